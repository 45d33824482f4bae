"""Cooperative cancellation (thoth_gpu_request_cancel): a cancel requested before a call ends every
book-pricing entry point without its launches, and after thoth_gpu_clear_cancel the same calls give
the same results; a cancel requested while a call runs ends that call.
"""
import threading
import time

import numpy as np
import pytest

from thoth_gb300 import abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def cancel(gpu):
    yield gpu.lib().thoth_gpu_request_cancel
    assert gpu.lib().thoth_gpu_clear_cancel() == abi.THOTH_GPU_OK


def one_tile_a_cta():
    """912 tiles of 256 paths: every CTA of the Heston kernel (six an SM) has one, a long one."""
    b = abi.Book(days=np.arange(2001), paths=912 * 256 - 1)
    a = b.add_heston(100.0, 0.04, 1.5, 0.04, 0.6, -0.7, 0.03)
    b.add_vanilla(a, 100.0, 2000, abi.CALL, zero_rate=0.03)
    return b


def refused(gpu, call):
    with pytest.raises(gpu.ThothGpuError) as e:
        call()
    assert e.value.code == abi.THOTH_GPU_E_CANCELLED


def test_a_cancel_before_the_call_launches_nothing(gpu, cancel):
    b = one_tile_a_cta()
    r = gpu.ResidentBook(b)
    first = r.run()
    full = min(r.run()["device_ms"] for _ in range(3)) * 1e-3
    assert cancel() == abi.THOTH_GPU_OK
    took = []
    for _ in range(5):
        t0 = time.perf_counter()
        refused(gpu, r.run)
        took.append(time.perf_counter() - t0)
    assert min(took) < 0.25 * full, (took, full)
    for call in (lambda: gpu.price_book(b), lambda: gpu.simulate_paths(W.gbm_call(paths=1000, greeks=False), 0),
                 lambda: gpu.bump_greeks(W.heston_grid(paths=1000)), lambda: gpu.autotune_book(b),
                 lambda: gpu.price_american(W.american_put(paths=1000), 0)):
        refused(gpu, call)
    assert gpu.lib().thoth_gpu_clear_cancel() == abi.THOTH_GPU_OK
    again = r.run()
    np.testing.assert_array_equal(again["premium"], first["premium"])
    np.testing.assert_array_equal(again["trust"], first["trust"])


def test_a_cancel_before_a_batch_replays_nothing(gpu, cancel):
    books = [W.heston_grid(paths=1 << 12), W.gbm_call(paths=1 << 13, greeks=False), W.lsv_book(paths=2000)]
    first = gpu.price_batch(books)
    gpu.price_batch(books)
    replays = gpu.batch_graph_replays()
    assert cancel() == abi.THOTH_GPU_OK
    refused(gpu, lambda: gpu.price_batch(books))
    assert gpu.batch_graph_replays() == replays
    assert gpu.lib().thoth_gpu_clear_cancel() == abi.THOTH_GPU_OK
    for a, f in zip(gpu.price_batch(books), first):
        np.testing.assert_array_equal(a["premium"], f["premium"])


@pytest.mark.parametrize("batch", [False, True])
def test_a_cancel_while_the_call_runs_ends_it(gpu, cancel, batch):
    """A call of many tiles a CTA (and, in a batch, many items a CTA), cancelled from another thread."""
    def call():
        if batch:
            return gpu.price_batch([W.heston_grid(paths=1 << 20 | k) for k in range(8)])
        b = one_tile_a_cta()
        b.paths *= 60
        return gpu.price_book(b)

    errors = []

    def run():
        try:
            while True:  # a request that lands between two calls ends the next one
                call()
        except gpu.ThothGpuError as e:
            errors.append(e.code)

    th = threading.Thread(target=run)
    th.start()
    time.sleep(0.5)
    assert cancel() == abi.THOTH_GPU_OK
    th.join(60)
    assert not th.is_alive() and errors == [abi.THOTH_GPU_E_CANCELLED]
