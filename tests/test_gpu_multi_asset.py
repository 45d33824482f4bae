"""Multi-asset books whose assets run in turn: observation slots in global memory where shared
memory would cap the CTAs, and the product sums laid out for the shape that keeps them shared.

The allocation-free entry point keeps the slots in shared memory, so the two entry points price
the same book on both layouts: every tile's FP32 sums are the same numbers, and only the FP64
sums over the CTAs differ in order (a few thousand terms: 1e-12 relative).
"""
import numpy as np
import pytest

import oracle
from thoth_gb300 import abi
from tests.test_gpu_parity import assert_shared_path_parity
from tests.test_zz_no_alloc import THREADS, _noalloc

pytestmark = pytest.mark.gpu


def book(models, n_products, paths, skip=0, steps=36):
    b = abi.Book(days=np.arange(steps + 1), paths=paths, sobol_skip=skip)
    for k, m in enumerate(models):
        if m == "gbm":
            b.add_gbm(90.0 + k, 0.2, 0.01)
            continue
        lev = None
        if m == "lsv":
            vals = 1.0 + 0.2 * np.sin(np.arange((steps + 1) * 12).reshape(steps + 1, 12))
            lev = (np.full(steps + 1, 0.05), np.full(steps + 1, 86, dtype=np.int64), vals)
        b.add_heston(90.0 + k, 0.05, 1.2, 0.05, 0.5, -0.5, 0.02, leverage=lev)
    na = len(models)
    for j in range(n_products):
        a, m = j % na, 1 + (7 * j) % steps
        kind = (j // na) % 4
        if kind == 0:
            b.add_vanilla(a, 95.0, m, abi.PUT if j % 2 else abi.CALL, zero_rate=0.02)
        elif kind == 1:
            b.add_barrier(a, 95.0, m, 80.0, up=False, knock_in=bool(j % 2), monitor=np.arange(1, m + 1), zero_rate=0.02,
                          quanto=0.01 * (j % 3))
        elif kind == 2:
            b.add_variance(a, m, strike_variance=0.04, notional=10.0, zero_rate=0.02)
        else:
            b.add_basket(list(range(na)), [1.0 / na] * na, 92.0, m, zero_rate=0.02)
    return b


@pytest.mark.parametrize("models,n_products,paths,skip", [
    (("lsv", "lsv"), 60, 4099, 0),              # no tile boundary at the last path
    (("gbm", "heston", "lsv"), 129, 2 ** 12, 5),  # more products than threads of a CTA
    (("heston", "gbm", "lsv", "lsv"), 300, 1000, 255),  # slots beyond what shared memory may hold
    (("lsv", "gbm"), 300, 1000, 255),  # more products than a tile has columns
    (("lsv", "heston"), 4, 300, 1),             # the few-product sums: slots stay shared
    (("lsv", "heston"), 5, 300, 1),
    (("heston",) * 8, 200, 513, 0),
    (("heston",) * 8, 40, 513, 0),
])
def test_assets_in_turn_slots_in_either_memory(gpu, models, n_products, paths, skip):
    b = book(models, n_products, paths, skip)
    if n_products * len(models) > 1000:  # refused wherever its slots would go
        with pytest.raises(gpu.ThothGpuError) as e:
            gpu.price_book(b)
        assert e.value.code == abi.THOTH_GPU_E_TOO_LARGE
        return
    if n_products > 256:
        b = book(models, n_products, paths, skip, steps=20)
    r = gpu.price_book(b)
    ref = oracle.price_book(b, threads=THREADS)
    assert_shared_path_parity(r, ref["premium"], ref["trust"], "book", scale=1.0)
    shared = _noalloc(gpu, b)
    for k in ("premium", "trust", "book_premium", "book_trust"):
        np.testing.assert_allclose(r[k], shared[k], rtol=1e-12, atol=1e-12)
    for x in gpu.price_batch([b, book(models, 6, 200), b]):  # both books' slots in one batch buffer
        if len(x["premium"]) == n_products:
            assert np.array_equal(x["premium"], r["premium"]) and np.array_equal(x["trust"], r["trust"])


def test_batch_slots_are_held_once_a_stream(gpu):
    """Slots in global memory are a book's only while its kernel runs: a larger batch of such books
    takes more plans, words and rows, but no more slots than its streams do, and prices as alone."""
    import torch

    def batch(n):
        return [book(("lsv", "heston", "lsv", "gbm", "lsv"), 50, 2 ** 18, skip=k) for k in range(n)]

    def grown(n):
        gpu.debug_fail_allocations(0)  # drops the engine's working buffers
        before = torch.cuda.mem_get_info()[0]
        res = gpu.price_batch(batch(n))
        return before - torch.cuda.mem_get_info()[0], res

    b = batch(1)[0]
    s = gpu.plan_summary(b)
    assert s["variant"] == 6 and s["slots"] > 40
    gpu.price_batch(batch(2))
    # 1025 tiles on 513 CTAs at least (two tiles each)
    slots = 4 * 257 * s["slots"] * 513
    small, _ = grown(16)
    large, res = grown(48)
    assert large - small < 32 * slots / 2, (small, large, slots)
    one = gpu.price_book(b)
    np.testing.assert_array_equal(res[0]["premium"], one["premium"])
    last = gpu.price_book(batch(48)[47])
    np.testing.assert_array_equal(res[47]["premium"], last["premium"])
