"""Books whose launch is small (at most three CTAs an SM), which run a kernel of their own.

Its sums are those of the ordinary kernel bit for bit, so each book is compared with the same book
priced in a batch, whose kernel has no small form (equal bits), with the entry point on the
caller's memory, which never takes the small form (1e-12: sums of the same FP32 rows), and with the
oracle on the same paths where that is quick.
"""
import os

import numpy as np
import pytest

import oracle
from thoth_gb300 import abi
from tests.test_gpu_multi_asset import _noalloc
from tests.test_gpu_parity import assert_shared_path_parity

pytestmark = pytest.mark.gpu

THREADS = max(1, min(16, os.cpu_count() or 1))
LINE = 3 * 152 * 256  # the last path count that fits three 256-path CTAs on each of 152 SMs


def book(models, paths, steps, uniform=True, skip=0, sobol=True):
    days = np.arange(steps + 1) if uniform else np.cumsum(np.r_[0, 1 + np.arange(steps) % 3])
    b = abi.Book(days=days, paths=paths, sobol_skip=skip, use_sobol=sobol)
    for k, m in enumerate(models):
        if m == "gbm":
            b.add_gbm(95.0 + k, 0.2, 0.01)
            continue
        lev = None
        if m == "lsv":
            vals = 1.0 + 0.2 * np.sin(np.arange((steps + 1) * 12).reshape(steps + 1, 12))
            lev = (np.full(steps + 1, 0.05), np.full(steps + 1, 86, dtype=np.int64), vals)
        b.add_heston(95.0 + k, 0.05, 1.2, 0.05, 0.5, -0.5, 0.02, leverage=lev)
        b.add_variance(k, steps, strike_variance=0.04, notional=10.0, zero_rate=0.02)
    for a in range(len(models)):
        for K in (85.0, 95.0, 105.0):
            b.add_vanilla(a, K, steps, abi.PUT, zero_rate=0.02)
        b.add_barrier(a, 95.0, steps, 80.0, up=False, knock_in=True, monitor=np.arange(1, steps + 1), zero_rate=0.02)
        b.add_vanilla(a, 95.0, max(1, steps // 2), abi.CALL, zero_rate=0.02)
    return b


@pytest.mark.parametrize("models,paths,steps,kw", [
    (("gbm",), 2, 1, {}),                                # fewer low words than the copies in flight
    (("heston",), 255, 2, dict(skip=3)),
    (("heston",), 300, 5, {}),                           # a second tile of a few paths
    (("lsv",), 257, 8, dict(uniform=False)),
    (("gbm",), LINE, 9, {}),                             # either side of the line of the dispatch
    (("gbm",), LINE + 1, 9, {}),
    (("heston",), LINE, 6, dict(uniform=False)),
    (("heston",), LINE + 1, 6, dict(uniform=False)),
    (("lsv",), LINE - 1, 6, {}),
    (("heston",), 40000, 255, dict(skip=12345)),         # tile parts in one chunk of 512, all but filled
    (("heston",), 40000, 256, {}),
    (("heston",), 4000, 257, {}),                        # and in two
    (("lsv",), 3000, 700, dict(uniform=False)),          # the step program stays in global memory
    (("gbm",), 3000, 2100, dict(uniform=False)),
    (("gbm",), 1500, 40, dict(sobol=False)),
    (("heston",), 513, 4200, {}),                        # beyond the Sobol dimensions
    (("heston", "gbm"), 5000, 30, {}),                   # assets in turn
    (("lsv", "heston", "gbm"), 777, 61, dict(uniform=False)),
])
def test_small_launch_has_the_ordinary_results(gpu, models, paths, steps, kw):
    b = book(models, paths, steps, **kw)
    r = gpu.price_book(b)
    pad = book(("gbm",), 300, 3)
    for x in gpu.price_batch([b, pad])[:1]:
        np.testing.assert_array_equal(r["premium"], x["premium"])
        np.testing.assert_array_equal(r["trust"], x["trust"])
        assert r["book_premium"] == x["book_premium"] and r["book_trust"] == x["book_trust"]
    try:
        own = _noalloc(gpu, b)
    except gpu.ThothGpuError as e:  # the longest books' tables exceed the fixed scratch
        assert e.code == abi.THOTH_GPU_E_TOO_LARGE and steps > 2000
        own = r
    for k in ("premium", "trust", "book_premium", "book_trust"):
        np.testing.assert_allclose(r[k], own[k], rtol=1e-12, atol=1e-12)
    if paths * steps <= 2000000 and kw.get("sobol", True) and steps < 2000:
        ref = oracle.price_book(b, threads=THREADS)
        assert_shared_path_parity(r, ref["premium"], ref["trust"], "book", scale=1.0)
