"""The exercise fit at the edges of its shares of paths, in shared and in global memory.

A CTA walks a run of whole 32-path chunks, split over its warps; the paths' cashflows and lists are
in shared memory where they fit (about 1.3 million paths of one contract on 152 SMs) and in global
memory beyond. The sums are exact and the arithmetic the reference's, so every case equals the
oracle on the stored paths bit for bit.
"""
import numpy as np
import pytest

from oracle import american as am
from thoth_gb300 import abi
from tests.test_gpu_american import DAYS, assert_same_fit, rates_of, vanilla_book

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths,K,typ,model", [
    (2, 100.0, abi.PUT, "gbm"),
    (31, 100.0, abi.PUT, "gbm"),
    (33, 103.7, abi.PUT, "heston"),             # a strike that is no float, a normaliser of 53 bits
    (129, 100.0, abi.CALL, "gbm"),              # a second CTA of one path
    (128 * 152, 96.25, abi.PUT, "heston"),      # one chunk a scheduler on every SM
    (128 * 152 + 1, 96.25, abi.CALL, "heston"),
    (100003, 99.9, abi.PUT, "gbm"),
    (60000, 260.0, abi.PUT, "gbm"),             # every path in the money, most below half the strike
    (700000, 100.0, abi.PUT, "heston"),
])
def test_fit_over_ragged_shares(gpu, paths, K, typ, model):
    b = vanilla_book(K=K, typ=typ, model=model, paths=paths, r=0.08 if typ == abi.PUT else 0.02)
    if typ == abi.CALL:
        b.assets[0]["carry"] = b.assets[0]["carry"] - 0.06
    r = gpu.price_american(b, 0, min_itm=5)
    S, _ = gpu.simulate_paths(b, 0)
    o = am.fit(S, b.t, rates_of(b), K, typ == abi.CALL, K, min_itm=5)
    if o["has_fit"].any():
        assert_same_fit(r, o, b.n_dates)
    else:
        assert r["fitted_dates"] == 0 and r["premium"] == o["premium"]


def test_fit_of_paths_in_global_memory(gpu):
    b = vanilla_book(paths=1500001, days=[0, 100, 200, 300, 365])
    r = gpu.price_american(b, 0)
    S, _ = gpu.simulate_paths(b, 0)
    assert_same_fit(r, am.fit(S, b.t, rates_of(b), 100.0, False, 100.0), b.n_dates)


@pytest.mark.parametrize("paths,n", [(20001, 3), (120000, 20)])  # shared; the 20 contracts' paths global
def test_contracts_that_share_a_fit(gpu, paths, n):
    b = abi.Book(days=np.asarray(DAYS), paths=paths)
    a = b.add_gbm(100.0, 0.30, 0.06)
    for k in range(n):
        b.add_vanilla(a, 80.0 + 2.37 * k, [13, 1, 7, 2][k % 4], abi.PUT if k % 3 else abi.CALL, zero_rate=0.06)
    together = gpu.price_american_book(b, list(range(n)))
    S, _ = gpu.simulate_paths(b, 0)
    for p in range(n):
        P = b.products[p]
        M = P["maturity"] + 1
        o = am.fit(S[:M], b.t, rates_of(b), P["strike"], P["option_type"] == abi.CALL, P["strike"])
        assert together[p]["premium"] == o["premium"] and together[p]["european"] == o["european"], p
        assert together[p]["fitted_dates"] == int(o["has_fit"].sum())
        np.testing.assert_array_equal(together[p]["beta"][:M][o["has_fit"]], o["beta"][o["has_fit"]])


@pytest.mark.parametrize("paths,n,days,K,carry", [
    (2, 1, DAYS, 1.0, 0.0),                              # one CTA, out of range on the first date walked
    (128 * 152, 1, range(0, 91), 1.0, 0.0),              # every SM
    (128 * 152 + 5, 1, range(0, 91), 1000.0 / 516, -2.0),  # in range at maturity, past it on the way to today
    (300000, 3, range(0, 61), 1000.0 / 516, -2.0),       # contracts that share the launch
    (120000, 20, range(0, 31), 1000.0 / 516, -2.0),      # paths in global memory
])
def test_moneyness_out_of_range_ends_the_fit(gpu, paths, n, days, K, carry):
    """A call far in the money (m = S / K >= 512, so m^4 >= 2^36) is refused, whichever date and CTA
    meets it first: every CTA's walkers and both its waiting warps leave the launch, on every repeat,
    and the next fit is the same as before."""
    good = vanilla_book(paths=5000)
    before = gpu.price_american(good, 0)
    b = abi.Book(days=np.asarray(list(days)), paths=paths)
    a = b.add_gbm(1000.0, 0.3, carry)
    for k in range(n):
        b.add_vanilla(a, K * (1.0 + 0.001 * k), b.n_dates - 1 - k % 3, abi.CALL, zero_rate=0.02)
    for _ in range(20):
        with pytest.raises(gpu.ThothGpuError) as e:
            gpu.price_american_book(b, list(range(n)), min_itm=1)
        assert e.value.code == abi.THOTH_GPU_E_INVALID
    after = gpu.price_american(good, 0)
    assert after["premium"] == before["premium"] and after["trust"] == before["trust"]
    np.testing.assert_array_equal(after["beta"], before["beta"])


@pytest.mark.parametrize("K,typ", [(55.0, abi.PUT), (260.0, abi.PUT), (99.9, abi.CALL)])
def test_lists_of_every_length_in_global_memory(gpu, K, typ):
    """Few, all and half of the paths in the money: blocks that are requested ahead of the walk end
    inside, at and past a warp's share of the paths and of its list."""
    b = vanilla_book(K=K, typ=typ, paths=1400003, days=[0, 120, 240, 365], r=0.08 if typ == abi.PUT else 0.02)
    if typ == abi.CALL:
        b.assets[0]["carry"] = b.assets[0]["carry"] - 0.06
    r = gpu.price_american(b, 0)
    S, _ = gpu.simulate_paths(b, 0)
    assert_same_fit(r, am.fit(S, b.t, rates_of(b), K, typ == abi.CALL, K), b.n_dates)
