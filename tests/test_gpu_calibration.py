"""LSV leverage calibration on the device (thoth_gpu_calibrate_leverage).

* layers against the oracle (Single::CalibrateLeverage restated, on the reference's Rng
  stream): the device draws the same stream, rounds every expression as the reference does
  and sums exactly, so the ensembles differ only where CUDA's exp / log / erfc differ from
  the host libm in the last bit;
* the reference test's degenerate limit (pricer/tests/test_lsv.cpp:77-103): flat 25 % target
  on a 30 % Heston base with vanishing vol of vol gives 25 / 30, and the calibrated LSV call
  prices at Black-Scholes 25 %;
* the defining property (test_lsv.cpp:42-60): LSV with the calibrated leverage reprices the
  target local-vol model's vanillas across strikes, within MC error plus the binned-particle
  bias the reference allows (0.10). The target is priced by the same engine as a local-vol
  model (an LSV asset whose variance stays at 1 and whose leverage is the local vol).
"""
import math

import numpy as np
import pytest

import oracle
from thoth_gb300 import abi, workloads as W

pytestmark = pytest.mark.gpu


def test_layers_match_the_oracle(gpu):
    c = W.lsv_calibration(horizon_days=90)
    L, ms = gpu.calibrate_leverage(c)
    ref = oracle.calibrate_leverage(c)
    assert ms > 0
    np.testing.assert_allclose(L, ref, rtol=1e-9, atol=0)


def test_layers_match_the_oracle_uneven_dates_and_particles(gpu):
    c = W.lsv_calibration(horizon_days=45, particles=5000)
    c.days = np.ascontiguousarray(np.r_[0, 1, 2, 5, 9, 14, 30, 45], dtype=np.int32)
    ls, off = W.layer_grids(c.days, 100.0, 0.22)
    c.ln_step, c.offset = ls, off
    x = (off[:, None] + np.arange(201)[None, :]) * ls[:, None]
    c.local_vol = np.ascontiguousarray(W.skew_local_vol(np.exp(x), (c.days / 365.0)[:, None]))
    c.carry = np.ascontiguousarray(np.linspace(0.01, 0.03, len(c.days)))
    c.leverage = np.zeros_like(c.local_vol)
    L, _ = gpu.calibrate_leverage(c)
    np.testing.assert_allclose(L, oracle.calibrate_leverage(c), rtol=1e-9, atol=0)


def test_degenerate_limit_prices_black_scholes(gpu):
    h = dict(v0=0.09, kappa=3.0, theta=0.09, xi=1e-4, rho=0.0)
    c = W.lsv_calibration(horizon_days=365, local_vol=lambda S, t: np.full(np.broadcast(S, t).shape, 0.25),
                          heston=h, carry=0.05)
    L, _ = gpu.calibrate_leverage(c)
    np.testing.assert_allclose(L, 0.25 / 0.30, rtol=2e-3)
    b = abi.Book(days=c.days, paths=200000)
    a = b.add_heston(100.0, h["v0"], h["kappa"], h["theta"], h["xi"], h["rho"], 0.05,
                     leverage=(c.ln_step, c.offset, L))
    b.add_vanilla(a, 100.0, 365, abi.CALL, zero_rate=0.05)
    r = gpu.price_book(b)
    bs = oracle.bs_price(100.0 * math.exp(0.05), 100.0, 1.0, 0.25, math.exp(-0.05), True)
    assert abs(r["premium"][0] - bs) <= 6.0 * r["trust"][0] + 0.06


def test_calibrated_lsv_reprices_the_local_vol_model(gpu):
    c = W.lsv_calibration(horizon_days=365)
    L, _ = gpu.calibrate_leverage(c)
    h = c.heston
    strikes = (80.0, 100.0, 120.0)

    def book(local_model):
        b = abi.Book(days=c.days, paths=1 << 18)
        if local_model:      # variance pinned at 1: the leverage is the local vol itself
            a = b.add_heston(100.0, 1.0, 1.0, 1.0, 1e-9, 0.0, 0.02, leverage=(c.ln_step, c.offset, c.local_vol))
        else:
            a = b.add_heston(100.0, h["v0"], h["kappa"], h["theta"], h["xi"], h["rho"], 0.02,
                             leverage=(c.ln_step, c.offset, L))
        for K in strikes:
            b.add_vanilla(a, K, 365, abi.PUT if K < 100 else abi.CALL, zero_rate=0.02)
        return b

    lv = gpu.price_book(book(True))
    lsv = gpu.price_book(book(False))
    for i, K in enumerate(strikes):
        se = math.hypot(lv["trust"][i], lsv["trust"][i])
        assert abs(lsv["premium"][i] - lv["premium"][i]) <= 6.0 * se + 0.10, (K, lsv["premium"][i], lv["premium"][i])
    # and the Heston base alone does not: the leverage is doing the work
    plain = abi.Book(days=c.days, paths=1 << 18)
    a = plain.add_heston(100.0, h["v0"], h["kappa"], h["theta"], h["xi"], h["rho"], 0.02)
    for K in strikes:
        plain.add_vanilla(a, K, 365, abi.PUT if K < 100 else abi.CALL, zero_rate=0.02)
    pr = gpu.price_book(plain)
    miss = [abs(pr["premium"][i] - lv["premium"][i]) - 6.0 * math.hypot(pr["trust"][i], lv["trust"][i]) - 0.10
            for i in range(len(strikes))]
    assert max(miss) > 0.0, miss


def test_invalid_inputs(gpu):
    c = W.lsv_calibration(horizon_days=10, particles=1024)
    c.bins = 500
    with pytest.raises(gpu.ThothGpuError) as e:
        gpu.calibrate_leverage(c)
    assert e.value.code == abi.THOTH_GPU_E_INVALID
    c = W.lsv_calibration(horizon_days=10, particles=1024)
    c.days = np.ascontiguousarray(c.days[::-1])
    with pytest.raises(gpu.ThothGpuError):
        gpu.calibrate_leverage(c)


@pytest.mark.parametrize("particles,bins,min_count", [(1000, 30, 20), (700, 12, 100), (4099, 1, 1)])
def test_uneven_ensembles_and_thin_bins_match_the_oracle(gpu, particles, bins, min_count):
    """Particle counts off the warp size, every bin thin (the ensemble mean everywhere), and
    one bin: the device follows the oracle."""
    c = W.lsv_calibration(horizon_days=30, particles=particles)
    c.bins, c.min_bin_count = bins, min_count
    L, _ = gpu.calibrate_leverage(c)
    np.testing.assert_allclose(L, oracle.calibrate_leverage(c), rtol=1e-9, atol=0)


@pytest.mark.parametrize("particles,points", [
    (16384, 2),          # the smallest layer
    (129, 201),          # one particle more than a CTA
    (77825, 64),         # more than one a thread: the ensemble in memory
])
def test_ensemble_and_layer_edges_match_the_oracle(gpu, particles, points):
    """The particles' places (registers, memory), a CTA with one particle, and the smallest layer,
    against the oracle; rounding differences alone, as in the tests above."""
    c = W.lsv_calibration(horizon_days=6, particles=particles)
    c.local_vol = np.ascontiguousarray(c.local_vol[:, (201 - points) // 2:][:, :points])
    c.offset = np.ascontiguousarray(c.offset + (201 - points) // 2)
    c.leverage = np.zeros_like(c.local_vol)
    L, _ = gpu.calibrate_leverage(c)
    np.testing.assert_allclose(L, oracle.calibrate_leverage(c), rtol=1e-9, atol=0)


def test_vanishing_vol_of_vol_keeps_its_errors_and_limits(gpu):
    """xi = 0 leaves no variance (psi = 0): refused, as the step's ratio is not a number; a tiny xi
    is the deterministic variance (the exact limit of the step)."""
    for xi, ok in ((0.0, False), (1e-100, True), (1e-13, True)):
        c = W.lsv_calibration(horizon_days=5, particles=1024, heston=dict(v0=0.04, kappa=1.0, theta=0.04, xi=xi, rho=0.0))
        if not ok:
            with pytest.raises(gpu.ThothGpuError):
                gpu.calibrate_leverage(c)
            continue
        L, _ = gpu.calibrate_leverage(c)
        np.testing.assert_allclose(L, oracle.calibrate_leverage(c), rtol=1e-9, atol=0)


@pytest.mark.parametrize("particles", [300, 16384, 60000, 200000])  # few CTAs, most of the SMs, every one, in memory
@pytest.mark.parametrize("heston", [
    dict(v0=0.04, kappa=1.0, theta=0.04, xi=0.0, rho=0.0),  # no variance after the first step, on every CTA
    dict(v0=1e9, kappa=2.0, theta=1e12, xi=1e5, rho=0.0),   # past 2^36 after some two weeks, CTA by CTA
])
def test_variance_out_of_range_ends_the_calibration(gpu, particles, heston):
    """A variance that is not a number or past 2^36 is refused, whichever CTA meets it first and
    wherever the others' waits are, on every repeat; the next calibration is the same as before."""
    good = W.lsv_calibration(horizon_days=10, particles=particles)
    before, _ = gpu.calibrate_leverage(good)
    before = np.array(before)
    for _ in range(20):
        c = W.lsv_calibration(horizon_days=40, particles=particles, heston=heston)
        with pytest.raises(gpu.ThothGpuError) as e:
            gpu.calibrate_leverage(c)
        assert e.value.code == abi.THOTH_GPU_E_INVALID
    after, _ = gpu.calibrate_leverage(good)
    np.testing.assert_array_equal(after, before)


def test_particles_lost_to_a_missing_local_vol_leave_the_others_as_they_are(gpu):
    """Local vols that are not a number far below the money: the particles that come there are lost
    (as the oracle's are), and the extremes, the bins and the layers of the others do not see them."""
    c = W.lsv_calibration(horizon_days=30)
    x = (c.offset[:, None] + np.arange(c.local_vol.shape[1])[None, :]) * c.ln_step[:, None]
    c.local_vol = np.where(x < math.log(100.0) - 0.12, np.nan, c.local_vol)
    L, _ = gpu.calibrate_leverage(c)
    ref = oracle.calibrate_leverage(c)
    assert np.isfinite(ref).any(axis=1).all() and np.isnan(ref).any()
    np.testing.assert_allclose(L, ref, rtol=1e-9, atol=0, equal_nan=True)


def test_an_ensemble_lost_at_once_ends_at_the_upper_bound(gpu):
    """Every particle outside the layer, at an end that has no local vol: no particle is left to form
    a conditional variance, and the layers behind are the least variance's, at the upper bound."""
    c = W.lsv_calibration(horizon_days=6, particles=300)
    c.offset = np.ascontiguousarray(c.offset + 1000)  # the grid lies above the ensemble
    c.local_vol[2, 0] = np.nan
    L, _ = gpu.calibrate_leverage(c)
    assert np.isnan(L[2, 0]) and np.isfinite(L[:2]).all()
    assert (L[3:] == 10.0).all()
