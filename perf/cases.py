"""Performance cases of the Monte-Carlo engine: what a user's program has it do.

Every case is one call (for training: one model's whole training) through the public Python
entry points of thoth_gb300, on seeded synthetic inputs of the engine's workloads
(thoth_gb300/workloads.py, thoth_gb300/surrogate.py). Books, calibration inputs and training
sets are host data by nature: the caller describes a book, the engine plans it, uploads it,
prices it and returns the sums, and all of that is a pass.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the inputs a program has in hand
  run(state)          one pass
  work(case)          bytes and operations the pass cannot do without
  exact(case, seed)   the pass's outputs in 64 bits, in plain torch and numpy
"""
import math
import pathlib

import numpy as np
import torch

import thoth_gb300 as G
from thoth_gb300 import abi, surrogate
from thoth_gb300 import workloads as W

FP64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one European call under GBM with pathwise delta and vega: the smallest call a pricing
        # server answers, one time step, where launches and host work are most of it
        dict(name="gbm_call", kind="book", model="gbm", payoff="call", paths=1 << 18, steps=1, greeks=True),
        # a Heston vanilla surface, 9 strikes x 7 maturities x call/put on 2^20 paths x 504 steps:
        # the benchmark workload
        dict(name="heston_grid", kind="grid", paths=1 << 20, months=24, maturities=7, strikes=9, calendar=False),
        # an ordinary request: a ragged path count, the calendar's daily steps, few strikes
        dict(name="heston_surface", kind="grid", paths=100003, months=12, maturities=4, strikes=5, calendar=True),
        # daily-monitored barriers on one name with a leverage surface
        dict(name="lsv_barriers", kind="book", model="lsv", payoff="barrier", paths=300001, steps=251, greeks=False),
        # a desk's book: 5 LSV names, 20 barriers, 10 variance swaps, 20 baskets, a year of daily dates
        dict(name="lsv_book", kind="lsv_book", paths=1 << 20, strikes=50, times=40, greeks=False),
        # an overnight batch of unequal single-name books in one call
        dict(name="ragged_batch", kind="batch", books=48, min_paths=1 << 14, max_paths=1 << 21, max_steps=730),
        # risk: every bump-and-revalue Greek of a Heston book of vanillas, a barrier and a variance swap
        dict(name="bump_greeks", kind="bump", model="heston", paths=1 << 18, steps=180),
        # American put on the monthly exercise grid, 300 000 GBM paths, all Greeks
        dict(name="american_monthly", kind="american", model="gbm", paths=300000, days=365, every=30, greeks=True),
        # American put with a year of daily exercise on 2^20 Heston paths
        dict(name="american_daily", kind="american", model="heston", paths=1 << 20, days=365, every=1, greeks=False),
        # the leverage surface of an LSV name, daily layers over a year, the default ensemble
        dict(name="lsv_calibration", kind="calibration", particles=16384, days=365),
        # training of one surrogate network (forward, backward and Adam): lattice labels of 512
        # parameter sets, 20 epochs
        dict(name="surrogate_train", kind="train", rows=512 * 252, batch=8192, epochs=20),
        # serving: a million cells of the surface by the mean of four networks
        dict(name="surrogate_lattice", kind="lattice", members=4, sets=4096, strikes=21, maturities=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["book", "grid", "lsv_book", "batch", "bump", "american", "calibration", "train", "lattice"])
    if kind == "book":
        model = rng.choice(["gbm", "heston", "lsv"])
        payoff = rng.choice(["call", "vanilla", "barrier", "variance"])
        return dict(kind=kind, model=model, payoff=payoff, paths=_log_int(rng, 1 << 14, 1 << 21),
                    steps=_log_int(rng, 1, 730), greeks=payoff == "call" and rng.random() < 0.5)
    if kind == "grid":
        months = rng.choice([3, 6, 12, 24])
        return dict(kind=kind, paths=_log_int(rng, 1 << 14, 1 << 20), months=months,
                    maturities=rng.randint(2, 7), strikes=rng.randint(1, 9), calendar=rng.random() < 0.5)
    if kind == "lsv_book":
        return dict(kind=kind, paths=_log_int(rng, 1 << 14, 1 << 20), strikes=rng.randint(20, 80),
                    times=rng.randint(4, 40), greeks=rng.random() < 0.25)
    if kind == "batch":
        return dict(kind=kind, books=rng.randint(5, 48), min_paths=1 << 14,
                    max_paths=_log_int(rng, 1 << 16, 1 << 20), max_steps=rng.choice([252, 365, 730]))
    if kind == "bump":
        return dict(kind=kind, model=rng.choice(["gbm", "heston"]), paths=_log_int(rng, 1 << 14, 1 << 18),
                    steps=rng.randint(30, 250))
    if kind == "american":
        every = rng.choice([1, 7, 30])
        return dict(kind=kind, model=rng.choice(["gbm", "heston"]), paths=_log_int(rng, 1 << 14, 1 << 19),
                    days=rng.randint(180, 365), every=every, greeks=rng.random() < 0.5)
    if kind == "calibration":
        return dict(kind=kind, particles=_log_int(rng, 4096, 65536), days=rng.randint(60, 365))
    if kind == "train":
        batch = rng.choice([1024, 2048, 4096, 8192, 16384])
        return dict(kind=kind, rows=batch * rng.randint(1, max(1, 131072 // batch)) + rng.randint(0, 127), batch=batch,
                    epochs=rng.randint(2, 12))
    return dict(kind=kind, members=rng.randint(1, 4), sets=_log_int(rng, 1, 4096), strikes=rng.randint(5, 21),
                maturities=rng.randint(2, 12))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _heston(rng):
    """Parameters around the benchmark's (kappa 1.5, theta 0.04, xi 0.6, rho -0.7, v0 0.04)."""
    u = rng.uniform(0.95, 1.05, 5)
    return dict(v0=0.04 * u[0], kappa=1.5 * u[1], theta=0.04 * u[2], xi=0.6 * u[3], rho=-0.7 * u[4])


def _add_asset(b, model, rng, carry):
    if model == "gbm":
        return b.add_gbm(100.0, 0.25 * rng.uniform(0.95, 1.05), carry)
    lev = None
    if model == "lsv":
        nd = b.n_dates
        step = (math.log(250.0) - math.log(30.0)) / 49
        surf = W._smooth(rng.uniform(0.7, 1.3, size=(8, 50)))
        lev = (np.full(nd, step), np.full(nd, int(math.floor(math.log(30.0) / step)), dtype=np.int64),
               surf[np.minimum(np.arange(nd) * 8 // nd, 7)])
    return b.add_heston(100.0, carry=carry, leverage=lev, **_heston(rng))


def _book(c, rng):
    n = c["steps"]
    days = [0, 365] if n == 1 else np.arange(n + 1)
    b = abi.Book(days=days, paths=c["paths"], greeks=(abi.GREEK_DELTA | abi.GREEK_VEGA) if c["greeks"] else 0)
    r = 0.03 * rng.uniform(0.9, 1.1)
    a = _add_asset(b, c["model"], rng, r - 0.01)
    if c["payoff"] == "call":
        b.add_vanilla(a, 100.0, n, abi.CALL, zero_rate=r)
    elif c["payoff"] == "vanilla":
        for k in (90.0, 100.0, 110.0):
            b.add_vanilla(a, k, n, abi.CALL, zero_rate=r)
            b.add_vanilla(a, k, n, abi.PUT, zero_rate=r)
    elif c["payoff"] == "barrier":
        mon = np.arange(1, n + 1)
        b.add_barrier(a, 100.0, n, 80.0, up=False, knock_in=False, monitor=mon, zero_rate=r)
        b.add_barrier(a, 100.0, n, 120.0, up=True, knock_in=True, monitor=mon, option_type=abi.PUT, zero_rate=r)
    else:
        b.add_variance(a, n, strike_variance=0.04, notional=100.0, zero_rate=r)
    return b


def _grid(c, rng):
    months = sorted({max(1, round(c["months"] * (j + 1) / c["maturities"])) for j in range(c["maturities"])})
    strikes = np.linspace(80.0, 120.0, c["strikes"]) if c["strikes"] > 1 else [100.0]
    if c["calendar"]:
        mats = [round(365 * m / 12) for m in months]
        b = abi.Book(days=np.arange(mats[-1] + 1), paths=c["paths"])
    else:
        mats = [21 * m for m in months]
        b = abi.Book(times=np.arange(mats[-1] + 1) / 252.0, paths=c["paths"])
    r = 0.03 * rng.uniform(0.9, 1.1)
    a = _add_asset(b, "heston", rng, r)
    for m in mats:
        for k in strikes:
            for typ in (abi.CALL, abi.PUT):
                b.add_vanilla(a, float(k), m, typ, zero_rate=r)
    return b


def _bump_book(c, rng):
    n = c["steps"]
    b = abi.Book(days=np.arange(n + 1), paths=c["paths"])
    r = 0.03 * rng.uniform(0.9, 1.1)
    a = _add_asset(b, c["model"], rng, r - 0.01)
    for k in (90.0, 100.0, 110.0):
        b.add_vanilla(a, k, n, abi.CALL, zero_rate=r)
        b.add_vanilla(a, k, n // 2, abi.PUT, zero_rate=r)
    b.add_barrier(a, 100.0, n, 80.0, up=False, knock_in=False, monitor=np.arange(1, n + 1), zero_rate=r)
    b.add_variance(a, n, strike_variance=0.04, notional=100.0, zero_rate=r)
    return b


def _american_book(c, rng):
    days = list(range(0, c["days"], c["every"]))
    b = abi.Book(days=np.asarray(days + [c["days"]]), paths=c["paths"])
    r = 0.03 * rng.uniform(0.9, 1.1) if c["model"] == "heston" else 0.08 * rng.uniform(0.9, 1.1)
    a = _add_asset(b, c["model"], rng, r)
    b.add_vanilla(a, 100.0, b.n_dates - 1, abi.PUT, zero_rate=r)
    return b


def _calibration(c, rng, seed):
    h = dict(v0=0.0324, kappa=2.0, theta=0.0676, xi=0.5, rho=-0.6)
    h = {k: v * rng.uniform(0.97, 1.03) for k, v in h.items()}
    return W.lsv_calibration(horizon_days=c["days"], particles=c["particles"], heston=h, seed=1 + seed)


def _sets(n, rng):
    """Heston parameter sets over the surrogate's training box."""
    lo, hi = surrogate.BOX_LO[2:], surrogate.BOX_HI[2:]
    return lo + rng.random((n, 5)) * (hi - lo)


H, KIN, NF = 128, 16, 7  # the network: 7 inputs (in 16 columns) -> 4 x 128 SiLU -> 1


def _weights(rng):
    """A network's parameters (Xavier-uniform, small biases) in the model's flat layout: W1 [128][16]
    (columns f and f + 7 hold input f's weight, the last two are empty), b1, then W, b of the
    hidden layers, then the head."""
    def u(rows, cols, fan):
        return rng.uniform(-1, 1, (rows, cols)) * math.sqrt(6.0 / (fan + rows))
    w1 = np.zeros((H, KIN))
    w1[:, :NF] = u(H, NF, NF)
    w1[:, NF:2 * NF] = w1[:, :NF]
    parts = [w1.ravel(), rng.uniform(-0.1, 0.1, H)]
    for _ in range(3):
        parts += [u(H, H, H).ravel(), rng.uniform(-0.1, 0.1, H)]
    parts += [u(1, H, H).ravel(), rng.uniform(-0.1, 0.1, 1)]
    return np.concatenate(parts).astype(np.float32)


def _training_set(c, rng):
    """Normalised inputs, targets and loss scales of the shape surrogate.train_targets() gives:
    a smooth O(1) target of the features with a little label noise."""
    x = rng.uniform(-1, 1, (c["rows"], NF)).astype(np.float32)
    y = 1.0 + 0.2 * np.sin(2 * x[:, 0] + x[:, 1]) + 0.1 * x[:, 2] * x[:, 6] + 1e-3 * rng.standard_normal(c["rows"])
    return x, y.astype(np.float32), rng.uniform(0.5, 1.5, c["rows"]).astype(np.float32)


def _axes(c):
    return np.linspace(-0.5, 0.5, c["strikes"]), np.linspace(1 / 12.0, 3.0, c["maturities"])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "book":
        s["book"] = _book(case, rng)
    elif kind == "grid":
        s["book"] = _grid(case, rng)
    elif kind == "lsv_book":
        s["book"] = _lsv_book(case, seed)
    elif kind == "batch":
        s["books"] = _batch(case, seed)
    elif kind == "bump":
        s["book"] = _bump_book(case, rng)
    elif kind == "american":
        s["book"] = _american_book(case, rng)
    elif kind == "calibration":
        s["calib"] = _calibration(case, rng, seed)
    elif kind == "train":
        s["p0"], s["set"] = _weights(rng), _training_set(case, rng)
        s["seed"] = seed
    else:
        s["sets"] = _sets(case["sets"], rng)
        s["model"] = surrogate.Ensemble(case["members"])
        for m in s["model"].members:
            m.set_params(_weights(rng))
    return s


def _lsv_book(case, seed):
    return W.lsv_book(paths=case["paths"], seed=seed, n_lev_strikes=case["strikes"], n_lev_times=case["times"],
                      greeks=case["greeks"])


def _batch(case, seed):
    """The ragged workload's mix. The sizes are the case's; the seed moves each book's parameters."""
    books = W.ragged_books(case["books"], seed=7, min_paths=case["min_paths"], max_paths=case["max_paths"],
                           max_steps=case["max_steps"])
    rng = np.random.default_rng(seed)
    for b in books:
        a = b.assets[0]
        for k in ("vol", "v0", "kappa", "theta", "xi", "rho"):
            if k in a:
                a[k] *= rng.uniform(0.95, 1.05)
    return books


SUMS = ("book_premium", "book_trust", "premium", "trust")
GREEKS = ("delta", "delta_trust", "vega", "vega_trust")


def run(state):
    kind = state["case"]["kind"]
    if kind in ("book", "grid", "lsv_book"):
        greeks = bool(state["book"].greeks)
        r = G.price_book(state["book"], greeks=greeks)
        return {k: r[k] for k in SUMS + (GREEKS if greeks else ())}
    if kind == "batch":
        rs = G.price_batch(state["books"])
        return {"book_premium": np.array([r["book_premium"] for r in rs]),
                "book_trust": np.array([r["book_trust"] for r in rs]),
                "premium": np.concatenate([r["premium"] for r in rs]),
                "trust": np.concatenate([r["trust"] for r in rs])}
    if kind == "bump":
        r = G.bump_greeks(state["book"])
        keys = ["premium", "delta", "gamma", "vega", "rho", "theta"]
        out = {k: r[k] for k in keys + ["vega_" + p for p in abi.PARAMS]}
        out["book"] = np.array([r["book"][k] for k in keys])
        return out
    if kind == "american":
        flags = abi.BUMP_DELTA | abi.BUMP_GAMMA | abi.BUMP_VEGA | abi.BUMP_RHO | abi.BUMP_THETA
        r = G.price_american(state["book"], 0, flags=flags if state["case"]["greeks"] else 0)
        keys = ["premium", "trust", "european"] + (["delta", "gamma", "vega", "rho", "theta"]
                                                   if state["case"]["greeks"] else [])
        return {**{k: r[k] for k in keys}, "beta": r["beta"], "fitted_dates": r["fitted_dates"]}
    if kind == "calibration":
        return G.calibrate_leverage(state["calib"])[0]
    if kind == "train":
        m = surrogate.Surrogate(seed=1)
        m.set_params(state["p0"])
        loss = m.train(*state["set"], epochs=state["case"]["epochs"], batch=state["case"]["batch"], lr=2e-3,
                       seed=state["seed"])
        out = {"params": m.params(), "loss": loss}
        m.close()
        return out
    return state["model"].price_lattice(state["sets"], *_axes(state["case"]))[0]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
PATH_STEP_FLOPS = dict(gbm=40, heston=96, lsv=112)  # per path and step: draws, bridge, step


def work(case):
    kind = case["kind"]
    if kind == "book":
        return dict(bytes=64.0 * case["steps"] + 1e3,
                    flops=float(case["paths"]) * case["steps"] * PATH_STEP_FLOPS[case["model"]])
    if kind == "grid":
        n = case["months"] * (21 if not case["calendar"] else 365 / 12)
        return dict(bytes=64.0 * n + 1e4, flops=case["paths"] * n * PATH_STEP_FLOPS["heston"])
    if kind == "lsv_book":
        return dict(bytes=5 * 8.0 * case["strikes"] * case["times"] + 1e4,
                    flops=5.0 * case["paths"] * 365 * PATH_STEP_FLOPS["lsv"])
    if kind == "batch":
        f = sum(float(b.paths) * (b.n_dates - 1) * PATH_STEP_FLOPS[("gbm", "heston", "lsv")[b.assets[0]["model"]]]
                for b in _batch(case, 0))
        return dict(bytes=1e5, flops=f)
    if kind == "bump":
        scenarios = 12 if case["model"] == "heston" else 7
        return dict(bytes=1e5, flops=float(scenarios) * case["paths"] * case["steps"] * PATH_STEP_FLOPS[case["model"]])
    if kind == "american":
        dates = case["days"] / case["every"]
        per = PATH_STEP_FLOPS[case["model"]]
        return dict(bytes=64.0 * dates,
                    flops=case["paths"] * dates * ((per + 30) + (5 * per + 30 if case["greeks"] else 0)))
    if kind == "calibration":
        return dict(bytes=case["days"] * W.LSV_GRID_POINTS * 16.0, flops=300.0 * case["particles"] * case["days"])
    layer = 2.0 * (KIN * H + 3 * H * H + H)
    if kind == "train":
        steps = case["epochs"] * (case["rows"] // case["batch"])
        return dict(bytes=case["rows"] * 36.0 + 2 * 52e3 * 4, flops=3 * layer * steps * case["batch"])
    cells = float(case["sets"]) * case["strikes"] * case["maturities"]
    return dict(bytes=4 * cells + 40.0 * case["sets"] + case["members"] * 2.1e5, flops=case["members"] * layer * cells)


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------
CHUNK = 18  # log2 paths simulated together


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


_directions = {}


def _direction_numbers():
    """Joe-Kuo direction numbers [4097][32] from the data table (primitive polynomials and m_i)."""
    if not _directions:
        raw = (pathlib.Path(W.__file__).resolve().parent / "data" / "joe_kuo_6_21201.bin").read_bytes()
        dims = int(np.frombuffer(raw, np.uint32, 1, 8)[0])
        u = np.frombuffer(raw, np.uint32, (len(raw) - 16) // 4, 16).astype(np.int64)
        S, A, MO, M = u[:dims], u[dims:2 * dims], u[2 * dims:3 * dims + 1], u[3 * dims + 1:]
        D = min(dims + 1, 4097)
        V = np.zeros((D, 32), dtype=np.int64)
        V[0] = 1 << np.arange(31, -1, -1)
        for d in range(1, D):
            s, a, m = int(S[d - 1]), int(A[d - 1]), M[MO[d - 1]:]
            for i in range(32):
                if i < s:
                    V[d, i] = int(m[i]) << (31 - i)
                else:
                    v = int(V[d, i - s]) ^ (int(V[d, i - s]) >> s)
                    for k in range(1, s):
                        if (a >> (s - 1 - k)) & 1:
                            v ^= int(V[d, i - k])
                    V[d, i] = v
        _directions["v"] = V
    return _directions["v"]


def _schedule(t):
    """Brownian-bridge construction order over dates 1..m: (date, left, right, weights, sd)."""
    m = len(t) - 1
    done = np.zeros(m, dtype=bool)
    done[m - 1] = True
    out = [(m, 0, m, 0.0, 0.0, math.sqrt(t[m]))]
    j = 0
    for _ in range(1, m):
        while done[j]:
            j += 1
        k = j
        while not done[k]:
            k += 1
        mid = j + ((k - 1 - j) >> 1)
        done[mid] = True
        a, b, x = j, k + 1, mid + 1  # left, right and middle dates
        span = t[b] - t[a]
        out.append((x, a, b, (t[b] - t[x]) / span, (t[x] - t[a]) / span,
                    math.sqrt((t[x] - t[a]) * (t[b] - t[x]) / span)))
        j = k + 1
        if j >= m:
            j = 0
    return out


def _normals(book):
    """Yields (valid, W [factors][dates][paths]) chunk by chunk: the Brownian paths of every factor."""
    dev = _dev()
    nd, na = book.n_dates, len(book.assets)
    F = na + sum(a["model"] != abi.MODEL_GBM for a in book.assets)
    dims = (nd - 1) * F
    V = torch.from_numpy(_direction_numbers()[:dims]).to(dev)
    lo = torch.zeros((dims, 1), dtype=torch.int32, device=dev)  # the points' low bits, Gray order
    v32 = V.to(torch.int32)
    for j in range(CHUNK):
        lo = torch.cat([lo, v32[:, j:j + 1] ^ lo.flip(1)], 1)
    sched = _schedule(book.t)
    first, last = book.sobol_skip + 1, book.sobol_skip + book.paths
    i = torch.arange(1 << CHUNK, device=dev)
    for c in range(first >> CHUNK, (last >> CHUNK) + 1):
        hi = v32[:, CHUNK - 1] if c & 1 else torch.zeros(dims, dtype=torch.int32, device=dev)
        g = c ^ (c >> 1)
        for k in range(32 - CHUNK):
            if (g >> k) & 1:
                hi = hi ^ v32[:, CHUNK + k]
        n = (c << CHUNK) + i
        ok = torch.nonzero((n >= first) & (n <= last)).flatten()
        p0, p1 = int(ok[0]), int(ok[-1]) + 1
        Wt = torch.zeros((F, nd, p1 - p0), dtype=FP64, device=dev)
        for s, (x, a, b, lw, rw, sd) in enumerate(sched):
            rows = slice(s * F, (s + 1) * F)
            u = ((lo[rows, p0:p1] ^ hi[rows, None]).to(torch.int64) & 0xFFFFFFFF).to(FP64) * 2.0 ** -32
            Wt[:, x] = lw * Wt[:, a] + rw * Wt[:, b] + sd * torch.special.ndtri(u)
        yield Wt


def _qe(v, z, e, kappa, theta, xi):
    m = theta + (v - theta) * e
    s2 = v * xi * xi * e / kappa * (1 - e) + theta * xi * xi / (2 * kappa) * (1 - e) ** 2
    psi = s2 / (m * m)
    c = torch.clamp(2.0 / psi, min=1.0)
    b2 = c - 1.0 + torch.sqrt(c * (c - 1.0))
    quad = m / (1.0 + b2) * (torch.sqrt(b2) + z) ** 2
    p = (psi - 1.0) / (psi + 1.0)
    up = torch.special.ndtr(-z)
    expo = torch.where(up >= 1.0 - p, torch.zeros_like(v),
                       torch.log((1.0 - p) / up) * m / torch.clamp(1.0 - p, min=1e-300))
    return torch.where(psi <= 1.5, quad, expo)


def _leverage(a, i, x):
    """Leverage of layer i at ln S = ln S0 + x, clamped linear interpolation."""
    row = torch.from_numpy(a["lev_values"][i]).to(x.device)
    f = (math.log(a["spot"]) + x) / float(a["lev_ln_step"][i]) - float(a["lev_offset"][i])
    f = torch.clamp(f, 0.0, float(len(row) - 1))
    k = torch.clamp(f.to(torch.int64), max=len(row) - 2)
    w = f - k.to(FP64)
    return (1.0 - w) * row[k] + w * row[k + 1]


def _simulate(book):
    """Yields (X, DX, B) per chunk: per asset the log-spot over S0 [dates][paths], its steps, and W."""
    t = book.t
    for Wt in _normals(book):
        X, B, nv = [], [], len(book.assets)
        for u, a in enumerate(book.assets):
            w = Wt[u]
            x = torch.zeros_like(w)
            v = torch.full_like(w[0], a.get("v0", 0.0))
            if a["model"] != abi.MODEL_GBM:
                wv = Wt[nv]
                nv += 1
            for i in range(1, book.n_dates):
                dt = t[i] - t[i - 1]
                z = (w[i] - w[i - 1]) / math.sqrt(dt)
                carry = a["carry"][i] * t[i] - a["carry"][i - 1] * t[i - 1]
                if a["model"] == abi.MODEL_GBM:
                    x[i] = x[i - 1] + carry - 0.5 * a["vol"] ** 2 * dt + a["vol"] * math.sqrt(dt) * z
                    continue
                k, th, xi, rho = a["kappa"], a["theta"], a["xi"], a["rho"]
                vn = _qe(v, (wv[i] - wv[i - 1]) / math.sqrt(dt), math.exp(-k * dt), k, th, xi)
                L = _leverage(a, i, x[i - 1]) if a["model"] == abi.MODEL_LSV else 1.0
                s = v + vn
                x[i] = (x[i - 1] + carry + L * (-rho * k * th / xi * dt + 0.5 * dt * k * rho / xi * s + rho / xi * (vn - v)
                                                + torch.sqrt(0.5 * dt * (1 - rho * rho) * s) * z)
                        - 0.25 * dt * L * L * s)
                v = vn
            X.append(x)
            B.append(w)
        yield X, B


def _flow(book, p, X):
    t, m = book.t, p["maturity"]
    df, q = math.exp(-t[m] * p["zero_rate"]), math.exp(-p["quanto"] * t[m])
    if p["kind"] == abi.VARIANCE:
        x = X[p["asset"]]
        dt = torch.from_numpy(np.diff(t[:m + 1])).to(x.device)[:, None]
        s2 = ((x[1:m + 1] - x[:m] - p["quanto"] * dt) ** 2).sum(0)
        total = p["total_year_fraction"] if p["total_year_fraction"] > 0 else t[m]
        return p["notional"] * ((p["past_variance"] + s2) / total - p["strike_variance"]) * df
    if p["kind"] == abi.BASKET:
        s = sum(w * book.assets[c]["spot"] * torch.exp(X[c][m]) for c, w in zip(p["components"], p["weights"])) * q
    else:
        s = book.assets[p["asset"]]["spot"] * torch.exp(X[p["asset"]][m]) * q
    f = torch.clamp(s - p["strike"] if p["option_type"] == abi.CALL else p["strike"] - s, min=0.0) * df
    if p["kind"] == abi.BARRIER:
        mon = torch.from_numpy(np.asarray(p["monitor"], dtype=np.int64)).to(s.device)
        y = X[p["asset"]][mon] - p["quanto"] * torch.from_numpy(t[p["monitor"]]).to(s.device)[:, None]
        level = math.log(p["barrier_level"] / book.assets[p["asset"]]["spot"])
        hit = (y >= level).any(0) if p["barrier_up"] else (y <= level).any(0)
        f = f * (hit if p["barrier_in"] else ~hit)
    return f


def _pathwise(book, p, X, B):
    """Pathwise delta and vega of one vanilla on a GBM or Heston asset (None where not given)."""
    a, m = book.assets[p["asset"]], p["maturity"]
    s = a["spot"] * torch.exp(X[p["asset"]][m])
    sgn = 1.0 if p["option_type"] == abi.CALL else -1.0
    live = (sgn * (s - p["strike"]) > 0).to(FP64) * sgn * math.exp(-book.t[m] * p["zero_rate"])
    vega = live * s * (B[p["asset"]][m] - a["vol"] * book.t[m]) if a["model"] == abi.MODEL_GBM else None
    return live * s / a["spot"], vega


def _price64(book, greeks=False):
    """Means and standard errors of every product and of the book, in FP64."""
    n = len(book.products)
    acc = np.zeros((n + 1 + 2 * n, 2))
    for X, B in _simulate(book):
        total = 0.0
        for j, p in enumerate(book.products):
            f = _flow(book, p, X)
            total = total + p["fx"] * f
            acc[j] += [float(f.sum()), float((f * f).sum())]
            if greeks:
                for q, g in enumerate(_pathwise(book, p, X, B)):
                    acc[n + 1 + 2 * j + q] += [float(g.sum()), float((g * g).sum())] if g is not None else np.nan
        acc[n] += [float(total.sum()), float((total * total).sum())]
    N = float(book.paths)
    mean = acc[:, 0] / N
    trust = np.sqrt(np.maximum(acc[:, 1] - acc[:, 0] ** 2 / N, 0.0) / (N - 1) / N)
    out = dict(premium=mean[:n], trust=trust[:n], book_premium=float(mean[n]), book_trust=float(trust[n]))
    if greeks:
        for q, k in enumerate(("delta", "vega")):
            out[k], out[k + "_trust"] = mean[n + 1 + q::2], trust[n + 1 + q::2]
    return out


def _bumped(book, kind, h):
    b = book.copy()
    for a in b.assets:
        if kind == "spot":
            a["spot"] *= 1.0 + h
        elif kind == "vol" and a["model"] == abi.MODEL_GBM:
            a["vol"] += h
        elif kind == "vol":
            a["v0"], a["theta"] = (math.sqrt(a["v0"]) + h) ** 2, (math.sqrt(a["theta"]) + h) ** 2
        elif kind == "rate":
            a["carry"] = a["carry"] + h
        elif kind in a:
            a[kind] += h
    if kind == "rate":
        for p in b.products:
            p["zero_rate"] += h
    return b


def _rolled(book):
    """The book one calendar day on; date 1 becomes today where it is tomorrow."""
    sh = 1 if book.days[1] == 1 and book.n_dates >= 3 else 0
    days = np.concatenate([[0], book.days[1 + sh:] - 1])
    b = abi.Book(days=days, paths=book.paths)
    for a in book.assets:
        c = a["carry"]
        new = np.full(len(days), c[1])
        new[1:] = (c[1 + sh:] * book.t[1 + sh:] - c[1] / 365.0) / b.t[1:]
        b.assets.append(dict(a, carry=new))
    for p in book.products:
        q = dict(p, maturity=max(p["maturity"] - sh, 0))
        if "monitor" in q:
            q["monitor"] = np.array([k - sh for k in q["monitor"] if k >= sh])
        b.products.append(q)
    return b


def _bump64(book):
    def price(b):
        r = _price64(b)
        return np.append(r["premium"], r["book_premium"])
    p0, S = price(book), book.assets[0]["spot"]
    up, dn = price(_bumped(book, "spot", 0.1)), price(_bumped(book, "spot", -0.1))
    out = dict(premium=p0, delta=(price(_bumped(book, "spot", 0.01)) - p0) / (0.01 * S),
               gamma=(up - 2 * p0 + dn) / (0.1 * S) ** 2, vega=price(_bumped(book, "vol", 0.01)) - p0,
               rho=(price(_bumped(book, "rate", 1e-4)) - p0) / 1e-4 * 0.01, theta=price(_rolled(book)) - p0)
    total = np.array([v[-1] for v in out.values()])
    heston = book.assets[0]["model"] != abi.MODEL_GBM
    for k in abi.PARAMS:
        out["vega_" + k] = (price(_bumped(book, k, 0.01)) - p0) / 0.01 if heston else np.full_like(p0, np.nan)
    return {**{k: v[:-1] for k, v in out.items()}, "book": total}


def _spots(book):
    a = book.assets[0]
    return torch.cat([a["spot"] * torch.exp(X[0]) for X, _ in _simulate(book)], 1)


def _exercise(book, S, policy=None):
    """Longstaff-Schwartz of the book's put on spots S [dates][paths]: fits on {1, m, m^2} of the
    in-the-money paths, or applies a fitted policy; (premium, trust, european, beta)."""
    p, t = book.products[0], book.t
    K, r, M = p["strike"], p["zero_rate"], len(t)
    iv = torch.clamp(K - S[-1], min=0.0)
    val = iv * math.exp(-r * t[-1])
    euro = float(val.mean())
    cf, beta = iv, np.full((M, 3), np.nan)
    for i in range(M - 2, 0, -1):
        cf = cf * math.exp(r * (t[i] - t[i + 1]))
        itm = torch.nonzero(S[i] < K).flatten()
        m, iv = S[i][itm] / K, K - S[i][itm]
        if policy is None:
            if len(itm) < 50:
                continue
            A = torch.stack([torch.ones_like(m), m, m * m])
            b = torch.linalg.solve((A @ A.T).cpu(), (A @ cf[itm]).cpu()).numpy()
        else:
            b = policy[i]
        if not np.isfinite(b).all():
            continue
        beta[i] = b
        ex = iv >= b[0] + b[1] * m + b[2] * m * m
        cf, val = cf.clone(), val.clone()
        cf[itm[ex]] = iv[ex]
        val[itm[ex]] = iv[ex] * math.exp(-r * t[i])
    n = S.shape[1]
    mean = float(val.mean())
    trust = math.sqrt((float((val * val).mean()) - mean * mean) / (n - 1))
    return max(mean, max(K - float(S[0, 0]), 0.0)), trust, euro, beta


def _american64(book, greeks):
    prem, trust, euro, beta = _exercise(book, _spots(book))
    out = dict(premium=prem, trust=trust, european=euro, beta=None, fitted_dates=None)
    if greeks:
        def frozen(b):
            return _exercise(b, _spots(b), beta)[0]
        S = book.assets[0]["spot"]
        out["delta"] = (frozen(_bumped(book, "spot", 0.01)) - prem) / (0.01 * S)
        out["gamma"] = (frozen(_bumped(book, "spot", 0.1)) - 2 * prem + frozen(_bumped(book, "spot", -0.1))) / (0.1 * S) ** 2
        out["vega"] = frozen(_bumped(book, "vol", 0.01)) - prem
        out["rho"] = (frozen(_bumped(book, "rate", 1e-4)) - prem) / 1e-4 * 0.01
        rolled = _rolled(book)
        out["theta"] = _exercise(rolled, _spots(rolled))[0] - prem
    return out


def _net(p):
    """The layers (W, b) of a flat parameter vector, in FP64."""
    p = torch.from_numpy(np.asarray(p, dtype=np.float64)).to(_dev())
    w1 = p[:H * KIN].reshape(H, KIN)[:, :NF]
    layers, o = [[w1, p[H * KIN:H * KIN + H]]], H * KIN + H
    for _ in range(3):
        layers.append([p[o:o + H * H].reshape(H, H), p[o + H * H:o + H * H + H]])
        o += H * H + H
    return layers + [[p[o:o + H].reshape(1, H), p[o + H:]]]


def _forward(layers, x):
    for w, b in layers[:-1]:
        x = torch.nn.functional.silu(x @ w.T + b)
    return (x @ layers[-1][0].T + layers[-1][1]).flatten()


class _Mt64:
    """The 64-bit Mersenne twister (Matsumoto and Nishimura), as C++'s mt19937_64."""

    def __init__(self, seed):
        s, mt = seed & (2 ** 64 - 1), []
        for i in range(312):
            mt.append(s)
            s = (6364136223846793005 * (s ^ (s >> 62)) + i + 1) & (2 ** 64 - 1)
        self.mt, self.out = np.array(mt, dtype=np.uint64), []

    def __call__(self):
        if not self.out:
            m, old = self.mt, self.mt.copy()
            u = np.uint64

            def twist(hi, lo, far):
                x = (hi & u(0xFFFFFFFF80000000)) | (lo & u(0x7FFFFFFF))
                return far ^ (x >> u(1)) ^ np.where(x & u(1), u(0xB5026F5AA96619E9), u(0))
            m[:156] = twist(old[:156], old[1:157], old[156:])
            m[156:311] = twist(old[156:311], old[157:312], m[:155])
            m[311:] = twist(old[311:], m[:1], m[155:156])
            y = m.copy()
            y ^= (y >> u(29)) & u(0x5555555555555555)
            y ^= (y << u(17)) & u(0x71D67FFFEDA60000)
            y ^= (y << u(37)) & u(0xFFF7EEE000000000)
            y ^= y >> u(43)
            self.out = [int(v) for v in y[::-1]]
        return self.out.pop()

    def below(self, n):
        """A uniform integer in [0, n) (Lemire's multiplication method)."""
        x = self() * n
        if (x & (2 ** 64 - 1)) < n:
            t = (2 ** 64 - n) % n
            while (x & (2 ** 64 - 1)) < t:
                x = self() * n
        return x >> 64


def _shuffle(idx, rng):
    """A Fisher-Yates shuffle that takes two positions from one draw, as the C++ library's."""
    n, i = len(idx), 1
    if n % 2 == 0:
        j = rng.below(2)
        idx[1], idx[j] = idx[j], idx[1]
        i = 2
    while i < n:
        a, b = divmod(rng.below((i + 1) * (i + 2)), i + 2)
        idx[i], idx[a] = idx[a], idx[i]
        idx[i + 1], idx[b] = idx[b], idx[i + 1]
        i += 2


def _train64(case, p0, data, seed):
    dev = _dev()
    x, y, sc = (torch.from_numpy(v.astype(np.float64)).to(dev) for v in data)
    n = case["rows"]
    B = min(case["batch"], n // 128 * 128)
    steps = n // B
    total = steps * case["epochs"]
    params = [w.clone().requires_grad_() for layer in _net(p0) for w in layer]
    m, v = [torch.zeros_like(w) for w in params], [torch.zeros_like(w) for w in params]
    idx, rng, k, loss = list(range(n)), _Mt64(seed), 0, 0.0
    for _ in range(case["epochs"]):
        _shuffle(idx, rng)
        perm = torch.tensor(idx, device=dev)
        for s in range(steps):
            rows = perm[s * B:(s + 1) * B]
            layers = [params[2 * j:2 * j + 2] for j in range(5)]
            e = _forward(layers, x[rows]) - y[rows]
            loss = (e * e / sc[rows] ** 2).mean()
            grads = torch.autograd.grad(loss, params)
            lr = 2e-3 * 0.5 * (1.0 + math.cos(math.pi * k / total)) + 1e-6
            k += 1
            with torch.no_grad():
                for w, g, mw, vw in zip(params, grads, m, v):
                    mw.mul_(0.9).add_(g, alpha=0.1)
                    vw.mul_(0.999).addcmul_(g, g, value=0.001)
                    w -= lr * (mw / (1 - 0.9 ** k)) / (torch.sqrt(vw / (1 - 0.999 ** k)) + 1e-8)
    w1 = torch.zeros((H, KIN), dtype=FP64, device=dev)
    w1[:, :NF] = w1[:, NF:2 * NF] = params[0].detach()
    flat = torch.cat([w1.flatten()] + [w.detach().flatten() for w in params[1:]])
    return dict(params=flat.cpu().numpy(), loss=float(loss))


def _lattice64(case, seed):
    rng = np.random.default_rng(seed)
    sets = _sets(case["sets"], rng)
    nets = [_net(_weights(rng)) for _ in range(case["members"])]
    lo, hi = surrogate.BOX_LO, surrogate.BOX_HI
    lm, T = _axes(case)
    dev = _dev()
    X = np.empty((len(sets), len(T), len(lm), NF))
    X[..., 0], X[..., 1], X[..., 2:] = lm[None, None, :], T[None, :, None], sets[:, None, None, :]
    X = torch.from_numpy(np.clip(X.reshape(-1, NF), lo, hi)).to(dev)
    lo, hi = torch.from_numpy(lo).to(dev), torch.from_numpy(hi).to(dev)
    xn = 2.0 * (X - lo) / (hi - lo) - 1.0
    y = torch.cat([sum(_forward(n, x) for n in nets) / len(nets) for x in xn.split(1 << 17)])
    kt = X[:, 2] * X[:, 1]
    sd = torch.sqrt((X[:, 3] + (X[:, 6] - X[:, 3]) * (1.0 - torch.exp(-kt)) / kt).clamp(min=1e-8) * X[:, 1])
    d1 = -X[:, 0] / sd + 0.5 * sd
    bs = torch.special.ndtr(d1) - torch.exp(X[:, 0]) * torch.special.ndtr(d1 - sd)
    return (y * torch.sqrt(bs * bs + surrogate.FLOOR ** 2)).cpu().numpy()


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "calibration":  # the ensemble's draws are one sequential stream: too long in numpy
        return None
    if kind == "train":
        p0 = _weights(rng)
        return _train64(case, p0, _training_set(case, rng), seed)
    if kind == "lattice":
        return _lattice64(case, seed)
    if kind == "batch":
        books = _batch(case, seed)
        if sum(float(b.paths) * b.n_dates for b in books) > 1e9:
            return None
        r = [_price64(b) for b in books]
        return {"book_premium": np.array([x["book_premium"] for x in r]),
                "book_trust": np.array([x["book_trust"] for x in r]),
                "premium": np.concatenate([x["premium"] for x in r]), "trust": np.concatenate([x["trust"] for x in r])}
    if kind == "book":
        s = _book(case, rng)
    elif kind == "grid":
        s = _grid(case, rng)
    elif kind == "lsv_book":
        s = _lsv_book(case, seed)
    elif kind == "bump":
        return _bump64(_bump_book(case, rng))
    else:
        return _american64(_american_book(case, rng), case["greeks"])
    if s.greeks and s.assets[0]["model"] == abi.MODEL_LSV:
        # the pathwise delta through a leverage surface has no plain counterpart here
        return {**_price64(s), **{k: None for k in GREEKS}}
    return _price64(s, greeks=bool(s.greeks))
