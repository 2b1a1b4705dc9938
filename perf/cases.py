"""Performance cases of the engine: the calls its users make, through the Python package.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)`` gives more from
the same ranges, ``prepare(case, seed)`` builds what a caller holds before the call (request objects,
and the resident handles a program keeps), ``run(state)`` makes the call and returns its results as
arrays, ``work(case)`` counts the bytes and operations the call cannot do without, and
``exact(case, seed)`` gives the same results in 64-bit arithmetic from numpy and torch alone.

Kinds of call:

* ``price``    one trade by ``price_put_leg``, or a common-random-number batch by ``price_scenarios``
* ``risk``     the central-difference batch of ``price_risk_batch`` (1 + 4·assets + 4 scenarios)
* ``replay``   ``materialize_paths``: a range of a priced trade's spot paths
* ``book``     ``price_book_trade_bumps``: every trade under its own 16 scenarios, in one call
* ``resident`` the same for a book that was uploaded once (``ResidentBook``)
* ``cube``     ``generate_correlated_block`` and ``gbm_evolve`` of the path cube
* ``backend``  one bump of the two-factor local-vol backend on resident buffers (``ResidentLv``)
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "riga-flow_gb300"))

from riga_gb300 import abi, gpu, pathcube  # noqa: E402
from riga_gb300.engine import default_engine  # noqa: E402
from riga_gb300.types import (BookRequest, BookTrade, EngineOptions, ImpliedVolGrid, MarketSnapshot,  # noqa: E402
                              PhoenixTrade, PriceRequest, SimulationConfig, VarianceReduction)

DAYS = 252
AS_OF = "2026-01-02"
UNIVERSE = 20  # assets of a book's universe
BOOK_YEARS = 5


# ---------------------------------------------------------------------- the cases -------------
def _price(name, assets, steps, paths, scenarios=0, smile=None, lane="sobol", precision="fp32", trace="off",
           kind="price"):
    """``smile``: (strikes, expiries, Dupire points) of a local-vol request, or None for flat vol;
    ``lane``: sobol (digital shift), owen (the reference's scramble, 512 dimensions), halton,
    stream (pseudo-random)."""
    k, t, g = smile or (0, 0, 0)
    return {"name": name, "kind": kind, "assets": assets, "steps": steps, "paths": paths, "scenarios": scenarios,
            "strikes": k, "expiries": t, "grid": g, "lane": lane, "precision": precision, "trace": trace}


def listed():
    return [
        # a quote while typing: the smallest request, latency only
        _price("quote_flat2", 2, 252, 4096),
        # a single trade of the serving mix: 3-asset Dupire local vol, 2^14 paths
        _price("serve_lv3", 3, 756, 1 << 14, smile=(40, 24, 40)),
        # the headline: one trade, base and 15 bumps in one common-random-number batch
        _price("crn16_lv3", 3, 756, 1 << 20, scenarios=16, smile=(40, 24, 40)),
        # the risk report of one trade: 17 scenarios on a ragged path count
        _price("risk_lv3", 3, 504, 100_003, smile=(40, 24, 40), kind="risk"),
        # a long-dated 5-asset trade on many paths, price only
        _price("large_lv5", 5, 1260, 1 << 21, smile=(64, 32, 64)),
        # the plain FP64 method: 3 assets, flat vol
        _price("plain_fp64", 3, 756, 1 << 16, precision="fp64"),
        # a request with every default of the configuration: FP64, pseudo-random stream, 30,000
        # paths, trace events, a market's own implied grid on the 96-point Dupire axis
        _price("default_stream", 2, 501, 30_000, smile=(13, 9, 96), lane="stream", precision="fp64", trace="aggregated"),
        # replay of the path range a reader asks for, on the reference's Owen-scrambled points
        _price("replay_owen", 2, 501, 4096, smile=(13, 9, 96), lane="owen", precision="fp64", kind="replay"),
        # a desk's book in one call: per-trade bumps on a 20-asset universe over five years
        {"name": "book_desk", "kind": "book", "trades": 64, "paths": 1 << 17},
        # a book kept on the device and repriced through the day
        {"name": "book_resident", "kind": "resident", "trades": 128, "paths": 1 << 14},
        # the path cube as arrays: correlated normals and their GBM evolution
        {"name": "cube_2x20000", "kind": "cube", "paths": 20_000, "steps": 252, "assets": 2},
        # the two-factor backend: one spot bump on resident normals and rows
        {"name": "backend_lv", "kind": "backend", "paths": 1 << 17, "steps": 252, "grid": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a shape of the listed ones with its sizes drawn over their range."""
    shape = rng.choice(["quote", "quote", "crn", "risk", "large", "plain", "stream", "replay", "book", "resident",
                        "cube", "backend"])
    smile = rng.choice([None, (rng.randint(13, 64), rng.randint(6, 32), rng.choice([40, 64, 96]))])
    steps = rng.randint(63, 1260)
    if shape == "quote":
        lane = rng.choice(["sobol", "sobol", "sobol", "owen", "halton"])
        c = _price("", rng.randint(1, 5), steps, _log_int(rng, 1000, 1 << 16), smile=smile, lane=lane)
    elif shape == "crn":
        c = _price("", rng.randint(1, 5), rng.randint(63, 756), _log_int(rng, 1 << 14, 1 << 19),
                   scenarios=rng.randint(2, 16), smile=smile)
    elif shape == "risk":
        c = _price("", rng.randint(1, 5), rng.randint(63, 756), _log_int(rng, 1 << 13, 1 << 18), smile=smile, kind="risk")
    elif shape == "large":
        c = _price("", rng.randint(1, 5), steps, _log_int(rng, 1 << 18, 1 << 21), smile=smile)
    elif shape == "plain":
        c = _price("", rng.randint(1, 5), rng.randint(63, 756), _log_int(rng, 1 << 12, 1 << 16), smile=smile,
                   lane=rng.choice(["sobol", "sobol", "owen"]), precision="fp64")
    elif shape == "stream":
        c = _price("", rng.randint(1, 3), rng.randint(63, 756), _log_int(rng, 4000, 40_000), smile=smile, lane="stream",
                   precision="fp64", trace="aggregated")
    elif shape == "replay":
        c = _price("", rng.randint(1, 3), rng.randint(63, 756), _log_int(rng, 64, 4096), smile=smile,
                   lane=rng.choice(["owen", "sobol"]), precision="fp64", kind="replay")
    elif shape == "book":
        c = {"kind": "book", "trades": _log_int(rng, 16, 128), "paths": _log_int(rng, 1 << 13, 1 << 17)}
    elif shape == "resident":
        c = {"kind": "resident", "trades": _log_int(rng, 16, 256), "paths": _log_int(rng, 1 << 12, 1 << 15)}
    elif shape == "cube":
        c = {"kind": "cube", "paths": _log_int(rng, 1000, 40_000), "steps": rng.randint(63, 504), "assets": rng.randint(1, 3)}
    else:
        c = {"kind": "backend", "paths": _log_int(rng, 4096, 1 << 17), "steps": rng.randint(63, 504),
             "grid": rng.choice([40, 64, 96])}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------- inputs ----------------
def _correlation(rng, n):
    """A one-factor correlation with loadings U[0.4, 0.85]."""
    b = [rng.uniform(0.4, 0.85) for _ in range(n)]
    return [[1.0 if i == j else b[i] * b[j] for j in range(n)] for i in range(n)]


def _terms(rng, n, steps, rate, name):
    """Phoenix terms of the benchmark configurations: quarterly memory coupons, daily knock-out."""
    return {"trade_id": name, "initial_spots": [100.0] * n, "maturity_years": steps / DAYS, "steps": steps,
            "strike": 1.0, "knock_in_barrier": rng.uniform(0.5, 0.7), "knock_out_barrier": rng.uniform(0.98, 1.08),
            "coupon_barrier": rng.uniform(0.6, 0.8), "coupon_rate": rate, "memory_coupon": True,
            "coupon_periods": max(1, round(steps / 63)), "fixed_first_coupon": False,
            "call_start_step": 63 if steps >= 126 else steps // 4}


def _grid(rng, strikes, expiries, years):
    """A seeded raw-SVI smile on `strikes` log-moneyness points and `expiries` maturities."""
    a, b, rho = rng.uniform(0.01, 0.04), rng.uniform(0.05, 0.2), rng.uniform(-0.7, -0.2)
    m, s = rng.uniform(-0.1, 0.1), rng.uniform(0.1, 0.3)
    ks = [-1.0 + 1.5 * i / (strikes - 1) for i in range(strikes)]
    row = [math.sqrt(a + b * (rho * (k - m) + math.sqrt((k - m) ** 2 + s * s))) for k in ks]
    return {"maturities_years": [years * (j + 1) / expiries for j in range(expiries)],
            "strikes": [100.0 * math.exp(k) for k in ks], "vols": [list(row) for _ in range(expiries)]}


def _market(rng, n):
    return {"as_of": AS_OF, "spots": [100.0 * rng.uniform(0.97, 1.03) for _ in range(n)],
            "vols": [rng.uniform(0.15, 0.45) for _ in range(n)], "risk_free_rate": rng.uniform(0.02, 0.04),
            "dividend_yields": [rng.uniform(0.0, 0.02) for _ in range(n)], "correlation": _correlation(rng, n)}


def _bumps(n):
    """The bump order of a scenario batch after the base: (spot factors, vol shifts, rate shift)."""
    one, zero = [1.0] * n, [0.0] * n

    def at(base, idx, v):
        out = list(base)
        for i in idx:
            out[i] = v
        return out

    pairs = [(i, j) for j in range(n) for i in range(j)]
    out = [(at(one, [f], 1.0 + h), zero, 0.0) for f in range(n) for h in (0.01, -0.01)]
    out += [(one, at(zero, [f], 0.01), 0.0) for f in range(n)] + [(one, zero, 1e-4)]
    out += [(at(one, p, 1.01), zero, 0.0) for p in pairs] + [(one, at(zero, [f], -0.01), 0.0) for f in range(n)]
    out += [(one, zero, -1e-4)] + [(at(one, p, 0.99), zero, 0.0) for p in pairs]
    out += [(at(one, range(n), 1.0 + h), zero, 0.0) for h in (0.01, -0.01, 0.02, -0.02, 0.05, -0.05, 0.1, -0.1)]
    return out


def _bumped(market, bump):
    spot, vol, rate = bump
    return {**market, "spots": [s * k for s, k in zip(market["spots"], spot)],
            "vols": [v + d for v, d in zip(market["vols"], vol)], "risk_free_rate": market["risk_free_rate"] + rate}


def _trade_inputs(case, seed):
    """Everything one trade's request is made from, as plain numbers."""
    rng = random.Random(f"trade {seed}")
    n, steps = case["assets"], case["steps"]
    market = _market(rng, n)
    terms = _terms(rng, n, steps, rng.uniform(0.01, 0.03), "trade")
    grids = [_grid(rng, case["strikes"], case["expiries"], steps / DAYS) for _ in range(n)] if case["strikes"] else None
    no_shift = [0.0] * n
    scenarios = [(market, no_shift)]
    if case["kind"] == "risk":
        one = [1.0] * n

        def up(f, h):
            return [1.0 + h if i == f else 1.0 for i in range(n)]

        def shift(f, h):
            return [h if i == f else 0.0 for i in range(n)]

        for f in range(n):
            scenarios += [(_bumped(market, (up(f, h), no_shift, 0.0)), no_shift) for h in (0.01, -0.01)]
            scenarios += [(_bumped(market, (one, shift(f, h), 0.0)), shift(f, h)) for h in (0.01, -0.01)]
        scenarios += [(_bumped(market, (one, no_shift, h)), no_shift) for h in (1e-4, -1e-4)]
        for h in (0.01, -0.01):
            corr = [[1.0 if i == j else c + h for j, c in enumerate(row)] for i, row in enumerate(market["correlation"])]
            scenarios.append(({**market, "correlation": corr}, no_shift))
    elif case["scenarios"]:
        scenarios += [(_bumped(market, b), b[1]) for b in _bumps(n)[: case["scenarios"] - 1]]
    return {"terms": terms, "market": market, "grids": grids, "scenarios": scenarios, "seed": rng.getrandbits(31)}


def _book_inputs(case, seed):
    rng = random.Random(f"book {seed}")
    loads = [[rng.uniform(0.2, 0.7) for _ in range(4)] for _ in range(UNIVERSE)]
    for row in loads:
        scale = min(1.0, math.sqrt(0.95 / sum(b * b for b in row)))
        row[:] = [b * scale for b in row]
    universe = _market(rng, UNIVERSE)
    universe["spots"] = [100.0] * UNIVERSE
    universe["correlation"] = [[1.0 if i == j else sum(a * b for a, b in zip(loads[i], loads[j]))
                                for j in range(UNIVERSE)] for i in range(UNIVERSE)]
    trades = []
    for j in range(case["trades"]):
        n = rng.randint(1, 5)
        under = rng.sample(range(UNIVERSE), n)
        trades.append((_terms(rng, n, DAYS * rng.randint(1, BOOK_YEARS), rng.uniform(0.01, 0.03), f"book-{j}"), under))
    return {"universe": universe, "trades": trades, "seed": rng.getrandbits(31)}


def _config(case, seed, dims):
    """The simulation configuration and engine options of a lane and precision."""
    lane = case.get("lane", "sobol")
    kind = {"sobol": "sobol", "owen": "sobol", "halton": "halton", "stream": "none"}[lane]
    vr = VarianceReduction(kind, 0 if kind == "none" else (512 if lane == "owen" else dims))
    config = SimulationConfig(case["paths"], 4096, seed, case.get("trace", "off"), vr)
    reference = lane in ("owen", "stream")
    options = EngineOptions(
        scrambler=abi.SCRAMBLE_OWEN if reference else abi.SCRAMBLE_DIGITAL_SHIFT,
        precision=abi.PRECISION_FP32 if case.get("precision", "fp32") == "fp32" else abi.PRECISION_FP64_PARITY,
        dim_mode=abi.DIM_WRAP_REFERENCE if reference else abi.DIM_FULL, lv_grid_x=case.get("grid", 0))
    return config, options


class _Handle:
    """Releases a resident handle's device memory with the state that holds it."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        self.handle.close()


def prepare(case, seed):
    engine = default_engine()
    kind = case["kind"]
    state = {"kind": kind, "engine": engine}
    if kind in ("price", "risk", "replay"):
        d = _trade_inputs(case, seed)
        config, options = _config(case, d["seed"], case["assets"] * case["steps"])
        state["request"] = PriceRequest(
            PhoenixTrade(**d["terms"]), MarketSnapshot(**d["market"]), config, AS_OF,
            [ImpliedVolGrid(**g) for g in d["grids"]] if d["grids"] else None, options)
        if case["scenarios"]:
            state["scenarios"] = [(MarketSnapshot(**m), shift) for m, shift in d["scenarios"]]
    elif kind in ("book", "resident"):
        d = _book_inputs(case, seed)
        steps = DAYS * BOOK_YEARS
        config, options = _config(case, d["seed"], UNIVERSE * steps)
        book = BookRequest(MarketSnapshot(**d["universe"]), steps, float(BOOK_YEARS),
                           [BookTrade(PhoenixTrade(**t), under) for t, under in d["trades"]], config, options)
        if kind == "book":
            state["book"] = book
        else:
            state["book"] = _Handle(engine.resident_book(book))
    elif kind == "cube":
        rng = random.Random(f"cube {seed}")
        m = _market(rng, case["assets"])
        state.update(seed=rng.getrandbits(31), paths=case["paths"], steps=case["steps"], market=m,
                     chol=np.linalg.cholesky(np.asarray(m["correlation"])))
    else:
        b = _backend_inputs(case, seed)
        state.update(b, lv=gpu.resident_lv(b["normals"], b["rows"], b["axis"], case["paths"], case["steps"], 1.0 / DAYS))
    return state


def _backend_inputs(case, seed):
    rng = np.random.default_rng(seed)
    paths, steps, gx = case["paths"], case["steps"], case["grid"]
    normals = rng.standard_normal(paths * steps * 2, dtype=np.float32)
    axis = np.tile(np.log(100.0) + np.linspace(-1.6, 0.55, gx), 2).astype(np.float32)
    k = np.linspace(-1.6, 0.55, gx)
    rows = []
    for _ in range(2):
        a, b, m, s = rng.uniform([0.02, 0.1, -0.1, 0.1], [0.05, 0.2, 0.1, 0.3])
        smile = np.sqrt(a + b * (-0.4 * (k - m) + np.sqrt((k - m) ** 2 + s * s)))
        rows.append(np.clip(smile[None, :] * np.linspace(1.1, 0.95, steps)[:, None], 0.1, 3.0))
    return {"normals": normals, "rows": np.concatenate([r.ravel() for r in rows]).astype(np.float32), "axis": axis,
            "spots": (100.0 * rng.uniform(0.97, 1.03, 2)).astype(np.float32), "refs": np.float32([100.0, 100.0]),
            "barrier": float(rng.uniform(1.02, 1.1)), "rate": 0.03, "dividends": np.float32([0.01, 0.0])}


# ---------------------------------------------------------------------- the calls -------------
def _results(results):
    """The numbers of a list of PriceResults: prices, errors, money sums and event counts."""
    r = np.frombuffer(b"".join(results), dtype=np.dtype(abi.PriceResult))
    return {"pv": r["pv"].copy(), "mc_error": r["mc_error"].copy(), "sums": r["path_sums"][:, :12].copy(),
            "counts": np.stack([r[k] for k in ("ko_count", "ki_count", "put_eligible_count", "coupon_path_count")],
                               axis=1).astype(np.int64)}


_RISK_FIELDS = ("spot_up_pv", "spot_down_pv", "vol_up_pv", "vol_down_pv", "spot_up_mc_error", "spot_down_mc_error",
                "vol_up_mc_error", "vol_down_mc_error")


def run(state):
    kind, engine = state["kind"], state["engine"]
    if kind == "price":
        if "scenarios" in state:
            return _results(engine.price_scenarios_raw(state["request"], state["scenarios"]))
        r = engine.price_raw(state["request"])
        out = _results([r])
        if state["request"].config.trace_level != "off":
            events = r.trace_events[: r.n_trace_events]
            out["trace_paths"] = np.array([e.path_id for e in events], dtype=np.int64)
            out["trace_times"] = np.array([e.time for e in events])
        return out
    if kind == "risk":
        rep = engine.price_risk_batch_raw(state["request"])
        assets = rep.assets[: rep.n_assets]
        out = _results([rep.base])
        out["greeks"] = np.array([[g.delta.value, g.gamma.value, g.vega.value] for g in assets])
        out["bumped"] = np.array([[getattr(g, f) for f in _RISK_FIELDS] for g in assets])
        out["market"] = np.array([rep.rate_up_pv, rep.rate_down_pv, rep.correlation_up_pv, rep.correlation_down_pv])
        out["transitions"] = np.array([[t.pv_impact, t.delta_impact, t.vega_impact] for t in rep.transitions])
        return out
    if kind == "replay":
        cube, _ = engine.materialize_paths(state["request"], with_records=False)
        return cube.data
    if kind == "book":
        return _results(engine.price_book_trade_bumps_raw(state["book"]))
    if kind == "resident":
        return _results(state["book"].handle.price_trade_bumps_raw())
    if kind == "cube":
        m = state["market"]
        block = pathcube.generate_correlated_block(state["seed"], state["paths"], state["steps"], state["chol"])
        cube = pathcube.gbm_evolve(m["spots"], m["vols"], m["risk_free_rate"], m["dividend_yields"], 1.0 / DAYS, block)
        return {"block": block.data, "cube": cube.data}
    state["lv"].run(state["spots"], state["refs"], state["barrier"], state["rate"], state["dividends"])
    terminal, ko = state["lv"].download()
    return {"terminal": terminal, "ko": ko}


# ---------------------------------------------------------------------- work ------------------
def work(case):
    """Operations (a fused multiply-add counts two): 35 per normal, N(N+1) + 3 per path, step and
    scenario for the correlation and the payoff, and per asset 19 for a local-vol step or 5 for a
    flat one.  Bytes: the arrays that cross the call or, on resident buffers, the device's memory."""
    kind = case["kind"]
    if kind in ("price", "risk", "replay"):
        n, units = case["assets"], case["paths"] * case["steps"]
        S = 9 + 4 * (n - 1) if kind == "risk" else max(1, case["scenarios"])
        step = n * (19 if case["strikes"] else 5) + n * (n + 1) + 3
        tables = 8 * n * case["strikes"] * case["expiries"] + 8 * S * case["steps"]
        cube = 4 * n * units if kind == "replay" else 0
        return {"bytes": tables + cube, "flops": units * (35 * n + S * step)}
    if kind in ("book", "resident"):
        steps = DAYS * BOOK_YEARS
        # a drawn trade has 3 underlyings and 3 years on average; a resident book holds its increments
        scan = case["trades"] * 16 * case["paths"] * 3 * DAYS * (3 * 5 + 3)
        gen = case["paths"] * steps * (35 * UNIVERSE + UNIVERSE * (UNIVERSE + 1))
        results = 16 * case["trades"] * 16 * 8
        incr = 4 * UNIVERSE * steps * case["paths"]
        if kind == "book":
            return {"bytes": results, "flops": scan + gen}
        return {"bytes": results + incr, "flops": scan}
    if kind == "cube":
        cells = case["paths"] * case["steps"] * case["assets"]
        return {"bytes": 3 * 4 * cells, "flops": cells * (60 + case["assets"] + 25)}
    units = case["paths"] * case["steps"]
    return {"bytes": 8 * units + 8 * case["steps"] * case["grid"] + 12 * case["paths"], "flops": units * 2 * 19}


# ---------------------------------------------------------------------- 64-bit results --------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_M64 = (1 << 64) - 1


def _mix64(z):
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M64
    return z ^ (z >> 31)


def _i64(v):
    """A 64-bit pattern as the signed value torch holds it in."""
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _lsr(t, k):
    return (t >> k) & ((1 << (64 - k)) - 1)


def _mix64_t(z):
    z = (z ^ _lsr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _lsr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _lsr(z, 31)


def _primitive_polynomials(count):
    """The first `count` primitive GF(2) polynomials of degree >= 2 in increasing order."""
    out, s = [], 2
    while len(out) < count:
        polys = np.arange((1 << s) + 1, 1 << (s + 1), 2, dtype=np.int64)

        def mulmod(a, b):
            r = np.zeros_like(polys)
            for i in reversed(range(s)):
                r = r << 1
                r = np.where(r >> s & 1, r ^ polys, r)
                r = np.where(b >> i & 1, r ^ a, r)
            return r

        def power_of_x(e):
            acc, base = np.ones_like(polys), np.full_like(polys, 2)
            while e:
                if e & 1:
                    acc = mulmod(acc, base)
                base = mulmod(base, base)
                e >>= 1
            return acc

        order = (1 << s) - 1
        ok, rest, p = power_of_x(order) == 1, order, 2
        while rest > 1:
            if rest % p == 0:
                if order != p or s > 1:
                    ok &= (power_of_x(order // p) != 1)
                while rest % p == 0:
                    rest //= p
            p = p + 1 if p * p <= rest else max(rest, p + 1)
        out += polys[ok].tolist()
        s += 1
    return out[:count]


def _directions(dims):
    """Sobol direction numbers [dims][32]: van der Corput, then the Joe-Kuo recurrence with unit
    initial values on the primitive polynomials."""
    v = np.zeros((dims, 32), dtype=np.int64)
    v[0] = [1 << (31 - k) for k in range(32)]
    polys = np.array(_primitive_polynomials(dims - 1), dtype=np.int64)
    deg = np.array([int(p).bit_length() - 1 for p in polys])
    for s in np.unique(deg):
        at = np.flatnonzero(deg == s)
        m = np.ones((len(at), 33), dtype=np.int64)
        for k in range(s + 1, 33):
            m[:, k] = (m[:, k - s] << s) ^ m[:, k - s]
            for i in range(1, s):
                m[:, k] ^= np.where(polys[at] >> (s - i) & 1, m[:, k - i] << i, 0)
        v[at + 1] = m[:, 1:] << np.arange(31, -1, -1)
    return v & 0xFFFFFFFF


def _probit(u):
    """Acklam's inverse normal."""
    a = (-3.969683028665376e1, 2.209460984245205e2, -2.759285104469687e2, 1.383577518672690e2, -3.066479806614716e1,
         2.506628277459239)
    b = (-5.447609879822406e1, 1.615858368580409e2, -1.556989798598866e2, 6.680131188771972e1, -1.328068155288572e1, 1.0)
    c = (-7.784894002430293e-3, -3.223964580411365e-1, -2.400758277161838, -2.549732539343734, 4.374664141464968,
         2.938163982698783)
    d = (7.784695709041462e-3, 3.224671290700398e-1, 2.445134137142996, 3.754408661907416, 1.0)

    def horner(k, x):
        r = torch.full_like(x, k[0])
        for v in k[1:]:
            r = r * x + v
        return r

    u = u.clamp(1e-12, 1.0 - 1e-12)
    q = u - 0.5
    mid = horner(a, q * q) * q / horner(b, q * q)
    t = torch.sqrt(-2.0 * torch.log(torch.minimum(u, 1.0 - u)))
    tail = horner(c, t) / horner(d, t) * torch.where(u < 0.5, 1.0, -1.0)
    return torch.where((u < 0.02425) | (u > 1.0 - 0.02425), tail, mid)


class _Lane:
    """The normals of a QMC lane, chunk by chunk: z[dim][path]."""

    def __init__(self, lane, seed, dims, chunk):
        self.lane, self.seed, self.dims, self.chunk = lane, seed, dims, chunk
        d = range(dims)
        if lane == "halton":
            primes, sieve = [], bytearray(max(64, int(dims * (math.log(dims + 6) + math.log(math.log(dims + 6))) + 64)))
            for p in range(2, len(sieve)):
                if not sieve[p]:
                    primes.append(p)
                    sieve[p * p::p] = b"\1" * len(range(p * p, len(sieve), p))
            self.base = torch.tensor(primes[:dims], device=_DEV)[:, None]
            self.key = torch.tensor([_i64(seed ^ ((k + 1) * 0xA0761D6478BD642F)) for k in d], device=_DEV)[:, None]
            return
        v = _directions(512 if lane == "owen" else dims)
        v = torch.tensor(v[np.arange(dims) % len(v)], device=_DEV)
        self.v = v
        self.shift = torch.tensor([_mix64(seed ^ ((k + 1) * 0xD1B54A32D192ED03) & _M64) >> 32 for k in d], device=_DEV)
        self.owen = torch.tensor([_i64(seed ^ (k * 0x9E3779B97F4A7C15)) for k in d], device=_DEV)[:, None]
        self.low = torch.zeros((dims, chunk), dtype=torch.int32, device=_DEV)
        n = torch.arange(chunk, device=_DEV)
        g = n ^ (n >> 1)
        v32 = torch.where(v >> 31 != 0, v - (1 << 32), v).to(torch.int32)
        for k in range(max(1, chunk.bit_length())):
            self.low ^= (g >> k & 1).to(torch.int32)[None, :] * v32[:, k:k + 1]

    def normals(self, first, lo, hi):
        """Points first + lo .. first + hi - 1, with `first` a multiple of the chunk."""
        if self.lane == "halton":
            n = torch.arange(first + lo, first + hi, device=_DEV)[None, :].expand(self.dims, -1).contiguous()
            R, B, i = torch.zeros_like(n), torch.ones_like(n), 0
            while bool((n > 0).any()):
                live = n > 0
                q = n // self.base
                h = _mix64_t(self.key ^ _i64((i + 1) * 0xE7037ED1A0B428DB))
                a = 1 + (((h & 0xFFFFFFFF) * (self.base - 1)) >> 32)
                c = (_lsr(h, 32) * self.base) >> 32
                R = torch.where(live, R * self.base + (a * (n - q * self.base) + c) % self.base, R)
                B = torch.where(live, B * self.base, B)
                n, i = q, i + 1
            return _probit(R.double() / B.double())
        g = first ^ (first >> 1)
        high = torch.zeros(self.dims, dtype=torch.int64, device=_DEV)
        for k in range(32):
            if g >> k & 1:
                high ^= self.v[:, k]
        if self.lane == "sobol":
            high ^= self.shift
        x = (self.low[:, lo:hi].long() & 0xFFFFFFFF) ^ high[:, None]
        if self.lane == "owen":
            y, prefix = torch.zeros_like(x), torch.zeros_like(x)
            for bit in range(31, -1, -1):
                h = _mix64_t(self.owen ^ _i64(bit * 0xD6E8FEB86659FD93) ^ (prefix * _i64(0xA24BAED4963EE407)))
                s = (x >> bit & 1) ^ _lsr(h, 63)
                y |= s << bit
                prefix = (prefix << 1) | s
            x = y
        return _probit((x.double() + 0.5) / 4294967296.0)


def _bridge(z, steps, dt):
    """Brownian increments [steps][n][path] of the depth-first bisection of [0, steps], node k of the
    preorder reading the normals z[k]."""
    W = torch.empty((steps + 1,) + z.shape[1:], dtype=torch.float64, device=z.device)
    W[0] = 0.0
    W[steps] = z[0] * math.sqrt(steps * dt)
    todo, k = [(0, steps)], 1
    while todo:
        lo, hi = todo.pop()
        if hi <= lo + 1:
            continue
        mid = (lo + hi) // 2
        W[mid] = 0.5 * (W[lo] + W[hi]) + z[k] * math.sqrt((hi - mid) * (mid - lo) / (hi - lo) * dt)
        k += 1
        todo += [(mid, hi), (lo, mid)]
    return W[1:] - W[:-1]


def _dupire(g, spot, rate, shift, gx):
    """(tenors, log-strike axis, local vol [tenor][axis]) of one implied grid: a spline per tenor in
    log-moneyness with the reference's coefficients, Dupire in total variance, clamped to [0.1, 3]."""
    T, K = np.asarray(g["maturities_years"]), np.asarray(g["strikes"])
    nt, nk = len(T), len(K)
    logs = np.linspace(math.log(K[0] * 0.55), math.log(K[-1] * 1.05), gx)
    w, wx, wxx, xa = (np.zeros((nt, gx)) for _ in range(4))
    for k in range(nt):
        fwd = spot * math.exp(rate * T[k])
        x, y = np.log(K / fwd), np.asarray(g["vols"][k]) + shift
        h = np.diff(x)
        y2 = np.zeros(nk)
        if nk >= 3:
            cp, dp = np.zeros(nk), np.zeros(nk)
            cp[0] = h[1] if 1 < nk - 1 else 0.0
            for i in range(1, nk):
                last = i == nk - 1
                b = 1.0 if last else 2.0 * (h[i - 1] + h[i])
                a = 0.0 if last else h[i]
                c = h[i + 1] if i + 1 < nk - 1 else 0.0
                d = 0.0 if last else 6.0 * ((y[i + 1] - y[i]) / h[i] - (y[i] - y[i - 1]) / h[i - 1])
                m = b - a * cp[i - 1]
                m = 1e-300 if abs(m) < 1e-300 else m
                cp[i], dp[i] = c / m, (d - a * dp[i - 1]) / m
            y2[-1] = dp[-1]
            for i in range(nk - 2, -1, -1):
                y2[i] = dp[i] - cp[i] * y2[i + 1]
        p = np.clip(logs - math.log(fwd), x[0], x[-1])
        s = np.minimum(np.searchsorted(x[1:nk - 1], p, side="left"), nk - 2)
        hs, t = h[s], np.clip((p - x[s]) / h[s], 0.0, 1.0)
        o = 1.0 - t
        f = o * y[s] + t * y[s + 1] + hs * hs / 6.0 * ((t ** 3 - t) * y2[s] + (o ** 3 - o) * y2[s + 1])
        f1 = (y[s + 1] - y[s] + hs * hs / 6.0 * ((3 * t * t - 1) * y2[s] - (3 * o * o - 1) * y2[s + 1])) / hs
        f2 = o * y2[s + 1] + t * y2[s]
        w[k], wx[k], wxx[k], xa[k] = f * f * T[k], 2 * f * T[k] * f1, 2 * T[k] * (f1 * f1 + f * f2), p
    lo, hi = np.maximum(np.arange(nt) - 1, 0), np.minimum(np.arange(nt) + 1, nt - 1)
    dw = (w[hi] - w[lo]) / np.maximum(T[hi] - T[lo], 1e-9)[:, None] if nt > 1 else w / max(T[0], 1e-9)
    ww = np.maximum(w, 1e-12)
    den = 1.0 - xa / ww * wx + 0.25 * (-0.25 - 1.0 / ww) * wx * wx + 0.5 * wxx
    ok = np.isfinite(den) & (np.abs(den) > 1e-12)
    lv2 = np.where(ok, dw / np.where(ok, den, 1.0), 0.01)
    return T, logs, np.sqrt(np.clip(lv2, 0.01, 9.0))


def _rows(surface, steps, dt):
    """The surface's row at each step's time [steps][axis]."""
    T, _, v = surface
    if len(T) == 1:
        return np.repeat(v, steps, axis=0)
    t = np.clip(np.arange(steps) * dt, T[0], T[-1])
    i = np.minimum(np.searchsorted(T[1:-1], t, side="left"), len(T) - 2)
    wt = ((t - T[i]) / (T[i + 1] - T[i]))[:, None]
    return (1.0 - wt) * v[i] + wt * v[i + 1]


def _scan(terms, rates, x, step, sums):
    """Runs the Phoenix machine on G (trade, scenario) rows that share a schedule and adds the path
    sums [G][16].  `terms`: one trade's terms per row; `step(t, x)` returns the log performances
    [G][n][path] after step t."""
    first = terms[0]
    steps, periods = first["steps"], first["coupon_periods"]
    dt = first["maturity_years"] / steps

    def col(values):
        return torch.tensor(values, dtype=torch.float64, device=_DEV)[:, None]

    ln_ko, ln_cb, ln_ki = (col([math.log(t[k]) for t in terms])
                           for k in ("knock_out_barrier", "coupon_barrier", "knock_in_barrier"))
    rate, coupon = col(rates), col([t["coupon_rate"] for t in terms])
    shape = (len(terms), x.shape[-1])
    qual, unpaid, cpv, mpv = (torch.zeros(shape, dtype=torch.float64, device=_DEV) for _ in range(4))
    alive, received = torch.ones(shape, dtype=torch.bool, device=_DEV), torch.zeros(shape, dtype=torch.bool, device=_DEV)
    ko_at = torch.full(shape, -1.0, dtype=torch.float64, device=_DEV)
    start = 0
    for t in range(steps):
        period = min(t * periods // steps, periods - 1)
        x = step(t, x)
        w = x.amin(1)
        qual += alive & (w >= ln_cb)
        if t >= first["call_start_step"]:
            hit = alive & (w >= ln_ko)
            ko_at.masked_fill_(hit, float(t))
            alive &= ~hit
        if t + 1 == steps or min((t + 1) * periods // steps, periods - 1) != period:
            # settle the period: paths knocked out in it at their own date, live ones at its end
            length = max(1, steps * (period + 1) // periods - steps * period // periods)
            due = qual * (coupon / length)
            out = ko_at >= start
            pay = (out | alive) & (due > 0.0)
            df = torch.exp(-rate * (torch.where(out, ko_at, float(t)) + 1.0) * dt)
            cpv += torch.where(pay, due * df, 0.0)
            mpv += torch.where(pay, unpaid * coupon * df, 0.0)
            received |= pay
            unpaid = torch.where(alive & ~pay, unpaid + 1.0, torch.where(pay, torch.zeros_like(unpaid), unpaid))
            qual.zero_()
            start = t + 1
    ko = ko_at >= 0.0
    df_end = torch.exp(-rate * first["maturity_years"])
    funding = torch.where(ko, torch.exp(-rate * (ko_at + 1.0) * dt), df_end)
    ki = w <= ln_ki
    strike = col([t["strike"] for t in terms])
    put = torch.where(ki & ~ko, (strike - torch.exp(w)).clamp(min=0.0) * df_end, 0.0)
    cn = cpv + mpv
    pv1 = funding - 1.0 + cn - put
    kof = torch.where(ko, funding - 1.0, 0.0)
    sums += torch.stack([pv1, pv1 * pv1, kof, kof * kof, put, put * put, cn, cn * cn, put, funding, 10.0 * cpv, 10.0 * mpv,
                         ko.double(), ki.double(), (ki & ~ko).double(), received.double()], dim=1).sum(2)


def _finish(sums, paths):
    """Prices and errors of the path sums, laid out as run() returns them."""
    s = sums.cpu().numpy()
    pv = s[:, 9] / paths + (s[:, 10] + s[:, 11]) / paths / 10.0 - s[:, 8] / paths
    err = np.sqrt((s[:, 1] - s[:, 0] ** 2 / paths) / (paths - 1) / paths)
    return {"pv": pv, "mc_error": err, "sums": s[:, :12], "counts": None}, s


def _stream(seed, count):
    """ChaCha8 (seeded through PCG32) feeding the 256-layer ziggurat: the first `count` normals."""
    state, key = seed, []
    for _ in range(8):
        state = (state * 6364136223846793005 + 11634580027462260723) & _M64
        xs, rot = (((state >> 18) ^ state) >> 27) & 0xFFFFFFFF, state >> 59
        key.append(((xs >> rot) | (xs << (32 - rot))) & 0xFFFFFFFF)
    blocks = (count + count // 32 + 8192) // 8
    s = [np.full(blocks, c, dtype=np.uint32) for c in (0x61707865, 0x3320646E, 0x79622D32, 0x6B206574, *key)]
    n = np.arange(blocks, dtype=np.uint64)
    s += [n.astype(np.uint32), (n >> np.uint64(32)).astype(np.uint32), np.zeros(blocks, np.uint32), np.zeros(blocks, np.uint32)]
    x = [a.copy() for a in s]

    def quarter(a, b, c, d):
        for i, j, k, r in ((a, b, d, 16), (c, d, b, 12), (a, b, d, 8), (c, d, b, 7)):
            x[i] += x[j]
            v = x[k] ^ x[i]
            x[k] = (v << np.uint32(r)) | (v >> np.uint32(32 - r))

    for _ in range(4):
        for q in ((0, 4, 8, 12), (1, 5, 9, 13), (2, 6, 10, 14), (3, 7, 11, 15),
                  (0, 5, 10, 15), (1, 6, 11, 12), (2, 7, 8, 13), (3, 4, 9, 14)):
            quarter(*q)
    words = np.stack([a + b for a, b in zip(x, s)], axis=1).astype("<u4").view("<u8").reshape(-1)
    R, V = 3.6541528853610088, 0.00492867323399
    zx = [V / math.exp(-R * R / 2.0), R]
    for _ in range(254):
        zx.append(math.sqrt(-2.0 * math.log(V / zx[-1] + math.exp(-zx[-1] ** 2 / 2.0))))
    zx.append(0.0)
    zf = np.array([float("%.18f" % math.exp(-v * v / 2.0)) for v in zx])
    zx = np.array([float("%.18f" % v) for v in zx])

    def unit(w, e):
        return ((w >> np.uint64(12)) | np.uint64((1023 + e) << 52)).view(np.float64)

    layer = (words & np.uint64(0xFF)).astype(np.int64)
    value = (unit(words, 1) - 3.0) * zx[layer]
    slow = np.flatnonzero(~(np.abs(value) < zx[layer + 1]))
    keep = np.ones(len(words), dtype=bool)
    pos = 0
    for at in slow[slow < len(words) - 1024].tolist():
        if at < pos:
            continue
        p = at
        while True:
            i, v = int(layer[p]), value[p]
            p += 1
            if abs(v) < zx[i + 1]:
                break
            if i == 0:
                while True:
                    a, b = (float(unit(words[p + j:p + j + 1], 0)[0]) - (1.0 - 2.0 ** -53) for j in (0, 1))
                    p += 2
                    e, f = math.log(a) / R, math.log(b)
                    if -2.0 * f >= e * e:
                        break
                v = e - R if v < 0.0 else R - e
                break
            u = float(words[p] >> np.uint64(11)) * 2.0 ** -53
            p += 1
            if zf[i + 1] + (zf[i] - zf[i + 1]) * u < math.exp(-v * v / 2.0):
                break
        value[at] = v
        keep[at + 1:p] = False
        pos = p
    return value[keep][:count]


def _trade_exact(case, seed):
    d = _trade_inputs(case, seed)
    n, steps, paths = case["assets"], case["steps"], case["paths"]
    sc, terms = d["scenarios"], d["terms"]
    S, dt = len(sc), terms["maturity_years"] / steps
    chunk = 1 << max(10, min(16, int(math.log2(4e8 / (n * steps)))))

    def tensor(v):
        return torch.tensor(np.asarray(v), dtype=torch.float64, device=_DEV)

    L = tensor([np.linalg.cholesky(np.asarray(m["correlation"])) for m, _ in sc])
    x0 = tensor([np.log(np.asarray(m["spots"]) / 100.0) for m, _ in sc])[:, :, None]
    mu = tensor([[(m["risk_free_rate"] - q) * dt for q in m["dividend_yields"]] for m, _ in sc])[:, :, None]
    vol = tensor([m["vols"] for m, _ in sc])[:, :, None]
    if d["grids"]:
        made = {}

        def surface(f, spot, rate, shift):
            key = (f, spot, rate, shift)
            if key not in made:
                made[key] = _dupire(d["grids"][f], spot, rate, shift, case["grid"])
            return made[key]

        surf = [[surface(f, m["spots"][f], m["risk_free_rate"], shift[f]) for f in range(n)] for m, shift in sc]
        rows = tensor([[_rows(s, steps, dt) for s in row] for row in surf])  # [S][n][steps][gx]
        logs = [[s[1] for s in row] for row in surf]
        lo = tensor([[a[0] for a in row] for row in logs])[:, :, None] - math.log(100.0)
        inv = tensor([[(len(a) - 1) / (a[-1] - a[0]) for a in row] for row in logs])[:, :, None]
        gx = case["grid"]
    sums = torch.zeros((S, 16), dtype=torch.float64, device=_DEV)
    cubes = []
    if case["lane"] == "stream":
        normals = torch.tensor(_stream(d["seed"], paths * steps * n)).view(paths, steps, n)
        spans = [(p, 0, min(chunk, paths - p)) for p in range(0, paths, chunk)]
    else:
        lane = _Lane(case["lane"], d["seed"], steps * n, chunk)
        # chunks of Sobol points aligned to the chunk size; path p reads point p + 1
        spans = [(k, 1 if k == 0 else 0, min(chunk, paths + 1 - k)) for k in range(0, paths + 1, chunk)]
        spans = [s for s in spans if s[2] > s[1]]
    for first, a, b in spans:
        if case["lane"] == "stream":
            dW = normals[first:first + b].to(_DEV).permute(1, 2, 0).contiguous() * math.sqrt(dt)
        else:
            dW = _bridge(lane.normals(first, a, b).view(steps, n, b - a), steps, dt)
        spot_rows = []

        def step(t, x):
            if d["grids"]:
                u = ((x - lo) * inv).clamp(0.0, gx - 1.0)
                j = u.long().clamp(max=gx - 2)
                r = rows[:, :, t, :]
                left, right = torch.gather(r, 2, j), torch.gather(r, 2, j + 1)
                sig = left + (u - j) * (right - left)
            else:
                sig = vol
            x = x + mu + sig * (L @ dW[t] - 0.5 * dt * sig)
            if case["kind"] == "replay":
                spot_rows.append(100.0 * torch.exp(x[0]))
            return x

        _scan([terms] * S, [m["risk_free_rate"] for m, _ in sc], x0.expand(S, n, b - a), step, sums)
        if spot_rows:
            cubes.append(torch.stack(spot_rows).permute(2, 0, 1).reshape(-1).cpu().numpy())
    if case["kind"] == "replay":
        return np.concatenate(cubes)
    out, s = _finish(sums, paths)
    if case["kind"] == "price":
        if case["trace"] != "off":
            out["trace_paths"] = out["trace_times"] = None
        return out
    # the risk report of the batch
    pv, err = out["pv"], out["mc_error"]
    total = {k: v[:1] if v is not None else None for k, v in out.items()}
    h = np.array([v * 0.01 for v in d["market"]["spots"]])
    up, down, vup, vdown = (1 + 4 * np.arange(n) + i for i in range(4))
    total["greeks"] = np.stack([(pv[up] - pv[down]) / (2 * h), (pv[up] - 2 * pv[0] + pv[down]) / h ** 2,
                                (pv[vup] - pv[vdown]) / 0.02], axis=1)
    total["bumped"] = np.stack([pv[up], pv[down], pv[vup], pv[vdown], err[up], err[down], err[vup], err[vdown]], axis=1)
    total["market"] = pv[1 + 4 * n:]
    impact = np.stack([s[:, 9] / paths * s[:, 12] / paths, -s[:, 8] / paths, (s[:, 10] + s[:, 11]) / paths / 10.0], axis=1)
    delta = ((impact[up] - impact[down]) / (2 * h[:, None])).sum(0)
    vega = ((impact[vup] - impact[vdown]) / 0.02).sum(0)
    total["transitions"] = np.stack([impact[0], delta, vega], axis=1)
    return total


def _trade_bumps(n):
    """A book trade's 15 bumps on its own underlyings, in the published order."""
    one, zero = [1.0] * n, [0.0] * n

    def at(base, idx, v):
        return [v if i in idx else b for i, b in enumerate(base)]

    pairs = [(i, j) for j in range(n) for i in range(j)]
    out = [(at(one, [f], 1.0 + h), zero, 0.0) for f in range(n) for h in (0.01, -0.01)]
    out += [(one, at(zero, [f], 0.01), 0.0) for f in range(n)] + [(one, zero, 1e-4)]
    out += [(at(one, p, 1.01), zero, 0.0) for p in pairs] + [(one, at(zero, [f], -0.01), 0.0) for f in range(n)]
    out += [(one, zero, -1e-4)] + [(at(one, p, 0.99), zero, 0.0) for p in pairs]
    for m in (2.0, 5.0, 10.0):
        out += [(at(one, [f], 1.0 + m * h), zero, 0.0) for f in range(n) for h in (0.01, -0.01)]
    out += [(one, at(zero, [f], h), 0.0) for f in range(n) for h in (0.02, -0.02)]
    out += [(one, zero, h) for h in (2e-4, -2e-4)]
    return out[:15]


def _book_exact(case, seed):
    d = _book_inputs(case, seed)
    u, paths, steps = d["universe"], case["paths"], DAYS * BOOK_YEARS
    dt, chunk = BOOK_YEARS / steps, 1 << 12
    lane = _Lane("sobol", d["seed"], UNIVERSE * steps, chunk)
    L = torch.tensor(np.linalg.cholesky(np.asarray(u["correlation"])), device=_DEV)
    groups = {}
    for j, (t, under) in enumerate(d["trades"]):
        groups.setdefault((len(under), t["steps"]), []).append(j)
    sums = torch.zeros((len(d["trades"]) * 16, 16), dtype=torch.float64, device=_DEV)
    for first in range(0, paths + 1, chunk):
        a, b = (1 if first == 0 else 0), min(chunk, paths + 1 - first)
        if b <= a:
            continue
        z = lane.normals(first, a, b).view(steps, UNIVERSE, b - a)
        dW = _bridge(L @ z, steps, dt)
        for (n, _), members in groups.items():
            markets = [{k: [u[k][i] for i in d["trades"][j][1]] for k in ("spots", "vols", "dividend_yields")}
                       | {"risk_free_rate": u["risk_free_rate"]} for j in members]
            rows = [_bumped(m, bump) for m in markets for bump in [([1.0] * n, [0.0] * n, 0.0)] + _trade_bumps(n)]
            idx = torch.tensor([d["trades"][j][1] for j in members], device=_DEV)

            def col(f):
                return torch.tensor([f(m) for m in rows], dtype=torch.float64, device=_DEV)[:, :, None]

            x0 = col(lambda m: [math.log(s / 100.0) for s in m["spots"]])
            sig = col(lambda m: m["vols"])
            mu = col(lambda m: [(m["risk_free_rate"] - q - 0.5 * v * v) * dt for q, v in zip(m["dividend_yields"], m["vols"])])

            def step(t, x):
                return x + mu + sig * dW[t][idx].repeat_interleave(16, dim=0)

            at = torch.tensor([j * 16 + k for j in members for k in range(16)], device=_DEV)
            part = torch.zeros((len(rows), 16), dtype=torch.float64, device=_DEV)
            _scan([d["trades"][j][0] for j in members for _ in range(16)], [m["risk_free_rate"] for m in rows],
                  x0.expand(-1, -1, b - a), step, part)
            sums[at] += part
    return _finish(sums, paths)[0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("price", "risk", "replay"):
        return _trade_exact(case, seed)
    if kind in ("book", "resident"):
        # the plain loop over every (trade, scenario) takes minutes on larger books
        return _book_exact(case, seed) if case["trades"] * case["paths"] <= 1 << 21 else None
    if kind == "cube":
        rng = random.Random(f"cube {seed}")
        m = _market(rng, case["assets"])
        z = _stream(rng.getrandbits(31), case["paths"] * case["steps"] * case["assets"])
        block = z.reshape(case["paths"], case["steps"], case["assets"]) @ np.linalg.cholesky(np.asarray(m["correlation"])).T
        vol, q = np.asarray(m["vols"]), np.asarray(m["dividend_yields"])
        drift = (m["risk_free_rate"] - q - 0.5 * vol * vol) / DAYS
        # the evolution reads the block in the 32 bits it is handed over in
        logs = np.cumsum(drift + vol * math.sqrt(1.0 / DAYS) * block.astype(np.float32).astype(np.float64), axis=1)
        return {"block": block.reshape(-1), "cube": (np.asarray(m["spots"]) * np.exp(logs)).reshape(-1)}
    b = _backend_inputs(case, seed)
    paths, steps, gx = case["paths"], case["steps"], case["grid"]

    def tensor(v):
        return torch.tensor(np.asarray(v, dtype=np.float64), device=_DEV)

    z = torch.tensor(b["normals"], device=_DEV).view(paths, steps, 2)
    rows, axis = tensor(b["rows"]).view(2, steps, gx), tensor(b["axis"]).view(2, gx)
    x = torch.log(tensor(b["spots"]))[:, None].expand(2, paths)
    mu = (b["rate"] - tensor(b["dividends"]))[:, None]
    dt = float(np.float32(1.0 / DAYS))
    for t in range(steps):
        u = ((x - axis[:, :1]) / (axis[:, -1:] - axis[:, :1]) * (gx - 1)).clamp(0.0, gx - 1.0)
        j = u.long().clamp(max=gx - 2)
        left, right = torch.gather(rows[:, t], 1, j), torch.gather(rows[:, t], 1, j + 1)
        sig = left + (u - j) * (right - left)
        x = x + (mu - 0.5 * sig * sig) * dt + sig * math.sqrt(dt) * z[:, t].T.double()
    return {"terminal": torch.exp(x).T.reshape(-1).cpu().numpy(), "ko": None}
