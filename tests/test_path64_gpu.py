"""The FP64 lane's kernels of an engine against the one-kernel form of the static entry point.

Both run the reference's arithmetic product by product, one path at a time, so every event count is
equal and the path sums differ only by the order of the FP64 additions over paths: at most `paths`
roundings of 2^-53 on sums of terms below 10 (coupon quotes are on the x10 scale).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from riga_gb300 import abi, workloads
from riga_gb300.build import build_library
from riga_gb300.engine import Engine
from riga_gb300.types import VarianceReduction

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    build_library()
    e = Engine(0)
    yield e
    e.close()


def _request(n, paths, steps, smile=None, lane="shift", **terms):
    if smile:
        req = workloads.lv3(paths, steps, fp32=False)
        req.local_vol, _ = workloads.svi_grids(n, seed=n, n_k=smile[0], n_t=smile[1], years=steps / 252)
        req.options.lv_grid_x = smile[2]
    else:
        req = workloads.plain3(paths, steps)
    req.trade = workloads.phoenix_trade(n, steps, steps / 252)
    m = req.market
    m.spots, m.vols = [100.0 + f for f in range(n)], [0.18 + 0.05 * f for f in range(n)]
    m.dividend_yields = [0.01] * n
    m.correlation = [[1.0 if i == j else 0.45 for j in range(n)] for i in range(n)]
    if lane == "owen":
        req.options.scrambler, req.options.dim_mode = abi.SCRAMBLE_OWEN, abi.DIM_WRAP_REFERENCE
    elif lane.startswith("halton"):
        req.config.variance_reduction = VarianceReduction("halton", n * steps)
        if lane == "halton512":
            req.options.dim_mode = abi.DIM_WRAP_REFERENCE
    for k, v in terms.items():
        setattr(req.trade, k, v)
    return req


def _check(engine, req):
    a = req.to_abi()
    want = abi.PriceResult()
    abi.check(engine.lib, engine.lib.rg_price_put_leg_static(a.ptr, C.byref(want)))
    got = engine.price_raw(req)
    assert list(got.path_sums)[12:] == list(want.path_sums)[12:]
    for x, y in zip(list(got.path_sums)[:12], list(want.path_sums)[:12]):
        assert abs(x - y) <= 10.0 * req.config.paths ** 2 * 2.0 ** -53
    return got


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("paths,steps", [(1, 1), (31, 2), (257, 63), (1000, 100)])
@pytest.mark.parametrize("smile", [None, (13, 1, 2), (20, 5, 96)])
def test_engine_and_static_kernels_agree(engine, n, paths, steps, smile):
    _check(engine, _request(n, paths, steps, smile))


@pytest.mark.parametrize("lane", ["owen", "halton", "halton512"])
@pytest.mark.parametrize("first", [0, 5, 31, 1000])
def test_lanes_and_offsets_agree(engine, lane, first):
    req = _request(3, 300, 40, (13, 3, 40), lane)
    req.options.first_path = first
    _check(engine, req)


@pytest.mark.parametrize("terms", [
    dict(coupon_periods=1), dict(coupon_periods=90), dict(coupon_periods=200), dict(fixed_first_coupon=True),
    dict(knock_out_barrier=None), dict(coupon_barrier=None), dict(memory_coupon=False), dict(call_start_step=0),
    dict(call_start_step=1000), dict(knock_out_barrier=0.5, call_start_step=0), dict(knock_in_barrier=5.0),
    dict(coupon_rate=None), dict(coupon_periods=7, fixed_first_coupon=True, call_start_step=3),
])
def test_schedules_agree(engine, terms):
    _check(engine, _request(2, 400, 90, None, **terms))


@pytest.mark.parametrize("vol,years", [(0.0, 1.0), (6.0, 30.0), (40.0, 60.0), (1e-9, 1e-6)])
def test_extreme_paths_agree(engine, vol, years):
    """Steps beyond the exponential's short range, spots that underflow to zero or overflow, and paths
    that do not move."""
    req = _request(3, 128, 30)
    req.trade.maturity_years = years
    req.market.vols = [vol] * 3
    _check(engine, req)


@pytest.mark.parametrize("init", [1e-3, 0.73, 1.0, 3.1, 1e6])
@pytest.mark.parametrize("terms", [dict(knock_out_barrier=None, coupon_barrier=None), dict(), dict(knock_out_barrier=1.0 / 3.0),
                                   dict(knock_out_barrier=1e300, coupon_barrier=1e300)])
def test_initial_spots_agree(engine, init, terms):
    """The engine's kernels compare spots with thresholds, the static one's ratios with barriers: the same
    events at initial spots whose ratios round differently, with barriers absent, ordinary and beyond reach."""
    req = _request(3, 500, 60, None, **terms)
    req.trade.initial_spots = [init * (1.0 + 0.1 * f) for f in range(3)]
    req.market.spots = [s * 1.01 for s in req.trade.initial_spots]
    _check(engine, req)


def _as_array(records):
    return np.ctypeslib.as_array(records)


@pytest.mark.parametrize("n,paths,steps,lane,smile", [
    (1, 9001, 15001, "shift", None), (3, 3205, 14999, "shift", None), (2, 5000, 15000, "owen", (13, 2, 40)),
    (5, 1801, 15013, "owen", None), (4, 2305, 15000, "none", None), (1, 8300, 16384, "none", (13, 2, 40))])
def test_windows_of_long_schedules_agree(engine, n, paths, steps, lane, smile):
    """Schedules too long for the buffer to hold all paths' normals pass through it in windows of steps, each
    path's state carried between them: the records of every path have the bytes of launches of a few paths,
    whose whole schedules it holds, and the path sums those of the records."""
    req = _request(n, paths, steps, smile, "owen" if lane == "none" else lane)
    if lane == "shift":
        req.options.dim_mode = abi.DIM_WRAP_REFERENCE
    if lane == "none":
        req.config.variance_reduction = VarianceReduction("none", n * steps)
    assert n * paths * steps * 8 > 1 << 30
    whole = _as_array(engine.run_paths_raw(req, 0, paths)).copy()
    cuts = [0, 1, 700, 1500, paths] if paths < 2400 else [0, 700, 701, paths // 2, paths]
    parts = [_as_array(engine.run_paths_raw(req, a, b - a)).copy() for a, b in zip(cuts, cuts[1:])]
    assert all(n * (b - a) * steps * 8 <= 1 << 30 for a, b in zip(cuts, cuts[1:]))
    split = np.concatenate(parts)
    for field in whole.dtype.names:
        np.testing.assert_array_equal(whole[field], split[field])
    got = engine.price_raw(req)
    assert got.ko_count == int((whole["knocked_out"] != 0).sum())
    assert abs(got.pv - whole["pv"].mean()) <= 10.0 * paths * 2.0 ** -53


def test_windows_fill_the_spot_cube(engine):
    """A cube of long paths, whose normals pass through the buffer in windows, equals its halves."""
    req = _request(1, 600, 240001, None, "owen")
    whole, _ = engine.materialize_paths(req, 0, 600)
    low, _ = engine.materialize_paths(req, 0, 299)
    high, _ = engine.materialize_paths(req, 299, 301)
    w = np.asarray(whole.data)
    assert np.array_equal(w[:299 * 240001], np.asarray(low.data))
    assert np.array_equal(w[299 * 240001:], np.asarray(high.data))


@pytest.mark.parametrize("n,lane,smile", [(1, "shift", None), (2, "owen", (13, 3, 40)), (3, "shift", (20, 5, 96)),
                                          (4, "owen", None), (5, "shift", (13, 3, 25))])
def test_records_have_the_oracles_bits(engine, n, lane, smile):
    """Per path the lane performs the oracle's operations (its portable exponential and logarithm) in the
    oracle's order, so every field of every record has the oracle's bits."""
    import oracle as O
    req = _request(n, 2000, 130, smile, lane)
    O.set_portable_math(True)
    try:
        want = O.run_paths(req, 0, 2000)
    finally:
        O.set_portable_math(False)
    got = _as_array(engine.run_paths_raw(req, 0, 2000))
    for f in ("worst_final", "ko_step", "ki_hit", "qualified_steps", "paid_periods", "put_payoff", "coupon_pv",
              "memory_coupon_pv", "funding", "pv"):
        np.testing.assert_array_equal(got[f], np.array([getattr(r, f) for r in want], got[f].dtype), err_msg=f)
