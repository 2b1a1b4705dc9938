"""GPU tests of the pseudo-random lane (ChaCha8Rng → StandardNormal generated on the device) and
of the PathCube drop-ins, against the oracle (which reproduces the reference's golden bit for bit).

Bars: the device normal stream equals the oracle's draw for draw (any seed, any offset);
generate_correlated_block equals the oracle's f32 block exactly; gbm_evolve within 1 f32 ulp
(CUDA's exp/log against the host libm, ≥ 99.9% of cells identical); the MC lane's per-path records
— KO step, coupon counts exact, payoffs within 1e-12 — and prices within 1e-12 of the oracle
(portable exp/log on both sides); and the reference's termsheet1 golden PriceResult (30,000
paths, Dupire local vol) reproduced on the GPU within the reference's 1e-12 with all 64 KO trace events exact.
"""
from __future__ import annotations

import copy
import math

import numpy as np
import pytest

import oracle as O
from conftest import json_close
from riga_gb300 import abi, pathcube
from riga_gb300.build import build_library
from riga_gb300.engine import Engine
from riga_gb300.types import result_to_json

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    build_library()
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("seed", [1, 7, 1729, (1 << 63) + 5])
def test_device_stream_equals_the_oracle(seed):
    n = 1 << 20
    want = np.frombuffer(O.chacha8_normals(seed, n), dtype=np.float64)
    got = pathcube.chacha8_normals(seed, 0, n)
    assert np.array_equal(got, want)
    for first, count in ((12345, 1000), (n - 777, 777), (0, 1)):
        assert np.array_equal(pathcube.chacha8_normals(seed, first, count), want[first:first + count])


@pytest.mark.parametrize("first,count", [
    (0, 1), (0, 31), (0, 2047), (0, 2049), (2040, 20),            # around one 2048-word segment
    (0, 128 * 2048 - 3000), (128 * 2048 - 4000, 8000),            # around one group of 128 segments
    (255 * 2048, 3 * 128 * 2048 + 77), (900_001, 1),
])
def test_stream_ranges_across_segments_and_groups(first, count):
    """The parallel parse at its seams: ranges that start, end and straddle the parse's segments and
    segment groups are the oracle's draws, bit for bit."""
    want = np.frombuffer(O.chacha8_normals(99, first + count), dtype=np.float64)[first:]
    assert np.array_equal(pathcube.chacha8_normals(99, first, count).view(np.uint64), want.view(np.uint64))


def test_correlated_block_equals_the_oracle():
    for corr in ([[1.0, 0.5], [0.5, 1.0]], [[1.0, 0.3, 0.1], [0.3, 1.0, 0.2], [0.1, 0.2, 1.0]]):
        L = O.cholesky(corr)
        got = pathcube.generate_correlated_block(7, 1024, 64, L)
        want = np.frombuffer(O.generate_correlated_block(7, 1024, 64, L), dtype=np.float32)
        assert np.array_equal(got.data, want)


def test_gbm_evolve_within_one_ulp_of_the_oracle():
    L = O.cholesky([[1.0, 0.5], [0.5, 1.0]])
    blk = pathcube.generate_correlated_block(7, 2048, 252, L)
    cube = pathcube.gbm_evolve([100.0, 50.0], [0.2, 0.3], 0.03, [0.01, 0.0], 1 / 252, blk)
    want = np.frombuffer(O.gbm_evolve([100.0, 50.0], [0.2, 0.3], 0.03, [0.01, 0.0], 1 / 252, blk.data,
                                      2048, 252), dtype=np.float32)
    ulps = np.abs(cube.data.view(np.int32).astype(np.int64) - want.view(np.int32).astype(np.int64))
    assert ulps.max() <= 1 and (ulps == 0).mean() >= 0.999


def test_mc_lane_records_match_the_oracle(engine, termsheet1):
    O.set_portable_math(True)
    try:
        r = copy.deepcopy(termsheet1.request)
        r.config.paths = 2048
        got = engine.run_paths_raw(r, 100, 512)
        want = O.run_paths(r, 100, 512)
    finally:
        O.set_portable_math(False)
    for g, w in zip(got, want):
        assert (g.path_id, g.knocked_out, g.ko_step, g.ki_hit, g.qualified_steps, g.paid_periods, g.sobol_index) == \
            (w.path_id, w.knocked_out, w.ko_step, w.ki_hit, w.qualified_steps, w.paid_periods, w.sobol_index)
        for f in ("pv", "put_payoff", "coupon_pv", "memory_coupon_pv", "funding", "worst_final"):
            a, b = getattr(g, f), getattr(w, f)
            assert abs(a - b) <= 1e-12 * max(abs(b), 1e-300), f


def test_termsheet1_golden_on_the_gpu(engine, termsheet1, golden_result):
    """The reference's golden vector (crates/riga-engine/src/lib.rs:489-498) priced by the GPU at
    the reference's own 1e-12: the device draws the same ChaCha8 stream, so every count and trace
    event is exact; the surfaces are calibrated from host-libm axes as the reference's, and only
    the per-path exp/log (portable, within 2 ulp of libm) differ in the last bits."""
    res = engine.price_raw(termsheet1.request)
    got = result_to_json(res, termsheet1.request)
    assert json_close(got, golden_result, tol=1e-12) == []
    assert got["determinism"] == golden_result["determinism"]
    O.set_portable_math(True)
    try:
        want = O.price_put_leg(termsheet1.request, threads=1)
    finally:
        O.set_portable_math(False)
    assert (res.ko_count, res.ki_count, res.put_eligible_count, res.coupon_path_count) == \
        (want.ko_count, want.ki_count, want.put_eligible_count, want.coupon_path_count)
    assert abs(res.pv - want.pv) <= 1e-12 * abs(want.pv)


def test_mc_lane_scenarios_share_the_stream(engine, termsheet1):
    r = copy.deepcopy(termsheet1.request)
    r.config.paths = 4096
    up = copy.deepcopy(r.market)
    up.spots = [s * 1.01 for s in up.spots]
    got = engine.price_scenarios_raw(r, [(r.market, None), (up, None)])
    O.set_portable_math(True)
    try:
        want = O.price_scenarios(r, [(r.market, None), (up, None)], threads=8)
    finally:
        O.set_portable_math(False)
    for g, w in zip(got, want):
        assert g.ko_count == w.ko_count and abs(g.pv - w.pv) <= 1e-12 * abs(w.pv)
