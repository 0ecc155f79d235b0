"""Points so close that their squared separations are subnormal: every kernel
counts them as the reference's float operations do (forced through the
neighbour lists and through the tiles).  Integer histograms equal the oracle's."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
TP = [(8, 0.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
JBJ = [(8, 0.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)]


@pytest.mark.parametrize("lists", ["1", "0"])
@pytest.mark.parametrize("sigma", [1e-18, 1e-19, 1e-20, 1e-21, 1e-22])
def test_triangles(monkeypatch, lists, sigma):
    monkeypatch.setenv("TPCF_TRI_LISTS", lists)
    rng = np.random.default_rng(1)
    d = np.concatenate([rng.normal(0, sigma, (90, 3)), rng.normal(0, 3.0, (40, 3))]).astype(np.float32)
    r = np.concatenate([rng.normal(0, sigma, (70, 3)), rng.normal(0, 3.0, (30, 3))]).astype(np.float32)
    with tpcf.Engine(0) as eng:
        h = {id(d): eng.catalog(d), id(r): eng.catalog(r)}
        for c, w in (([d, d, d], 0), ([d, d, r], 1), ([d, r, r], 1)):
            j = eng.job([h[id(x)] for x in c])
            loop = tpcf.LOOP_ONE if w else tpcf.LOOP_SAME
            got = eng.count(tpcf.make_spec(tpcf.TRIANGLE, loop, TP, nan_policy=NAN), j)
            want = oracle.triangle(c, w, TP, nan_zero=NAN == tpcf.NAN_ZERO)[0]
            assert np.array_equal(got, want), (w, int((got != want).sum()))
            got = eng.count(tpcf.make_spec(tpcf.TRIANGLE_JBJ, loop, JBJ, nan_policy=NAN), j)
            want = oracle.triangle_jbj(c, w, JBJ)[0]
            assert np.array_equal(got, want), (w, int((got != want).sum()))


@pytest.mark.parametrize("near", ["1", "0"])
@pytest.mark.parametrize("axis", [(16, 0.0, 20.0), (7, 0.0, 1e-19), (5, 3e-20, 2e-19)])
def test_sides_and_pairs(monkeypatch, near, axis):
    monkeypatch.setenv("TPCF_NEAR", near)
    rng = np.random.default_rng(1)
    for sigma in (1e-18, 1e-20, 1e-21, 1e-22):
        d = np.concatenate([rng.normal(0, sigma, (90, 3)), rng.normal(0, 3.0, (40, 3))]).astype(np.float32)
        with tpcf.Engine(0) as eng:
            h = eng.catalog(d)
            for overflow in (tpcf.OVERFLOW_COMPAT, tpcf.OVERFLOW_CLEAN):
                want, _ = oracle.three_side([d] * 3, axis[1], axis[2], axis[0], clean=overflow == tpcf.OVERFLOW_CLEAN)
                s = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], overflow=overflow)
                assert np.array_equal(eng.count(s, eng.job([h] * 3)), want), (sigma, overflow)
            want, _ = oracle.pair([d, d], 0, axis[1], axis[2], axis[0])
            assert np.array_equal(eng.count(tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_SAME, [axis]), eng.job([h, h])), want)
