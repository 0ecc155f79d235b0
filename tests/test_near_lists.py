"""Three-side counts from neighbour lists: every class of job (one catalog, two
catalogs in each role order, three views) in the reference's mode and in clean
mode, at list sizes around one block, more than one list holds, and more near
tiles than a list of tiles holds; points on bin edges, lower edges above 0.
Counts equal the oracle's, or the plain FP64 kernel's where the loop is large
(integer histograms, tolerance 0)."""
import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

AXES = [(16, 0.0, 40.0), (32, 0.0, 32.0), (5, 3.0, 11.0), (1, 0.0, 9.0)]


def _both(eng, cats, handles, axis, ranges=None):
    sub = cats if ranges is None else [c[a:b] for c, (a, b) in zip(cats, ranges)]
    job = eng.job(handles, ranges)
    for overflow in (tpcf.OVERFLOW_COMPAT, tpcf.OVERFLOW_CLEAN):
        want, _ = oracle.three_side(sub, axis[1], axis[2], axis[0], clean=overflow == tpcf.OVERFLOW_CLEAN)
        s = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], overflow=overflow)
        assert np.array_equal(eng.count(s, job), want), (axis, overflow, ranges)


@pytest.mark.parametrize("n,m", [(1, 2), (3, 64), (31, 33), (65, 70), (150, 129), (333, 200)])
def test_classes(n, m):
    d = synth.lattice_mix(n, box=22.0, frac=0.5, seed=n)
    r = synth.lattice_mix(m, box=45.0, frac=0.3, seed=100 + m)
    t = synth.blobs(m, n_blobs=2, sigma=4.0, box=30.0, seed=200 + m)
    with tpcf.Engine(0) as eng:
        h = {id(c): eng.catalog(c) for c in (d, r, t)}
        for cats in ([d, d, d], [d, d, r], [d, r, r], [d, r, d], [r, d, t], [t, t, d]):
            for axis in AXES:
                _both(eng, cats, [h[id(c)] for c in cats], axis)
        if n > 60:  # overlapping ranges of one catalog: views of their own
            _both(eng, [d, d, d], [h[id(d)]] * 3, AXES[0], [(0, n), (5, 50), (20, n - 3)])
            _both(eng, [d, d, d], [h[id(d)]] * 3, AXES[1], [(5, 50)] * 3)


@pytest.mark.parametrize("axis", [(16, 0.0, 40.0), (20, 1.0, 15.0)])
def test_lists_that_overflow(axis):
    """Up to 1,500 neighbours a point (a list holds 1,024, or 512 of two)."""
    d = synth.blobs(1500, n_blobs=1, sigma=3.0, box=20.0, seed=1)
    r = synth.uniform(700, box=30.0, seed=2)
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        for hs in ([hd, hd, hd], [hd, hr, hr], [hr, hd, hd], [hd, hr, hd]):
            for overflow in (tpcf.OVERFLOW_COMPAT, tpcf.OVERFLOW_CLEAN):
                got, want = [eng.count(tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], overflow=overflow,
                                                      precision=p), eng.job(hs))
                             for p in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64)]
                assert np.array_equal(got, want), (hs, overflow)
        # two lists at once: ranges of one catalog
        job = eng.job([hd, hd, hr], [(0, 300), (100, 1500), (0, 700)])
        got, want = [eng.count(tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], precision=p), job)
                     for p in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64)]
        assert np.array_equal(got, want)


def test_too_many_near_tiles(monkeypatch):
    """Tiles of eight points: 290 near tiles, more than are listed; the launch
    is counted by tile triples instead."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    d = synth.blobs(2320, n_blobs=1, sigma=2.0, box=10.0, seed=3)
    with tpcf.Engine(0) as eng:
        h = eng.catalog(d)
        got, want = [eng.count(tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [(8, 0.0, 30.0)], precision=p),
                               eng.job([h, h, h])) for p in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64)]
        assert np.array_equal(got, want)


def test_summed_outputs():
    """Jobs of several classes and modes added into shared outputs."""
    d = synth.lattice_mix(300, box=30.0, frac=0.5, seed=4)
    r = synth.uniform(280, box=40.0, seed=5)
    axis = (16, 0.0, 20.0)
    combos = [[d, d, d], [d, d, r], [r, r, r], [d, r, d], [r, d, d]]
    want = [oracle.three_side(c, axis[1], axis[2], axis[0])[0] for c in combos]
    with tpcf.Engine(0) as eng:
        h = {id(d): eng.catalog(d), id(r): eng.catalog(r)}
        s = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis])
        for _ in range(3):  # planned, autotuned, replayed
            got = eng.count_batch_into([s] * 5, [eng.job([h[id(x)] for x in c]) for c in combos], [0, 1, 0, 1, 1], 2)
            assert np.array_equal(got[0], want[0] + want[2])
            assert np.array_equal(got[1], want[1] + want[3] + want[4])
