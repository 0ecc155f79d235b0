"""Pair kernels at the sizes where tiles, half tiles and chunks of tiles end:
counts equal the oracle's for one catalog (self pairs and j >= i), two catalogs
under every loop nest, index ranges, and separations on bin edges, through both
pair entry points; NaN and infinite coordinates are counted nowhere.
Integer histograms: tolerance 0."""
import numpy as np
import pytest

import oracle
import synth
import tpcf
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu

# bins wide and narrow, lower edge above 0, more bins than fit a table of 700
AXES = [(700, 0.0, 70.0), (32, 0.0, 32.0), (10, 5.0, 9.0), (3000, 1.0, 50.0)]


@pytest.fixture(scope="module")
def eng():
    e = tpcf.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("n,m", [(1, 1), (2, 63), (31, 65), (64, 64), (65, 33), (127, 129), (515, 64), (2113, 700)])
def test_tile_edges(eng, n, m):
    d = synth.lattice_mix(n, box=40.0, frac=0.5, seed=n)
    r = synth.lattice_mix(m, box=60.0, frac=0.5, seed=1000 + m)
    hd, hr = eng.catalog(d), eng.catalog(r)
    for axis in AXES:
        for cats, hs, loop, which in (([d, d], [hd, hd], tpcf.LOOP_SAME, 0), ([d, r], [hd, hr], tpcf.LOOP_ONE, 1),
                                      ([d, r], [hd, hr], tpcf.LOOP_SAME, 0), ([r, d], [hr, hd], tpcf.LOOP_ALL, 1)):
            want, _ = oracle.pair(cats, which, axis[1], axis[2], axis[0])
            for precision in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64):
                got = eng.count(tpcf.make_spec(tpcf.PAIR, loop, [axis], precision=precision), eng.job(hs))
                assert np.array_equal(got, want), (axis, loop, precision)
            assert np.array_equal(_noalloc(cats[0], cats[1], loop, axis, cats[0] is cats[1]), want), (axis, loop)
    eng.release(hd)
    eng.release(hr)


def test_many_jobs_and_empty_ranges(eng):
    """More jobs than one step of the job search, empty ranges among them."""
    d = synth.uniform(900, box=50.0, seed=5)
    h = eng.catalog(d)
    spec = tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_SAME, [(40, 0.0, 20.0)])
    ranges = [(7 * k % 800, 7 * k % 800 + (0 if k % 5 == 0 else 1 + 13 * k % 97)) for k in range(75)]
    got = eng.count_batch([spec] * 75, [eng.job([h, h], [r, r]) for r in ranges])
    for (a, b), g in zip(ranges, got):
        want = oracle.pair([d[a:b], d[a:b]], 0, 0.0, 20.0, 40)[0] if b > a else np.zeros(40, np.uint64)
        assert np.array_equal(g, want), (a, b)
    eng.release(h)


def test_points_that_are_not_numbers(eng):
    d = synth.uniform(300, box=30.0, seed=6)
    bad = d.copy()
    bad[::7, 0], bad[3::11, 1], bad[5::50, 2] = np.nan, np.inf, -np.inf
    good = bad[np.isfinite(bad).all(1)]
    axis = (40, 0.0, 20.0)
    want, _ = oracle.pair([good, d], 1, axis[1], axis[2], axis[0])
    hb, hd = eng.catalog(bad), eng.catalog(d)
    assert np.array_equal(eng.count(tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_ONE, [axis]), eng.job([hb, hd])), want)
    assert np.array_equal(_noalloc(bad, d, tpcf.LOOP_ONE, axis, False), want)
    eng.release(hb)
    eng.release(hd)
