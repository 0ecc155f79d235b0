"""The device planner at its edges: catalogs around one window of tiles, every
loop nest and role order, more units than the unit list first holds, and many
jobs with empty ranges.  Integer histograms equal the oracle's."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

TP = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN


@pytest.mark.parametrize("n,m", [(1, 3), (63, 65), (64, 129), (257, 40), (260, 320), (530, 200)])
def test_windows_and_role_orders(n, m):
    """One to nine tiles per catalog (windows of four): a last window of one
    tile, tiles of one point, and each role order, with and without pruning."""
    d = synth.blobs(n, n_blobs=3, sigma=5.0, box=40.0, seed=n)
    r = synth.uniform(m, box=40.0, seed=m)
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        h = {id(d): hd, id(r): hr}
        combos = [([d, d, d], 0), ([d, d, r], 1), ([d, r, r], 1), ([r, d, r], 1), ([r, r, d], 1), ([d, r, d], 0),
                  ([r, r, r], 0)]
        want = [oracle.triangle(c, w, TP, nan_zero=NAN == tpcf.NAN_ZERO)[0] for c, w in combos]
        jobs = [eng.job([h[id(x)] for x in c]) for c, _ in combos]
        for prune in (True, False):
            for precision in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64):
                specs = [tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE if w else tpcf.LOOP_SAME, TP, precision=precision,
                                        nan_policy=NAN, prune=prune) for _, w in combos]
                for _ in range(2):  # planned, then repeated
                    for g, w in zip(eng.count_batch(specs, jobs), want):
                        assert np.array_equal(g, w), (prune, precision)


def test_unit_list_overflow(monkeypatch):
    """Tiles of eight points: 2.1 million tile triples, twice what the unit list
    first holds; the list grows and the count is exact, also when repeated."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    d = synth.uniform(1100, box=50.0, seed=1)
    r = synth.lattice_mix(1000, box=50.0, frac=0.5, seed=2)
    axis = (10, 0.0, 20.0)
    want, _ = oracle.three_side([d, r, r], axis[1], axis[2], axis[0])
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        spec = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], prune=False)
        for _ in range(3):
            assert np.array_equal(eng.count(spec, eng.job([hd, hr, hr])), want)
            assert eng.stats()["tasks"] == 138 * 125 * 125


def test_many_jobs_with_empty_ranges():
    d = synth.blobs(700, n_blobs=4, sigma=5.0, box=40.0, seed=3)
    spec = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, TP, nan_policy=NAN)
    ranges = [(5 * k % 600, 5 * k % 600 + (0 if k % 7 == 0 else 1 + 11 * k % 90)) for k in range(130)]
    with tpcf.Engine(0) as eng:
        h = eng.catalog(d)
        jobs = [eng.job([h, h, h], [r, r, r]) for r in ranges]
        got = eng.count_batch([spec] * len(jobs), jobs)
        units = 0
        for (a, b), g in zip(ranges, got):
            if b > a:
                want, n = oracle.triangle([d[a:b]] * 3, 0, TP, nan_zero=NAN == tpcf.NAN_ZERO)
                units += n
            else:
                want = np.zeros_like(g)
            assert np.array_equal(g, want), (a, b)
        eng.count_batch([spec] * len(jobs), jobs)
        assert eng.stats()["loop_units"] == units
