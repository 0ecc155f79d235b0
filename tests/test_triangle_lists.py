"""Triangle and JBJ counts from neighbour lists (forced, as small catalogs keep
the tile kernel): every loop nest and role order, lists around 32 and 64
entries and many times that, more near tiles than are kept, duplicate points
and equal sides (lattices: the longest side shared), shares of centres, and
histograms of several outputs beside one another or one at a time.  Integer
histograms equal the oracle's, in FP64 geometry the exhaustive kernel's."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
TP = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
FINE = [(50, 2.0, 12.0), (16, 0.9, 4.1), (25, 0.0, 1.0)]  # one output's histogram in shared memory
JBJ = [(8, 2.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)]


@pytest.fixture
def lists(monkeypatch):
    monkeypatch.setenv("TPCF_TRI_LISTS", "1")


def _check(cats, kind, axes):
    d, r = cats
    combos = [([d, d, d], 0), ([d, d, r], 1), ([d, r, r], 1), ([r, d, r], 1), ([d, r, d], 0), ([r, r, d], 1), ([r, r, r], 0)]
    with tpcf.Engine(0) as eng:
        h = {id(d): eng.catalog(d), id(r): eng.catalog(r)}
        specs = [tpcf.make_spec(kind, tpcf.LOOP_ONE if w else tpcf.LOOP_SAME, axes, nan_policy=NAN) for _, w in combos]
        jobs = [eng.job([h[id(x)] for x in c]) for c, _ in combos]
        for _ in range(2):  # planned, then autotuned
            got = eng.count_batch(specs, jobs)
            for (c, w), g in zip(combos, got):
                want = (oracle.triangle(c, w, axes, nan_zero=NAN == tpcf.NAN_ZERO) if kind == tpcf.TRIANGLE
                        else oracle.triangle_jbj(c, w, axes))[0]
                assert np.array_equal(g, want), (w, [len(x) for x in c])


@pytest.mark.parametrize("n,m", [(1, 2), (3, 31), (33, 64), (65, 32), (129, 200), (420, 150)])
@pytest.mark.parametrize("name", ["tp", "fine", "jbj"])
def test_blobs(lists, n, m, name):
    kind, axes = {"tp": (tpcf.TRIANGLE, TP), "fine": (tpcf.TRIANGLE, FINE), "jbj": (tpcf.TRIANGLE_JBJ, JBJ)}[name]
    _check((synth.blobs(n, n_blobs=2, sigma=4.0, box=25.0, seed=n), synth.uniform(m, box=35.0, seed=m)), kind, axes)


@pytest.mark.parametrize("name", ["tp", "jbj"])
def test_lattices_and_duplicates(lists, name):
    kind, axes = {"tp": (tpcf.TRIANGLE, TP), "jbj": (tpcf.TRIANGLE_JBJ, JBJ)}[name]
    base = synth.lattice_mix(140, box=14.0, frac=1.0, seed=1)
    _check((np.concatenate([base, base[:50]]), synth.lattice_mix(150, box=18.0, frac=0.7, seed=2)), kind, axes)


def test_more_near_tiles_than_are_kept(lists, monkeypatch):
    """Tiles of eight points: some 90 near tiles, found again at every pass."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    _check((synth.blobs(700, n_blobs=1, sigma=4.0, box=20.0, seed=3), synth.uniform(300, box=30.0, seed=4)),
           tpcf.TRIANGLE, TP)


@pytest.mark.parametrize("cap", ["16", ""])
def test_geometry_and_recheck_overflow(lists, monkeypatch, cap):
    if cap:
        monkeypatch.setenv("TPCF_RECHECK_CAP", cap)
        monkeypatch.setenv("TPCF_GRAPHS", "0")
    d = synth.lattice_mix(400, box=20.0, frac=0.6, seed=5)
    far = np.concatenate([d, np.array([[2e15, 2e15, 2e15]], np.float32)])  # the exhaustive kernel
    with tpcf.Engine(0) as eng:
        s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, TP, precision=tpcf.GEOMETRY_FP64, nan_policy=NAN)
        got = [eng.count(s, eng.job([h, h, h])) for h in (eng.catalog(d), eng.catalog(far))]
        assert np.array_equal(*got) and got[0].sum() > 0
        s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, TP, nan_policy=NAN)
        h = eng.catalog(d)
        assert np.array_equal(eng.count(s, eng.job([h, h, h])), oracle.triangle([d] * 3, 0, TP, nan_zero=NAN == tpcf.NAN_ZERO)[0])
        assert eng.stats()["recheck_regrows"] == (0 if not cap else eng.stats()["recheck_regrows"])


def test_routes_agree_at_the_rules_edges(monkeypatch):
    """Sparse catalogs and large histograms, which take the lists by themselves,
    against the tile kernel."""
    for axes, n in ((TP, 1500), (FINE, 500)):
        d = synth.lightcone(n, clustered=True, n_blobs=n // 25, half_angle_deg=2.5, seed=6)
        r = synth.lightcone(n, half_angle_deg=2.5, seed=7)
        res = []
        for env in (None, "0"):
            if env is None:
                monkeypatch.delenv("TPCF_TRI_LISTS", raising=False)
            else:
                monkeypatch.setenv("TPCF_TRI_LISTS", env)
            with tpcf.Engine(0) as eng:
                hd, hr = eng.catalog(d), eng.catalog(r)
                loops = [tpcf.LOOP_SAME, tpcf.LOOP_ONE, tpcf.LOOP_ONE, tpcf.LOOP_SAME]
                specs = [tpcf.make_spec(tpcf.TRIANGLE, lp, axes, nan_policy=NAN) for lp in loops]
                res.append(eng.count_batch(specs, [eng.job(h) for h in ([hd] * 3, [hd, hd, hr], [hd, hr, hr], [hr] * 3)]))
        for a, b in zip(*res):
            assert np.array_equal(a, b)
        assert sum(int(a.sum()) for a in res[0]) > 0
