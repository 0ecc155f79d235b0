"""Batches whose plan passes its limits are counted in parts that add up: the
limits lowered so far that small batches are halved and single jobs go by a few
A tiles at a time, for every kernel that has a unit list, every loop nest and
role order.  Integer histograms equal the oracle's."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

TP = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
JBJ = [(8, 2.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)]
THREE = [(16, 0.0, 20.0)]
NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
NESTS = [("ddd", 0), ("ddr", 1), ("drr", 1), ("rdr", 1), ("rrd", 1), ("drd", 0), ("rrr", 0)]


def _want(kind, cats, which, axes):
    if kind == tpcf.THREE_SIDE:
        return oracle.three_side(cats, axes[0][1], axes[0][2], axes[0][0])[0]
    if kind == tpcf.TRIANGLE_JBJ:
        return oracle.triangle_jbj(cats, which, axes)[0]
    return oracle.triangle(cats, which, axes, nan_zero=NAN == tpcf.NAN_ZERO)[0]


def _check(monkeypatch, limit, value, kind, axes, precision, launches):
    """launches: of one count of a job that is not cut."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    monkeypatch.setenv("TPCF_NEAR", "0")
    monkeypatch.setenv("TPCF_TRI_LISTS", "0")
    monkeypatch.setenv("TPCF_AUTOTUNE", "0")
    cat = {"d": synth.lattice_mix(117, box=22.0, frac=0.5, seed=1), "r": synth.blobs(90, n_blobs=2, sigma=4.0, box=25.0, seed=2)}
    with tpcf.Engine(0) as eng:
        h = {k: eng.catalog(v) for k, v in cat.items()}
        jobs = [eng.job([h[x] for x in roles]) for roles, _ in NESTS]
        specs = [tpcf.make_spec(kind, tpcf.LOOP_ALL if kind == tpcf.THREE_SIDE else tpcf.LOOP_ONE if w else tpcf.LOOP_SAME,
                                axes, precision=precision, nan_policy=NAN) for _, w in NESTS]
        want = [_want(kind, [cat[x] for x in roles], w, axes) for roles, w in NESTS]
        whole = [eng.count(s, j) for s, j in zip(specs, jobs)]
        monkeypatch.setenv(limit, str(value))
        for s, j, a, w in zip(specs, jobs, whole, want):
            assert np.array_equal(a, w)
            assert np.array_equal(eng.count(s, j), w)
            assert eng.stats()["kernel_launches"] > launches
            assert eng.stats()["loop_units"] == eng.loop_units(s, j)
        assert all(np.array_equal(g, w) for g, w in zip(eng.count_batch(specs, jobs), want))
        assert eng.stats()["kernel_launches"] > launches * len(jobs)
        into = eng.count_batch_into(specs, jobs, [k % 2 for k in range(len(jobs))], 2)
        assert np.array_equal(into[0], sum(want[0::2])) and np.array_equal(into[1], sum(want[1::2]))
        tickets = [eng.submit(s, j) for s, j in zip(specs, jobs)]
        assert all(np.array_equal(eng.wait(t, s), w) for t, s, w in zip(tickets, specs, want))


KINDS = {
    "tp": (tpcf.TRIANGLE, TP, tpcf.GUARDED_FP32, 2),
    "tp64": (tpcf.TRIANGLE, TP, tpcf.PLAIN_FP64, 1),
    "jbj": (tpcf.TRIANGLE_JBJ, JBJ, tpcf.GUARDED_FP32, 1),
    "jbj64": (tpcf.TRIANGLE_JBJ, JBJ, tpcf.PLAIN_FP64, 1),
    "three": (tpcf.THREE_SIDE, THREE, tpcf.GUARDED_FP32, 1),
}


@pytest.mark.parametrize("name", sorted(KINDS))
def test_more_units_than_a_plan_may_have(monkeypatch, name):
    monkeypatch.setenv("TPCF_GROUP_TASKS", "1")  # (units of one tile triple, also of the fast kernel)
    _check(monkeypatch, "TPCF_MAX_UNITS", 300, *KINDS[name])


def test_a_tile_with_more_units_than_a_plan_may_have(monkeypatch):
    monkeypatch.setenv("TPCF_MAX_UNITS", "1")
    monkeypatch.setenv("TPCF_TRI_LISTS", "0")
    with tpcf.Engine(0) as eng:
        h = eng.catalog(synth.blobs(400, n_blobs=2, sigma=4.0, box=25.0, seed=3))
        with pytest.raises(tpcf.EngineError) as e:
            eng.count(tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, TP), eng.job([h] * 3))
        assert e.value.status == -1  # TPCF_ERR_INVALID


@pytest.mark.parametrize("name", sorted(KINDS))
def test_more_rows_than_a_plan_may_have(monkeypatch, name):
    _check(monkeypatch, "TPCF_MAX_ROWS", 17, *KINDS[name])


@pytest.mark.parametrize("precision", [tpcf.GUARDED_FP32, tpcf.PLAIN_FP64])
def test_pairs_with_more_items_than_a_plan_may_have(monkeypatch, precision):
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    monkeypatch.setenv("TPCF_MAX_ROWS", "60")  # (items of one tile pair)
    axis = (40, 0.0, 30.0)
    d, r = synth.lattice_mix(203, box=40.0, frac=0.5, seed=1), synth.uniform(150, box=40.0, seed=2)
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        cases = [([d, d], [hd, hd], tpcf.LOOP_SAME, 0), ([d, r], [hd, hr], tpcf.LOOP_ONE, 1),
                 ([r, d], [hr, hd], tpcf.LOOP_SAME, 0), ([r, r], [hr, hr], tpcf.LOOP_ALL, 1)]
        want = [oracle.pair(c, w, axis[1], axis[2], axis[0])[0] for c, _, _, w in cases]
        specs = [tpcf.make_spec(tpcf.PAIR, loop, [axis], precision=precision) for _, _, loop, _ in cases]
        jobs = [eng.job(h) for _, h, _, _ in cases]
        for s, j, w in zip(specs, jobs, want):
            assert np.array_equal(eng.count(s, j), w)
            assert eng.stats()["kernel_launches"] > 4
        assert all(np.array_equal(g, w) for g, w in zip(eng.count_batch(specs, jobs), want))


@pytest.mark.parametrize("kind,axes,env", [(tpcf.THREE_SIDE, THREE, "TPCF_NEAR"), (tpcf.TRIANGLE, TP, "TPCF_TRI_LISTS"),
                                           (tpcf.TRIANGLE_JBJ, JBJ, "TPCF_TRI_LISTS")])
def test_lists_with_more_items_than_a_plan_may_have(monkeypatch, kind, axes, env):
    """A batch of lists is halved to single jobs; one whose own lists pass the
    limit is counted from tiles."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    monkeypatch.setenv(env, "1")
    d, r = synth.lattice_mix(117, box=22.0, frac=0.5, seed=1), synth.uniform(17, box=20.0, seed=2)
    combos = [([d, r, r], 1), ([r, d, r], 1), ([d, d, d], 0), ([r, r, r], 0)]
    want = [_want(kind, c, w, axes) for c, w in combos]
    with tpcf.Engine(0) as eng:
        h = {id(d): eng.catalog(d), id(r): eng.catalog(r)}
        specs = [tpcf.make_spec(kind, tpcf.LOOP_ALL if kind == tpcf.THREE_SIDE else tpcf.LOOP_ONE if w else tpcf.LOOP_SAME,
                                axes, nan_policy=NAN) for _, w in combos]
        jobs = [eng.job([h[id(x)] for x in c]) for c, _ in combos]
        for limit in (200, 2000, 20000):
            monkeypatch.setenv("TPCF_MAX_ROWS", str(limit))
            assert all(np.array_equal(g, w) for g, w in zip(eng.count_batch(specs, jobs), want))
