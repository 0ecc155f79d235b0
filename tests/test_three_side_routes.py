"""Which way a three-side batch is counted: from tiles where most triples are in
range or few tiles are in reach, from neighbour lists elsewhere, and from tiles
again and again (planned once, replayed) where the lists were refused.  The lists
as such, forced wherever they are possible, at the sizes of test_near_lists."""
import numpy as np
import pytest

import synth
import test_near_lists
import tpcf

pytestmark = pytest.mark.gpu


def _spec(overflow, axis, precision=tpcf.GUARDED_FP32):
    return tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [axis], overflow=overflow, precision=precision)


@pytest.mark.parametrize("overflow", [tpcf.OVERFLOW_COMPAT, tpcf.OVERFLOW_CLEAN])
@pytest.mark.parametrize("n,hi,bins,tiles", [
    (1000, 180.0, 16, {tpcf.OVERFLOW_COMPAT: True, tpcf.OVERFLOW_CLEAN: False}),
    (1000, 40.0, 16, {tpcf.OVERFLOW_COMPAT: False, tpcf.OVERFLOW_CLEAN: False}),
    (1000, 8.0, 32, {tpcf.OVERFLOW_COMPAT: False, tpcf.OVERFLOW_CLEAN: True}),
    (300, 40.0, 16, {tpcf.OVERFLOW_COMPAT: False, tpcf.OVERFLOW_CLEAN: False}),
])
def test_rule(monkeypatch, overflow, n, hi, bins, tiles):
    d = synth.uniform(n, box=100.0, seed=n)
    with tpcf.Engine(0) as eng:
        j = eng.job([eng.catalog(d)] * 3)
        s = _spec(overflow, (bins, 0.0, hi))
        got = eng.count(s, j)
        tasks = {"default": eng.stats()["tasks"]}
        for env in "01":
            monkeypatch.setenv("TPCF_NEAR", env)
            assert np.array_equal(eng.count(s, j), got)
            tasks[env] = eng.stats()["tasks"]
        assert tasks["0"] != tasks["1"]
        assert tasks["default"] == tasks["0" if tiles[overflow] else "1"]
    assert got.sum() > 0


@pytest.mark.parametrize("overflow", [tpcf.OVERFLOW_COMPAT, tpcf.OVERFLOW_CLEAN])
def test_sets_of_small_jobs_go_to_the_tiles(monkeypatch, overflow):
    """Every job of such a set would make a launch's CTAs change accumulators."""
    d = synth.uniform(20000, box=200.0, seed=7)
    begin = np.random.default_rng(1).integers(0, 19900, (50, 3))
    tasks = {}
    with tpcf.Engine(0) as eng:
        h = eng.catalog(d)
        jobs = [eng.job([h] * 3, [(int(x), int(x) + 100) for x in b]) for b in begin]
        res = []
        for env in (None, "0", "1"):
            if env:
                monkeypatch.setenv("TPCF_NEAR", env)
            res.append(eng.count_batch([_spec(overflow, (16, 0.0, 32.0))] * len(jobs), jobs))
            tasks[env] = eng.stats()["tasks"]
        assert all(np.array_equal(a, b) and np.array_equal(a, c) for a, b, c in zip(*res))
    assert tasks[None] == tasks["0"] != tasks["1"]


def test_refused_lists_are_not_tried_again(monkeypatch):
    """Tiles of eight points: 290 near tiles, more than are listed."""
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    monkeypatch.setenv("TPCF_AUTOTUNE", "0")
    d = synth.blobs(2320, n_blobs=1, sigma=2.0, box=10.0, seed=3)
    with tpcf.Engine(0) as eng:
        h = eng.catalog(d)
        want = eng.count(_spec(tpcf.OVERFLOW_CLEAN, (8, 0.0, 30.0), tpcf.PLAIN_FP64), eng.job([h] * 3))
        for call in range(3):
            assert np.array_equal(eng.count(_spec(tpcf.OVERFLOW_CLEAN, (8, 0.0, 30.0)), eng.job([h] * 3)), want)
            assert eng.stats()["graph_replays"] == (1 if call else 0)


@pytest.fixture
def near(monkeypatch):
    monkeypatch.setenv("TPCF_NEAR", "1")


@pytest.mark.parametrize("n,m", [(1, 2), (3, 64), (31, 33), (65, 70), (150, 129), (333, 200)])
def test_lists_at_small_sizes(near, n, m):
    test_near_lists.test_classes(n, m)


@pytest.mark.parametrize("axis", [(16, 0.0, 40.0), (20, 1.0, 15.0)])
def test_lists_that_overflow(near, axis):
    test_near_lists.test_lists_that_overflow(axis)


def test_summed_outputs(near):
    test_near_lists.test_summed_outputs()
