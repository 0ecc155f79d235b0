"""Triangle tile kernel: which points of a unit are listed.  Groups of eight
points, one tile each, in triples whose three distances lie below, on and above
the limits that the listing tests (the s range, that range times the largest
ratio, the largest side), in exact steps and a few units in the last place
apart.  Integer histograms equal the oracle's."""
import itertools
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN


def _groups(limits, spread, seed):
    """Triples of groups 4096 apart: A at 0, B at b along x, C at c along x or y."""
    rng = np.random.default_rng(seed)
    out = []
    near = [f * x for x in limits for f in (1 - 2e-6, 1.0, 1 + 2e-6)]
    for k, (b, c, along) in enumerate(itertools.product(near, near, "xy")):
        o = np.array([0.0, 4096.0 * (k % 16), 4096.0 * (k // 16)])
        for at in (np.zeros(3), np.array([b, 0, 0]), np.array([c, 0, 0] if along == "x" else [0, c, 0])):
            step = rng.integers(-1, 2, (8, 3)) * spread
            out.append(o + at + step * (1, 1, 0))
    return np.concatenate(out).astype(np.float32)


@pytest.mark.parametrize("spread", [0.0, 1e-5, 0.25])
@pytest.mark.parametrize("name", ["tp", "flat", "jbj"])
def test_limits(monkeypatch, name, spread):
    kind, axes, limits = {
        "tp": (tpcf.TRIANGLE, [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)], (2.0, 10.0, 30.0, 40.0)),
        "flat": (tpcf.TRIANGLE, [(4, 2.0, 10.0), (4, 0.5, 1.0), (8, 0.0, 1.0)], (2.0, 10.0, 20.0)),
        "jbj": (tpcf.TRIANGLE_JBJ, [(8, 2.0, 10.0), (8, 0.25, 1.0), (10, 0.0, 1.0)], (2.0, 10.0, 40.0, 50.0)),
    }[name]
    monkeypatch.setenv("TPCF_TRI_LISTS", "0")
    monkeypatch.setenv("TPCF_TILE_POINTS", "8")
    d = _groups(limits, spread, seed=1)[:1200]
    r = d[::-1][:600] + np.float32(0.5)
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        for c, h, w in (([d, d, d], [hd, hd, hd], 0), ([d, r, r], [hd, hr, hr], 1)):
            s = tpcf.make_spec(kind, tpcf.LOOP_ONE if w else tpcf.LOOP_SAME, axes, nan_policy=NAN)
            got = eng.count(s, eng.job(h))
            want = (oracle.triangle(c, w, axes, nan_zero=NAN == tpcf.NAN_ZERO) if kind == tpcf.TRIANGLE
                    else oracle.triangle_jbj(c, w, axes))[0]
            assert np.array_equal(got, want)


def test_points_that_are_not_numbers():
    """A point outside every box, whose sides are all in the s range's first
    bin where int(NaN) is 0: no point may be left out for its distance from it."""
    d, r = synth.blobs(50, n_blobs=2, sigma=6.0, box=40.0, seed=50), synth.uniform(70, box=60.0, seed=70)
    d[17, 1] = r[23, 2] = np.nan
    axes = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE, axes, nan_policy=tpcf.NAN_ZERO, prune=False)
        want = oracle.triangle([r, d, r], 1, axes, nan_zero=True)[0]
        assert np.array_equal(eng.count(s, eng.job([hr, hd, hr])), want)
