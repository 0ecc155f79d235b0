"""The double-precision geometry through the fast kernel (float sides, wide
guard bands, the rest recomputed in double) against the exhaustive kernel that
evaluates every triangle in double.  A catalog with one coordinate beyond 1e15
takes the exhaustive kernel; the point lies out of every other point's reach,
so the counts have to be the same.  Integer histograms: tolerance 0."""
import platform

import numpy as np
import pytest

import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
AXES = {
    "benchmark": [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)],
    "default": [(50, 2.0, 12.0), (16, 0.9, 4.1), (25, 0.0, 1.0)],
    "part of theta": [(5, 1.0, 11.0), (7, 1.5, 2.9), (9, 0.2, 0.6)],
    "from zero": [(10, 0.0, 10.0), (8, 1.0, 5.0), (10, 0.0, 1.0)],
    "one wide bin": [(1, 3.0, 9.0), (1, 1.0, 8.0), (1, 0.0, 1.0)],
}


def _line(n, seed):
    """Nearly collinear points, some repeated: cosines at and around +-1."""
    rng = np.random.default_rng(seed)
    t = rng.uniform(0, 40, n)
    p = np.stack([t, 0.5 * t, 2.0 * t], 1) * 0.3 + rng.normal(0, 1, (n, 3)) * rng.choice([0, 1e-6, 1e-3, 0.05], (n, 1))
    p[::9] = p[0]
    return p.astype(np.float32)


CATALOGS = {
    "blobs": (synth.blobs(420, n_blobs=2, sigma=4.0, box=30.0, seed=1), synth.uniform(300, box=40.0, seed=2)),
    "lattice": (synth.lattice_mix(400, box=20.0, frac=1.0, seed=3), synth.lattice_mix(330, box=25.0, frac=0.5, seed=4)),
    "line": (_line(300, 5), _line(260, 6)),
    "far from the origin": (synth.blobs(350, n_blobs=2, sigma=4.0, box=20.0, seed=7) + np.float32(3000.0),
                            synth.uniform(300, box=30.0, seed=8) + np.float32(3000.0)),
}


@pytest.mark.parametrize("axes", sorted(AXES))
@pytest.mark.parametrize("cats", sorted(CATALOGS))
def test_equals_the_exhaustive_kernel(cats, axes):
    d, r = CATALOGS[cats]
    far = np.array([[2e15, -2e15, 3e15]], dtype=np.float32)
    loops = [tpcf.LOOP_SAME, tpcf.LOOP_ONE, tpcf.LOOP_ONE, tpcf.LOOP_SAME, tpcf.LOOP_ALL]
    specs = [tpcf.make_spec(tpcf.TRIANGLE, lp, AXES[axes], precision=tpcf.GEOMETRY_FP64, nan_policy=NAN) for lp in loops]
    got = []
    with tpcf.Engine(0) as eng:
        for extra in (None, far):
            # (last, so that the loop indices of the others stay)
            hd, hr = [eng.catalog(c if extra is None else np.concatenate([c, extra])) for c in (d, r)]
            jobs = [eng.job(h) for h in ([hd, hd, hd], [hd, hd, hr], [hd, hr, hr], [hr, hr, hr], [hd, hr, hd])]
            got.append(eng.count_batch(specs, jobs))
            fast = eng.stats()
            assert (fast["evaluated_units"] == fast["binned_units"]) == (extra is not None)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert sum(int(a.sum()) for a in got[0]) > 0
