"""Degenerate triangles (points on a line, whose rounded cosines pass +-1 and give
the reference NaN) in angle binnings whose edges are and are not at 0 and pi: in
the reference a NaN angle has bin 0 or none, by the machine, wherever 0 and pi
lie.  From tiles and from lists; integer histograms equal the oracle's."""
import numpy as np
import pytest

import oracle
import tpcf

pytestmark = pytest.mark.gpu

ANGLES = [(16, 0.0, 1.0), (1, 0.1, 0.5), (1, 0.25, 0.75), (4, -0.1, 1.1), (3, 0.0, 0.7), (25, 0.1, 1.0), (2, -1.0, 3.0), (5, 0.03, 1.03)]


def _lines(n, seed):
    """Points at random steps along lines in random directions, near the origin and far from it."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(6):
        d = rng.normal(size=3)
        t = rng.uniform(0, 40, (n, 1))
        out.append(rng.uniform(-1, 1, 3) * (10.0 ** k / 100) + t * d / np.linalg.norm(d))
    return np.concatenate(out).astype(np.float32)


@pytest.mark.parametrize("lists", ["0", "1"])
@pytest.mark.parametrize("nan", [tpcf.NAN_ZERO, tpcf.NAN_INT_MIN])
def test_points_on_lines(monkeypatch, lists, nan):
    monkeypatch.setenv("TPCF_TRI_LISTS", lists)
    d, r = _lines(45, 1), _lines(25, 2)
    total = 0
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        for angle in ANGLES:
            axes = [(8, 1.0, 30.0), (4, 0.9, 4.1), angle]
            for c, h, w in (([d] * 3, [hd] * 3, 0), ([d, d, r], [hd, hd, hr], 1)):
                s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE if w else tpcf.LOOP_SAME, axes, nan_policy=nan)
                want = oracle.triangle(c, w, axes, nan_zero=nan == tpcf.NAN_ZERO)[0]
                assert np.array_equal(eng.count(s, eng.job(h)), want), (angle, w)
                total += int(want.sum())
    assert total > 0
