"""evaluated_units of the triangle lists where one warp has more than 2^32 pairs to
test: two clumps of 70,000 points seen from outside (enough centres that none is
cut into shares)."""
import numpy as np
import pytest

import synth
import tpcf

pytestmark = pytest.mark.gpu


def test_a_centre_with_more_than_32_bits_of_pairs(monkeypatch):
    monkeypatch.setenv("TPCF_TRI_LISTS", "1")
    n = 70000
    clump = [synth.uniform(n, box=0.25, seed=k) for k in (1, 2)]
    outside = np.array([[5.0, 0.0, 0.0]], np.float32)
    with tpcf.Engine(0) as eng:
        h = [eng.catalog(c) for c in [outside] + clump]
        spec = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ALL, [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)])
        eng.count(spec, eng.job(h))
        # the point outside has every pair of the clumps, each of theirs the other clump's with it
        assert eng.stats()["evaluated_units"] == 3 * n * n
