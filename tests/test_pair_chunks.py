"""Pair counts at catalog sizes on both sides of each number of tiles B per item
(1 below 1,520 tile pairs, 8 above, 16 and 32 from some 97,000 and 195,000 on),
against the plain FP64 kernel, whose items have one, through both pair entry
points.  Integer histograms: tolerance 0."""
import numpy as np
import pytest

import synth
import tpcf
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(2400, 2500), (2560, 2600), (20100, 19500), (28400, 28000)])
def test_items_of_every_size(n, m):
    d, r = synth.lattice_mix(n, box=90.0, frac=0.5, seed=n), synth.uniform(m, box=100.0, seed=m)
    axis = (40, 0.0, 12.0)
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        for a, b, ha, hb, loop in ((d, d, hd, hd, tpcf.LOOP_SAME), (d, r, hd, hr, tpcf.LOOP_ONE), (r, d, hr, hd, tpcf.LOOP_SAME)):
            want, got = [eng.count(tpcf.make_spec(tpcf.PAIR, loop, [axis], precision=p), eng.job([ha, hb]))
                         for p in (tpcf.PLAIN_FP64, tpcf.GUARDED_FP32)]
            assert want.sum() > 0
            assert np.array_equal(got, want)
            assert np.array_equal(_noalloc(a, b, loop, axis, a is b), want)
