"""The largest triangle histograms that the tile kernels take (46,464 bins beside
their tables in 227 KB of shared memory), in every mode that has tables of its
own, and one bin row more, which is refused.  Integer histograms equal the
oracle's."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
MOST = [(44, 2.0, 10.0), (33, 0.9, 4.2), (32, 0.0, 1.0)]  # 46,464 bins
MORE = [(44, 2.0, 10.0), (33, 0.9, 4.2), (33, 0.0, 1.0)]
JBJ = [(44, 2.0, 10.0), (33, 0.2, 1.0), (32, 0.0, 1.0)]


@pytest.mark.parametrize("lists", ["0", None])
def test_the_largest(monkeypatch, lists):
    if lists:
        monkeypatch.setenv("TPCF_TRI_LISTS", lists)
    d = synth.blobs(150, n_blobs=2, sigma=4.0, box=25.0, seed=1)
    with tpcf.Engine(0) as eng:
        j = eng.job([eng.catalog(d)] * 3)
        want = oracle.triangle([d] * 3, 0, MOST, nan_zero=NAN == tpcf.NAN_ZERO)[0]
        assert want.sum() > 0
        for precision in (tpcf.GUARDED_FP32, tpcf.PLAIN_FP64):
            s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, MOST, precision=precision, nan_policy=NAN)
            assert np.array_equal(eng.count(s, j), want)
        # FP64 geometry, also by the exhaustive kernel (coordinates past 1e15)
        far = np.concatenate([d, np.array([[2e15, 2e15, 2e15]], np.float32)])
        s = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, MOST, precision=tpcf.GEOMETRY_FP64, nan_policy=NAN)
        assert np.array_equal(eng.count(s, j), eng.count(s, eng.job([eng.catalog(far)] * 3)))
        s = tpcf.make_spec(tpcf.TRIANGLE_JBJ, tpcf.LOOP_SAME, JBJ)
        assert np.array_equal(eng.count(s, j), oracle.triangle_jbj([d] * 3, 0, JBJ)[0])
        with pytest.raises(tpcf.EngineError) as e:
            eng.count(tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, MORE, nan_policy=NAN), j)
        assert e.value.status == -1  # TPCF_ERR_INVALID
