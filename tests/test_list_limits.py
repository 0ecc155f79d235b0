"""Triangle lists where their buffers end: the recheck queue overflows and grows
(in every mode that has one), and a CTA's 32-bit histogram is emptied before it
can run over.  The first against the oracle and the count that needed no growth,
the second against the tiles."""
import platform

import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

NAN = tpcf.NAN_ZERO if platform.machine() == "aarch64" else tpcf.NAN_INT_MIN
TP = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
JBJ = [(8, 2.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)]


@pytest.mark.parametrize("kind,axes,precision", [(tpcf.TRIANGLE, TP, tpcf.GUARDED_FP32), (tpcf.TRIANGLE, TP, tpcf.GEOMETRY_FP64),
                                                 (tpcf.TRIANGLE_JBJ, JBJ, tpcf.GUARDED_FP32)])
def test_recheck_queue_overflow(monkeypatch, kind, axes, precision):
    monkeypatch.setenv("TPCF_TRI_LISTS", "1")
    monkeypatch.setenv("TPCF_GRAPHS", "0")
    d = synth.lattice_mix(400, box=20.0, frac=0.6, seed=5)
    spec = tpcf.make_spec(kind, tpcf.LOOP_SAME, axes, precision=precision, nan_policy=NAN)
    res = []
    for cap in (None, "16"):
        if cap:
            monkeypatch.setenv("TPCF_RECHECK_CAP", cap)
        with tpcf.Engine(0) as eng:  # (a fresh engine: its queue has not grown)
            res.append(eng.count(spec, eng.job([eng.catalog(d)] * 3)))
            st = eng.stats()
        assert st["recheck_units"] > 16
        assert st["recheck_regrows"] >= 1 if cap else st["recheck_regrows"] == 0
    assert np.array_equal(*res) and res[0].sum() > 0
    if kind == tpcf.TRIANGLE_JBJ:
        assert np.array_equal(res[0], oracle.triangle_jbj([d] * 3, 0, axes)[0])
    elif precision == tpcf.GUARDED_FP32:
        assert np.array_equal(res[0], oracle.triangle([d] * 3, 0, axes, nan_zero=NAN == tpcf.NAN_ZERO)[0])


def test_histograms_emptied_before_they_run_over(monkeypatch):
    """More than 2^28 triangles for each of the launch's CTAs (three per SM)."""
    d = synth.blobs(11000, n_blobs=1, sigma=5.0, box=10.0, seed=1)
    spec = tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, TP, nan_policy=NAN)
    res = []
    with tpcf.Engine(0) as eng:
        j = eng.job([eng.catalog(d)] * 3)
        for lists in ("0", "1"):
            monkeypatch.setenv("TPCF_TRI_LISTS", lists)
            res.append(eng.count(spec, j))
        assert eng.stats()["binned_units"] > 3 * 152 * 2**28
    assert np.array_equal(*res)
