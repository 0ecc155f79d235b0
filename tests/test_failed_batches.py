"""A batch that fails for lack of memory leaves the batches planned before it
right: their plans are not used with buffers that have moved meanwhile."""
import numpy as np
import pytest

import oracle
import synth
import tpcf

pytestmark = pytest.mark.gpu

AXIS = (16, 0.0, 20.0)


def test_accumulators_that_moved(monkeypatch):
    d, r = synth.lattice_mix(300, box=30.0, frac=0.5, seed=1), synth.uniform(280, box=40.0, seed=2)
    want = [oracle.three_side(c, AXIS[1], AXIS[2], AXIS[0])[0] for c in ([d] * 3, [d, r, r])]
    spec = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [AXIS])
    with tpcf.Engine(0) as eng:
        hd, hr = eng.catalog(d), eng.catalog(r)
        jobs = [eng.job([hd] * 3), eng.job([hd, hr, hr])]
        many = [jobs[k % 2] for k in range(100)]
        # the histograms of the large batch exist before the small one is planned
        monkeypatch.setenv("TPCF_NEAR", "0")
        eng.count_batch([spec] * len(many), many)
        monkeypatch.setenv("TPCF_NEAR", "1")

        def small():
            assert all(np.array_equal(g, w) for g, w in zip(eng.count_batch([spec] * 2, jobs), want))

        small()
        small()
        try:
            # accumulators of 44 KB a job: more than a block may have
            tpcf.lib().tpcf_debug_alloc_limit(1 << 20)
            with pytest.raises(tpcf.EngineError) as e:
                eng.count_batch([spec] * len(many), many)
            assert e.value.status == -4  # TPCF_ERR_OOM
        finally:
            tpcf.lib().tpcf_debug_alloc_limit(2**64 - 1)
        # the released accumulators (a block of 128 KB) become a catalog's points
        extra = [eng.catalog(synth.uniform(8000, box=500.0, seed=k)) for k in range(4)]
        eng.resident_bytes()
        small()
        small()
        pair = tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_SAME, [(10, 0.0, 50.0)])
        for k, h in enumerate(extra):
            p = synth.uniform(8000, box=500.0, seed=k)
            assert np.array_equal(eng.count(pair, eng.job([h, h])), oracle.pair([p, p], 0, 0.0, 50.0, 10)[0])
        assert all(np.array_equal(g, want[k % 2]) for k, g in enumerate(eng.count_batch([spec] * len(many), many)))
