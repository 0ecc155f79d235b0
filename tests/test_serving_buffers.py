"""A serving lane takes no memory from the driver for a batch (that would wait for
the other lanes' kernels): its buffers, sized when the engine is made, hold what
every kind of batch needs."""
import numpy as np
import pytest

import synth
import tpcf

pytestmark = pytest.mark.gpu

TP = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
FINE = [(50, 2.0, 12.0), (16, 0.9, 4.1), (25, 0.0, 1.0)]
JBJ = [(8, 2.0, 10.0), (8, 0.2, 1.0), (10, 0.0, 1.0)]


def test_batches_allocate_nothing(monkeypatch):
    monkeypatch.setenv("TPCF_NEAR", "1")
    with tpcf.Engine(0) as eng:
        h = [eng.catalog(synth.blobs(n, n_blobs=2, sigma=5.0, box=60.0, seed=n)) for n in (300, 700, 3000)]
        kinds = [(tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [(32, 0.0, 32.0)]), 3),
                 (tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [(60, 0.0, 32.0)]), 3),
                 (tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE, TP), 3),
                 (tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE, FINE), 3),
                 (tpcf.make_spec(tpcf.TRIANGLE_JBJ, tpcf.LOOP_SAME, JBJ), 3),
                 (tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_SAME, [(700, 0.0, 70.0)]), 2)]
        jobs = [(s, eng.job([h[(k + r) % 3] for r in range(nc)])) for s, nc in kinds for k in range(3)]
        want = [eng.count(s, j) for s, j in jobs]  # (and every view is built)
        before = tpcf.lib().tpcf_debug_allocations()
        for burst in range(4):
            tickets = [(eng.submit(s, j), s, w) for (s, j), w in zip(jobs, want)]
            assert all(np.array_equal(eng.wait(t, s), w) for t, s, w in tickets)
        assert tpcf.lib().tpcf_debug_allocations() == before
