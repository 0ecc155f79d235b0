"""The 32-bit counters of the three-side neighbour lists at the most that they
can take between two flushes: three catalogs with every triple in one bin, the
lists as long as they get (256 near tiles of 64 points), and enough centres for
every pipeline to draw the largest item at once."""
import numpy as np
import pytest

import synth
import tpcf

pytestmark = pytest.mark.gpu


def test_two_lists_in_one_bin(monkeypatch):
    monkeypatch.setenv("TPCF_NEAR", "1")
    # 2,432 centres: an item of four for each of 152 x 4 pipelines
    cats = [synth.uniform(n, box=5.0, seed=k) for k, n in enumerate((2432, 16384, 16384))]
    # many centres in the batch, none near another, so that an item is as large as it gets
    far = np.stack(np.meshgrid(*[np.arange(35) * 1000.0] * 3), -1).reshape(-1, 3).astype(np.float32)
    with tpcf.Engine(0) as eng:
        h, hf = [eng.catalog(c) for c in cats], eng.catalog(far)
        spec = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [(1, 0.0, 100.0)])
        got = eng.count_batch([spec] * 2, [eng.job(h), eng.job([hf] * 3)])
        assert got[0].tolist() == [2432 * 16384 * 16384]
        assert got[1].tolist() == [len(far)]  # i == j == k
