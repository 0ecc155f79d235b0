"""Into how many parts the planner cuts the units of small batches: not at all
where a part would repeat most of its unit's work (three-side counts in plain FP64
or clean mode), into quarters elsewhere.  Counts equal the oracle's either way."""
import os
import re
import subprocess
import sys

import pytest

import tpcf

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = {paths!r}
import numpy as np, oracle, synth, tpcf
d = synth.uniform(400, box=60.0, seed=1)
r = synth.uniform(300, box=60.0, seed=2)
want = oracle.three_side([d, r, r], 0.0, 30.0, 8, clean={clean})[0]
with tpcf.Engine(0) as eng:
    hd, hr = eng.catalog(d), eng.catalog(r)
    s = tpcf.make_spec(tpcf.THREE_SIDE, tpcf.LOOP_ALL, [(8, 0.0, 30.0)], overflow={clean}, precision={precision})
    assert np.array_equal(eng.count(s, eng.job([hd, hr, hr])), want)
"""


@pytest.mark.parametrize("clean,precision,parts", [(0, tpcf.GUARDED_FP32, 4), (1, tpcf.GUARDED_FP32, 1),
                                                   (0, tpcf.PLAIN_FP64, 1), (1, tpcf.PLAIN_FP64, 1)])
def test_parts_of_a_small_three_side_batch(clean, precision, parts):
    env = dict(os.environ, TPCF_PLAN_TRACE="1", TPCF_NEAR="0")  # (the trace is read once in a process)
    r = subprocess.run([sys.executable, "-c", CODE.format(paths=sys.path, clean=clean, precision=precision)], env=env,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert re.findall(r"tpcf plan: .* parts (\d+)", r.stderr) == [str(parts)]
