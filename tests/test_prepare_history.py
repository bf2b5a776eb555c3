"""wf_prepare_run grows the histories that the run fills, also where the run
replays no graph: the cluster run, the tile run, phase timing. Seen as device
memory: 40 million steps take a history of 512 MB. In a process of its own, whose
pool holds no memory of earlier domains."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
import sys
import torch
import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W
d = wf.Domain(wf.WF_MIXED)
W.apply(d, W.config(0, scale=({n}, {n}, {n})))
if {timing}:
    d.set_phase_timing(True)
d.init()
d.sync()
before = torch.cuda.mem_get_info()[0]
d.prepare_run(40_000_000)
d.sync()
print(before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.gpu
@pytest.mark.parametrize("n,timing", [(10, False), (20, False), (20, True)])
def test_prepare_run_grows_the_history(n, timing):
    r = subprocess.run([sys.executable, "-c", SRC.format(n=n, timing=timing)], cwd=ROOT,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) >= 8 * 40_000_000
