"""sw_score_noalloc loads every kernel in the first call on a device: the
profiler sees no lazy loading in a later call, whatever its query's length."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.join(os.path.dirname(__file__), "..")

CHILD = r'''
import numpy as np, torch
from swhybrid_b200 import capi, synth
rec = torch.from_numpy(synth.query(1, 3000)).to("cuda:0")
off = torch.tensor([0, 3000], dtype=torch.int64, device="cuda:0")
out = torch.zeros(1, dtype=torch.int32, device="cuda:0")
queries = [torch.from_numpy(synth.query(2, n)).to("cuda:0")
           for n in (100, 200, 300, 500, 700, 1000, 1500, 2000, 5000, 9000, 100)]
p = capi.default_params()
def call(q, n):
    st = capi.score_noalloc(0, p, q.data_ptr(), q.numel(), rec.data_ptr(), off.data_ptr(), n,
                            out.data_ptr())
    assert st == capi.SW_OK, st
call(queries[0], 0)
from torch.profiler import ProfilerActivity, profile
with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
    for q in queries:
        call(q, 1)
names = [e.name for e in prof.events()]
print("names", sorted(set(names)))
if not any("sw_score_noalloc" in n for n in names):
    raise SystemExit(77)                 # the profiler sees no kernels here
loads = [n for n in names if "load" in n.lower()]
assert loads == [], loads
'''


def test_later_calls_load_nothing():
    env = dict(os.environ, PYTHONPATH=ROOT, CUDA_MODULE_LOADING="LAZY")
    out = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, env=env,
                         cwd=ROOT, timeout=300)
    if out.returncode == 77:
        pytest.skip("the profiler is not available")
    assert out.returncode == 0, out.stdout + out.stderr
