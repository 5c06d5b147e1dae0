"""Optional forms are configured by the first call that takes one: also when that call is the
first of its process and is captured.  The replay gives the bits of a later direct call."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = '''
import sys
sys.path[:0] = [%r, %r]
import torch
from namsa_gb300 import engine
from test_gpu_stream import DEV, case
ny, nx, S, P = map(int, sys.argv[1:])
x = case(ny, nx, S, P, 3)
plan = engine.Plan(ny, nx)
out = torch.zeros((P, ny, nx), device=DEV)
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    plan.multislice(*x, out=out)
g.replay()
torch.cuda.synchronize()
plan.check()
want = plan.multislice(*x)
torch.cuda.synchronize()
assert bool(torch.isfinite(out).all()) and float(out.abs().sum()) > 0 and torch.equal(out, want)
print('equal')
''' % (ROOT, os.path.join(ROOT, 'tests'))


# all slices in one kernel, clusters, schedules of few lines, the two passes
@pytest.mark.parametrize('shape', ['512 512 3 3', '128 128 3 2', '64 384 3 5', '1024 64 2 3'])
def test_first_call_under_capture(shape):
    r = subprocess.run([sys.executable, '-c', SRC, *shape.split()], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and 'equal' in r.stdout, r.stderr
