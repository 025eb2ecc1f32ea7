"""Laying out the adjoint takes host memory for the plan's lists, whatever the chunk size."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = """
import resource
import numpy as np
import torch
from cbm.plan import Plan

p = Plan(np.array([0, 1, 2], np.int32), np.array([1, 0], np.int32), np.ones(2, np.float32), 2, 2,
         np.array([0], np.int32), np.zeros(0, np.int32), np.zeros(0, np.int32), host=True)
g = torch.tensor([[1.0], [2.0]], device="cuda")
dx = torch.empty_like(g)
p.adjoint("ax", g, dx)
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
p.tune(chunk_nnz=2**31 - 1)  # never split
p.adjoint("ax", g, dx)
assert dx.flatten().tolist() == [2.0, 1.0]
print("grown", resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before)  # KiB
"""


def test_largest_chunk_size_allocates_by_the_lists():
    out = subprocess.run([sys.executable, "-c", _SCRIPT], capture_output=True, text=True, timeout=300,
                         env={**__import__("os").environ, "PYTHONPATH": ":".join(sys.path)})
    assert out.returncode == 0, out.stderr
    assert int(out.stdout.split()[-1]) < 1 << 20  # a vector of chunk_nnz / 4 counters is 4 GiB
