"""The allocation-free sum's first call of a process takes no device memory, whatever was loaded on
the device before it: the driver places modules in blocks of 2 MiB, so how full the last one is
decides whether one more module would need another."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIRST_CALL = r"""
import sys
import numpy as np
import torch
import bohrium_b200 as bh
from tests.test_zz_no_alloc import _noalloc

rt = bh.Runtime(bh.NativeExecutor())
for k in range(int(sys.argv[1])):  # one more loaded kernel each
    a = bh.array(rt, np.ones(1000))
    for _ in range(k + 1):
        a = bh.sqrt(a + 1.0)
    a.numpy()
core, f = _noalloc()
x = torch.ones(1_000_003, dtype=torch.float64, device="cuda")
out = torch.zeros(1, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
assert f(x.data_ptr(), x.numel(), out.data_ptr(), None) == 0, core.bhb_last_error()
torch.cuda.synchronize()
assert torch.cuda.mem_get_info()[0] == before, (before, torch.cuda.mem_get_info()[0])
assert float(out.item()) == 1_000_003.0
"""


@pytest.mark.gpu
@pytest.mark.parametrize("kernels", [0, 1, 2, 4, 8, 16, 32])
def test_first_call_of_a_process(kernels):
    r = subprocess.run([sys.executable, "-c", FIRST_CALL, str(kernels)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
