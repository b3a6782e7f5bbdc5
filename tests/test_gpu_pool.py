"""Workspaces come from a pool that keeps memory between calls. A cudaMalloc of the same process that
would not fit otherwise gets that memory from the driver, so keeping it costs other allocators of the
process nothing."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
from gammcor_gb300 import api
n, rank = 200, 1200
g = torch.Generator(device="cuda").manual_seed(1)
L = torch.randn(rank, n * (n + 1) // 2, dtype=torch.float64, device="cuda", generator=g).t()
C = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g))[0]
co = C[:, :24].contiguous()
before = torch.cuda.mem_get_info()[0]
out = api.tran4_factored(n, L, C, co, C, co, precision="fp64tc5")
torch.cuda.synchronize()
torch.cuda.empty_cache()
kept = before - torch.cuda.mem_get_info()[0] - out.numel() * 8
assert kept > 256 << 20, kept                    # the call's workspaces stay in the pool
x = torch.empty(torch.cuda.mem_get_info()[0] + kept // 2, dtype=torch.uint8, device="cuda")
del x
torch.cuda.empty_cache()
assert torch.equal(api.tran4_factored(n, L, C, co, C, co, precision="fp64tc5"), out)
"""


def test_kept_workspaces_give_way_to_other_allocations(gpu_lib):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=Path(__file__).resolve().parent.parent,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
