"""readtwoint called once per chunk of a file: the chunks' results, and the device memory that a
small chunk of a large basis takes."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

from gammcor_gb300 import api
from oracle import sorter_ref as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROOT = Path(__file__).resolve().parent.parent


# Chunks on both sides of the rule that chooses the one-pass road (n = 300: a bitmap of 127 MB,
# against 64 MB or 64 bytes per integral), a pair repeated within one chunk and across chunks
@pytest.mark.parametrize("fmt,n,sizes", [("pqrs", 9, (1, 40, 300)), ("dalton8", 9, (1, 40, 300)),
                                         ("dalton16", 9, (1, 40, 300)),
                                         ("pqrs", 300, (1000, 2200000, 3)),
                                         ("dalton16", 300, (1000, 2200000, 3))])
def test_chunks_of_one_file(gpu_lib, fmt, n, sizes):
    rng = np.random.default_rng(n)
    ntr = n * (n + 1) // 2
    ref, got = torch.zeros(ntr, ntr, dtype=torch.float64, device=DEV), None
    for cnt in sizes:
        p, q, r, s = rng.integers(1, n + 1, (4, cnt))
        if fmt != "pqrs":
            p, q, r, s = np.minimum(p, q), np.maximum(p, q), np.minimum(r, s), np.maximum(r, s)
        for x in (p, q, r, s):
            x[0], x[-1] = 1, 1       # (11|11) opens and closes every chunk
        lab = {"pqrs": lambda: np.stack([p, q, r, s], 1).ravel(),
               "dalton8": lambda: p | q << 8 | r << 16 | s << 24,
               "dalton16": lambda: np.stack([r | s << 16, p | q << 16], 1).ravel()}[fmt]()
        lab = lab.astype(np.uint32).view(np.int32)
        vals = rng.standard_normal(cnt)
        if n < 50:
            ref = torch.as_tensor(S.readtwoint(n, vals, lab, fmt, out=ref.cpu().numpy()), device=DEV)
        else:  # the oracle's rule, vectorised: the last integral of a slot stays
            a, b, c, d = np.minimum(p, q), np.maximum(p, q), np.minimum(r, s), np.maximum(r, s)
            pq, rs = a + b * (b - 1) // 2 - 1, c + d * (d - 1) // 2 - 1
            both = np.ones(cnt, bool) if fmt == "pqrs" else pq < rs
            slot = np.stack([rs * ntr + pq, np.where(both, pq * ntr + rs, rs * ntr + pq)], 1).ravel()
            last = len(slot) - 1 - np.unique(slot[::-1], return_index=True)[1]
            ref.view(-1)[torch.as_tensor(slot[last], device=DEV)] = torch.as_tensor(
                np.repeat(vals, 2)[last], device=DEV)
        got = api.readtwoint(n, torch.as_tensor(vals, device=DEV), torch.as_tensor(lab, device=DEV),
                             fmt, out=got)
    assert torch.equal(got, ref)


PROGRAM = """
import sys
import torch
from gammcor_gb300 import api
n, cnt, dev = 300, int(sys.argv[1]), "cuda:0"
ntr = n * (n + 1) // 2

def pair(x):  # 0-based pair index -> 1-based p <= q
    d = ((torch.sqrt(8.0 * x.double() + 1) - 1) * 0.5).long()
    d -= (d * (d + 1) // 2 > x).long()
    d += ((d + 1) * (d + 2) // 2 <= x).long()
    return x - d * (d + 1) // 2 + 1, d + 1

def chunk(t0, c, fmt_n):
    hi, lo = pair(torch.arange(t0, t0 + c, device=dev))     # lo <= hi: one unordered pair each
    lo, hi = hi - 1, lo - 1
    lo, hi = torch.minimum(lo, hi), torch.maximum(lo, hi)
    (p, q), (r, s) = pair(lo), pair(hi)
    return lo, hi, torch.stack([r | s << 16, p | q << 16], 1).reshape(-1).to(torch.int32)

small = torch.zeros(36, 36, dtype=torch.float64, device=dev)  # loads every kernel
one = torch.ones(2, dtype=torch.float64, device=dev)
api.readtwoint(8, one, torch.tensor([1 | 1 << 16] * 4, dtype=torch.int32, device=dev), "dalton16", out=small)
lo, hi, lab = chunk(10 ** 8, cnt, n)
val = torch.randn(cnt, dtype=torch.float64, device=dev)
out = torch.zeros(ntr, ntr, dtype=torch.float64, device=dev)
torch.cuda.synchronize()
torch.cuda.empty_cache()
before = torch.cuda.mem_get_info()[0]
if len(sys.argv) > 2:                                        # leave that many MB
    fill = torch.empty(before - (int(sys.argv[2]) << 20), dtype=torch.uint8, device=dev)
api.readtwoint(n, val, lab, "dalton16", out=out)
torch.cuda.synchronize()
if len(sys.argv) > 2:
    del fill
    torch.cuda.empty_cache()
    assert torch.equal(out[hi, lo], val) and torch.equal(out[lo, hi], val)
    assert int((out != 0).sum()) == 2 * cnt - int((lo == hi).sum())
else:
    print("grown", before - torch.cuda.mem_get_info()[0])
"""


def run(*args):
    r = subprocess.run([sys.executable, "-c", PROGRAM, *args], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


def test_small_chunk_takes_no_bitmap_of_a_large_basis(gpu_lib):
    """n = 300: a bitmap of 127 MB for a chunk of 1000 integrals of 16 KB in all."""
    assert int(run("1000").split()[-1]) < 64 << 20


def test_sort_without_room_for_the_bitmap(gpu_lib):
    """The exact passes need one byte per integral, where the bitmap of 127 MB does not fit."""
    run("4500000", "70")
