"""AC0-CAS: the device memory of a call, integrals whose (rs|pq) and (pq|rs) differ, and calls from
several threads."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

MEMORY = """
import numpy as np
import torch
from gammcor_gb300 import api, synth

def call(n, nin, nact):
    occ = np.r_[np.ones(nin), np.linspace(0.96, 0.05, nact), np.zeros(n - nin - nact)]
    xone = np.zeros(synth.ntri(n))
    xone[np.cumsum(np.arange(1, n + 1)) - 1] = np.linspace(-30.0, 10.0, n)
    o, e = occ[nin:nin + nact], np.eye(nact)
    rdm = synth.pack_rdm2act(2 * np.einsum("p,q,pr,qs->pqrs", o, o, e, e)
                             - np.einsum("p,q,ps,qr->pqrs", o, o, e, e))
    indn, nocc = api.pair_space(occ, nin + nact // 2), nin + nact
    fo = 1e-2 * torch.randn(n * nocc, 40, dtype=torch.float64, device="cuda")
    fofo, ffoo = fo @ fo.T, torch.zeros(nocc * nocc, n * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    api.ac0cas_fofo(occ, xone, indn, nact, nin, ffoo, fofo, rdm)
    torch.cuda.synchronize()
    return (before - torch.cuda.mem_get_info()[0]) / (8 * len(indn) ** 2)

call(20, 2, 4)   # loads the kernels
print(call(200, 20, 6))
"""


def test_ac0_holds_four_matrices(gpu_lib):
    """A+-B(0) and A+-' are all that is held in N x N (174 MB each here): the workspace pool grows by
    less than 4.6 of them (the rest: intermediates of the assembly and rounding of the pool)."""
    r = subprocess.run([sys.executable, "-c", MEMORY], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert 3.5 < float(r.stdout.split()[-1]) < 4.6, r.stdout
