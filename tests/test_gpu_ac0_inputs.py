"""AC0-CAS: the device memory of a call, integrals whose (rs|pq) and (pq|rs) differ, and calls from
several threads."""
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest
import torch

from gammcor_gb300 import api, synth
from oracle import ac0_ref as A
from oracle import ac_cas_ref as R

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


def system(n, nin, nact):
    """Orthogonal orbitals, a dominant one-electron diagonal and a mean-field 2-RDM: stable blocks."""
    rng = np.random.default_rng(n)
    lf = synth.make_lfac(n, 3 * n, rng) * 0.1
    occ = np.r_[np.ones(nin), np.linspace(0.96, 0.05, nact), np.zeros(n - nin - nact)]
    ffoo, fofo = R.transform_fofo_ffoo(np.linalg.qr(rng.standard_normal((n, n)))[0], lf @ lf.T, nin, nact)
    xone = 0.05 * rng.standard_normal(synth.ntri(n))
    xone[np.cumsum(np.arange(1, n + 1)) - 1] = np.linspace(-30.0, 10.0, n)
    o, e = occ[nin:nin + nact], np.eye(nact)
    rdm = synth.pack_rdm2act(2 * np.einsum("p,q,pr,qs->pqrs", o, o, e, e)
                             - np.einsum("p,q,ps,qr->pqrs", o, o, e, e))
    return occ, xone, R.pair_space(occ, nin + nact // 2), nin, nact, ffoo, fofo, rdm


def energy(s, fofo, ctx=None):
    occ, xone, indn, nin, nact, ffoo, _, rdm = s
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda:0")
    return api.ac0cas_fofo(occ, xone, indn, nact, nin, dev(ffoo), dev(fofo), rdm, ctx=ctx)[0]


# The energy sums over all pairs of pairs with a symmetric factor. A part of FOFO with
# (rs|pq) = -(pq|rs), for virtual p, r and inactive q, s, all different, leaves A+- alone once
# symmetrised and must leave the energy alone too.
@pytest.mark.parametrize("n,nin,nact", [(21, 3, 4), (45, 4, 2)])
def test_ac0_takes_both_of_rs_pq_and_pq_rs(gpu_lib, n, nin, nact):
    s = system(n, nin, nact)
    occ, xone, indn, nin, nact, ffoo, fofo, rdm = s
    nocc = nin + nact
    q, p = np.divmod(np.arange(n * nocc), n)
    ok = ((p[:, None] >= nocc) & (p >= nocc) & (q[:, None] < nin) & (q < nin)
          & (p[:, None] != p) & (q[:, None] != q))
    d = np.random.default_rng(1).standard_normal(fofo.shape)
    odd = fofo + np.where(ok, 0.3 * (d - d.T), 0.0)
    ref = A.ac0cas_fofo(occ, xone, np.eye(n), indn, nin, nact, ffoo, odd, rdm)[0]
    assert abs(ref - A.ac0cas_fofo(occ, xone, np.eye(n), indn, nin, nact, ffoo, fofo, rdm)[0]) < 1e-12
    assert abs(energy(s, fofo) - ref) < 1e-9
    assert abs(energy(s, odd) - ref) < 1e-9


def test_ac0_from_threads_with_blocks_of_different_size(gpu_lib):
    """Blocks of 45 pairs and of one pair at the same time: no call may take its shared-memory limit
    from the other's."""
    def repeat(s):
        ctx = api.Context(0, torch.cuda.Stream())
        try:
            return {round(energy(s, s[6], ctx), 9) for _ in range(600)}
        finally:
            ctx.close()
    with ThreadPoolExecutor(2) as ex:
        for got in ex.map(repeat, [system(14, 0, 10), system(9, 2, 2)]):
            assert len(got) == 1
