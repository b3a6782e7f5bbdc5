"""The work that a user of this library has it do, as cases that can be timed and checked.

Each case calls the public entry points of gammcor_gb300.api on inputs made from a seed. The
sizes are those of the package's own shapes (synth.CFG_SMALL, synth.batched_shapes): basis
sizes 50 to 250, 5 to 25 inactive orbitals, CAS(2,2) to CAS(6,6), ERI factor rank 6 n.
`exact` restates the same quantities in plain FP64 torch, independently of the library.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gammcor_gb300 import api, synth

DEV = "cuda"
F8 = torch.float64


def listed():
    return [
        # AO->MO transform of the small named shape: one call of a few milliseconds' worth of
        # launches, as a program makes it for every small molecule.
        dict(name="fofo_n64", kind="fofo", n=64, nin=6, nact=4, rank=300, prec="fp64tc5"),
        # The same at the top of the batch's range: the largest FOFO block that the batch forms.
        dict(name="fofo_n249", kind="fofo", n=249, nin=22, nact=6, rank=1494, prec="fp64tc5"),
        # FFOO at an odd middle size: its two sides have different orbital blocks.
        dict(name="ffoo_n153", kind="ffoo", n=153, nin=13, nact=4, rank=918, prec="fp64tc5"),
        # The reference-shaped route: AO integrals in sorted records, plain FP64, the precision
        # that the parity runs use.
        dict(name="gen_n64_fp64", kind="gen", n=64, nin=6, nact=4, rank=300, prec="fp64"),
        # A+B and A-B of a small system: a chain of small kernels, where launches count.
        dict(name="ab_n64", kind="ab", n=64, nin=6, nact=4, alpha=0.5),
        # ... and of the largest system of the batch (NDimX 6335).
        dict(name="ab_n249", kind="ab", n=249, nin=22, nact=6, alpha=0.02),
        # One lambda point of the production form: ERPA solve (FP32 start, refined) and W.
        dict(name="point_n110", kind="point", n=110, nin=10, nact=4, lam=0.5, prec="fp64tc5"),
        # The integrand alone, given the solutions, at a large order (NDimX 3774).
        dict(name="integrand_n190", kind="integrand", n=190, nin=18, nact=4, prec="fp64tc5"),
        # AC0-CAS: the non-iterative energy, from integrals to the energy.
        dict(name="ac0_n120", kind="ac0", n=120, nin=11, nact=6),
        # A whole batch of uneven systems, 8 points each, from ERI factors to energies, with the
        # widest tensor-core arithmetic: what a screening run does.
        dict(name="batch_6", kind="batch", count=6, nmax=96, prec="fp64tc6"),
        # One training step of the integrand network on a full batch.
        dict(name="mlp_b256", kind="mlp", batch=256, hidden=256),
        # Sorting the AO integral file's labels and values into records, once per molecule.
        dict(name="sort_n96", kind="sort", n=96, fmt="dalton16"),
    ]


def draw(rng):
    kind = rng.choice(["fofo", "fofo", "ffoo", "gen", "ab", "ab", "point", "integrand", "ac0",
                       "batch", "mlp", "sort"])
    nact = rng.choice([2, 4, 6])
    if kind in ("fofo", "ffoo"):
        n = rng.randint(50, 249) if kind == "fofo" else rng.randint(50, 200)
        return dict(kind=kind, n=n, nin=rng.randint(5, 22 if n > 80 else 14), nact=nact,
                    rank=6 * n, prec=rng.choice(["fp64tc5", "fp64tc5", "fp64tc6"]))
    if kind == "gen":
        n = rng.randint(40, 72)
        return dict(kind=kind, n=n, nin=rng.randint(4, 9), nact=nact, rank=6 * n,
                    prec=rng.choice(["fp64", "fp64tc5"]))
    if kind == "ab":
        n = rng.randint(50, 249)
        return dict(kind=kind, n=n, nin=rng.randint(5, 22 if n > 80 else 14), nact=nact,
                    alpha=rng.choice([0.0, 0.02, 0.5, 0.98, 1.0]))
    if kind == "point":
        return dict(kind=kind, n=rng.randint(50, 110), nin=rng.randint(5, 10), nact=nact,
                    lam=round(rng.uniform(0.02, 0.98), 3), prec="fp64tc5")
    if kind == "integrand":
        return dict(kind=kind, n=rng.randint(50, 190), nin=rng.randint(5, 18), nact=nact,
                    prec="fp64tc5")
    if kind == "ac0":
        return dict(kind=kind, n=rng.randint(50, 120), nin=rng.randint(5, 11), nact=nact)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 6), nmax=rng.randint(56, 96), prec="fp64tc6")
    if kind == "mlp":
        return dict(kind=kind, batch=rng.randint(16, 320), hidden=256)
    return dict(kind="sort", n=rng.randint(30, 96), fmt=rng.choice(["dalton8", "dalton16", "pqrs"]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _factor(n, rank, gen):
    """ERI factor as (rank, ntr), i.e. column-major with Fortran meaning (ntr, rank)."""
    p, q = synth.tri_index(n)
    p, q = torch.as_tensor(p, device=DEV), torch.as_tensor(q, device=DEV)
    g = torch.randn(rank, p.numel(), dtype=F8, device=DEV, generator=gen)
    g *= torch.exp(-(p - q).abs().to(F8) / 8.0)[None, :] * synth.ERI_SCALE
    g *= torch.exp(-torch.arange(rank, dtype=F8, device=DEV) / 60.0)[:, None]
    return g


def _orbitals(n, gen):
    return torch.linalg.qr(torch.randn(n, n, dtype=F8, device=DEV, generator=gen))[0].contiguous()


def _square(lf, n):
    p, q = synth.tri_index(n)
    p, q = torch.as_tensor(p, device=DEV), torch.as_tensor(q, device=DEV)
    m = torch.empty(lf.shape[0], n, n, dtype=F8, device=DEV)
    m[:, p, q] = lf
    m[:, q, p] = lf
    return m


def _half(lf, n, CA, CB):
    """B[P, b, a] = (CA^T L_P CB)[a, b], the pair index a fastest."""
    out = torch.empty(lf.shape[0], CB.shape[1], CA.shape[1], dtype=F8, device=DEV)
    for s in range(0, lf.shape[0], 256):
        m = _square(lf[s:s + 256], n)
        out[s:s + 256] = (CB.t() @ m) @ CA
    return out.reshape(lf.shape[0], -1)


def _integrals(lf, n, nocc, C):
    """FFOO and FOFO records in the library's layout (row = record, column = element)."""
    co = C[:, :nocc]
    fo, oo, ff = _half(lf, n, C, co), _half(lf, n, co, co), _half(lf, n, C, C)
    return oo.t() @ ff, fo.t() @ fo


def _occ(nin, nact, n, rng):
    """Natural occupations: inactive 1, active pairs (1 - x, x), virtual 0; the x well apart,
    as A-B is divided by differences of their roots."""
    x = 0.03 + 0.04 * np.arange(nact // 2) + rng.uniform(0.0, 0.02, nact // 2)
    occ = np.zeros(n)
    occ[:nin] = 1.0
    occ[nin:nin + nact] = np.concatenate([1.0 - x, x[::-1]])
    return occ


def _mean_field_rdm(occ, nin, nact, rng):
    """Packed active 2-RDM: the mean-field part plus a small symmetric correlated part."""
    o = occ[nin:nin + nact]
    e = np.eye(nact)
    g = 2 * np.einsum("p,q,pr,qs->pqrs", o, o, e, e) - np.einsum("p,q,ps,qr->pqrs", o, o, e, e)
    return synth.pack_rdm2act(g + 0.0) + 0.01 * rng.standard_normal(nact ** 2 * (nact ** 2 + 1) // 2)


def _model_system(case, seed):
    """A system's arrays without an SCF: what the assembly and the integrand read."""
    n, nin, nact = case["n"], case["nin"], case["nact"]
    gen, rng = _gen(seed), np.random.default_rng(seed)
    C = _orbitals(n, gen)
    ffoo, fofo = _integrals(_factor(n, min(6 * n, 320), gen), n, nin + nact, C)
    occ = _occ(nin, nact, n, rng)
    h = np.diag(np.sort(rng.uniform(-20.0, 5.0, n))) + 0.05 * rng.standard_normal((n, n))
    return dict(n=n, nin=nin, nact=nact, occ=occ, xone=synth.pack_sym(0.5 * (h + h.T)),
                rdm=_mean_field_rdm(occ, nin, nact, rng), ffoo=ffoo, fofo=fofo,
                indn=api.pair_space(occ, nin + nact // 2))


def _cas_system(n, nin, nact, seed):
    """A system after SCF and CAS-CI (the package's generator), resampled until A+B is positive
    definite at both ends of the lambda range, as the benchmark does."""
    for k in range(20):
        s = synth.make_system_device(n, nin, nact, 6 * n, 1000 * seed + k, device=DEV)
        C = torch.as_tensor(s.cmo, device=DEV)
        lf = torch.as_tensor(np.ascontiguousarray(s.lfac.T), device=DEV)
        ffoo, fofo = _integrals(lf, n, s.nocc, C)
        d = dict(n=n, nin=nin, nact=nact, occ=s.occ, xone=s.xone, rdm=s.rdm2act, ffoo=ffoo,
                 fofo=fofo, indn=api.pair_space(s.occ, s.nele), system=s)
        d["ends"] = [_ab(d, lam) for lam in (0.0, 1.0)]
        if all(int(torch.linalg.cholesky_ex(_sym(e[0]))[1]) == 0 for e in d["ends"]):
            return d
    raise RuntimeError("no seed with a positive definite A+B")


def _batch_shapes(case):
    """Uneven sizes from 50 to nmax, active spaces of 2, 4 and 6 orbitals in turn."""
    c = case["count"]
    return [(int(50 + (case["nmax"] - 50) * i / max(1, c - 1)), 5 + (3 * i) % 8, (2, 4, 6)[i % 3])
            for i in range(c)]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("fofo", "ffoo", "gen"):
        n, nocc, gen = case["n"], case["nin"] + case["nact"], _gen(seed)
        lf = _factor(n, case["rank"], gen)
        C = _orbitals(n, gen)
        st = dict(case=case, C=C, co=C[:, :nocc].contiguous())
        if kind == "gen":
            st["ao"] = lf.t() @ lf
        else:
            st["lfac"] = lf.t()
        return st
    if kind == "ab":
        return dict(case=case, **_model_system(case, seed))
    if kind == "integrand":
        st = _model_system(case, seed)
        N, gen = len(st["indn"]), _gen(seed + 1)
        mix = torch.randn(N, N, dtype=F8, device=DEV, generator=gen) * (0.1 / math.sqrt(N))
        q = torch.linalg.qr(mix + torch.eye(N, dtype=F8, device=DEV))[0]
        w = torch.rand(N, dtype=F8, device=DEV, generator=gen) * 30.0 + 0.2
        y = (0.7 + 0.02 * torch.rand(N, dtype=F8, device=DEV, generator=gen))[:, None] * q.t()
        w[::97] = -0.3   # unstable modes, which the integrand drops
        return dict(case=case, evec=y.contiguous().t(), eig=w, **st)
    if kind == "point":
        st = _cas_system(case["n"], case["nin"], case["nact"], seed)
        lam, (a0, a1) = case["lam"], st.pop("ends")
        # column-major, as the assembly returns them
        st["abp"] = ((1 - lam) * a0[0] + lam * a1[0]).t().contiguous().t()
        st["abm"] = ((1 - lam) * a0[1] + lam * a1[1]).t().contiguous().t()
        return dict(case=case, **st)
    if kind == "ac0":
        st = _cas_system(case["n"], case["nin"], case["nact"], seed)
        del st["ends"]
        return dict(case=case, **st)
    if kind == "batch":
        ds = [_cas_system(n, nin, nact, 50 * seed + i)
              for i, (n, nin, nact) in enumerate(_batch_shapes(case))]
        return dict(case=case, ds=ds, batch=api.BatchInputs([d.pop("system") for d in ds]))
    if kind == "mlp":
        gen = _gen(seed)
        net = api.Mlp(29, case["hidden"], 6, seed=seed)
        x = torch.randn(case["batch"], 29, device=DEV, generator=gen)
        t = torch.tanh(x[:, :6] + 0.5 * x[:, 6:12]) + 0.1 * torch.randn(
            case["batch"], 6, device=DEV, generator=gen)
        return dict(case=case, net=net, x=x, t=t.contiguous(), p0=net.params().clone())
    n, rng = case["n"], np.random.default_rng(seed)
    ntr, gen = synth.ntri(n), _gen(seed)
    rs, pq = torch.tril_indices(ntr, ntr, device=DEV)     # pq <= rs
    keep = torch.rand(rs.numel(), device=DEV, generator=gen) < 0.7   # screened integrals
    rs, pq = rs[keep], pq[keep]
    a, b = (torch.as_tensor(v, device=DEV, dtype=torch.int32) + 1 for v in synth.tri_index(n))
    p, q, r, s = a[pq], b[pq], a[rs], b[rs]
    lab = {"dalton8": lambda: p | q << 8 | r << 16 | s << 24,
           "dalton16": lambda: torch.stack([r | s << 16, p | q << 16], 1),
           "pqrs": lambda: torch.stack([p, q, r, s], 1)}[case["fmt"]]().contiguous()
    return dict(case=case, val=torch.randn(rs.numel(), dtype=F8, device=DEV, generator=gen),
                lab=lab, rs=rs, pq=pq, ntr=ntr)


# --------------------------------------------------------------------- run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "fofo":
        return api.tran4_factored(case["n"], st["lfac"], st["C"], st["co"], st["C"], st["co"],
                                  precision=case["prec"])
    if kind == "ffoo":
        return api.tran4_factored(case["n"], st["lfac"], st["co"], st["co"], st["C"], st["C"],
                                  precision=case["prec"])
    if kind == "gen":
        return api.tran4_gen(case["n"], st["C"], st["co"], st["C"], st["co"], st["ao"],
                             precision=case["prec"])
    if kind == "ab":
        return api.ab_cas_fofo(st["occ"], st["xone"], st["indn"], st["nact"], st["nin"],
                               st["ffoo"], st["fofo"], st["rdm"], case["alpha"])
    if kind == "point":
        y, eig = api.erpasymm1(st["abp"], st["abm"], mode="refined", precision=case["prec"])
        return eig, api.ace_ne_erpa_fofo(y, eig, st["occ"], st["indn"], st["nact"], st["nin"],
                                         st["fofo"], precision=case["prec"])
    if kind == "integrand":
        return api.ace_ne_erpa_fofo(st["evec"], st["eig"], st["occ"], st["indn"], st["nact"],
                                    st["nin"], st["fofo"], precision=case["prec"])
    if kind == "ac0":
        return api.ac0cas_fofo(st["occ"], st["xone"], st["indn"], st["nact"], st["nin"],
                               st["ffoo"], st["fofo"], st["rdm"])
    if kind == "batch":
        return api.ac_energy_batched(st["batch"], ngrid=8, precision=case["prec"],
                                     erpa_mode="refined", nstreams=4)
    if kind == "mlp":
        loss = st["net"].train_step(st["x"], st["t"], 1e-3)
        return loss, st["net"].params()
    return api.readtwoint(case["n"], st["val"], st["lab"], case["fmt"])


# -------------------------------------------------------------------- work
def _pairs(n, nin, nact):
    return nin * (n - nin) + nact * (n - nin - nact) + nact * (nact - 1) // 2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        fl = by = 0.0
        for n, nin, nact in _batch_shapes(case):
            N, ntr = _pairs(n, nin, nact), n * (n + 1) // 2
            # per point: the factor, L^T A L, tridiagonalisation with vectors, Y, the integrand
            fl += 8 * (1 / 3 + 2 + 4 + 1 + 1) * N ** 3
            by += 8.0 * (ntr * 6 * n + n * n)
        return {"bytes": by, "flops": fl}
    if kind == "mlp":
        h, b = case["hidden"], case["batch"]
        w = 29 * h + 2 * h * h + 6 * h
        # weights and both moments read and written, FP32
        return {"bytes": 4.0 * (6 * w + 35 * b), "flops": 6.0 * b * w}
    n = case["n"]
    ntr = n * (n + 1) // 2
    if kind == "sort":
        cnt = 0.7 * ntr * (ntr + 1) / 2
        return {"bytes": cnt * (8 + {"dalton8": 4, "dalton16": 8, "pqrs": 16}[case["fmt"]])
                + 8.0 * ntr * ntr, "flops": 0}
    nin, nact = case["nin"], case["nact"]
    o = nin + nact
    N, fo = _pairs(n, nin, nact), n * o
    if kind in ("fofo", "ffoo"):
        r = case["rank"]
        oo, ff = o * (o + 1) // 2, ntr
        # the occupied index first, and every distinct product once
        half = 2.0 * r * (n * n * o + (n * o * n if kind == "fofo" else o * o * n + n ** 3 + n * n * n / 2))
        full = r * fo * (fo + 1.0) if kind == "fofo" else 2.0 * r * oo * ff
        return {"bytes": 8.0 * (ntr * r + fo * fo), "flops": half + full}
    if kind == "gen":
        return {"bytes": 8.0 * (ntr * ntr + fo * fo),
                "flops": 2.0 * (ntr + fo) * (n * n * o + n * o * n)}
    ints = 8.0 * (fo * fo + o * o * n * n)
    z = 2.0 * nact ** 4 * (5 * n * n + 5 * n * o)
    if kind == "ab":
        return {"bytes": ints + 16.0 * N * N, "flops": 12.0 * N * N + z + 2.0 * n * o ** 4}
    if kind == "ac0":
        return {"bytes": ints, "flops": 24.0 * N * N + 2 * z + 10.0 * N * N * (nact + 2)}
    if kind == "integrand":
        return {"bytes": 8.0 * (fo * fo + N * N), "flops": 1.0 * N ** 3}
    return {"bytes": 8.0 * (fo * fo + 2 * N * N), "flops": (1 / 3 + 2 + 4 + 1 + 1) * N ** 3}


# ------------------------------------------------------- 64-bit restatement
def _sym(a):
    return 0.5 * (a + a.t())


def _rv(d):
    """RDM2val(i, j, k, l) = FRDM2(i, k, j, l) over the occupied orbitals."""
    nin, nact = d["nin"], d["nact"]
    o = nin + nact
    f = np.zeros((o,) * 4)
    occ = d["occ"][:o]
    one = (occ[:, None] == 1.0) | (occ[None, :] == 1.0)
    nn = np.where(one, occ[:, None] * occ[None, :], 0.0)
    e = np.eye(o)
    f += 2 * np.einsum("pq,pr,qs->pqrs", nn, e, e) - np.einsum("pq,ps,qr->pqrs", nn, e, e)
    f[nin:, nin:, nin:, nin:] = synth.unpack_rdm2act(d["rdm"], nact)
    return torch.as_tensor(np.ascontiguousarray(f.transpose(0, 2, 1, 3)), device=DEV)


def _ci(occ):
    return np.where(occ >= 0.5, np.sqrt(occ), -np.sqrt(occ))


def _tables(d):
    p, q = (torch.as_tensor(d["indn"][:, k] - 1, device=DEV) for k in (0, 1))
    c = torch.as_tensor(_ci(d["occ"]), device=DEV)
    o = torch.as_tensor(d["occ"], device=DEV)
    g = torch.zeros(d["n"], dtype=torch.long, device=DEV)
    g[d["nin"]:] = 1
    g[d["nin"] + d["nact"]:] = 2
    return p, q, c, o, g


def _views(d):
    """(ab|cd) as F[a, b, c, d] from FOFO (b, d occupied) and G[a, b, c, d] from FFOO (c, d occupied)."""
    n, o = d["n"], d["nin"] + d["nact"]
    F = d["fofo"].view(o, n, o, n).permute(1, 0, 3, 2)
    G = d["ffoo"].view(o, o, n, n).permute(3, 2, 1, 0)
    return F, G


def _ab(d, lam, ab1=False):
    """A+B, A-B (rows pq, columns rs) and E_CAS by the in-core formulas in FP64 torch."""
    n, nin, nact = d["n"], d["nin"], d["nact"]
    o = nin + nact
    p, q, c, oc, g = _tables(d)
    F, G = _views(d)
    rv = _rv(d)
    same = 0.0 if ab1 else 1.0

    def ac(a, b, e, f):
        return torch.where((a == b) & (b == e) & (e == f), same, lam).to(F8)

    h = torch.as_tensor(synth.unpack_sym(d["xone"], n), device=DEV)
    go, oo = g[:o], oc[:o]
    jv = torch.einsum("ijkk->ijk", G)
    kv = torch.einsum("jkik->ijk", F)
    gi, gj, gk = g[:, None, None], g[None, :, None], go[None, None, :]
    corr = torch.where((gi == gj) & (gk != gi), oo * (2 * jv - kv), 0.0).sum(-1)
    t = oo * (2 * ac(gi, gj, gk, gk) * jv - ac(gi, gi, gj, gk) * kv)
    auxi, auxio = t.sum(-1), t[..., :nin].sum(-1)
    eq = g[:, None] == g[None, :]
    hno = torch.where(eq, -corr if ab1 else h + (1 - lam) * corr, lam * h)
    e1, e2 = (oo * torch.diagonal(h)[:o]).sum(), torch.einsum("ijkl,ijkl->", rv, G[:o, :o])
    w = ac(g[:, None, None, None], go[None, :, None, None], go[None, None, :, None],
           go[None, None, None, :]) * F[:o, :, :, :].permute(2, 3, 0, 1)   # (kl|ij): [k, l, i, j]
    wmat = torch.zeros(n, n, dtype=F8, device=DEV)
    wmat[:, :o] = torch.einsum("klij,ijrl->kr", w, rv)
    del w, t, jv, kv, corr

    act = slice(nin, o)
    Fa, ra = F[act, act], rv[act, act, act, act]                 # (TU|ab), [T, U, ...]
    z1 = torch.einsum("tuab,tucd->abcd", Fa, ra)
    f4 = F[:, act, :, act]                                       # (rU|pT): [r, u, p, t]
    z4, z7 = torch.einsum("rupt,tqsu->prqs", f4, ra), torch.einsum("rupt,tqus->prqs", f4, ra)
    f5 = F[act, :, :, act]                                       # (Tq|rU): [t, q, r, u]
    z5, z6 = torch.einsum("tqru,tpsu->rqps", f5, ra), torch.einsum("tqru,tpus->rqps", f5, ra)
    z8 = torch.einsum("tuqs,tupr->qspr", Fa[:, :, :o], ra)
    z9 = torch.einsum("prkl,qskl->prqs", G[:, :, act, act], ra)
    g10 = G[:o, act, :, act]                                     # (qT|sU): [q, t, s, u]
    z10, z13 = torch.einsum("qtsu,tpru->qspr", g10, ra), torch.einsum("qtsu,tpur->qspr", g10, ra)
    g11 = G[:, act, :, act]
    z11, z12 = torch.einsum("ptsu,tqru->psqr", g11, ra), torch.einsum("ptsu,tqur->psqr", g11, ra)

    N = p.numel()
    gp, gq, gr, gs = g[p][:, None], g[q][:, None], g[p][None, :], g[q][None, :]
    P, Q, R, S = p[:, None], q[:, None], p[None, :], q[None, :]
    Pa, Qa, Ra, Sa = ((x - nin).clamp(0, max(nact - 1, 0)) for x in (P, Q, R, S))

    def at(x, *i):
        return x[tuple(v.expand(N, N) for v in i)]

    def X(a, b, ga, gb):
        m = (ga <= 1) & (gb <= 1) & ~((ga == 1) & (gb == 1))
        return torch.where(m, oc[a] * oc[b], 0.0)

    x1 = X(P, R, gp, gr) + X(Q, S, gq, gs) - X(Q, R, gq, gr) - X(P, S, gp, gs)
    x1 = torch.where((R >= nin) & (P >= nin), ac(gp, gq, gr, gs) * x1, 0.0)
    mo = 4 * x1 * at(F, R, S, P, Q)
    a = x1 * at(F, R, Q, P, S)
    s = -x1 * at(G, P, R, Q, S)
    del x1
    pa, qa, ra_, sa, pv, rvir = gp == 1, gq == 1, gr == 1, gs == 1, P >= nin, R >= nin

    def add(dst, cond, coef, z, i, sign=1.0):
        if nact:
            m = cond.expand(N, N).nonzero()
            i = [v.expand(N, N)[m[:, 0], m[:, 1]] for v in i]
            dst[m[:, 0], m[:, 1]] += sign * coef.expand(N, N)[m[:, 0], m[:, 1]] * z[tuple(i)]

    one = torch.ones_like(gp)
    cps, cqr = ac(gp, gs, one, one), ac(gq, gr, one, one)
    cpr, cqs = ac(gp, gr, one, one), ac(gq, gs, one, one)
    add(a, pv & ra_ & qa, cps, z1, (P, S, Qa, Ra))
    add(a, rvir & sa & pa, cqr, z1, (R, Q, Pa, Sa))
    m4 = rvir & sa & qa & pv
    add(s, m4, cpr, z4, (P, R, Qa, Sa))
    add(a, m4, cpr, z7, (P, R, Qa, Sa), -1.0)
    add(s, m4, cpr, z9, (P, R, Qa, Sa))
    m5 = rvir & sa & pa
    add(a, m5, cqr, z5, (R, Q, Pa, Sa))
    add(s, m5, cqr, z6, (R, Q, Pa, Sa), -1.0)
    m8 = ra_ & pa
    add(s, m8, cqs, z8, (Q, S, Pa, Ra))
    add(s, m8, cqs, z10, (Q, S, Pa, Ra))
    add(a, m8, cqs, z13, (Q, S, Pa, Ra), -1.0)
    m11 = ra_ & qa & pv
    add(a, m11, cps, z11, (P, S, Qa, Ra))
    add(s, m11, cps, z12, (P, S, Qa, Ra), -1.0)

    def aux(ga, gb, x, y):
        both = (ga <= 1) & (gb <= 1)
        aa = (ga == 1) & (gb == 1)
        return torch.where(aa, auxio[x, y], torch.where(both, auxi[x, y], 0.0))

    def onebody(dst, cond, x, y, na_, nb, ga, gb):
        m = cond.nonzero()
        i, j = m[:, 0], m[:, 1]
        x, y, na_, nb, ga, gb = (v.expand(N, N)[i, j] for v in (x, y, na_, nb, ga, gb))
        dst[i, j] += (oc[na_] - oc[nb]) * hno[x, y] - wmat[x, y] + oc[na_] * aux(ga, gb, x, y)

    onebody(s, P == R, Q, S, P, S, gp, gr)
    onebody(s, Q == S, P, R, Q, R, gq, gs)
    onebody(a, Q == R, P, S, Q, S, gq, gr)
    onebody(a, P == S, Q, R, P, R, gp, gs)
    plus, minus = c[p] + c[q], c[p] - c[q]
    dp, dm = plus[:, None] * plus[None, :], minus[:, None] * minus[None, :]
    abp = (s + a) / torch.where(dp == 0, 1.0, dp)
    abm = (s - a + mo) / torch.where(dm == 0, 1.0, dm)
    if ab1:
        abp, abm = _sym(abp), _sym(abm)
    return abp, abm, float(2 * e1 + e2)


def _kernel(d):
    """Mask, weights and (rs|pq) of the integrand."""
    p, q, c, o, g = _tables(d)
    F, _ = _views(d)
    f = F[p[None, :], q[None, :], p[:, None], q[:, None]]
    m = ~((g[p] == g[q])[:, None] & (g[p][:, None] == g[p][None, :]) & (g[p][:, None] == g[q][None, :]))
    cc = c[p] + c[q]
    return torch.where(m, f, 0.0), cc, o[p] * (1 - o[q]) + o[q] * (1 - o[p])


def _w(d, y, eig):
    f, cc, dn = _kernel(d)
    y = torch.where((eig > 1e-3) & (eig < 1e8), y, 0.0)
    return float(2 * (f * cc[:, None] * cc[None, :] * (y @ y.t())).sum() - (dn * torch.diagonal(f)).sum())


def _erpa(abp, abm):
    L = torch.linalg.cholesky(_sym(abp))
    w2, u = torch.linalg.eigh(_sym(L.t() @ _sym(abm) @ L))
    ok = w2 > 1e-6
    om = torch.where(ok, w2.clamp_min(1e-6).sqrt(), w2)
    return (L @ u) / torch.where(ok, (2 * om.abs()).sqrt(), 1.0), om


def _ac0(d):
    a0p, a0m, etot = _ab(d, 0.0)
    a1p, a1m, _ = _ab(d, 1.0, ab1=True)
    pn, qn = d["indn"][:, 0] - 1, d["indn"][:, 1] - 1
    nin, o, N = d["nin"], d["nin"] + d["nact"], len(pn)
    blocks, single = {}, []
    for i, (p, q) in enumerate(zip(pn, qn)):
        if p >= o and q < nin:
            single.append(i)
        else:
            blocks.setdefault(("v", p) if p >= o else (("i", q) if q < nin else ("a",)), []).append(i)
    hp, hm = a0p.cpu().numpy(), a0m.cpu().numpy()
    Y, X, eig = np.zeros((N, N)), np.zeros((N, N)), np.zeros(N)
    for idx in blocks.values():
        ix = np.ix_(idx, idx)
        A, B = 0.5 * (hp[ix] + hp[ix].T), 0.5 * (hm[ix] + hm[ix].T)
        e, v = np.linalg.eigh(A)
        R = (v * np.sqrt(np.abs(e))) @ v.T
        H = R @ B @ R
        w2, z = np.linalg.eigh(0.5 * (H + H.T))
        y = R @ z
        for k, wk in enumerate(w2):
            eig[idx[k]] = wk
            if wk > 1e-6:
                om = math.sqrt(wk)
                s = 2 / om * (y[:, k] @ B @ y[:, k])
                yk = y[:, k] / math.sqrt(s) if s > 0 else 0 * y[:, k]
                Y[idx, idx[k]], X[idx, idx[k]], eig[idx[k]] = yk, B @ yk / om, om
    for i in single:
        eig[i] = hp[i, i]
        Y[i, i] = X[i, i] = math.sqrt(0.5)
    Y, X, eig = (torch.as_tensor(v, device=DEV) for v in (Y, X, eig))
    den = eig[:, None] + eig[None, :]
    live = (eig != 0)[:, None] & (eig != 0)[None, :]
    work_ = torch.where(live, 2 * (X.t() @ a1p @ X - Y.t() @ a1m @ Y) / den, 0.0)
    f, cc, _ = _kernel(d)
    return float((cc[:, None] * cc[None, :] * (Y @ work_ @ Y.t()) * f).sum()), etot


def exact(case, seed):
    kind = case["kind"]
    st = prepare(case, seed)
    if kind in ("fofo", "ffoo"):
        lf, n = st["lfac"].t(), case["n"]
        if kind == "fofo":
            z = _half(lf, n, st["C"], st["co"])
            return z.t() @ z
        return _half(lf, n, st["co"], st["co"]).t() @ _half(lf, n, st["C"], st["C"])
    if kind == "gen":
        n = case["n"]
        t = _half(st["ao"], n, st["C"], st["co"])              # (rs, ab)
        return _half(t.t().contiguous(), n, st["C"], st["co"])
    if kind == "ab":
        return _ab(st, case["alpha"])
    if kind == "point":
        y, eig = _erpa(st["abp"], st["abm"])
        return eig, _w(st, y, eig)
    if kind == "integrand":
        return _w(st, st["evec"], st["eig"])
    if kind == "ac0":
        return _ac0(st)
    if kind == "batch":
        x, wt = np.polynomial.legendre.leggauss(8)
        x, wt = 0.5 * (x + 1), 0.5 * wt
        ecas, wl = [], []
        for d in st["ds"]:
            (p0, m0, e), (p1, m1, _) = d["ends"]
            ecas.append(e)
            wl.append([_w(d, *_erpa((1 - t) * p0 + t * p1, (1 - t) * m0 + t * m1)) for t in x])
        wl = np.array(wl)
        return wl @ wt, np.array(ecas), wl, np.zeros(len(wl), dtype=np.int32)
    if kind == "mlp":
        return _mlp(st)
    out = torch.zeros(st["ntr"], st["ntr"], dtype=F8, device=DEV)
    out[st["rs"], st["pq"]] = st["val"]
    out[st["pq"], st["rs"]] = st["val"]
    return out


def _mlp(st):
    """One Adam step from fresh moments; the products read BF16 copies of the weights."""
    h = st["case"]["hidden"]
    shapes = [(h, 29), (h,), (h, h), (h,), (h, h), (h,), (6, h), (6,)]
    p0 = st["p0"].to(F8)
    parts, at = [], 0
    for k, s in enumerate(shapes):
        v = st["p0"][at:at + math.prod(s)].view(s)
        at += math.prod(s)
        parts.append((v.to(torch.bfloat16) if k % 2 == 0 else v).to(F8).requires_grad_())
    a = st["x"].to(F8)
    for k in range(4):
        a = a @ parts[2 * k].t() + parts[2 * k + 1]
        if k < 3:
            a = torch.nn.functional.gelu(a)
    loss = ((a - st["t"].to(F8)) ** 2).mean()
    g = torch.cat([v.reshape(-1) for v in torch.autograd.grad(loss, parts)])
    return float(loss), p0 - 1e-3 * g / (g.abs() + 1e-8)
