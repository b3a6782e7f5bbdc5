"""Kernels at the sizes where their tiling can go wrong, against the oracle.

Inputs need no SCF here: random orthogonal orbitals and occupations, so that the sizes
are free. Tolerances as in the parity tests.
"""
import numpy as np
import pytest
import torch

from gammcor_gb300 import api, synth
from oracle import ac_cas_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=DEV)


def model(n, nin, nact, seed=0):
    """Integrals, one-electron part, occupations and 2-RDM without an SCF."""
    rng = np.random.default_rng(seed)
    lf = synth.make_lfac(n, 3 * n, rng) * 0.1
    C, _ = np.linalg.qr(rng.standard_normal((n, n)))
    occ = np.zeros(n)
    occ[:nin] = 1.0
    occ[nin:nin + nact] = np.linspace(0.96, 0.05, nact)
    ffoo, fofo = R.transform_fofo_ffoo(C, lf @ lf.T, nin, nact)
    return dict(n=n, nin=nin, nact=nact, occ=occ, xone=rng.standard_normal(synth.ntri(n)),
                rdm=rng.standard_normal(nact ** 2 * (nact ** 2 + 1) // 2), ffoo=ffoo, fofo=fofo,
                indn=R.pair_space(occ, nin + nact // 2), lf=lf, C=C)


def assembled(m, indn, lam, ab1=False):
    return api.ab_cas_fofo(m["occ"], m["xone"], indn, m["nact"], m["nin"], t(m["ffoo"]),
                           t(m["fofo"]), m["rdm"], lam, ab1=ab1)


# no inactive, no active, more than one 32-wide chunk of occupied and of all orbitals, sizes
# around the 8 x 4 row tiles, an inactive occupation below 1 and an active one of exactly 1
@pytest.mark.parametrize("n,nin,nact,ab1,odd_occ", [(9, 0, 3, False, False), (13, 4, 0, False, False),
                                                    (40, 33, 2, False, True), (33, 3, 5, True, True),
                                                    (17, 5, 1, False, False)])
def test_assembly_tiles(gpu_lib, n, nin, nact, ab1, odd_occ):
    m = model(n, nin, nact, seed=n)
    if odd_occ:
        m["occ"][0], m["occ"][nin] = 0.99, 1.0
        m["occ"][-1] = 1e-3   # virtual occupations that differ: the general form of every element
    rng = np.random.default_rng(1)
    indn = m["indn"][rng.permutation(len(m["indn"]))]
    rp, rm, re = R.ab_cas_fofo(m["occ"], m["xone"], np.eye(n), indn, nin, nact, m["ffoo"],
                               m["fofo"], m["rdm"], 0.3, ab1=ab1)
    gp, gm, ge = assembled(m, indn, 0.3, ab1)
    assert np.abs(gp.cpu().numpy() - rp).max() < 1e-10 * np.abs(rp).max()
    assert np.abs(gm.cpu().numpy() - rm).max() < 1e-10 * np.abs(rm).max()
    assert abs(ge - re) < 1e-9


def test_assembly_shows_a_nonfinite_integral_with_zero_weight(gpu_lib):
    """(01|23) of four inactive orbitals has no weight in A+-B, but stays visible."""
    m = model(17, 5, 2)
    m["fofo"][0 + 1 * m["n"], 2 + 3 * m["n"]] = np.nan
    gp, gm, _ = assembled(m, m["indn"], 0.5)
    assert not torch.isfinite(gp).all() and not torch.isfinite(gm).all()


# AC0 blocks of odd and even size, of one pair, and an active-active block of 55 pairs; with a
# one-electron part whose order is turned, A+ of some blocks is not positive definite
@pytest.mark.parametrize("n,nin,nact,turn", [(12, 2, 1, 0), (14, 1, 2, 0), (21, 2, 5, 0), (30, 0, 11, 0),
                                             (21, 2, 5, 1), (18, 3, 4, 1)])
def test_ac0_block_sizes(gpu_lib, n, nin, nact, turn):
    from oracle import ac0_ref as A
    m = model(n, nin, nact, seed=n)
    # a dominant one-electron diagonal keeps the zeroth-order blocks stable
    m["xone"] *= 0.05
    d = np.cumsum(np.arange(1, n + 1)) - 1
    m["xone"][d] = np.linspace(-30.0, 10.0, n)
    if turn:
        m["xone"][d[nin:nin + nact]] = m["xone"][d[nin:nin + nact]][::-1]
    m["rdm"] = np.zeros_like(m["rdm"])
    o = m["occ"][nin:nin + nact]
    e = np.eye(nact)
    m["rdm"] = synth.pack_rdm2act(2 * np.einsum("p,q,pr,qs->pqrs", o, o, e, e)
                                  - np.einsum("p,q,ps,qr->pqrs", o, o, e, e))
    e0, etot = A.ac0cas_fofo(m["occ"], m["xone"], np.eye(n), m["indn"], nin, nact, m["ffoo"],
                             m["fofo"], m["rdm"])
    ge, get = api.ac0cas_fofo(m["occ"], m["xone"], m["indn"], nact, nin, t(m["ffoo"]),
                              t(m["fofo"]), m["rdm"])
    assert abs(ge - e0) < 1e-9 * max(1.0, abs(e0))
    assert abs(get - etot) < 1e-9 * max(1.0, abs(etot))


def sliced_product(A, B, S):
    """C = A B^T by the balanced base-128 slicing with exact integer sums: the bits that the
    sliced GEMM has to give (up to 5 slices; every weight's sum fits an int64)."""
    def cut(X):
        e = np.where((X != 0).any(1), np.frexp(np.abs(X).max(1))[1], 0)
        n = np.rint(np.ldexp(X, (7 * S - e)[:, None])).astype(np.int64)
        d = []
        for _ in range(S - 1):
            d.append(((n + 64) & 127) - 64)
            n = (n - d[-1]) >> 7
        return e, [n] + d[::-1]
    ea, a = cut(A)
    eb, b = cut(B)
    acc = sum((a[t] @ b[u].T) << (7 * (S - 1 - t - u)) for t in range(S) for u in range(S - t))
    return np.ldexp(acc.astype(np.float64), ea[:, None] + eb[None, :] - 7 * (S + 1))


# rows and K around the 32-row and 64-value tiles of the slicing, zero rows, ties, subnormals
@pytest.mark.parametrize("S", [4, 5])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 31, 63), (65, 97, 64), (130, 40, 129)])
def test_sliced_gemm_bits(gpu_lib, S, m, n, k):
    rng = np.random.default_rng(m * k)
    A = rng.standard_normal((m, k)) * 2.0 ** rng.integers(-30, 4, (m, k))
    B = rng.standard_normal((n, k)) * 2.0 ** rng.integers(-30, 4, (n, k))
    A[::7] = np.round(A[::7] * 2 ** 10) / 2 ** 10     # exact ties among the roundings
    A[-1] = 0.0
    if m > 2:
        A[1] = 3.0 * 2.0 ** -1070 * rng.integers(-5, 6, k)
    C = api.tc_gemm_nt(t(A), t(B), f"fp64tc{S}").cpu().numpy()
    assert np.array_equal(C, sliced_product(A, B, S))


# Products whose waves of tiles make the default another width than the forced one, with ragged
# rows, columns and K: plain, symmetric (FOFO with one pair of blocks) and reduced (integrand)
@pytest.mark.parametrize("S", [4, 5])
def test_sliced_gemm_tile_choice(gpu_lib, S):
    g = torch.Generator(device=DEV).manual_seed(S)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device=DEV, generator=g)
    n, nin, nact, prec = 76, 28, 4, f"fp64tc{S}"
    occ = np.r_[np.ones(nin), 0.9, 0.7, 0.2, 0.1, np.zeros(n - nin - nact)]
    indn = R.pair_space(occ, nin + 2)
    N, nocc = len(indn), nin + nact
    A, B, L = rnd(19401, 33), rnd(141, 33), rnd(64, 101 * 100 // 2).t()
    C = torch.linalg.qr(rnd(100, 100))[0]
    Co = C[:, :30].contiguous()
    Y, fofo = torch.linalg.qr(rnd(N, N))[0], rnd(n * nocc, n * nocc)
    eig = torch.linspace(0.1, 9.0, N, dtype=torch.float64, device=DEV)
    eig[::5] = -0.1  # dropped modes: Y Y^T is no unit matrix
    got = []
    for width in (0, 64):
        ctx = api.Context(0)
        try:
            ctx.set_gemm_tile(width)
            got.append((api.tc_gemm_nt(A, B, prec, ctx=ctx),
                        api.tran4_factored(100, L, C, Co, C, Co, precision=prec, ctx=ctx),
                        api.ace_ne_erpa_fofo(Y, eig, occ, indn, nact, nin, fofo, precision=prec,
                                             ctx=ctx)))
        finally:
            ctx.close()
    assert torch.equal(got[0][0], got[1][0])
    assert torch.equal(got[0][1], got[1][1])
    # N^2 terms, each within 2^-52 of itself, added in another grouping
    assert abs(got[0][2] - got[1][2]) <= 1e-12 * N * fofo.abs().max().item()


# widths (nA, nB, nC, nD); -1 repeats the block before it, so that the pair index is symmetric
@pytest.mark.parametrize("n,widths", [(33, (33, 5, 33, 5)), (33, (5, -1, 33, -1)), (20, (3, 17, 9, -1)),
                                      (20, (7, -1, 4, 11)), (65, (2, 65, 2, 65)), (5, (1, 1, 5, 2)),
                                      (130, (3, -1, 130, -1))])
@pytest.mark.parametrize("entry", ["factored", "gen"])
@pytest.mark.parametrize("precision", ["fp64tc5", "fp64"])
def test_transform_block_shapes(gpu_lib, n, widths, entry, precision):
    rng = np.random.default_rng(n)
    lf = synth.make_lfac(n, 2 * n + 1, rng) * 0.1
    C, blocks = np.linalg.qr(rng.standard_normal((n, n)))[0], []
    for i, w in enumerate(widths):
        blocks.append(blocks[-1] if w < 0 else t(np.roll(C, i // 2, axis=1)[:, :w]))
    if widths[:2] == widths[2:]:
        blocks[2:] = blocks[:2]
    ref = R.tran4_gen(n, *[b.cpu().numpy() for b in blocks], lf @ lf.T)
    if entry == "factored":
        out = api.tran4_factored(n, t(lf), *blocks, precision=precision)
    else:
        out = api.tran4_gen(n, *blocks, t(lf @ lf.T), precision=precision)
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-10


# pair counts below, at and above the 32-wide tiles and the GEMM's column tiles, dropped modes,
# and (rs|pq) that differs from (pq|rs): both enter
@pytest.mark.parametrize("precision", ["fp64tc5", "fp64tc6"])
@pytest.mark.parametrize("n,nin,nact", [(4, 1, 1), (13, 2, 2), (17, 4, 2), (33, 3, 5)])
def test_integrand_tiles(gpu_lib, precision, n, nin, nact):
    m = model(n, nin, nact, seed=n)
    rng = np.random.default_rng(2)
    N = len(m["indn"])
    m["fofo"] = m["fofo"] * (1.0 + 0.1 * rng.standard_normal(m["fofo"].shape))
    y = np.linalg.qr(rng.standard_normal((N, N)))[0] * 0.7
    e = rng.uniform(0.1, 20.0, N)
    e[::5], e[1::7] = -0.1, 2e8
    ref = R.ac_ene_erpa_fofo(y, e, m["occ"], nin, nact, m["indn"], m["fofo"])
    w = api.ace_ne_erpa_fofo(t(y.T).t(), t(e), m["occ"], m["indn"], nact, nin, t(m["fofo"]),
                             precision=precision)
    assert abs(w - ref) < 5e-9


# ragged row blocks, units that are no multiple of 8 or 32, wide outputs, and a layer beyond the
# fused kernels' width
@pytest.mark.parametrize("din,hid,dout,B", [(29, 256, 6, 5), (3, 37, 33, 1), (64, 8, 1, 307),
                                            (5, 258, 3, 9)])
def test_mlp_sizes(gpu_lib, din, hid, dout, B):
    from oracle import mlp_ref
    rng = np.random.default_rng(B)
    net = api.Mlp(din, hid, dout, seed=2)
    x = rng.standard_normal((B, din)).astype(np.float32)
    y = rng.standard_normal((B, dout)).astype(np.float32)
    p = net.params().cpu().numpy()
    dims = [din, hid, hid, hid, dout]
    ref, _, _ = mlp_ref.forward(p, dims, x)
    assert np.abs(net.forward(x).cpu().numpy() - ref).max() < 1e-4 * np.abs(ref).max()
    loss_ref, g_ref = mlp_ref.loss_and_grad(p, dims, x, y)
    loss, g = net.gradients(x, y)
    assert abs(loss - loss_ref) < 1e-4 * loss_ref
    g, off = g.cpu().numpy(), 0
    for l in range(4):
        for size in (dims[l] * dims[l + 1], dims[l + 1]):
            a, b = g[off:off + size], g_ref[off:off + size]
            assert np.abs(a - b).max() < 1e-4 * max(np.abs(b).max(), 1e-12), (l, size)
            off += size
    # one Adam step from fresh moments moves every parameter by lr g / (|g| + eps)
    assert abs(net.train_step(x, y, 1e-3) - loss) < 1e-5 * loss
    step = p - net.params().cpu().numpy()
    assert np.abs(step - 1e-3 * g / (np.abs(g) + 1e-8)).max() < 1e-6


# every pair of pair indices at most once (the one-pass road), and one repeated pair far away in
# the input, beside it in a warp, or mirrored (the exact resolution)
@pytest.mark.parametrize("fmt", ["pqrs", "dalton8", "dalton16"])
@pytest.mark.parametrize("repeat", [None, "far", "near", "mirror"])
@pytest.mark.parametrize("n", [1, 2, 9])
def test_sort_single_and_repeated_pairs(gpu_lib, fmt, repeat, n):
    from oracle import sorter_ref as S
    rng = np.random.default_rng(n)
    tri = [(a, b) for b in range(1, n + 1) for a in range(1, b + 1)]
    lab = [(tri[x], tri[y]) for y in range(len(tri)) for x in range(y + 1) if rng.random() < 0.8 or n < 3]
    if repeat == "far":
        lab.append(lab[0])
    elif repeat == "near":
        lab.insert(1, lab[0])
    elif repeat == "mirror":
        lab.append((lab[-1][1], lab[-1][0]))
    p, q, r, s = (np.array([x[i][j] for x in lab]) for i in (0, 1) for j in (0, 1))
    lab = {"pqrs": lambda: np.stack([p, q, r, s], 1).ravel(),
           "dalton8": lambda: p | q << 8 | r << 16 | s << 24,
           "dalton16": lambda: np.stack([r | s << 16, p | q << 16], 1).ravel()}[fmt]()
    lab = lab.astype(np.uint32).view(np.int32)
    vals = rng.standard_normal(len(p))
    got = api.readtwoint(n, torch.as_tensor(vals, device=DEV), torch.as_tensor(lab, device=DEV), fmt)
    assert np.array_equal(got.cpu().numpy(), S.readtwoint(n, vals, lab, fmt))
