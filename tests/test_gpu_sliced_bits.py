"""The sliced GEMM's result bits: every element is the rounded sum of exact integer products of the
balanced base-128 digits of its row and column, whatever the tile, the K chunks and the
order in which the products of a chunk complete."""
import pytest
import torch

from gammcor_gb300 import api

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def two(e):
    """2^e in FP64, exactly, from its bits (torch.ldexp takes a power in FP32)."""
    return ((e.long() + 1023) << 52).view(torch.float64)


def digits(X, S):
    """Exponent of each row's largest entry, and the S digits of rint(x 2^(7 S - e))."""
    e = torch.where((X != 0).any(1), torch.frexp(X.abs().amax(1))[1].long(), 0)
    n = torch.round(X * two(7 * S - e)[:, None]).long()
    d = []
    for _ in range(S - 1):
        d.append(((n + 64) & 127) - 64)
        n = (n - d[-1]) >> 7
    return e, [x.double() for x in [n] + d[::-1]]


def sliced_product(A, B, S):
    """C = A B^T of the digits. The sums of a weight are integers below 2^53, so FP64 products give
    them exactly. Six slices: the lowest weight of each chunk of 480 K is rounded to 2^7."""
    (ea, a), (eb, b) = digits(A, S), digits(B, S)
    top, chunk = min(S, 5), 480 if S == 6 else A.shape[1]
    acc = torch.zeros(A.shape[0], B.shape[0], dtype=torch.int64, device=A.device)
    for k in range(0, A.shape[1], chunk):
        for d in range(S):
            v = sum(a[t][:, k:k + chunk] @ b[d - t][:, k:k + chunk].T for t in range(d + 1))
            acc += v.long() << 7 * (top - 1 - d) if d < top else torch.round(v / 128).long()
    return acc.double() * two(ea[:, None] + eb[None, :] - 7 * (top + 1))


def operands(m, n, k, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda r: (torch.randn(r, k, dtype=torch.float64, device=DEV, generator=g)
                     * 2.0 ** torch.randint(-12, 3, (r, k), device=DEV, generator=g))
    return rnd(m), rnd(n)


# Several K chunks (672, 576 and 480 long) with every tile width: 32 for at most 32 columns, 48
# where two of its waves are one of the wider tiles', the others forced. Each product is
# repeated: the MMAs of a chunk are issued back to back, two CTAs of the narrow tiles share an SM.
@pytest.mark.parametrize("S,m,n,k,width", [(4, 700, 30, 2100, 0), (5, 700, 30, 2100, 0),
                                           (6, 700, 30, 2100, 0), (4, 38900, 47, 1400, 0),
                                           (5, 38900, 47, 1400, 0), (4, 600, 300, 2100, 64),
                                           (5, 600, 300, 2100, 64), (6, 600, 300, 2100, 64),
                                           (4, 600, 300, 2100, 96), (5, 600, 300, 2100, 96),
                                           (4, 600, 300, 2100, 128)])
def test_bits_over_several_chunks(gpu_lib, S, m, n, k, width):
    A, B = operands(m, n, k, S)
    ref = sliced_product(A, B, S)
    ctx = api.Context(0)
    try:
        ctx.set_gemm_tile(width)
        for _ in range(30):
            assert torch.equal(api.tc_gemm_nt(A, B, f"fp64tc{S}", ctx=ctx), ref)
    finally:
        ctx.close()


# The 32-wide tile of six slices (three stages of 32 K): fewer K blocks than stages, as many, more
@pytest.mark.parametrize("k", [1, 33, 96, 129, 250])
def test_six_slices_in_the_narrow_tile(gpu_lib, k):
    A, B = operands(300, 17, k, k)
    assert torch.equal(api.tc_gemm_nt(A, B, "fp64tc6"), sliced_product(A, B, 6))


def test_narrow_tiles_of_several_kernels_share_sms(gpu_lib):
    """32- and 48-wide tiles and the split-BF16 GEMM from four threads at once: CTAs of different
    kernels on one SM, each with its own slices in the collector buffer, leave each other's bits alone."""
    from concurrent.futures import ThreadPoolExecutor
    jobs = [("fp64tc5", *operands(20000, 30, 700, 1)), ("fp64tc4", *operands(20000, 31, 700, 2)),
            ("fp64tc5", *operands(38900, 47, 300, 3)), ("bf16x6", *operands(3000, 700, 700, 4))]
    torch.cuda.synchronize()

    def repeat(job):
        prec, A, B = job
        stream = torch.cuda.Stream()
        ctx = api.Context(0, stream)
        try:
            with torch.cuda.stream(stream):
                ref = api.tc_gemm_nt(A, B, prec, ctx=ctx)
                same = all(torch.equal(api.tc_gemm_nt(A, B, prec, ctx=ctx), ref) for _ in range(40))
                return same and (prec == "bf16x6" or torch.equal(ref, sliced_product(A, B, int(prec[-1]))))
        finally:
            ctx.close()
    with ThreadPoolExecutor(4) as ex:
        assert all(ex.map(repeat, jobs))
