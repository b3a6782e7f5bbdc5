// AO -> MO four-index transform into the FFOO / FOFO record layout.
//
// gc_tran4_gen follows tran4_gen (tran.f90:313-423): phase 1 contracts every
// AO pair record rs with CA^T . M . CB, phase 2 contracts every (ab| column
// over the unpacked rs index with CC^T . M . CD. Out-of-core files become
// HBM buffers: the AOTWOSORT tensor, the half-transformed TMPMO intermediate
// (ntr x nA*nB) and the output all stay resident. Packed triangles are
// expanded by the unpack kernels below (triang_to_sq, tran.f90:1221-1247).
//
// gc_tran4_factored produces the same records from the ERI factor L:
// B_P = CA^T L_P CB for every P, then (ab|cd) = sum_P B_P(ab) B'_P(cd).
//
// In FP64 and in the sliced precisions the packed triangles are the operands
// themselves (half_fp64, tc_half_packed); in the sliced ones a block of orbitals
// given twice (the same pointer and width) makes its pair index symmetric
// (tc_pair_product). The split-BF16 precisions expand the triangles.
#include "gc_internal.cuh"
#include "gc_tc_gemm.cuh"

namespace {

const size_t kChunkBytes = size_t(1) << 30;  // staging per chunk

__host__ __device__ inline long long tri_pack(int p, int q) {  // p <= q, 0-based
  return (long long)p + (long long)q * (q + 1) / 2;
}

// Expand records [rs0, rs0+cnt) of the packed tensor G (ntr x ntr, record-major)
// into cnt column-major n x n matrices.
__global__ void unpack_records(const double *__restrict__ G, long long ntr, int n, long long rs0,
                               int cnt, double *__restrict__ M) {
  long long total = (long long)cnt * n * n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int p = (int)(t % n);
    long long r = t / n;
    int q = (int)(r % n);
    long long k = r / n;
    long long pq = p <= q ? tri_pack(p, q) : tri_pack(q, p);
    M[t] = G[(rs0 + k) * ntr + pq];
  }
}

// Mt[c][rs] = H[rs][c0 + c]: columns [c0, c0+cnt) of H (ntr x ncol, column fastest) as packed
// records.
__global__ void transpose_columns(const double *__restrict__ H, long long ntr, long long ncol,
                                  long long c0, int cnt, double *__restrict__ Mt) {
  __shared__ double tile[32][33];
  const long long rs0 = (long long)blockIdx.x * 32, cb = (long long)blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int i = ty; i < 32; i += 8)
    if (rs0 + i < ntr && cb + tx < cnt) tile[i][tx] = H[(rs0 + i) * ncol + c0 + cb + tx];
  __syncthreads();
  for (int j = ty; j < 32; j += 8)
    if (cb + j < cnt && rs0 + tx < ntr) Mt[(cb + j) * ntr + rs0 + tx] = tile[tx][j];
}

// Expand columns [c0, c0+cnt) of H (ntr x ncol, row index = packed rs, column
// fastest) into cnt column-major n x n matrices. Tiled through shared memory so
// that both the H reads (along columns) and the M writes (along packed rs,
// i.e. along r for fixed s) are contiguous.
__global__ void unpack_columns(const double *__restrict__ H, long long ntr, long long ncol, int n,
                               long long c0, int cnt, double *__restrict__ M) {
  __shared__ double tile[32][33];
  long long rs_base = (long long)blockIdx.x * 32;
  long long c_base = (long long)blockIdx.y * 32;
  int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int i = ty; i < 32; i += 8) {
    long long rs = rs_base + i;
    long long c = c_base + tx;
    tile[i][tx] = (rs < ntr && c < cnt) ? H[rs * ncol + c0 + c] : 0.0;
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    long long c = c_base + j;
    long long rs = rs_base + tx;
    if (c >= cnt || rs >= ntr) continue;
    // invert rs = r + s(s+1)/2, r <= s
    int s = (int)((sqrt(8.0 * (double)rs + 1.0) - 1.0) * 0.5);
    while ((long long)s * (s + 1) / 2 > rs) s--;
    while ((long long)(s + 1) * (s + 2) / 2 <= rs) s++;
    int r = (int)(rs - (long long)s * (s + 1) / 2);
    double v = tile[tx][j];
    double *Mc = M + c * (long long)n * n;
    Mc[r + (long long)s * n] = v;
    Mc[s + (long long)r * n] = v;
  }
}

// L (ntr x rank, column-major) -> rank column-major n x n matrices.
__global__ void unpack_factor(const double *__restrict__ L, long long ntr, int n, int P0, int cnt,
                              double *__restrict__ M) {
  long long total = (long long)cnt * n * n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int p = (int)(t % n);
    long long r = t / n;
    int q = (int)(r % n);
    long long P = r / n;
    long long pq = p <= q ? tri_pack(p, q) : tri_pack(q, p);
    M[t] = L[(P0 + P) * ntr + pq];
  }
}

// T[p + n (f + nf k)] = sum_q M_k(p, q) C[q + n f] in FP64 for symmetric n x n matrices given by
// their packed triangles (M_k at M + k ld, element (p, q), p <= q, at p + q (q + 1) / 2). A warp
// takes 32 rows p and FB columns f of one matrix. Bound by the FP64 pipe (64 cycles per warp
// instruction and quarter of an SM): the triangle is read in place, element by element, since
// even its uncoalesced half (q < p: a sector per lane, four q long) hides behind FB FMAs.
// Measured for the AOTWOSORT transform at n = 64, nocc = 10: 0.21 ms in two launches (85% of the
// pipe's rate); the whole call 2.28 -> 0.53 ms, of which DGEMM takes 0.30.
template <int FB>
__global__ void __launch_bounds__(128) k_half_fp64(int n, int cnt, int nf, int ngf,
                                                   const double *__restrict__ M, long long ld,
                                                   const double *__restrict__ C,
                                                   double *__restrict__ T) {
  const int lane = threadIdx.x & 31, nch = (n + 31) / 32;
  const long long items = (long long)cnt * nch * ngf;
  for (long long w = (blockIdx.x * 128ll + threadIdx.x) >> 5; w < items; w += gridDim.x * 4ll) {
    const int g = (int)(w % ngf), ch = (int)((w / ngf) % nch);
    const long long k = w / ((long long)ngf * nch);
    const int p = ch * 32 + lane, f0 = g * FB;
    const int pc = min(p, n - 1);  // lanes beyond n repeat the last row
    const double *__restrict__ m = M + k * ld;
    const double *__restrict__ row = m + (long long)pc * (pc + 1) / 2;
    const double *__restrict__ c[FB];
#pragma unroll
    for (int f = 0; f < FB; ++f) c[f] = C + (long long)min(f0 + f, nf - 1) * n;
    double acc[FB] = {};
#pragma unroll 4
    for (int q = 0; q < n; ++q) {
      const double v = q <= pc ? row[q] : m[pc + (long long)q * (q + 1) / 2];
#pragma unroll
      for (int f = 0; f < FB; ++f) acc[f] = fma(v, c[f][q], acc[f]);
    }
    if (p < n)
#pragma unroll
      for (int f = 0; f < FB; ++f)
        if (f0 + f < nf) T[p + n * (f0 + f + (long long)nf * k)] = acc[f];
  }
}

// out_k = CX^T M_k CY (nX x nY, column-major, consecutive) for cnt such matrices in FP64: the
// narrower block first (k_half_fp64), the other one by one DGEMM over all matrices (batched where
// the first block is CX).
int half_fp64(gc_context *ctx, int n, long long cnt, const double *M, int nX, const double *CX,
              int nY, const double *CY, double *out) {
  const bool y1 = nY <= nX;
  const int nf = y1 ? nY : nX;
  // at most 8 columns per thread, shared out evenly
  const int ngf = (nf + 7) / 8, fb = (nf + ngf - 1) / ngf;
  const long long ld = (long long)n * (n + 1) / 2;
  const int cs = (int)std::max<long long>(
      1, std::min<long long>({cnt, (long long)kChunkBytes / (8ll * n * nf), 0x7fffffffll / ((long long)n * nf)}));
  gc::DevBuf<double> T;
  GC_TRY(T.alloc(ctx, (size_t)cs * n * nf));
  const double one = 1.0, zero = 0.0;
  for (long long k0 = 0; k0 < cnt; k0 += cs) {
    const int c = (int)std::min<long long>(cs, cnt - k0);
    const long long items = (long long)c * ((n + 31) / 32) * ngf;
    const unsigned grid = (unsigned)std::min<long long>((items + 3) / 4, 152 * 256);
    const double *Mk = M + k0 * ld, *Cf = y1 ? CY : CX;
    auto go = [&](auto kern) { kern<<<grid, 128, 0, ctx->stream>>>(n, c, nf, ngf, Mk, ld, Cf, T.p); };
    switch (fb) {
      case 1: go(k_half_fp64<1>); break;
      case 2: go(k_half_fp64<2>); break;
      case 3: go(k_half_fp64<3>); break;
      case 4: go(k_half_fp64<4>); break;
      case 5: go(k_half_fp64<5>); break;
      case 6: go(k_half_fp64<6>); break;
      case 7: go(k_half_fp64<7>); break;
      default: go(k_half_fp64<8>);
    }
    GC_LAUNCHED(ctx);
    double *o = out + k0 * nX * nY;
    if (y1)
      GC_CUBLAS(ctx, cublasDgemm(ctx->cublas, CUBLAS_OP_T, CUBLAS_OP_N, nX, c * nY, n, &one, CX, n, T.p,
                                 n, &zero, o, nX));
    else
      GC_CUBLAS(ctx, cublasDgemmStridedBatched(ctx->cublas, CUBLAS_OP_T, CUBLAS_OP_N, nX, nY, n, &one,
                                               T.p, n, (long long)n * nX, CY, n, 0, &zero, o, nX,
                                               (long long)nX * nY, c));
  }
  return GC_OK;
}

int check_dims(gc_context *ctx, int nbas, int nA, int nB, int nC, int nD) {
  if (nbas <= 0 || nA <= 0 || nB <= 0 || nC <= 0 || nD <= 0 || nA > nbas || nB > nbas ||
      nC > nbas || nD > nbas)
    return gc::set_error(ctx, GC_EINVAL, "tran4: bad dimensions nbas=%d nA=%d nB=%d nC=%d nD=%d",
                         nbas, nA, nB, nC, nD);
  return GC_OK;
}

}  // namespace

extern "C" int gc_tran4_gen(gc_context *ctx, int nbas, int nA, const double *CA, int nB,
                            const double *CB, int nC, const double *CC, int nD, const double *CD,
                            const double *G, double *out, int precision) {
  if (!ctx) return GC_EINVAL;
  gc::PhaseScope ph(ctx, GC_PHASE_TRANSFORM);
  GC_TRY(check_dims(ctx, nbas, nA, nB, nC, nD));
  if (precision < GC_PREC_FP64 || precision > GC_PREC_FP64TC4)
    return gc::set_error(ctx, GC_EINVAL, "tran4_gen: unknown precision %d", precision);
  const int n = nbas;
  const long long ntr = (long long)n * (n + 1) / 2;
  const long long nAB = (long long)nA * nB, nCD = (long long)nC * nD;
  const long long n2 = (long long)n * n;
  gc::DevBuf<double> H, M, T1;
  GC_TRY(H.alloc(ctx, ntr * nAB));
  const bool sliced = gc::is_sliced(precision);
  if (sliced || precision == GC_PREC_FP64) {
    auto half = [&](int cnt, const double *packed, int nX, const double *CX, int nY, const double *CY,
                    double *o) -> int {
      if (!sliced) return half_fp64(ctx, n, cnt, packed, nX, CX, nY, CY, o);
      const gc::HalfOut h{nX, CX, nY, CY, o};
      return gc::tc_half_packed(ctx, precision, n, cnt, packed, ntr, 1, &h);
    };
    GC_TRY(half((int)ntr, G, nA, CA, nB, CB, H.p));
    const int cs = (int)std::max<long long>(1, std::min<long long>(nAB, kChunkBytes / (8 * ntr)));
    GC_TRY(M.alloc(ctx, (size_t)cs * ntr));
    for (long long c0 = 0; c0 < nAB; c0 += cs) {
      const int cnt = (int)std::min<long long>(cs, nAB - c0);
      transpose_columns<<<dim3(gc::ceil_div(ntr, 32), gc::ceil_div(cnt, 32)), dim3(32, 8), 0,
                          ctx->stream>>>(H.p, ntr, nAB, c0, cnt, M.p);
      GC_LAUNCHED(ctx);
      GC_TRY(half(cnt, M.p, nC, CC, nD, CD, out + c0 * nCD));
    }
    return sliced ? gc::check_flag(ctx) : GC_OK;
  }
  int cs = (int)std::max<long long>(1, std::min<long long>(ntr, kChunkBytes / (8 * n2)));
  GC_TRY(M.alloc(ctx, (size_t)cs * n2));
  int tmax = std::max(nA, nC);
  GC_TRY(T1.alloc(ctx, (size_t)cs * n * tmax));
  // phase 1: (ab| for every rs
  for (long long rs0 = 0; rs0 < ntr; rs0 += cs) {
    int cnt = (int)std::min<long long>(cs, ntr - rs0);
    unsigned grid = std::min<unsigned>(gc::ceil_div((size_t)cnt * n2, 256), 152u * 32u);
    unpack_records<<<grid, 256, 0, ctx->stream>>>(G, ntr, n, rs0, cnt, M.p);
    GC_LAUNCHED(ctx);
    GC_TRY(gc::tc_two_sided(ctx, precision, n, cnt, M.p, nA, CA, nB, CB, T1.p, H.p + rs0 * nAB, nAB));
  }
  // phase 2: |cd) for every ab
  for (long long c0 = 0; c0 < nAB; c0 += cs) {
    int cnt = (int)std::min<long long>(cs, nAB - c0);
    dim3 grid(gc::ceil_div(ntr, 32), gc::ceil_div(cnt, 32));
    unpack_columns<<<grid, dim3(32, 8), 0, ctx->stream>>>(H.p, ntr, nAB, n, c0, cnt, M.p);
    GC_LAUNCHED(ctx);
    GC_TRY(gc::tc_two_sided(ctx, precision, n, cnt, M.p, nC, CC, nD, CD, T1.p, out + c0 * nCD, nCD));
  }
  return gc::check_flag(ctx);
}

extern "C" int gc_tran4_factored(gc_context *ctx, int nbas, int rank, const double *L, int nA,
                                 const double *CA, int nB, const double *CB, int nC,
                                 const double *CC, int nD, const double *CD, double *out,
                                 int precision) {
  if (!ctx) return GC_EINVAL;
  gc::PhaseScope ph(ctx, GC_PHASE_TRANSFORM);
  GC_TRY(check_dims(ctx, nbas, nA, nB, nC, nD));
  if (rank <= 0) return gc::set_error(ctx, GC_EINVAL, "tran4_factored: rank=%d", rank);
  const int n = nbas;
  const long long ntr = (long long)n * (n + 1) / 2;
  const long long nAB = (long long)nA * nB, nCD = (long long)nC * nD;
  const long long n2 = (long long)n * n;
  const bool same = (CA == CC && CB == CD && nA == nC && nB == nD);
  gc::DevBuf<double> Y, Z, M, T1;
  GC_TRY(Y.alloc(ctx, nAB * rank));
  if (!same) GC_TRY(Z.alloc(ctx, nCD * rank));
  if (gc::is_sliced(precision)) {
    const bool symAB = CA == CB && nA == nB, symCD = CC == CD && nC == nD;
    const gc::HalfOut half[2] = {{nA, CA, nB, CB, Y.p, symAB}, {nC, CC, nD, CD, Z.p, symCD}};
    GC_TRY(gc::tc_half_packed(ctx, precision, n, rank, L, ntr, same ? 1 : 2, half));
    GC_TRY(gc::tc_pair_product(ctx, precision, rank, nC, nD, symCD, same ? Y.p : Z.p, nA, nB, symAB,
                               Y.p, out));
    return gc::check_flag(ctx);
  }
  int cs = (int)std::max<long long>(1, std::min<long long>(rank, kChunkBytes / (8 * n2)));
  if (precision == GC_PREC_FP64) {
    GC_TRY(half_fp64(ctx, n, rank, L, nA, CA, nB, CB, Y.p));
    if (!same) GC_TRY(half_fp64(ctx, n, rank, L, nC, CC, nD, CD, Z.p));
    cs = rank;
  } else {
    GC_TRY(M.alloc(ctx, (size_t)cs * n2));
    GC_TRY(T1.alloc(ctx, (size_t)cs * n * std::max(nA, nC)));
  }
  for (int P0 = 0; P0 < rank && precision != GC_PREC_FP64; P0 += cs) {
    int cnt = std::min(cs, rank - P0);
    unsigned grid = std::min<unsigned>(gc::ceil_div((size_t)cnt * n2, 256), 152u * 32u);
    unpack_factor<<<grid, 256, 0, ctx->stream>>>(L, ntr, n, P0, cnt, M.p);
    GC_LAUNCHED(ctx);
    GC_TRY(gc::tc_two_sided(ctx, precision, n, cnt, M.p, nA, CA, nB, CB, T1.p, Y.p + P0 * nAB, nAB));
    if (!same)
      GC_TRY(gc::tc_two_sided(ctx, precision, n, cnt, M.p, nC, CC, nD, CD, T1.p, Z.p + P0 * nCD, nCD));
  }
  // out (nCD x nAB, column-major == record-major) = Z . Y^T
  const double *Zp = same ? Y.p : Z.p;
  GC_TRY(gc::tc_gemm_nt(ctx, precision, (int)nCD, (int)nAB, rank, Zp, (int)nCD, Y.p, (int)nAB, out,
                        (int)nCD));
  return precision == GC_PREC_FP64 ? GC_OK : gc::check_flag(ctx);
}
