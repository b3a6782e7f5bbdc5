// AC0-CAS correlation energy, AC0CAS_FOFO (abfofo.f90:1485-1750).
//
// At lambda = 0 the ERPA matrices are block diagonal once the pairs are grouped
// (create_AC0_blocks_1/2, abfofo.f90:1374-1484): the active-active pairs, the
// (active, q) pairs of every inactive q, the (p, active) pairs of every virtual
// p, and the (virtual, inactive) pairs, whose block is diagonal. The AC0
// energy is first order in lambda:
//   C = Y [2 (X^T A+' X - Y^T A-' Y)_ij / (omega_i + omega_j)] Y^T,
//   ECorr = sum_{pq, rs not in one group} (C_p + C_q)(C_r + C_s) C[pq, rs] (rs|pq),
// with Y, X, omega the block-diagonal zeroth-order ERPA solution (ERPASYMM0,
// interpa.f:1496-1650, per block) and A+-' the AB1 matrices (the lambda
// derivative of A+-B, AB_CAS_FOFO with AB1 = .true.).
//
// Here the pair list is put in block order before the assembly, so that A+-B(0)
// and A+-' come out in block order directly (as ABPM0_FOFO assembles them) and
// every block is a contiguous square. Then:
//   k_ac0_block_erpa  one CTA per block: ERPASYMM0 in FP64 shared memory (two
//                     Jacobi eigensolves), Y, X and omega of the block;
//   k_ac0_iv          the (virtual, inactive) pairs: omega = A+(ii,ii), Y = X = 1/sqrt 2;
//   k_ac0_right       T+ = A+' Xbd, T- = A-' Ybd (block-diagonal right products);
//   k_ac0_weights     K: the masked, CI-weighted FOFO integrals, symmetrised;
//   k_ac0_right_k     TK = K Ybd;
//   k_ac0_work        the energy sum_{r<=c} of 2 (Xbd^T T+ - Ybd^T T-) / (omega_r + omega_c) times
//                     Ybd^T TK, one partial sum per block.
// Every pass is O(N^2 m) for blocks of size m (at most nact(nact-1)/2): there is
// no O(N^3) step, unlike the ERPA solves of the lambda quadrature.
#include <algorithm>
#include <cmath>
#include <vector>

#include "gc_internal.cuh"
#include "gc_math.cuh"

namespace {

constexpr int kMaxBlock = 64;  // largest block
constexpr int kRow = kMaxBlock;  // row stride of the block-diagonal factors Yrow / Xrow
const double kSmall = 1e-6;     // interpa.f:1511

constexpr int kBlkThreads = 256;

// Shared scratch of the block solve.
struct BlockSh {
  double red[2 * (kBlkThreads / 32)];
  double c[kMaxBlock], s[kMaxBlock];  // x_i' = c_i x_i + s_i x_w(i)
  int w[kMaxBlock];                   // the index that i is rotated with (i itself: none)
  int p[kMaxBlock / 2];               // pair k: p[k] < q = w[p[k]], or w[p[k]] = p[k]
};

// Jacobi (Golub and Van Loan, Alg. 8.5.3, and 8.5.6 for the parallel ordering) on the symmetric
// m x m matrix A (row stride ld >= m) in shared memory; V <- eigenvectors (columns), the
// eigenvalues are left on the diagonal of A; T is scratch of A's size. Returns false if 40
// sweeps did not bring the off-diagonal norm below 1e-30 of the total (uniform across the
// block).
//
// A chain of rotations is bound by the latency of each, and a warp's FP64 instruction occupies
// its quarter of the SM for 64 cycles however few of its lanes are live. So a sweep takes the
// m (m - 1) / 2 pairs as rounds of m / 2 disjoint pairs (round robin); one thread per pair
// forms its rotation with eight FP64 instructions; then every element of the upper triangle
// is one thread's (six instructions, from A into T and back in turn), and so is every pair of
// elements of V. A pair's element shrinks by the FP32 tangent's error only, which the second-order
// terms of the other pairs exceed.
// Measured for k_ac0_block_erpa with a 15 x 15 block (CAS(6,6), two eigensolves): one rotation
// at a time 2.67 ms, rounds with FP64 angles and one thread per 2 x 2 block 0.53 ms, this 0.27 ms.
__device__ bool block_jacobi(double *A, double *V, double *T, int m, int ld, BlockSh &sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = m + (m & 1), np = M / 2;
  const int wd = (m & 1) ? m : m + 1;  // folded triangle: row a beside row m - a or m - 1 - a
  double *src = A, *dst = T;
  for (int e = tid; e < m * m; e += kBlkThreads) {
    const int i = e / m, j = e - i * m;
    V[i * ld + j] = i == j ? 1.0 : 0.0;
  }
  for (int sweep = 0; sweep < 40; ++sweep) {
    __syncthreads();
    double off = 0.0, tot = 0.0;
    for (int e = tid; e < m * m; e += kBlkThreads) {
      const int i = e / m, j = e - i * m;
      const double v = src[i * ld + j] * src[i * ld + j];
      tot += v;
      if (i != j) off += v;
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_down_sync(0xffffffffu, off, o);
      tot += __shfl_down_sync(0xffffffffu, tot, o);
    }
    if (lane == 0) {
      sh.red[2 * warp] = off;
      sh.red[2 * warp + 1] = tot;
    }
    __syncthreads();
    off = tot = 0.0;
    for (int w = 0; w < kBlkThreads / 32; ++w) {
      off += sh.red[2 * w];
      tot += sh.red[2 * w + 1];
    }
    if (off <= 1e-30 * tot) {  // uniform: every thread added the same values
      if (src != A) {
        for (int e = tid; e < m * m; e += kBlkThreads) {
          const int i = e / m, j = e - i * m;
          A[i * ld + j] = src[i * ld + j];
        }
        __syncthreads();
      }
      return true;
    }
    for (int k = 0; k < M - 1; ++k) {
      if (tid < np) {
        const int x = tid == 0 ? M - 1 : (k + tid) % (M - 1);
        const int y = tid == 0 ? k : (k - tid + M - 1) % (M - 1);
        const int p = min(x, y), q = max(x, y);
        double c = 1.0, sn = 0.0;
        if (q < m) {
          const double h = src[p * ld + q], d = src[q * ld + q] - src[p * ld + p];
          if ((__double_as_longlong(h) << 1) != 0) gc::jacobi_rotation(h, d, &c, &sn);
          sh.w[q] = p;
          sh.c[q] = c;
          sh.s[q] = sn;
        }
        sh.w[p] = q < m ? q : p;
        sh.c[p] = c;
        sh.s[p] = -sn;
        sh.p[tid] = p;
      }
      __syncthreads();
      for (int e = tid; e < (m + 1) / 2 * wd; e += kBlkThreads) {
        const int a = e / wd, b = e - a * wd;
        const bool first = b < m - a;
        const int i = first ? a : ((m & 1) ? m - a : m - 1 - a), j = first ? a + b : i + b - (m - a);
        if (j >= m) continue;
        const int iw = sh.w[i], jw = sh.w[j];
        const double ci = sh.c[i], si = sh.s[i], cj = sh.c[j], sj = sh.s[j];
        const double x = cj * src[i * ld + j] + sj * src[i * ld + jw];
        const double y = cj * src[iw * ld + j] + sj * src[iw * ld + jw];
        const double v = ci * x + si * y;
        dst[i * ld + j] = v;
        dst[j * ld + i] = v;
      }
      for (int e = kBlkThreads - 1 - tid; e < m * np; e += kBlkThreads) {
        const int i = e / np, r = sh.p[e - i * np], u = sh.w[r];
        if (u == r) continue;
        const double x = V[i * ld + r], y = V[i * ld + u];
        V[i * ld + r] = sh.c[r] * x + sh.s[r] * y;
        V[i * ld + u] = sh.c[u] * y + sh.s[u] * x;
      }
      __syncthreads();
      double *t = src;
      src = dst;
      dst = t;
    }
  }
  return false;
}

// A = L L^T (lower, zero above) of the symmetric m x m matrix A, in place, right-looking; false,
// with A half done, at the first pivot that is not positive (uniform across the block).
__device__ bool block_cholesky(double *A, int m, int ld) {
  for (int k = 0; k < m; ++k) {
    const double d = A[k * ld + k];  // every thread reads the same pivot
    if (!(d > 0.0)) return false;
    const double r = rsqrt(d);
    __syncthreads();
    for (int i = k + threadIdx.x; i < m; i += kBlkThreads) A[i * ld + k] *= r;
    __syncthreads();
    const int w = m - k - 1;
    for (int e = threadIdx.x; e < w * w; e += kBlkThreads) {
      const int i = k + 1 + e / w, j = k + 1 + e % w;
      if (j <= i) A[i * ld + j] -= A[i * ld + k] * A[j * ld + k];
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < m * m; e += kBlkThreads)
    if (e % m > e / m) A[(e / m) * ld + e % m] = 0.0;
  __syncthreads();
  return true;
}

// ERPASYMM0 of every block (one CTA each): block b covers the block-order positions
// bstart[b] .. bstart[b] + bsize[b] - 1 of the column-major N x N matrices ap, am (A+-B at
// lambda = 0). Writes Yrow/Xrow[(s + i) * kRow + c] = Y/X(i, c) of the block and eig[s + c]; a
// Jacobi that does not converge sets *flag. The largest block (active-active pairs) sets
// the time: its eigensolves are a chain of rotations. A positive definite A+ is factored, L
// takes the place of A+^1/2 (L^T A- L has the eigenvalues of A+^1/2 A- A+^1/2, and L u is the
// same mode), and one of the two eigensolves falls away: 149 us for CAS(6,6), 270 with two.
__global__ void __launch_bounds__(kBlkThreads) k_ac0_block_erpa(
    int N, const double *__restrict__ ap, const double *__restrict__ am,
    const int *__restrict__ bstart, const int *__restrict__ bsize, int rows, int ld,
    double *__restrict__ Yrow, double *__restrict__ Xrow, double *__restrict__ eig, int *flag) {
  extern __shared__ double sm[];
  __shared__ BlockSh sh;
  __shared__ double w2[kMaxBlock];
  const int s = bstart[blockIdx.x], m = bsize[blockIdx.x], tid = threadIdx.x;
  const size_t sz = (size_t)rows * ld;
  double *A = sm, *B = A + sz, *P = B + sz, *H = P + sz, *V = H + sz;
  auto each = [&](auto f) {  // f(i, j) over the m x m elements
    for (int e = tid; e < m * m; e += kBlkThreads) f(e / m, e % m);
    __syncthreads();
  };
  auto dot = [&](const double *x, int sx, const double *y, int sy) {
    double v = 0.0;
    for (int k = 0; k < m; ++k) v += x[k * sx] * y[k * sy];
    return v;
  };
  // symmetrised blocks (interpa.f:1532-1540)
  each([&](int j, int i) {  // i fastest: consecutive threads read consecutive rows
    const size_t e = (size_t)(s + i) + (size_t)(s + j) * N, t = (size_t)(s + j) + (size_t)(s + i) * N;
    A[i * ld + j] = 0.5 * (ap[e] + ap[t]);
    B[i * ld + j] = 0.5 * (am[e] + am[t]);
  });
  each([&](int i, int j) { P[i * ld + j] = A[i * ld + j]; });
  if (!block_cholesky(P, m, ld)) {
    if (!block_jacobi(A, V, H, m, ld, sh)) {
      if (tid == 0) atomicOr(flag, 1);
      return;  // uniform
    }
    if (tid < m) w2[tid] = sqrt(fabs(A[tid * ld + tid]));
    __syncthreads();
    // P = V diag(sqrt|e|) V^T = A+^1/2 (interpa.f:1546-1568)
    each([&](int i, int j) {
      double v = 0.0;
      for (int k = 0; k < m; ++k) v += V[i * ld + k] * w2[k] * V[j * ld + k];
      P[i * ld + j] = v;
    });
  }
  // H = A- P, then A <- P^T H (the symmetrised problem, interpa.f:1578-1581)
  each([&](int i, int j) { H[i * ld + j] = dot(B + i * ld, 1, P + j, ld); });
  each([&](int i, int j) {  // the lower triangle, as the eigensolver reads it
    if (i >= j) A[i * ld + j] = A[j * ld + i] = dot(P + i, ld, H + j, ld);
  });
  if (!block_jacobi(A, V, H, m, ld, sh)) {
    if (tid == 0) atomicOr(flag, 1);
    return;
  }
  if (tid < m) w2[tid] = A[tid * ld + tid];
  // Y = P Z into H, A- Y into A
  each([&](int i, int j) { H[i * ld + j] = dot(P + i * ld, 1, V + j, ld); });
  each([&](int i, int j) { A[i * ld + j] = dot(B + i * ld, 1, H + j, ld); });
  // mode nu: normalise 2/omega y^T A- y = 1, X = A- y / omega (interpa.f:1598-1648)
  if (tid < m) {
    const int nu = tid;
    double om = w2[nu], f = 0.0, g = 0.0;
    if (om > kSmall) {
      om = sqrt(om);
      const double sum = 2.0 / om * dot(H + nu, ld, A + nu, ld);
      f = sum > 0.0 ? 1.0 / sqrt(sum) : 0.0;
      g = f / om;
    }
    for (int i = 0; i < m; ++i) {
      Yrow[(size_t)(s + i) * kRow + nu] = f * H[i * ld + nu];
      Xrow[(size_t)(s + i) * kRow + nu] = g * A[i * ld + nu];
    }
    eig[s + nu] = om;  // omega, or omega^2 where omega^2 <= Small
  }
}

// (virtual, inactive) pairs, positions iv0..N-1: omega = A+(ii,ii), Y = X = 1/sqrt 2
// (AC0CAS_FOFO, abfofo.f90:1600-1614; the 1/sqrt 2 factor of abpm_tran, tran.f90:634).
__global__ void k_ac0_iv(int N, int iv0, const double *__restrict__ ap, double *__restrict__ Yrow,
                         double *__restrict__ Xrow, double *__restrict__ eig) {
  const int i = iv0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double fac = 1.0 / sqrt(2.0);
  eig[i] = ap[(size_t)i + (size_t)i * N];
  Yrow[(size_t)i * kRow] = fac;
  Xrow[(size_t)i * kRow] = fac;
}

// T+ = A+' Xbd and T- = A-' Ybd with the block-diagonal Xbd, Ybd (the sum over k in the block of
// c, positions bs[c] .. bs[c] + bz[c] - 1). The rows up to the end of c's block are all that
// k_ac0_work reads. Threads along r: coalesced columns.
__global__ void k_ac0_right(int N, const double *__restrict__ a1p, const double *__restrict__ a1m,
                            const int *__restrict__ bs, const int *__restrict__ bz,
                            const double *__restrict__ Xrow, const double *__restrict__ Yrow,
                            double *__restrict__ tp, double *__restrict__ tm) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  for (int c = blockIdx.y; c < N; c += gridDim.y) {
    const int s = bs[c], m = bz[c], cc = c - s;
    if (r >= s + m) continue;
    double vp = 0.0, vm = 0.0;
    for (int b = 0; b < m; ++b) {
      const size_t e = (size_t)r + (size_t)(s + b) * N;
      vp += a1p[e] * Xrow[(size_t)(s + b) * kRow + cc];
      vm += a1m[e] * Yrow[(size_t)(s + b) * kRow + cc];
    }
    const size_t o = (size_t)r + (size_t)c * N;
    tp[o] = vp;
    tm[o] = vm;
  }
}

// K = (K0 + K0^T) / 2 of the energy's weights K0[r, k] = (C_p + C_q)(C_r' + C_s') (r's'|pq) for
// pairs r = (p, q), k = (r', s') not in one orbital group: the energy sums over all r, k with a
// symmetric factor, so both of (r's'|pq) and (pq|r's') enter, which may differ (FOFO blocks are
// symmetric to the rounding of their transform). One block per 32 x 32 tile of the lower triangle; its
// mirror tile is gathered with the same coalescing and turned in shared memory, and both are
// stored. K is formed once, where it was gathered again for every column of a block, and takes the
// place of A+', as TK then takes that of A-': four N x N matrices are held.
__global__ void __launch_bounds__(256)
    k_ac0_weights(int N, int n, int nocc, const int *__restrict__ pp, const int *__restrict__ pq,
                  const double *__restrict__ cpl, const int *__restrict__ grp,
                  const double *__restrict__ fofo, double *__restrict__ kw) {
  __shared__ double mirror[32][33], turned[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const size_t ld = (size_t)n * nocc;
  auto el = [&](int i, int j) -> double {
    const int p = pp[i], q = pq[i], r = pp[j], s = pq[j];
    if (grp[p] == grp[q] && grp[q] == grp[r] && grp[r] == grp[s]) return 0.0;
    return cpl[i] * cpl[j] * fofo[((size_t)r + (size_t)s * n) * ld + p + (size_t)q * n];
  };
  const int nt = (N + 31) / 32, i0 = blockIdx.x * 32;
  for (int tj = blockIdx.y; tj <= (int)blockIdx.x && tj < nt; tj += gridDim.y) {
    const int j0 = tj * 32;
    __syncthreads();  // the tiles of the last turn
    for (int k = ty; k < 32; k += 8) {
      const int i = j0 + tx, j = i0 + k;
      mirror[k][tx] = i < N && j < N ? el(i, j) : 0.0;
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
      const int i = i0 + tx, j = j0 + k;
      const double v = i < N && j < N ? 0.5 * (el(i, j) + mirror[tx][k]) : 0.0;
      if (i < N && j < N) kw[i + (size_t)j * N] = v;
      turned[k][tx] = v;
    }
    __syncthreads();
    if (i0 != j0)
      for (int k = ty; k < 32; k += 8) {
        const int i = j0 + tx, j = i0 + k;
        if (i < N && j < N) kw[i + (size_t)j * N] = turned[tx][k];
      }
  }
}

// TK = K Ybd, the rows of k_ac0_right.
__global__ void k_ac0_right_k(int N, const double *__restrict__ kw, const int *__restrict__ bs,
                              const int *__restrict__ bz, const double *__restrict__ Yrow,
                              double *__restrict__ tk) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  for (int c = blockIdx.y; c < N; c += gridDim.y) {
    const int s = bs[c], m = bz[c], cc = c - s;
    if (r >= s + m) continue;
    double v = 0.0;
    for (int b = 0; b < m; ++b)
      v += kw[(size_t)r + (size_t)(s + b) * N] * Yrow[(size_t)(s + b) * kRow + cc];
    tk[(size_t)r + (size_t)c * N] = v;
  }
}

// The energy sum_{r,c} work[r, c] (Ybd^T K Ybd)[r, c] with
// work[r, c] = 2 ((Xbd^T T+)[r, c] - (Ybd^T T-)[r, c]) / (omega_r + omega_c) where both
// omegas are nonzero, else 0 (AC0CAS_FOFO, abfofo.f90:1625-1720, with the back-transform Ybd work
// Ybd^T moved to the symmetric weights). Both factors are symmetric: r <= c, the others counted
// twice. One partial sum per block. Measured at NDimX 1832 (n = 120, CAS(6,6)): k_ac0_right 25 us,
// k_ac0_weights 27, k_ac0_right_k 16, this 137, where the products, the back-transform and the energy loop
// over all r, c took 280.
__global__ void __launch_bounds__(256)
    k_ac0_work(int N, const double *__restrict__ tp, const double *__restrict__ tm,
               const double *__restrict__ tk, const int *__restrict__ bs, const int *__restrict__ bz,
               const double *__restrict__ Xrow, const double *__restrict__ Yrow,
               const double *__restrict__ eig, double *__restrict__ part) {
  __shared__ double red[256];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (r < N) {
    const double er = eig[r];
    const int s = bs[r], m = bz[r], rr = r - s;
    for (int c = blockIdx.y; c < N; c += gridDim.y) {
      const double ec = eig[c];
      if (c < r || er == 0.0 || ec == 0.0) continue;
      double xp = 0.0, ym = 0.0, yk = 0.0;
      for (int b = 0; b < m; ++b) {
        const size_t t = (size_t)(s + b) + (size_t)c * N;
        const double y = Yrow[(size_t)(s + b) * kRow + rr];
        xp += Xrow[(size_t)(s + b) * kRow + rr] * tp[t];
        ym += y * tm[t];
        yk += y * tk[t];
      }
      e += (r == c ? 2.0 : 4.0) * (xp - ym) * yk / (er + ec);
    }
  }
  red[threadIdx.x] = e;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x + (size_t)gridDim.x * blockIdx.y] = red[0];
}

// out[0] = sum of part[0 .. cnt) (one block, fixed order).
__global__ void k_sum(size_t cnt, const double *__restrict__ part, double *__restrict__ out) {
  __shared__ double red[1024];
  double s = 0.0;
  for (size_t i = threadIdx.x; i < cnt; i += blockDim.x) s += part[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

}  // namespace

extern "C" int gc_ac0cas_fofo(gc_context *ctx, int nbas, int ninact, int nact, int ndimx,
                              const double *occ, const double *ure, const double *xone,
                              const int *indn, const double *rdm2act, const double *ffoo,
                              const double *fofo, double *ecorr, double *etot) {
  if (!ctx) return GC_EINVAL;
  if (!occ || !xone || !indn || !ffoo || !fofo || !ecorr || ndimx <= 0 || nbas <= 0 ||
      ninact < 0 || nact < 0 || ninact + nact > nbas)
    return gc::set_error(ctx, GC_EINVAL, "ac0cas_fofo: bad arguments");
  const int n = nbas, nocc = ninact + nact, N = ndimx;
  // Block order of the pairs (create_AC0_blocks_1/2): AA, AI for q = 1..nin, AV for
  // p = nocc+1..n, then the (virtual, inactive) pairs.
  auto grp = [&](int i) { return i < ninact ? 0 : (i < nocc ? 1 : 2); };
  std::vector<int> aa, iv;
  std::vector<std::vector<int>> ai(ninact), av(n > nocc ? n - nocc : 0);
  for (int i = 0; i < N; ++i) {
    const int p = indn[2 * i] - 1, q = indn[2 * i + 1] - 1;
    if (p <= q || p >= n || q < 0 || q >= nocc)
      return gc::set_error(ctx, GC_EINVAL, "ac0cas_fofo: pair %d = (%d,%d) is not valid", i + 1,
                           p + 1, q + 1);
    const int gp = grp(p), gq = grp(q);
    if (gp == 1 && gq == 1) aa.push_back(i);
    else if (gp == 1 && gq == 0) ai[q].push_back(i);
    else if (gp == 2 && gq == 1) av[p - nocc].push_back(i);
    else if (gp == 2 && gq == 0) iv.push_back(i);
    else
      return gc::set_error(ctx, GC_EINVAL, "ac0cas_fofo: pair (%d,%d) in no AC0 block", p + 1, q + 1);
  }
  std::vector<int> order, bstart, bsize, pos_s(N), pos_m(N);
  auto add_block = [&](const std::vector<int> &b) {
    if (b.empty()) return;
    bstart.push_back((int)order.size());
    bsize.push_back((int)b.size());
    for (int i : b) order.push_back(i);
  };
  add_block(aa);
  for (auto &b : ai) add_block(b);
  for (auto &b : av) add_block(b);
  const int iv0 = (int)order.size();
  for (int i : iv) order.push_back(i);
  int mmax = 1;
  for (size_t b = 0; b < bstart.size(); ++b) {
    mmax = std::max(mmax, bsize[b]);
    for (int k = 0; k < bsize[b]; ++k) {
      pos_s[bstart[b] + k] = bstart[b];
      pos_m[bstart[b] + k] = bsize[b];
    }
  }
  for (int k = iv0; k < N; ++k) {
    pos_s[k] = k;
    pos_m[k] = 1;
  }
  if (mmax > kMaxBlock)
    return gc::set_error(ctx, GC_EUNSUPPORTED, "ac0cas_fofo: an AC0 block of %d pairs (limit %d)",
                         mmax, kMaxBlock);
  std::vector<int> indn_blk(2 * (size_t)N);
  for (int k = 0; k < N; ++k) {
    indn_blk[2 * k] = indn[2 * order[k]];
    indn_blk[2 * k + 1] = indn[2 * order[k] + 1];
  }
  // A+-B(0) and the AB1 matrices, assembled in block order
  gc::SysDev sd;
  GC_TRY(gc::sys_upload(ctx, sd, n, ninact, nact, N, occ, xone, indn_blk.data(), rdm2act));
  if (ure) GC_TRY(gc::rotate_h(ctx, sd, ure));
  const size_t NN = (size_t)N * N;
  gc::DevBuf<double> a0p, a0m, a1p, a1m, Yrow, Xrow, eig;
  GC_TRY(a0p.alloc(ctx, NN));
  GC_TRY(a0m.alloc(ctx, NN));
  GC_TRY(a1p.alloc(ctx, NN));
  GC_TRY(a1m.alloc(ctx, NN));
  GC_TRY(gc::assemble_ab_pair(ctx, sd, ffoo, fofo, {{0.0, 0, a0p.p, a0m.p}, {1.0, 1, a1p.p, a1m.p}}, etot));
  GC_TRY(Yrow.alloc(ctx, (size_t)N * kRow));
  GC_TRY(Xrow.alloc(ctx, (size_t)N * kRow));
  GC_TRY(eig.alloc(ctx, N));
  GC_CUDA(ctx, cudaMemsetAsync(Yrow.p, 0, (size_t)N * kRow * sizeof(double), ctx->stream));
  GC_CUDA(ctx, cudaMemsetAsync(Xrow.p, 0, (size_t)N * kRow * sizeof(double), ctx->stream));
  gc::DevBuf<int> dbs, dbz, pbs, pbz, flag;
  const int nblk = (int)bstart.size();
  if (nblk > 0) {
    GC_TRY(dbs.upload(ctx, bstart.data(), nblk));
    GC_TRY(dbz.upload(ctx, bsize.data(), nblk));
  }
  GC_TRY(pbs.upload(ctx, pos_s.data(), N));
  GC_TRY(pbz.upload(ctx, pos_m.data(), N));
  GC_TRY(flag.alloc(ctx, 1));
  GC_CUDA(ctx, cudaMemsetAsync(flag.p, 0, sizeof(int), ctx->stream));
  if (nblk > 0) {
    const int ld = mmax + 1;
    const size_t smem = 5 * (size_t)mmax * ld * sizeof(double);
    // always the largest block's: a smaller limit could come between this and another thread's launch
    constexpr int kMaxSmem = 5 * kMaxBlock * (kMaxBlock + 1) * (int)sizeof(double);
    GC_CUDA(ctx, cudaFuncSetAttribute(k_ac0_block_erpa, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kMaxSmem));
    k_ac0_block_erpa<<<nblk, kBlkThreads, smem, ctx->stream>>>(
        N, a0p.p, a0m.p, dbs.p, dbz.p, mmax, ld, Yrow.p, Xrow.p, eig.p, flag.p);
    GC_LAUNCHED(ctx);
  }
  if (iv0 < N) {
    k_ac0_iv<<<gc::ceil_div(N - iv0, 256), 256, 0, ctx->stream>>>(N, iv0, a0p.p, Yrow.p, Xrow.p,
                                                                 eig.p);
    GC_LAUNCHED(ctx);
  }
  // Products with the block-diagonal factors; T+ and T- go into a0p and a0m, then K into a1p and TK
  // into a1m.
  gc::DevBuf<double> part, res;
  const dim3 gr(gc::ceil_div(N, 256), std::min(N, 65535));
  k_ac0_right<<<gr, 256, 0, ctx->stream>>>(N, a1p.p, a1m.p, pbs.p, pbz.p, Xrow.p, Yrow.p, a0p.p, a0m.p);
  GC_LAUNCHED(ctx);
  double *kw = a1p.p, *tk = a1m.p;
  const unsigned nt = gc::ceil_div(N, 32);
  k_ac0_weights<<<dim3(nt, std::min(nt, 65535u)), 256, 0, ctx->stream>>>(
      N, n, nocc, sd.pair_p.p, sd.pair_q.p, sd.cpl.p, sd.grp.p, fofo, kw);
  GC_LAUNCHED(ctx);
  k_ac0_right_k<<<gr, 256, 0, ctx->stream>>>(N, kw, pbs.p, pbz.p, Yrow.p, tk);
  GC_LAUNCHED(ctx);
  const unsigned gy = (unsigned)std::min(N, 256);
  const size_t npart = (size_t)gc::ceil_div(N, 256) * gy;
  GC_TRY(part.alloc(ctx, npart));
  GC_TRY(res.alloc(ctx, 1));
  k_ac0_work<<<dim3(gc::ceil_div(N, 256), gy), 256, 0, ctx->stream>>>(
      N, a0p.p, a0m.p, tk, pbs.p, pbz.p, Xrow.p, Yrow.p, eig.p, part.p);
  GC_LAUNCHED(ctx);
  k_sum<<<1, 1024, 0, ctx->stream>>>(npart, part.p, res.p);
  GC_LAUNCHED(ctx);
  int hflag = 0;
  GC_CUDA(ctx, cudaMemcpyAsync(ecorr, res.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaMemcpyAsync(&hflag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (hflag)
    return gc::set_error(ctx, GC_ECUSOLVER, "ac0cas_fofo: a block eigensolve did not converge");
  if (!std::isfinite(*ecorr))
    return gc::set_error(ctx, GC_ENONFINITE, "ac0cas_fofo: the energy is not finite");
  return GC_OK;
}
