// Split-precision tensor-core GEMM on tcgen05 (sm_103a).
//
//   C[m, n] = sum_pass sum_k A_pa(pass)[m, k] * B_pb(pass)[n, k]
//
// FP64 operands are split into BF16 planes x = x0 + x1 (+ x2) by pack_planes;
// a pass list selects the plane products that are kept (3 passes for
// hi*hi + hi*lo + lo*hi, 6 passes with a third plane, which brings the
// product error to the FP32 level). All passes accumulate into one FP32
// accumulator in tensor memory.
//
// Kernel structure (one CTA per 128 x BN output tile, 192 threads):
//   warp 0  TMA producer: 64-wide K slices of A and B into a STAGES-deep
//           shared-memory ring (128B swizzle), completion on mbarriers;
//   warp 1  allocates TMEM, one elected thread issues tcgen05.mma
//           (M=128, N=BN, K=16) and tcgen05.commit to release ring slots;
//   warps 2-5 epilogue: tcgen05.ld of the accumulator, then either a FP64
//           store or a fused dot product with an FP64 matrix (integrand).
// Every pipeline wait is bounded by the context's limit (1 s unless a test
// shortens it). On expiry the CTA records an error in a device flag and stops
// issuing work; before it frees TMEM and exits, the producer waits for the TMA
// copies it issued and the MMA thread commits the MMAs it issued and waits for
// them, both under their own fixed 1 s limit.
#include <cuda.h>
#include <cuda_bf16.h>

#include <memory>
#include <mutex>

#include "gc_tc_gemm.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // bf16 elements per K slice = one 128-byte swizzle row
constexpr int STAGES = 4;
constexpr int MAXPASS = 8;
constexpr unsigned long long kDrainNs = 1000000000ull;  // limit of the waits of the abort path

struct PassList {
  int n;
  int pa[MAXPASS];
  int pb[MAXPASS];
};

struct Epi {
  int mode;             // 0: store C (FP64); 1: partial[cta] = sum C .* R
  double *c;            // mode 0 output
  long long ldn;        // element (m, n) at c[b*sb + m + n*ldn]
  long long sb;
  const double *r;      // mode 1 matrix, same indexing
  double *partial;      // mode 1: one double per CTA
};

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(addr), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded parity wait: returns false if the phase did not complete within limit_ns.
// try_wait itself suspends the thread for a while, so the timer is read once per
// unsuccessful attempt (never when the first attempt succeeds).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          unsigned long long limit_ns) {
  const uint32_t addr = smem_u32(bar);
  if (mbar_try(addr, parity)) return true;
  const unsigned long long t0 = globaltimer();
  for (;;) {
    if (mbar_try(addr, parity)) return true;
    if (globaltimer() - t0 > limit_ns) return false;
  }
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0,
                                            int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Shared-memory matrix descriptor: K-major tile, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), version 1 (bits 46-47), layout SWIZZLE_128B (bits 61-63 = 2).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;            // LBO (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // SBO
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}

// As smem_desc for 64-byte rows (32 BF16 of K) in the 64-byte swizzle: 8-row groups
// 512 bytes apart, layout SWIZZLE_64B (bits 61-63 = 4).
__device__ __forceinline__ uint64_t smem_desc64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;           // LBO (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;  // SBO
  d |= (uint64_t)1 << 46;           // descriptor version
  d |= (uint64_t)4 << 61;           // SWIZZLE_64B
  return d;
}

// Instruction descriptor, kind::f16: D=F32, A=B=BF16, both K-major, M=128, N=bn.
__host__ __device__ constexpr uint32_t instr_desc(int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) |
         ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
}

// As mma_bf16, with a use of the A collector buffer: C = 1 reads A from shared memory
// and keeps it in the buffer, 2 reads the buffer, 3 reads it and releases it, 0 discards it (the
// plain form). The same A descriptor is given with every use.
template <int C>
__device__ __forceinline__ void mma_bf16_ca(uint32_t tmem, uint64_t ad, uint64_t bd,
                                            uint32_t idesc, uint32_t accumulate) {
  if constexpr (C == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
  else if constexpr (C == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16.collector::a::use [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
  else if constexpr (C == 3)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
  else
    mma_bf16(tmem, ad, bd, idesc, accumulate);
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 8 columns of 32-bit TMEM words, issued without waiting (several loads
// can be in flight before one tmem_ld_wait()).
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld4_issue(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One lane of a converged warp, the same one every time.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok));
  return ok != 0;
}

// ------------------------------------------------------------------- kernel
template <int BN>
__global__ void __launch_bounds__(192, 1)
    k_tc_gemm(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
              int M, int N, int kblocks, int a_batched, int b_batched, PassList passes, Epi epi,
              int *err_flag, unsigned long long wait_ns) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
  uint8_t *sA = smem;
  uint8_t *sB = smem + STAGES * A_BYTES;
  uint64_t *full = (uint64_t *)(sB + STAGES * B_BYTES);
  uint64_t *empty = full + STAGES;
  uint64_t *accf = empty + STAGES;
  uint32_t *tmem_slot = (uint32_t *)(accf + 1);
  __shared__ int abort_flag;
  volatile int *abort_v = &abort_flag;
  __shared__ double red[4];

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN, b = blockIdx.z;
  const int total = passes.n * kblocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accf, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer
    int issued = 0;
    for (int it = 0; it < total; ++it) {
      int s = it % STAGES;
      uint32_t ph = (it / STAGES) & 1;
      if (!mbar_wait(&empty[s], ph ^ 1, wait_ns)) {
        atomicExch(&abort_flag, 1);
        break;
      }
      if (*abort_v) break;
      int pass = it / kblocks, kb = it % kblocks;
      mbar_expect_tx(&full[s], A_BYTES + B_BYTES);
      tma_load_4d(sA + s * A_BYTES, &mapA, &full[s], kb * BK, m0, a_batched ? b : 0,
                  passes.pa[pass]);
      tma_load_4d(sB + s * B_BYTES, &mapB, &full[s], kb * BK, n0, b_batched ? b : 0,
                  passes.pb[pass]);
      issued = it + 1;
    }
    if (*abort_v) {
      // Drain the copies already issued into the ring before the CTA exits. Loads older
      // than the last STAGES were consumed by the MMA thread (their slot was released
      // before it was reused), so only the last STAGES can still be in flight.
      for (int it = (issued > STAGES ? issued - STAGES : 0); it < issued; ++it)
        mbar_wait(&full[it % STAGES], (it / STAGES) & 1, kDrainNs);
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    constexpr uint32_t idesc = instr_desc(BN);
    bool ok = true;
    for (int it = 0; it < total && ok; ++it) {
      int s = it % STAGES;
      uint32_t ph = (it / STAGES) & 1;
      if (!mbar_wait(&full[s], ph, wait_ns) || *abort_v) {
        atomicExch(&abort_flag, 1);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t a_addr = smem_u32(sA + s * A_BYTES), b_addr = smem_u32(sB + s * B_BYTES);
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) {
        uint64_t ad = smem_desc(a_addr + kk * 32), bd = smem_desc(b_addr + kk * 32);
        mma_bf16(tmem, ad, bd, idesc, (it > 0 || kk > 0) ? 1u : 0u);
      }
      mma_commit(&empty[s]);
    }
    mma_commit(accf);  // arrives once all issued MMAs have completed
    // TMEM is freed after the final barrier: wait here for every MMA this thread
    // issued, whatever the epilogue saw (on the abort path it may have given up).
    if (!mbar_wait(accf, 0, kDrainNs)) atomicExch(&abort_flag, 1);
  } else if (warp >= 2) {
    // ---------------- epilogue
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    const int m = m0 + q * 32 + lane;
    bool ok = mbar_wait(accf, 0, wait_ns);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    double acc = 0.0;
    if (ok && !*abort_v) {
      for (int c0 = 0; c0 < BN; c0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
        if (m < M) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            int n = n0 + c0 + j;
            if (n < N) {
              long long o = (long long)b * epi.sb + m + (long long)n * epi.ldn;
              if (epi.mode == 0)
                epi.c[o] = (double)v[j];
              else
                acc += (double)v[j] * epi.r[o];
            }
          }
        }
      }
    } else {
      atomicExch(&abort_flag, 1);
    }
    if (epi.mode == 1) {
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
      if (lane == 0) red[warp - 2] = acc;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (epi.mode == 1 && threadIdx.x == 0) {
    long long cta = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
    epi.partial[cta] = red[0] + red[1] + red[2] + red[3];
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(err_flag, 1);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)BN));
  }
}

// ------------------------------------------------ FP64-accurate (sliced) GEMM
// Each row r of A is scaled by 2^-e_r (e_r: exponent of its largest entry) and
// cut into S integer slices a = sum_t alpha_t 2^-7(t+1), |alpha_0| <= 128,
// |alpha_t>0| <= 64, every alpha exact in BF16; likewise the rows of B with f_c.
// C[r,c] = 2^(e_r+f_c) sum_{t+u<S} 2^-7(t+u+2) sum_k alpha_t[r,k] beta_u[c,k].
// The products of one weight d = t+u share a TMEM accumulator; K is cut into
// chunks short enough that every FP32 partial sum is an integer below 2^24, so
// each chunk is exact, and the epilogue adds the chunks in int64 registers.
// Column tile (TBN rows of B): the S weight accumulators take S * TBN of the 512 TMEM
// columns, so TBN = 128 for S = 4, 96 for S = 5 and 64 for S = 6 at most (half of them where two
// CTAs share an SM: 48 for S <= 5, 32). A wider
// tile reads fewer operand bytes per product (shared memory and L2); a narrower
// one gives more CTAs to a small product. oz_tile() picks one per GEMM; every
// width gives the same result bits (each element's integer sums are the same).
constexpr int OZ_BK = 32;      // K per stage: 32 BF16 = one 64-byte swizzled row
// Each stage holds every slice of A and of B. The 32- and 48-wide tiles of 4 and 5 slices (the
// occupied block of a transform; products with a short K) take two, so that two CTAs share an SM and
// one's epilogue runs beside the other's products (372006 x 28 x 249, 5 slices: 177 us, with the
// 64-wide tile 268). Two CTAs of six slices do not fit an SM's shared memory, so they take
// three stages (372006 x 28 x 249: 255 us, with two 266, with the 64-wide tile 308; x 512: 416, 561,
// 499).
__host__ __device__ constexpr int oz_ctas(int S, int tbn) { return S < 6 && tbn < 64 ? 2 : 1; }
__host__ __device__ constexpr int oz_stages(int S, int tbn) { return oz_ctas(S, tbn) == 2 ? 2 : 3; }
// TMEM columns allocated: a power of two that holds the weight accumulators.
__host__ __device__ constexpr int oz_tmem_cols(int weights, int tbn) {
  return weights * tbn <= 128 ? 128 : (weights * tbn <= 256 ? 256 : 512);
}
// Row exponent of a row holding a NaN or an infinity: its slices are zero and
// every product element of the row comes out NaN, so non-finite inputs stay
// visible in the result (the integer slices cannot carry them).
constexpr int kBadExp = 0x7fffffff;

constexpr int OZ_GROUP_M = 8;  // row tiles per raster group
// Epilogue: four warps (one per TMEM lane quarter) per 16 columns of the tile. It is a chain of
// integer operations per column, bound by latency, so more warps with fewer columns each
// shorten it: with 32 columns per warp 140454 x 153 x 64 took 219 us instead of 197 (64-wide), with
// 48 columns 191 us instead of 141 (48-wide). From 96 columns on 16 would leave too few registers
// (or more than 1024 threads), and gained nothing.
__host__ __device__ constexpr int oz_epi_cols(int tbn) { return tbn >= 96 ? 32 : 16; }
__host__ __device__ constexpr int oz_epi_warps(int tbn) { return 4 * (tbn / oz_epi_cols(tbn)); }
__host__ __device__ constexpr int oz_threads(int tbn) {  // TMA warp, MMA warp, epilogue
  return 64 + 32 * oz_epi_warps(tbn);
}
__host__ __device__ constexpr int oz_max_tile(int S) { return S <= 4 ? 128 : (S == 5 ? 96 : 64); }

struct OzPlan {
  int S;          // slices per operand
  int chunk_kb;   // OZ_BK-wide K blocks per exact chunk
};

struct OzEpi {
  int mode;              // 0 store, 1 dot with the strict lower triangle of r (GRAM instances),
                         // 2 subtract from the lower triangle of c,
                         // 3 store the lower triangle of c and its mirror image
  double *c;
  long long ldn, sb;
  const double *r;
  double *partial;
  const int *ea;         // row exponents of A, [batch][rows] (batch stride 0 if shared)
  const int *eb;         // row exponents of B
  long long ea_sb, eb_sb;
  int tri_period;        // > 0: skip tiles wholly above the diagonal of each
                         // tri_period-wide column block (C lower-triangular per block)
  int tri_upper;         // 1: skip the tiles wholly below the diagonals instead
};

// t 2^sc where the result is subnormal, overflows or is next to it: exact steps, one rounding.
__device__ __noinline__ double scaled_double_edge(long long t, int sc) {
  double x = (double)t;
  for (; sc < -1000; sc += 1000) x *= 0x1p-1000;
  for (; sc > 1000; sc -= 1000) x *= 0x1p1000;
  return x * __longlong_as_double((long long)(sc + 1023) << 52);
}

// t 2^sc as ldexp((double)t, sc) gives it (t rounded to nearest even), by integer operations
// without a branch: with an FP64 conversion and an FP64 scaling per element the narrow FP64
// pipe took 12 us per 128 x 96 tile, as long as the products of K = 256.
__device__ __forceinline__ double scaled_double(long long t, int sc) {
  const unsigned long long u = t < 0 ? 0ull - (unsigned long long)t : (unsigned long long)t;
  const int lz = __clzll((long long)u);
  const int E = 63 - lz + sc + 1023;
  if (u != 0 && (E < 1 || E > 2045)) return scaled_double_edge(t, sc);
  const unsigned long long v = u << (lz & 63);  // leading bit at 63 (u != 0)
  const unsigned long long m = v >> 11;         // 53 bits; rounding may carry into the exponent
  const unsigned long long up = ((v & 0x7ff) + 0x3ff + (m & 1)) >> 11;
  const unsigned long long b = ((unsigned long long)E << 52) + (m - (1ull << 52)) + up;
  return u == 0 ? 0.0 : __longlong_as_double((long long)(b | ((unsigned long long)t & (1ull << 63))));
}

// GRAM: the integrand's product (mode 1). It keeps one weight more, the products with t + u = S:
// dotted with integrals, the dropped ones made up most of the error of W, which was 2 to 10 times that
// of the form with Kt Yk (CPU emulation and batch systems of 600 to 1000 pairs); with them it is that
// form's or less, as the digits alone then limit it.
template <int S, int TBN, bool GRAM = false>
__global__ void __launch_bounds__(oz_threads(TBN), oz_ctas(S, TBN))
    k_tc_gemm_oz(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                 int M, int N, int kblocks, int a_batched, int b_batched, OzPlan plan, OzEpi epi,
                 int *err_flag, unsigned long long wait_ns) {
  // One stage = the K block [kb*32, kb*32+32) of all S slices of the A tile (128 rows)
  // and of the B tile (TBN rows): every slice product t+u < S of the block is
  // issued from it, so each slice tile crosses L2 -> shared memory once per block.
  constexpr int NW = GRAM ? S + 1 : S;  // weights
  static_assert(NW * TBN <= 512 / oz_ctas(S, TBN) && TBN % 16 == 0, "weight accumulators exceed TMEM");
  constexpr int EPI = oz_epi_warps(TBN), STG = oz_stages(S, TBN);
  constexpr uint32_t TCOLS = oz_tmem_cols(NW, TBN);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr uint32_t A_BYTES = BM * OZ_BK * 2, B_BYTES = TBN * OZ_BK * 2;
  constexpr uint32_t STAGE_BYTES = S * (A_BYTES + B_BYTES);
  uint64_t *full = (uint64_t *)(smem + STG * STAGE_BYTES);
  uint64_t *empty = full + STG;
  uint64_t *accf = empty + STG;
  uint64_t *acce = accf + 1;
  uint64_t *drainb = acce + 1;  // abort path: completion of the MMAs already issued
  uint32_t *tmem_slot = (uint32_t *)(drainb + 1);
  __shared__ int abort_flag;
  volatile int *abort_v = &abort_flag;
  __shared__ double red[EPI];

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int role = __shfl_sync(0xffffffffu, warp, 0);  // warp, uniform for the compiler too
  // Grouped raster: CTAs are scheduled roughly in linear order, so consecutive ones
  // take OZ_GROUP_M row tiles before moving to the next column tile. A wave of CTAs
  // then shares a few A and B panels in L2 instead of sweeping every A panel
  // (which does not fit in L2 at large M) once per column tile.
  int mt, nt;
  {
    const int ntm = gridDim.x, ntn = gridDim.y;
    const long long t = blockIdx.x + (long long)ntm * blockIdx.y;
    const long long per_group = (long long)OZ_GROUP_M * ntn;
    const int first_m = (int)(t / per_group) * OZ_GROUP_M;
    const int gm = min(ntm - first_m, OZ_GROUP_M);
    const int r = (int)(t % per_group);
    mt = first_m + r % gm;
    nt = r / gm;
  }
  const int m0 = mt * BM, n0 = nt * TBN, b = blockIdx.z;
  const int nchunks = (kblocks + plan.chunk_kb - 1) / plan.chunk_kb;
  if (epi.tri_period > 0) {  // whole CTA, before any barrier or TMEM is set up
    const int c0 = n0 % epi.tri_period;
    const bool inside = c0 + TBN <= epi.tri_period;  // all columns in one block
    if (inside && (epi.tri_upper ? c0 + TBN <= m0 : c0 >= m0 + BM)) {
      if (GRAM && threadIdx.x == 0)
        epi.partial[blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = 0.0;
      return;
    }
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STG; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accf, 1);
    mbar_init(acce, EPI);
    mbar_init(drainb, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The exponents of the tile's rows and columns, read while the pipeline starts: read one by
  // one between the stores of the result (which the compiler cannot move loads across) each
  // column waits for a load.
  __shared__ int eb_s[TBN];
  int ea = 0;
  if (warp >= 2) {
    const int t = threadIdx.x - 64, m = m0 + (warp & 3) * 32 + lane;
    if (t < TBN) eb_s[t] = n0 + t < N ? epi.eb[(long long)b * epi.eb_sb + n0 + t] : 0;
    if (m < M) ea = epi.ea[(long long)b * epi.ea_sb + m];
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    int issued = 0;
    for (int kb = 0; kb < kblocks && !*abort_v; ++kb) {
      const int s = kb % STG;
      if (!mbar_wait(&empty[s], ((kb / STG) & 1) ^ 1, wait_ns)) {
        atomicExch(&abort_flag, 1);
        break;
      }
      mbar_expect_tx(&full[s], STAGE_BYTES);
      uint8_t *st = smem + s * STAGE_BYTES;
#pragma unroll
      for (int t = 0; t < S; ++t)
        tma_load_4d(st + t * A_BYTES, &mapA, &full[s], kb * OZ_BK, m0, a_batched ? b : 0, t);
#pragma unroll
      for (int u = 0; u < S; ++u)
        tma_load_4d(st + S * A_BYTES + u * B_BYTES, &mapB, &full[s], kb * OZ_BK, n0,
                    b_batched ? b : 0, u);
      issued = kb + 1;
    }
    if (*abort_v)  // only the last STG loads can still be in flight
      for (int j = (issued > STG ? issued - STG : 0); j < issued; ++j)
        mbar_wait(&full[j % STG], (j / STG) & 1, kDrainNs);
  } else if (role == 1 && elect_one()) {
    bool ok = true;
    for (int g = 0; g < nchunks && ok; ++g) {
      if (g > 0 && !mbar_wait(acce, (g - 1) & 1, wait_ns)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int kb0 = g * plan.chunk_kb, kb1 = min(kblocks, kb0 + plan.chunk_kb);
      for (int kb = kb0; kb < kb1; ++kb) {
        const int s = kb % STG;
        if (!mbar_wait(&full[s], (kb / STG) & 1, wait_ns) || *abort_v) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_base = smem_u32(smem + s * STAGE_BYTES);
        const uint32_t b_base = a_base + S * A_BYTES;
        // One product per pair of slices, weight t + u always in its own TBN columns: the order in
        // which MMAs take effect is only guaranteed between those of one accumulator and one
        // shape. A slice t meets its B slices back to back, so that it is read from shared memory
        // once and then from the collector buffer (a product without it takes 1.15 times as long
        // at 96 columns, 1.3 at 64). The first product into a weight of the chunk is t = 0 (t = 1 for
        // weight S) at kb0, kk 0. The issuing thread is elected and its descriptors are an addition
        // to a warp-uniform base: with lane 0 of a divided warp and descriptors put together
        // per product, issuing took longer than the product (6290^3 FP64TC5: 5.58 ms, so 4.23).
        const uint64_t da = smem_desc64(a_base), db = smem_desc64(b_base);
#pragma unroll
        for (int t = 0; t < S; ++t)
#pragma unroll
          for (int kk = 0; kk < OZ_BK / 16; ++kk) {
            const uint64_t ad = da + (uint64_t)((t * A_BYTES + kk * 32) >> 4);
            constexpr uint32_t idesc = instr_desc(TBN);
            const int last = S < NW - t ? S - 1 : NW - 1 - t;
#pragma unroll
            for (int u = 0; u <= last; ++u) {
              const uint64_t bd = db + (uint64_t)((u * B_BYTES + kk * 32) >> 4);
              const uint32_t d = tmem + (uint32_t)((t + u) * TBN);
              const bool first = t == 0 || (t == 1 && u == S - 1);
              const uint32_t acc_in = (kb == kb0 && first && kk == 0) ? 0u : 1u;
              if (last == 0)
                mma_bf16_ca<0>(d, ad, bd, idesc, acc_in);
              else if (u == 0)
                mma_bf16_ca<1>(d, ad, bd, idesc, acc_in);
              else if (u < last)
                mma_bf16_ca<2>(d, ad, bd, idesc, acc_in);
              else
                mma_bf16_ca<3>(d, ad, bd, idesc, acc_in);
            }
          }
        mma_commit(&empty[s]);
      }
      mma_commit(accf);
    }
    if (!ok) atomicExch(&abort_flag, 1);
    // TMEM is freed after the final barrier, and the epilogue may have given up on the
    // last chunk: commit every MMA issued so far (a chunk may be half issued) to a
    // barrier of its own and wait until they have completed.
    mma_commit(drainb);
    if (!mbar_wait(drainb, 0, kDrainNs)) atomicExch(&abort_flag, 1);
  } else if (warp >= 2) {
    // Every chunk's FP32 sums v_d are integers below 2^24, so the weights fold into one int64
    // per column, t = sum_d v_d 2^(7 (SI - 1 - d)), exact for the first SI = min(NW, 5) weights
    // (|t| < 2^52 per chunk); what comes after is rounded to units of the fifth first (2^-42 of the
    // scaled product per chunk, beside six slices cut at 2^-42 each). Two weights at a time fit 32 bits
    // (128 |v_0| + |v_1| and 128 |v_2| + |v_3| are below 2^31: v_0 sums products up to 2^14, v_2
    // up to 2 2^13 + 2^12, over at most 672 K), and two 32 x 32 + 64 multiply-adds put the pairs
    // in place: the MMAs of the next chunk wait for this.
    // Four warps per NC columns (one per TMEM lane quarter, q = warp % 4); warp group
    // h = (warp - 2) / 4 owns columns [NC h, NC h + NC) of the tile.
    constexpr int SI = NW < 5 ? NW : 5;
    constexpr int NC = oz_epi_cols(TBN), LW = NC == 16 ? 4 : 8;
    const int q = warp & 3;
    const int h = (warp - 2) / 4;
    const int m = m0 + q * 32 + lane;
    long long acc[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) acc[j] = 0;
    bool ok = true;
    for (int g = 0; g < nchunks && ok; ++g) {
      if (!mbar_wait(accf, g & 1, wait_ns) || *abort_v) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c0 = 0; c0 < NC; c0 += LW) {
        uint32_t r[NW][LW];
#pragma unroll
        for (int d = 0; d < NW; ++d) {
          const uint32_t a = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(d * TBN + h * NC + c0);
          if constexpr (LW == 8)
            tmem_ld8_issue(a, r[d]);
          else
            tmem_ld4_issue(a, r[d]);
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < LW; ++j) {
          int v[SI];
#pragma unroll
          for (int d = 0; d < SI; ++d) v[d] = __float2int_rn(__uint_as_float(r[d][j]));
          if (NW == SI + 1) v[SI - 1] += __float2int_rn(__uint_as_float(r[SI][j]) * 0.0078125f);
          if (NW == SI + 2)
            v[SI - 1] += __float2int_rn((__uint_as_float(r[SI + 1][j]) * 0.0078125f +
                                         __uint_as_float(r[SI][j])) * 0.0078125f);
          const int p0 = v[0] * 128 + v[1], p1 = v[2] * 128 + v[3];
          long long t = acc[c0 + j];
          if (SI == 5) {
            t += (long long)p0 * (1 << 21);
            t += (long long)p1 * 128;
            t += v[SI - 1];
          } else {
            t += (long long)p0 * (1 << 14);
            t += p1;
          }
          acc[c0 + j] = t;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acce)) : "memory");
    }
    if (!ok) atomicExch(&abort_flag, 1);
    double dot = 0.0;
    if (ok) {
      const int er = ea - 7 * (SI + 1);
      const long long o0 = (long long)b * epi.sb + m + (long long)(n0 + h * NC) * epi.ldn;
      // FP64 results first, then one short loop per mode: a tile runs this code once, so its
      // length counts (this part of a 128 x 64 tile: 6.7 us as one unrolled loop over modes and
      // edge cases, 4.1 us so).
      double cv[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int eb = eb_s[h * NC + j];
        const double v = scaled_double(acc[j], eb == kBadExp || ea == kBadExp ? 0 : er + eb);
        cv[j] = eb == kBadExp || ea == kBadExp ? __longlong_as_double(0x7ff8000000000000ll) : v;
      }
      const int n1 = n0 + h * NC, nn = m < M ? min(NC, N - n1) : 0;
      if constexpr (GRAM) {
        const int last = min(nn, m - n1);  // columns below the diagonal
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < last) dot += cv[j] * epi.r[o0 + j * epi.ldn];
      } else if (epi.mode == 0) {
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < nn) epi.c[o0 + j * epi.ldn] = cv[j];
      } else if (epi.mode == 3) {
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < nn && m >= n1 + j) epi.c[o0 + j * epi.ldn] = cv[j];
        // the mirror image, turned in shared memory (the stages are free: every load was
        // consumed by a product that has completed): stores of NC consecutive elements
        double *tr = reinterpret_cast<double *>(smem) + (warp - 2) * (NC * 33);
#pragma unroll
        for (int j = 0; j < NC; ++j) tr[j * 33 + lane] = cv[j];
        __syncwarp();
        const int n = n1 + lane % NC, mb = m0 + q * 32 + lane / NC;
        for (int i = 0; i < NC; ++i) {
          const int k = i * (32 / NC), mm = mb + k;
          if (mm < M && n < N && mm >= n)
            epi.c[n + (long long)mm * epi.ldn] = tr[(lane % NC) * 33 + k + lane / NC];
        }
      } else {
        const int last = min(nn, m - n1 + 1);  // columns up to the diagonal
#pragma unroll
        for (int j0 = 0; j0 < NC; j0 += 8) {  // the loads of a group before its stores
          double old[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) old[j] = j0 + j < last ? epi.c[o0 + (j0 + j) * epi.ldn] : 0.0;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j0 + j < last) epi.c[o0 + (j0 + j) * epi.ldn] = old[j] - cv[j0 + j];
        }
      }
    }
    if (GRAM) {
      for (int off = 16; off > 0; off >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, off);
      if (lane == 0) red[warp - 2] = dot;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (GRAM && threadIdx.x == 0) {
    long long cta = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
    double sum = 0.0;
    for (int w = 0; w < EPI; ++w) sum += red[w];
    epi.partial[cta] = sum;
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(err_flag, 1);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
  }
}

// |x| as its bit pattern without the sign: for finite values the unsigned integer order is
// the order of |x|, and a value with the exponent field all ones is an infinity or a NaN.
__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
// 1 + ilogb of the value whose |x| bits are m (m > 0, finite), from the bits.
__device__ __forceinline__ int exp_of_bits(unsigned long long m) {
  const int E = (int)(m >> 52);
  return E > 0 ? E - 1022 : -1010 - __clzll((long long)m);
}
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;

// e = 1 + ilogb of the row's largest |x| (its bits mx): 0 for a zero row, kBadExp for a row
// with a non-finite element.
__device__ __forceinline__ int row_exponent(unsigned long long mx) {
  return mx >= kInfBits ? kBadExp : (mx ? exp_of_bits(mx) : 0);
}

// Balanced base-128 digits of n = rint(x 2^(7S - e)) (|x| < 2^e, so |n| <= 2^(7S)):
// n = sum_s a_s 128^(S-1-s), |a_0| <= 128, |a_s| <= 64 otherwise, as FP32 bit patterns whose
// upper half is the BF16 value. Rounding is to nearest even, as __double2ll_rn(ldexp(x, 7S - e))
// rounds (that scaling is exact unless the result is below 1/2, which rounds to 0 either way).
// Integer operations but for one FP32 addition per digit: GB300's FP64 pipe is narrow, and
// integer-to-float conversions share a quarter-rate pipe. With B = 64 (1 + 128 + ...) added
// once, the lower digits are plain 7-bit fields minus 64 and the carries are already in place.
template <int S>
__device__ __forceinline__ void digits(double x, int e, uint32_t *d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = (b & 0xfffffffffffffull) | (E ? 1ull << 52 : 0ull);
  // x = +-m 2^(max(E, 1) - 1075); |x| < 2^e makes the shift at least 53 - 7S > 0, unless the
  // whole row is subnormal
  const int sft = e == kBadExp ? 64 : 1075 - max(E, 1) - 7 * S + e;
  long long n = 0;
  if (sft < 1)
    n = (long long)(m << -sft);
  else if (sft <= 63)
    n = (long long)((m + ((1ull << (sft - 1)) - 1) + ((m >> sft) & 1)) >> sft);
  if (b >> 63) n = -n;
  unsigned long long bias = 0;
#pragma unroll
  for (int s = 1; s < S; ++s) bias = bias * 128 + 64;
  const long long u = n + (long long)bias;
#pragma unroll
  for (int s = 1; s < S; ++s) {
    const int v = (int)(u >> (7 * (S - 1 - s))) & 127;
    d[s] = __float_as_uint(__int_as_float(0x4B400000 - 64 + v) - 12582912.f);
  }
  d[0] = __float_as_uint(__int_as_float(0x4B400000 + (int)(u >> (7 * (S - 1)))) - 12582912.f);
}

// Four consecutive elements of one row into their S planes, 8 bytes per plane.
template <int S>
__device__ __forceinline__ void store_digits4(const double *x, int e, long long plane, long long o,
                                              __nv_bfloat16 *__restrict__ planes) {
  uint32_t d[4][S];
#pragma unroll
  for (int i = 0; i < 4; ++i) digits<S>(x[i], e, d[i]);
#pragma unroll
  for (int s = 0; s < S; ++s)
    *reinterpret_cast<uint2 *>(planes + s * plane + o) =
        make_uint2(__byte_perm(d[0][s], d[1][s], 0x7632), __byte_perm(d[2][s], d[3][s], 0x7632));
}

// Row exponents and integer slices, planes[t][b][r][kp] = alpha_t of x[b,r,k] 2^-e[b][r], of an
// operand whose K elements are contiguous: TPR threads per row, each holding its elements of
// the row in registers between the maximum and the digits (kOzHold groups of four; rows longer
// than TPR * 4 * kOzHold are read again for the rest). Bound by HBM: 8 bytes read and 2 S written per element. One
// warp per row up to 1024 elements, so that short rows fill a block; a block per longer row.
// Measured (5 slices): 3774 x 3774 62 us = 4.1 TB/s, where a pass for the exponents and a pass
// with 2-byte stores took 155 us.
template <int S, int TPR, int kOzHold>
__global__ void __launch_bounds__(256) k_oz_rows(const double *__restrict__ x, int rows, int K, int Kp,
                                                 long long nrr, long long sr, long long sb,
                                                 int *__restrict__ e,
                                                 __nv_bfloat16 *__restrict__ planes) {
  __shared__ unsigned long long part[8];
  const int t = threadIdx.x % TPR;
  const long long rr = blockIdx.x * (long long)(256 / TPR) + threadIdx.x / TPR;
  const bool live = rr < nrr;
  const long long bb = live ? rr / rows : 0;
  const double *__restrict__ xr = x + (live ? bb * sb + (rr - bb * rows) * sr : 0);
  double v[kOzHold][4];
  unsigned long long mx = 0;
  const int ng = Kp / 4;
#pragma unroll
  for (int g = 0; g < kOzHold; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = (t + g * TPR) * 4 + i;
      v[g][i] = live && k < K ? xr[k] : 0.0;
    }
#pragma unroll
  for (int g = 0; g < kOzHold; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) mx = max(mx, abs_bits(v[g][i]));
  if (live)
    for (int k = TPR * 4 * kOzHold + t; k < K; k += TPR) mx = max(mx, abs_bits(xr[k]));
  for (int off = 16; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if (TPR > 32) {
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = max(mx, part[w]);
  }
  if (!live) return;
  const int ex = row_exponent(mx);
  if (t == 0) e[rr] = ex;
  const long long plane = nrr * Kp;
#pragma unroll
  for (int g = 0; g < kOzHold; ++g)
    if (t + g * TPR < ng) store_digits4<S>(v[g], ex, plane, rr * Kp + (t + g * TPR) * 4, planes);
  for (int g = t + kOzHold * TPR; g < ng; g += TPR) {
    double w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = g * 4 + i < K ? xr[g * 4 + i] : 0.0;
    store_digits4<S>(w, ex, plane, rr * Kp + g * 4, planes);
  }
}

// Offset c + d n of the packed pair r = c + d (d + 1) / 2, c <= d.
__device__ __forceinline__ long long tri_offset(int r, int n) {
  int d = (int)((sqrtf(8.f * (float)r + 1.f) - 1.f) * 0.5f);
  while ((long long)d * (d + 1) / 2 > r) --d;
  while ((long long)(d + 1) * (d + 2) / 2 <= r) ++d;
  return r - (long long)d * (d + 1) / 2 + (long long)d * n;
}

// What k_oz_cols does beside slicing: columns k of x outside (lo, hi) by eig[k] count as zero,
// and sq[b][r] = sum_k x[b,r,k]^2 in FP64 (the integrand's dropped modes and its diagonal term).
// One kernel up to this K: a transform of n = 64 (K = 300) takes 11 us instead of two launches.
constexpr int kOzShortK = 512;
struct OzColsOpt {
  const double *eig = nullptr;
  double lo = 0.0, hi = 0.0;
  double *sq = nullptr;
};

// Element (b, r, k) of an operand with any strides (in use: consecutive rows contiguous, K the
// slow index), rows by pair index (tri > 0: row r is the pair (c, d), c <= d, of a tri x tri
// matrix, r = c + d (d + 1) / 2) and columns dropped by opt.eig.
struct OzColView {
  const double *x;
  int rows, K, tri;
  long long sr, sk, sb;
  OzColsOpt opt;
  __device__ __forceinline__ const double *row(long long bb, int r) const {
    return x + bb * sb + (tri > 0 ? tri_offset(r, tri) : r) * sr;
  }
  // lo < eig < hi for 0 < lo < hi, as integers: the FP64 pipe is narrow
  __device__ __forceinline__ bool kept(int k) const {
    if (!opt.eig) return true;
    const long long b = __double_as_longlong(opt.eig[k]);
    return b > __double_as_longlong(opt.lo) && b < __double_as_longlong(opt.hi);
  }
  __device__ __forceinline__ double at(const double *xr, int r, int k) const {
    double v = r < rows && k < K ? xr[k * sk] : 0.0;
    if (k < K && !kept(k)) v = 0.0;
    return v;
  }
};

// Such operands in one kernel, for short K (Cholesky panels, small transforms: one launch). A
// block takes 16 rows: the maximum with the lanes along the rows, then 128 values of K at a time
// through shared memory, read along the rows and written along K. The position of k within
// its 128 is (k / 4) + 32 (k % 4), so that four consecutive k are read without bank conflicts.
template <int S>
__global__ void __launch_bounds__(512) k_oz_cols(OzColView X, int Kp, int nb, int *__restrict__ e,
                                                 __nv_bfloat16 *__restrict__ planes) {
  constexpr int ROWS = 16, TY = 32;
  __shared__ double tile[ROWS][129];
  __shared__ unsigned long long part[TY][ROWS];
  __shared__ double psq[TY][ROWS];
  __shared__ int es[ROWS];
  const int tx = threadIdx.x % ROWS, ty = threadIdx.x / ROWS;
  const int r0 = blockIdx.x * ROWS, r = r0 + tx;
  const int lr = threadIdx.x / 32, lk = threadIdx.x % 32;  // row and group of four in the write
  const long long plane = (long long)nb * X.rows * Kp;
  for (int bb = blockIdx.y; bb < nb; bb += gridDim.y) {
    const double *xr = X.row(bb, r);
    unsigned long long mx = 0;
    double q = 0.0;
#pragma unroll 4
    for (int k = ty; k < X.K; k += TY) {
      const double v = X.at(xr, r, k);
      mx = max(mx, abs_bits(v));
      if (X.opt.sq) q += v * v;
    }
    part[ty][tx] = mx;
    psq[ty][tx] = q;
    __syncthreads();
    if (ty == 0) {
      for (int w = 1; w < TY; ++w) mx = max(mx, part[w][tx]);
      es[tx] = row_exponent(mx);
      if (r < X.rows) {
        e[(long long)bb * X.rows + r] = es[tx];
        if (X.opt.sq) {
          for (int w = 1; w < TY; ++w) q += psq[w][tx];
          X.opt.sq[(long long)bb * X.rows + r] = q;
        }
      }
    }
    for (int k0 = 0; k0 < Kp; k0 += 128) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = ty + TY * i;
        tile[tx][(k >> 2) + 32 * (k & 3)] = X.at(xr, r, k0 + k);
      }
      __syncthreads();
      if (r0 + lr < X.rows && k0 + lk * 4 < Kp) {
        const double v[4] = {tile[lr][lk], tile[lr][lk + 32], tile[lr][lk + 64], tile[lr][lk + 96]};
        store_digits4<S>(v, es[lr], plane, ((long long)bb * X.rows + r0 + lr) * Kp + k0 + lk * 4, planes);
      }
    }
    __syncthreads();
  }
}

// ... and in two kernels for longer K, so that both passes have blocks enough for the chip:
// the maxima (and squares) of 64 rows over a share of K, then the digits of 64 x 64 tiles (512
// contiguous bytes per load). part[share][b][r], psq likewise. Measured (5 slices): 6972 x 1494
// 19 + 46 us, where one kernel with 16 rows per block took 89 us, with 32 rows 76 us, and a
// cluster of CTAs sharing the maxima 108 us; 3774 x 3774 with eig and sq 62 + 78 us (one kernel
// 171 us).
constexpr int kColW = 64;
constexpr int kColShare = 1024;  // K per block of k_oz_col_max at most
__global__ void __launch_bounds__(256) k_oz_col_max(OzColView X, int nb, int share,
                                                    unsigned long long *__restrict__ part,
                                                    double *__restrict__ psq) {
  __shared__ unsigned long long pm[4][kColW];
  __shared__ double ps[4][kColW];
  __shared__ unsigned char keep[kColShare];
  const int tx = threadIdx.x % kColW, ty = threadIdx.x / kColW, r = blockIdx.x * kColW + tx;
  const int k0 = blockIdx.y * share, k1 = min(X.K, k0 + share);
  if (X.opt.eig) {
    for (int k = k0 + threadIdx.x; k < k1; k += 256) keep[k - k0] = X.kept(k);
    __syncthreads();
  }
  for (int bb = blockIdx.z; bb < nb; bb += gridDim.z) {
    const double *xr = X.row(bb, min(r, X.rows - 1));
    unsigned long long mx = 0;
    double q = 0.0;
    int k = k0 + ty;
    for (; k + 28 < k1; k += 32) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = xr[(k + 4 * i) * X.sk];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (X.opt.eig && !keep[k + 4 * i - k0]) v[i] = 0.0;
        mx = max(mx, abs_bits(v[i]));
        if (X.opt.sq) q += v[i] * v[i];
      }
    }
    for (; k < k1; k += 4) {
      const double v = !X.opt.eig || keep[k - k0] ? xr[k * X.sk] : 0.0;
      mx = max(mx, abs_bits(v));
      if (X.opt.sq) q += v * v;
    }
    pm[ty][tx] = mx;
    ps[ty][tx] = q;
    __syncthreads();
    if (ty == 0 && r < X.rows) {
      for (int w = 1; w < 4; ++w) {
        mx = max(mx, pm[w][tx]);
        q += ps[w][tx];
      }
      const size_t o = ((size_t)blockIdx.y * nb + bb) * X.rows + r;
      part[o] = mx;
      if (X.opt.sq) psq[o] = q;
    }
    __syncthreads();
  }
}

template <int S>
__global__ void __launch_bounds__(256) k_oz_col_digits(OzColView X, int Kp, int nb, int nshare,
                                                       const unsigned long long *__restrict__ part,
                                                       const double *__restrict__ psq,
                                                       int *__restrict__ e,
                                                       __nv_bfloat16 *__restrict__ planes) {
  __shared__ double tile[kColW][65];  // k of the 64 at (k / 4) + 16 (k % 4)
  __shared__ int es[kColW];
  __shared__ unsigned char keep[64];
  const int tx = threadIdx.x % kColW, ty = threadIdx.x / kColW;
  const int r0 = blockIdx.x * kColW, r = r0 + tx, k0 = blockIdx.y * 64;
  const int lr = threadIdx.x / 16, lk = threadIdx.x % 16;
  const long long plane = (long long)nb * X.rows * Kp;
  for (int bb = blockIdx.z; bb < nb; bb += gridDim.z) {
    const double *xr = X.row(bb, min(r, X.rows - 1));
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int k = k0 + ty + 4 * i;
      v[i] = r < X.rows && k < X.K ? xr[k * X.sk] : 0.0;
    }
    if (threadIdx.x < 64) keep[threadIdx.x] = k0 + threadIdx.x >= X.K || X.kept(k0 + threadIdx.x);
#pragma unroll
    for (int i = 0; i < 16; ++i) tile[tx][i + 16 * ty] = v[i];
    if (ty == 0 && r < X.rows) {
      unsigned long long mx = 0;
      double q = 0.0;
      for (int c = 0; c < nshare; ++c) {
        const size_t o = ((size_t)c * nb + bb) * X.rows + r;
        mx = max(mx, part[o]);
        if (X.opt.sq) q += psq[o];
      }
      es[tx] = row_exponent(mx);
      if (blockIdx.y == 0) {
        e[(long long)bb * X.rows + r] = es[tx];
        if (X.opt.sq) X.opt.sq[(long long)bb * X.rows + r] = q;
      }
    }
    __syncthreads();
#pragma unroll
    for (int l = lr; l < kColW; l += 16)
      if (r0 + l < X.rows) {
        double w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = keep[lk * 4 + i] ? tile[l][lk + 16 * i] : 0.0;
        store_digits4<S>(w, es[l], plane, ((long long)bb * X.rows + r0 + l) * Kp + k0 + lk * 4, planes);
      }
    __syncthreads();
  }
}

// Row exponents and slices of symmetric n x n matrices read from their packed triangles
// (matrix k at x + k ld, element (p, q), p <= q, at p + q (q + 1) / 2): the operand has a row
// (k, p) for every p, without the unpacked FP64 matrices ever being written. One block per
// matrix (blockIdx.y: a share of its tiles): the maxima of all rows from one sweep over the
// triangle (high words only: the exponent is all that is wanted), then the triangle again in
// 64 x 64 tiles through shared memory, each of which gives the digits of its rows and, with their
// own exponents, of its columns. A tile is loaded along p, contiguous in the triangle.
// Measured for 1494 matrices with n = 249: 0.37 ms (4.5 TB/s; both sweeps come from HBM), with a
// warp per row that gathers the elements beyond the diagonal 0.40, with a cluster of four
// blocks per matrix 0.41, and unpacking, exponents and digits apart 1.2 ms.
template <int S>
__global__ void __launch_bounds__(256) k_oz_packed(const double *__restrict__ x, long long ld, int n,
                                                   int Kp, int cnt, int *__restrict__ e,
                                                   __nv_bfloat16 *__restrict__ planes) {
  extern __shared__ unsigned rmax[];
  // [q][p], row q at (q / 4) + 16 (q % 4): four consecutive q of a column from four rows without
  // bank conflicts, four consecutive p of a row as two 16-byte reads
  __shared__ __align__(16) double tile[64][66];
  auto at = [](int q) { return (q >> 2) + 16 * (q & 3); };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double *__restrict__ xk = x + blockIdx.x * ld;
  for (int p = threadIdx.x; p < n; p += 256) rmax[p] = 0;
  __syncthreads();
  for (int q = warp; q < n; q += 8) {
    const double *__restrict__ c = xk + (long long)q * (q + 1) / 2;
    unsigned mx = 0;
#pragma unroll 4
    for (int p = lane; p <= q; p += 32) {
      const unsigned h = (unsigned)__double2hiint(c[p]) & 0x7fffffffu;
      atomicMax(&rmax[p], h);
      mx = max(mx, h);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) atomicMax(&rmax[q], mx);
  }
  __syncthreads();
  const long long row0 = blockIdx.x * (long long)n, plane = (long long)cnt * n * Kp;
  auto exponent = [&](int p) {
    const int E = (int)(rmax[p] >> 20);
    return E == 0x7ff ? kBadExp : max(E, 1) - 1022;  // 2^-1021 bounds a subnormal or zero row
  };
  if (blockIdx.y == 0)
    for (int p = threadIdx.x; p < n; p += 256) e[row0 + p] = exponent(p);
  const int nt = Kp / 64, tx = threadIdx.x & 63, ty = threadIdx.x >> 6;  // load: p along tx
  const int lr = threadIdx.x >> 4, lk = threadIdx.x & 15;                // write: row, group of 4
  for (int t = blockIdx.y; t < nt * (nt + 1) / 2; t += gridDim.y) {
    int tq = 0;  // tile (tp, tq), tp <= tq
    while ((tq + 1) * (tq + 2) / 2 <= t) ++tq;
    const int p0 = (t - tq * (tq + 1) / 2) * 64, q0 = tq * 64;
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int q = q0 + ty + 4 * i, p = p0 + tx;
      v[i] = q < n && p <= q ? xk[p + (long long)q * (q + 1) / 2] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) tile[at(ty + 4 * i)][tx] = v[i];
    __syncthreads();
    if (p0 == q0) {  // the diagonal tile's other half
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int q = ty + 4 * i;
        if (tx > q) tile[at(q)][tx] = tile[at(tx)][q];
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // rows q, K along p
      const int l = lr + 16 * i;
      if (q0 + l < n) {
        const double2 a = *reinterpret_cast<const double2 *>(&tile[at(l)][lk * 4]);
        const double2 b = *reinterpret_cast<const double2 *>(&tile[at(l)][lk * 4 + 2]);
        const double w[4] = {a.x, a.y, b.x, b.y};
        store_digits4<S>(w, exponent(q0 + l), plane, (row0 + q0 + l) * Kp + p0 + lk * 4, planes);
      }
    }
    if (p0 != q0)
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // rows p, K along q
        const int l = lr + 16 * i;
        if (p0 + l < n) {
          const double w[4] = {tile[lk][l], tile[lk + 16][l], tile[lk + 32][l], tile[lk + 48][l]};
          store_digits4<S>(w, exponent(p0 + l), plane, (row0 + p0 + l) * Kp + q0 + lk * 4, planes);
        }
      }
  }
}

// out[cd + nCD ab] from the product over pairs (row index cd or its packed form, column index
// ab or its packed form): every element of the pair blocks from the triangles.
__global__ void k_expand_pairs(const double *__restrict__ cp, long long ldc, int nC, int nD, int symCD,
                               int nA, int nB, int symAB, double *__restrict__ out) {
  const int cd = blockIdx.x * blockDim.x + threadIdx.x;
  if (cd >= nC * nD) return;
  const int c = cd % nC, d = cd / nC;
  auto tri = [](int a, int b) { return a <= b ? a + (long long)b * (b + 1) / 2 : b + (long long)a * (a + 1) / 2; };
  const long long r = symCD ? tri(c, d) : cd;
  for (int ab = blockIdx.y; ab < nA * nB; ab += gridDim.y) {
    const long long k = symAB ? tri(ab % nA, ab / nA) : ab;
    out[cd + (long long)nC * nD * ab] = cp[r + k * ldc];
  }
}

// ------------------------------------------------------------ operand packing
// planes[s][b][r][kp] (bf16) from x[b*sb + r*sr + k*sk] (FP64): x = x0 + x1 + x2 + ...
__global__ void k_pack_planes(const double *__restrict__ x, int rows, int K, int Kp, int nb,
                              long long sr, long long sk, long long sb, int S,
                              __nv_bfloat16 *__restrict__ planes) {
  long long plane = (long long)nb * rows * Kp;
  long long total = plane;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int k = (int)(t % Kp);
    long long rr = t / Kp;
    int r = (int)(rr % rows);
    long long bb = rr / rows;
    double v = k < K ? x[bb * sb + r * sr + (long long)k * sk] : 0.0;
    for (int s = 0; s < S; ++s) {
      __nv_bfloat16 h = __double2bfloat16(v);
      planes[s * plane + t] = h;
      v -= (double)__bfloat162float(h);
    }
  }
}

// Same, for operands whose K index is the slow one (sk >> sr): a 32 x 32 tile
// is staged in shared memory so that reads run along rows and writes along K.
__global__ void k_pack_planes_t(const double *__restrict__ x, int rows, int K, int Kp, int nb,
                                long long sr, long long sk, long long sb, int S,
                                __nv_bfloat16 *__restrict__ planes) {
  __shared__ double tile[32][33];
  int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32, bb = blockIdx.z;
  int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int i = ty; i < 32; i += 8) {
    int k = k0 + i, r = r0 + tx;
    tile[i][tx] = (k < K && r < rows) ? x[bb * sb + (long long)r * sr + (long long)k * sk] : 0.0;
  }
  __syncthreads();
  long long plane = (long long)nb * rows * Kp;
  for (int i = ty; i < 32; i += 8) {
    int r = r0 + i, k = k0 + tx;
    if (r >= rows || k >= Kp) continue;
    double v = tile[tx][i];
    long long o = ((long long)bb * rows + r) * Kp + k;
    for (int s = 0; s < S; ++s) {
      __nv_bfloat16 h = __double2bfloat16(v);
      planes[s * plane + o] = h;
      v -= (double)__bfloat162float(h);
    }
  }
}

// ----------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// Operand planes [S][nb][rows][Kp] bf16 and their 4-D tensor map.
struct Operand {
  gc::DevBuf<__nv_bfloat16> buf;
  CUtensorMap map;
  int rows = 0, Kp = 0, nb = 1, S = 0;
};

int make_operand(gc_context *ctx, Operand &op, const double *x, int rows, int K, int nb,
                 long long sr, long long sk, long long sb, int S, int box_rows) {
  op.rows = rows;
  op.Kp = (K + BK - 1) / BK * BK;
  op.nb = nb;
  op.S = S;
  size_t plane = (size_t)nb * rows * op.Kp;
  GC_TRY(op.buf.alloc(ctx, plane * S));
  if (sk == 1) {
    unsigned grid = std::min<unsigned>(gc::ceil_div(plane, 256), 152u * 32u);
    k_pack_planes<<<grid, 256, 0, ctx->stream>>>(x, rows, K, op.Kp, nb, sr, sk, sb, S, op.buf.p);
  } else {
    dim3 grid(gc::ceil_div(rows, 32), gc::ceil_div(op.Kp, 32), nb);
    k_pack_planes_t<<<grid, dim3(32, 8), 0, ctx->stream>>>(x, rows, K, op.Kp, nb, sr, sk, sb, S,
                                                           op.buf.p);
  }
  GC_LAUNCHED(ctx);
  EncodeTiledFn enc = encode_fn();
  if (!enc) return gc::set_error(ctx, GC_ECUDA, "cuTensorMapEncodeTiled entry point unavailable");
  cuuint64_t dims[4] = {(cuuint64_t)op.Kp, (cuuint64_t)rows, (cuuint64_t)nb, (cuuint64_t)S};
  cuuint64_t strides[3] = {(cuuint64_t)op.Kp * 2, (cuuint64_t)rows * op.Kp * 2,
                           (cuuint64_t)nb * rows * op.Kp * 2};
  cuuint32_t box[4] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(&op.map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, op.buf.p, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return gc::set_error(ctx, GC_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return GC_OK;
}

PassList pass_list(int precision, int *S) {
  PassList p{};
  if (precision == GC_PREC_BF16X3) {
    *S = 2;
    p.n = 3;
    int a[3] = {1, 0, 0}, b[3] = {0, 1, 0};
    for (int i = 0; i < 3; ++i) p.pa[i] = a[i], p.pb[i] = b[i];
  } else {  // six passes over three planes: every product x_i y_j with i + j <= 2
    *S = 3;
    p.n = 6;
    int a[6] = {2, 1, 0, 1, 0, 0}, b[6] = {0, 1, 2, 0, 1, 0};
    for (int i = 0; i < 6; ++i) p.pa[i] = a[i], p.pb[i] = b[i];
  }
  return p;
}

constexpr int BN_T = 128;

size_t smem_bytes(int bn) {
  return 1024 + STAGES * (size_t)(BM * BK * 2 + bn * BK * 2) + (2 * STAGES + 1) * 8 + 16;
}

// C = A . B^T over prepared operands; A may be shared across the batch.
int run_gemm(gc_context *ctx, const Operand &A, const Operand &B, int M, int N, int nbatch,
             const PassList &pl, const Epi &epi) {
  if (A.Kp != B.Kp) return gc::set_error(ctx, GC_EINVAL, "tc_gemm: K mismatch");
  // on every call: the setting holds for one device
  GC_CUDA(ctx, cudaFuncSetAttribute(k_tc_gemm<BN_T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem_bytes(BN_T)));
  dim3 grid(gc::ceil_div(M, BM), gc::ceil_div(N, BN_T), nbatch);
  k_tc_gemm<BN_T><<<grid, 192, smem_bytes(BN_T), ctx->stream>>>(
      A.map, B.map, M, N, A.Kp / BK, A.nb > 1 ? 1 : 0, B.nb > 1 ? 1 : 0, pl, epi, ctx->dev_flag,
      ctx->wait_ns);
  GC_LAUNCHED(ctx);
  return GC_OK;
}



// ---- sliced (FP64-accurate) operands and launch
struct OzOperand {
  gc::DevBuf<__nv_bfloat16> buf;
  gc::DevBuf<int> exps;
  CUtensorMap map;
  int rows = 0, Kp = 0, nb = 1, S = 0, box_rows = 0;
  const __nv_bfloat16 *planes = nullptr;  // buf.p, or another operand's planes (alias)
  const int *ex = nullptr;                // exps.p, or another operand's exponents
};

bool is_oz(int precision) { return gc::is_sliced(precision); }

OzPlan oz_plan(int precision) {
  OzPlan p{};
  p.S = precision == GC_PREC_FP64TC6 ? 6 : (precision == GC_PREC_FP64TC4 ? 4 : 5);
  // exact FP32 partial sums: (S+2) 2^12 c < 2^24 and 2^14 c < 2^24
  int c = (4096 / (p.S + 2)) / OZ_BK * OZ_BK;
  if ((long long)(p.S + 2) * 4096 * c >= (1ll << 24)) c -= OZ_BK;
  p.chunk_kb = c / OZ_BK;
  return p;
}

// The 4-D TMA map [S][nb][rows][Kp] of an operand's slice planes, box OZ_BK x box_rows.
int encode_oz_map(gc_context *ctx, OzOperand &op) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return gc::set_error(ctx, GC_ECUDA, "cuTensorMapEncodeTiled entry point unavailable");
  cuuint64_t dims[4] = {(cuuint64_t)op.Kp, (cuuint64_t)op.rows, (cuuint64_t)op.nb,
                        (cuuint64_t)op.S};
  cuuint64_t strides[3] = {(cuuint64_t)op.Kp * 2, (cuuint64_t)op.rows * op.Kp * 2,
                           (cuuint64_t)op.nb * op.rows * op.Kp * 2};
  cuuint32_t box[4] = {(cuuint32_t)OZ_BK, (cuuint32_t)op.box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(&op.map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void *)op.planes, dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return gc::set_error(ctx, GC_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return GC_OK;
}

template <int S>
int slice_operand(gc_context *ctx, OzOperand &op, const double *x, int rows, int K, int nb,
                  long long sr, long long sk, long long sb, int tri, const OzColsOpt &opt) {
  const long long nrr = (long long)nb * rows;
  const bool plain = !tri && !opt.eig && !opt.sq;
  if (sk == 1 && plain) {
    // One warp holds a row up to K = 256 (140454 x 153: 182 -> 115 us against the instance for
    // 1024, which has twice the registers) and, for rows enough to fill the chip, up to 1024;
    // else a block holds it, with the registers for its length (1390 x 1390: 12 us, with the registers for K = 8192 20 us).
    const bool warp_row = op.Kp <= 256 || (op.Kp <= 1024 && nrr >= 152 * 16);
    auto kern = op.Kp <= 256 ? k_oz_rows<S, 32, 2>
                             : (warp_row ? k_oz_rows<S, 32, 8>
                                         : (op.Kp <= 1024 ? k_oz_rows<S, 256, 1>
                                                          : (op.Kp <= 2048 ? k_oz_rows<S, 256, 2>
                                                                           : k_oz_rows<S, 256, 8>)));
    kern<<<warp_row ? gc::ceil_div(nrr, 8) : (unsigned)nrr, 256, 0, ctx->stream>>>(
        x, rows, K, op.Kp, nrr, sr, sb, op.exps.p, op.buf.p);
  } else {
    const OzColView X{x, rows, K, tri, sr, sk, sb, opt};
    if (op.Kp <= kOzShortK) {
      k_oz_cols<S><<<dim3(gc::ceil_div(rows, 16), std::min(nb, 65535)), 512, 0, ctx->stream>>>(
          X, op.Kp, nb, op.exps.p, op.buf.p);
    } else {
      const int nshare = std::max(std::min(16, (K + 255) / 256), (K + kColShare - 1) / kColShare);
      const int share = (K + nshare - 1) / nshare;
      gc::DevBuf<unsigned long long> part;
      gc::DevBuf<double> psq;
      GC_TRY(part.alloc(ctx, (size_t)nshare * nrr));
      if (opt.sq) GC_TRY(psq.alloc(ctx, (size_t)nshare * nrr));
      const unsigned gz = std::min(nb, 65535);
      k_oz_col_max<<<dim3(gc::ceil_div(rows, kColW), nshare, gz), 256, 0, ctx->stream>>>(X, nb, share,
                                                                                      part.p, psq.p);
      GC_LAUNCHED(ctx);
      k_oz_col_digits<S><<<dim3(gc::ceil_div(rows, kColW), op.Kp / 64, gz), 256, 0,
                           ctx->stream>>>(X, op.Kp, nb, nshare, part.p, psq.p, op.exps.p, op.buf.p);
    }
  }
  GC_LAUNCHED(ctx);
  return GC_OK;
}

int make_oz_operand(gc_context *ctx, OzOperand &op, const double *x, int rows, int K, int nb,
                    long long sr, long long sk, long long sb, int S, int box_rows, int tri = 0,
                    const OzColsOpt &opt = OzColsOpt()) {
  op.rows = rows;
  op.box_rows = box_rows;
  op.Kp = (K + BK - 1) / BK * BK;
  op.nb = nb;
  op.S = S;
  size_t plane = (size_t)nb * rows * op.Kp;
  GC_TRY(op.exps.alloc(ctx, (size_t)nb * rows));
  GC_TRY(op.buf.alloc(ctx, plane * S));
  switch (S) {
    case 4: GC_TRY(slice_operand<4>(ctx, op, x, rows, K, nb, sr, sk, sb, tri, opt)); break;
    case 5: GC_TRY(slice_operand<5>(ctx, op, x, rows, K, nb, sr, sk, sb, tri, opt)); break;
    default: GC_TRY(slice_operand<6>(ctx, op, x, rows, K, nb, sr, sk, sb, tri, opt));
  }
  op.planes = op.buf.p;
  op.ex = op.exps.p;
  return encode_oz_map(ctx, op);
}

// The operand of cnt packed symmetric n x n matrices, one row per (matrix, p).
int make_oz_packed(gc_context *ctx, OzOperand &op, const double *x, long long ld, int n, int cnt,
                   int S) {
  op.rows = cnt * n;
  op.box_rows = BM;
  op.Kp = (n + BK - 1) / BK * BK;
  op.nb = 1;
  op.S = S;
  GC_TRY(op.exps.alloc(ctx, (size_t)op.rows));
  GC_TRY(op.buf.alloc(ctx, (size_t)op.rows * op.Kp * S));
  // two blocks per SM at least, where a matrix has the tiles for it
  const unsigned nt = op.Kp / 64, tiles = nt * (nt + 1) / 2;
  const dim3 grid(cnt, std::max(1u, std::min(gc::ceil_div(304, cnt), tiles)));
  const size_t sm = (size_t)n * sizeof(unsigned);
  constexpr size_t kMaxSm = 188 * 1024;  // n <= 48128, beyond the 46340 whose n^2 fits an int
  if (sm > kMaxSm) return gc::set_error(ctx, GC_EUNSUPPORTED, "packed operand: n=%d", n);
  auto kern = S == 4 ? k_oz_packed<4> : (S == 5 ? k_oz_packed<5> : k_oz_packed<6>);
  if (sm > 8 * 1024)
    GC_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSm));
  kern<<<grid, 256, sm, ctx->stream>>>(x, ld, n, op.Kp, cnt, op.exps.p, op.buf.p);
  GC_LAUNCHED(ctx);
  op.planes = op.buf.p;
  op.ex = op.exps.p;
  return encode_oz_map(ctx, op);
}

// A second view of src's slice planes with another TMA box height (src must outlive it).
int alias_oz_operand(gc_context *ctx, const OzOperand &src, OzOperand &op, int box_rows) {
  op.rows = src.rows;
  op.Kp = src.Kp;
  op.nb = src.nb;
  op.S = src.S;
  op.box_rows = box_rows;
  op.planes = src.planes;
  op.ex = src.ex;
  return encode_oz_map(ctx, op);
}

// alignment pad, stages, 2 * stages + 3 barriers, TMEM slot
constexpr size_t oz_smem_bytes(int S, int tbn) {
  return 1024 + oz_stages(S, tbn) * (size_t)S * (BM * OZ_BK * 2 + tbn * OZ_BK * 2) +
         (2 * oz_stages(S, tbn) + 3) * 8 + 16;
}
static_assert(oz_smem_bytes(4, 128) <= 232448 && oz_smem_bytes(5, 96) <= 232448 &&
                  oz_smem_bytes(6, 64) <= 232448,
              "sliced GEMM stages exceed the 227 KB of shared memory per CTA");
// 228 KB per SM, 1 KB of it reserved per CTA, and less than 1 KB of static shared memory each
static_assert(2 * (oz_smem_bytes(5, 48) + 2048) <= 233472 && 2 * (oz_smem_bytes(5, 32) + 2048) <= 233472,
              "the narrow tiles' two CTAs do not fit the shared memory of an SM");

// Time in us of one wave of tiles (152 CTAs, 304 of the 48-wide tile) for K = 64 kb: the
// pipeline's start and the epilogue, and the products. Measured on GB300 at 140454 x 153 for
// K = 64..2048, where the waves so come out within 9%. The 48-wide tile's two CTAs per SM run
// one's epilogue beside the other's products: the best of the widths up to K of about 300 with 5
// slices and 500 with 4 (5 slices, K = 64: 137 us against 183 with 96 columns and 197 with 64;
// K = 256: 254, 260, 284; K = 512: 407, 356, 398), where the epilogue is longer than the products.
double oz_wave_us(int S, int tbn, double kb) {
  const bool s4 = S == 4;
  switch (tbn) {
    case 48: return s4 ? 7.0 + 1.68 * kb : 6.6 + 2.57 * kb;
    case 64: return s4 ? 7.2 + 1.08 * kb : 7.5 + 1.42 * kb;
    case 96: return s4 ? 9.6 + 1.43 * kb : 10.3 + 1.93 * kb;
    default: return 12.3 + 1.61 * kb;
  }
}

// Tile width for an M x N x K x nbatch product: the one whose waves of CTAs finish first by the
// times above. tri: only the tiles that reach the lower triangle of an M x M product are
// computed (N = M). Products of at most 32 columns take the 32-wide tile, and six slices 64 columns
// otherwise: two CTAs of 48 would not fit TMEM, and 32 columns are slower unless the product leaves most
// SMs idle (140454 x 153 x 256: 334 us with 64, 388 with 32; 6290 x 6290 x 249: 511, 700; but
// 512^3: 25 and 19).
int oz_tile(const gc_context *ctx, int S, long long M, long long N, long long K, long long nbatch,
            bool tri = false) {
  const int widest = oz_max_tile(S);
  if (ctx->oz_tile > 0) return std::min(ctx->oz_tile, widest);
  if (N <= 32 && !tri) return 32;
  if (widest == 64) return 64;
  int best = 0;
  double best_us = 0.0;
  for (int tbn : {64, 48, 96, 128}) {
    if (tbn > widest) continue;
    const long long ntm = (M + BM - 1) / BM, ntn = (N + tbn - 1) / tbn;
    long long ctas = ntm * ntn;
    if (tri) {
      ctas = 0;
      for (long long i = 0; i < ntm; ++i) ctas += std::min(ntn, (std::min((i + 1) * BM, M) + tbn - 1) / tbn);
    }
    const int per_wave = tbn == 48 ? 304 : 152;
    const double us = (double)((ctas * nbatch + per_wave - 1) / per_wave) *
                      oz_wave_us(S, tbn, (double)((K + BK - 1) / BK));
    if (best == 0 || us < best_us) {
      best = tbn;
      best_us = us;
    }
  }
  return best;
}

template <int S, int TBN, bool GRAM = false>
int launch_oz(gc_context *ctx, const OzOperand &A, const OzOperand &B, int M, int N, int nbatch,
              const OzPlan &pl, const OzEpi &epi) {
  // on every call: the setting holds for one device
  GC_CUDA(ctx, cudaFuncSetAttribute(k_tc_gemm_oz<S, TBN, GRAM>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)oz_smem_bytes(S, TBN)));
  dim3 grid(gc::ceil_div(M, BM), gc::ceil_div(N, TBN), nbatch);
  k_tc_gemm_oz<S, TBN, GRAM><<<grid, oz_threads(TBN), oz_smem_bytes(S, TBN), ctx->stream>>>(
      A.map, B.map, M, N, A.Kp / OZ_BK, A.nb > 1 ? 1 : 0, B.nb > 1 ? 1 : 0, pl, epi, ctx->dev_flag,
      ctx->wait_ns);
  GC_LAUNCHED(ctx);
  return GC_OK;
}

constexpr int kGramTile = 64;

// The B operand's TMA box height is the column tile width of the launch.
int run_oz(gc_context *ctx, const OzOperand &A, const OzOperand &B, int M, int N, int nbatch,
           const OzPlan &pl, OzEpi epi) {
  if (A.Kp != B.Kp) return gc::set_error(ctx, GC_EINVAL, "oz_gemm: K mismatch");
  epi.ea = A.ex;
  epi.eb = B.ex;
  epi.ea_sb = A.nb > 1 ? A.rows : 0;
  epi.eb_sb = B.nb > 1 ? B.rows : 0;
  const int w = B.box_rows;
  if (epi.mode == 1) {  // one width: S + 1 accumulators of 96 columns would not fit TMEM for S = 5
    if (pl.S == 6) return launch_oz<6, kGramTile, true>(ctx, A, B, M, N, nbatch, pl, epi);
    if (pl.S == 5) return launch_oz<5, kGramTile, true>(ctx, A, B, M, N, nbatch, pl, epi);
    return launch_oz<4, kGramTile, true>(ctx, A, B, M, N, nbatch, pl, epi);
  }
  if (pl.S == 6 && w == 32) return launch_oz<6, 32>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 5 && w == 32) return launch_oz<5, 32>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 4 && w == 32) return launch_oz<4, 32>(ctx, A, B, M, N, nbatch, pl, epi);
  if (w == 48) {
    if (pl.S == 5) return launch_oz<5, 48>(ctx, A, B, M, N, nbatch, pl, epi);
    if (pl.S == 4) return launch_oz<4, 48>(ctx, A, B, M, N, nbatch, pl, epi);
  }
  if (pl.S == 6 && w == 64) return launch_oz<6, 64>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 5 && w == 64) return launch_oz<5, 64>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 5 && w == 96) return launch_oz<5, 96>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 4 && w == 64) return launch_oz<4, 64>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 4 && w == 96) return launch_oz<4, 96>(ctx, A, B, M, N, nbatch, pl, epi);
  if (pl.S == 4 && w == 128) return launch_oz<4, 128>(ctx, A, B, M, N, nbatch, pl, epi);
  return gc::set_error(ctx, GC_EINVAL, "oz_gemm: no kernel for %d slices and tile %d", pl.S, w);
}

}  // namespace

namespace gc {

int check_flag(gc_context *ctx) {
  int flag = 0;
  GC_CUDA(ctx, cudaMemcpyAsync(&flag, ctx->dev_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (flag) {
    GC_CUDA(ctx, cudaMemsetAsync(ctx->dev_flag, 0, sizeof(int), ctx->stream));
    return gc::set_error(ctx, GC_ETIMEOUT, "tc_gemm: a bounded mbarrier wait expired");
  }
  return GC_OK;
}

int tc_half_packed(gc_context *ctx, int precision, int n, int cnt, const double *M, long long ld,
                   int nhalf, const HalfOut *half) {
  if (!is_oz(precision))
    return set_error(ctx, GC_EINVAL, "half_packed: needs a sliced FP64-accurate precision");
  const OzPlan pl = oz_plan(precision);
  // The matrices of a chunk have at most 1 GiB of slice planes (and fit the row counts).
  const long long per = (long long)n * ((n + BK - 1) / BK * BK) * 2 * pl.S;
  const int cs = (int)std::max<long long>(
      1, std::min<long long>({(long long)cnt, (1ll << 30) / per, 0x7fffffffll / ((long long)n * n),
                              65535ll}));
  struct Side {
    OzOperand first, second;  // the block contracted first (GEMM B) and the other one
  };
  std::vector<std::unique_ptr<Side>> side;
  for (int h = 0; h < nhalf; ++h) {
    const HalfOut &o = half[h];
    side.push_back(std::make_unique<Side>());
    // M_k is symmetric: the narrower block is contracted first, n x min(nX, nY) instead of
    // n x nX intermediate columns (FOFO at n = 249, nocc = 28: 5 times fewer products).
    const bool y1 = o.nY <= o.nX;
    const int nf = y1 ? o.nY : o.nX;
    GC_TRY(make_oz_operand(ctx, side[h]->first, y1 ? o.CY : o.CX, nf, n, 1, n, 1, 0, pl.S,
                           oz_tile(ctx, pl.S, (long long)n * cs, nf, n, 1)));
    if (y1)
      GC_TRY(make_oz_operand(ctx, side[h]->second, o.CX, o.nX, n, 1, n, 1, 0, pl.S, BM));
    else
      GC_TRY(make_oz_operand(ctx, side[h]->second, o.CY, o.nY, n, 1, n, 1, 0, pl.S,
                             oz_tile(ctx, pl.S, o.nX, o.nY, n, cs)));
  }
  for (int k0 = 0; k0 < cnt; k0 += cs) {
    const int c = std::min(cs, cnt - k0);
    OzOperand A;
    GC_TRY(make_oz_packed(ctx, A, M + k0 * ld, ld, n, c, pl.S));
    for (int h = 0; h < nhalf; ++h) {
      const HalfOut &o = half[h];
      const bool y1 = o.nY <= o.nX;
      const int nf = y1 ? o.nY : o.nX;
      double *out = o.out + (long long)k0 * o.nX * o.nY;
      DevBuf<double> T;  // T[(k, p) + f (c n)] = sum_q M_k[p, q] C_first[q, f]
      GC_TRY(T.alloc(ctx, (size_t)c * n * nf));
      OzEpi e{0, T.p, (long long)c * n, 0, nullptr, nullptr, nullptr, nullptr, 0, 0};
      GC_TRY(run_oz(ctx, A, side[h]->first, c * n, nf, 1, pl, e));
      OzOperand B;
      if (y1) {
        // out[x + nX (y + nY k)] = sum_p CX[p, x] T[(k, p), y]: one product, columns (k, y)
        GC_TRY(make_oz_operand(ctx, B, T.p, nf, n, c, (long long)c * n, 1, n, pl.S,
                               oz_tile(ctx, pl.S, o.nX, (long long)c * nf, n, 1)));
        B.rows = c * nf;
        B.nb = 1;
        GC_TRY(encode_oz_map(ctx, B));
        // a block with itself: x <= y is all that tc_pair_product reads
        const bool sym = o.sym;
        OzEpi e2{0, out, o.nX, 0, nullptr, nullptr, nullptr, nullptr, 0, 0, sym ? nf : 0, sym ? 1 : 0};
        GC_TRY(run_oz(ctx, side[h]->second, B, o.nX, c * nf, 1, pl, e2));
      } else {
        GC_TRY(make_oz_operand(ctx, B, T.p, nf, n, c, (long long)c * n, 1, n, pl.S, BM));
        OzEpi e2{0, out, o.nX, (long long)o.nX * o.nY, nullptr, nullptr, nullptr, nullptr, 0, 0};
        GC_TRY(run_oz(ctx, B, side[h]->second, o.nX, o.nY, c, pl, e2));
      }
    }
  }
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_pair_product(gc_context *ctx, int precision, int rank, int nC, int nD, bool symCD,
                    const double *Z, int nA, int nB, bool symAB, const double *Y, double *out) {
  if (!is_oz(precision))
    return set_error(ctx, GC_EINVAL, "pair_product: needs a sliced FP64-accurate precision");
  const OzPlan pl = oz_plan(precision);
  const int nCD = nC * nD, nAB = nA * nB;
  const int R = symCD ? nC * (nC + 1) / 2 : nCD, Q = symAB ? nA * (nA + 1) / 2 : nAB;
  const bool same = Y == Z && symAB == symCD;
  DevBuf<double> cp;
  double *C = out;
  if (symCD || symAB) {
    GC_TRY(cp.alloc(ctx, (size_t)R * Q));
    C = cp.p;
  }
  OzOperand a, b;
  GC_TRY(make_oz_operand(ctx, a, Z, R, rank, 1, 1, nCD, 0, pl.S, BM, symCD ? nC : 0));
  if (same) {  // symmetric: the lower triangle and its mirror image
    GC_TRY(alias_oz_operand(ctx, a, b, oz_tile(ctx, pl.S, R, Q, rank, 1, true)));
    OzEpi e{3, C, R, 0, nullptr, nullptr, nullptr, nullptr, 0, 0, R};
    GC_TRY(run_oz(ctx, a, b, R, Q, 1, pl, e));
  } else {
    GC_TRY(make_oz_operand(ctx, b, Y, Q, rank, 1, 1, nAB, 0, pl.S, oz_tile(ctx, pl.S, R, Q, rank, 1),
                           symAB ? nA : 0));
    OzEpi e{0, C, R, 0, nullptr, nullptr, nullptr, nullptr, 0, 0};
    GC_TRY(run_oz(ctx, a, b, R, Q, 1, pl, e));
  }
  if (C != out) {
    k_expand_pairs<<<dim3(ceil_div(nCD, 256), std::min(nAB, 65535)), 256, 0, ctx->stream>>>(
        C, R, nC, nD, symCD, nA, nB, symAB, out);
    GC_LAUNCHED(ctx);
  }
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_two_sided(gc_context *ctx, int precision, int n, int cnt, const double *M, int nX,
                 const double *CX, int nY, const double *CY, double *T1, double *out,
                 long long ostride) {
  int S;
  PassList pl = pass_list(precision, &S);
  // step 1: T1[(k,q), x] = sum_p M_k[p, q] CX[p, x]   (T1 column-major, ld = n*cnt)
  {
    Operand A, B;
    GC_TRY(make_operand(ctx, A, M, n * cnt, n, 1, n, 1, 0, S, BM));
    GC_TRY(make_operand(ctx, B, CX, nX, n, 1, n, 1, 0, S, BN_T));
    Epi e{0, T1, (long long)n * cnt, 0, nullptr, nullptr};
    GC_TRY(run_gemm(ctx, A, B, n * cnt, nX, 1, pl, e));
  }
  // step 2: out_k[x, y] = sum_q T1[(k,q), x] CY[q, y]   (batched over k)
  {
    Operand A, B;
    // A rows x, K = q: T1[(k*n + q) + x*(n*cnt)]
    GC_TRY(make_operand(ctx, A, T1, nX, n, cnt, (long long)n * cnt, 1, n, S, BM));
    GC_TRY(make_operand(ctx, B, CY, nY, n, 1, n, 1, 0, S, BN_T));
    Epi e{0, out, nX, ostride, nullptr, nullptr};
    GC_TRY(run_gemm(ctx, A, B, nX, nY, cnt, pl, e));
  }
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_gemm_nt(gc_context *ctx, int precision, int m, int n, int k, const double *A, int lda,
               const double *B, int ldb, double *C, int ldc) {
  if (precision == GC_PREC_FP64) {
    const double one = 1.0, zero = 0.0;
    GC_CUBLAS(ctx, cublasDgemm(ctx->cublas, CUBLAS_OP_N, CUBLAS_OP_T, m, n, k, &one, A, lda, B, ldb,
                               &zero, C, ldc));
    return GC_OK;
  }
  if (is_oz(precision)) {
    OzPlan pl = oz_plan(precision);
    OzOperand a, b;
    GC_TRY(make_oz_operand(ctx, a, A, m, k, 1, 1, lda, 0, pl.S, BM));
    GC_TRY(make_oz_operand(ctx, b, B, n, k, 1, 1, ldb, 0, pl.S, oz_tile(ctx, pl.S, m, n, k, 1)));
    OzEpi e{0, C, ldc, 0, nullptr, nullptr, nullptr, nullptr, 0, 0};
    GC_TRY(run_oz(ctx, a, b, m, n, 1, pl, e));
    return GC_OK;  // the device flag is read at the caller's next sync point
  }
  int S;
  PassList pl = pass_list(precision, &S);
  Operand a, b;
  // A (m x k) column-major: row i, k stride lda
  GC_TRY(make_operand(ctx, a, A, m, k, 1, 1, lda, 0, S, BM));
  GC_TRY(make_operand(ctx, b, B, n, k, 1, 1, ldb, 0, S, BN_T));
  Epi e{0, C, ldc, 0, nullptr, nullptr};
  GC_TRY(run_gemm(ctx, a, b, m, n, 1, pl, e));
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_gemm_strided(gc_context *ctx, int precision, int M, int N, int K, const double *A,
                    long long sam, long long sak, const double *B, long long sbn, long long sbk,
                    double *C, long long ldc) {
  if (precision == GC_PREC_FP64 || !is_oz(precision))
    return set_error(ctx, GC_EINVAL, "gemm_strided: needs a sliced FP64-accurate precision");
  OzPlan pl = oz_plan(precision);
  OzOperand a, b;
  GC_TRY(make_oz_operand(ctx, a, A, M, K, 1, sam, sak, 0, pl.S, BM));
  GC_TRY(make_oz_operand(ctx, b, B, N, K, 1, sbn, sbk, 0, pl.S, oz_tile(ctx, pl.S, M, N, K, 1)));
  OzEpi e{0, C, ldc, 0, nullptr, nullptr, nullptr, nullptr, 0, 0};
  GC_TRY(run_oz(ctx, a, b, M, N, 1, pl, e));
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_gemm_strided_lower(gc_context *ctx, int precision, int M, int N, int K, const double *A,
                          long long sam, long long sak, const double *B, long long sbn,
                          long long sbk, double *C, long long ldc, int period) {
  if (!is_oz(precision))
    return set_error(ctx, GC_EINVAL, "gemm_strided_lower: needs a sliced FP64-accurate precision");
  OzPlan pl = oz_plan(precision);
  OzOperand a, b;
  GC_TRY(make_oz_operand(ctx, a, A, M, K, 1, sam, sak, 0, pl.S, BM));
  GC_TRY(make_oz_operand(ctx, b, B, N, K, 1, sbn, sbk, 0, pl.S, oz_tile(ctx, pl.S, M, N, K, 1)));
  OzEpi e{0, C, ldc, 0, nullptr, nullptr, nullptr, nullptr, 0, 0, period};
  GC_TRY(run_oz(ctx, a, b, M, N, 1, pl, e));
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_syrk_sub_lower(gc_context *ctx, int precision, int M, int K, const double *P, long long sm,
                      long long sk, double *C, long long ldc, int nbatch, long long sb) {
  if (!is_oz(precision))
    return set_error(ctx, GC_EINVAL, "syrk_sub_lower: needs a sliced FP64-accurate precision");
  OzPlan pl = oz_plan(precision);
  OzOperand a, b;
  GC_TRY(make_oz_operand(ctx, a, P, M, K, nbatch, sm, sk, sb, pl.S, BM));
  GC_TRY(alias_oz_operand(ctx, a, b, oz_tile(ctx, pl.S, M, M, K, nbatch, true)));
  OzEpi e{2, C, ldc, nbatch > 1 ? sb : 0, nullptr, nullptr, nullptr, nullptr, 0, 0, M};
  GC_TRY(run_oz(ctx, a, b, M, M, nbatch, pl, e));
  return GC_OK;  // the device flag is read at the caller's next sync point
}

int tc_gram_dot(gc_context *ctx, int precision, int N, const double *Y, const double *eig, double lo,
                double hi, const double *Klow, double *sq, DevBuf<double> &part) {
  if (!is_oz(precision))
    return set_error(ctx, GC_EINVAL, "gram_dot: needs a sliced FP64-accurate precision");
  const OzPlan pl = oz_plan(precision);
  OzOperand a, b;
  OzColsOpt opt;
  opt.eig = eig;
  opt.lo = lo;
  opt.hi = hi;
  opt.sq = sq;
  GC_TRY(make_oz_operand(ctx, a, Y, N, N, 1, 1, N, 0, pl.S, BM, 0, opt));
  GC_TRY(alias_oz_operand(ctx, a, b, kGramTile));
  GC_TRY(part.alloc(ctx, (size_t)ceil_div(N, BM) * ceil_div(N, b.box_rows)));
  OzEpi e{1, nullptr, N, 0, Klow, part.p, nullptr, nullptr, 0, 0, N};
  return run_oz(ctx, a, b, N, N, 1, pl, e);
}

int tc_dot_gemm(gc_context *ctx, int precision, int N, const double *Ksym, const double *Y,
                double *result) {
  int S;
  PassList pl = pass_list(precision, &S);
  Operand a, b;
  // rows i of the symmetric Kt (= its columns), rows nu of Y^T (= columns of Y)
  GC_TRY(make_operand(ctx, a, Ksym, N, N, 1, N, 1, 0, S, BM));
  GC_TRY(make_operand(ctx, b, Y, N, N, 1, N, 1, 0, S, BN_T));
  size_t ncta = (size_t)ceil_div(N, BM) * ceil_div(N, BN_T);
  DevBuf<double> part;
  GC_TRY(part.alloc(ctx, ncta));
  Epi e{1, nullptr, N, 0, Y, part.p};
  GC_TRY(run_gemm(ctx, a, b, N, N, 1, pl, e));
  std::vector<double> h(ncta);
  GC_CUDA(ctx, cudaMemcpyAsync(h.data(), part.p, ncta * sizeof(double), cudaMemcpyDeviceToHost,
                               ctx->stream));
  GC_TRY(check_flag(ctx));
  double s = 0.0;
  for (double v : h) s += v;
  *result = s;
  return GC_OK;
}

}  // namespace gc

extern "C" int gc_tc_gemm_nt(gc_context *ctx, int precision, int m, int n, int k, const double *A,
                             int lda, const double *B, int ldb, double *C, int ldc) {
  if (!ctx) return GC_EINVAL;
  if (m <= 0 || n <= 0 || k <= 0 || lda < m || ldb < n || ldc < m || !A || !B || !C)
    return gc::set_error(ctx, GC_EINVAL, "tc_gemm_nt: bad arguments");
  GC_TRY(gc::tc_gemm_nt(ctx, precision, m, n, k, A, lda, B, ldb, C, ldc));
  return gc::check_flag(ctx);
}

// Deterministic operands for gc_tc_gemm_time: x = u 2^-k with u uniform in
// [-1, 1) and k in 0..19 from a hash of the element index, so that every row
// mixes magnitudes over six decades (what the slicing sees on real operands).
__global__ void k_fill_mixed(size_t n, unsigned long long seed, double *__restrict__ x) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull ^ seed;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    const double u = (double)(h >> 11) * 0x1.0p-53 * 2.0 - 1.0;
    x[i] = ldexp(u, -(int)((h >> 3) % 20));
  }
}

// CUDA event pair destroyed on every return path.
struct EventPair {
  cudaEvent_t a = nullptr, b = nullptr;
  ~EventPair() {
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
  }
};

extern "C" int gc_tc_gemm_time(gc_context *ctx, int precision, int m, int n, int k, int reps,
                               double *ms_per_launch) {
  if (!ctx) return GC_EINVAL;
  if (m <= 0 || n <= 0 || k <= 0 || reps <= 0 || !ms_per_launch ||
      (precision != GC_PREC_BF16X3 && precision != GC_PREC_BF16X6 && !is_oz(precision)))
    return gc::set_error(ctx, GC_EINVAL, "tc_gemm_time: bad arguments");
  gc::DevBuf<double> a, b, c;
  GC_TRY(a.alloc(ctx, (size_t)m * k));
  GC_TRY(b.alloc(ctx, (size_t)n * k));
  GC_TRY(c.alloc(ctx, (size_t)m * n));
  k_fill_mixed<<<152 * 8, 256, 0, ctx->stream>>>((size_t)m * k, 0x1234567ull, a.p);
  GC_LAUNCHED(ctx);
  k_fill_mixed<<<152 * 8, 256, 0, ctx->stream>>>((size_t)n * k, 0x7654321ull, b.p);
  GC_LAUNCHED(ctx);
  EventPair ev;
  GC_CUDA(ctx, cudaEventCreate(&ev.a));
  GC_CUDA(ctx, cudaEventCreate(&ev.b));
  float ms = 0.f;
  if (is_oz(precision)) {
    OzPlan pl = oz_plan(precision);
    OzOperand A, B;
    GC_TRY(make_oz_operand(ctx, A, a.p, m, k, 1, k, 1, 0, pl.S, BM));
    GC_TRY(make_oz_operand(ctx, B, b.p, n, k, 1, k, 1, 0, pl.S, oz_tile(ctx, pl.S, m, n, k, 1)));
    OzEpi e{0, c.p, m, 0, nullptr, nullptr, nullptr, nullptr, 0, 0};
    GC_TRY(run_oz(ctx, A, B, m, n, 1, pl, e));  // warm-up
    GC_CUDA(ctx, cudaEventRecord(ev.a, ctx->stream));
    for (int r = 0; r < reps; ++r) GC_TRY(run_oz(ctx, A, B, m, n, 1, pl, e));
    GC_CUDA(ctx, cudaEventRecord(ev.b, ctx->stream));
    GC_CUDA(ctx, cudaEventSynchronize(ev.b));
    GC_CUDA(ctx, cudaEventElapsedTime(&ms, ev.a, ev.b));
  } else {
    int S;
    PassList pl = pass_list(precision, &S);
    Operand A, B;
    GC_TRY(make_operand(ctx, A, a.p, m, k, 1, k, 1, 0, S, BM));
    GC_TRY(make_operand(ctx, B, b.p, n, k, 1, k, 1, 0, S, BN_T));
    Epi e{0, c.p, m, 0, nullptr, nullptr};
    GC_TRY(run_gemm(ctx, A, B, m, n, 1, pl, e));  // warm-up
    GC_CUDA(ctx, cudaEventRecord(ev.a, ctx->stream));
    for (int r = 0; r < reps; ++r) GC_TRY(run_gemm(ctx, A, B, m, n, 1, pl, e));
    GC_CUDA(ctx, cudaEventRecord(ev.b, ctx->stream));
    GC_CUDA(ctx, cudaEventSynchronize(ev.b));
    GC_CUDA(ctx, cudaEventElapsedTime(&ms, ev.a, ev.b));
  }
  *ms_per_launch = ms / reps;
  return gc::check_flag(ctx);
}
