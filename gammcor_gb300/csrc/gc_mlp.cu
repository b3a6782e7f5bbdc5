// Integrand surrogate: a multilayer perceptron with hand-written training and
// inference kernels.
//
// Layers: in -> H -> H -> H -> out, GELU after every hidden layer. The forward
// pass reads BF16 copies of the weights and accumulates in FP32; training keeps
// FP32 master weights and Adam moments and refreshes the BF16 copies after every
// step.
//
// A step of the surrogate's sizes (batches of some hundred rows, 256 units) is bound by launches
// and by the latency of its chain of layers, not by its 0.2 GFLOP. Layers up to kFusedWidth
// units therefore take two kernels: k_mlp_rows carries a few rows through all layers forward and,
// in training, the loss and the data gradient back (everything of a row is local to it, the
// activations stay in shared memory); k_mlp_dw forms all weight and bias gradients and
// applies Adam to them. Wider layers, whose weights every block of k_mlp_rows would read
// again, go through one tiled shared-memory kernel
//   C[m, n] = sum_k A(m, k) B(n, k)   (A, B with arbitrary strides, B in BF16 or FP32)
// per product.
//
// Parameter layout (flattened FP32): W1 (H x in), b1 (H), W2 (H x H), b2,
// W3 (H x H), b3, W4 (out x H), b4; W row-major (row = output unit).
#include <cuda_bf16.h>

#include <cmath>
#include <random>

#include "gc_internal.cuh"

struct gc_mlp {
  int in = 0, hid = 0, out = 0;
  int nlayer = 4;
  size_t nparam = 0;
  size_t woff[4], boff[4];
  int din[4], dout[4];
  gc::DevBuf<float> master, grad, m1, m2;
  gc::DevBuf<__nv_bfloat16> wbf;  // BF16 copy of the whole parameter vector
  gc::DevBuf<float> act;           // activations / pre-activations for the largest batch seen
  int act_batch = 0;
  gc::DevBuf<float> lossbuf;       // loss partials of the row blocks, then the loss
  long long step = 0;
};

namespace {

constexpr int T = 16;  // tile edge of the product kernel

__device__ __forceinline__ float load_el(const float *p, long long i) { return p[i]; }
__device__ __forceinline__ float load_el(const __nv_bfloat16 *p, long long i) {
  return __bfloat162float(p[i]);
}

// C[m*ldc + n] (+)= sum_k A[m*sam + k*sak] * B[n*sbn + k*sbk] (+ bias[n]);
// act 1: also writes GELU(C) to H[m*ldc + n] (C keeps the pre-activation).
template <typename TB>
__global__ void k_prod(int M, int N, int K, const float *__restrict__ A, long long sam,
                       long long sak, const TB *__restrict__ B, long long sbn, long long sbk,
                       float *__restrict__ C, long long ldc, const float *__restrict__ bias,
                       int accumulate, int act, float *__restrict__ H) {
  __shared__ float as[T][T + 1], bs[T][T + 1];
  int tx = threadIdx.x, ty = threadIdx.y;
  int m = blockIdx.y * T + ty, n = blockIdx.x * T + tx;
  float acc = 0.f;
  for (int k0 = 0; k0 < K; k0 += T) {
    int ka = k0 + tx;
    as[ty][tx] = (m < M && ka < K) ? A[(long long)m * sam + (long long)ka * sak] : 0.f;
    int nb = blockIdx.x * T + ty;
    bs[ty][tx] = (nb < N && ka < K) ? load_el(B, (long long)nb * sbn + (long long)ka * sbk) : 0.f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < T; ++k) acc += as[ty][k] * bs[tx][k];
    __syncthreads();
  }
  if (m < M && n < N) {
    long long o = (long long)m * ldc + n;
    float v = acc + (bias ? bias[n] : 0.f);
    if (accumulate) v += C[o];
    C[o] = v;
    if (act) H[o] = 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
  }
}

// dZ = dH * GELU'(Z)
__global__ void k_gelu_bwd(long long total, const float *__restrict__ Z, const float *__restrict__ dH,
                           float *__restrict__ dZ) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    float z = Z[t];
    float g = 0.5f * (1.f + erff(z * 0.70710678118654752f)) +
              z * 0.3989422804014327f * expf(-0.5f * z * z);
    dZ[t] = dH[t] * g;
  }
}

// db[n] = sum_m dZ[m, n]
__global__ void k_colsum(int M, int N, const float *__restrict__ dZ, float *__restrict__ db) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float s = 0.f;
  for (int m = 0; m < M; ++m) s += dZ[(long long)m * N + n];
  db[n] = s;
}

// MSE: loss partials and dY = 2 (Y - T) / (M N)
__global__ void k_mse(long long total, float inv, const float *__restrict__ Y,
                      const float *__restrict__ Tt, float *__restrict__ dY, float *__restrict__ part) {
  __shared__ float red[256];
  float s = 0.f;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    float d = Y[t] - Tt[t];
    s += d * d;
    dY[t] = 2.f * d * inv;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_adam(long long n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, __nv_bfloat16 *__restrict__ wbf) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    float gt = g[t];
    float mt = b1 * m[t] + (1.f - b1) * gt;
    float vt = b2 * v[t] + (1.f - b2) * gt * gt;
    m[t] = mt;
    v[t] = vt;
    float wt = w[t] - lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    w[t] = wt;
    wbf[t] = __float2bfloat16(wt);
  }
}

__global__ void k_to_bf16(long long n, const float *__restrict__ w, __nv_bfloat16 *__restrict__ o) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    o[t] = __float2bfloat16(w[t]);
}

// Layer table of a network as the fused kernels read it.
struct Layers {
  int din[4], dout[4];
  long long woff[4], boff[4];
  float *h[4];   // inputs of layers 1..3 kept for the weight gradient (h[l]: output of layer l)
  float *dz[4];  // dL/dZ of every layer
};

constexpr int kFusedWidth = 256;   // widest layer of the fused kernels: one unit per thread
constexpr int kRowThreads = 256, kRowWarps = kRowThreads / 32;

__device__ __forceinline__ float gelu(float v) { return 0.5f * v * (1.f + erff(v * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.3989422804014327f * expf(-0.5f * z * z);
}

// Layer weights in shared memory: row o (BF16) at w + o * ld. Rows of a multiple of 8 weights on
// 16-byte boundaries are copied 16 bytes at a time with all copies in flight, and padded by
// 16 bytes, so that a thread per row reads 16 bytes without bank conflicts (vec).
struct Staged {
  const __nv_bfloat16 *w;
  int ld;
  bool vec;
};
__device__ __forceinline__ Staged stage_weights(const __nv_bfloat16 *w, int din, int dout,
                                                unsigned char *dst) {
  const bool vec = (din & 7) == 0 && ((uintptr_t)w & 15) == 0;
  const int ld = vec ? din + 8 : din;
  __syncthreads();  // the buffer's last readers
  if (vec) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n16 = din / 8;
    for (int c = threadIdx.x; c < dout * n16; c += kRowThreads) {
      const int o = c / n16, k = c - o * n16;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 2 * (o * ld + 8 * k)),
                   "l"(w + (size_t)o * din + 8 * k)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  } else {
    __nv_bfloat16 *p = reinterpret_cast<__nv_bfloat16 *>(dst);
#pragma unroll 4
    for (int c = threadIdx.x; c < dout * din; c += kRowThreads) p[c] = w[c];
  }
  __syncthreads();
  return {reinterpret_cast<const __nv_bfloat16 *>(dst), ld, vec};
}

// out[r][o] = sum_i in[r][i] W[o, i]: a thread per unit, the sum in one chain in the order of i
// (as the tiled kernel of wider layers adds it).
template <int R>
__device__ __forceinline__ void layer_forward(const float *in, int ld, const Staged &w, int din,
                                              int dout, float *out) {
  const int o = threadIdx.x;
  if (o >= dout) return;
  const __nv_bfloat16 *wo = w.w + o * w.ld;
  float acc[R] = {};
  if (w.vec) {
#pragma unroll 4
    for (int i = 0; i < din; i += 8) {
      const uint4 q = *reinterpret_cast<const uint4 *>(wo + i);
      const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 a = *reinterpret_cast<const float4 *>(in + r * ld + i);
        const float4 b = *reinterpret_cast<const float4 *>(in + r * ld + i + 4);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 8; ++k)
          acc[r] += v[k] * __uint_as_float((k & 1) ? u[k / 2] & 0xffff0000u : u[k / 2] << 16);
      }
    }
  } else {
#pragma unroll 4
    for (int i = 0; i < din; ++i) {
      const float wv = __bfloat162float(wo[i]);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] += in[r * ld + i] * wv;
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) out[r * ld + o] = acc[r];
}

// put(i, r, sum_o dz[r][o] W[o, i]): a thread per input, the sum in one chain in the order of o.
template <int R, class F>
__device__ __forceinline__ void layer_backward(const float *dz, int ld, const Staged &w, int din,
                                               int dout, F put) {
  const int i = threadIdx.x;
  if (i >= din) return;
  float acc[R] = {};
  int o = 0;
#pragma unroll 2
  for (; o + 4 <= dout; o += 4) {
    float wv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) wv[k] = __bfloat162float(w.w[(o + k) * w.ld + i]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 z = *reinterpret_cast<const float4 *>(dz + r * ld + o);
      acc[r] += z.x * wv[0];
      acc[r] += z.y * wv[1];
      acc[r] += z.z * wv[2];
      acc[r] += z.w * wv[3];
    }
  }
  for (; o < dout; ++o)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] += dz[r * ld + o] * __bfloat162float(w.w[o * w.ld + i]);
#pragma unroll
  for (int r = 0; r < R; ++r) put(i, r, acc[r]);
}

// R rows through all layers; with t also the loss partial and dL/dZ of every layer. The chain of
// layers is bound by latency, so each layer's weights come into shared memory with all copies in
// flight at once, and the arithmetic then reads shared memory and registers only. Measured at 256
// rows, 256 units: 33 us; a whole training step 221 -> 76 us with this and k_mlp_dw in
// place of 20 kernels.
template <int R>
constexpr size_t rows_smem() {  // weights, two activation buffers, pre-activations
  return 2 * (size_t)kFusedWidth * (kFusedWidth + 8) + sizeof(float) * kFusedWidth * R * (2 + 3);
}

template <int R>
__global__ void __launch_bounds__(kRowThreads)
    k_mlp_rows(int B, Layers L, const __nv_bfloat16 *__restrict__ W, const float *__restrict__ P,
               const float *__restrict__ x, const float *__restrict__ t, float inv,
               float *__restrict__ y, float *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int LD = kFusedWidth;
  float *cur = reinterpret_cast<float *>(sm + 2 * (size_t)LD * (LD + 8)), *nxt = cur + R * LD,
        *zs = nxt + R * LD;
  __shared__ float lred[kRowWarps], bias[4 * kFusedWidth];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * R, nr = min(R, B - b0);
  for (int e = tid; e < R * L.din[0]; e += kRowThreads) {
    const int r = e / L.din[0], i = e - r * L.din[0];
    cur[r * LD + i] = r < nr ? x[(long long)(b0 + r) * L.din[0] + i] : 0.f;
  }
  for (int l = 0; l < 4; ++l)
    if (tid < L.dout[l]) bias[l * LD + tid] = P[L.boff[l] + tid];
  Staged w{};
  for (int l = 0; l < 4; ++l) {
    const int din = L.din[l], dout = L.dout[l];
    w = stage_weights(W + L.woff[l], din, dout, sm);
    layer_forward<R>(cur, LD, w, din, dout, nxt);
    __syncthreads();
    for (int e = tid; e < R * dout; e += kRowThreads) {
      const int r = e / dout, o = e - r * dout;
      const float v = nxt[r * LD + o] + bias[l * LD + o];
      const float h = l == 3 ? v : gelu(v);
      nxt[r * LD + o] = h;
      if (l == 3) {
        if (r < nr && y) y[(long long)(b0 + r) * dout + o] = v;
      } else if (t) {
        zs[(l * R + r) * LD + o] = v;
        if (r < nr) L.h[l][(long long)(b0 + r) * dout + o] = h;
      }
    }
    __syncthreads();
    float *s = cur;
    cur = nxt;
    nxt = s;
  }
  if (!t) return;
  // loss partial and dL/dY
  const int nout = L.dout[3];
  float ls = 0.f;
  for (int e = tid; e < R * nout; e += kRowThreads) {
    const int r = e / nout, o = e - r * nout;
    float dv = 0.f;
    if (r < nr) {
      const float d = cur[r * LD + o] - t[(long long)(b0 + r) * nout + o];
      ls += d * d;
      dv = 2.f * d * inv;
      L.dz[3][(long long)(b0 + r) * nout + o] = dv;
    }
    cur[r * LD + o] = dv;
  }
  for (int off = 16; off > 0; off >>= 1) ls += __shfl_down_sync(0xffffffffu, ls, off);
  if (lane == 0) lred[warp] = ls;
  __syncthreads();
  if (tid == 0) {
    float v = 0.f;
    for (int k = 0; k < kRowWarps; ++k) v += lred[k];
    part[blockIdx.x] = v;
  }
  // dH = dZ W, dZ of the layer below = dH GELU'(Z); the last layer's weights are in place
  for (int l = 3; l >= 1; --l) {
    const int din = L.din[l], dout = L.dout[l];
    if (l < 3) w = stage_weights(W + L.woff[l], din, dout, sm);
    auto put = [&](int i, int r, float v) {
      const float g = v * gelu_grad(zs[((l - 1) * R + r) * LD + i]);
      nxt[r * LD + i] = g;
      if (r < nr) L.dz[l - 1][(long long)(b0 + r) * din + i] = g;
    };
    layer_backward<R>(cur, LD, w, din, dout, put);
    __syncthreads();
    float *s = cur;
    cur = nxt;
    nxt = s;
  }
}

struct AdamArgs {
  int on;  // 0: write the gradients
  float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void adam_one(const AdamArgs &a, long long k, float g, float *w, float *m,
                                         float *v, __nv_bfloat16 *wbf) {
  const float mt = a.b1 * m[k] + (1.f - a.b1) * g;
  const float vt = a.b2 * v[k] + (1.f - a.b2) * g * g;
  m[k] = mt;
  v[k] = vt;
  const float wt = w[k] - a.lr * (mt / a.c1) / (sqrtf(vt / a.c2) + a.eps);
  w[k] = wt;
  wbf[k] = __float2bfloat16(wt);
}

// dW_l[o, i] = sum_b dZ_l[b, o] in_l[b, i] and db_l[o] = sum_b dZ_l[b, o] of every layer, one
// 32 x 32 tile per block (first[l]: first block of layer l), followed by Adam or stored. Block
// 0 also turns the loss partials into the loss.
// All rows of a chunk are read at once, then each output is one chain of additions in the order
// of the rows (15 us at 256 rows, 256 units).
constexpr int kDwB = 256;  // rows per chunk
constexpr size_t kDwSmem = sizeof(float) * kDwB * (36 + 33);
__global__ void __launch_bounds__(256)
    k_mlp_dw(int B, Layers L, int4 first, const float *__restrict__ x, float *__restrict__ grad,
             float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
             __nv_bfloat16 *__restrict__ wbf, AdamArgs ad, int npart, float *__restrict__ lossbuf,
             double nout) {
  extern __shared__ __align__(16) float dws[];
  float *zt = dws, *at = dws + kDwB * 36;  // [row][36], [row][33]
  const int blk = blockIdx.x;
  const int l = blk >= first.w ? 3 : (blk >= first.z ? 2 : (blk >= first.y ? 1 : 0));
  const int t0 = blk - (l == 0 ? first.x : (l == 1 ? first.y : (l == 2 ? first.z : first.w)));
  const int din = L.din[l], dout = L.dout[l], nti = (din + 31) / 32;
  const int o0 = (t0 / nti) * 32, i0 = (t0 % nti) * 32;
  const float *dz = L.dz[l], *in = l == 0 ? x : L.h[l - 1];
  const int tid = threadIdx.x;
  const int tx = tid & 31, ty = tid >> 5;  // the thread's outputs: i0 + tx; o0 + 4 ty + k
  float acc[4] = {}, db = 0.f;
  for (int b = 0; b < B; b += kDwB) {
    const int nb = min(kDwB, B - b);
#pragma unroll 16
    for (int r = ty; r < nb; r += 8) {
      zt[r * 36 + tx] = o0 + tx < dout ? dz[(long long)(b + r) * dout + o0 + tx] : 0.f;
      at[r * 33 + tx] = i0 + tx < din ? in[(long long)(b + r) * din + i0 + tx] : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < nb; ++r) {
      const float a = at[r * 33 + tx];
      const float4 z = *reinterpret_cast<const float4 *>(zt + r * 36 + 4 * ty);
      acc[0] += z.x * a;
      acc[1] += z.y * a;
      acc[2] += z.z * a;
      acc[3] += z.w * a;
    }
    if (i0 == 0 && ty == 0)
#pragma unroll 8
      for (int r = 0; r < nb; ++r) db += zt[r * 36 + tx];
    __syncthreads();
  }
  auto put = [&](long long k, float g) {
    if (ad.on)
      adam_one(ad, k, g, w, m, v, wbf);
    else
      grad[k] = g;
  };
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int o = o0 + 4 * ty + k, i = i0 + tx;
    if (o < dout && i < din) put(L.woff[l] + (long long)o * din + i, acc[k]);
  }
  if (i0 == 0 && ty == 0 && o0 + tx < dout) put(L.boff[l] + o0 + tx, db);
  if (blk == 0 && ty == 1) {
    double s = 0.0;
    for (int k = tx; k < npart; k += 32) s += lossbuf[k];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (tx == 0) lossbuf[npart] = (float)(s / nout);
  }
}

template <typename TB>
int prod(gc_context *ctx, int M, int N, int K, const float *A, long long sam, long long sak,
         const TB *B, long long sbn, long long sbk, float *C, long long ldc, const float *bias,
         int accumulate, int act, float *H) {
  dim3 grid(gc::ceil_div(N, T), gc::ceil_div(M, T));
  k_prod<TB><<<grid, dim3(T, T), 0, ctx->stream>>>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, bias,
                                                   accumulate, act, H);
  GC_LAUNCHED(ctx);
  return GC_OK;
}

// activation workspace: per layer l: Z_l (B x dout), H_l (B x dout); plus dA, dB (B x max)
size_t layer_floats(const gc_mlp *m, int batch) {
  size_t s = 0;
  for (int l = 0; l < m->nlayer; ++l) s += 2 * (size_t)batch * m->dout[l];
  return s;
}

int max_width(const gc_mlp *m) { return std::max(std::max(m->in, m->hid), m->out); }

int ensure_act(gc_context *ctx, gc_mlp *m, int batch) {
  if (batch <= m->act_batch) return GC_OK;
  GC_TRY(m->act.alloc(ctx, layer_floats(m, batch) + 2 * (size_t)batch * max_width(m)));
  m->act_batch = batch;
  return GC_OK;
}

bool fused(const gc_mlp *m) { return max_width(m) <= kFusedWidth; }

// The layer table with H_l and dL/dZ_l in the activation workspace.
int fused_layers(gc_context *ctx, gc_mlp *m, int B, Layers &L) {
  GC_TRY(ensure_act(ctx, m, B));
  float *p = m->act.p;
  for (int l = 0; l < 4; ++l) {
    L.din[l] = m->din[l];
    L.dout[l] = m->dout[l];
    L.woff[l] = (long long)m->woff[l];
    L.boff[l] = (long long)m->boff[l];
    L.dz[l] = p;
    p += (size_t)m->act_batch * m->dout[l];
    L.h[l] = p;
    p += (size_t)m->act_batch * m->dout[l];
  }
  return GC_OK;
}

// Rows per block: 2 while that gives one block per SM at most (their shared memory leaves room for
// one), 4 above.
int fused_rows_per_block(int B) { return B <= 2 * 152 ? 2 : 4; }

// Forward of x (y), or with t the loss partials and dL/dZ of every layer too.
template <int R>
int fused_rows(gc_context *ctx, gc_mlp *m, int B, const Layers &L, const float *x, const float *t,
               float *y) {
  // on every call: the setting holds for one device
  GC_CUDA(ctx, cudaFuncSetAttribute(k_mlp_rows<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)rows_smem<R>()));
  k_mlp_rows<R><<<gc::ceil_div(B, R), kRowThreads, rows_smem<R>(), ctx->stream>>>(
      B, L, m->wbf.p, m->master.p, x, t, 1.f / (float)((long long)B * m->out), y, m->lossbuf.p);
  GC_LAUNCHED(ctx);
  return GC_OK;
}
int fused_rows(gc_context *ctx, gc_mlp *m, int B, const Layers &L, const float *x, const float *t,
               float *y) {
  return fused_rows_per_block(B) == 2 ? fused_rows<2>(ctx, m, B, L, x, t, y)
                                      : fused_rows<4>(ctx, m, B, L, x, t, y);
}

// Loss (host, when asked for) and gradient of one batch, stored (ad.on = 0) or applied.
int fused_step(gc_context *ctx, gc_mlp *m, int B, const float *x, const float *t, float *loss,
               const AdamArgs &ad) {
  Layers L;
  GC_TRY(fused_layers(ctx, m, B, L));
  const int nblk = gc::ceil_div(B, fused_rows_per_block(B));
  if (m->lossbuf.n < (size_t)nblk + 1) GC_TRY(m->lossbuf.alloc(ctx, nblk + 1));
  GC_TRY(fused_rows(ctx, m, B, L, x, t, nullptr));
  int first[5] = {0};
  for (int l = 0; l < 4; ++l)
    first[l + 1] = first[l] + (int)(gc::ceil_div(L.dout[l], 32) * gc::ceil_div(L.din[l], 32));
  GC_CUDA(ctx, cudaFuncSetAttribute(k_mlp_dw, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kDwSmem));
  k_mlp_dw<<<first[4], 256, kDwSmem, ctx->stream>>>(B, L, make_int4(first[0], first[1], first[2], first[3]), x,
                                              m->grad.p, m->master.p, m->m1.p, m->m2.p, m->wbf.p, ad,
                                              nblk, m->lossbuf.p, (double)B * m->out);
  GC_LAUNCHED(ctx);
  if (loss) {
    GC_CUDA(ctx, cudaMemcpyAsync(loss, m->lossbuf.p + nblk, sizeof(float), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return GC_OK;
}

// Forward through all layers; Z_l and H_l (H of the last layer = output) kept in act.
int forward(gc_context *ctx, gc_mlp *m, int B, const float *x, float **Z, float **H) {
  GC_TRY(ensure_act(ctx, m, B));
  float *p = m->act.p;
  const int stride = m->act_batch;
  for (int l = 0; l < m->nlayer; ++l) {
    Z[l] = p;
    p += (size_t)stride * m->dout[l];
    H[l] = p;
    p += (size_t)stride * m->dout[l];
  }
  const float *in = x;
  for (int l = 0; l < m->nlayer; ++l) {
    const bool last = l == m->nlayer - 1;
    GC_TRY(prod(ctx, B, m->dout[l], m->din[l], in, m->din[l], 1, m->wbf.p + m->woff[l],
                (long long)m->din[l], 1, last ? H[l] : Z[l], m->dout[l], m->master.p + m->boff[l],
                0, last ? 0 : 1, H[l]));
    in = H[l];
  }
  return GC_OK;
}

// Loss and gradient of the FP32 master parameters for one batch.
int loss_grad(gc_context *ctx, gc_mlp *m, int B, const float *x, const float *t, float *loss) {
  float *Z[4], *H[4];
  GC_TRY(forward(ctx, m, B, x, Z, H));
  float *dA = m->act.p + layer_floats(m, m->act_batch);
  float *dB = dA + (size_t)m->act_batch * max_width(m);
  const long long nout = (long long)B * m->out;
  const int nb = 64;
  gc::DevBuf<float> part;
  GC_TRY(part.alloc(ctx, nb));
  k_mse<<<nb, 256, 0, ctx->stream>>>(nout, 1.f / (float)nout, H[m->nlayer - 1], t, dA, part.p);
  GC_LAUNCHED(ctx);
  // dA holds dL/dZ of the current layer (the last layer has no activation)
  for (int l = m->nlayer - 1; l >= 0; --l) {
    const float *inp = l == 0 ? x : H[l - 1];
    // dW_l[o, i] = sum_b dZ[b, o] inp[b, i]
    GC_TRY(prod(ctx, m->dout[l], m->din[l], B, dA, 1, m->dout[l], inp, 1, m->din[l],
                m->grad.p + m->woff[l], m->din[l], nullptr, 0, 0, nullptr));
    k_colsum<<<gc::ceil_div(m->dout[l], 128), 128, 0, ctx->stream>>>(B, m->dout[l], dA,
                                                                      m->grad.p + m->boff[l]);
    GC_LAUNCHED(ctx);
    if (l == 0) break;
    // dH_{l-1}[b, i] = sum_o dZ[b, o] W_l[o, i]
    GC_TRY(prod(ctx, B, m->din[l], m->dout[l], dA, m->dout[l], 1, m->wbf.p + m->woff[l], 1,
                m->din[l], dB, m->din[l], nullptr, 0, 0, nullptr));
    long long tot = (long long)B * m->din[l];
    k_gelu_bwd<<<std::min<unsigned>(gc::ceil_div(tot, 256), 4096u), 256, 0, ctx->stream>>>(
        tot, Z[l - 1], dB, dA);
    GC_LAUNCHED(ctx);
  }
  if (loss) {
    float hp[nb];
    GC_CUDA(ctx, cudaMemcpyAsync(hp, part.p, sizeof hp, cudaMemcpyDeviceToHost, ctx->stream));
    GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    double s = 0;
    for (int i = 0; i < nb; ++i) s += hp[i];
    *loss = (float)(s / (double)nout);
  }
  return GC_OK;
}

}  // namespace

extern "C" {

int gc_mlp_create(gc_context *ctx, int in_dim, int hidden, int out_dim, unsigned long long seed,
                  gc_mlp **out) {
  if (!ctx || !out || in_dim <= 0 || hidden <= 0 || out_dim <= 0) return GC_EINVAL;
  gc_mlp *m = new gc_mlp();
  m->in = in_dim;
  m->hid = hidden;
  m->out = out_dim;
  int dims[5] = {in_dim, hidden, hidden, hidden, out_dim};
  size_t off = 0;
  for (int l = 0; l < 4; ++l) {
    m->din[l] = dims[l];
    m->dout[l] = dims[l + 1];
    m->woff[l] = off;
    off += (size_t)dims[l] * dims[l + 1];
    m->boff[l] = off;
    off += dims[l + 1];
  }
  m->nparam = off;
  std::vector<float> h(off, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < 4; ++l) {
    std::normal_distribution<float> nd(0.f, 1.f / std::sqrt((float)m->din[l]));
    for (size_t i = 0; i < (size_t)m->din[l] * m->dout[l]; ++i) h[m->woff[l] + i] = nd(rng);
  }
  int r;
  if ((r = m->master.upload(ctx, h.data(), off)) != GC_OK || (r = m->grad.alloc(ctx, off)) != GC_OK ||
      (r = m->m1.alloc(ctx, off)) != GC_OK || (r = m->m2.alloc(ctx, off)) != GC_OK ||
      (r = m->wbf.alloc(ctx, off)) != GC_OK) {
    delete m;
    return r;
  }
  cudaMemsetAsync(m->m1.p, 0, off * 4, ctx->stream);
  cudaMemsetAsync(m->m2.p, 0, off * 4, ctx->stream);
  k_to_bf16<<<gc::ceil_div(off, 256), 256, 0, ctx->stream>>>(off, m->master.p, m->wbf.p);
  ctx->launches++;
  *out = m;
  return GC_OK;
}

int gc_mlp_destroy(gc_mlp *m) {
  delete m;
  return GC_OK;
}

long long gc_mlp_num_params(const gc_mlp *m) { return m ? (long long)m->nparam : 0; }

int gc_mlp_set_params(gc_context *ctx, gc_mlp *m, const float *params_dev) {
  if (!ctx || !m || !params_dev) return GC_EINVAL;
  GC_CUDA(ctx, cudaMemcpyAsync(m->master.p, params_dev, m->nparam * 4, cudaMemcpyDeviceToDevice,
                               ctx->stream));
  k_to_bf16<<<gc::ceil_div(m->nparam, 256), 256, 0, ctx->stream>>>(m->nparam, m->master.p, m->wbf.p);
  GC_LAUNCHED(ctx);
  return GC_OK;
}

int gc_mlp_get_params(gc_context *ctx, gc_mlp *m, float *params_dev) {
  if (!ctx || !m || !params_dev) return GC_EINVAL;
  GC_CUDA(ctx, cudaMemcpyAsync(params_dev, m->master.p, m->nparam * 4, cudaMemcpyDeviceToDevice,
                               ctx->stream));
  return GC_OK;
}

int gc_mlp_forward(gc_context *ctx, gc_mlp *m, int batch, const float *x_dev, float *y_dev) {
  if (!ctx || !m || batch <= 0 || !x_dev || !y_dev) return GC_EINVAL;
  float *Z[4], *H[4];
  if (fused(m)) {
    Layers L;
    GC_TRY(fused_layers(ctx, m, batch, L));
    return fused_rows(ctx, m, batch, L, x_dev, nullptr, y_dev);
  }
  GC_TRY(forward(ctx, m, batch, x_dev, Z, H));
  GC_CUDA(ctx, cudaMemcpyAsync(y_dev, H[3], (size_t)batch * m->out * 4, cudaMemcpyDeviceToDevice,
                               ctx->stream));
  return GC_OK;
}

int gc_mlp_gradients(gc_context *ctx, gc_mlp *m, int batch, const float *x_dev, const float *t_dev,
                     float *grad_dev, float *loss_host) {
  if (!ctx || !m || batch <= 0 || !x_dev || !t_dev) return GC_EINVAL;
  if (fused(m))
    GC_TRY(fused_step(ctx, m, batch, x_dev, t_dev, loss_host, AdamArgs{}));
  else
    GC_TRY(loss_grad(ctx, m, batch, x_dev, t_dev, loss_host));
  if (grad_dev)
    GC_CUDA(ctx, cudaMemcpyAsync(grad_dev, m->grad.p, m->nparam * 4, cudaMemcpyDeviceToDevice,
                                 ctx->stream));
  return GC_OK;
}

int gc_mlp_train_step(gc_context *ctx, gc_mlp *m, int batch, const float *x_dev, const float *t_dev,
                      float lr, float *loss_host) {
  if (!ctx || !m || batch <= 0 || !x_dev || !t_dev || !(lr > 0.f)) return GC_EINVAL;
  const float b1 = 0.9f, b2 = 0.999f;
  if (fused(m)) {
    const float s = (float)(m->step + 1);
    GC_TRY(fused_step(ctx, m, batch, x_dev, t_dev, loss_host,
                      AdamArgs{1, lr, b1, b2, 1e-8f, 1.f - std::pow(b1, s), 1.f - std::pow(b2, s)}));
    m->step++;
    return GC_OK;
  }
  GC_TRY(loss_grad(ctx, m, batch, x_dev, t_dev, loss_host));
  m->step++;
  float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
  k_adam<<<std::min<unsigned>(gc::ceil_div(m->nparam, 256), 4096u), 256, 0, ctx->stream>>>(
      m->nparam, lr, b1, b2, 1e-8f, c1, c2, m->master.p, m->grad.p, m->m1.p, m->m2.p, m->wbf.p);
  GC_LAUNCHED(ctx);
  return GC_OK;
}

}  // extern "C"
