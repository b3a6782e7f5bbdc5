// ERPA A+B / A-B assembly in gather form.
//
// AB_CAS_FOFO (abfofo.f90:8-293) streams FOFO and FFOO records through
// JK_loop (abfofo.f90:4468-5053) and scatters contributions into
// ABPLUS(ipq,irs). Here every output element (ipq, irs) is computed by one
// thread from closed forms of the same terms:
//   * integral terms read FOFO / FFOO elements directly,
//   * the 2-RDM terms T1..T6 read small intermediates Z (sums over two
//     active indices of an integral times RDM2val) built once per system,
//   * the one-body part reads HNO, AuxI, AuxIO and WMAT (n x n), which the
//     reference accumulates in the same loops.
// Every coefficient is 1, lambda or (1 - lambda), so A+-B is affine in lambda.
#include <cmath>
#include <cstring>
#include <memory>

#include "gc_internal.cuh"

namespace {

// h(i, j): a full matrix (column-major), or the packed triangle (hpk).
__device__ __forceinline__ double one_el(const double *__restrict__ h, int hpk, int n, int i, int j) {
  if (!hpk) return h[i + (size_t)j * n];
  return i <= j ? h[i + (size_t)j * (j + 1) / 2] : h[j + (size_t)i * (i + 1) / 2];
}

struct Geo {
  int n, nin, nact, nocc;
};

// One pair A+-B of an assembly: what depends on lambda and the AB1 switch.
// AB1 = .false.: AuxCoeff = 1 for four equal groups, HNO kept inside a group with the
// (1 - lambda) inactive/active correction. AB1 = .true. (the lambda derivative,
// abfofo.f90:109-156 and HNOCoef, abfofo.f90:167-171, 4494-4500): AuxCoeff = 0 there,
// HNO zeroed inside a group and the correction taken with coefficient -1.
struct Setting {
  double lam;
  double same;   // AuxCoeff of four equal groups
  int ab1;
  double2 *ct;                        // ct[q + nocc s], see k_ab (nocc x nocc)
  double *hno, *auxi, *auxio, *wmat;  // n x n, column-major
  double *abp, *abm;
};
constexpr int kMaxSet = 2;
struct Settings {
  Setting s[kMaxSet];
};

__device__ __forceinline__ double Fofo(const double *__restrict__ f, const Geo &g, int a, int b,
                                       int c, int d) {  // (ab|cd), b, d < nocc
  size_t ld = (size_t)g.n * g.nocc;
  return f[(size_t)(a + (size_t)b * g.n) * ld + c + (size_t)d * g.n];
}
__device__ __forceinline__ double Ffoo(const double *__restrict__ f, const Geo &g, int a, int b,
                                       int c, int d) {  // (ab|cd), c, d < nocc
  size_t ld = (size_t)g.n * g.n;
  return f[(size_t)(c + (size_t)d * g.nocc) * ld + a + (size_t)b * g.n];
}
// AuxCoeff(g1,g2,g3,g4): st.same if the four orbital groups are equal, else lambda.
__device__ __forceinline__ double AC(const Setting &st, int a, int b, int c, int d) {
  return (a == b && b == c && c == d) ? st.same : st.lam;
}
// AuxInd(g1,g2) of AB_CAS_FOFO: 1 for inactive/active combinations other than
// active-active, 2 for active-active, 0 otherwise.
__device__ __forceinline__ int AuxInd(int a, int b) {
  if (a <= 1 && b <= 1) return (a == 1 && b == 1) ? 2 : 1;
  return 0;
}

// RDM2val(i, j, k, l) of active orbitals (abfofo.f90:84-92), indices within the active block.
__device__ __forceinline__ double RVa(const double *__restrict__ rv, int na, int i, int j, int k,
                                      int l) {
  return rv[i + na * (j + na * (k + (size_t)na * l))];
}

// The buffers between the two kernels of an assembly. The 2-RDM intermediates hold, per
// element, the part that enters A+B and A-B with one sign (x) and the part that enters them with
// opposite signs (y); nv = n - nin.
//   za[p, s, q, r]  x = -Z12            y = Z1[p,s,q,r] + Z11   (p >= nin, s < nocc; q, r active)
//   zb[r, q, p, s]  x = -Z6             y = Z1[r,q,p,s] + Z5    (r >= nin, q < nocc; p, s active)
//   zc[p, r, q, s]  x = Z4 + Z9         y = -Z7                 (p, r >= nin; q, s active)
//   zd[q, s, p, r]  x = Z8 + Z10        y = -Z13                (q, s < nocc; p, r active)
// with, over active t, u, k, l (capitals: their orbital indices):
//   Z1[a,b,c,d] = sum (ab|TU) RV[t,u,c,d]    Z4[p,r,q,s] = sum (rU|pT) RV[t,q,s,u]
//   Z5[r,q,p,s] = sum (rU|Tq) RV[t,p,s,u]    Z6[r,q,p,s] = sum (rU|Tq) RV[t,p,u,s]
//   Z7[p,r,q,s] = sum (rU|pT) RV[t,q,u,s]    Z8[q,s,p,r] = sum (TU|qs) RV[t,u,p,r]
//   Z9[p,r,q,s] = sum (pr|KL) RV[q,s,k,l]    Z10[q,s,p,r] = sum (Tq|sU) RV[t,p,r,u]
//   Z11[p,s,q,r] = sum (Tp|sU) RV[t,q,r,u]   Z12[p,s,q,r] = sum (Tp|sU) RV[t,q,u,r]
//   Z13[q,s,p,r] = sum (Tq|sU) RV[t,p,u,r]
struct Inter {
  double2 *za, *zb, *zc, *zd;
  double *part;  // kEtotWarps partial sums of E_CAS
};

constexpr int kEtotWarps = 256;

// Everything that the element kernel reads, in one launch: the parts do not depend on one
// another, and each of them alone is a short kernel that leaves most of the chip idle at
// small n. The unit of work is one warp: 32 consecutive values of the fastest index
// (coalesced along FOFO / FFOO records) for one value of the others, which are then uniform
// over the warp. Bound at large n by the FP64 pipe: 6 nact^2 FMAs per element of zc, and
// ten per element of za and zb. Measured at n = 249, nocc = 28, nact = 6: 0.53 ms (FP64 pipe
// 89%), against 1.14 ms for a kernel per part and a DGEMM with K = nocc^3 for WMAT; at n = 64
// 25 us, against 126 us.
struct InterWork {  // first warp of each part
  int wc, wab, wd, wone, wwm, wct, wet, end;
};

__global__ void __launch_bounds__(256)
    k_intermediates(Geo g, InterWork W, const double *__restrict__ h, int hpk,
                    const double *__restrict__ occ, const int *__restrict__ grp,
                    const double *__restrict__ fofo, const double *__restrict__ ffoo,
                    const double *__restrict__ rv, const __grid_constant__ Settings sets, Inter I) {
  const int lane = threadIdx.x & 31;
  const int n = g.n, nin = g.nin, na = g.nact, nocc = g.nocc, nv = n - nin;
  const size_t ldo = (size_t)n * nocc, ldf = (size_t)n * n;
  for (int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w < W.end;
       w += (int)((gridDim.x * blockDim.x) >> 5)) {
    if (w < W.wab) {  // zc
      const int ch = (nv + 31) / 32;
      int t0 = w;
      const int p = (t0 % ch) * 32 + lane + nin;
      t0 /= ch;
      const int r = t0 % nv + nin;
      t0 /= nv;
      const int q = t0 % na, s = t0 / na;
      if (p >= n) continue;
      double x = 0.0, y = 0.0;
      for (int u = 0; u < na; ++u) {
        // (rU|pT): record (r, U), element p + T n;  (pr|KL): record (K, L), element p + r n
        const double *fr = fofo + ((size_t)r + (size_t)(nin + u) * n) * ldo + p + (size_t)nin * n;
        const double *ff = ffoo + ((size_t)nin + (size_t)(nin + u) * nocc) * ldf + p + (size_t)r * n;
#pragma unroll 2
        for (int t = 0; t < na; ++t) {
          const double f = fr[(size_t)t * n];
          x += f * RVa(rv, na, t, q, s, u);
          y -= f * RVa(rv, na, t, q, u, s);
          x += ff[(size_t)t * ldf] * RVa(rv, na, q, s, t, u);
        }
      }
      I.zc[(p - nin) + (size_t)nv * ((r - nin) + (size_t)nv * (q + na * s))] = make_double2(x, y);
    } else if (w < W.wd) {  // za and zb at (a, b, c, d)
      const int ch = (nv + 31) / 32;
      int t0 = w - W.wab;
      const int a = (t0 % ch) * 32 + lane + nin;
      t0 /= ch;
      const int b = t0 % nocc;
      t0 /= nocc;
      const int c = t0 % na, d = t0 / na;
      if (a >= n) continue;
      double z1 = 0.0, z5 = 0.0, z6 = 0.0, z11 = 0.0, z12 = 0.0;
      for (int u = 0; u < na; ++u) {
        const int U = nin + u;
#pragma unroll 2
        for (int t = 0; t < na; ++t) {
          const int T = nin + t;
          const double rx = RVa(rv, na, t, c, d, u), ry = RVa(rv, na, t, c, u, d);
          z1 += Fofo(fofo, g, T, U, a, b) * RVa(rv, na, t, u, c, d);  // (ab|TU) as (TU|ab)
          const double f5 = Fofo(fofo, g, T, b, a, U);               // (rU|Tq) as (Tq|rU)
          z5 += f5 * rx;
          z6 += f5 * ry;
          const double f11 = Ffoo(ffoo, g, a, T, b, U);              // (Tp|sU) as (pT|sU)
          z11 += f11 * rx;
          z12 += f11 * ry;
        }
      }
      const size_t o = (a - nin) + (size_t)nv * (b + (size_t)nocc * (c + na * d));
      I.za[o] = make_double2(-z12, z1 + z11);
      I.zb[o] = make_double2(-z6, z1 + z5);
    } else if (w < W.wone) {  // zd
      const int ch = (nocc + 31) / 32;
      int t0 = w - W.wd;
      const int q = (t0 % ch) * 32 + lane;
      t0 /= ch;
      const int s = t0 % nocc;
      t0 /= nocc;
      const int p = t0 % na, r = t0 / na;
      if (q >= nocc) continue;
      double x = 0.0, y = 0.0;
      for (int u = 0; u < na; ++u)
#pragma unroll 2
        for (int t = 0; t < na; ++t) {
          const double f10 = Ffoo(ffoo, g, q, nin + t, s, nin + u);  // (Tq|sU) as (qT|sU)
          x += Fofo(fofo, g, nin + t, nin + u, q, s) * RVa(rv, na, t, u, p, r);
          x += f10 * RVa(rv, na, t, p, r, u);
          y -= f10 * RVa(rv, na, t, p, u, r);
        }
      I.zd[q + (size_t)nocc * (s + (size_t)nocc * (p + na * r))] = make_double2(x, y);
    } else if (w < W.wwm) {  // HNO, AuxI, AuxIO at (i, j)
      const int ch = (n + 31) / 32;
      const Setting &st = sets.s[(w - W.wone) / (ch * n)];
      const int t0 = (w - W.wone) % (ch * n);
      const int i = (t0 % ch) * 32 + lane, j = t0 / ch;
      if (i >= n) continue;
      const int gi = grp[i], gj = grp[j];
      const double hv = one_el(h, hpk, n, i, j);
      double corr = 0.0, ai = 0.0, aio = 0.0;
#pragma unroll 4
      for (int k = 0; k < nocc; ++k) {
        const int gk = grp[k];
        const double ok = occ[k];
        const double jv = Ffoo(ffoo, g, i, j, k, k);  // (ij|kk)
        const double kv = Fofo(fofo, g, j, k, i, k);  // (jk|ik)
        if (gi == gj && gk != gi) corr += ok * (2.0 * jv - kv);
        const double t = ok * (2.0 * AC(st, gi, gj, gk, gk) * jv - AC(st, gi, gi, gj, gk) * kv);
        ai += t;
        if (k < nin) aio += t;
      }
      const size_t o = i + (size_t)j * n;
      st.hno[o] = (gi != gj) ? st.lam * hv : (st.ab1 ? -corr : hv + (1.0 - st.lam) * corr);
      st.auxi[o] = ai;
      st.auxio[o] = aio;
    } else if (w < W.wct) {
      // WMAT(k, r) = sum_{i,j,l < nocc} AuxCoeff(k,l,i,j) (ij|kl) RDM2val(i,j,r,l), 0 for
      // r >= nocc. RDM2val(i,j,r,l) is 2 n_i n_r delta_ij delta_rl - n_i n_r delta_il delta_rj
      // unless i and r are both active (and only where one of n_i, n_r is 1), and the active
      // 2-RDM for four active orbitals: 2 nocc + nact^3 terms instead of nocc^3.
      const int ch = (n + 31) / 32;
      const Setting &st = sets.s[(w - W.wwm) / (ch * n)];
      const int t0 = (w - W.wwm) % (ch * n);
      const int k = (t0 % ch) * 32 + lane, r = t0 / ch;
      if (k >= n) continue;
      double v = 0.0;
      if (r < nocc) {
        const int gk = grp[k], gr = grp[r];
        const double nr = occ[r];
#pragma unroll 4
        for (int i = 0; i < nocc; ++i) {
          const double ni = occ[i];
          const int gi = grp[i];
          const double c = ((i >= nin && r >= nin) || !(ni == 1.0 || nr == 1.0)) ? 0.0 : ni * nr;
          v += c * (2.0 * AC(st, gk, gr, gi, gi) * Fofo(fofo, g, i, i, k, r) -
                    AC(st, gk, gi, gi, gr) * Fofo(fofo, g, i, r, k, i));
        }
        if (r >= nin) {
          const double c = AC(st, gk, 1, 1, 1);
          double a = 0.0;
#pragma unroll 8
          for (int t = 0; t < na * na * na; ++t) {  // flat: eight loads in flight
            const int i = t % na, j = (t / na) % na, l = t / (na * na);
            a += Fofo(fofo, g, nin + i, nin + j, k, nin + l) * RVa(rv, na, i, j, r - nin, l);
          }
          v += c * a;
        }
      }
      st.wmat[k + (size_t)r * n] = v;
    } else if (w < W.wet) {
      const int chc = (nocc * nocc + 31) / 32;
      const Setting &st = sets.s[(w - W.wct) / chc];
      const int t = (w - W.wct) % chc * 32 + lane;
      if (t >= nocc * nocc) continue;
      const int q = t % nocc, s = t / nocc;
      // C = sign(n - 1/2) sqrt(n); a sum or difference of 0 is not divided by
      auto ci = [&](int a) { return occ[a] >= 0.5 ? sqrt(occ[a]) : -sqrt(occ[a]); };
      const double cv = ci(n - 1), cq = ci(q), cs = ci(s);
      const double dp = (cv + cq) * (cv + cs), dm = (cv - cq) * (cv - cs);
      const double x = grp[q] + grp[s] <= 1 ? st.lam * (occ[q] * occ[s]) : 0.0;
      st.ct[t] = make_double2(dp != 0.0 ? x / dp : x, dm != 0.0 ? x / dm : x);
    } else {
      // E_CAS = 2 sum_i n_i h_ii + sum RDM2val(i,j,k,l) (ij|kl), kEtotWarps partial sums in a
      // fixed order. Every integral is read, also those with a zero RDM2val, so that a
      // non-finite one shows in the energy.
      const int e = w - W.wet;
      double v = 0.0;
      for (int i = e * 32 + lane; i < nocc; i += 32 * kEtotWarps)
        v += 2.0 * occ[i] * one_el(h, hpk, n, i, i);
      const unsigned o2 = (unsigned)nocc * nocc;
      for (unsigned rec = e; rec < o2; rec += kEtotWarps) {  // record (k, l), elements (i, j)
        const int k = rec % nocc, l = rec / nocc;
        const double *fr = ffoo + (size_t)rec * ldf;
#pragma unroll 4
        for (unsigned t = lane; t < o2; t += 32) {
          const int j = t / nocc, i = t - j * nocc;
          double c = 0.0;
          if (i >= nin && j >= nin && k >= nin && l >= nin) {
            c = RVa(rv, na, i - nin, j - nin, k - nin, l - nin);
          } else if ((i == j && k == l) || (i == l && k == j)) {
            const double ni = occ[i], nk = occ[k];
            if (ni == 1.0 || nk == 1.0)
              c = ((i == j && k == l) ? 2.0 * ni * nk : 0.0) - ((i == l && k == j) ? ni * nk : 0.0);
          }
          v += c * fr[i + (size_t)j * n];
        }
      }
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) I.part[e] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// A+B and A-B, element (row = pair i, column = pair j), column-major N x N.
//
// Bound by the FP64 pipe (2 FMAs per cycle per SM), then by the three gathers, so whatever is
// not a product of the element itself is kept off that pipe: groups, zero and NaN tests are
// integer work, the addresses are a row part (held by the thread over `cols` columns) plus a
// column part that is uniform over the warp. Nine in ten elements of a large system have p
// and r virtual and q, s not both active. There the element is
//   A+B = t (f2 - f3) / ((C_p + C_q)(C_r + C_s)),  A-B = t (4 f1 - f2 - f3) / ((C_p - C_q)(C_r - C_s))
// with t = lambda n_q n_s (0 beside an active pair), and as long as the virtual occupations
// are all the same (`vuni`) the factors depend on q and s alone: they come from the table ct,
// and the element takes 5 FP64 operations instead of 19. Measured at NDimX 6335: 0.73 ms,
// with the general form for every element 1.46 ms, without the row order and with the same
// conditional products for every element 2.10 ms.
// The rows go through `slot`, an order of the pairs in which a warp holds 8 consecutive p
// times 4 consecutive q of one pair of orbital groups: the branches are then uniform over
// almost every warp, the gathers use whole sectors (8 consecutive elements of a record) and
// so do the stores, whichever of p and q is the outer index of the caller's pair list.
constexpr int kAbWarps = 4;

__device__ __forceinline__ bool nonzero(double x) {
  return (__double_as_longlong(x) << 1) != 0;  // integer test: the FP64 pipe is the bound
}
__device__ __forceinline__ bool nonfinite(double x) {
  return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000;
}

__global__ void __launch_bounds__(32 * kAbWarps)
    k_ab(Geo g, int N, int cols, const int *__restrict__ slot, const int *__restrict__ pp,
         const int *__restrict__ pq, const double *__restrict__ occ, const int *__restrict__ grp,
         const double *__restrict__ fofo, const double *__restrict__ ffoo, Inter I,
         const __grid_constant__ Setting st, int vuni, const double *__restrict__ rpl,
         const double *__restrict__ rmi) {
  double *__restrict__ abp = st.abp, *__restrict__ abm = st.abm;
  const int sl = (blockIdx.x * kAbWarps + (threadIdx.x >> 5)) * 32 + (threadIdx.x & 31);
  if (sl >= N) return;
  const int i = slot[sl];
  const int n = g.n, nin = g.nin, nocc = g.nocc, na = g.nact, nv = n - nin;
  const size_t ldo = (size_t)n * nocc, ldf = (size_t)n * n;
  const int p = pp[i], q = pq[i], gp = grp[p], gq = grp[q];
  const double op = occ[p], oq = occ[q];
  const double ri_p = rpl[i], ri_m = rmi[i];
  const bool zi_p = nonzero(ri_p), zi_m = nonzero(ri_m);
  const bool pa = gp == 1, qa = gq == 1;
  const int pA = p - nin, qA = q - nin;
  const double *f1 = fofo + p + (size_t)q * n;        // (rs|pq): record (r, s)
  const double *f2 = fofo + (size_t)q * n * ldo + p;  // (rq|ps): record (r, q)
  const double *f3 = ffoo + (size_t)q * ldf + p;      // (pr|qs): record (q, s)
  // The assembly of the reference sums over every (ij|kl) with i, j, l occupied, most of them
  // with a zero coefficient. A non-finite one must still show in A+-B: each thread looks at its
  // share of them and adds a NaN to its elements where it finds one.
  bool bad = false;
  {
    const size_t rec = (size_t)n * nocc, cnt = (size_t)nocc * nocc * rec,
                 nth = (size_t)N * gridDim.y;
    for (size_t e = (size_t)blockIdx.y * N + sl; e < cnt; e += nth) {
      const size_t ij = e / rec;
      bad |= nonfinite(fofo[((ij % nocc) + (ij / nocc) * n) * ldo + (e - ij * rec)]);
    }
  }
  auto aux = [&](int ga, int gb, int x, int y) -> double {
    const int a = AuxInd(ga, gb);
    if (a == 1) return st.auxi[x + (size_t)y * n];
    if (a == 2) return st.auxio[x + (size_t)y * n];
    return 0.0;
  };
  const bool vrow = vuni && gp == 2;
  const int j1 = min(N, (int)(blockIdx.y + 1) * cols);
  for (int j = blockIdx.y * cols; j < j1; ++j) {
    const int r = pp[j], s = pq[j], gr = grp[r], gs = grp[s];
    const bool ra = gr == 1, sa = gs == 1;
    const double orr = occ[r], os = occ[s];
    const double rj_p = rpl[j], rj_m = rmi[j];
    const size_t o = i + (size_t)j * N;
    if (vrow && gr == 2 && !(qa && sa)) {
      const double2 k = st.ct[q + nocc * s];
      const double v1 = f1[((size_t)r + (size_t)s * n) * ldo], v2 = f2[(size_t)r * ldo + (size_t)s * n],
                   v3 = f3[(size_t)s * nocc * ldf + (size_t)r * n];
      double vp = k.x * (v2 - v3), vm = k.y * fma(4.0, v1, -(v2 + v3));
      if (p == r || q == s) {  // the one-body part (q = r and p = s cannot be)
        double ob = 0.0;
        if (p == r)
          ob = (op - os) * st.hno[q + (size_t)s * n] - st.wmat[q + (size_t)s * n] + op * aux(gp, gr, q, s);
        if (q == s)
          ob += (oq - orr) * st.hno[p + (size_t)r * n] - st.wmat[p + (size_t)r * n] + oq * aux(gq, gs, p, r);
        vp += (zi_p && nonzero(rj_p)) ? ob * (ri_p * rj_p) : ob;
        vm += (zi_m && nonzero(rj_m)) ? ob * (ri_m * rj_m) : ob;
      }
      abp[o] = bad ? __longlong_as_double(0x7ff8000000000000ll) : vp;
      abm[o] = bad ? __longlong_as_double(0x7ff8000000000000ll) : vm;
      continue;
    }
    // Every term enters A+B and A-B either with the same sign (S) or with opposite signs
    // (A); A+B = S + A, A-B = S - A + the Coulomb term Mo.
    double S = bad ? __longlong_as_double(0x7ff8000000000000ll) : 0.0, A = 0.0, Mo = 0.0;
    if (r >= nin && p >= nin) {
      // AuxInd = 1: both inactive or active, not both active (a virtual orbital takes no part)
      double x1 = 0.0;
      if (gp + gr <= 1) x1 = op * orr;
      if (gq + gs <= 1) x1 = fma(oq, os, x1);
      if (gq + gr <= 1) x1 = fma(-oq, orr, x1);
      if (gp + gs <= 1) x1 = fma(-op, os, x1);
      const double t = AC(st, gp, gq, gr, gs) * x1;
      // A- += 4 t (rs|pq); anti: t (ps|rq), read as (rq|ps); sym: -t (pr|qs)
      Mo = 4.0 * t * f1[((size_t)r + (size_t)s * n) * ldo];
      A = t * f2[(size_t)r * ldo + (size_t)s * n];
      S = fma(-t, f3[(size_t)s * nocc * ldf + (size_t)r * n], S);
    }
    if (ra && qa && p >= nin) {  // FOFO T1 (p -> q), FFOO T2 (p -> q) and T5
      const double2 z = I.za[(p - nin) + (size_t)nv * (s + (size_t)nocc * (qA + na * (r - nin)))];
      const double c = AC(st, gp, gs, 1, 1);
      S = fma(c, z.x, S);
      A = fma(c, z.y, A);
    }
    if (sa && r >= nin) {
      if (pa) {  // FOFO T3, T4 (p -> q) and T6
        const double2 z = I.zb[(r - nin) + (size_t)nv * (q + (size_t)nocc * (pA + na * (s - nin)))];
        const double c = AC(st, gq, gr, 1, 1);
        S = fma(c, z.x, S);
        A = fma(c, z.y, A);
      }
      if (qa && p >= nin) {  // FOFO T4 and T6 (p -> q), FFOO T3
        const double2 z = I.zc[(p - nin) + (size_t)nv * ((r - nin) + (size_t)nv * (qA + na * (s - nin)))];
        const double c = AC(st, gp, gr, 1, 1);
        S = fma(c, z.x, S);
        A = fma(c, z.y, A);
      }
    }
    if (ra && pa) {  // FFOO T1, T2 and T5 (p -> q)
      const double2 z = I.zd[q + (size_t)nocc * (s + (size_t)nocc * (pA + na * (r - nin)))];
      const double c = AC(st, gq, gs, 1, 1);
      S = fma(c, z.x, S);
      A = fma(c, z.y, A);
    }
    // one-body part (final loop of AB_CAS_FOFO): sym (p = r, q = s) and anti (q = r, p = s)
    if (p == r || q == s || q == r || p == s) {
      if (p == r)
        S += (op - os) * st.hno[q + (size_t)s * n] - st.wmat[q + (size_t)s * n] + op * aux(gp, gr, q, s);
      if (q == s)
        S += (oq - orr) * st.hno[p + (size_t)r * n] - st.wmat[p + (size_t)r * n] + oq * aux(gq, gs, p, r);
      if (q == r)
        A += (oq - os) * st.hno[p + (size_t)s * n] - st.wmat[p + (size_t)s * n] + oq * aux(gq, gr, p, s);
      if (p == s)
        A += (op - orr) * st.hno[q + (size_t)r * n] - st.wmat[q + (size_t)r * n] + op * aux(gp, gs, q, r);
    }
    double vp = S + A, vm = S - A + Mo;
    // divide by (C_p + C_q)(C_r + C_s) and (C_p - C_q)(C_r - C_s) where they are not 0,
    // as products of the pair reciprocals (no FP64 square root or division per element)
    if (zi_p && nonzero(rj_p)) vp *= ri_p * rj_p;
    if (zi_m && nonzero(rj_m)) vm *= ri_m * rj_m;
    abp[o] = vp;
    abm[o] = vm;
  }
}

__global__ void k_unpack_h(int n, const double *__restrict__ xone, double *__restrict__ h) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) h[i + (size_t)blockIdx.y * n] = one_el(xone, 1, n, i, blockIdx.y);
}

// sq_symmetrize (tran.f90:1303-1319): a(i,j) = a(j,i) = (a(i,j) + a(j,i)) / 2.
__global__ void k_sym_avg(int N, double *__restrict__ a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= N || j >= N || j <= i) return;
  const size_t u = i + (size_t)j * N, l = j + (size_t)i * N;
  const double v = 0.5 * (a[u] + a[l]);
  a[u] = v;
  a[l] = v;
}

}  // namespace

namespace gc {

std::vector<int> coalesced_pair_order(const int *indn, int ndimx) {
  if (!indn || ndimx <= 0) return {};
  std::vector<int> idx(ndimx);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) {
    const int qa = indn[2 * a + 1], qb = indn[2 * b + 1];
    return qa != qb ? qa < qb : indn[2 * a] < indn[2 * b];
  });
  std::vector<int> out(2 * (size_t)ndimx);
  for (int k = 0; k < ndimx; ++k) {
    out[2 * k] = indn[2 * idx[k]];
    out[2 * k + 1] = indn[2 * idx[k] + 1];
  }
  return out;
}

int rotate_h(gc_context *ctx, SysDev &sd, const double *ure_host) {
  // HNO = URe . h . URe^T, then sq_symmetrize (abfofo.f90:97-100)
  const int n = sd.n;
  DevBuf<double> u, w;
  GC_TRY(u.upload(ctx, ure_host, (size_t)n * n));
  GC_TRY(w.alloc(ctx, (size_t)n * n));
  GC_TRY(sd.h.alloc(ctx, (size_t)n * n));
  k_unpack_h<<<dim3(ceil_div(n, 128), n), 128, 0, ctx->stream>>>(n, sd.xone.p, sd.h.p);
  GC_LAUNCHED(ctx);
  const double one = 1.0, zero = 0.0;
  GC_CUBLAS(ctx, cublasDgemm(ctx->cublas, CUBLAS_OP_N, CUBLAS_OP_N, n, n, n, &one, u.p, n, sd.h.p, n,
                             &zero, w.p, n));
  GC_CUBLAS(ctx, cublasDgemm(ctx->cublas, CUBLAS_OP_N, CUBLAS_OP_T, n, n, n, &one, w.p, n, u.p, n,
                             &zero, sd.h.p, n));
  dim3 bs(32, 8), gs(ceil_div(n, 32), ceil_div(n, 8));
  k_sym_avg<<<gs, bs, 0, ctx->stream>>>(n, sd.h.p);
  GC_LAUNCHED(ctx);
  return GC_OK;
}

int set_error(gc_context *ctx, int code, const char *fmt, ...) {
  if (ctx) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    ctx->err = buf;
  }
  return code;
}

int sys_upload(gc_context *ctx, SysDev &sd, int nbas, int ninact, int nact, int ndimx,
               const double *occ, const double *xone, const int *indn, const double *rdm2act) {
  if (nbas <= 0 || ninact < 0 || nact < 0 || ninact + nact > nbas || ndimx <= 0 || !occ ||
      !indn || (!rdm2act && nact > 0))
    return set_error(ctx, GC_EINVAL, "system: bad arguments nbas=%d ninact=%d nact=%d ndimx=%d",
                     nbas, ninact, nact, ndimx);
  const int n = nbas, nocc = ninact + nact;
  auto finite = [](const double *x, size_t cnt) {
    for (size_t i = 0; i < cnt; ++i)
      if (!std::isfinite(x[i])) return false;
    return true;
  };
  if (!finite(occ, n) || (xone && !finite(xone, (size_t)n * (n + 1) / 2)) ||
      (nact > 0 && !finite(rdm2act, (size_t)nact * nact * (nact * nact + 1) / 2)))
    return set_error(ctx, GC_ENONFINITE,
                     "system: non-finite value in the occupations, one-electron integrals or 2-RDM");
  sd.n = n;
  sd.nin = ninact;
  sd.nact = nact;
  sd.nocc = nocc;
  sd.ndimx = ndimx;
  sd.vuni = n > nocc;
  for (int i = nocc; i < n; ++i)
    if (occ[i] != occ[nocc]) sd.vuni = 0;
  std::vector<int> grp(n), pp(ndimx), pq(ndimx);
  for (int i = 0; i < n; ++i) grp[i] = i < ninact ? 0 : (i < nocc ? 1 : 2);
  for (int i = 0; i < ndimx; ++i) {
    int a = indn[2 * i] - 1, b = indn[2 * i + 1] - 1;
    if (a < 0 || b < 0 || a >= n || b >= n || a <= b || b >= nocc)
      return set_error(ctx, GC_EINVAL, "system: pair %d = (%d,%d) is not a p>q pair with q occupied",
                       i + 1, a + 1, b + 1);
    pp[i] = a;
    pq[i] = b;
  }
  std::vector<double> cpl(ndimx), rpl(ndimx), rmi(ndimx), dnq(ndimx);
  {
    std::vector<double> ci(n);
    for (int i = 0; i < n; ++i) ci[i] = occ[i] >= 0.5 ? std::sqrt(occ[i]) : -std::sqrt(occ[i]);
    for (int i = 0; i < ndimx; ++i) {
      const double cp = ci[pp[i]], cq = ci[pq[i]], op = occ[pp[i]], oq = occ[pq[i]];
      cpl[i] = cp + cq;
      rpl[i] = cp + cq != 0.0 ? 1.0 / (cp + cq) : 0.0;
      rmi[i] = cp - cq != 0.0 ? 1.0 / (cp - cq) : 0.0;
      dnq[i] = op * (1.0 - oq) + oq * (1.0 - op);
    }
  }
  // Active block of RDM2val(i,j,k,l) = FRDM2(i,k,j,l) (abfofo.f90:84-92, interpa.f:5244-5272);
  // outside it RDM2val is products of occupations, which the kernels form themselves.
  std::vector<double> rv(std::max<size_t>((size_t)nact * nact * nact * nact, 1), 0.0);
  {
    size_t t = 0;
    for (int l = 0; l < nact; ++l)
      for (int k = 0; k < nact; ++k)
        for (int j = 0; j < nact; ++j)
          for (int i = 0; i < nact; ++i, ++t) {
            const long long a = (long long)i * nact + k + 1, b = (long long)j * nact + l + 1;
            const long long mx = std::max(a, b), mn = std::min(a, b);
            rv[t] = rdm2act[mx * (mx - 1) / 2 + mn - 1];
          }
  }
  // Row order of the element kernel: pairs by orbital groups, then tiles of 8 p x 4 q. The
  // pairs are listed per (p, q) cell (head, next) and the cells are walked in that order.
  std::vector<int> slot, head((size_t)n * nocc, -1), next(ndimx);
  for (int i = ndimx - 1; i >= 0; --i) {
    int &c = head[pp[i] + (size_t)pq[i] * n];
    next[i] = c;
    c = i;
  }
  slot.reserve(ndimx);
  const int pb[4] = {0, ninact, nocc, n}, qb[3] = {0, ninact, nocc};
  for (int gq = 0; gq < 2; ++gq)
    for (int gp = gq; gp < 3; ++gp)
      for (int p0 = pb[gp]; p0 < pb[gp + 1]; p0 += 8)
        for (int q0 = qb[gq]; q0 < qb[gq + 1]; q0 += 4)
          for (int q = q0; q < std::min(q0 + 4, qb[gq + 1]); ++q)
            for (int p = p0; p < std::min(p0 + 8, pb[gp + 1]); ++p)
              for (int i = head[p + (size_t)q * n]; i >= 0; i = next[i]) slot.push_back(i);
  // One staging buffer, one allocation, one copy: a copy from pageable memory costs some
  // microseconds whatever its size.
  struct Part {
    const void *src;
    size_t bytes;
    void **dst;
  };
  const size_t N = ndimx, ntr = (size_t)n * (n + 1) / 2;
  const Part parts[] = {
      {occ, n * sizeof(double), (void **)&sd.occ.p},
      {xone, xone ? ntr * sizeof(double) : 0, (void **)&sd.xone.p},
      {rv.data(), rv.size() * sizeof(double), (void **)&sd.rv.p},
      {cpl.data(), N * sizeof(double), (void **)&sd.cpl.p},
      {rpl.data(), N * sizeof(double), (void **)&sd.rpl.p},
      {rmi.data(), N * sizeof(double), (void **)&sd.rmi.p},
      {dnq.data(), N * sizeof(double), (void **)&sd.dnq.p},
      {grp.data(), n * sizeof(int), (void **)&sd.grp.p},
      {pp.data(), N * sizeof(int), (void **)&sd.pair_p.p},
      {pq.data(), N * sizeof(int), (void **)&sd.pair_q.p},
      {slot.data(), N * sizeof(int), (void **)&sd.slot.p},
  };
  std::vector<char> stage;
  for (const Part &p : parts) stage.resize((stage.size() + p.bytes + 15) / 16 * 16);
  GC_TRY(sd.blob.alloc(ctx, stage.size()));
  size_t at = 0;
  for (const Part &p : parts) {
    if (p.bytes) std::memcpy(stage.data() + at, p.src, p.bytes);
    *p.dst = sd.blob.p + at;
    at += (p.bytes + 15) / 16 * 16;
  }
  GC_CUDA(ctx, cudaMemcpyAsync(sd.blob.p, stage.data(), stage.size(), cudaMemcpyHostToDevice,
                               ctx->stream));
  return GC_OK;
}

int assemble(gc_context *ctx, const SysDev &sd, const double *ffoo, const double *fofo, int ns,
             const AbSpec *spec, double *etot_host) {
  auto ph = std::make_unique<PhaseScope>(ctx, GC_PHASE_ASSEMBLY);  // of the first pair
  Geo g{sd.n, sd.nin, sd.nact, sd.nocc};
  const int n = sd.n, N = sd.ndimx, nocc = sd.nocc, nv = n - sd.nin;
  const size_t na2 = (size_t)sd.nact * sd.nact, n2 = (size_t)n * n;
  const size_t sab = (size_t)nv * nocc * na2, sc = (size_t)nv * nv * na2,
               o2 = (size_t)nocc * nocc, sdd = o2 * na2;
  DevBuf<double> buf;
  GC_TRY(buf.alloc(ctx, 2 * (2 * sab + sc + sdd + ns * o2) + 4 * ns * n2 + kEtotWarps));
  Inter I;
  I.za = reinterpret_cast<double2 *>(buf.p);
  I.zb = I.za + sab;
  I.zc = I.zb + sab;
  I.zd = I.zc + sc;
  double2 *ct = I.zd + sdd;
  double *d = reinterpret_cast<double *>(ct + ns * o2);
  Settings sets{};
  for (int e = 0; e < ns; ++e, d += 4 * n2)
    sets.s[e] = Setting{spec[e].alpha, spec[e].ab1 ? 0.0 : 1.0, spec[e].ab1, ct + e * o2,
                        d, d + n2, d + 2 * n2, d + 3 * n2, spec[e].abplus, spec[e].abmin};
  I.part = d;
  const long long chv = ceil_div(nv, 32), chn = ceil_div(n, 32), cho = ceil_div(nocc, 32);
  const long long cnt[7] = {chv * nv * (long long)na2, chv * nocc * (long long)na2,
                            cho * nocc * (long long)na2, ns * chn * n, ns * chn * n,
                            (long long)ns * ceil_div(o2, 32), etot_host ? kEtotWarps : 0};
  long long first[8] = {0};
  for (int k = 0; k < 7; ++k) first[k + 1] = first[k] + cnt[k];
  if (first[7] > 0x7fffffffll - (1 << 24))
    return set_error(ctx, GC_EUNSUPPORTED, "assembly: nbas=%d nact=%d too large", n, sd.nact);
  const InterWork W{(int)first[0], (int)first[1], (int)first[2], (int)first[3],
                    (int)first[4], (int)first[5], (int)first[6], (int)first[7]};
  k_intermediates<<<std::min<unsigned>(ceil_div((size_t)W.end, 8), 152u * 64u), 256, 0,
                    ctx->stream>>>(g, W, sd.h.p ? sd.h.p : sd.xone.p, sd.h.p ? 0 : 1, sd.occ.p,
                                   sd.grp.p, fofo, ffoo, sd.rv.p, sets, I);
  GC_LAUNCHED(ctx);
  // Columns per warp: up to 8 share the row part of a warp's work; fewer where 8 would leave
  // the chip with less than 32 warps per SM (N = 570: 30 us with 8, 20 us with 2).
  const int cols = (int)std::min<long long>(8, std::max<long long>(1, (long long)ceil_div(N, 32) * N / (152 * 32)));
  const dim3 g3(ceil_div(N, 32 * kAbWarps), ceil_div(N, cols));
  if (g3.y > 65535)
    return set_error(ctx, GC_EUNSUPPORTED, "assembly: ndimx=%d too large", N);
  for (int e = 0; e < ns; ++e) {
    if (e > 0) ph = nullptr, ph = std::make_unique<PhaseScope>(ctx, GC_PHASE_ASSEMBLY);
    k_ab<<<g3, 32 * kAbWarps, 0, ctx->stream>>>(g, N, cols, sd.slot.p, sd.pair_p.p, sd.pair_q.p,
                                                sd.occ.p, sd.grp.p, fofo, ffoo, I, sets.s[e], sd.vuni,
                                                sd.rpl.p, sd.rmi.p);
    GC_LAUNCHED(ctx);
    if (spec[e].ab1) {  // AB_CAS_FOFO symmetrises the AB1 matrices (sq_symmetrize, abfofo.f90:260-263)
      dim3 bs(32, 8), gs(ceil_div(N, 32), ceil_div(N, 8));
      k_sym_avg<<<gs, bs, 0, ctx->stream>>>(N, spec[e].abplus);
      GC_LAUNCHED(ctx);
      k_sym_avg<<<gs, bs, 0, ctx->stream>>>(N, spec[e].abmin);
      GC_LAUNCHED(ctx);
    }
  }
  if (etot_host) {
    double hpart[kEtotWarps];
    GC_CUDA(ctx, cudaMemcpyAsync(hpart, I.part, sizeof hpart, cudaMemcpyDeviceToHost, ctx->stream));
    GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    double e = 0.0;
    for (double v : hpart) e += v;
    *etot_host = e;
  }
  return GC_OK;
}

int assemble_ab(gc_context *ctx, const SysDev &sd, const double *ffoo, const double *fofo,
                double alpha, double *abplus, double *abmin, double *etot_host, int ab1) {
  const AbSpec spec{alpha, ab1, abplus, abmin};
  return assemble(ctx, sd, ffoo, fofo, 1, &spec, etot_host);
}

int assemble_ab_pair(gc_context *ctx, const SysDev &sd, const double *ffoo, const double *fofo,
                     const AbSpec (&spec)[2], double *etot_host) {
  return assemble(ctx, sd, ffoo, fofo, 2, spec, etot_host);
}

}  // namespace gc

extern "C" int gc_ab_cas_fofo_ex(gc_context *ctx, int nbas, int ninact, int nact, int ndimx,
                                 const double *occ, const double *ure, const double *xone,
                                 const int *indn, const double *rdm2act, const double *ffoo,
                                 const double *fofo, double alpha, int ab1, double *abplus,
                                 double *abmin, double *etot) {
  if (!ctx) return GC_EINVAL;
  if (!xone || !ffoo || !fofo || !abplus || !abmin)
    return gc::set_error(ctx, GC_EINVAL, "ab_cas_fofo: null pointer");
  if (ure)
    for (size_t i = 0; i < (size_t)nbas * nbas; ++i)
      if (!std::isfinite(ure[i]))
        return gc::set_error(ctx, GC_ENONFINITE, "ab_cas_fofo: non-finite value in URe");
  gc::SysDev sd;
  GC_TRY(gc::sys_upload(ctx, sd, nbas, ninact, nact, ndimx, occ, xone, indn, rdm2act));
  if (ure) GC_TRY(gc::rotate_h(ctx, sd, ure));
  GC_TRY(gc::assemble_ab(ctx, sd, ffoo, fofo, alpha, abplus, abmin, etot, ab1 ? 1 : 0));
  return GC_OK;
}

extern "C" int gc_ab_cas_fofo(gc_context *ctx, int nbas, int ninact, int nact, int ndimx,
                              const double *occ, const double *xone, const int *indn,
                              const double *rdm2act, const double *ffoo, const double *fofo,
                              double alpha, double *abplus, double *abmin, double *etot) {
  return gc_ab_cas_fofo_ex(ctx, nbas, ninact, nact, ndimx, occ, nullptr, xone, indn, rdm2act, ffoo,
                           fofo, alpha, 0, abplus, abmin, etot);
}
