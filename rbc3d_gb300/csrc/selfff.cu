// selfff.cu -- RBC_SingInt (ModRbcSingInt.F90:29-90) for the FP32D mode: the
// own-cell polar-patch quadrature in float-float arithmetic on the FP32 pipe.
//
// GB300 issues FP64 at about 1/76 of its FP32 FMA rate (1.06 against 78
// TFLOP/s measured), and the FP64 patch kernel is bound by that pipe.  Here
// every quantity is an unevaluated sum hi + lo of two FP32 numbers (48
// significant bits):
//   * the Spline_Interp sums are compensated dot products (Ogita, Rump and
//     Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26, 2005):
//     each product w v split exactly by the FMA form of TwoProduct, the high
//     parts summed error-free, the rounding errors and the lo-part cross
//     terms summed in FP32.  The sums start from a power of two `off` at
//     least twice a bound on their sum of |w v| (the per-cell maxima of the
//     node values times the weight-sum bounds 1, h/4 and h^2/16), so every
//     partial sum stays above every product in magnitude and Dekker's
//     FastTwoSum (3 operations) is exact where Knuth's TwoSum takes 6; off
//     is subtracted exactly at the end.  The FP32 correction term is rounded
//     on the scale of off, so for the position x, whose interpolant is
//     differenced against the target, the bound covers the 12 derivative
//     terms only: off is subtracted before the 4 value terms, which are
//     added with TwoSum (all 16 from the larger offset: the corrections
//     move from 2.3e-12 to 2.3e-11 of the FP64 patch);
//   * the Ewald kernel (EwaldCoeff_SL / _DL, ModEwaldFunc.F90:86-180, the
//     same tables as hi/lo) is evaluated with Dekker's float-float product
//     and sum, and 1/r by rsqrtf, an FP32 Newton step and a float-float
//     Newton step.
// The patch corrections agree with the FP64 kernel to a few 1e-12 relative
// (rel-L2, 256-cell workload); the interpolation sums carry errors of a few
// 1e-12 of sum |w v| (x) or of the cell's maxima (f, g, a3).
//
// By latitude rings, as selfring.cu does it in FP64: the points of a ring's
// targets share their colatitudes and pair up about the meridian, so per point
// pair (class) and column j the theta part U_j, D_j (4 terms each) is computed
// once for the ring, and a point takes the 4 terms of the phi part from the
// columns j and j + 1.  About 500 packed instructions of interpolation a point
// against 900 with 16 terms, and 0.4 KB of loads against 1.7 KB.  256 cells,
// SL+DL: 6.5 -> 4.8 ms against one warp per target, the FP32D matvec 10.66 -> 8.89.
//
// Data layout.  Per row i and slot d (u, u_th, u_ph, u_thph) the 12 values x
// (relative to the cell centre), f and g density sets and a3 (three
// components each) are stored as three quads in column order; a quad's hi and
// lo parts form one 32-byte entry, read with one 256-bit load, so that a warp
// reads 32 consecutive entries: [cell][row][slot][quad][column].
// Consecutive values share one weight, so they run in pairs as packed FP32x2
// operations; the weights are stored doubled, as the pairs' operands.  Target
// positions are the FP32M hi/lo records relative to the same cell centre.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ctx.hpp"

namespace {

constexpr int FF_ROW = 12;   // 32-byte entries of a node: 4 slots x 3 quads
constexpr int FF_CHUNK = 2;  // classes between two barriers: the rows' entries are loaded once for both

// A class of patch points (RingClass) in hi/lo parts, each weight as the
// operands (h, h, l, l): the theta weights of (u, u', u_th, u'_th), per side
// the phi weights of (U_j, U_j+1, D_j, D_j+1).
struct FFClass {
  int i1, j[2], pad;
  float4 x[4], y[2][4];
  float2 w, pad2;
};
static_assert(sizeof(FFClass) % 16 == 0, "vector loads of the weights");

// ---------------------------------------------------------------------------
// float-float arithmetic
struct ff {
  float h, l;
};
__device__ __forceinline__ ff two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ ff fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ ff ff_norm(ff a) { return fast_two_sum(a.h, a.l); }
__device__ __forceinline__ ff ff_add(ff a, ff b) {
  ff s = two_sum(a.h, b.h);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ ff ff_sub(ff a, ff b) {
  ff s = two_sum(a.h, -b.h);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fsub_rn(a.l, b.l)));
}
// product without the final renormalisation: |l| stays ~2^-23 |h|
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return {p, e};
}
__device__ __forceinline__ bool ff_ge(ff a, ff b) { return a.h > b.h || (a.h == b.h && a.l >= b.l); }

// lazy accumulator: hi parts summed exactly, errors and lo parts in FP32
struct ffacc {
  float s, c;
  __device__ __forceinline__ void add(ff v) {
    const ff t = two_sum(s, v.h);
    s = t.h;
    c = __fadd_rn(c, __fadd_rn(t.l, v.l));
  }
};

// one 32-byte read-only load (hi quad, lo quad of one node)
__device__ __forceinline__ void ld8(const float4* p, float4& h, float4& l) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(h.x), "=f"(h.y), "=f"(h.z), "=f"(h.w), "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w)
      : "l"(p));
}

// packed FP32x2 helpers (round to nearest, as the scalar forms)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}

// Compensated dot-product accumulator for two values sharing a weight.
struct Dot2 {
  float2 s, c;
  // s + c += w * v with w = (wh, wl), v = (vh, vl) per half; nwh = -wh.
  // FAST: s has been kept above every product in magnitude (FastTwoSum)
  template <bool FAST>
  __device__ __forceinline__ void add(float2 wh, float2 nwh, float2 wl, float2 vh, float2 vl) {
    const float2 p = __fmul2_rn(wh, vh);
    const float2 ne = __ffma2_rn(nwh, vh, p);  // p - wh vh: minus the product's rounding error
    const float2 t = __fadd2_rn(s, p);
    float2 err;
    if (FAST) {
      err = sub2(p, sub2(t, s));
    } else {
      const float2 bb = sub2(t, s);
      err = __fadd2_rn(sub2(s, sub2(t, bb)), sub2(p, bb));
    }
    s = t;
    c = __ffma2_rn(wh, vl, c);
    c = __ffma2_rn(wl, vh, c);
    c = __fadd2_rn(c, sub2(err, ne));
  }
  // FAST with the weight's stored operands (h, h, l, l)
  template <bool FAST>
  __device__ __forceinline__ void add(float4 w, float2 vh, float2 vl) {
    add<FAST>(make_float2(w.x, w.y), make_float2(-w.x, -w.y), make_float2(w.z, w.w), vh, vl);
  }
};

struct FFArgs {
  int nt, ncell, nlat, nlon, m, NC, G, parts;
  const double* tA;
  double* v;
  const float4* rec;    // [cell][row][slot][quad][column][hi, lo]
  const FFClass* cls;   // [latitude][NC]
  const float4* thi;    // target positions relative to the cell centre, hi
  const float4* tlo;    // and lo
  const float4* tab;    // [3][EWALD_NTAB]: {T_i hi, T_i lo, (T_i+1 - T_i) hi, lo}
  const uint4* bnd;     // [set x f g a3][cell]: max |u|, |u_th|, |u_ph|, |u_thph| (float bits)
  float hq1, hq2;       // derivative weight-sum bounds: h_th / 4, h_ph / 4
  const int* celltype;
  ff c1;                // c1
  ff c2B[RBC3D_MAX_CELLTYPES];  // c2 Bcoef per cell type
  ff rc2, r_eps, ntab_over_rc;
};

__device__ __forceinline__ ff ld_ff(float2 v) { return {v.x, v.y}; }

// T + D f1 for table t at index it
__device__ __forceinline__ ff tab_lerp(const float4* tab, int t, int it, ff f1) {
  const float4 e = __ldg(tab + (size_t)t * EWALD_NTAB + it);
  return ff_add({e.x, e.y}, ff_mul({e.z, e.w}, f1));
}

__device__ __forceinline__ ff dot3(const ff* a, const ff* b) {
  return ff_add(ff_add(ff_mul(a[0], b[0]), ff_mul(a[1], b[1])), ff_mul(a[2], b[2]));
}

// The pairs of values: (x.x x.y) (x.z f.x) (f.y f.z) (g.x g.y) (g.z a.x) (a.y a.z),
// value 3 set + component in the order x, f, g, a3.
constexpr int FF_PAIRS = 6, FF_XPAIRS = 2;  // the first two hold x: value terms by TwoSum
// Offsets of one cell's sums: of U and D (theta part) and of the point (phi
// part), the x pairs' for their derivative terms only; and c2 Bcoef.
struct FFCell {
  float2 u[FF_PAIRS], d[FF_PAIRS], p[FF_PAIRS];
  float2 c2m, pad;
};

// smallest power of two at least twice b (with a margin for b's rounding)
__device__ __forceinline__ float sum_offset(float b) {
  int e;
  frexpf(2.f * 1.01f * b, &e);
  return ldexpf(1.f, e);
}

__device__ __forceinline__ void cell_offsets(const FFArgs& a, int cell, FFCell& C) {
  float ou[4], od[4], op[4];
  for (int s = 0; s < 4; ++s) {
    const uint4 b = __ldg(a.bnd + (size_t)s * a.ncell + cell);
    const float u = __uint_as_float(b.x), ut = __uint_as_float(b.y), up = __uint_as_float(b.z), utp = __uint_as_float(b.w);
    const float D = up + a.hq1 * utp, U = u + a.hq1 * ut;  // bounds of |D_j|, |U_j|
    const bool x = s == 0;
    ou[s] = sum_offset(x ? a.hq1 * ut : U);
    od[s] = sum_offset(D);
    op[s] = sum_offset(x ? a.hq2 * D : U + a.hq2 * D);
  }
  // f shares its first pair with x: the derivative terms' offset there too
  const uint4 b = __ldg(a.bnd + (size_t)a.ncell + cell);
  const float fD = __uint_as_float(b.z) + a.hq1 * __uint_as_float(b.w);
  const float fu = sum_offset(a.hq1 * __uint_as_float(b.y)), fp = sum_offset(a.hq2 * fD);
  C.u[0] = make_float2(ou[0], ou[0]); C.u[1] = make_float2(ou[0], fu); C.u[2] = make_float2(ou[1], ou[1]);
  C.u[3] = make_float2(ou[2], ou[2]); C.u[4] = make_float2(ou[2], ou[3]); C.u[5] = make_float2(ou[3], ou[3]);
  C.d[0] = make_float2(od[0], od[0]); C.d[1] = make_float2(od[0], od[1]); C.d[2] = make_float2(od[1], od[1]);
  C.d[3] = make_float2(od[2], od[2]); C.d[4] = make_float2(od[2], od[3]); C.d[5] = make_float2(od[3], od[3]);
  C.p[0] = make_float2(op[0], op[0]); C.p[1] = make_float2(op[0], fp); C.p[2] = make_float2(op[1], op[1]);
  C.p[3] = make_float2(op[2], op[2]); C.p[4] = make_float2(op[2], op[3]); C.p[5] = make_float2(op[3], op[3]);
  const ff c2 = a.c2B[a.celltype[cell]];
  C.c2m = make_float2(c2.h, c2.l);
}

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// RBC_SingInt's loop body at interpolated values v (s and c of the 6 pairs)
// for a target at xi: c1 and c2 terms added to the sums acc (stride st).
template <bool SL, bool DL>
__device__ __forceinline__ void patch_point(const FFArgs& a, const Dot2* d2, const ff* xi, ff c2m, ff wq, float2* acc,
                                            int st) {
  ff xx[3], F[3], G[3], A[3];
  xx[0] = ff_sub(fast_two_sum(d2[0].s.x, d2[0].c.x), xi[0]);
  xx[1] = ff_sub(fast_two_sum(d2[0].s.y, d2[0].c.y), xi[1]);
  xx[2] = ff_sub(fast_two_sum(d2[1].s.x, d2[1].c.x), xi[2]);
  if (SL) {
    F[0] = fast_two_sum(d2[1].s.y, d2[1].c.y);
    F[1] = fast_two_sum(d2[2].s.x, d2[2].c.x);
    F[2] = fast_two_sum(d2[2].s.y, d2[2].c.y);
  }
  if (DL) {
    G[0] = fast_two_sum(d2[3].s.x, d2[3].c.x);
    G[1] = fast_two_sum(d2[3].s.y, d2[3].c.y);
    G[2] = fast_two_sum(d2[4].s.x, d2[4].c.x);
    A[0] = fast_two_sum(d2[4].s.y, d2[4].c.y);
    A[1] = fast_two_sum(d2[5].s.x, d2[5].c.x);
    A[2] = fast_two_sum(d2[5].s.y, d2[5].c.y);
  }
  const ff r2 = ff_add(ff_add(ff_mul(xx[0], xx[0]), ff_mul(xx[1], xx[1])), ff_mul(xx[2], xx[2]));
  if (ff_ge(r2, a.rc2)) return;  // rr >= rc (ModRbcSingInt.F90:65)
  if (!(r2.h > 0.f)) return;
  // 1/r: rsqrtf, an FP32 Newton step, a float-float Newton step
  float y = rsqrtf(r2.h);
  y = y * fmaf(-0.5f * r2.h, y * y, 1.5f);
  const float y2 = __fmul_rn(y, y), y2e = fmaf(y, y, -y2);
  const float t0 = __fmul_rn(r2.h, y2);
  const float t1 = fmaf(r2.h, y2, -t0) + fmaf(r2.h, y2e, r2.l * y2);
  const float eps = __fsub_rn(__fsub_rn(1.f, t0), t1);  // 1 - r2 y^2
  const ff ir = fast_two_sum(y, 0.5f * y * eps);
  const ff rv = ff_norm(ff_mul(r2, ir));
  // EwaldCoeff_SL / _DL share the table position; below r_eps or beyond
  // the table both are zero
  if (!ff_ge(rv, a.r_eps)) return;
  const ff sp = ff_norm(ff_mul(rv, a.ntab_over_rc));
  float fi = floorf(sp.h);
  if (sp.h == fi && sp.l < 0.f) fi -= 1.f;
  const int it = (int)fi;
  if (it < 0 || it >= EWALD_NTAB) return;
  const ff f1 = two_sum(__fsub_rn(sp.h, fi), sp.l);
  const ff ir2 = ff_mul(ir, ir);
  ff cx = {0.f, 0.f}, cf = {0.f, 0.f};  // dv += cx xx + cf f
  if (SL) {
    const ff cs1 = tab_lerp(a.tab, 0, it, f1), cs2 = tab_lerp(a.tab, 1, it, f1);
    const ff c1ir = ff_mul(cs1, ir);
    const ff EA = ff_mul(ff_add(c1ir, cs2), ir2), EB = ff_sub(c1ir, cs2);
    // c1 wq (EA xx (xx . f) + EB f)
    const ff sw = ff_mul(a.c1, wq);
    cx = ff_mul(sw, ff_mul(EA, dot3(xx, F)));
    cf = ff_mul(sw, EB);
  }
  if (DL) {
    // c2 Bcoef wq EA xx (xx . g)(xx . a3), EA = cd / r^5
    const ff cd = tab_lerp(a.tab, 2, it, f1);
    const ff EA = ff_mul(cd, ff_mul(ir2, ff_mul(ir2, ir)));
    const ff t = ff_mul(ff_mul(ff_mul(c2m, wq), EA), ff_mul(dot3(xx, G), dot3(xx, A)));
    cx = SL ? ff_add(cx, t) : t;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 z = acc[k * st];
    ffacc s = {z.x, z.y};
    s.add(ff_mul(cx, xx[k]));
    if (SL) s.add(ff_mul(cf, F[k]));
    acc[k * st] = make_float2(s.s, s.c);
  }
}

// One block: a ring of G cells, thread = column (cols = G nlon; more than 256
// columns: several a thread).  Per chunk of FF_CHUNK classes the theta parts
// go to shared memory, then every column evaluates the points in the interval
// [j, j + 1]: of the targets j - j[0] and j - j[1] (mod nlon), whose sums lie
// in shared memory, a side each, so no two threads meet between two barriers.
template <bool SL, bool DL>
__global__ void __launch_bounds__(256, 2) k_self_ff(FFArgs a) {
  constexpr int NP = DL ? (SL ? 6 : 5) : 3;  // pairs kept; without SL the pair (f.y f.z) is left out
  extern __shared__ __align__(16) unsigned char smem_ff[];
  const int nlon = a.nlon, cols = a.G * nlon;
  float4* ex = reinterpret_cast<float4*>(smem_ff);            // [FF_CHUNK][NP][U, D][cols]: (s, s, c, c)
  FFCell* sC = reinterpret_cast<FFCell*>(ex + (size_t)FF_CHUNK * NP * 2 * cols);  // [G]
  float2* acc = reinterpret_cast<float2*>(sC + a.G);          // [2 sides][3][cols]
  float2* sT = acc + 6 * cols;                                // [3][cols] target positions
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int ring = b % a.nlat, cell0 = (b / a.nlat) * a.G;
  const int ncl = min(a.G, a.ncell - cell0), ncol = ncl * nlon;
  const int nv = a.nlat * nlon;
  for (int t = threadIdx.x; t < ncl; t += blockDim.x) cell_offsets(a, cell0 + t, sC[t]);
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = t / nlon, j = t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const float4 h = a.thi[p], l = a.tlo[p];
    sT[t] = make_float2(h.x, l.x); sT[cols + t] = make_float2(h.y, l.y); sT[2 * cols + t] = make_float2(h.z, l.z);
    for (int k = 0; k < 6; ++k) acc[k * cols + t] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  const FFClass* cls = a.cls + (size_t)ring * a.NC;
  for (int kb = k0; kb < k1; kb += FF_CHUNK) {
    for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
      const int lc = t / nlon, j = t - lc * nlon;
      const FFCell& C = sC[lc];
      const float4* rc = a.rec + 2 * ((size_t)(cell0 + lc) * a.m * FF_ROW * nlon + j);
#pragma unroll
      for (int q = 0; q < (DL ? 3 : 2); ++q) {
        float4 rh[8], rl[8];  // row i1: slots 0..3, row i1 + 1: slots 0..3
        int have = -1;
#pragma unroll
        for (int kk = 0; kk < FF_CHUNK; ++kk) {
          if (kb + kk >= k1) break;
          const FFClass& c = cls[kb + kk];
          if (c.i1 != have) {
            have = c.i1;
            const int i2 = have + 1 == a.m ? 0 : have + 1;
#pragma unroll
            for (int d = 0; d < 4; ++d) {
              ld8(rc + 2 * (size_t)((have * FF_ROW + 3 * d + q) * nlon), rh[d], rl[d]);
              ld8(rc + 2 * (size_t)((i2 * FF_ROW + 3 * d + q) * nlon), rh[4 + d], rl[4 + d]);
            }
          }
          const float4 w0 = __ldg(c.x), w1 = __ldg(c.x + 1), w2 = __ldg(c.x + 2), w3 = __ldg(c.x + 3);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int P = 2 * q + e;
            if ((!DL && P >= 3) || (!SL && P == 2)) continue;
            const int S = (!SL && P > 2) ? P - 1 : P;
            auto vh = [&](int i) { return e ? hi2(rh[i]) : lo2(rh[i]); };
            auto vl = [&](int i) { return e ? hi2(rl[i]) : lo2(rl[i]); };
            Dot2 U, D;
            const float2 ou = C.u[P], od = C.d[P];
            U.s = ou; U.c = make_float2(0.f, 0.f);
            U.add<true>(w2, vh(1), vl(1));
            U.add<true>(w3, vh(5), vl(5));
            if (P < FF_XPAIRS) {  // off/2 <= s <= 3 off/2: the subtraction is exact
              U.s = sub2(U.s, ou);
              U.add<false>(w0, vh(0), vl(0));
              U.add<false>(w1, vh(4), vl(4));
            } else {
              U.add<true>(w0, vh(0), vl(0));
              U.add<true>(w1, vh(4), vl(4));
              U.s = sub2(U.s, ou);
            }
            D.s = od; D.c = make_float2(0.f, 0.f);
            D.add<true>(w2, vh(3), vl(3));
            D.add<true>(w3, vh(7), vl(7));
            D.add<true>(w0, vh(2), vl(2));
            D.add<true>(w1, vh(6), vl(6));
            D.s = sub2(D.s, od);
            float4* o = ex + (size_t)((kk * NP + S) * 2) * cols + t;
            o[0] = make_float4(U.s.x, U.s.y, U.c.x, U.c.y);
            o[cols] = make_float4(D.s.x, D.s.y, D.c.x, D.c.y);
          }
        }
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int kk = 0; kk < FF_CHUNK && kb + kk < k1; ++kk) {
      const FFClass& c = cls[kb + kk];
      for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
        const int lc = t / nlon, j = t - lc * nlon, base = t - j;
        const int tn = j + 1 == nlon ? base : t + 1;
        const FFCell& C = sC[lc];
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
          const int js = c.j[side];
          if (js < 0) break;  // the points on the meridian have no mirror image
          const int q = base + (j >= js ? j - js : j - js + nlon);  // the target's column
          const float4* y = c.y[side];
          const float4 w0 = __ldg(y), w1 = __ldg(y + 1), w2 = __ldg(y + 2), w3 = __ldg(y + 3);
          Dot2 d2[FF_PAIRS];
#pragma unroll
          for (int P = 0; P < FF_PAIRS; ++P) {
            if ((!DL && P >= 3) || (!SL && P == 2)) continue;
            const int S = (!SL && P > 2) ? P - 1 : P;
            const float4* o = ex + (size_t)((kk * NP + S) * 2) * cols;
            const float4 D0 = o[cols + t], D1 = o[cols + tn], U0 = o[t], U1 = o[tn];
            const float2 off = C.p[P];
            Dot2& d = d2[P];
            d.s = off; d.c = make_float2(0.f, 0.f);
            d.add<true>(w2, lo2(D0), hi2(D0));
            d.add<true>(w3, lo2(D1), hi2(D1));
            if (P < FF_XPAIRS) {
              d.s = sub2(d.s, off);
              d.add<false>(w0, lo2(U0), hi2(U0));
              d.add<false>(w1, lo2(U1), hi2(U1));
            } else {
              d.add<true>(w0, lo2(U0), hi2(U0));
              d.add<true>(w1, lo2(U1), hi2(U1));
              d.s = sub2(d.s, off);
            }
          }
          const ff xi[3] = {ld_ff(sT[q]), ld_ff(sT[cols + q]), ld_ff(sT[2 * cols + q])};
          patch_point<SL, DL>(a, d2, xi, ld_ff(C.c2m), ld_ff(__ldg(&c.w)), acc + 3 * side * cols + q, cols);
        }
      }
      __syncthreads();  // the next class's sums may meet these
    }
  }
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = t / nlon, j = t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const double iA = 1.0 / a.tA[p];
    for (int k = 0; k < 3; ++k) {
      const float2 z0 = acc[k * cols + t], z1 = acc[(3 + k) * cols + t];
      const double dv = (((double)z0.x + (double)z1.x) + ((double)z0.y + (double)z1.y)) * iA;
      if (a.parts == 1) a.v[p + (size_t)k * a.nt] += dv;
      else atomicAdd(a.v + p + (size_t)k * a.nt, dv);
    }
  }
}

// hi/lo split of an FP64 value
__device__ __forceinline__ void split(double v, float* h, float* l) {
  const float hv = (float)v;
  *h = hv;
  *l = (float)(v - (double)hv);
}

// Node records of the spline sets named in `sets` (bit 0 x, 1 f, 2 g, 3 a3):
// value 3 s + c of slot d goes to component (3 s + c) % 4 of quad (3 s + c) / 4.
// bnd[s][cell] collects max |value| per slot (float bits, rounded up).  A block
// takes 4 rows x 16 columns of one cell through shared memory (the tables are
// in row order, the records in column order).
__global__ void __launch_bounds__(128) k_ff_rec(int ncell, int m, int n, const double* __restrict__ spl,
                                                const double* __restrict__ xc, float* __restrict__ out,
                                                unsigned* __restrict__ bnd, int sets) {
  __shared__ double s[4][16][4][SPL_NODE];  // set, column, row, value
  __shared__ unsigned smax[16];
  const int nti = (m + 3) / 4, ntj = (n + 15) / 16;
  const int jt = blockIdx.x % ntj, it = (blockIdx.x / ntj) % nti, cell = blockIdx.x / (ntj * nti);
  const int src[4] = {SPL_X, SPL_F, SPL_G, SPL_A3};
  if (threadIdx.x < 16) smax[threadIdx.x] = 0;
  __syncthreads();
  for (int k = 0; k < 4; ++k) {
    if (!(sets & (1 << k))) continue;
    const double* in = spl + ((size_t)cell * SPL_NSET + src[k]) * (size_t)m * n * SPL_NODE;
    for (int e = threadIdx.x; e < 16 * 4 * SPL_NODE; e += blockDim.x) {
      const int q = e % SPL_NODE, r = (e / SPL_NODE) % 4, c = e / (4 * SPL_NODE);
      const int j = 16 * jt + c, i = 4 * it + r;
      double v = 0.;
      if (j < n && i < m) v = in[((size_t)j * m + i) * SPL_NODE + q];
      if (k == 0 && q < 3 && j < n && i < m) v -= xc[3 * cell + q];
      s[k][c][r][q] = v;
      const unsigned mx = __float_as_uint(__double2float_ru(fabs(v)));
      atomicMax(&smax[4 * k + q / 3], mx);
    }
  }
  __syncthreads();
  if (threadIdx.x < 16 && (sets & (1 << (threadIdx.x / 4))))
    atomicMax(bnd + ((size_t)(threadIdx.x / 4) * ncell + cell) * 4 + threadIdx.x % 4, smax[threadIdx.x]);
  for (int e = threadIdx.x; e < 4 * FF_ROW * 16; e += blockDim.x) {
    const int c = e % 16, dq = (e / 16) % FF_ROW, r = e / (16 * FF_ROW);
    const int j = 16 * jt + c, i = 4 * it + r;
    if (j >= n || i >= m) continue;
    float* o = out + 8 * ((((size_t)cell * m + i) * FF_ROW + dq) * n + j);
    float h[4], l[4];
    int have = 0;
    for (int k = 0; k < 4; ++k) {
      const int val = 4 * (dq % 3) + k, set = val / 3;
      h[k] = l[k] = 0.f;
      if (!(sets & (1 << set))) continue;
      split(s[set][c][r][3 * (dq / 3) + val % 3], h + k, l + k);
      have |= 1 << k;
    }
    if (have == 15) {
      *reinterpret_cast<float4*>(o) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(o + 4) = make_float4(l[0], l[1], l[2], l[3]);
    } else {
      for (int k = 0; k < 4; ++k)
        if (have & (1 << k)) { o[k] = h[k]; o[4 + k] = l[k]; }
    }
  }
}

inline ff hsplit(double v) {
  const float h = (float)v;
  return {h, (float)(v - (double)h)};
}

}  // namespace

// Ewald tables as {T_i, T_i+1 - T_i} hi/lo (ModEwaldFunc.F90:96-104, 151-162).
rbc3d_status self_ff_tables(rbc3d_ctx* ctx, const std::vector<double>& c1, const std::vector<double>& c2,
                            const std::vector<double>& dl) {
  const int N = EWALD_NTAB;
  std::vector<float4> t(3 * (size_t)N);
  const std::vector<double>* src[3] = {&c1, &c2, &dl};
  for (int k = 0; k < 3; ++k)
    for (int i = 0; i < N; ++i) {
      const double v = (*src[k])[i], d = (*src[k])[i + 1] - v;
      const ff a = hsplit(v), b = hsplit(d);
      t[(size_t)k * N + i] = make_float4(a.h, a.l, b.h, b.l);
    }
  CUDA_TRY(ctx->ff_tab.upload(t.data(), t.size(), ctx->st));
  CUDA_TRY(cudaStreamSynchronize(ctx->st));
  return RBC3D_OK;
}

// The ring classes in hi/lo parts (the value weights complete: 1 - x[0] for u).
rbc3d_status self_ff_grid(rbc3d_ctx* ctx, const std::vector<RingClass>& R) {
  auto op = [](double v) {
    const ff e = hsplit(v);
    return make_float4(e.h, e.h, e.l, e.l);
  };
  std::vector<FFClass> C(R.size());
  for (size_t i = 0; i < R.size(); ++i) {
    const RingClass& r = R[i];
    FFClass& c = C[i];
    c.i1 = r.i1; c.j[0] = r.j[0]; c.j[1] = r.j[1]; c.pad = 0;
    c.x[0] = op(1. - r.x[0]); c.x[1] = op(r.x[0]); c.x[2] = op(r.x[1]); c.x[3] = op(r.x[2]);
    for (int s = 0; s < 2; ++s) {
      c.y[s][0] = op(1. - r.y[s][0]); c.y[s][1] = op(r.y[s][0]); c.y[s][2] = op(r.y[s][1]); c.y[s][3] = op(r.y[s][2]);
    }
    const ff w = hsplit(r.w);
    c.w = make_float2(w.h, w.l);
    c.pad2 = make_float2(0.f, 0.f);
  }
  CUDA_TRY(ctx->ff_cls.upload(reinterpret_cast<const char*>(C.data()), C.size() * sizeof(FFClass), ctx->st));
  CUDA_TRY(cudaStreamSynchronize(ctx->st));
  return RBC3D_OK;
}

// Node records are rebuilt on first use after the positions or densities change.
void self_ff_invalidate(rbc3d_ctx* ctx, bool geom, bool f, bool g) {
  const int gone = (geom ? 1 | 8 : 0) | (f ? 2 : 0) | (g ? 4 : 0);
  ctx->ff_sets &= ~gone;
  ctx->ring_sets &= ~gone;
}

// The float-float node records of the sets in `need` (bit 0 x, 1 f, 2 g,
// 3 a3) that are out of date, on the current stream.
rbc3d_status self_ff_records(rbc3d_ctx* ctx, int need) {
  const size_t per = 2 * (size_t)ctx->m * ctx->nlon * FF_ROW;  // float4 a cell
  if (!ctx->ff_rec.p || ctx->ff_rec.n < ctx->ncell * per) {
    CUDA_TRY(ctx->ff_rec.alloc(ctx->ncell * per));
    ctx->ff_sets = 0;
  }
  CUDA_TRY(ctx->ff_bnd.alloc(16 * (size_t)ctx->ncell));
  const int build = need & ~ctx->ff_sets;
  if (build) {
    for (int k = 0; k < 4; ++k)
      if (build & (1 << k))
        CUDA_TRY(cudaMemsetAsync(ctx->ff_bnd.p + 4 * (size_t)k * ctx->ncell, 0, 16 * (size_t)ctx->ncell, ctx->st));
    const long long nb = (long long)ctx->ncell * ((ctx->m + 3) / 4) * ((ctx->nlon + 15) / 16);
    { k_ff_rec<<<(int)nb, 128, 0, ctx->st>>>(ctx->ncell, ctx->m, ctx->nlon, ctx->spl.p, ctx->mix_xc.p,
                                             reinterpret_cast<float*>(ctx->ff_rec.p), ctx->ff_bnd.p, build); ++ctx->launches; }
    CUDA_TRY(cudaGetLastError());
    ctx->ff_sets |= build;
  }
  return RBC3D_OK;
}

rbc3d_status run_self_ff(rbc3d_ctx* ctx, int tlist, double c1, double c2) {
  TargetSet& t = ctx->tl[tlist];
  if (tlist != RBC3D_TLIST_RBC || t.n == 0 || ctx->ncell == 0) return RBC3D_OK;
  if (!ctx->phi_uniform) return ctx_fail(ctx, RBC3D_ERR_ARG, "FP32D needs phi(j) = j*2*pi/nlon");
  const bool sl = c1 != 0 && ctx->has_f, dl = c2 != 0 && ctx->has_g;
  if (!sl && !dl) return RBC3D_OK;
  const int np = dl ? (sl ? 6 : 5) : 3;
  auto smem = [&](int G) {
    const size_t cols = (size_t)G * ctx->nlon;
    return sizeof(float4) * FF_CHUNK * np * 2 * cols + sizeof(FFCell) * G + sizeof(float2) * 9 * cols;
  };
  // a ring wider than shared memory holds (about 500 columns) goes to the FP64 patch
  if (smem(1) > 227 * 1024) return run_self_corr(ctx, tlist, sl ? c1 : 0., dl ? c2 : 0.);
  // records this call reads: x always, f for SL, g and a3 for DL
  rbc3d_status s = self_ff_records(ctx, 1 | (sl ? 2 : 0) | (dl ? 4 | 8 : 0));
  if (s) return s;
  FFArgs a;
  a.nt = t.n; a.ncell = ctx->ncell; a.nlat = ctx->nlat; a.nlon = ctx->nlon; a.m = ctx->m;
  a.tA = t.Acoef.p; a.v = t.v.p; a.rec = ctx->ff_rec.p;
  a.cls = reinterpret_cast<const FFClass*>(ctx->ff_cls.p);
  a.thi = ctx->mix_thi.p; a.tlo = ctx->mix_tlo.p; a.tab = ctx->ff_tab.p; a.celltype = ctx->celltype.p;
  a.bnd = reinterpret_cast<const uint4*>(ctx->ff_bnd.p);
  a.hq1 = (float)(RBC3D_TWO_PI / ctx->m / 4); a.hq2 = (float)(RBC3D_TWO_PI / ctx->nlon / 4);
  const ff z = {0.f, 0.f};
  a.c1 = sl ? hsplit(c1) : z;
  for (int l = 0; l < RBC3D_MAX_CELLTYPES; ++l) a.c2B[l] = dl ? hsplit(c2 * ctx->Bcoef[l]) : z;
  a.rc2 = hsplit(ctx->prm.rc * ctx->prm.rc);
  a.r_eps = hsplit(ctx->T.r_eps);
  a.ntab_over_rc = hsplit(ctx->T.ntab_over_rc);
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device);
  a.NC = ctx->nrad * (ctx->nazm / 2 + 1);
  a.G = ring_cells(ctx->ncell, ctx->nlon);
  const int blocks = (ctx->ncell + a.G - 1) / a.G * ctx->nlat, thr = std::min(256, (a.G * ctx->nlon + 31) / 32 * 32);
  a.parts = ring_parts(a.NC, blocks, nsm);
  const size_t bytes = smem(a.G);
  auto launch = [&](auto kern) -> rbc3d_status {
    CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    kern<<<blocks * a.parts, thr, bytes, ctx->st>>>(a);
    ++ctx->launches;
    CUDA_TRY(cudaGetLastError());
    return RBC3D_OK;
  };
  if (sl && dl) return launch(k_self_ff<true, true>);
  if (sl) return launch(k_self_ff<true, false>);
  return launch(k_self_ff<false, true>);
}
