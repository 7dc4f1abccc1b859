// selfff.cu -- RBC_SingInt (ModRbcSingInt.F90:29-90) for the FP32D mode: the
// own-cell polar-patch quadrature in float-float arithmetic on the FP32 pipe.
//
// GB300 issues FP64 at about 1/76 of its FP32 FMA rate (1.06 against 78
// TFLOP/s measured), and the FP64 patch kernel is bound by that pipe.  Here
// every quantity is an unevaluated sum hi + lo of two FP32 numbers (48
// significant bits):
//   * the Spline_Interp sums are compensated dot products (Ogita, Rump and
//     Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26, 2005):
//     the high parts summed error-free, the rounding errors and the lo-part
//     cross terms summed in FP32.  The sums start from a power of two `off` at
//     least twice a bound on their sum of |w v| (the per-cell maxima of the
//     node values times the weight-sum bounds 1 and h/4), so every partial sum
//     stays above every product in magnitude and one fused multiply-add takes
//     the place of product and sum with a recoverable error (Dot2); off is
//     subtracted exactly at the end.  The FP32 correction term is rounded
//     on the scale of off, so for the position x, whose interpolant is
//     differenced against the target, the bound covers the derivative terms
//     only: off is subtracted before the value terms, which are added with
//     Knuth's TwoSum (all from the larger offset: the corrections move from
//     2.3e-12 to 2.3e-11 of the FP64 patch);
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
// columns j and j + 1; the two points of a class run as the halves of packed
// FP32x2 operations.  256 cells, SL+DL: 6.5 -> 3.5 ms against one warp per
// target with 16-term sums (the FP32D matvec 10.63 -> 7.62 ms); of that 4.8 ->
// 3.9 by loading a quad's U and D slots in turn (32 registers of node values
// instead of 64, no spills), -> 3.5 by the fused 6-operation sums (Dot2).
// ncu at 64 cells: FMA pipe 56%, L1 data pipe 56%, issue 44% at 16 warps an
// SM (registers); measured and not kept: three blocks an SM (80 registers,
// spills: 3.8), two classes between barriers (3.9 against 3.9), loads past L1.
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
// Targets of a ring segment's block: 44 KB of shared memory, five blocks of three
// warps an SM (63 and 127 targets within 3 % of it at 260 to 1,000 columns)
constexpr int FF_SEG = 95;

// A class of patch points (RingClass) in hi/lo parts, each weight as the
// operands (h, h, l, l): the theta weights of (u, u', u_th, u'_th), per side
// the phi weights of (U_j, U_j+1, D_j, D_j+1).
struct FFClass {
  int i1, j[2], pad;
  float4 x[4], y[2][4], w;  // w: quadrature weights (h, l) of the sides; a point without mirror image stands
};                          // on both sides, with weight 0 on the second
static_assert(sizeof(FFClass) % 16 == 0, "vector loads of the weights");

// ---------------------------------------------------------------------------
// float-float arithmetic
struct ff {
  float h, l;
};
__device__ __forceinline__ bool ff_ge(ff a, ff b) { return a.h > b.h || (a.h == b.h && a.l >= b.l); }

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

// Compensated dot-product accumulator for two values sharing a weight:
// s + c += w v with the weight's stored operands (h, h, l, l).
struct Dot2 {
  float2 s, c;
  // FAST: s has been kept at off/2 .. 3 off/2 with |w v| <= off/2, so the fused
  // t = RN(s + wh vh) leaves t - s exact, and wh vh - (t - s), rounded once, is
  // what t lost: 6 operations where a separate product and FastTwoSum take 9
  template <bool FAST>
  __device__ __forceinline__ void add(float4 w, float2 vh, float2 vl) {
    const float2 wh = make_float2(w.x, w.y), wl = make_float2(w.z, w.w);
    if (FAST) {
      const float2 t = __ffma2_rn(wh, vh, s);
      const float2 lost = __ffma2_rn(wh, vh, sub2(s, t));
      s = t;
      c = __ffma2_rn(wh, vl, c);
      c = __ffma2_rn(wl, vh, c);
      c = __fadd2_rn(c, lost);
    } else {
      const float2 np = __fmul2_rn(make_float2(-w.x, -w.y), vh);  // minus the product
      const float2 e = __ffma2_rn(wh, vh, np);
      const float2 t = sub2(s, np), bb = sub2(t, s);
      const float2 err = sub2(sub2(s, sub2(t, bb)), __fadd2_rn(np, bb));
      s = t;
      c = __ffma2_rn(wh, vl, c);
      c = __ffma2_rn(wl, vh, c);
      c = __fadd2_rn(c, __fadd2_rn(err, e));
    }
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
  const float4* tab;    // [EWALD_NTAB][3]: {T_i hi, T_i lo, (T_i+1 - T_i) hi, lo}
  const uint4* bnd;     // [set x f g a3][cell]: max |u|, |u_th|, |u_ph|, |u_thph| (float bits)
  float hq1, hq2;       // derivative weight-sum bounds: h_th / 4, h_ph / 4
  const int* celltype;
  ff c1;                // c1
  ff c2B[RBC3D_MAX_CELLTYPES];  // c2 Bcoef per cell type
  ff rc2, r_eps, ntab_over_rc;
  int seg, segs;        // targets of a ring segment's block, blocks a ring
};

// float-float arithmetic on two points at once (packed FP32x2)
struct ff2 {
  float2 h, l;
};
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ ff2 two_sum2(float2 a, float2 b) {
  const float2 s = __fadd2_rn(a, b), bb = sub2(s, a);
  return {s, __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ ff2 fast_two_sum2(float2 a, float2 b) {  // |a| >= |b| or a == 0, per half
  const float2 s = __fadd2_rn(a, b);
  return {s, sub2(b, sub2(s, a))};
}
// a + b without the final renormalisation
__device__ __forceinline__ ff2 add2(ff2 a, ff2 b) {
  const ff2 s = two_sum2(a.h, b.h);
  return {s.h, __fadd2_rn(s.l, __fadd2_rn(a.l, b.l))};
}
// product without the final renormalisation: |l| stays ~2^-23 |h|
__device__ __forceinline__ ff2 mul2(ff2 a, ff2 b) {
  const float2 p = __fmul2_rn(a.h, b.h);
  float2 e = __ffma2_rn(a.h, b.h, neg2(p));
  e = __ffma2_rn(a.h, b.l, e);
  e = __ffma2_rn(a.l, b.h, e);
  return {p, e};
}
// compensated dot product, not renormalised
__device__ __forceinline__ ff2 dot3(const ff2* a, const ff2* b) {
  ff2 r = mul2(a[0], b[0]);
#pragma unroll
  for (int k = 1; k < 3; ++k) {
    const float2 p = __fmul2_rn(a[k].h, b[k].h), e = __ffma2_rn(a[k].h, b[k].h, neg2(p));
    const ff2 t = two_sum2(r.h, p);
    r.h = t.h;
    r.l = __ffma2_rn(a[k].h, b[k].l, r.l);
    r.l = __ffma2_rn(a[k].l, b[k].h, r.l);
    r.l = __fadd2_rn(r.l, __fadd2_rn(t.l, e));
  }
  return r;
}
__device__ __forceinline__ ff2 both(ff a) { return {make_float2(a.h, a.h), make_float2(a.l, a.l)}; }
// T + D f1 for table t at the indices ia, ib (|D f1| <= |T|), not renormalised
__device__ __forceinline__ ff2 tab_lerp(const float4* tab, int t, int ia, int ib, ff2 f1) {
  const float4 a = __ldg(tab + 3 * ia + t), b = __ldg(tab + 3 * ib + t);
  const ff2 p = mul2({make_float2(a.z, b.z), make_float2(a.w, b.w)}, f1);
  const ff2 r = fast_two_sum2(make_float2(a.x, b.x), p.h);
  return {r.h, __fadd2_rn(r.l, __fadd2_rn(make_float2(a.y, b.y), p.l))};
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

__device__ __forceinline__ ff2 vx(const Dot2& a, const Dot2& b) {
  return {make_float2(a.s.x, b.s.x), make_float2(a.c.x, b.c.x)};
}
__device__ __forceinline__ ff2 vy(const Dot2& a, const Dot2& b) {
  return {make_float2(a.s.y, b.s.y), make_float2(a.c.y, b.c.y)};
}
__device__ __forceinline__ ff2 norm2(ff2 a) { return fast_two_sum2(a.h, a.l); }
// v - t for the targets' positions ta, tb (h, l)
__device__ __forceinline__ ff2 from_target(ff2 v, float2 ta, float2 tb) {
  v = norm2(v);
  const ff2 s = two_sum2(v.h, make_float2(-ta.x, -tb.x));
  return fast_two_sum2(s.h, __fadd2_rn(s.l, sub2(v.l, make_float2(ta.y, tb.y))));
}
// whether a patch point at squared distance (h, l) counts: not rr >= rc
// (ModRbcSingInt.F90:65), not zero, not NaN
__device__ __forceinline__ bool in_range(const FFArgs& a, float h, float l) {
  return h > 0.f && (h < a.rc2.h || (h == a.rc2.h && l < a.rc2.l));
}
__device__ __forceinline__ int table_index(float h, float l) {
  const float fi = floorf(h);
  return (int)(h == fi && l < 0.f ? fi - 1.f : fi);
}

// RBC_SingInt's loop body for the two points of a class, interpolated values
// A and B (s and c of the 6 pairs): their c1 and c2 terms added to the sums
// accA and accB (stride st) of the targets at tA and tB (stride st).
template <bool SL, bool DL>
__device__ __forceinline__ void patch_points(const FFArgs& a, const Dot2* A, const Dot2* B, const float2* tA,
                                             const float2* tB, ff c2m, float4 wq, float2* accA, float2* accB, int st) {
  ff2 xx[3], F[3], Gv[3], N[3];
  xx[0] = from_target(vx(A[0], B[0]), tA[0], tB[0]);
  xx[1] = from_target(vy(A[0], B[0]), tA[st], tB[st]);
  xx[2] = from_target(vx(A[1], B[1]), tA[2 * st], tB[2 * st]);
  if (SL) { F[0] = vy(A[1], B[1]); F[1] = vx(A[2], B[2]); F[2] = vy(A[2], B[2]); }
  if (DL) {
    Gv[0] = vx(A[3], B[3]); Gv[1] = vy(A[3], B[3]); Gv[2] = vx(A[4], B[4]);
    // xx . a3 cancels to the surface's curvature times r^2: normalised
    N[0] = norm2(vy(A[4], B[4])); N[1] = norm2(vx(A[5], B[5])); N[2] = norm2(vy(A[5], B[5]));
  }
  ff2 r2 = norm2(dot3(xx, xx));
  bool oka = in_range(a, r2.h.x, r2.l.x), okb = in_range(a, r2.h.y, r2.l.y);
  r2.h = make_float2(oka ? r2.h.x : 1.f, okb ? r2.h.y : 1.f);
  r2.l = make_float2(oka ? r2.l.x : 0.f, okb ? r2.l.y : 0.f);
  // 1/r: rsqrtf, an FP32 Newton step, a float-float Newton step
  const float2 half = make_float2(0.5f, 0.5f);
  float2 y = make_float2(rsqrtf(r2.h.x), rsqrtf(r2.h.y));
  const float2 hr = __fmul2_rn(make_float2(-0.5f, -0.5f), r2.h);
  y = __fmul2_rn(y, __ffma2_rn(hr, __fmul2_rn(y, y), make_float2(1.5f, 1.5f)));
  const float2 y2 = __fmul2_rn(y, y), y2e = __ffma2_rn(y, y, neg2(y2));
  const float2 t0 = __fmul2_rn(r2.h, y2);
  const float2 t1 = __fadd2_rn(__ffma2_rn(r2.h, y2, neg2(t0)), __ffma2_rn(r2.h, y2e, __fmul2_rn(r2.l, y2)));
  const float2 eps = sub2(sub2(make_float2(1.f, 1.f), t0), t1);  // 1 - r2 y^2
  const ff2 ir = fast_two_sum2(y, __fmul2_rn(__fmul2_rn(half, y), eps));
  const ff2 rv = norm2(mul2(r2, ir));
  // EwaldCoeff_SL / _DL share the table position; below r_eps or beyond the
  // table both are zero
  const ff2 sp = norm2(mul2(rv, both(a.ntab_over_rc)));
  const int ia = table_index(sp.h.x, sp.l.x), ib = table_index(sp.h.y, sp.l.y);
  oka = oka && ff_ge({rv.h.x, rv.l.x}, a.r_eps) && (unsigned)ia < (unsigned)EWALD_NTAB;
  okb = okb && ff_ge({rv.h.y, rv.l.y}, a.r_eps) && (unsigned)ib < (unsigned)EWALD_NTAB;
  const int ja = oka ? ia : 0, jb = okb ? ib : 0;
  // sp.h - ia is 0 or at least an ulp of sp.h
  const ff2 f1 = fast_two_sum2(sub2(sp.h, make_float2((float)ia, (float)ib)), sp.l);
  const ff2 ir2 = mul2(ir, ir);
  const ff2 w = {make_float2(wq.x, wq.z), make_float2(wq.y, wq.w)};
  ff2 cx, cf;  // dv += cx xx + cf f
  if (SL) {
    const ff2 cs1 = tab_lerp(a.tab, 0, ja, jb, f1), cs2 = tab_lerp(a.tab, 1, ja, jb, f1);
    const ff2 c1ir = mul2(cs1, ir);
    const ff2 EA = mul2(add2(c1ir, cs2), ir2), EB = add2(c1ir, {neg2(cs2.h), neg2(cs2.l)});
    // c1 wq (EA xx (xx . f) + EB f)
    const ff2 sw = mul2(both(a.c1), w);
    cx = mul2(sw, mul2(EA, dot3(xx, F)));
    cf = mul2(sw, EB);
  }
  if (DL) {
    // c2 Bcoef wq EA xx (xx . g)(xx . a3), EA = cd / r^5
    const ff2 cd = tab_lerp(a.tab, 2, ja, jb, f1);
    const ff2 EA = mul2(cd, mul2(ir2, mul2(ir2, ir)));
    const ff2 t = mul2(mul2(mul2(both(c2m), w), EA), mul2(dot3(xx, Gv), dot3(xx, N)));
    cx = SL ? add2(cx, t) : t;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 za = accA[k * st], zb = accB[k * st];
    ff2 v = mul2(cx, xx[k]);
    ff2 s = two_sum2(make_float2(za.x, zb.x), v.h);
    float2 c = __fadd2_rn(make_float2(za.y, zb.y), __fadd2_rn(s.l, v.l));
    if (SL) {
      v = mul2(cf, F[k]);
      s = two_sum2(s.h, v.h);
      c = __fadd2_rn(c, __fadd2_rn(s.l, v.l));
    }
    if (oka) accA[k * st] = make_float2(s.h.x, c.x);
    if (okb) accB[k * st] = make_float2(s.h.y, c.y);
  }
}

// One block: a ring of G cells, thread = column (cols = G nlon; more than 256
// columns: several a thread).  Per class the theta parts go to shared memory,
// then every column evaluates the points in the interval [j, j + 1]: of the
// targets j - j[0] and j - j[1] (mod nlon), whose sums lie in shared memory, a
// side each, so no two threads meet between two barriers.
// WIDE: a segment of the targets of one cell's ring, thread = target; the theta
// parts of a class are of the columns that these targets' points fall into, for
// each side apart (so each twice in a ring).
template <bool SL, bool DL, bool WIDE>
__global__ void __launch_bounds__(WIDE ? FF_SEG + 1 : 256, WIDE ? 5 : 2) k_self_ff(FFArgs a) {
  constexpr int NP = DL ? (SL ? 6 : 5) : 3;  // pairs kept; without SL the pair (f.y f.z) is left out
  extern __shared__ __align__(16) unsigned char smem_ff[];
  const int nlon = a.nlon, cols = WIDE ? 2 * (a.seg + 1) : a.G * nlon, ntg = WIDE ? a.seg : cols;
  float4* ex = reinterpret_cast<float4*>(smem_ff);            // [2, WIDE 1][NP][U, D][cols]: (s, s, c, c)
  FFCell* sC = reinterpret_cast<FFCell*>(ex + (size_t)(WIDE ? 2 : 4) * NP * cols);  // [G]
  float2* acc = reinterpret_cast<float2*>(sC + a.G);          // [2 sides][3][ntg]
  float2* sT = acc + 6 * ntg;                                 // [3][ntg] target positions
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int q0 = WIDE ? b % a.segs * a.seg : 0;               // the first target
  if (WIDE) b /= a.segs;
  const int ring = b % a.nlat, cell0 = (b / a.nlat) * a.G;
  const int ncl = min(a.G, a.ncell - cell0), ncol = WIDE ? min(a.seg, nlon - q0) : ncl * nlon;
  const int nv = a.nlat * nlon;
  for (int t = threadIdx.x; t < ncl; t += blockDim.x) cell_offsets(a, cell0 + t, sC[t]);
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = WIDE ? 0 : t / nlon, j = q0 + t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const float4 h = a.thi[p], l = a.tlo[p];
    sT[t] = make_float2(h.x, l.x); sT[ntg + t] = make_float2(h.y, l.y); sT[2 * ntg + t] = make_float2(h.z, l.z);
    for (int k = 0; k < 6; ++k) acc[k * ntg + t] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  const FFClass* cls = a.cls + (size_t)ring * a.NC;
  for (int k = k0; k < k1; ++k) {
    const FFClass& c = cls[k];
    float4* buf = WIDE ? ex : ex + (size_t)((k & 1) * NP * 2) * cols;
    const int i1 = c.i1, i2 = i1 + 1 == a.m ? 0 : i1 + 1;
    if (WIDE) __syncthreads();  // the previous class's values are done with
    for (int t = threadIdx.x; t < (WIDE ? 2 * (ncol + 1) : ncol); t += blockDim.x) {
      int lc = 0, j;
      if (WIDE) {
        const int side = t > ncol;
        j = q0 + t - side * (ncol + 1) + c.j[side];
        if (j >= nlon) j -= nlon;
      } else {
        lc = t / nlon;
        j = t - lc * nlon;
      }
      const FFCell& C = sC[lc];
      const float4* rc = a.rec + 2 * ((size_t)(cell0 + lc) * a.m * FF_ROW * nlon + j);
      const float4 w0 = __ldg(c.x), w1 = __ldg(c.x + 1), w2 = __ldg(c.x + 2), w3 = __ldg(c.x + 3);
#pragma unroll
      for (int qh = 0; qh < (DL ? 6 : 4); ++qh) {
        const int q = qh >> 1, h = qh & 1;  // quad; 0: U from the slots u, u_th, 1: D from u_ph, u_thph
        float4 rh[4], rl[4];                // slots 2h, 2h + 1 of row i1, then of row i2
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          ld8(rc + 2 * (size_t)((i1 * FF_ROW + 3 * (2 * h + d) + q) * nlon), rh[d], rl[d]);
          ld8(rc + 2 * (size_t)((i2 * FF_ROW + 3 * (2 * h + d) + q) * nlon), rh[2 + d], rl[2 + d]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int P = 2 * q + e;
          if ((!DL && P >= 3) || (!SL && P == 2)) continue;
          const int S = (!SL && P > 2) ? P - 1 : P;
          auto vh = [&](int i) { return e ? hi2(rh[i]) : lo2(rh[i]); };
          auto vl = [&](int i) { return e ? hi2(rl[i]) : lo2(rl[i]); };
          const float2 off = h ? C.d[P] : C.u[P];
          Dot2 d;
          d.s = off; d.c = make_float2(0.f, 0.f);
          d.add<true>(w2, vh(1), vl(1));
          d.add<true>(w3, vh(3), vl(3));
          if (h == 0 && P < FF_XPAIRS) {  // off/2 <= s <= 3 off/2: the subtraction is exact
            d.s = sub2(d.s, off);
            d.add<false>(w0, vh(0), vl(0));
            d.add<false>(w1, vh(2), vl(2));
          } else {
            d.add<true>(w0, vh(0), vl(0));
            d.add<true>(w1, vh(2), vl(2));
            d.s = sub2(d.s, off);
          }
          buf[(size_t)(2 * S + h) * cols + t] = make_float4(d.s.x, d.s.y, d.c.x, d.c.y);
        }
      }
    }
    // one barrier a class: the next class's values go to the other buffer, and
    // nobody is past this barrier before the previous class's sums are in
    __syncthreads();
    for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
      const int lc = WIDE ? 0 : t / nlon, j = t - lc * nlon, base = t - j;
      const int tn = !WIDE && j + 1 == nlon ? base : t + 1;
      const FFCell& C = sC[lc];
      const int qa = WIDE ? t : base + (j >= c.j[0] ? j - c.j[0] : j - c.j[0] + nlon);  // the targets' columns
      const int qb = WIDE ? t : base + (j >= c.j[1] ? j - c.j[1] : j - c.j[1] + nlon);
      Dot2 da[FF_PAIRS], db[FF_PAIRS];
#pragma unroll
      for (int P = 0; P < FF_PAIRS; ++P) {
        if ((!DL && P >= 3) || (!SL && P == 2)) continue;
        const int S = (!SL && P > 2) ? P - 1 : P;
        const float4* o = buf + (size_t)(2 * S) * cols;
        float4 D0 = o[cols + t], D1 = o[cols + tn], U0 = o[t], U1 = o[tn];
        const float2 off = C.p[P];
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          if (WIDE && side) {
            const int u = ncol + 1 + t;
            D0 = o[cols + u]; D1 = o[cols + u + 1]; U0 = o[u]; U1 = o[u + 1];
          }
          const float4* y = c.y[side];
          const float4 w0 = __ldg(y), w1 = __ldg(y + 1), w2 = __ldg(y + 2), w3 = __ldg(y + 3);
          Dot2& d = side ? db[P] : da[P];
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
      }
      patch_points<SL, DL>(a, da, db, sT + qa, sT + qb, {C.c2m.x, C.c2m.y}, __ldg(&c.w), acc + qa, acc + 3 * ntg + qb, ntg);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = WIDE ? 0 : t / nlon, j = q0 + t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const double iA = 1.0 / a.tA[p];
    for (int k = 0; k < 3; ++k) {
      const float2 z0 = acc[k * ntg + t], z1 = acc[(3 + k) * ntg + t];
      const double dv = (((double)z0.x + (double)z1.x) + ((double)z0.y + (double)z1.y)) * iA;
      if (a.parts == 1) a.v[p + (size_t)k * a.nt] += dv;
      else atomicAdd(a.v + p + (size_t)k * a.nt, dv);
    }
  }
}

// hi/lo split of an FP64 value, both parts rounded to nearest.  In integer
// arithmetic where both parts are normal: the conversions run on the FP64 pipe.
__device__ __forceinline__ void split(double v, float& h, float& l) {
  const unsigned long long b = __double_as_longlong(v);
  const int e = (int)(b >> 52) & 0x7ff;  // |v| in [2^(e-1023), 2^(e-1022))
  if (e >= 1023 - 70 && e < 1023 + 120) {
    // hi: 24 of the 53 bits, rounded by the addition's carry; the remainder
    // of the 29 bits below as a signed integer in units of 2^(e-1075)
    const unsigned long long r = b + (1ull << 28);
    h = __int_as_float((int)((b >> 32) & 0x80000000u) | ((((int)(r >> 52) & 0x7ff) - 1023 + 127) << 23) |
                       ((int)(r >> 29) & 0x7fffff));
    const int low = (int)(r & 0x1fffffff) - (1 << 28);
    const float u = __int_as_float((e - 1075 + 127) << 23);
    l = (float)low * (b >> 63 ? -u : u);
  } else {
    h = (float)v;
    l = (float)(v - (double)h);
  }
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
  const int nti = (m + 3) / 4, ntj = (n + 15) / 16;
  const int jt = blockIdx.x % ntj, it = (blockIdx.x / ntj) % nti, cell = blockIdx.x / (ntj * nti);
  const int src[4] = {SPL_X, SPL_F, SPL_G, SPL_A3};
  for (int k = 0; k < 4; ++k) {
    if (!(sets & (1 << k))) continue;
    const double* in = spl + ((size_t)cell * SPL_NSET + src[k]) * (size_t)m * n * SPL_NODE;
    for (int e = threadIdx.x; e < 16 * 4 * SPL_NODE; e += blockDim.x) {
      const int q = e % SPL_NODE, r = (e / SPL_NODE) % 4, c = e / (4 * SPL_NODE);
      const int j = 16 * jt + c, i = 4 * it + r;
      double v = 0.;
      if (j < n && i < m) {
        v = in[((size_t)j * m + i) * SPL_NODE + q];
        if (k == 0 && q < 3) v -= xc[3 * cell + q];
      }
      s[k][c][r][q] = v;
    }
  }
  __syncthreads();
  {  // 8 threads per (set, slot): the largest magnitude, compared as integers
    const int k = threadIdx.x >> 5, d = (threadIdx.x >> 3) & 3, o = threadIdx.x & 7;
    unsigned long long mx = 0;
    if (sets & (1 << k))
      for (int node = o; node < 64; node += 8)
        for (int c = 0; c < 3; ++c) {
          const unsigned long long v = __double_as_longlong(s[k][node >> 2][node & 3][3 * d + c]) & 0x7fffffffffffffffull;
          mx = v > mx ? v : mx;
        }
    for (int w = 4; w > 0; w >>= 1) {
      const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, w);
      mx = v > mx ? v : mx;
    }
    if (o == 0 && (sets & (1 << k)))
      atomicMax(bnd + ((size_t)k * ncell + cell) * 4 + d, __float_as_uint(__double2float_ru(__longlong_as_double(mx))));
  }
  for (int e = threadIdx.x; e < 4 * FF_ROW * 16; e += blockDim.x) {
    const int c = e % 16, dq = (e / 16) % FF_ROW, r = e / (16 * FF_ROW);
    const int j = 16 * jt + c, i = 4 * it + r;
    if (j >= n || i >= m) continue;
    float* o = out + 8 * ((((size_t)cell * m + i) * FF_ROW + dq) * n + j);
    float h[4], l[4];
    int have = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int val = 4 * (dq % 3) + k, set = val / 3;
      h[k] = l[k] = 0.f;
      if (!(sets & (1 << set))) continue;
      split(s[set][c][r][3 * (dq / 3) + val % 3], h[k], l[k]);
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
      t[3 * (size_t)i + k] = make_float4(a.h, a.l, b.h, b.l);
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
    const bool two = r.j[1] >= 0;
    c.i1 = r.i1; c.j[0] = r.j[0]; c.j[1] = r.j[two]; c.pad = 0;
    c.x[0] = op(1. - r.x[0]); c.x[1] = op(r.x[0]); c.x[2] = op(r.x[1]); c.x[3] = op(r.x[2]);
    for (int s = 0; s < 2; ++s) {
      const double* y = r.y[s && two];
      c.y[s][0] = op(1. - y[0]); c.y[s][1] = op(y[0]); c.y[s][2] = op(y[1]); c.y[s][3] = op(y[2]);
    }
    const ff w = hsplit(r.w);
    c.w = make_float4(w.h, w.l, two ? w.h : 0.f, two ? w.l : 0.f);
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
  // A ring of more columns than threads goes by segments, unless it fits in
  // shared memory (498 columns) and leaves few threads without a second column
  // (us, whole ring / segments: 4 cells of 16 x 260 706 / 670, 16 x 300 774 /
  // 749, 2 cells of 40 x 264 1470 / 1310, of 16 x 480 665 / 692).  Over that it
  // went to the FP64 patch: 2 cells of 16 x 520 2165 -> 775, of 16 x 1000 5115 -> 2410.
  const size_t column = sizeof(float4) * 4 * np + sizeof(float2) * 9;
  const bool wide = ctx->nlon > RING_MAX_NLON &&
                    (ctx->nlon < 432 || column * ctx->nlon + sizeof(FFCell) > SMEM_BLOCK);
  a.G = wide ? 1 : ring_cells(ctx->ncell, ctx->nlon);
  a.seg = wide ? ring_segment(ctx->nlon, FF_SEG) : 0;
  a.segs = wide ? (ctx->nlon + a.seg - 1) / a.seg : 1;
  const int blocks = (ctx->ncell + a.G - 1) / a.G * ctx->nlat * a.segs;
  const int thr = std::min(256, ((wide ? a.seg + 1 : a.G * ctx->nlon) + 31) / 32 * 32);
  a.parts = ring_parts(a.NC, blocks, nsm);
  const size_t cols = wide ? a.seg : a.G * ctx->nlon, ent = wide ? 2 * (a.seg + 1) : 2 * cols;  // (both buffers)
  const size_t bytes = sizeof(float4) * 2 * np * ent + sizeof(FFCell) * a.G + sizeof(float2) * 9 * cols;
  auto launch = [&](auto kern) -> rbc3d_status {
    CUDA_TRY(smem_opt_in(kern, bytes));
    kern<<<blocks * a.parts, thr, bytes, ctx->st>>>(a);
    ++ctx->launches;
    CUDA_TRY(cudaGetLastError());
    return RBC3D_OK;
  };
  if (sl && dl) return wide ? launch(k_self_ff<true, true, true>) : launch(k_self_ff<true, true, false>);
  if (sl) return wide ? launch(k_self_ff<true, false, true>) : launch(k_self_ff<true, false, false>);
  return wide ? launch(k_self_ff<false, true, true>) : launch(k_self_ff<false, true, false>);
}
