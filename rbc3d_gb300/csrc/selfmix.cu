// selfmix.cu -- RBC_SingInt (ModRbcSingInt.F90:29-90) for the FP32M mode:
// the own-cell polar-patch quadrature with FP64-accurate geometry and FP32
// arithmetic.
//
// The only cancellation-prone quantity of the patch quadrature is the
// separation xx = x(patch point) - x(target), as small as 1e-2 for the first
// radial ring.  Positions are stored relative to each cell's centre as FP32
// (hi, lo) pairs computed in FP64, and the stencil's values enter as offsets
// (X_hi - T_hi) + (X_lo - T_lo) from nearby target positions, formed before any
// weight is applied, so xx carries ~1e-7 relative error instead of the ~1e-5 of
// plain FP32 positions.  Densities, normals, weights and the Ewald kernel are
// FP32 (erfc as exp(-x^2) t Q(t), the fit of fit_erfcx, pair.cu), accumulated
// with Kahan compensation per target.
//
// By latitude rings, as selfring.cu and selfff.cu: per point pair (class) of a
// ring and column j the theta part once, relative to the ring's target T_j of
// that column; a point of target q takes it from the columns j and j + 1 with
// T_j - T_q and T_j+1 - T_q added.  About 240 packed instructions for the two
// points of a class and 0.4 KB of loads a point, against 300 scalar ones and
// 0.8 KB a point with one warp per target and 16-term sums, bound by L1.
#include <cmath>
#include <vector>

#include "ctx.hpp"

namespace {

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// Node record: 13 float4 in column order, [cell][row][MIX_ROW][column]: slot d (u,
// u_th, u_ph, u_thph) has the 12 values x, f, g, a3 in quads 3 d .. 3 d + 2 (x
// of slot u: the hi parts relative to the cell centre), quad 12 the lo parts.
constexpr int MIX_ROW = 13;

// A class of patch points (RingClass): theta weights of (u, u', u_th, u'_th),
// per side the phi weights of (U_j, U_j+1, D_j, D_j+1), the sides' quadrature
// weights (0 for a point without mirror image, which stands on both sides).
struct MixClass {
  int i1, j[2], pad;
  float x[4], y[2][4], w[2], pad2[2];
};

// mean of each cell's grid points (x SoA, 3 x npt)
__global__ void k_cell_mean(int nv, long long npt, const double* __restrict__ x, double* __restrict__ xc) {
  __shared__ double red[3][32];
  const int cell = blockIdx.x;
  double s[3] = {0, 0, 0};
  for (int r = threadIdx.x; r < nv; r += blockDim.x)
    for (int k = 0; k < 3; ++k) s[k] += x[(size_t)cell * nv + r + k * npt];
  for (int k = 0; k < 3; ++k) {
    double v = warp_sum(s[k]);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
    xc[3 * cell + threadIdx.x] = t / nv;
  }
}

// Node records of the sets in `sets` (bit 0 x and a3, 1 f, 2 g): a block takes
// 4 rows x 16 columns of one cell through shared memory (the tables are in row
// order, the records in column order).
__global__ void __launch_bounds__(128) k_mix_rec(int m, int n, const double* __restrict__ spl,
                                                 const double* __restrict__ xc, float* __restrict__ out, int sets) {
  __shared__ float s[4][16][4][SPL_NODE];  // set x f g a3, column, row, value
  __shared__ float lo[16][4][3];
  const int nti = (m + 3) / 4, ntj = (n + 15) / 16;
  const int jt = blockIdx.x % ntj, it = (blockIdx.x / ntj) % nti, cell = blockIdx.x / (ntj * nti);
  const int src[4] = {SPL_X, SPL_F, SPL_G, SPL_A3}, bit[4] = {1, 2, 4, 1};
  for (int k = 0; k < 4; ++k) {
    if (!(sets & bit[k])) continue;
    const double* in = spl + ((size_t)cell * SPL_NSET + src[k]) * (size_t)m * n * SPL_NODE;
    for (int e = threadIdx.x; e < 16 * 4 * SPL_NODE; e += blockDim.x) {
      const int q = e % SPL_NODE, r = (e / SPL_NODE) % 4, c = e / (4 * SPL_NODE);
      const int j = 16 * jt + c, i = 4 * it + r;
      if (j >= n || i >= m) continue;
      double v = in[((size_t)j * m + i) * SPL_NODE + q];
      if (k == 0 && q < 3) {
        v -= xc[3 * cell + q];
        lo[c][r][q] = (float)(v - (double)(float)v);
      }
      s[k][c][r][q] = (float)v;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 4 * MIX_ROW * 16; e += blockDim.x) {
    const int c = e % 16, dq = (e / 16) % MIX_ROW, r = e / (16 * MIX_ROW);
    const int j = 16 * jt + c, i = 4 * it + r;
    if (j >= n || i >= m) continue;
    float* o = out + 4 * ((((size_t)cell * m + i) * MIX_ROW + dq) * n + j);
    for (int k = 0; k < 4; ++k) {
      if (dq == 12) {
        if (sets & 1) o[k] = k < 3 ? lo[c][r][k] : 0.f;
        continue;
      }
      const int val = 4 * (dq % 3) + k, set = val / 3;
      if (sets & bit[set]) o[k] = s[set][c][r][3 * (dq / 3) + val % 3];
    }
  }
}

// Interpolated own position of every cell point (Spline_Interp at the grid
// point, as RBC_SingInt does), relative to the cell centre, as hi/lo.
__global__ void k_mix_targets(int npt, int nlat, int nlon, int m, const double* __restrict__ th,
                              const double* __restrict__ phi, const double* __restrict__ spl,
                              const double* __restrict__ xc, float4* __restrict__ thi, float4* __restrict__ tlo) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npt) return;
  int nv = nlat * nlon, cell = p / nv, r = p - cell * nv;
  int ilat = r % nlat, ilon = r / nlat;
  SplW W;
  spline_weights(th[ilat], phi[ilon], m, nlon, W);
  double x[3];
  spline_eval(spl + ((size_t)cell * SPL_NSET + SPL_X) * (size_t)m * nlon * SPL_NODE, W, 3, x);
  float h[3], l[3];
  for (int k = 0; k < 3; ++k) {
    double d = x[k] - xc[3 * cell + k];
    h[k] = (float)d;
    l[k] = (float)(d - (double)h[k]);
  }
  thi[p] = make_float4(h[0], h[1], h[2], 0.f);
  tlo[p] = make_float4(l[0], l[1], l[2], 0.f);
}

struct MixArgs {
  int nt, ncell, nlat, nlon, m, NC, G, parts;
  const double* tA;
  double* v;
  const float4* rec;
  const MixClass* cls;  // [latitude][NC]
  const float4* thi;
  const float4* tlo;
  const int* celltype;
  double B[RBC3D_MAX_CELLTYPES];
  float c1, c2;
  float rc2, sqpa, two_isqa, m8_ispi, q75_spi;
  float erfcx_q[ERFCX_DEG + 1];
};

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// One block: a ring of G cells, thread = column (cols = G nlon; more than 256
// columns: several a thread); values in pairs (x.x x.y) (x.z f.x) (f.y f.z)
// (g.x g.y) (g.z a.x) (a.y a.z).  One barrier a class: the theta parts
// alternate between two buffers; the targets' sums lie in shared memory, a side
// each, so no two threads meet between two barriers.
template <bool SL, bool DL>
__global__ void __launch_bounds__(256, 3) k_self_mix(MixArgs a) {
  constexpr int NP = DL ? (SL ? 6 : 5) : 3;  // pairs kept; without SL (f.y f.z) is left out
  extern __shared__ __align__(16) unsigned char smem_mix[];
  const int nlon = a.nlon, cols = a.G * nlon;
  float4* ex = reinterpret_cast<float4*>(smem_mix);              // [2][NP][cols]: U pair, D pair
  float2* acc = reinterpret_cast<float2*>(ex + 2 * NP * cols);   // [2 sides][3][cols]: Kahan sum and error
  float2* sT = acc + 6 * cols;                                   // [3][cols]: target position hi, lo
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int ring = b % a.nlat, cell0 = (b / a.nlat) * a.G;
  const int ncol = min(a.G, a.ncell - cell0) * nlon, nv = a.nlat * nlon;
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = t / nlon, j = t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const float4 h = a.thi[p], l = a.tlo[p];
    sT[t] = make_float2(h.x, l.x); sT[cols + t] = make_float2(h.y, l.y); sT[2 * cols + t] = make_float2(h.z, l.z);
    for (int k = 0; k < 6; ++k) acc[k * cols + t] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  const MixClass* cls = a.cls + (size_t)ring * a.NC;
  for (int kc = k0; kc < k1; ++kc) {
    const MixClass& c = cls[kc];
    float4* buf = ex + (size_t)((kc & 1) * NP) * cols;
    const int i1 = c.i1, i2 = i1 + 1 == a.m ? 0 : i1 + 1;
    for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
      const int lc = t / nlon, j = t - lc * nlon;
      const float4* r1 = a.rec + ((size_t)(cell0 + lc) * a.m + i1) * MIX_ROW * nlon + j;
      const float4* r2 = a.rec + ((size_t)(cell0 + lc) * a.m + i2) * MIX_ROW * nlon + j;
      const float4 w = *reinterpret_cast<const float4*>(c.x);
      const float2 w0 = dup(w.x), w1 = dup(w.y), w2 = dup(w.z), w3 = dup(w.w);
      const float2 T0 = sT[t], T1 = sT[cols + t], T2 = sT[2 * cols + t];
      const float4 l1 = __ldg(r1 + 12 * nlon), l2 = __ldg(r2 + 12 * nlon);
#pragma unroll
      for (int q = 0; q < (DL ? 3 : 2); ++q) {
        float4 p[4], r[4];  // the quad's slots of row i1 and of row i2
#pragma unroll
        for (int d = 0; d < 4; ++d) { p[d] = __ldg(r1 + (3 * d + q) * nlon); r[d] = __ldg(r2 + (3 * d + q) * nlon); }
        if (q == 0) {  // x as offsets from T_j (f.x passes unchanged)
          const float2 hxy = make_float2(T0.x, T1.x), lxy = make_float2(T0.y, T1.y);
          float2 v = __fadd2_rn(sub2(make_float2(p[0].x, p[0].y), hxy), sub2(make_float2(l1.x, l1.y), lxy));
          p[0].x = v.x; p[0].y = v.y;
          v = __fadd2_rn(sub2(make_float2(r[0].x, r[0].y), hxy), sub2(make_float2(l2.x, l2.y), lxy));
          r[0].x = v.x; r[0].y = v.y;
          p[0].z = __fadd_rn(__fsub_rn(p[0].z, T2.x), __fsub_rn(l1.z, T2.y));
          r[0].z = __fadd_rn(__fsub_rn(r[0].z, T2.x), __fsub_rn(l2.z, T2.y));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int P = 2 * q + e;
          if ((!DL && P >= 3) || (!SL && P == 2)) continue;
          const int S = (!SL && P > 2) ? P - 1 : P;
          auto lo = [&](const float4& v) { return e ? make_float2(v.z, v.w) : make_float2(v.x, v.y); };
          const float2 U = fma2(w3, lo(r[1]), fma2(w2, lo(p[1]), fma2(w1, lo(r[0]), mul2(w0, lo(p[0])))));
          const float2 D = fma2(w3, lo(r[3]), fma2(w2, lo(p[3]), fma2(w1, lo(r[2]), mul2(w0, lo(p[2])))));
          buf[(size_t)S * cols + t] = make_float4(U.x, U.y, D.x, D.y);
        }
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
      const int lc = t / nlon, j = t - lc * nlon, base = t - j;
      const int tn = j + 1 == nlon ? base : t + 1;
      const int qs[2] = {base + (j >= c.j[0] ? j - c.j[0] : j - c.j[0] + nlon),
                         base + (j >= c.j[1] ? j - c.j[1] : j - c.j[1] + nlon)};
      float2 val[2][6];
      {
        float2 Tj[3], Tn[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) { Tj[k] = sT[k * cols + t]; Tn[k] = sT[k * cols + tn]; }
#pragma unroll
        for (int P = 0; P < 6; ++P) {
          if ((!DL && P >= 3) || (!SL && P == 2)) continue;
          const int S = (!SL && P > 2) ? P - 1 : P;
          const float4 A = buf[(size_t)S * cols + t], B = buf[(size_t)S * cols + tn];
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            const float4 y = *reinterpret_cast<const float4*>(c.y[side]);
            float2 U0 = make_float2(A.x, A.y), U1 = make_float2(B.x, B.y);
            if (P < 2) {  // x: offsets from T_q
              const int q = qs[side];
              const float2 a0 = sT[2 * P * cols + q], z = make_float2(0.f, 0.f);
              const float2 a1 = P == 0 ? sT[cols + q] : z, j1 = P == 0 ? Tj[1] : z, n1 = P == 0 ? Tn[1] : z;
              U0 = __fadd2_rn(U0, __fadd2_rn(sub2(make_float2(Tj[2 * P].x, j1.x), make_float2(a0.x, a1.x)),
                                             sub2(make_float2(Tj[2 * P].y, j1.y), make_float2(a0.y, a1.y))));
              U1 = __fadd2_rn(U1, __fadd2_rn(sub2(make_float2(Tn[2 * P].x, n1.x), make_float2(a0.x, a1.x)),
                                             sub2(make_float2(Tn[2 * P].y, n1.y), make_float2(a0.y, a1.y))));
            }
            val[side][P] = fma2(dup(y.w), make_float2(B.z, B.w),
                                fma2(dup(y.z), make_float2(A.z, A.w), fma2(dup(y.y), U1, mul2(dup(y.x), U0))));
          }
        }
      }
      // both points at once: x = side 0, y = side 1
      auto vx = [&](int P) { return make_float2(val[0][P].x, val[1][P].x); };
      auto vy = [&](int P) { return make_float2(val[0][P].y, val[1][P].y); };
      const float2 xx = vx(0), yy = vy(0), zz = vx(1);
      float2 r2 = fma2(xx, xx, fma2(yy, yy, mul2(zz, zz)));
      const bool ok[2] = {r2.x < a.rc2, r2.y < a.rc2};  // not rr >= rc (ModRbcSingInt.F90:65)
      r2 = make_float2(ok[0] ? r2.x : 1.f, ok[1] ? r2.y : 1.f);
      const float2 ri = make_float2(rsqrtf(r2.x), rsqrtf(r2.y)), ir2 = mul2(ri, ri);
      const float2 st = mul2(mul2(r2, ri), dup(a.sqpa));
      const float2 exn = make_float2(__expf(-st.x * st.x), __expf(-st.y * st.y));
      // erfc(st) = exp(-st^2) t Q(t), t = 1/(1 + st/2) (fit_erfcx)
      const float2 den = fma2(dup(0.5f), st, dup(1.f)), tq = make_float2(__fdividef(1.f, den.x), __fdividef(1.f, den.y));
      float2 Q = dup(a.erfcx_q[ERFCX_DEG]);
#pragma unroll
      for (int k = ERFCX_DEG - 1; k >= 0; --k) Q = fma2(Q, tq, dup(a.erfcx_q[k]));
      const float2 e1 = mul2(exn, mul2(tq, Q)), wq = *reinterpret_cast<const float2*>(c.w);
      float2 cx, cf;  // dv = cx xx + cf f
      if (SL) {
        const float2 e1r = mul2(e1, ri), e2 = mul2(dup(a.two_isqa), exn), sw = mul2(dup(a.c1), wq);
        const float2 d = fma2(xx, vy(1), fma2(yy, vx(2), mul2(zz, vy(2))));
        cx = mul2(mul2(sw, mul2(__fadd2_rn(e1r, e2), ir2)), d);
        cf = mul2(sw, sub2(e1r, e2));
      }
      if (DL) {
        const float c2m = (float)(a.c2 * a.B[a.celltype[cell0 + lc]]);
        const float2 cdl = mul2(dup(a.m8_ispi), fma2(exn, mul2(st, fma2(st, st, dup(1.5f))), mul2(dup(a.q75_spi), e1)));
        const float2 Ad = mul2(mul2(mul2(cdl, ir2), ir2), ri);
        const float2 dg = fma2(xx, vx(3), fma2(yy, vy(3), mul2(zz, vx(4))));
        const float2 da = fma2(xx, vy(4), fma2(yy, vx(5), mul2(zz, vy(5))));
        const float2 tt = mul2(mul2(mul2(dup(c2m), wq), Ad), mul2(dg, da));
        cx = SL ? __fadd2_rn(cx, tt) : tt;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float2 v = mul2(cx, k == 0 ? xx : k == 1 ? yy : zz);
        if (SL) v = fma2(cf, k == 0 ? vy(1) : k == 1 ? vx(2) : vy(2), v);
        float2* s0 = acc + k * cols + qs[0];
        float2* s1 = acc + (3 + k) * cols + qs[1];
        const float2 z0 = *s0, z1 = *s1;  // (sum, error)
        const float2 sum = make_float2(z0.x, z1.x), y = sub2(v, make_float2(z0.y, z1.y));
        const float2 n = __fadd2_rn(sum, y), err = sub2(sub2(n, sum), y);
        if (ok[0]) *s0 = make_float2(n.x, err.x);
        if (ok[1]) *s1 = make_float2(n.y, err.y);
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = t / nlon, j = t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const double iA = 1.0 / a.tA[p];
    for (int k = 0; k < 3; ++k) {
      const float2 z0 = acc[k * cols + t], z1 = acc[(3 + k) * cols + t];
      const double dv = (((double)z0.x - (double)z0.y) + ((double)z1.x - (double)z1.y)) * iA;
      if (a.parts == 1) a.v[p + (size_t)k * a.nt] += dv;
      else atomicAdd(a.v + p + (size_t)k * a.nt, dv);
    }
  }
}

}  // namespace

// The ring classes in FP32.
rbc3d_status self_mixed_grid(rbc3d_ctx* ctx, const std::vector<RingClass>& R) {
  std::vector<MixClass> C(R.size());
  for (size_t i = 0; i < R.size(); ++i) {
    const RingClass& r = R[i];
    const bool two = r.j[1] >= 0;
    MixClass c{};
    c.i1 = r.i1; c.j[0] = r.j[0]; c.j[1] = r.j[two];
    c.x[0] = (float)(1. - r.x[0]);
    for (int k = 0; k < 3; ++k) c.x[1 + k] = (float)r.x[k];
    for (int s = 0; s < 2; ++s) {
      const double* y = r.y[s && two];
      c.y[s][0] = (float)(1. - y[0]);
      for (int k = 0; k < 3; ++k) c.y[s][1 + k] = (float)y[k];
    }
    c.w[0] = (float)r.w; c.w[1] = two ? (float)r.w : 0.f;
    C[i] = c;
  }
  CUDA_TRY(ctx->mix_cls.upload((const char*)C.data(), C.size() * sizeof(MixClass), ctx->st));
  CUDA_TRY(cudaStreamSynchronize(ctx->st));
  return RBC3D_OK;
}

// FP32 node records and target positions for the current geometry.
rbc3d_status self_mixed_geom(rbc3d_ctx* ctx) {
  self_ff_invalidate(ctx, true, false, false);
  ctx->rep_valid = false;  // the near pass's FP32 replay records follow the geometry
  const int nv = ctx->nlat * ctx->nlon;
  // cell centres (mean of the grid points) from the uploaded positions
  CUDA_TRY(ctx->mix_xc.alloc(3 * (size_t)ctx->ncell));
  { k_cell_mean<<<ctx->ncell, 256, 0, ctx->st>>>(nv, ctx->npt, ctx->x.p, ctx->mix_xc.p); ++ctx->launches; }
  // the node records are built on first use (run_self_mixed); the target
  // positions serve the float-float patch too
  ctx->mix_sets = 0;
  CUDA_TRY(ctx->mix_thi.alloc(ctx->npt));
  CUDA_TRY(ctx->mix_tlo.alloc(ctx->npt));
  { k_mix_targets<<<nblk(ctx->npt, 128), 128, 0, ctx->st>>>(ctx->npt, ctx->nlat, ctx->nlon, ctx->m, ctx->th.p,
                                                             ctx->phi.p, ctx->spl.p, ctx->mix_xc.p, ctx->mix_thi.p,
                                                             ctx->mix_tlo.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  return RBC3D_OK;
}

rbc3d_status self_mixed_density(rbc3d_ctx* ctx, bool f, bool g) {
  self_ff_invalidate(ctx, false, f, g);
  if (f) ctx->mix_sets &= ~2;
  if (g) ctx->mix_sets &= ~4;
  return RBC3D_OK;
}

rbc3d_status run_self_mixed(rbc3d_ctx* ctx, int tlist, double c1, double c2) {
  TargetSet& t = ctx->tl[tlist];
  if (tlist != RBC3D_TLIST_RBC || t.n == 0 || ctx->ncell == 0) return RBC3D_OK;
  const bool sl = c1 != 0 && ctx->has_f, dl = c2 != 0 && ctx->has_g;
  if (!sl && !dl) return RBC3D_OK;
  const int np = dl ? (sl ? 6 : 5) : 3;
  auto smem = [&](int G) {
    const size_t cols = (size_t)G * ctx->nlon;
    return sizeof(float4) * 2 * np * cols + sizeof(float2) * 9 * cols;
  };
  // a ring wider than shared memory holds (about 850 columns) goes to the FP64 patch
  if (smem(1) > 227 * 1024) return run_self_corr(ctx, tlist, sl ? c1 : 0., dl ? c2 : 0.);
  // FP32 node records of the current geometry and densities (bit 0 geometry, 1 f, 2 g)
  const size_t per = 4 * (size_t)ctx->m * ctx->nlon * MIX_ROW;
  if (!ctx->mix_rec.p || ctx->mix_rec.n < ctx->ncell * per) {
    CUDA_TRY(ctx->mix_rec.alloc(ctx->ncell * per));
    ctx->mix_sets = 0;
  }
  const int build = (1 | (sl ? 2 : 0) | (dl ? 4 : 0)) & ~ctx->mix_sets;
  if (build) {
    const long long nb = (long long)ctx->ncell * ((ctx->m + 3) / 4) * ((ctx->nlon + 15) / 16);
    { k_mix_rec<<<(int)nb, 128, 0, ctx->st>>>(ctx->m, ctx->nlon, ctx->spl.p, ctx->mix_xc.p, ctx->mix_rec.p, build); ++ctx->launches; }
    CUDA_TRY(cudaGetLastError());
    ctx->mix_sets |= build;
  }
  MixArgs a;
  a.nt = t.n; a.ncell = ctx->ncell; a.nlat = ctx->nlat; a.nlon = ctx->nlon; a.m = ctx->m;
  a.tA = t.Acoef.p; a.v = t.v.p; a.rec = reinterpret_cast<const float4*>(ctx->mix_rec.p);
  a.cls = reinterpret_cast<const MixClass*>(ctx->mix_cls.p);
  a.thi = ctx->mix_thi.p; a.tlo = ctx->mix_tlo.p; a.celltype = ctx->celltype.p;
  for (int l = 0; l < RBC3D_MAX_CELLTYPES; ++l) a.B[l] = ctx->Bcoef[l];
  a.c1 = (float)c1;
  a.c2 = (float)c2;
  a.rc2 = (float)(ctx->prm.rc * ctx->prm.rc);
  a.sqpa = (float)std::sqrt(RBC3D_PI / ctx->prm.alpha);
  a.two_isqa = (float)(2.0 / std::sqrt(ctx->prm.alpha));
  a.m8_ispi = (float)(-8.0 / std::sqrt(RBC3D_PI));
  a.q75_spi = (float)(0.75 * std::sqrt(RBC3D_PI));
  erfcx_coeffs(ctx);
  for (int k = 0; k <= ERFCX_DEG; ++k) a.erfcx_q[k] = ctx->erfcx_q[k];
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
  if (sl && dl) return launch(k_self_mix<true, true>);
  if (sl) return launch(k_self_mix<true, false>);
  return launch(k_self_mix<false, true>);
}
