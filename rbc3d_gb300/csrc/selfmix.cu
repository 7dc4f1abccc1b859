// selfmix.cu -- RBC_SingInt (ModRbcSingInt.F90:29-90) for the FP32M mode:
// the own-cell polar-patch quadrature with FP64-accurate geometry and FP32
// arithmetic.
//
// The cancellation-prone quantities of the patch quadrature are the separation
// xx = x(patch point) - x(target), as small as 1e-2 for the first radial ring,
// and its product with the normal.  Positions are stored relative to each
// cell's centre as FP32 (hi, lo) pairs computed in FP64, and each stencil node's
// offset from the target, (X_hi - t_hi) + (X_lo - t_lo), is formed before the
// bicubic weights are applied, so xx carries ~1e-7 relative error instead of
// the ~1e-5 of plain FP32 positions.  Densities, normals, weights and the Ewald
// kernel are FP32 (erfc as exp(-x^2) t Q(t), the fit of fit_erfcx, pair.cu),
// accumulated with Kahan compensation per target.
//
// By latitude rings, as selfring.cu and selfff.cu: the two points of a class
// that fall into a column interval share their four stencil nodes, so a thread
// (column) loads the nodes' positions and normals once for both (their sums
// keep all 16 terms: any other order moves xx . a3 near the target by its
// rounding, 2e-6 of the velocities), and the densities go through the theta
// part computed once per column and class.  0.4 KB of loads a point instead of
// 0.8 KB with one warp per target, which L1 bound: 256 cells, SL+DL, 3.08 ->
// 1.72 ms alone (two blocks an SM 1.82).  With the theta part for the positions
// and normals too, relative to the ring's target, 1.41 ms, but outputs 1.3e-7
// from these by rounding alone.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ctx.hpp"

namespace {

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// Node record: 13 float4 in column order, [cell][row][MIX_ROW][column]: floats
// x hi(3) lo(3), a3(3), then u_th, u_ph, u_thph of x (9) and of a3 (9), pad;
// from quad 7 on f and g (6 floats) of the slots u, u_th, u_ph, u_thph.
constexpr int MIX_ROW = 13, MIX_XA = 7;
constexpr int MIX_SEG = 127;  // targets of a ring segment's block

// A class of patch points (RingClass): theta weights of (u, u', u_th, u'_th);
// per side the phi weights of (U_j, U_j+1, D_j, D_j+1) and, per stencil node
// (row i1: columns j, j + 1; the next row: j, j + 1), the products for (u,
// u_th, u_ph, u_thph); the sides' quadrature weights (0 for a point without
// mirror image, which stands on both sides).
struct MixClass {
  int i1, j[2], pad;
  float x[4], y[2][4], n[2][4][4], w[2], pad2[2];
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
  __shared__ float s[16][4][4 * MIX_ROW + 1];  // column, row, float of the record
  const int nti = (m + 3) / 4, ntj = (n + 15) / 16;
  const int jt = blockIdx.x % ntj, it = (blockIdx.x / ntj) % nti, cell = blockIdx.x / (ntj * nti);
  const int src[4] = {SPL_X, SPL_A3, SPL_F, SPL_G}, bit[4] = {1, 1, 2, 4};
  for (int k = 0; k < 4; ++k) {
    if (!(sets & bit[k])) continue;
    const double* in = spl + ((size_t)cell * SPL_NSET + src[k]) * (size_t)m * n * SPL_NODE;
    for (int e = threadIdx.x; e < 16 * 4 * SPL_NODE; e += blockDim.x) {
      const int q = e % SPL_NODE, r = (e / SPL_NODE) % 4, c = e / (4 * SPL_NODE), d = q / 3, v3 = q % 3;
      const int j = 16 * jt + c, i = 4 * it + r;
      if (j >= n || i >= m) continue;
      double v = in[((size_t)j * m + i) * SPL_NODE + q];
      float* o = s[c][r];
      if (k == 0) {
        if (d == 0) {
          v -= xc[3 * cell + v3];
          o[3 + v3] = (float)(v - (double)(float)v);
          if (v3 == 0) o[4 * MIX_XA - 1] = 0.f;
        }
        o[d == 0 ? v3 : 9 + 3 * (d - 1) + v3] = (float)v;
      } else if (k == 1) {
        o[d == 0 ? 6 + v3 : 18 + 3 * (d - 1) + v3] = (float)v;
      } else {
        o[4 * MIX_XA + 6 * d + 3 * (k - 2) + v3] = (float)v;
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 4 * MIX_ROW * 16; e += blockDim.x) {
    const int c = e % 16, dq = (e / 16) % MIX_ROW, r = e / (16 * MIX_ROW);
    const int j = 16 * jt + c, i = 4 * it + r;
    if (j >= n || i >= m) continue;
    float* o = out + 4 * ((((size_t)cell * m + i) * MIX_ROW + dq) * n + j);
    for (int k = 0; k < 4; ++k) {
      const int f = 4 * dq + k;  // the record's float, and the set it belongs to
      const int b = dq < MIX_XA ? 1 : (f - 4 * MIX_XA) % 6 < 3 ? 2 : 4;
      if (sets & b) o[k] = s[c][r][f];
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
  int seg, segs;  // as FFArgs (selfff.cu)
};

// One block: a ring of G cells, thread = column (cols = G nlon; more than 256
// columns: several a thread).  One barrier a class: the densities' theta parts
// alternate between two buffers; the targets' sums lie in shared memory, a side
// each, so no two threads meet between two barriers.  WIDE: a segment of the targets of one cell's ring, as k_self_ff.
template <bool SL, bool DL, bool WIDE>
__global__ void __launch_bounds__(WIDE ? MIX_SEG + 1 : 256, WIDE ? 5 : 3) k_self_mix(MixArgs a) {
  extern __shared__ __align__(16) unsigned char smem_mix[];
  const int nlon = a.nlon, cols = WIDE ? 2 * (a.seg + 1) : a.G * nlon, ntg = WIDE ? a.seg : cols;
  float4* ex = reinterpret_cast<float4*>(smem_mix);            // [2][3][cols]: (f0 f1) (f2 g0) (g1 g2) of U, D
  float2* acc = reinterpret_cast<float2*>(ex + 2 * 3 * cols);  // [2 sides][3][ntg]: Kahan sum and error
  float2* sT = acc + 6 * ntg;                                   // [3][ntg]: target position hi, lo
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int q0 = WIDE ? b % a.segs * a.seg : 0;                // the first target
  if (WIDE) b /= a.segs;
  const int ring = b % a.nlat, cell0 = (b / a.nlat) * a.G;
  const int ncol = WIDE ? min(a.seg, nlon - q0) : min(a.G, a.ncell - cell0) * nlon, nv = a.nlat * nlon;
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = WIDE ? 0 : t / nlon, j = q0 + t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const float4 h = a.thi[p], l = a.tlo[p];
    sT[t] = make_float2(h.x, l.x); sT[ntg + t] = make_float2(h.y, l.y); sT[2 * ntg + t] = make_float2(h.z, l.z);
    for (int k = 0; k < 6; ++k) acc[k * ntg + t] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  const MixClass* cls = a.cls + (size_t)ring * a.NC;
  const float c1 = a.c1;
  for (int kc = k0; kc < k1; ++kc) {
    const MixClass& c = cls[kc];
    float4* buf = ex + (size_t)((kc & 1) * 3) * cols;
    const int i1 = c.i1, i2 = i1 + 1 == a.m ? 0 : i1 + 1;
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
      const float4* r1 = a.rec + (((size_t)(cell0 + lc) * a.m + i1) * MIX_ROW + MIX_XA) * nlon + j;
      const float4* r2 = a.rec + (((size_t)(cell0 + lc) * a.m + i2) * MIX_ROW + MIX_XA) * nlon + j;
      const float4 w = *reinterpret_cast<const float4*>(c.x);
      float o[2][6];  // U (slots u, u_th), D (u_ph, u_thph) of f and g
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float p[12], r[12];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float4 u = __ldg(r1 + (3 * h + q) * nlon), v = __ldg(r2 + (3 * h + q) * nlon);
          p[4 * q] = u.x; p[4 * q + 1] = u.y; p[4 * q + 2] = u.z; p[4 * q + 3] = u.w;
          r[4 * q] = v.x; r[4 * q + 1] = v.y; r[4 * q + 2] = v.z; r[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) o[h][k] = fmaf(w.w, r[6 + k], fmaf(w.z, p[6 + k], fmaf(w.y, r[k], w.x * p[k])));
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
        buf[q * cols + t] = make_float4(o[0][2 * q], o[0][2 * q + 1], o[1][2 * q], o[1][2 * q + 1]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
      // the sides' targets, columns and places of their theta parts
      int lc = 0, qs[2] = {t, t}, js[2], jn[2], ts[2] = {t, ncol + 1 + t}, tn[2] = {t + 1, ncol + 2 + t};
      if (WIDE) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          js[s] = q0 + t + c.j[s];
          if (js[s] >= nlon) js[s] -= nlon;
          jn[s] = js[s] + 1 == nlon ? 0 : js[s] + 1;
        }
      } else {
        lc = t / nlon;
        const int j = t - lc * nlon, base = t - j;
        js[0] = js[1] = j;
        jn[0] = jn[1] = j + 1 == nlon ? 0 : j + 1;
        ts[1] = t;
        tn[0] = tn[1] = base + jn[0];
#pragma unroll
        for (int s = 0; s < 2; ++s) qs[s] = base + (j >= c.j[s] ? j - c.j[s] : j - c.j[s] + nlon);
      }
      float xx[2][3], A3[2][3], FG[2][6], th_[2][3], tl_[2][3];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float2 T = sT[k * ntg + qs[s]];
          th_[s][k] = T.x; tl_[s][k] = T.y;
          xx[s][k] = 0.f; A3[s][k] = 0.f;
        }
      const float4* rows = a.rec + (size_t)(cell0 + lc) * a.m * MIX_ROW * nlon;
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // the stencil nodes
        float v[4 * MIX_XA];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (WIDE || s == 0) {  // the sides share a column unless WIDE
            const float4* r = rows + (size_t)(k < 2 ? i1 : i2) * MIX_ROW * nlon + (k & 1 ? jn[s] : js[s]);
#pragma unroll
            for (int q = 0; q < MIX_XA; ++q) {
              if (!DL && q >= 5) continue;  // a3's derivatives
              const float4 u = __ldg(r + q * nlon);
              v[4 * q] = u.x; v[4 * q + 1] = u.y; v[4 * q + 2] = u.z; v[4 * q + 3] = u.w;
            }
          }
          const float4 w = *reinterpret_cast<const float4*>(c.n[s][k]);
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const float d = __fadd_rn(__fsub_rn(v[e], th_[s][e]), __fsub_rn(v[3 + e], tl_[s][e]));
            // in this order: it decides the rounding of xx . a3 near the target
            xx[s][e] = __fadd_rn(xx[s][e], fmaf(w.w, v[15 + e], fmaf(w.z, v[12 + e], fmaf(w.x, d, __fmul_rn(w.y, v[9 + e])))));
            if (DL)
              A3[s][e] = __fadd_rn(A3[s][e], fmaf(w.w, v[24 + e], fmaf(w.z, v[21 + e],
                                                                       fmaf(w.x, v[6 + e], __fmul_rn(w.y, v[18 + e])))));
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        float4 A = buf[q * cols + ts[0]], B = buf[q * cols + tn[0]];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (WIDE && s) { A = buf[q * cols + ts[1]]; B = buf[q * cols + tn[1]]; }
          const float4 y = *reinterpret_cast<const float4*>(c.y[s]);
          FG[s][2 * q] = fmaf(y.w, B.z, fmaf(y.z, A.z, fmaf(y.y, B.x, y.x * A.x)));
          FG[s][2 * q + 1] = fmaf(y.w, B.w, fmaf(y.z, A.w, fmaf(y.y, B.y, y.x * A.y)));
        }
      }
      const float c2m = DL ? (float)(a.c2 * a.B[a.celltype[cell0 + lc]]) : 0.f;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const float* x = xx[s];
        const float r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (r2 >= a.rc2) continue;  // rr >= rc (ModRbcSingInt.F90:65)
        const float rinv = rsqrtf(r2), rv = r2 * rinv, ir2 = rinv * rinv;
        const float st = rv * a.sqpa, exn = __expf(-st * st);
        // erfc(st) = exp(-st^2) t Q(t), t = 1/(1 + st/2) (fit_erfcx)
        const float tq = __fdividef(1.f, fmaf(0.5f, st, 1.f));
        float Qp = a.erfcx_q[ERFCX_DEG];
#pragma unroll
        for (int k = ERFCX_DEG - 1; k >= 0; --k) Qp = fmaf(Qp, tq, a.erfcx_q[k]);
        const float e1 = exn * (tq * Qp), e2 = a.two_isqa * exn;
        const float wq = c.w[s];
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        if (SL) {
          const float A = (e1 * rinv + e2) * ir2, Bc = e1 * rinv - e2;
          const float f0 = wq * FG[s][0], f1 = wq * FG[s][1], f2 = wq * FG[s][2];
          const float d = x[0] * f0 + x[1] * f1 + x[2] * f2;
          v0 = c1 * (A * x[0] * d + Bc * f0);
          v1 = c1 * (A * x[1] * d + Bc * f1);
          v2 = c1 * (A * x[2] * d + Bc * f2);
        }
        if (DL) {
          const float cdl = a.m8_ispi * (exn * (st * (1.5f + st * st)) + a.q75_spi * e1);
          const float Ad = cdl * ir2 * ir2 * rinv;
          const float dg = wq * (x[0] * FG[s][3] + x[1] * FG[s][4] + x[2] * FG[s][5]);
          const float da = fmaf(x[2], A3[s][2], fmaf(x[0], A3[s][0], __fmul_rn(x[1], A3[s][1])));
          const float tt = c2m * Ad * dg * da;
          v0 += tt * x[0]; v1 += tt * x[1]; v2 += tt * x[2];
        }
        float2* z = acc + 3 * s * ntg + qs[s];
        const float v[3] = {v0, v1, v2};
#pragma unroll
        for (int k = 0; k < 3; ++k) {  // Kahan: (sum, error)
          const float2 o = z[k * ntg];
          const float y = __fsub_rn(v[k], o.y), n = __fadd_rn(o.x, y);
          z[k * ntg] = make_float2(n, __fsub_rn(__fsub_rn(n, o.x), y));
        }
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
    const int lc = WIDE ? 0 : t / nlon, j = q0 + t - lc * nlon, p = (cell0 + lc) * nv + j * a.nlat + ring;
    const double iA = 1.0 / a.tA[p];
    for (int k = 0; k < 3; ++k) {
      const float2 z0 = acc[k * ntg + t], z1 = acc[(3 + k) * ntg + t];
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
    for (int s = 0; s < 2; ++s)
      for (int k = 0; k < 4; ++k) {  // u, u_th, u_ph, u_thph of node (row k / 2, column k % 2)
        const float xu = c.x[k / 2], xd = c.x[2 + k / 2], yu = c.y[s][k % 2], yd = c.y[s][2 + k % 2];
        c.n[s][k][0] = xu * yu; c.n[s][k][1] = xd * yu; c.n[s][k][2] = xu * yd; c.n[s][k][3] = xd * yd;
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
  // a ring that does not fit in shared memory (about 1,300 columns) goes by
  // segments; under that a ring of more than 256 columns, several a thread, is
  // the faster (us, whole ring / segments: 4 cells of 16 x 260 585 / 610, 2 of
  // 16 x 520 606 / 639, of 16 x 1000 2270 / 2270).  Over it a ring went to the
  // FP64 patch: 1 cell of 10 x 1400 1820 -> 790.
  constexpr size_t COLUMN = sizeof(float4) * 2 * 3 + sizeof(float2) * 9;
  const bool wide = COLUMN * ctx->nlon > SMEM_BLOCK;
  a.G = wide ? 1 : ring_cells(ctx->ncell, ctx->nlon);
  a.seg = wide ? ring_segment(ctx->nlon, MIX_SEG) : 0;
  a.segs = wide ? (ctx->nlon + a.seg - 1) / a.seg : 1;
  const int blocks = (ctx->ncell + a.G - 1) / a.G * ctx->nlat * a.segs;
  const int thr = std::min(256, ((wide ? a.seg + 1 : a.G * ctx->nlon) + 31) / 32 * 32);
  a.parts = ring_parts(a.NC, blocks, nsm);
  const size_t cols = wide ? a.seg : a.G * ctx->nlon, ent = wide ? 2 * (a.seg + 1) : cols;
  const size_t bytes = sizeof(float4) * 2 * 3 * ent + sizeof(float2) * 9 * cols;
  auto launch = [&](auto kern) -> rbc3d_status {
    CUDA_TRY(smem_opt_in(kern, bytes));
    kern<<<blocks * a.parts, thr, bytes, ctx->st>>>(a);
    ++ctx->launches;
    CUDA_TRY(cudaGetLastError());
    return RBC3D_OK;
  };
  if (sl && dl) return wide ? launch(k_self_mix<true, true, true>) : launch(k_self_mix<true, true, false>);
  if (sl) return wide ? launch(k_self_mix<true, false, true>) : launch(k_self_mix<true, false, false>);
  return wide ? launch(k_self_mix<false, true, true>) : launch(k_self_mix<false, true, false>);
}
