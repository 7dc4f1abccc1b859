// selfring.cu -- RBC_SingInt (ModRbcSingInt.F90:29-90) in FP64 by latitude
// rings: the own-cell polar-patch quadrature of the FP64 and FP32C modes on a
// uniform longitude grid.
//
// The patch points of the targets of one latitude ring sit at the same
// colatitudes, shifted by whole longitude columns, and the patch is symmetric
// about the target's meridian: the points at azimuth +-a share their
// colatitude and mirror their longitude.  So the bicubic interpolation of
// Spline_Interp splits into
//   * per point pair (a "class") and column j, the theta part
//       U_j = u + x1 (u' - u) + x2 u_th + x3 u'_th   (rows i1 and i1 + 1 = '),
//       D_j the same of u_ph, u_thph,
//     once for the whole ring: 3 FMA for each of U, D and value;
//   * per point, the phi part U_j + y1 (U_j+1 - U_j) + y2 D_j + y3 D_j+1:
//     3 FMA a value, the difference shared by the pair.
// One point alone takes 16 FMA a value, here it is 3.3 + 3.5.  A thread owns a
// column j of a cell: it computes U_j and D_j, hands them to its neighbour
// through shared memory, and evaluates both points of the class that fall
// into the interval [j, j+1]: those of the targets j - jA and j - jB, whose
// positions and sums are in shared memory (a side each, so that no two
// threads meet).
//
// Bound by the FP64 pipe (2 lanes a clock and SM): about 140 FP64
// instructions a patch point, against about 350 (counting conversions) with one
// warp per target and 16-term interpolations.  256
// cells, SL+DL, inside the FP32C matvec: 46.1 -> 19.6 ms, the matvec 46.5 ->
// 20.1.  The node values are kept per row in column
// order (rec, built when positions or densities change), so that a warp reads
// consecutive columns: [cell][row][slot][value][column], slots u, u' - u,
// u_th, u_ph, u'_ph - u_ph, u_thph, values x, f, g, a3.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ctx.hpp"

namespace {

constexpr int RSLOT = 6, RVAL = 12;

struct RingArgs {
  int ncell, nlat, nlon, m, NC, G, parts, nt;
  const double* rec;
  const RingClass* cls;  // [latitude][NC]
  const double* spl;
  const double* th;
  const double* phi;
  const double* tA;
  double* v;
  const int* celltype;
  const double* Bc;
  Tables T;
  double c1, c2;
  int seg, segs;  // targets of a ring segment's block, blocks a ring (last: k_self_ring is
                  // 0.3 % slower with these before the pointers)
};

// Node values of the sets in `sets` (bit 0 x, 1 f, 2 g, 3 a3) in column order;
// a block takes 4 rows x 32 columns of one set of one cell.
__global__ void __launch_bounds__(128) k_ring_rec(int m, int n, const double* __restrict__ spl,
                                                  double* __restrict__ rec, int sets) {
  __shared__ double s[5][32][SPL_NODE + 1];
  const int nti = (m + 3) / 4, ntj = (n + 31) / 32;
  int b = blockIdx.x;
  const int jt = b % ntj; b /= ntj;
  const int it = b % nti; b /= nti;
  const int set = b % 4, cell = b / 4;
  if (!(sets & (1 << set))) return;
  const int src[4] = {SPL_X, SPL_F, SPL_G, SPL_A3};
  const double* in = spl + ((size_t)cell * SPL_NSET + src[set]) * (size_t)m * n * SPL_NODE;
  for (int e = threadIdx.x; e < 32 * 5 * SPL_NODE; e += blockDim.x) {
    const int q = e % SPL_NODE, r = (e / SPL_NODE) % 5, c = e / (5 * SPL_NODE);
    const int j = 32 * jt + c, i = (4 * it + r) % m;
    if (j < n) s[r][c][q] = in[((size_t)j * m + i) * SPL_NODE + q];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 4 * RSLOT * 3 * 32; e += blockDim.x) {
    const int c = e % 32, k = (e / 32) % 3, sl = (e / 96) % RSLOT, r = e / (96 * RSLOT);
    const int j = 32 * jt + c, i = 4 * it + r;
    if (j >= n || i >= m) continue;
    // spline kinds u, u_th, u_ph, u_thph are 0, 1, 2, 3
    const int kind[RSLOT] = {0, 0, 1, 2, 2, 3};
    const int q = 3 * kind[sl] + k;
    double v = s[r][c][q];
    if (sl == 1 || sl == 4) v = s[r + 1][c][q] - v;
    rec[(((size_t)cell * m + i) * RSLOT * RVAL + (size_t)sl * RVAL + 3 * set + k) * n + j] = v;
  }
}

// The values of a node or point: x, f, g, a3.
template <bool SL, bool DL>
struct RingVal {
  static constexpr int NV = 3 + (SL ? 3 : 0) + (DL ? 6 : 0), OF = 3, OG = 3 + (SL ? 3 : 0), OA = OG + 3;
  // U_j and D_j of a class from the column's node values (rc: row 0)
  static __device__ __forceinline__ void theta(const RingArgs& a, const RingClass& c, const double* rc, double* U,
                                               double* D) {
    const int nlon = a.nlon;
    const size_t rowlen = (size_t)RSLOT * RVAL * nlon;
    const double* r1 = rc + (size_t)c.i1 * rowlen;
    const double* r2 = rc + (size_t)(c.i1 + 1 == a.m ? 0 : c.i1 + 1) * rowlen;
    const double x1 = c.x[0], x2 = c.x[1], x3 = c.x[2];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int rv = (v < 3 || SL) ? v : v + 3;  // without f: g and a3 follow x
      U[v] = fma(x3, __ldg(r2 + (2 * RVAL + rv) * nlon),
                 fma(x2, __ldg(r1 + (2 * RVAL + rv) * nlon), fma(x1, __ldg(r1 + (RVAL + rv) * nlon), __ldg(r1 + rv * nlon))));
      D[v] = fma(x3, __ldg(r2 + (5 * RVAL + rv) * nlon),
                 fma(x2, __ldg(r1 + (5 * RVAL + rv) * nlon),
                     fma(x1, __ldg(r1 + (4 * RVAL + rv) * nlon), __ldg(r1 + (3 * RVAL + rv) * nlon))));
    }
  }
  // the point's term is cx p + cf f, p relative to the target; false: none
  static __device__ __forceinline__ bool term(const RingArgs& a, const double* p, double w1, double w2, bool dl,
                                              double& cx, double& cf) {
    const double r2 = fma(p[0], p[0], fma(p[1], p[1], p[2] * p[2]));
    double EA, EB, ED;
    if (!ewald_coef64<SL, DL>(a.T, r2, EA, EB, ED)) return false;  // rr >= rc: ModRbcSingInt.F90:65
    cx = cf = 0.;
    if (SL) {
      cx = w1 * EA * fma(p[0], p[OF], fma(p[1], p[OF + 1], p[2] * p[OF + 2]));
      cf = w1 * EB;
    }
    if (DL && dl) {
      const double dg = fma(p[0], p[OG], fma(p[1], p[OG + 1], p[2] * p[OG + 2]));
      const double da = fma(p[0], p[OA], fma(p[1], p[OA + 1], p[2] * p[OA + 2]));
      cx = fma(w2 * ED * dg, da, cx);
    }
    return true;
  }
};

// FEW: the form for few points, the same code with another shared-memory split
// (a kernel's split is the process's, as its opt-in: run_self_ring).
template <bool SL, bool DL, bool FEW>
__global__ void __launch_bounds__(256, 1) k_self_ring(RingArgs a) {
  using V = RingVal<SL, DL>;
  constexpr int NV = V::NV;
  extern __shared__ double sm[];
  const int t = threadIdx.x, W = blockDim.x, nlon = a.nlon;
  double* exU = sm;             // [NV][W]
  double* exD = exU + NV * W;   // [NV][W]
  double* sT = exD + NV * W;    // [3][W] target positions
  double* acc = sT + 3 * W;     // [2 sides][3][W]
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int ring = b % a.nlat, cell = (b / a.nlat) * a.G + t / nlon, j = t % nlon;
  const bool valid = t < a.G * nlon && cell < a.ncell;
  const int base = t - j;  // first column of this cell
  const int jn = j + 1 == nlon ? base : t + 1;
  double c2m = 0.;
  if (valid) {
    SplW sw;
    double xi[3];
    spline_weights(a.th[ring], a.phi[j], a.m, nlon, sw);
    spline_eval(a.spl + ((size_t)cell * SPL_NSET + SPL_X) * (size_t)a.m * nlon * SPL_NODE, sw, 3, xi);
    for (int k = 0; k < 3; ++k) sT[k * W + t] = xi[k];
    if (DL) c2m = a.c2 * a.Bc[a.celltype[cell]];
  }
  for (int k = 0; k < 6; ++k) acc[k * W + t] = 0.;
  const double* rc = a.rec + (size_t)(valid ? cell : 0) * a.m * RSLOT * RVAL * nlon + j;
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  for (int kc = k0; kc < k1; ++kc) {
    const RingClass& c = a.cls[(size_t)ring * a.NC + kc];
    double U[NV], D[NV];
    if (valid) V::theta(a, c, rc, U, D);
    __syncthreads();  // the previous class's values and sums are done with
    if (valid) {
#pragma unroll
      for (int v = 0; v < NV; ++v) { exU[v * W + t] = U[v]; exD[v * W + t] = D[v]; }
    }
    __syncthreads();
    if (!valid) continue;
    double dU[NV], E[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) { dU[v] = exU[v * W + jn] - U[v]; E[v] = exD[v * W + jn]; }
    const double w1 = SL ? a.c1 * c.w : 0., w2 = DL ? c2m * c.w : 0.;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int js = c.j[side];
      if (js < 0) break;  // the points on the meridian have no mirror image
      const int q = base + (j >= js ? j - js : j - js + nlon);  // the target's column
      const double y1 = c.y[side][0], y2 = c.y[side][1], y3 = c.y[side][2];
      double p[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) p[v] = fma(y3, E[v], fma(y2, D[v], fma(y1, dU[v], U[v])));
      for (int k = 0; k < 3; ++k) p[k] -= sT[k * W + q];
      double cx, cf;
      if (!V::term(a, p, w1, w2, c2m != 0., cx, cf)) continue;
      double* s = acc + 3 * side * W + q;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        double z = s[k * W];
        if (SL) z = fma(cf, p[V::OF + k], z);
        s[k * W] = fma(cx, p[k], z);
      }
    }
  }
  __syncthreads();
  if (!valid) return;
  const int p = cell * a.nlat * nlon + j * a.nlat + ring;
  const double iA = 1.0 / a.tA[p];
  for (int k = 0; k < 3; ++k) {
    const double dv = (acc[k * W + t] + acc[(3 + k) * W + t]) * iA;
    if (a.parts == 1) a.v[p + (size_t)k * a.nt] += dv;
    else atomicAdd(a.v + p + (size_t)k * a.nt, dv);
  }
}

// Rings of more than RING_MAX_NLON columns: a block takes a segment of the
// targets of one cell's ring, a thread a target.  Per class and side the theta
// parts of the segment's columns (and the next) go through shared memory to
// the neighbour as above, each column's twice in a ring (a side each), 6.6 +
// 3.5 FMA a value; the sums stay in registers.  FP32C matvecs against one warp per
// target and 16-term interpolations (us): 4 cells of 16 x 260 2210 -> 1300, 2 cells
// of 40 x 264 5290 -> 2830, of 16 x 520 2400 -> 1450, of 16 x 1000 5843 -> 3610.
template <bool SL, bool DL>
__global__ void __launch_bounds__(256, 1) k_self_ring_wide(RingArgs a) {
  using V = RingVal<SL, DL>;
  constexpr int NV = V::NV;
  extern __shared__ double sm[];
  const int t = threadIdx.x, W = blockDim.x, nlon = a.nlon;
  double* exU = sm;            // [NV][W]
  double* exD = exU + NV * W;  // [NV][W]
  int b = blockIdx.x;
  const int part = b % a.parts; b /= a.parts;
  const int q0 = b % a.segs * a.seg; b /= a.segs;
  const int ring = b % a.nlat, cell = b / a.nlat, n = min(a.seg, nlon - q0);
  double xi[3] = {0, 0, 0}, dv[3] = {0, 0, 0}, c2m = 0.;
  if (t < n) {
    SplW sw;
    spline_weights(a.th[ring], a.phi[q0 + t], a.m, nlon, sw);
    spline_eval(a.spl + ((size_t)cell * SPL_NSET + SPL_X) * (size_t)a.m * nlon * SPL_NODE, sw, 3, xi);
    if (DL) c2m = a.c2 * a.Bc[a.celltype[cell]];
  }
  const double* rc = a.rec + (size_t)cell * a.m * RSLOT * RVAL * nlon;
  const int k0 = (int)((long long)a.NC * part / a.parts), k1 = (int)((long long)a.NC * (part + 1) / a.parts);
  for (int kc = k0; kc < k1; ++kc) {
    const RingClass& c = a.cls[(size_t)ring * a.NC + kc];
    const double w1 = SL ? a.c1 * c.w : 0., w2 = DL ? c2m * c.w : 0.;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      if (c.j[side] < 0) break;  // the points on the meridian have no mirror image
      double U[NV], D[NV];
      if (t <= n) {
        const int j = q0 + t + c.j[side];
        V::theta(a, c, rc + (j >= nlon ? j - nlon : j), U, D);
      }
      __syncthreads();  // the previous values are done with
      if (t <= n) {
#pragma unroll
        for (int v = 0; v < NV; ++v) { exU[v * W + t] = U[v]; exD[v * W + t] = D[v]; }
      }
      __syncthreads();
      if (t >= n) continue;
      const double y1 = c.y[side][0], y2 = c.y[side][1], y3 = c.y[side][2];
      double p[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v)
        p[v] = fma(y3, exD[v * W + t + 1], fma(y2, D[v], fma(y1, exU[v * W + t + 1] - U[v], U[v])));
      for (int k = 0; k < 3; ++k) p[k] -= xi[k];
      double cx, cf;
      if (!V::term(a, p, w1, w2, c2m != 0., cx, cf)) continue;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (SL) dv[k] = fma(cf, p[V::OF + k], dv[k]);
        dv[k] = fma(cx, p[k], dv[k]);
      }
    }
  }
  if (t >= n) return;
  const int p = cell * a.nlat * nlon + (q0 + t) * a.nlat + ring;
  const double iA = 1.0 / a.tA[p];
  for (int k = 0; k < 3; ++k) {
    if (a.parts == 1) a.v[p + (size_t)k * a.nt] += dv[k] * iA;
    else atomicAdd(a.v + p + (size_t)k * a.nt, dv[k] * iA);
  }
}

}  // namespace

// Targets of one block of a wide ring, `most` at most (a block's threads are
// these and one column more): the most lanes in use.
int ring_segment(int nlon, int most) {
  int best = most;
  double top = -1.;
  for (int segs = (nlon + most - 1) / most; segs <= 2 * ((nlon + most - 1) / most) + 1; ++segs) {
    const int seg = (nlon + segs - 1) / segs, thr = (seg + 32) / 32 * 32;
    const double used = (double)nlon / ((double)segs * thr);
    if (used > top + 1e-9) { top = used; best = seg; }
  }
  return best;
}

// Cells per block: the most lanes in use (full warps of columns, no empty
// places in the last block).
int ring_cells(int ncell, int nlon) {
  int best = 1;
  double top = -1.;
  for (int G = 1; G == 1 || G * nlon <= 256; ++G) {
    const int thr = (G * nlon + 31) / 32 * 32;
    const double used = (double)ncell * nlon / ((double)((ncell + G - 1) / G) * thr);
    if (used > top + 1e-9) { top = used; best = G; }
  }
  return best;
}

// Under 12 blocks an SM several share a ring's classes, at least 8 each, and
// add their sums atomically (a block's set-up costs about half a class).
int ring_parts(int classes, int blocks, int nsm) {
  return std::max(1, std::min(classes / 8, (12 * nsm + blocks - 1) / blocks));
}

// Classes of the patch points per latitude: the points (irad, ia) and (irad,
// nazm - ia), in the order of their spline rows.
std::vector<RingClass> ring_classes(const rbc3d_ctx* ctx, const std::vector<double>& thG,
                                    const std::vector<double>& phiA, const std::vector<double>& pw) {
  const int nlat = ctx->nlat, nlon = ctx->nlon, m = 2 * nlat, nrad = ctx->nrad, nazm = ctx->nazm;
  const double hx = RBC3D_TWO_PI / m, hy = RBC3D_TWO_PI / nlon;
  const int NC = nrad * (nazm / 2 + 1);
  std::vector<RingClass> C((size_t)nlat * NC);
  for (int i0 = 0; i0 < nlat; ++i0) {
    RingClass* c = &C[(size_t)i0 * NC];
    for (int ia = 0; ia <= nazm / 2; ++ia)
      for (int ir = 0; ir < nrad; ++ir, ++c) {
        const size_t q = (size_t)i0 * nrad * nazm + ir;
        const double x = thG[q + (size_t)nrad * ia] * (1. / hx);
        const int i1 = (int)std::floor(x);
        const double s = x - i1;
        c->i1 = ((i1 % m) + m) % m;
        c->x[0] = s * s * (3. - 2. * s);
        c->x[1] = hx * s * (1. + s * (-2. + s));
        c->x[2] = hx * s * s * (-1. + s);
        c->w = pw[ir];
        for (int side = 0; side < 2; ++side) {
          c->j[side] = -1;
          if (side == 1 && (ia == 0 || 2 * ia == nazm)) continue;
          const double y = phiA[q + (size_t)nrad * (side ? nazm - ia : ia)] * (1. / hy);
          const int j1 = (int)std::floor(y);
          const double t = y - j1;
          c->j[side] = ((j1 % nlon) + nlon) % nlon;
          c->y[side][0] = t * t * (3. - 2. * t);
          c->y[side][1] = hy * t * (1. + t * (-2. + t));
          c->y[side][2] = hy * t * t * (-1. + t);
        }
      }
    std::stable_sort(&C[(size_t)i0 * NC], c, [](const RingClass& p, const RingClass& q) { return p.i1 < q.i1; });
  }
  return C;
}

rbc3d_status self_ring_grid(rbc3d_ctx* ctx, const std::vector<RingClass>& C) {
  CUDA_TRY(ctx->ring_cls.upload(reinterpret_cast<const char*>(C.data()), C.size() * sizeof(RingClass), ctx->st));
  CUDA_TRY(cudaStreamSynchronize(ctx->st));
  return RBC3D_OK;
}

// The Ewald tables as (value, step) pairs, entry by entry.
rbc3d_status self_ring_tables(rbc3d_ctx* ctx, const std::vector<double>& c1, const std::vector<double>& c2,
                              const std::vector<double>& dl) {
  std::vector<double> t(6 * (size_t)EWALD_NTAB);
  const std::vector<double>* src[3] = {&c1, &c2, &dl};
  for (int i = 0; i < EWALD_NTAB; ++i)
    for (int k = 0; k < 3; ++k) {
      t[6 * (size_t)i + 2 * k] = (*src[k])[i];
      t[6 * (size_t)i + 2 * k + 1] = (*src[k])[i + 1] - (*src[k])[i];
    }
  CUDA_TRY(ctx->ring_tab.upload(t.data(), t.size(), ctx->st));
  CUDA_TRY(cudaStreamSynchronize(ctx->st));
  return RBC3D_OK;
}

// FP64 own-cell patch on a uniform longitude grid.
rbc3d_status run_self_ring(rbc3d_ctx* ctx, int tlist, double c1, double c2) {
  TargetSet& t = ctx->tl[tlist];
  const bool sl = c1 != 0, dl = c2 != 0;
  if (!sl && !dl) return RBC3D_OK;
  const size_t per = (size_t)ctx->m * ctx->nlon * RSLOT * RVAL;
  if (!ctx->ring_rec.p || ctx->ring_rec.n < per * ctx->ncell) {
    CUDA_TRY(ctx->ring_rec.alloc(per * ctx->ncell));
    ctx->ring_sets = 0;
  }
  const int build = (1 | (sl ? 2 : 0) | (dl ? 4 | 8 : 0)) & ~ctx->ring_sets;
  if (build) {
    const long long nb = 4ll * ctx->ncell * ((ctx->m + 3) / 4) * ((ctx->nlon + 31) / 32);
    { k_ring_rec<<<(int)nb, 128, 0, ctx->st>>>(ctx->m, ctx->nlon, ctx->spl.p, ctx->ring_rec.p, build); ++ctx->launches; }
    CUDA_TRY(cudaGetLastError());
    ctx->ring_sets |= build;
  }
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device);
  RingArgs a;
  a.ncell = ctx->ncell; a.nlat = ctx->nlat; a.nlon = ctx->nlon; a.m = ctx->m; a.nt = t.n;
  a.NC = ctx->nrad * (ctx->nazm / 2 + 1);
  const bool wide = ctx->nlon > RING_MAX_NLON;
  a.G = wide ? 1 : ring_cells(ctx->ncell, ctx->nlon);
  a.seg = wide ? ring_segment(ctx->nlon, RING_MAX_NLON - 1) : 0;
  a.segs = wide ? (ctx->nlon + a.seg - 1) / a.seg : 1;
  const int blocks = (ctx->ncell + a.G - 1) / a.G * ctx->nlat * a.segs;
  const int thr = ((wide ? a.seg + 1 : a.G * ctx->nlon) + 31) / 32 * 32;
  a.parts = ring_parts(a.NC, blocks, nsm);
  a.rec = ctx->ring_rec.p; a.cls = reinterpret_cast<const RingClass*>(ctx->ring_cls.p); a.spl = ctx->spl.p;
  a.th = ctx->th.p; a.phi = ctx->phi.p; a.tA = t.Acoef.p; a.v = t.v.p; a.celltype = ctx->celltype.p; a.Bc = ctx->dBcoef.p;
  a.T = ctx->T;
  a.c1 = c1; a.c2 = c2;
  // few points: the pair kernels' shared-memory split of the SM, as no block
  // of another split starts beside this one (3 cells of 12 x 24: matvec 661 ->
  // 459 us, of 14 x 28 841 -> 617; of 25 x 50 1224 -> 1281, where the L1 counts)
  const bool few = t.n <= 2000;
  auto launch = [&](auto kern, int nv) -> rbc3d_status {
    const size_t bytes = sizeof(double) * (size_t)thr * (2 * nv + (wide ? 0 : 9));
    CUDA_TRY(smem_opt_in(kern, bytes));
    if (few && !wide)
      CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    kern<<<blocks * a.parts, thr, bytes, ctx->st>>>(a);
    ++ctx->launches;
    CUDA_TRY(cudaGetLastError());
    return RBC3D_OK;
  };
  if (wide) {
    if (sl && dl) return launch(k_self_ring_wide<true, true>, 12);
    if (sl) return launch(k_self_ring_wide<true, false>, 6);
    return launch(k_self_ring_wide<false, true>, 9);
  }
  if (sl && dl) return few ? launch(k_self_ring<true, true, true>, 12) : launch(k_self_ring<true, true, false>, 12);
  if (sl) return few ? launch(k_self_ring<true, false, true>, 6) : launch(k_self_ring<true, false, false>, 6);
  return few ? launch(k_self_ring<false, true, true>, 9) : launch(k_self_ring<false, true, false>, 9);
}
