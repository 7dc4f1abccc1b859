// pair.cu -- cell lists and the real-space Stokeslet / stresslet pair sums of
// AddIntOnRbcs (ModIntOnRbcs.F90:47-112) on the GPU.
//
// Cell list: the linked lists hoc/next of HashTable_Build (ModHashTable.F90:
// 23-62) become a stable radix sort of the points by cell id plus
// [start, end) ranges per cell.  The same Nc = max(floor(L/rc), 3) cells are
// used, so a target visits its 27 neighbour cells exactly as the reference.
//
// Pair kernel (k_pair, both precisions): a warp per work unit, the targets of
// one hash cell (equal-sized units, heaviest launched first): 32 targets of a
// lane each, or 16 or 8 of two or four lanes (pair_sub), the block's four warps
// together on a unit where targets are few (PAIR_SPLIT_MAX*).  A warp stages
// the tiles of 128 sources of the 27 neighbour cells whose boxes come within
// rc of its targets, skipping chunks of 32 that do not; every lane marks its
// candidates in bit lists and evaluates them, so lanes work on sources of
// their own.  Cell targets: the own cell's pairs (79% of the pairs of dense
// suspensions) go to a dense pass per cell (k_pair_own32, k_pair_own64), which
// evaluates a pair once for both points (cells that nearly meet their own
// image keep to the walk: k_own_records).
// FP32: sources carry hi/lo FP32
// coordinates relative to their own cell centre (from FP64, once per
// position update) and the targets are shifted into each neighbour cell's
// frame with an error-free difference, so x_j - x_i keeps full FP32 accuracy
// regardless of the box size; each target accumulates with Kahan
// compensation.  FP64 (the plain form): positions relative to the target
// cell centre, reference table arithmetic.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctx.hpp"

namespace {

constexpr int TILE = 128;
// Up to this many targets a block shares a unit (SPLIT of k_pair).  Measured,
// warps apart -> together (real part, us): FP64 3750 targets 1516 -> 770,
// 10000 2176 -> 1598, 25000 3909 -> 3676 (the whole matvec 7.06 -> 6.59 ms),
// 40000 6986 -> 6613 but the matvec 11.58 -> 11.63, 80000 19.48 -> 19.93; FP32
// 6250 targets 249 -> 168, 10000 325 -> 240 (matvec 600 -> 564), 13750
// 334 -> 280 but the matvec 663 -> 675, 16250 640 -> 693: blocks that wait for
// their longest warp hold shared memory that the patch beside them lacks.
constexpr int PAIR_SPLIT_MAX64 = 24000, PAIR_SPLIT_MAX32 = 12000;

// Sort keys: the hash cell; for targets (MORTON) followed by the place in the
// cell's 8 x 8 x 8 sub-cells along the Morton curve, so that the targets of a
// warp lie together and its box reaches few sources.
constexpr int MORTON_BITS = 9;
template <bool MORTON>
__global__ void k_hash_keys(int n, const double* __restrict__ x, int Nc0, int Nc1, int Nc2, double s0, double s1,
                            double s2, int* __restrict__ key, int* __restrict__ idx) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  // HashTable_Index, ModHashTable.F90:67-94 (single node): modulo(floor(x*Nc/L), Nc)
  const double u[3] = {x[p] * s0, x[p + n] * s1, x[p + 2 * (size_t)n] * s2};
  const double f[3] = {floor(u[0]), floor(u[1]), floor(u[2])};
  const int cell = imod((int)f[0], Nc0) + Nc0 * (imod((int)f[1], Nc1) + Nc1 * imod((int)f[2], Nc2));
  if (MORTON) {
    int m = 0;
    for (int d = 0; d < 3; ++d) {
      const int i = min(7, max(0, (int)(8.f * (float)(u[d] - f[d]))));
      m |= (i & 1) << d | (i & 2) << (d + 2) | (i & 4) << (d + 4);
    }
    key[p] = cell << MORTON_BITS | m;
  } else {
    key[p] = cell;
  }
  idx[p] = p;
}

__global__ void k_cell_ranges(int n, int shift, const int* __restrict__ key, int* __restrict__ cs, int* __restrict__ ce) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int k = key[p] >> shift;
  if (p == 0 || key[p - 1] >> shift != k) cs[k] = p;
  if (p == n - 1 || key[p + 1] >> shift != k) ce[k] = p + 1;
}

// Lists built on the device from sorted cell ranges (no host round trip).
// Every list has a fixed capacity (an upper bound on its length); the
// entries past its true length are empty (zero counts) and their consumers
// skip them.

// pieces[c] = ceil(count of cell c / P); pieces[nc] = 0 (the scan's total)
__global__ void k_piece_counts(int nc, const int* __restrict__ cs, const int* __restrict__ ce, int P,
                               int* __restrict__ pieces) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > nc) return;
  pieces[c] = c < nc ? (ce[c] - cs[c] + P - 1) / P : 0;
}

// (first, count) of the P-sized pieces of every cell, at off[c] (exclusive
// scan of the piece counts); entries [off[nc], cap) are cleared
__global__ void k_fill_pieces(int nc, const int* __restrict__ cs, const int* __restrict__ ce, int P,
                              const int* __restrict__ off, int cap, int2* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) {
    const int b0 = cs[c], e = ce[c];
    int k = off[c];
    for (int b = b0; b < e; b += P) out[k++] = make_int2(b, min(P, e - b));
  }
  for (int i = off[nc] + c; i < cap; i += gridDim.x * blockDim.x) out[i] = make_int2(0, 0);
}

// Work units of the pair sums (the cells' targets in equal-sized units of at
// most `tile`), keyed by their work: targets x the sources of the 27
// neighbour cells.  Unit counts first (k_piece_counts), then the units at the
// scanned offsets.
__global__ void k_fill_units(int nc, int tile, int Nc0, int Nc1, int Nc2, const int* __restrict__ cs, const int* __restrict__ ce,
                             const int* __restrict__ ss, const int* __restrict__ se, const int* __restrict__ off,
                             int cap, int4* __restrict__ units, long long* __restrict__ key, int* __restrict__ idx) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) {
    const int cnt = ce[c] - cs[c];
    if (cnt > 0) {
      const int ci = c % Nc0, cj = (c / Nc0) % Nc1, ck = c / (Nc0 * Nc1);
      long long nsrc = 0;
      for (int nb = 0; nb < 27; ++nb) {
        const int ni = (ci + nb % 3 - 1 + Nc0) % Nc0, nj = (cj + (nb / 3) % 3 - 1 + Nc1) % Nc1;
        const int nk = (ck + nb / 9 - 1 + Nc2) % Nc2;
        const int q = ni + Nc0 * (nj + Nc1 * nk);
        nsrc += se[q] - ss[q];
      }
      const int k = (cnt + tile - 1) / tile, per = (cnt + k - 1) / k;
      int u = off[c];
      for (int b = 0; b < cnt; b += per, ++u) {
        const int m = min(per, cnt - b);
        units[u] = make_int4(c, cs[c] + b, m, 0);
        key[u] = nsrc * m + 1;
        idx[u] = u;
      }
    }
  }
  for (int i = off[nc] + c; i < cap; i += gridDim.x * blockDim.x) {
    units[i] = make_int4(0, 0, 0, 0);
    key[i] = 0;
    idx[i] = i;
  }
}
__global__ void k_gather_units(int cap, const int* __restrict__ idx, const int4* __restrict__ in,
                               int4* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cap) out[i] = in[idx[i]];
}

// Gather cell-point geometry into cell-list order; clears the cells' flags of k_own_records.
__global__ void k_gather_src(int n, int nlat, int nv, const int* __restrict__ order, const double* __restrict__ x,
                             double* __restrict__ sx, int4* __restrict__ meta, int* __restrict__ wide) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  if (q < n / nv) wide[q] = 0;
  int p = order[q];
  for (int k = 0; k < 3; ++k) sx[q + (size_t)k * n] = x[p + (size_t)k * n];
  int cell = p / nv, r = p - cell * nv;
  meta[q] = make_int4(cell + 1, r % nlat, r / nlat, p);
}

// The sources' normals, sorted (FP64) and as FP32 records.
__global__ void k_gather_a3(int n, const int* __restrict__ order, const double* __restrict__ a3,
                            double* __restrict__ sa3, float4* __restrict__ a4) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int p = order[q];
  double v[3];
  for (int k = 0; k < 3; ++k) {
    v[k] = a3[p + (size_t)k * n];
    sa3[q + (size_t)k * n] = v[k];
  }
  a4[q] = make_float4((float)v[0], (float)v[1], (float)v[2], 0.f);
}

__device__ __forceinline__ double min_image(double d, double L, double iL) { return d - round(d * iL) * L; }

// FP32 pair-sum records of the sorted sources (see PairArgs); the normals'
// records come from k_gather_a3.
__global__ void k_src_records(int n, const double* __restrict__ sx, const int4* __restrict__ meta,
                              const float4* __restrict__ usph, int nlat, int Nc0, int Nc1, int Nc2, double h0,
                              double h1, double h2, double L0, double L1, double L2, float4* __restrict__ p0,
                              float4* __restrict__ p1, float4* __restrict__ u4) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int Nc[3] = {Nc0, Nc1, Nc2};
  const double h[3] = {h0, h1, h2}, L[3] = {L0, L1, L2};
  float hi[3], lo[3];
  for (int k = 0; k < 3; ++k) {
    const double x = sx[q + (size_t)k * n];
    const int c = imod((int)floor(x * (Nc[k] / L[k])), Nc[k]);  // HashTable_Index
    const double r = min_image(x - (c + 0.5) * h[k], L[k], 1.0 / L[k]);
    hi[k] = (float)r;
    lo[k] = (float)(r - (double)hi[k]);
  }
  const int4 m = meta[q];
  p0[q] = make_float4(hi[0], hi[1], hi[2], __int_as_float(m.x));
  p1[q] = make_float4(lo[0], lo[1], lo[2], __int_as_float(m.y | (m.z << 16)));
  u4[q] = usph[m.y + nlat * m.z];
}

// Bounding box of each tile (TILE consecutive sources of one cell), from the
// hi coordinates, with the range of the sources' surfaces in w (int bits);
// tiles listed as (first source, count).
__global__ void k_tile_boxes(const int2* __restrict__ tiles, const float4* __restrict__ p0, float4* __restrict__ box) {
  const int2 t = tiles[blockIdx.x];
  const float big = 3.0e38f;
  float3 lo = make_float3(big, big, big), hi = make_float3(-big, -big, -big);
  int smin = INT_MAX, smax = INT_MIN;
  for (int i = threadIdx.x; i < t.y; i += blockDim.x) {
    const float4 p = p0[t.x + i];
    lo.x = fminf(lo.x, p.x); lo.y = fminf(lo.y, p.y); lo.z = fminf(lo.z, p.z);
    hi.x = fmaxf(hi.x, p.x); hi.y = fmaxf(hi.y, p.y); hi.z = fmaxf(hi.z, p.z);
    smin = min(smin, __float_as_int(p.w)); smax = max(smax, __float_as_int(p.w));
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    smin = min(smin, __shfl_xor_sync(0xffffffffu, smin, o));
    smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, o));
  }
  __shared__ float3 red[32][2];
  __shared__ int sred[32][2];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { red[w][0] = lo; red[w][1] = hi; sred[w][0] = smin; sred[w][1] = smax; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      lo.x = fminf(lo.x, red[k][0].x); lo.y = fminf(lo.y, red[k][0].y); lo.z = fminf(lo.z, red[k][0].z);
      hi.x = fmaxf(hi.x, red[k][1].x); hi.y = fmaxf(hi.y, red[k][1].y); hi.z = fmaxf(hi.z, red[k][1].z);
      smin = min(smin, sred[k][0]); smax = max(smax, sred[k][1]);
    }
    box[2 * blockIdx.x] = make_float4(lo.x, lo.y, lo.z, __int_as_float(smin));
    box[2 * blockIdx.x + 1] = make_float4(hi.x, hi.y, hi.z, __int_as_float(smax));
  }
}

// Point-order records of the own-cell pair sums: hi/lo FP32 of the position
// relative to the cell's first point (at the minimum image), the grid indices, and
// the point's sorted source position.  The difference of two such positions is
// the pair's minimum image, or the pair is out of reach, while every component
// is under L - rc; a cell with a component of (L - rc) / 2 or more is flagged
// in wide[cell], and its own pairs stay in the cell-list walk.
__global__ void k_own_records(int n, int nlat, int nv, const double* __restrict__ x, const int* __restrict__ order,
                              double L0, double L1, double L2, double rc, float4* __restrict__ op0,
                              float4* __restrict__ op1, int* __restrict__ sinv, int* __restrict__ wide) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) sinv[order[q]] = q;
  const int p = q;
  if (p >= n) return;
  const int cell = p / nv, r = p - cell * nv;
  const double L[3] = {L0, L1, L2};
  float hi[3], lo[3];
  for (int k = 0; k < 3; ++k) {
    const double d = min_image(x[p + (size_t)k * n] - x[(size_t)cell * nv + (size_t)k * n], L[k], 1.0 / L[k]);
    if (2.0 * fabs(d) >= L[k] - 1.000001 * rc) wide[cell] = 1;  // (margin: the FP32 cutoff)
    hi[k] = (float)d;
    lo[k] = (float)(d - (double)hi[k]);
  }
  op0[p] = make_float4(hi[0], hi[1], hi[2], __int_as_float((r % nlat) | ((r / nlat) << 16)));
  op1[p] = make_float4(lo[0], lo[1], lo[2], 0.f);
}

// c1 f dS and c2 g dS Bcoef of the sorted sources in FP32 (per call).
__global__ void k_src_dens4(int n, double c1, double c2, const double* __restrict__ sf, const double* __restrict__ sg,
                            int do_f, int do_g, float4* __restrict__ F, float4* __restrict__ Gv) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  F[q] = do_f ? make_float4((float)(c1 * sf[q]), (float)(c1 * sf[q + n]), (float)(c1 * sf[q + 2 * (size_t)n]), 0.f)
              : make_float4(0.f, 0.f, 0.f, 0.f);
  if (do_g)
    Gv[q] = make_float4((float)(c2 * sg[q]), (float)(c2 * sg[q + n]), (float)(c2 * sg[q + 2 * (size_t)n]), 0.f);
}

// FP64 records of the sorted sources, 12 doubles each: position relative to
// the source's hash-cell centre, c1 f dS, c2 g dS Bcoef, a3 (per call).
__global__ void k_src_rec64(int n, double c1, double c2, const double* __restrict__ sx, const double* __restrict__ sf,
                            const double* __restrict__ sg, const double* __restrict__ sa3, int Nc0, int Nc1, int Nc2,
                            double h0, double h1, double h2, double L0, double L1, double L2, int do_f, int do_g,
                            double* __restrict__ rec) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int Nc[3] = {Nc0, Nc1, Nc2};
  const double h[3] = {h0, h1, h2}, L[3] = {L0, L1, L2};
  double* o = rec + 12 * (size_t)q;
  for (int k = 0; k < 3; ++k) {
    const double x = sx[q + (size_t)k * n];
    const int c = imod((int)floor(x * (Nc[k] / L[k])), Nc[k]);  // HashTable_Index
    o[k] = min_image(x - (c + 0.5) * h[k], L[k], 1.0 / L[k]);
    o[3 + k] = do_f ? c1 * sf[q + (size_t)k * n] : 0.;
    o[6 + k] = do_g ? c2 * sg[q + (size_t)k * n] : 0.;
    o[9 + k] = sa3[q + (size_t)k * n];
  }
}

// SourceList_UpdateDensity (ModSourceList.F90:160-189): f*dS, g*dS with
// dS = detJ*w(ilat); the sorted copy of g also carries Bcoef of the cell type.
__global__ void k_density(int n, int nlat, int nv, const double* __restrict__ f, const double* __restrict__ detJ,
                          const double* __restrict__ w, double* __restrict__ sf) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int ilat = (p % nv) % nlat;
  double ds = detJ[p] * w[ilat];
  for (int k = 0; k < 3; ++k) sf[p + (size_t)k * n] = f[p + (size_t)k * n] * ds;
}
__global__ void k_gather_density(int n, int nv, const int* __restrict__ order, const double* __restrict__ sf,
                                 const double* __restrict__ sg, const int* __restrict__ celltype,
                                 const double* __restrict__ Bc, double* __restrict__ ssf, double* __restrict__ ssg,
                                 int do_f, int do_g) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int p = order[q];
  double B = Bc[celltype[p / nv]];
  for (int k = 0; k < 3; ++k) {
    if (do_f) ssf[q + (size_t)k * n] = sf[p + (size_t)k * n];
    if (do_g) ssg[q + (size_t)k * n] = sg[p + (size_t)k * n] * B;
  }
}

struct PairArgs {
  // targets
  int nt;
  const double* tx;
  const double* tA;
  const int4* tmeta;
  const int* torder;
  const int4* units;
  int nunits;
  double* v;  // 3*nt accumulator
  // sources (sorted)
  int ns;
  const int* cs;
  const int* ce;
  // FP32 source records (sorted order) and tile boxes
  const float4* sp0;   // (x, y, z) hi relative to the source's hash-cell centre, surf bits
  const float4* sp1;   // (x, y, z) lo, id bits (ilat | ilon << 16)
  const float4* su;    // unit-sphere coordinates of the grid point
  const float4* sa4;   // a3
  const float4* sF4;   // c1 f dS
  const float4* sG4;   // c2 g dS Bcoef
  const int* toff;     // per hash cell: first tile (TILE consecutive sources per tile)
  const float4* tbox;  // per tile: lo, hi (relative to the cell centre)
  const int* coff;     // per hash cell: first 32-source chunk
  const float4* cbox;  // per chunk: lo, hi
  // grid
  int Nc[3];
  double h[3], L[3], iL[3];
  const double* th;
  const double* phi;
  const float4* usph;
  int nlat, nlon, nhalf;
  const double* mtab64;  // MaskFunc of same-cell grid pairs, (ilat_i, ilat_j, |dlon|), or null
  const float* mtab32;   // 1 - mask in FP32
  double radius, inv_radius;
  float inv_radius_f, chord2_max;
  double rc2;
  const double* rec64;  // FP64 source records
  const double* px;     // the points' positions (k_pair_own64)
  float rc2_f, reps2_f;
  float rc2_loose;  // (rc + 1e-3)^2: hi-part reject threshold of the FP32 pair kernel
  float rthr2_f;  // FP32 path: cross-surface pairs closer than this are left to the FP64 near-singular pass
  float sqpa_f, two_isqa_f, m8_ispi_f, q75_spi_f;  // sqrt(pi/alpha), 2/sqrt(alpha), -8/sqrt(pi), 0.75 sqrt(pi)
  float erfcx_q[ERFCX_DEG + 1];  // erfc(x) exp(x^2) = t Q(t), t = 1/(1 + x/2), on [0, rc sqrt(pi/alpha)]
  Tables T;
  // near-singular work list
  int collect;
  int4* items;
  int cap;
  unsigned long long* cnt;  // [0] items, [1] pairs, [2] overflow
  // own-cell pairs (cell targets, same-cell weight table): the dense pass takes
  // them and k_pair skips same-surface sources, but for the cells in wide
  int own_split;
  const int* wide;
  const float4* op0;  // per point (point order): (x, y, z) hi relative to its cell's first point, id bits
  const float4* op1;  // lo
  const int* sinv;    // point -> sorted source position
};


struct NbrList {
  int n;
  int surf[RBC3D_NBR_MAX];
  int idx[RBC3D_NBR_MAX];  // ilat | ilon << 16
  float d2[RBC3D_NBR_MAX];
  int overflow;
  __device__ __forceinline__ void insert(int s, int id, float d) {
    for (int e = 0; e < n; ++e)
      if (surf[e] == s) {
        if (d < d2[e]) { d2[e] = d; idx[e] = id; }
        return;
      }
    if (n < RBC3D_NBR_MAX) { surf[n] = s; idx[n] = id; d2[n] = d; ++n; }
    else overflow = 1;
  }
};

// Box-to-box distance test of the tile culling: true if every point of box
// [alo, ahi] is farther than sqrt(rc2) from every point of [blo, bhi].  The
// boxes hold FP32 coordinates; the margin absorbs their rounding.
__device__ __forceinline__ bool boxes_apart(float3 alo, float3 ahi, float3 blo, float3 bhi, float rc2) {
  float gx = fmaxf(0.f, fmaxf(alo.x - bhi.x, blo.x - ahi.x));
  float gy = fmaxf(0.f, fmaxf(alo.y - bhi.y, blo.y - ahi.y));
  float gz = fmaxf(0.f, fmaxf(alo.z - bhi.z, blo.z - ahi.z));
  float g = sqrtf(gx * gx + gy * gy + gz * gz) - 1e-3f;
  return g > 0.f && g * g > rc2;
}

__device__ __forceinline__ void warp_minmax(float3& lo, float3& hi) {
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
}

// Error-free a - b = s + e (Knuth TwoSum).
__device__ __forceinline__ void two_diff(float a, float b, float& s, float& e) {
  s = a - b;
  float bb = a - s;
  e = (a - (s + bb)) + (bb - b);
}

__device__ __forceinline__ float3 f3sub(float3 a, float3 d) { return make_float3(a.x - d.x, a.y - d.y, a.z - d.z); }

__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float2 ld2(const float* p, int j) { return *reinterpret_cast<const float2*>(p + j); }

// The coefficients of the Ewald real-space kernels (EwaldCoeff_SL /
// EwaldCoeff_DL, ModEwaldFunc.F90:86-180) at two pair distances at once, in
// packed FP32x2 arithmetic: the Stokeslet term A (x.f) x + B f and the
// stresslet factor Adl of (x.g)(x.n) x, for squared distances r2 (a pair of
// weight 0 enters with r^2 = 1, harmless).
template <bool SL, bool DL>
__device__ __forceinline__ void ewald_coef2(const PairArgs& a, float2 r2, float wa, float wb, float2& A, float2& B,
                                            float2& Adl) {
  const float2 sqpa2 = f2(a.sqpa_f, a.sqpa_f), half2 = f2(0.5f, 0.5f), one2 = f2(1.f, 1.f);
  const float2 tisqa2 = f2(a.two_isqa_f, a.two_isqa_f);
  const float2 rs = f2(wa != 0.f ? r2.x : 1.f, wb != 0.f ? r2.y : 1.f);
  const float2 rinv = f2(rsqrtf(rs.x), rsqrtf(rs.y));
  const float2 r = __fmul2_rn(rs, rinv);
  const float2 st = __fmul2_rn(r, sqpa2);
  const float2 ex = f2(__expf(-st.x * st.x), __expf(-st.y * st.y));
  const float2 den = __ffma2_rn(half2, st, one2);
  const float2 tq = f2(__fdividef(1.f, den.x), __fdividef(1.f, den.y));
  float2 Q = f2(a.erfcx_q[ERFCX_DEG], a.erfcx_q[ERFCX_DEG]);
#pragma unroll
  for (int k = ERFCX_DEG - 1; k >= 0; --k) Q = __ffma2_rn(Q, tq, f2(a.erfcx_q[k], a.erfcx_q[k]));
  const float2 c1 = __fmul2_rn(ex, __fmul2_rn(tq, Q)), c2 = __fmul2_rn(tisqa2, ex);
  const float2 ir2 = __fmul2_rn(rinv, rinv);
  if (SL) {
    const float2 c1r = __fmul2_rn(c1, rinv);
    A = __fmul2_rn(__fadd2_rn(c1r, c2), ir2);
    B = __fadd2_rn(c1r, f2(-c2.x, -c2.y));
  }
  if (DL) {
    const float2 st2 = __fmul2_rn(st, st);
    const float2 cdl = __fmul2_rn(f2(a.m8_ispi_f, a.m8_ispi_f),
                                  __ffma2_rn(ex, __fmul2_rn(st, __fadd2_rn(f2(1.5f, 1.5f), st2)),
                                             __fmul2_rn(f2(a.q75_spi_f, a.q75_spi_f), c1)));
    Adl = __fmul2_rn(__fmul2_rn(cdl, __fmul2_rn(ir2, ir2)), rinv);
  }
}

// A (x.f) x + B f + Adl (x.g)(x.n) x for two pairs (SL: the first two terms, DL: the last)
template <bool SL, bool DL>
__device__ __forceinline__ void ewald_apply2(float2 xx, float2 yy, float2 zz, float2 A, float2 B, float2 Adl,
                                             float2 fx, float2 fy, float2 fz, float2 gx, float2 gy, float2 gz,
                                             float2 nx, float2 ny, float2 nz, float2& vx, float2& vy, float2& vz) {
  if (SL) {
    const float2 Ad = __fmul2_rn(A, __ffma2_rn(xx, fx, __ffma2_rn(yy, fy, __fmul2_rn(zz, fz))));
    vx = __ffma2_rn(Ad, xx, __fmul2_rn(B, fx));
    vy = __ffma2_rn(Ad, yy, __fmul2_rn(B, fy));
    vz = __ffma2_rn(Ad, zz, __fmul2_rn(B, fz));
  }
  if (DL) {
    const float2 dg = __ffma2_rn(xx, gx, __ffma2_rn(yy, gy, __fmul2_rn(zz, gz)));
    const float2 da = __ffma2_rn(xx, nx, __ffma2_rn(yy, ny, __fmul2_rn(zz, nz)));
    const float2 t = __fmul2_rn(__fmul2_rn(Adl, dg), da);
    vx = SL ? __ffma2_rn(t, xx, vx) : __fmul2_rn(t, xx);
    vy = SL ? __ffma2_rn(t, yy, vy) : __fmul2_rn(t, yy);
    vz = SL ? __ffma2_rn(t, zz, vz) : __fmul2_rn(t, zz);
  }
}

// A warp's tile of up to TILE sources.  FP32: records of NQ float4 (hi
// coordinates and surface, lo coordinates and grid index, f, g, a3), read by
// lanes at sources of their own with 16-byte loads.  FP64: the FP32 hi
// coordinates of the tests and the FP64 values as a structure of arrays.
template <int NQ>
struct WarpTile32 {
  float4 r[TILE][NQ];
};
struct WarpTile64 {
  float4 p0[TILE];
  int id[TILE];
  double v[12][TILE];  // xyz, f, g, a3
};
template <typename R, bool SL, bool DL>
constexpr size_t warp_tile_bytes() {
  return sizeof(R) == 8 ? sizeof(WarpTile64) : sizeof(WarpTile32<2 + SL + 2 * DL>);
}

// Real-space pair sums (EwaldCoeff_SL / EwaldCoeff_DL of ModEwaldFunc over the
// 27 neighbour hash cells, AddIntOnRbcs ModIntOnRbcs.F90:25-160), one warp per
// unit of up to 32/SUB targets of one hash cell, SUB lanes per target.
//
// FP32: sources carry hi/lo coordinates relative to their own cell centre; per
// neighbour cell the targets are shifted into that frame with an error-free
// difference, so the pair vector keeps full FP32 accuracy however far from the
// origin the cells are; two sources at once in packed FP32x2 arithmetic, plain
// sums per 32-source chunk, Kahan-compensated across them.  FP64 (the plain form):
// the same frames in FP64, reference table arithmetic.
//
// Per tile (TILE consecutive sources of a cell; tiles and 32-source chunks
// whose bounding box is out of the warp's reach are skipped) a lane tests all
// its sources in FP32 (with a margin) and collects the survivors as bits; then
// the lanes pop their own bits, so a step evaluates a pair in every lane that
// has one left.  Before, all lanes walked the same sources and about 7 of 32
// had a pair to evaluate.  FP64 is bound by its pipe, FP32 by issue.
//
// SUB = 2, 4: that many lanes share a target, each with two or one of the
// tile's 32-source chunks, and merge sums and neighbour lists at the end: a
// half or a quarter of the serial work per warp where there are few targets
// (see pair_sub).
//
// SPLIT = 4: the four warps of a block share a unit as well, each with every
// fourth live tile, and merge in the same way.
template <typename R, bool SL, bool DL, int SUB, int SPLIT>
__global__ void __launch_bounds__(TILE, sizeof(R) == 8 ? 3 : 5) k_pair(PairArgs a) {
  constexpr bool F64 = sizeof(R) == 8;
  extern __shared__ __align__(16) unsigned char smem_pair[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int wu = SPLIT > 1 ? blockIdx.x : blockIdx.x * (TILE / 32) + wid;  // this warp's unit
  if (wu >= a.nunits) return;
  const int4 unit = a.units[wu];
  if (unit.z == 0) return;  // the empty tail
  constexpr int NQ = 2 + SL + 2 * DL;
  unsigned char* tile = smem_pair + wid * warp_tile_bytes<R, SL, DL>();
  WarpTile32<NQ>& C = *reinterpret_cast<WarpTile32<NQ>*>(tile);  // FP32
  WarpTile64& D = *reinterpret_cast<WarpTile64*>(tile);          // FP64
  const int cell = unit.x, sub = lane % SUB;
  const bool active = lane / SUB < unit.z;
  const int ci = cell % a.Nc[0], cj = (cell / a.Nc[0]) % a.Nc[1], ck = cell / (a.Nc[0] * a.Nc[1]);
  const double c0[3] = {(ci + 0.5) * a.h[0], (cj + 0.5) * a.h[1], (ck + 0.5) * a.h[2]};
  const int ti = active ? a.torder[unit.y + lane / SUB] : 0;
  double t64[3] = {0, 0, 0};
  float th_[3] = {0, 0, 0}, tl_[3] = {0, 0, 0};
  int surf_i = -2, own = -7, tlat = 0, tlon = 0;  // own: the surface whose pairs the dense pass takes
  bool grid = false;
  if (active) {
    for (int k = 0; k < 3; ++k) {
      t64[k] = min_image(a.tx[ti + (size_t)k * a.nt] - c0[k], a.L[k], a.iL[k]);
      th_[k] = (float)t64[k];
      tl_[k] = (float)(t64[k] - (double)th_[k]);
    }
    const int4 m = a.tmeta[ti];
    surf_i = m.x;
    if (a.own_split && !a.wide[m.x - 1]) own = m.x;
    if (m.y >= 0) { tlat = m.y; tlon = m.z; grid = true; }
  }
  float3 wlo0, whi0;
  {
    const float big = 3.0e38f;
    wlo0 = active ? make_float3(th_[0], th_[1], th_[2]) : make_float3(big, big, big);
    whi0 = active ? make_float3(th_[0], th_[1], th_[2]) : make_float3(-big, -big, -big);
    warp_minmax(wlo0, whi0);
  }
  Kahan3 acc;
  acc.zero();
  double acc64[3] = {0, 0, 0};
  NbrList L;
  L.n = 0; L.overflow = 0;
  int run_surf = -3, run_id = -1;
  R run_d2 = (R)3.4e38f;
  unsigned npairs = 0;  // < 2^32 pairs per target
  // own-cell pairs left to the dense pass: the warp's surface when all its
  // targets share one (whole tiles and chunks of it are skipped), else -7
  int wsurf = -7;
  if (a.own_split) {
    const int s0 = __shfl_sync(0xffffffffu, own, 0);
    wsurf = __all_sync(0xffffffffu, !active || own == s0) ? s0 : -7;
  }

  // 1 - MaskFunc of a pair on one cell
  auto same_weight = [&](int idj, int q) -> R {
    if (F64) {
      double m = 0.;
      if (a.mtab64) {
        int dl = abs((idj >> 16) - tlon);
        dl = min(dl, a.nlon - dl);
        m = __ldg(a.mtab64 + ((size_t)tlat * a.nlat + (idj & 0xffff)) * a.nhalf + dl);
      } else if (grid) {
        const double dth = dist_on_sphere(a.th[tlat], a.phi[tlon], a.th[idj & 0xffff], a.phi[idj >> 16]);
        m = mask64(a.T, dth * a.inv_radius);
      }
      return (R)(1. - m);
    }
    float w = 1.f;
    if (a.mtab32) {
      int dl = abs((idj >> 16) - tlon);
      dl = min(dl, a.nlon - dl);
      w = __ldg(a.mtab32 + (size_t)tlat * a.nlat * a.nhalf + (idj & 0xffff) * a.nhalf + dl);
    } else if (grid) {
      const float4 u = a.su[q], ui = a.usph[tlat + a.nlat * tlon];
      const float ex = ui.x - u.x, ey = ui.y - u.y, ez = ui.z - u.z;
      const float ch2 = ex * ex + ey * ey + ez * ez;
      if (ch2 < a.chord2_max) {
        const float t = 2.f * asinf(0.5f * sqrtf(ch2)) * a.inv_radius_f;
        const float sx = t * (float)MASK_NTAB;
        const int i = (int)sx;
        if (i < MASK_NTAB) {
          const float2 e = __ldg(a.T.mask32 + i);
          w = 1.f - (e.x + (sx - (float)i) * e.y);
        }
      }
    }
    return (R)w;
  };
  // bookkeeping of a source within rc (sorted index q), in source order: pair
  // count, neighbour-surface runs (each run's closest point merged into L by
  // surface), the weight (FP32: 0 for pairs left to the near-singular pass)
  auto weight = [&](int sj, int idj, int q, R r2) -> R {
    ++npairs;
    if (sj == surf_i) return same_weight(idj, q);
    if (a.collect) {
      if (sj != run_surf) {
        if (run_id >= 0) L.insert(run_surf, run_id, (float)run_d2);
        run_surf = sj; run_id = -1; run_d2 = (R)3.4e38f;
      }
      if (r2 < run_d2) { run_d2 = r2; run_id = idj; }
      if (!F64 && r2 < (R)a.rthr2_f) return (R)0;
    }
    return (R)1;
  };

  int turn = 0;  // SPLIT: live tiles so far, the same for the block's warps
  for (int nb = 0; nb < 27; ++nb) {
    const int dx = nb % 3 - 1, dy = (nb / 3) % 3 - 1, dz = nb / 9 - 1;
    const int ni = imod(ci + dx, a.Nc[0]), nj = imod(cj + dy, a.Nc[1]), nk = imod(ck + dz, a.Nc[2]);
    const int ncell = ni + a.Nc[0] * (nj + a.Nc[1] * nk);
    const int sbeg = a.cs[ncell], send = a.ce[ncell];
    if (sbeg >= send) continue;
    const double d64[3] = {dx * a.h[0], dy * a.h[1], dz * a.h[2]};
    const float3 dh = make_float3((float)d64[0], (float)d64[1], (float)d64[2]);
    float tsh[3], tsl[3];  // the target in the neighbour's frame
    {
      const float dl[3] = {(float)(d64[0] - (double)dh.x), (float)(d64[1] - (double)dh.y), (float)(d64[2] - (double)dh.z)};
      const float d3[3] = {dh.x, dh.y, dh.z};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float e;
        two_diff(th_[k], d3[k], tsh[k], e);
        tsl[k] = (tl_[k] - dl[k]) + e;
      }
    }
    const double tn[3] = {t64[0] - d64[0], t64[1] - d64[1], t64[2] - d64[2]};
    const float3 wlo = f3sub(wlo0, dh), whi = f3sub(whi0, dh);
    for (int base = sbeg, tt = a.toff[ncell], cc = a.coff[ncell]; base < send; base += TILE, ++tt, cc += TILE / 32) {
      const float4 blo = a.tbox[2 * tt], bhi = a.tbox[2 * tt + 1];
      if (boxes_apart(wlo, whi, make_float3(blo.x, blo.y, blo.z), make_float3(bhi.x, bhi.y, bhi.z), a.rc2_f)) continue;
      if (__float_as_int(blo.w) == wsurf && __float_as_int(bhi.w) == wsurf) continue;  // own cell only
      const int cnt = min(TILE, send - base);
      unsigned live = 0;  // chunks within reach (uniform over the warp)
#pragma unroll
      for (int w = 0; w < TILE / 32; ++w) {
        if (32 * w >= cnt) break;
        const float4 clo = a.cbox[2 * (cc + w)], chi = a.cbox[2 * (cc + w) + 1];
        if (!boxes_apart(wlo, whi, make_float3(clo.x, clo.y, clo.z), make_float3(chi.x, chi.y, chi.z), a.rc2_f) &&
            !(__float_as_int(clo.w) == wsurf && __float_as_int(chi.w) == wsurf))
          live |= 1u << w;
      }
      if (!live || (SPLIT > 1 && (turn++ & (SPLIT - 1)) != wid)) continue;
      __syncwarp();
#pragma unroll
      for (int w = 0; w < TILE / 32; ++w) {
        const int j = 32 * w + lane;
        if (!(live & (1u << w))) continue;
        if (j >= cnt) {  // padding: out of every target's reach
          const float4 far = make_float4(1.0e18f, 0.f, 0.f, __int_as_float(-9));
          if constexpr (F64) D.p0[j] = far;
          else C.r[j][0] = far;
          continue;
        }
        const int q = base + j;
        const float4 p0 = a.sp0[q], p1 = a.sp1[q];
        if constexpr (F64) {
          D.p0[j] = p0;
          D.id[j] = __float_as_int(p1.w);
          const double2* r = reinterpret_cast<const double2*>(a.rec64) + 6 * (size_t)q;
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            if ((!SL && (k == 2)) || (!DL && k >= 3)) continue;  // values 4, 5 (f) or 6.. (g, a3) unused
            const double2 v = r[k];
            D.v[2 * k][j] = v.x; D.v[2 * k + 1][j] = v.y;
          }
        } else {
          C.r[j][0] = p0;
          C.r[j][1] = p1;
          if (SL) C.r[j][2] = a.sF4[q];
          if (DL) { C.r[j][2 + SL] = a.sG4[q]; C.r[j][3 + SL] = a.sa4[q]; }
        }
      }
      __syncwarp();
      // the lane's candidates: bits of TILE/32/SUB words
      constexpr int NW = TILE / 32 / SUB;
      unsigned bits[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        bits[w] = 0;
        const int word = SUB == 1 ? w : w * SUB + sub;
        if (!active || !(live & (1u << word))) continue;
        unsigned m = 0;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
          const float4 p = F64 ? D.p0[32 * word + j] : C.r[32 * word + j][0];
          const float hx = p.x - tsh[0], hy = p.y - tsh[1], hz = p.z - tsh[2];
          const float h2 = fmaf(hx, hx, fmaf(hy, hy, hz * hz));
          if (h2 <= a.rc2_loose && __float_as_int(p.w) != own) m |= 1u << j;
        }
        bits[w] = m;
      }
      // a step: every lane that has a bit left evaluates its next source (FP32:
      // its next two of one chunk)
      int w = 0;
      unsigned m = bits[0];
      float cx = 0.f, cy = 0.f, cz = 0.f;
      for (;;) {
        if (NW > 1 && m == 0 && w < NW - 1) {  // the lane's next chunk
          acc.add(0, cx); acc.add(1, cy); acc.add(2, cz);
          cx = cy = cz = 0.f;
#pragma unroll
          for (int k = 1; k < NW; ++k)
            if (m == 0 && w < k) { w = k; m = bits[k]; }
        }
        if (!__any_sync(0xffffffffu, m != 0)) break;
        if (m == 0) continue;
        const int j0 = 32 * (SUB == 1 ? w : w * SUB + sub);
        const int ja = j0 + __ffs(m) - 1;
        m &= m - 1;
        if constexpr (F64) {
          const double x = D.v[0][ja] - tn[0], y = D.v[1][ja] - tn[1], z = D.v[2][ja] - tn[2];
          const double r2 = fma(x, x, fma(y, y, z * z));
          if (r2 > a.rc2) continue;
          const double wt = weight(__float_as_int(D.p0[ja].w), D.id[ja], base + ja, r2);
          double EA, EB, ED;
          if (!ewald_coef64<SL, DL>(a.T, r2, EA, EB, ED)) continue;
          double t = 0., b = 0.;
          if (SL) { t = EA * fma(x, D.v[3][ja], fma(y, D.v[4][ja], z * D.v[5][ja])); b = wt * EB; }
          if (DL) {
            const double dg = fma(x, D.v[6][ja], fma(y, D.v[7][ja], z * D.v[8][ja]));
            const double da = fma(x, D.v[9][ja], fma(y, D.v[10][ja], z * D.v[11][ja]));
            t = fma(ED * dg, da, t);
          }
          t *= wt;
          acc64[0] = fma(t, x, acc64[0]); acc64[1] = fma(t, y, acc64[1]); acc64[2] = fma(t, z, acc64[2]);
          if (SL) {
            acc64[0] = fma(b, D.v[3][ja], acc64[0]); acc64[1] = fma(b, D.v[4][ja], acc64[1]);
            acc64[2] = fma(b, D.v[5][ja], acc64[2]);
          }
        } else {
          const bool two = m != 0;
          const int jb = two ? j0 + __ffs(m) - 1 : ja;
          m &= m - 1;  // 0 stays 0
          const float4 pa = C.r[ja][0], pb = C.r[jb][0], la = C.r[ja][1], lb = C.r[jb][1];
          const float2 xx = __fadd2_rn(f2(pa.x - tsh[0], pb.x - tsh[0]), f2(la.x - tsl[0], lb.x - tsl[0]));
          const float2 yy = __fadd2_rn(f2(pa.y - tsh[1], pb.y - tsh[1]), f2(la.y - tsl[1], lb.y - tsl[1]));
          const float2 zz = __fadd2_rn(f2(pa.z - tsh[2], pb.z - tsh[2]), f2(la.z - tsl[2], lb.z - tsl[2]));
          const float2 r2 = __ffma2_rn(xx, xx, __ffma2_rn(yy, yy, __fmul2_rn(zz, zz)));
          float wa = 0.f, wb = 0.f;
          if (r2.x <= a.rc2_f) {
            wa = weight(__float_as_int(pa.w), __float_as_int(la.w), base + ja, r2.x);
            if (r2.x < a.reps2_f) wa = 0.f;
          }
          if (two && r2.y <= a.rc2_f) {
            wb = weight(__float_as_int(pb.w), __float_as_int(lb.w), base + jb, r2.y);
            if (r2.y < a.reps2_f) wb = 0.f;
          }
          if (wa == 0.f && wb == 0.f) continue;
          const float2 z2 = f2(0.f, 0.f);
          float2 A, B, Adl, vx, vy, vz, fx = z2, fy = z2, fz = z2, gx = z2, gy = z2, gz = z2, nx = z2, ny = z2, nz = z2;
          if (SL) {
            const float4 u = C.r[ja][2], v = C.r[jb][2];
            fx = f2(u.x, v.x); fy = f2(u.y, v.y); fz = f2(u.z, v.z);
          }
          if (DL) {
            const float4 u = C.r[ja][2 + SL], v = C.r[jb][2 + SL], s = C.r[ja][3 + SL], t = C.r[jb][3 + SL];
            gx = f2(u.x, v.x); gy = f2(u.y, v.y); gz = f2(u.z, v.z);
            nx = f2(s.x, t.x); ny = f2(s.y, t.y); nz = f2(s.z, t.z);
          }
          ewald_coef2<SL, DL>(a, r2, wa, wb, A, B, Adl);
          ewald_apply2<SL, DL>(xx, yy, zz, A, B, Adl, fx, fy, fz, gx, gy, gz, nx, ny, nz, vx, vy, vz);
          cx = fmaf(wb, vx.y, fmaf(wa, vx.x, cx));
          cy = fmaf(wb, vy.y, fmaf(wa, vy.x, cy));
          cz = fmaf(wb, vz.y, fmaf(wa, vz.x, cz));
        }
      }
      if (!F64) { acc.add(0, cx); acc.add(1, cy); acc.add(2, cz); }
    }
  }
  if (run_id >= 0) L.insert(run_surf, run_id, (float)run_d2);
  double sum[3];
  for (int k = 0; k < 3; ++k) sum[k] = F64 ? acc64[k] : (double)acc.s[k] - (double)acc.c[k];
  if (SUB > 1) {
    // the target's lanes: their sums, and their neighbour lists into lane 0's
    for (int o = 1; o < SUB; o <<= 1)
      for (int k = 0; k < 3; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    if (a.collect) {
      L.overflow = __any_sync(0xffffffffu, L.overflow);
      for (int r = 1; r < SUB; ++r) {
        const int src = (lane & ~(SUB - 1)) + r;
        const int nr = __shfl_sync(0xffffffffu, L.n, src);
        const int most = __reduce_max_sync(0xffffffffu, nr);
        for (int e = 0; e < most; ++e) {
          const int k = min(e, RBC3D_NBR_MAX - 1);
          const int sj = __shfl_sync(0xffffffffu, L.surf[k], src), id = __shfl_sync(0xffffffffu, L.idx[k], src);
          const float d = __shfl_sync(0xffffffffu, L.d2[k], src);
          if (sub == 0 && e < nr) L.insert(sj, id, d);
        }
      }
    }
  }
  if (SPLIT > 1) {
    // the block's warps: sums and lists of their targets to warp 0
    constexpr int NT = 32 / SUB;
    struct Merge {
      double sum[SPLIT][NT][3];
      int n[SPLIT][NT], surf[SPLIT][NT][RBC3D_NBR_MAX], idx[SPLIT][NT][RBC3D_NBR_MAX];
      float d2[SPLIT][NT][RBC3D_NBR_MAX];
    };
    static_assert(sizeof(Merge) <= TILE / 32 * warp_tile_bytes<R, SL, DL>(), "fits the tiles' shared memory");
    __syncthreads();
    Merge& M = *reinterpret_cast<Merge*>(smem_pair);
    const int t = lane / SUB;
    if (wid > 0 && sub == 0) {
      for (int k = 0; k < 3; ++k) M.sum[wid][t][k] = sum[k];
      M.n[wid][t] = L.overflow ? -1 : L.n;
      for (int e = 0; e < L.n; ++e) { M.surf[wid][t][e] = L.surf[e]; M.idx[wid][t][e] = L.idx[e]; M.d2[wid][t][e] = L.d2[e]; }
    }
    __syncthreads();
    if (wid == 0 && sub == 0)
      for (int r = 1; r < SPLIT; ++r) {
        for (int k = 0; k < 3; ++k) sum[k] += M.sum[r][t][k];
        if (M.n[r][t] < 0) L.overflow = 1;
        for (int e = 0; e < M.n[r][t]; ++e) L.insert(M.surf[r][t][e], M.idx[r][t][e], M.d2[r][t][e]);
      }
  }
  if (active && sub == 0 && (SPLIT == 1 || wid == 0)) {
    const double iA = 1.0 / a.tA[ti];
    // (beside the own-cell pass)
    for (int k = 0; k < 3; ++k) atomicAdd(a.v + ti + (size_t)k * a.nt, sum[k] * iA);
    if (a.collect) {
      if (L.overflow) atomicAdd(a.cnt + 2, 1ull);
      for (int e = 0; e < L.n; ++e) {
        const unsigned long long pos = atomicAdd(a.cnt + 0, 1ull);
        if (pos < (unsigned long long)a.cap) a.items[pos] = make_int4(ti, L.surf[e], L.idx[e] & 0xffff, L.idx[e] >> 16);
      }
    }
  }
  unsigned long long np = npairs;
  for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
  if (lane == 0 && np) atomicAdd(a.cnt + 1, np);
}

// Own-cell pairs of the FP32 modes: the pairs of AddIntOnRbcs whose source
// lies on the target's own cell with the weight 1 - MaskFunc of the same-cell
// table (ModIntOnRbcs.F90:77-80).  Every point of a biconcave cell lies
// within rc of every other (79% of the pairs within rc on the 256-cell
// workload), so per cell this is a dense all-pairs pass over tiles of
// OWN_TILE points in ring-major order, one CTA per (target tile T, source
// tile S >= T).  Pair (i, j) and pair (j, i) share the distance, the weight
// (the table is symmetric) and the kernel coefficients, so off the diagonal
// a CTA evaluates them once and adds both: to its target i (registers) and
// to its source j (per-warp sums in shared memory; at step s lane l takes
// the source pair (l + s) mod OWN_TILE/2, so the lanes of a warp touch
// distinct sources and read consecutive ones).  A diagonal CTA (S = T) takes
// every ordered pair of its tile one way.  The pair arithmetic is k_pair's
// (ewald_coef2 / ewald_apply2), positions hi/lo FP32 relative to the cell's
// first point, FP32 sums per 32 sources (Kahan-compensated across them) and
// per warp, added to the accumulator in FP64 atomically, beside k_pair.
// The target tile's at most (OWN_TILE - 1) / nlon + 2
// latitude rings' rows of the weight table sit in shared memory.
constexpr int OWN_TILE = 128;
// FP64: fewer than this many blocks of 128 points go in tiles of 32 (8 blocks
// of 4 warps an SM).  FP64 matvec, 128 -> 32 (us): 3 cells (165 blocks)
// 1761 -> 1533, 3 cells of 12 x 24 839 -> 675, 8 cells 3085 -> 2797, 12 cells
// 3850 -> 3800, 20 cells (1100) 6596 -> 6589, 64 cells (3520) 19927 -> 20133.
constexpr int OWN64_BLOCKS = 1216;
constexpr size_t OWN_MASK_MAX = 160 * 1024;  // weight-table rows of a block; wider grids keep their pairs in the walk
template <bool SL, bool DL>
__global__ void __launch_bounds__(OWN_TILE) k_pair_own32(PairArgs a) {
  __shared__ __align__(16) float s_src[15][OWN_TILE];  // hi xyz, lo xyz, f xyz, g xyz, normal xyz
  __shared__ __align__(16) int s_id[OWN_TILE];
  __shared__ __align__(16) float s_rev[OWN_TILE / 32][3][OWN_TILE];  // per warp: the sources' sums
  extern __shared__ float s_mask[];  // rows lat0.. of the table, nlat * nhalf each
  const int nlat = a.nlat, nlon = a.nlon, nv = nlat * nlon, rowlen = nlat * a.nhalf;
  const int ntile = (nv + OWN_TILE - 1) / OWN_TILE, npt = ntile * (ntile + 1) / 2;
  const int cell = blockIdx.x / npt;
  if (a.wide[cell]) return;  // k_pair takes this cell's pairs
  int r = blockIdx.x - cell * npt, T = 0;
  while (r >= ntile - T) { r -= ntile - T; ++T; }
  const int S = T + r;
  const bool diag = S == T;
  const int tid = threadIdx.x, wid = tid >> 5;
  const int k = T * OWN_TILE + tid;  // ring-major index of the target in its cell
  const bool active = k < nv;
  const int tlat = active ? k / nlon : 0, tlon = active ? k - tlat * nlon : 0;
  const int lat0 = T * OWN_TILE / nlon;
  const int nrow = min(nlat - 1, (T * OWN_TILE + OWN_TILE - 1) / nlon) - lat0 + 1;
  for (int i = tid; i < nrow * rowlen; i += OWN_TILE) s_mask[i] = a.mtab32[(size_t)lat0 * rowlen + i];
  const int p = cell * nv + tlon * nlat + tlat;  // the target's point index (= its target index)
  // the source tile, and the per-warp sums cleared
  const int js = S * OWN_TILE + tid;
  int ps = 0;
  if (js < nv) {
    const int sl = js / nlon;
    ps = cell * nv + (js - sl * nlon) * nlat + sl;
    const int q = a.sinv[ps];
    const float4 q0 = a.op0[ps], q1 = a.op1[ps], f = a.sF4[q];
    s_src[0][tid] = q0.x; s_src[1][tid] = q0.y; s_src[2][tid] = q0.z;
    s_src[3][tid] = q1.x; s_src[4][tid] = q1.y; s_src[5][tid] = q1.z;
    s_src[6][tid] = f.x; s_src[7][tid] = f.y; s_src[8][tid] = f.z;
    s_id[tid] = __float_as_int(q0.w);
    if (DL) {
      const float4 g = a.sG4[q], an = a.sa4[q];
      s_src[9][tid] = g.x; s_src[10][tid] = g.y; s_src[11][tid] = g.z;
      s_src[12][tid] = an.x; s_src[13][tid] = an.y; s_src[14][tid] = an.z;
    }
  } else {  // padding: a source beyond rc of every target
    for (int c = 0; c < 15; ++c) s_src[c][tid] = 0.f;
    s_src[0][tid] = 1.0e18f;
    s_id[tid] = 0;
  }
  for (int w = 0; w < OWN_TILE / 32; ++w)
    for (int c = 0; c < 3; ++c) s_rev[w][c][tid] = 0.f;
  // the target: position, and off the diagonal its densities for the reverse terms
  float4 t0 = make_float4(0.f, 0.f, 0.f, 0.f), t1 = t0, tf = t0, tg = t0, tn = t0;
  if (active) {
    t0 = a.op0[p];
    t1 = a.op1[p];
    if (!diag) {
      const int q = a.sinv[p];
      tf = a.sF4[q];
      if (DL) { tg = a.sG4[q]; tn = a.sa4[q]; }
    }
  }
  __syncthreads();
  const float2 nth0 = f2(-t0.x, -t0.x), nth1 = f2(-t0.y, -t0.y), nth2 = f2(-t0.z, -t0.z);
  const float2 ntl0 = f2(-t1.x, -t1.x), ntl1 = f2(-t1.y, -t1.y), ntl2 = f2(-t1.z, -t1.z);
  const float2 tfx = f2(tf.x, tf.x), tfy = f2(tf.y, tf.y), tfz = f2(tf.z, tf.z);
  const float2 tgx = f2(tg.x, tg.x), tgy = f2(tg.y, tg.y), tgz = f2(tg.z, tg.z);
  const float2 tnx = f2(-tn.x, -tn.x), tny = f2(-tn.y, -tn.y), tnz = f2(-tn.z, -tn.z);  // (x.g)(-x.n) x: reverse sign
  const float* mrow = s_mask + (tlat - lat0) * rowlen;
  Kahan3 acc;
  acc.zero();
  unsigned npairs = 0;
  const float2 z2 = f2(0.f, 0.f);
  float cx = 0.f, cy = 0.f, cz = 0.f;
  for (int step = 0; step < OWN_TILE / 2; ++step) {
    if (active) {
      const int j = 2 * ((tid + step) & (OWN_TILE / 2 - 1));
      const float2 xx = __fadd2_rn(__fadd2_rn(ld2(s_src[0], j), nth0), __fadd2_rn(ld2(s_src[3], j), ntl0));
      const float2 yy = __fadd2_rn(__fadd2_rn(ld2(s_src[1], j), nth1), __fadd2_rn(ld2(s_src[4], j), ntl1));
      const float2 zz = __fadd2_rn(__fadd2_rn(ld2(s_src[2], j), nth2), __fadd2_rn(ld2(s_src[5], j), ntl2));
      const float2 r2 = __ffma2_rn(xx, xx, __ffma2_rn(yy, yy, __fmul2_rn(zz, zz)));
      const bool oka = r2.x <= a.rc2_f, okb = r2.y <= a.rc2_f;
      npairs += ((unsigned)oka + (unsigned)okb) * (diag ? 1u : 2u);
      const int2 id = *reinterpret_cast<const int2*>(s_id + j);
      float wa = 0.f, wb = 0.f;
      if (oka && !(r2.x < a.reps2_f)) {
        int dl = abs((id.x >> 16) - tlon);
        dl = min(dl, nlon - dl);
        wa = mrow[(id.x & 0xffff) * a.nhalf + dl];
      }
      if (okb && !(r2.y < a.reps2_f)) {
        int dl = abs((id.y >> 16) - tlon);
        dl = min(dl, nlon - dl);
        wb = mrow[(id.y & 0xffff) * a.nhalf + dl];
      }
      if (wa != 0.f || wb != 0.f) {
        float2 A, B, Adl, vx, vy, vz;
        ewald_coef2<SL, DL>(a, r2, wa, wb, A, B, Adl);
        ewald_apply2<SL, DL>(xx, yy, zz, A, B, Adl, ld2(s_src[6], j), ld2(s_src[7], j), ld2(s_src[8], j),
                         DL ? ld2(s_src[9], j) : z2, DL ? ld2(s_src[10], j) : z2, DL ? ld2(s_src[11], j) : z2,
                         DL ? ld2(s_src[12], j) : z2, DL ? ld2(s_src[13], j) : z2, DL ? ld2(s_src[14], j) : z2, vx,
                         vy, vz);
        cx = fmaf(wb, vx.y, fmaf(wa, vx.x, cx));
        cy = fmaf(wb, vy.y, fmaf(wa, vy.x, cy));
        cz = fmaf(wb, vz.y, fmaf(wa, vz.x, cz));
        if (!diag) {  // pair (j, i): the vector is -x, so only the stresslet term changes sign
          ewald_apply2<SL, DL>(xx, yy, zz, A, B, Adl, tfx, tfy, tfz, tgx, tgy, tgz, tnx, tny, tnz, vx, vy, vz);
          const float2 w2 = f2(wa, wb);
          float2* rx = reinterpret_cast<float2*>(&s_rev[wid][0][j]);
          float2* ry = reinterpret_cast<float2*>(&s_rev[wid][1][j]);
          float2* rz = reinterpret_cast<float2*>(&s_rev[wid][2][j]);
          *rx = __ffma2_rn(w2, vx, *rx);
          *ry = __ffma2_rn(w2, vy, *ry);
          *rz = __ffma2_rn(w2, vz, *rz);
        }
      }
      if ((step & 15) == 15) {
        acc.add(0, cx);
        acc.add(1, cy);
        acc.add(2, cz);
        cx = cy = cz = 0.f;
      }
    }
    __syncwarp();  // the lanes' per-warp sums of this step are written before the next step's
  }
  __syncthreads();
  if (active) {
    const double iA = 1.0 / a.tA[p];
    for (int c = 0; c < 3; ++c) atomicAdd(a.v + p + (size_t)c * a.nt, ((double)acc.s[c] - (double)acc.c[c]) * iA);
  }
  if (!diag && js < nv) {
    const double iA = 1.0 / a.tA[ps];
    for (int c = 0; c < 3; ++c) {
      float sum = 0.f;
      for (int w = 0; w < OWN_TILE / 32; ++w) sum += s_rev[w][c][tid];
      atomicAdd(a.v + ps + (size_t)c * a.nt, (double)sum * iA);
    }
  }
  unsigned long long np = npairs;
  for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
  if ((tid & 31) == 0 && np) atomicAdd(a.cnt + 1, np);
}

// The same in FP64: one source a step (at step s lane l takes source
// (l + s) mod OT), coefficients by the reference's tables.  Bound by the
// FP64 pipe: about 66 instructions for both orders of a pair, against 75 and
// more for each order in the cell-list walk.
// Tiles of 32 where 128 would leave SMs short of blocks (OWN64_BLOCKS).
template <bool SL, bool DL, int OT>
__global__ void __launch_bounds__(OT) k_pair_own64(PairArgs a) {
  __shared__ double s_src[12][OT];  // xyz (relative to the cell's first point), f, g, normal
  __shared__ int s_id[OT];
  __shared__ double s_rev[OT / 32][3][OT];  // per warp: the sources' sums
  extern __shared__ double s_mask64[];  // rows lat0.. of the table, nlat * nhalf each
  const int nlat = a.nlat, nlon = a.nlon, nv = nlat * nlon, rowlen = nlat * a.nhalf;
  const int ntile = (nv + OT - 1) / OT, npt = ntile * (ntile + 1) / 2;
  const int cell = blockIdx.x / npt;
  if (a.wide[cell]) return;  // k_pair takes this cell's pairs
  int r = blockIdx.x - cell * npt, T = 0;
  while (r >= ntile - T) { r -= ntile - T; ++T; }
  const int S = T + r;
  const bool diag = S == T;
  const int tid = threadIdx.x, wid = tid >> 5;
  const int k = T * OT + tid;
  const bool active = k < nv;
  const int tlat = active ? k / nlon : 0, tlon = active ? k - tlat * nlon : 0;
  const int lat0 = T * OT / nlon;
  const int nrow = min(nlat - 1, (T * OT + OT - 1) / nlon) - lat0 + 1;
  for (int i = tid; i < nrow * rowlen; i += OT) s_mask64[i] = a.mtab64[(size_t)lat0 * rowlen + i];
  const int p = cell * nv + tlon * nlat + tlat, first = cell * nv;
  auto relative = [&](int point, int c) {
    return min_image(a.px[point + (size_t)c * a.ns] - a.px[first + (size_t)c * a.ns], a.L[c], a.iL[c]);
  };
  const int js = S * OT + tid;
  int ps = 0;
  if (js < nv) {
    const int sl = js / nlon;
    ps = cell * nv + (js - sl * nlon) * nlat + sl;
    const double* rec = a.rec64 + 12 * (size_t)a.sinv[ps];
    for (int c = 0; c < 3; ++c) s_src[c][tid] = relative(ps, c);
    for (int c = 3; c < 12; ++c)
      if ((SL && c < 6) || (DL && c >= 6)) s_src[c][tid] = rec[c];
    s_id[tid] = sl | ((js - sl * nlon) << 16);
  } else {  // padding: a source beyond rc of every target
    for (int c = 0; c < 12; ++c) s_src[c][tid] = 0.;
    s_src[0][tid] = 1.0e18;
    s_id[tid] = 0;
  }
  for (int w = 0; w < OT / 32; ++w)
    for (int c = 0; c < 3; ++c) s_rev[w][c][tid] = 0.;
  double tx[3] = {0, 0, 0}, tf[3] = {0, 0, 0}, tg[3] = {0, 0, 0}, tn[3] = {0, 0, 0};
  if (active) {
    const double* rec = a.rec64 + 12 * (size_t)a.sinv[p];
    for (int c = 0; c < 3; ++c) {
      tx[c] = relative(p, c);
      if (SL) tf[c] = rec[3 + c];
      if (DL) { tg[c] = rec[6 + c]; tn[c] = rec[9 + c]; }
    }
  }
  __syncthreads();
  const double* mrow = s_mask64 + (tlat - lat0) * rowlen;
  double acc[3] = {0, 0, 0};
  unsigned npairs = 0;
  for (int step = 0; step < OT; ++step) {
    if (active) {
      const int j = (tid + step) & (OT - 1);
      const double x = s_src[0][j] - tx[0], y = s_src[1][j] - tx[1], z = s_src[2][j] - tx[2];
      const double r2 = fma(x, x, fma(y, y, z * z));
      npairs += r2 <= a.rc2 ? (diag ? 1u : 2u) : 0u;
      double EA, EB, ED;
      if (ewald_coef64<SL, DL>(a.T, r2, EA, EB, ED)) {
        const int id = s_id[j];
        int dl = abs((id >> 16) - tlon);
        dl = min(dl, nlon - dl);
        const double wt = 1. - mrow[(id & 0xffff) * a.nhalf + dl];
        double t = 0., u = 0., b = 0., dg, da;
        if (SL) {
          EA *= wt;
          b = wt * EB;
          t = EA * fma(x, s_src[3][j], fma(y, s_src[4][j], z * s_src[5][j]));
        }
        if (DL) {
          ED *= wt;
          dg = fma(x, s_src[6][j], fma(y, s_src[7][j], z * s_src[8][j]));
          da = fma(x, s_src[9][j], fma(y, s_src[10][j], z * s_src[11][j]));
          t = fma(ED * dg, da, t);
        }
        acc[0] = fma(t, x, acc[0]); acc[1] = fma(t, y, acc[1]); acc[2] = fma(t, z, acc[2]);
        if (SL) {
          acc[0] = fma(b, s_src[3][j], acc[0]); acc[1] = fma(b, s_src[4][j], acc[1]); acc[2] = fma(b, s_src[5][j], acc[2]);
        }
        if (!diag) {  // pair (j, i): the vector is -x, so only the stresslet term changes sign
          if (SL) u = EA * fma(x, tf[0], fma(y, tf[1], z * tf[2]));
          if (DL) {
            dg = fma(x, tg[0], fma(y, tg[1], z * tg[2]));
            da = fma(x, tn[0], fma(y, tn[1], z * tn[2]));
            u = fma(-ED * dg, da, u);
          }
          const double xs[3] = {x, y, z};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            double v = fma(u, xs[c], s_rev[wid][c][j]);
            if (SL) v = fma(b, tf[c], v);
            s_rev[wid][c][j] = v;
          }
        }
      }
    }
    __syncwarp();  // the lanes' per-warp sums of this step are written before the next step's
  }
  __syncthreads();
  if (active) {
    const double iA = 1.0 / a.tA[p];
    for (int c = 0; c < 3; ++c) atomicAdd(a.v + p + (size_t)c * a.nt, acc[c] * iA);
  }
  if (!diag && js < nv) {
    const double iA = 1.0 / a.tA[ps];
    for (int c = 0; c < 3; ++c) {
      double sum = 0.;
      for (int w = 0; w < OT / 32; ++w) sum += s_rev[w][c][tid];
      atomicAdd(a.v + ps + (size_t)c * a.nt, sum * iA);
    }
  }
  unsigned long long np = npairs;
  for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
  if ((tid & 31) == 0 && np) atomicAdd(a.cnt + 1, np);
}

// AddLinearInt (ModIntOnRbcs.F90:162-201): xvint = sum Bcoef * x * (g.a3) dS
__global__ void k_linear_reduce(int n, int nv, const double* __restrict__ x, const double* __restrict__ sg,
                                const double* __restrict__ a3, const int* __restrict__ celltype,
                                const double* __restrict__ Bc, double* __restrict__ out) {
  double acc[3] = {0, 0, 0};
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    double vn = sg[p] * a3[p] + sg[p + n] * a3[p + n] + sg[p + 2 * (size_t)n] * a3[p + 2 * (size_t)n];
    double B = Bc[celltype[p / nv]];
    for (int k = 0; k < 3; ++k) acc[k] += B * x[p + (size_t)k * n] * vn;
  }
  for (int k = 0; k < 3; ++k) {
    double s = warp_sum(acc[k]);
    if ((threadIdx.x & 31) == 0) atomicAdd(out + k, s);
  }
}
__global__ void k_linear_add(int nt, const double* __restrict__ tA, const double* __restrict__ xv, double scale,
                             double* __restrict__ v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  double iA = 1.0 / tA[i];
  for (int k = 0; k < 3; ++k) v[i + (size_t)k * nt] += scale * xv[k] * iA;
}

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

rbc3d_status sort_points(rbc3d_ctx* ctx, int n, const double* x_dev, DBuf<int>& order, DBuf<int>& cs, DBuf<int>& ce,
                         bool targets = false) {
  const HashGrid& hg = ctx->hg;
  DBuf<int>&key = ctx->sort_key, &key2 = ctx->sort_key2, &idx = ctx->sort_idx;
  CUDA_TRY(key.alloc(n)); CUDA_TRY(key2.alloc(n)); CUDA_TRY(idx.alloc(n)); CUDA_TRY(order.alloc(n));
  CUDA_TRY(cs.alloc(hg.ncells)); CUDA_TRY(ce.alloc(hg.ncells));
  int bits = 1;
  while ((1ll << bits) < hg.ncells) ++bits;
  const bool morton = targets && bits + MORTON_BITS < 31;
  const int shift = morton ? MORTON_BITS : 0;
  auto keys = [&](auto kern) {
    kern<<<nblk(n, 256), 256, 0, ctx->st>>>(n, x_dev, hg.Nc[0], hg.Nc[1], hg.Nc[2], hg.Nc[0] / hg.L[0],
                                            hg.Nc[1] / hg.L[1], hg.Nc[2] / hg.L[2], key.p, idx.p);
    ++ctx->launches;
  };
  if (morton) keys(k_hash_keys<true>);
  else keys(k_hash_keys<false>);
  size_t tmp = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tmp, key.p, key2.p, idx.p, order.p, n, 0, bits + shift, ctx->st);
  DBuf<char>& tbuf = ctx->sort_tmp;
  CUDA_TRY(tbuf.alloc(tmp + 1));
  CUDA_TRY(cub::DeviceRadixSort::SortPairs(tbuf.p, tmp, key.p, key2.p, idx.p, order.p, n, 0, bits + shift, ctx->st));
  CUDA_TRY(cudaMemsetAsync(cs.p, 0, sizeof(int) * hg.ncells, ctx->st));
  CUDA_TRY(cudaMemsetAsync(ce.p, 0, sizeof(int) * hg.ncells, ctx->st));
  { k_cell_ranges<<<nblk(n, 256), 256, 0, ctx->st>>>(n, shift, key2.p, cs.p, ce.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  return RBC3D_OK;
}

// off = exclusive scan of cnt[0..nc] (nc + 1 entries; off[nc] the total), on the context stream
rbc3d_status scan_counts(rbc3d_ctx* ctx, int nc, const int* cnt, int* off) {
  size_t tmp = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tmp, cnt, off, nc + 1, ctx->st);
  DBuf<char>& tb = ctx->scan_tmp;
  CUDA_TRY(tb.alloc(tmp + 1));
  CUDA_TRY(cub::DeviceScan::ExclusiveSum(tb.p, tmp, cnt, off, nc + 1, ctx->st));
  return RBC3D_OK;
}

// The units of `tile` targets at most into `units` (cap entries, the empty
// tail last): per-cell counts, their scan, the units, a stable sort by work.
rbc3d_status fill_units(rbc3d_ctx* ctx, const DBuf<int>& cs, const DBuf<int>& ce, const int* ss, const int* se,
                        int tile, long long nsrc, int cap, DBuf<int4>& units) {
  const int nc = ctx->hg.ncells;
  rbc3d_status s;
  DBuf<int>& cnt = ctx->unit_cnt;
  CUDA_TRY(cnt.alloc(nc + 1)); CUDA_TRY(ctx->unit_off.alloc(nc + 1));
  CUDA_TRY(ctx->unit_tmp.alloc(cap)); CUDA_TRY(units.alloc(cap));
  CUDA_TRY(ctx->unit_key.alloc(2 * (size_t)cap)); CUDA_TRY(ctx->unit_idx.alloc(2 * (size_t)cap));
  const int g1 = nblk(nc + 1, 256);
  { k_piece_counts<<<g1, 256, 0, ctx->st>>>(nc, cs.p, ce.p, tile, cnt.p); ++ctx->launches; }
  if ((s = scan_counts(ctx, nc, cnt.p, ctx->unit_off.p))) return s;
  long long* key = ctx->unit_key.p;
  int* idx = ctx->unit_idx.p;
  { k_fill_units<<<g1, 256, 0, ctx->st>>>(nc, tile, ctx->hg.Nc[0], ctx->hg.Nc[1], ctx->hg.Nc[2], cs.p, ce.p, ss, se,
                                          ctx->unit_off.p, cap, ctx->unit_tmp.p, key, idx); ++ctx->launches; }
  // heaviest units first, so the last wave holds the light ones; the radix
  // sort is stable, so equal work keeps cell order (as a stable host sort);
  // the empty tail (key 0) stays last.  A key is at most tile times the sources, 24 of 64 bits at
  // 320,000: three of the sort's passes instead of eight (12 us each).
  int bits = 1;
  while (bits < 62 && (1ll << bits) <= (long long)tile * nsrc + 1) ++bits;
  size_t tmp = 0;
  cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, key, key + cap, idx, idx + cap, cap, 0, bits, ctx->st);
  DBuf<char>& tb = ctx->sort_tmp;
  CUDA_TRY(tb.alloc(tmp + 1));
  CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(tb.p, tmp, key, key + cap, idx, idx + cap, cap, 0, bits, ctx->st));
  { k_gather_units<<<nblk(cap, 256), 256, 0, ctx->st>>>(cap, idx + cap, ctx->unit_tmp.p, units.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  return RBC3D_OK;
}

// Lanes per target of the pair sums.  With one lane each and few units the
// longest warps set the time (256 cells: the walk's SMs active 74 % of its
// time); more lanes a target cost tile walks.  FP32D, the pair stage alone and
// the whole matvec (us) with 1 / 2 / 4 lanes, the own-cell pass beside the walk:
// 8 cells of 1,250 points 728 / 434 / 233 and 812 / 613 / 433; 24 cells 1112 / 689 /
// 570 and 1589 / 1223 / 1070; 40 cells 1287 / 818 / 654 and 1905 / 1394 / 1418; 64
// cells 1163 / 736 / 752 and 2012 / 1803 / 1915; 97 cells 1499 / 993 / 1103 and 3036 /
// 2634 / 2845; 128 cells 1519 / 1195 / 1506 and 3573 / 3532 / 3839; 160 cells 1746 /
// 1501 / 1886 and 4507 / 4475 / 4845 (FP32M 3369 / 3505 / 3884); 256 cells 2106 /
// 2250 / 2840 and 6468 / 6624 / 7204; 512 cells 13446 / 13781 / 14941.  FP64 matvecs
// (ms): 64 cells 19.3 / 19.2 / 19.5, 160 cells 50.9 / 50.9 / 51.9.
int pair_sub(int n) { return n <= 50000 ? 4 : n <= 180000 ? 2 : 1; }

rbc3d_status make_units(rbc3d_ctx* ctx, TargetSet& t, const DBuf<int>& cs, const DBuf<int>& ce) {
  const int nc = ctx->hg.ncells;
  // sources per cell: the source list's ranges (or the targets' own when
  // there is no source list)
  const bool src = ctx->npt > 0 && ctx->s_cstart.p;
  const int* ss = src ? ctx->s_cstart.p : cs.p;
  const int* se = src ? ctx->s_cend.p : ce.p;
  if (!src) {  // no sources: every unit weighs 0
    CUDA_TRY(ctx->unit_zero.alloc(nc));
    CUDA_TRY(cudaMemsetAsync(ctx->unit_zero.p, 0, sizeof(int) * nc, ctx->st));
    ss = se = ctx->unit_zero.p;
  }
  t.sub = pair_sub(t.n);
  const int tile = 32 / t.sub;
  // capacity: every non-empty cell gives at most count / tile + 1 units
  const int cap = nc + (t.n + tile - 1) / tile;
  t.nunits = cap;
  return fill_units(ctx, cs, ce, ss, se, tile, src ? (long long)ctx->npt : 0, cap, t.units);
}

}  // namespace


// erfc(x) exp(x^2) on [0, X] as t Q(t) with t = 1/(1 + x/2) (the variable of
// the Chebyshev erfc fit of Press et al., Numerical Recipes, sec. 6.2) and Q
// a degree-ERFCX_DEG polynomial: the truncated Chebyshev series of Q over the
// t-interval (projection on 64 Chebyshev nodes, FP64 std::erfc), converted to
// monomial coefficients in t.  Max relative error ~3e-7 in FP32 Horner for
// X = 4.24 (eps = 1e-6 at rc = 3), against ~1e-9 of the series itself.
void fit_erfcx(double X, float* q) {  // declared in ctx.hpp
  const int N = 64, D = ERFCX_DEG;
  const double tlo = 1.0 / (1.0 + 0.5 * X);
  const double a = 2.0 / (1.0 - tlo), b = -(1.0 + tlo) / (1.0 - tlo);  // s = a t + b in [-1, 1]
  double c[D + 1] = {0};
  for (int j = 0; j < N; ++j) {
    const double th = RBC3D_PI * (j + 0.5) / N, sj = std::cos(th), t = (sj - b) / a, x = 2.0 * (1.0 / t - 1.0);
    const double g = std::erfc(x) * std::exp(x * x) / t;
    for (int k = 0; k <= D; ++k) c[k] += 2.0 / N * g * std::cos(k * th);
  }
  c[0] *= 0.5;
  // sum c_k T_k(s), s = a t + b, as a polynomial in t: T_{k+1} = 2 s T_k - T_{k-1}
  double Tm[D + 1] = {0}, Tk[D + 1] = {0}, out[D + 1] = {0};
  Tm[0] = 1.0;                  // T_0
  Tk[0] = b; Tk[1] = a;         // T_1 = s
  for (int i = 0; i <= D; ++i) out[i] += c[0] * Tm[i];
  for (int k = 1; k <= D; ++k) {
    for (int i = 0; i <= D; ++i) out[i] += c[k] * Tk[i];
    double Tn[D + 1] = {0};
    for (int i = 0; i <= D; ++i) {
      Tn[i] += 2.0 * b * Tk[i] - Tm[i];
      if (i + 1 <= D) Tn[i + 1] += 2.0 * a * Tk[i];
    }
    for (int i = 0; i <= D; ++i) { Tm[i] = Tk[i]; Tk[i] = Tn[i]; }
  }
  for (int i = 0; i <= D; ++i) q[i] = (float)out[i];
}


rbc3d_status sort_points_by_cell(rbc3d_ctx* ctx, int n, const double* x_dev, DBuf<int>& order, DBuf<int>& cs,
                                DBuf<int>& ce) {
  return sort_points(ctx, n, x_dev, order, cs, ce);
}

rbc3d_status build_source_list(rbc3d_ctx* ctx, bool with_normals) {
  int n = ctx->npt;
  rbc3d_status s = sort_points(ctx, n, ctx->x.p, ctx->s_order, ctx->s_cstart, ctx->s_cend);
  if (s) return s;
  CUDA_TRY(ctx->s_x.alloc(3 * (size_t)n)); CUDA_TRY(ctx->s_a3.alloc(3 * (size_t)n)); CUDA_TRY(ctx->s_meta.alloc(n));
  CUDA_TRY(ctx->s_f.alloc(3 * (size_t)n)); CUDA_TRY(ctx->s_g.alloc(3 * (size_t)n));
  CUDA_TRY(ctx->s_wide.alloc(ctx->ncell));
  { k_gather_src<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->nlat, ctx->nlat * ctx->nlon, ctx->s_order.p, ctx->x.p,
                                                   ctx->s_x.p, ctx->s_meta.p, ctx->s_wide.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  // FP32 pair-sum records and tile boxes
  CUDA_TRY(ctx->s_p0.alloc(n)); CUDA_TRY(ctx->s_p1.alloc(n)); CUDA_TRY(ctx->s_u4.alloc(n)); CUDA_TRY(ctx->s_a4.alloc(n));
  if (with_normals && (s = source_normals(ctx))) return s;
  {
    const HashGrid& hg = ctx->hg;
    k_src_records<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->s_x.p, ctx->s_meta.p, ctx->usph.p, ctx->nlat,
                                                     hg.Nc[0], hg.Nc[1], hg.Nc[2], hg.h[0], hg.h[1], hg.h[2], hg.L[0],
                                                     hg.L[1], hg.L[2], ctx->s_p0.p, ctx->s_p1.p, ctx->s_u4.p);
    ++ctx->launches;
    CUDA_TRY(ctx->s_op0.alloc(n)); CUDA_TRY(ctx->s_op1.alloc(n)); CUDA_TRY(ctx->s_inv.alloc(n));
    { k_own_records<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->nlat, ctx->nlat * ctx->nlon, ctx->x.p, ctx->s_order.p,
                                                       hg.L[0], hg.L[1], hg.L[2], ctx->prm.rc, ctx->s_op0.p,
                                                       ctx->s_op1.p, ctx->s_inv.p, ctx->s_wide.p); ++ctx->launches; }
    CUDA_TRY(cudaGetLastError());
    const int nc = hg.ncells;
    // tiles of TILE and chunks of 32 consecutive sources of one cell, with
    // their offsets per cell and bounding boxes
    const int capt = nc + (n + TILE - 1) / TILE, capc = nc + (n + 31) / 32;
    CUDA_TRY(ctx->s_toff.alloc(nc + 1)); CUDA_TRY(ctx->s_coff.alloc(nc + 1));
    CUDA_TRY(ctx->unit_cnt.alloc(nc + 1));
    DBuf<int2>& lt = ctx->list_tmp;
    CUDA_TRY(lt.alloc((size_t)capc + capt));
    CUDA_TRY(ctx->s_cbox.alloc(2 * (size_t)capc + 2)); CUDA_TRY(ctx->s_tbox.alloc(2 * (size_t)capt + 2));
    const int g1 = nblk(nc + 1, 256);
    { k_piece_counts<<<g1, 256, 0, ctx->st>>>(nc, ctx->s_cstart.p, ctx->s_cend.p, 32, ctx->unit_cnt.p); ++ctx->launches; }
    if ((s = scan_counts(ctx, nc, ctx->unit_cnt.p, ctx->s_coff.p))) return s;
    { k_fill_pieces<<<g1, 256, 0, ctx->st>>>(nc, ctx->s_cstart.p, ctx->s_cend.p, 32, ctx->s_coff.p, capc, lt.p); ++ctx->launches; }
    { k_piece_counts<<<g1, 256, 0, ctx->st>>>(nc, ctx->s_cstart.p, ctx->s_cend.p, TILE, ctx->unit_cnt.p); ++ctx->launches; }
    if ((s = scan_counts(ctx, nc, ctx->unit_cnt.p, ctx->s_toff.p))) return s;
    { k_fill_pieces<<<g1, 256, 0, ctx->st>>>(nc, ctx->s_cstart.p, ctx->s_cend.p, TILE, ctx->s_toff.p, capt, lt.p + capc);
      ++ctx->launches; }
    { k_tile_boxes<<<capc, 32, 0, ctx->st>>>(lt.p, ctx->s_p0.p, ctx->s_cbox.p); ++ctx->launches; }
    { k_tile_boxes<<<capt, TILE, 0, ctx->st>>>(lt.p + capc, ctx->s_p0.p, ctx->s_tbox.p); ++ctx->launches; }
    CUDA_TRY(cudaGetLastError());
    ctx->s_ntiles = capt;
  }
  ctx->src_sorted = true;
  ctx->pme.cplan.valid = false;  // the PME tiles follow the source positions
  // tlist_rbc shares the source order
  TargetSet& t = ctx->tl[RBC3D_TLIST_RBC];
  t.sorted = false;
  return RBC3D_OK;
}

// The sorted sources' normals (a3 in source order and the FP32 records),
// once a3 is on the device.
rbc3d_status source_normals(rbc3d_ctx* ctx) {
  const int n = ctx->npt;
  if (n == 0) return RBC3D_OK;
  { k_gather_a3<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->s_order.p, ctx->a3.p, ctx->s_a3.p, ctx->s_a4.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  return RBC3D_OK;
}

rbc3d_status build_source_density(rbc3d_ctx* ctx) {
  int n = ctx->npt, nv = ctx->nlat * ctx->nlon;
  if (n == 0) return RBC3D_OK;
  const double* Bc = ctx->dBcoef.p;
  if (ctx->has_f) { k_density<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->nlat, nv, ctx->f.p, ctx->detJ.p, ctx->w.p, ctx->sf.p); ++ctx->launches; }
  if (ctx->has_g) { k_density<<<nblk(n, 256), 256, 0, ctx->st>>>(n, ctx->nlat, nv, ctx->g.p, ctx->detJ.p, ctx->w.p, ctx->sg.p); ++ctx->launches; }
  { k_gather_density<<<nblk(n, 256), 256, 0, ctx->st>>>(n, nv, ctx->s_order.p, ctx->sf.p, ctx->sg.p, ctx->celltype.p,
                                                       Bc, ctx->s_f.p, ctx->s_g.p, ctx->has_f, ctx->has_g); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  ctx->src_density = true;
  return RBC3D_OK;
}

rbc3d_status sort_targets(rbc3d_ctx* ctx, int tlist) {
  TargetSet& t = ctx->tl[tlist];
  if (t.sorted) return RBC3D_OK;
  rbc3d_status s;
  if (tlist == RBC3D_TLIST_RBC) {
    // same points in the same order as the sources
    CUDA_TRY(t.order.alloc(ctx->npt)); CUDA_TRY(t.cstart.alloc(ctx->hg.ncells)); CUDA_TRY(t.cend.alloc(ctx->hg.ncells));
    CUDA_TRY(cudaMemcpyAsync(t.order.p, ctx->s_order.p, sizeof(int) * ctx->npt, cudaMemcpyDeviceToDevice, ctx->st));
    CUDA_TRY(cudaMemcpyAsync(t.cstart.p, ctx->s_cstart.p, sizeof(int) * ctx->hg.ncells, cudaMemcpyDeviceToDevice, ctx->st));
    CUDA_TRY(cudaMemcpyAsync(t.cend.p, ctx->s_cend.p, sizeof(int) * ctx->hg.ncells, cudaMemcpyDeviceToDevice, ctx->st));
  } else {
    if ((s = sort_points(ctx, t.n, t.x.p, t.order, t.cstart, t.cend, true))) return s;
  }
  if ((s = make_units(ctx, t, t.cstart, t.cend))) return s;
  t.sorted = true;
  return RBC3D_OK;
}

rbc3d_status run_pair_sum(rbc3d_ctx* ctx, int tlist, double c1, double c2, int prec, bool collect_nbr) {
  if (ctx->npt == 0) return RBC3D_OK;
  TargetSet& t = ctx->tl[tlist];
  if (t.n == 0) return RBC3D_OK;
  rbc3d_status s = sort_targets(ctx, tlist);
  if (s) return s;
  PairArgs a;
  a.nt = t.n; a.tx = t.x.p; a.tA = t.Acoef.p; a.tmeta = t.meta.p; a.torder = t.order.p; a.v = t.v.p;
  a.units = t.units.p; a.nunits = t.nunits;
  a.ns = ctx->npt; a.cs = ctx->s_cstart.p; a.ce = ctx->s_cend.p;
  a.sp0 = ctx->s_p0.p; a.sp1 = ctx->s_p1.p; a.su = ctx->s_u4.p; a.sa4 = ctx->s_a4.p;
  a.toff = ctx->s_toff.p; a.tbox = ctx->s_tbox.p; a.coff = ctx->s_coff.p; a.cbox = ctx->s_cbox.p;
  for (int d = 0; d < 3; ++d) { a.Nc[d] = ctx->hg.Nc[d]; a.h[d] = ctx->hg.h[d]; a.L[d] = ctx->hg.L[d]; a.iL[d] = ctx->iLb[d]; }
  a.th = ctx->th.p; a.phi = ctx->phi.p; a.usph = ctx->usph.p; a.nlat = ctx->nlat;
  a.nlon = ctx->nlon; a.nhalf = ctx->nlon / 2 + 1;
  a.mtab64 = ctx->phi_uniform ? ctx->mtab64.p : nullptr;
  a.mtab32 = ctx->phi_uniform ? ctx->mtab32.p : nullptr;
  a.radius = ctx->radius; a.inv_radius = 1.0 / ctx->radius; a.inv_radius_f = (float)(1.0 / ctx->radius);
  double cm = 2.0 * sin(0.5 * ctx->radius) * (1.0 + 1e-6);
  a.chord2_max = (float)(cm * cm);
  a.rc2 = ctx->prm.rc * ctx->prm.rc; a.rc2_f = (float)a.rc2;
  a.px = ctx->x.p;
  a.rc2_loose = (float)((ctx->prm.rc + 1e-3) * (ctx->prm.rc + 1e-3)); a.reps2_f = (float)(ctx->T.r_eps * ctx->T.r_eps);
  const double rthr = near_rthr_now(ctx);
  a.rthr2_f = (float)(rthr * rthr);
  a.sqpa_f = (float)sqrt(RBC3D_PI / ctx->prm.alpha);
  a.two_isqa_f = (float)(2.0 / sqrt(ctx->prm.alpha));
  a.m8_ispi_f = (float)(-8.0 / sqrt(RBC3D_PI));
  a.q75_spi_f = (float)(0.75 * sqrt(RBC3D_PI));
  erfcx_coeffs(ctx);
  for (int k = 0; k <= ERFCX_DEG; ++k) a.erfcx_q[k] = ctx->erfcx_q[k];
  a.T = ctx->T;
  a.collect = collect_nbr ? 1 : 0;
  a.items = ctx->items.p; a.cap = ctx->items_cap; a.cnt = ctx->dcnt.p;
  const bool dl = c2 != 0.0 && ctx->has_g, sl = c1 != 0.0 && ctx->has_f;
  const int n = ctx->npt, nb = (t.nunits + TILE / 32 - 1) / (TILE / 32);
  const HashGrid& hg = ctx->hg;
  // own-cell pairs of the cell targets by the dense pass when the same-cell
  // weights come from the table (uniform longitudes)
  const bool f64 = prec == RBC3D_FP64;
  const int nv = ctx->nlat * ctx->nlon;
  // FP64 own-cell tiles: 128 points, or 32 where those are under OWN64_BLOCKS
  auto own_blocks = [&](int tile) {
    const long long nt = (nv + tile - 1) / tile;
    return ctx->ncell * (nt * (nt + 1) / 2);
  };
  const int own_tile = f64 && own_blocks(OWN_TILE) < OWN64_BLOCKS ? 32 : OWN_TILE;
  const int nrow = std::min(ctx->nlat, (own_tile - 1) / std::max(ctx->nlon, 1) + 2);
  const size_t own_sm = (f64 ? sizeof(double) : sizeof(float)) * (size_t)nrow * ctx->nlat * a.nhalf;
  const bool own = tlist == RBC3D_TLIST_RBC && a.mtab32 && t.n == n && ctx->s_op0.p && own_sm <= OWN_MASK_MAX;
  a.own_split = own ? 1 : 0;
  a.op0 = ctx->s_op0.p; a.op1 = ctx->s_op1.p; a.sinv = ctx->s_inv.p; a.wide = ctx->s_wide.p;
  if (f64) {
    CUDA_TRY(ctx->s_rec64.alloc(12 * (size_t)n));
    a.rec64 = ctx->s_rec64.p;
    { k_src_rec64<<<nblk(n, 256), 256, 0, ctx->st>>>(n, c1, c2, ctx->s_x.p, ctx->s_f.p, ctx->s_g.p, ctx->s_a3.p, hg.Nc[0],
                                                     hg.Nc[1], hg.Nc[2], hg.h[0], hg.h[1], hg.h[2], hg.L[0], hg.L[1],
                                                     hg.L[2], sl, dl, ctx->s_rec64.p); ++ctx->launches; }
  } else {
    CUDA_TRY(ctx->s_F4.alloc(n));
    if (dl) CUDA_TRY(ctx->s_G4.alloc(n));
    a.sF4 = ctx->s_F4.p; a.sG4 = ctx->s_G4.p;
    { k_src_dens4<<<nblk(n, 256), 256, 0, ctx->st>>>(n, c1, c2, ctx->s_f.p, ctx->s_g.p, sl, dl,
                                                     ctx->s_F4.p, ctx->s_G4.p); ++ctx->launches; }
  }
  auto launch = [&](auto kern, int blocks, size_t bytes, size_t most, int threads = TILE) -> rbc3d_status {
    // (static and dynamic shared memory together may pass the 48 KB that need no opt-in)
    CUDA_TRY(smem_opt_in(kern, bytes, most));
    kern<<<blocks, threads, bytes, ctx->st>>>(a);
    ++ctx->launches;
    CUDA_TRY(cudaGetLastError());
    return RBC3D_OK;
  };
  auto pairs = [&](auto R, auto SL, auto DL) -> rbc3d_status {
    using T = decltype(R);
    const size_t bytes = TILE / 32 * warp_tile_bytes<T, SL.value, DL.value>();
    if (t.sub == 4 && t.n <= (sizeof(T) == 8 ? PAIR_SPLIT_MAX64 : PAIR_SPLIT_MAX32)) return launch(k_pair<T, SL.value, DL.value, 4, 4>, t.nunits, bytes, bytes);
    if (t.sub == 4) return launch(k_pair<T, SL.value, DL.value, 4, 1>, nb, bytes, bytes);
    if (t.sub == 2) return launch(k_pair<T, SL.value, DL.value, 2, 1>, nb, bytes, bytes);
    return launch(k_pair<T, SL.value, DL.value, 1, 1>, nb, bytes, bytes);
  };
  auto own_pairs = [&](auto R, auto SL, auto DL) -> rbc3d_status {
    const int blocks = (int)own_blocks(own_tile);
    if (sizeof(R) == 4) return launch(k_pair_own32<SL.value, DL.value>, blocks, own_sm, OWN_MASK_MAX);
    if (own_tile == 32) return launch(k_pair_own64<SL.value, DL.value, 32>, blocks, own_sm, OWN_MASK_MAX, 32);
    return launch(k_pair_own64<SL.value, DL.value, OWN_TILE>, blocks, own_sm, OWN_MASK_MAX);
  };
  const std::true_type yes{};
  const std::false_type no{};
  auto run = [&](auto R) -> rbc3d_status {
    // without a density the walk still counts pairs and lists neighbours: as the single layer of zeros
    // The own-cell pass on a low-priority stream beside the walk, where it
    // fills the SMs that the walk's last units leave idle.  After it / beside it
    // (us): 256 cells pair stage 2700 / 2122, FP32D matvec 7156 / 6936, FP32M
    // 5502 / 5253; 97 cells 2743 / 2619; 8 cells 558 / 513; 2048 cells 54787 /
    // 54844.  At the walk's priority 7018 and 5417.  FP64 with PME on the side
    // stream: 3 cells 1490 / 1218, 3 cells of 12 x 24 525 / 459, 8 cells 2812 /
    // 2770, 64 cells 19385 / 19287, 9 cells of 36 x 72 9203 / 9317.
    const bool beside = own && ctx->st3;
    if (beside) {
      CUDA_TRY(cudaEventRecord(ctx->ev_pair, ctx->st));
      CUDA_TRY(cudaStreamWaitEvent(ctx->st3, ctx->ev_pair, 0));
    }
    rbc3d_status e = sl && dl ? pairs(R, yes, yes) : dl ? pairs(R, no, yes) : pairs(R, yes, no);
    if (e || !own) return e;
    if (beside) std::swap(ctx->st, ctx->st3);
    e = sl && dl ? own_pairs(R, yes, yes) : dl ? own_pairs(R, no, yes) : own_pairs(R, yes, no);
    if (beside) {
      std::swap(ctx->st, ctx->st3);
      CUDA_TRY(cudaEventRecord(ctx->ev_own, ctx->st3));
      CUDA_TRY(cudaStreamWaitEvent(ctx->st, ctx->ev_own, 0));
    }
    return e;
  };
  return f64 ? run(0.0) : run(0.f);
}

rbc3d_status run_linear(rbc3d_ctx* ctx, int tlist, double c2) {
  if (c2 == 0.0 || ctx->npt == 0 || !ctx->has_g) return RBC3D_OK;
  TargetSet& t = ctx->tl[tlist];
  const double* Bc = ctx->dBcoef.p;
  CUDA_TRY(ctx->xvint.alloc(3));
  CUDA_TRY(cudaMemsetAsync(ctx->xvint.p, 0, 3 * sizeof(double), ctx->st));
  { k_linear_reduce<<<304, 256, 0, ctx->st>>>(ctx->npt, ctx->nlat * ctx->nlon, ctx->x.p, ctx->sg.p, ctx->a3.p,
                                            ctx->celltype.p, Bc, ctx->xvint.p); ++ctx->launches; }
  double pil = ctx->iLb[0] * ctx->iLb[1] * ctx->iLb[2];
  if (t.n) { k_linear_add<<<nblk(t.n, 256), 256, 0, ctx->st>>>(t.n, t.Acoef.p, ctx->xvint.p, c2 * (-8 * RBC3D_PI * pil), t.v.p); ++ctx->launches; }
  CUDA_TRY(cudaGetLastError());
  return RBC3D_OK;
}

void erfcx_coeffs(rbc3d_ctx* ctx) {
  const double X = ctx->prm.rc * std::sqrt(RBC3D_PI / ctx->prm.alpha);
  if (ctx->erfcx_X != X) {
    ctx->erfcx_X = X;
    fit_erfcx(X, ctx->erfcx_q);
  }
}
