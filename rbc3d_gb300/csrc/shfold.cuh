// shfold.cuh -- longitude sums of the spherical-harmonic transforms on a quarter
// of the columns.  With phi_j = phi_0 + 2 pi j / nlon and nlon even, the columns
// j, nlon - j, nlon/2 - j and nlon/2 + j have the same |cos m phi| and |sin m phi|:
//   cos: 1, 1, (-1)^m, (-1)^m     sin: 1, -1, -(-1)^m, (-1)^m.
// The analysis adds the four columns once, for every m, and sums over j <= nlon/4;
// the synthesis sums the even and odd m of the cosine and the sine terms apart
// and combines them four ways.  Bound by the FP64 pipe (2 lanes a clock and SM):
// of the 14 and 7 operations a column and m of the plain sums 2 to 4 stay.
// Angles are taken from phi_0, which turns the coefficients and changes no
// field value.  256 cells of 25 x 50: a spline table set (degree 12) 268 -> 124
// us, the gradient of 768 fields (degree 25) 682 -> 195 us; what is left is the
// FP64 pipe (about 70 and 130 us) and the barriers between the sums.  Blocks of
// 128 threads, six or more an SM: one wave of 768 blocks.
#pragma once
#include <cmath>
#include <vector>

namespace {

// cos, sin, m cos, m sin of 2 pi m j / nlon, [m][j], j <= nlon / 4
inline std::vector<Fold4> fold_table(int L, int nlon) {
  const int nq = nlon / 4 + 1;
  std::vector<Fold4> t((size_t)L * nq);
  for (int m = 0; m < L; ++m)
    for (int j = 0; j < nq; ++j) {
      const double x = RBC3D_TWO_PI * (((long long)m * j) % nlon) / nlon, c = std::cos(x), s = std::sin(x);
      t[(size_t)m * nq + j] = Fold4{c, s, m * c, m * s};
    }
  return t;
}

// g[i + nrow j], in place: column j <- cosine sums of even m, nlon/2 - j of odd m,
// nlon/2 + j <- sine sums of even m, nlon - j of odd m.  At j = 0 (no sines) and
// j = nlon/4 exactly (no cosines of odd m, no sines of even m) columns coincide.
__device__ __forceinline__ void fold_columns(int nrow, int nlon, double* g) {
  const int N2 = nlon / 2, nq = nlon / 4 + 1;
  for (int t = threadIdx.x; t < nrow * nq; t += blockDim.x) {
    const int j = t / nrow;
    double* p = g + (t - j * nrow);
    if (j == 0) {
      const double a = p[0], c = p[nrow * N2];
      p[0] = a + c;
      p[nrow * N2] = a - c;
    } else if (2 * j == N2) {
      const double a = p[nrow * j], b = p[nrow * (nlon - j)];
      p[nrow * j] = a + b;
      p[nrow * (nlon - j)] = a - b;
    } else {
      double &a = p[nrow * j], &b = p[nrow * (nlon - j)], &c = p[nrow * (N2 - j)], &d = p[nrow * (N2 + j)];
      const double ab = a + b, cd = c + d, am = a - b, dc = d - c;
      a = ab + cd;
      c = ab - cd;
      d = am + dc;
      b = am - dc;
    }
  }
}

// C_m(i) = sum_j g cos(m phi_j), S_m(i) likewise, times wf_i, from the folded
// columns; C, S [m][i]
__device__ __forceinline__ void fold_analysis(int L, int nrow, int nlon, const double* g, const Fold4* __restrict__ tab,
                                              const double* __restrict__ wf, double* C, double* S) {
  const int N2 = nlon / 2, nq = nlon / 4 + 1, q1 = (N2 - 1) / 2;  // q1: the last j of four distinct columns
  for (int t = threadIdx.x; t < L * nrow; t += blockDim.x) {
    const int m = t / nrow, i = t - m * nrow, odd = m & 1;
    const double* gc = g + i + (odd ? nrow * N2 : 0);
    const double* gs = g + i + nrow * (odd ? nlon : N2);
    const int dc = odd ? -nrow : nrow;
    const Fold4* q = tab + (size_t)m * nq;
    double c = gc[0], s = 0;
    for (int j = 1; j <= q1; ++j) {
      const double2 w = *reinterpret_cast<const double2*>(q + j);
      c = fma(gc[j * dc], w.x, c);
      s = fma(gs[j * dc], w.y, s);
    }
    if (nq - 1 > q1) {  // j = nlon / 4
      const double2 w = *reinterpret_cast<const double2*>(q + nq - 1);
      if (odd) s = fma(gs[(nq - 1) * dc], w.y, s);
      else c = fma(gc[(nq - 1) * dc], w.x, c);
    }
    C[t] = c * wf[i];
    S[t] = s * wf[i];
  }
}

// a(m, n), b(m, n) (n >= m) of C, S; A, B [m][n], n < m untouched; P [i][m][n]
__device__ __forceinline__ void legendre_analysis(int L, int nrow, const double* __restrict__ P, const double* C,
                                                  const double* S, double* A, double* B) {
  // rows m and L - 1 - m together hold L + 1 entries
  for (int t = threadIdx.x; t < L * (L + 1) / 2; t += blockDim.x) {
    const int k = t / (L + 1), r = t - k * (L + 1);
    const int m = r < L - k ? k : L - 1 - k, n = m + (r < L - k ? r : r - (L - k));
    double sa = 0, sb = 0;
    for (int i = 0; i < nrow; ++i) {
      const double p = P[((size_t)i * L + m) * L + n];
      sa = fma(p, C[m * nrow + i], sa);
      sb = fma(-p, S[m * nrow + i], sb);
    }
    A[m * L + n] = sa;
    B[m * L + n] = m > 0 ? sb : 0.0;
  }
}

// G_m(r) = sum_n p a, H_m(r) = sum_n p b, Gd, Hd with dp, [m][r]; m = 0 halved
__device__ __forceinline__ void legendre_synthesis(int L, int nrow, const double* __restrict__ P,
                                                   const double* __restrict__ DP, const double* A, const double* B,
                                                   double* G, double* H, double* Gd, double* Hd) {
  for (int t = threadIdx.x; t < L * nrow; t += blockDim.x) {
    const int m = t / nrow, r = t - m * nrow;
    const size_t row = ((size_t)r * L + m) * L;
    double gs = 0, hs = 0, gd = 0, hd = 0;
    for (int n = m; n < L; ++n) {
      const double p = P[row + n], dp = DP[row + n], a = A[m * L + n], b = B[m * L + n];
      gs = fma(p, a, gs);
      hs = fma(p, b, hs);
      gd = fma(dp, a, gd);
      hd = fma(dp, b, hd);
    }
    const double h = m == 0 ? 0.5 : 1.0;
    G[t] = h * gs; H[t] = h * hs; Gd[t] = h * gd; Hd[t] = h * hd;
  }
}

// Even and odd sums of one row and column pair, and the four columns' values in
// the order j, nlon - j, nlon/2 - j, nlon/2 + j: of sum g cos - h sin, and of
// its phi derivative -sum m (g sin + h cos) from the sums over m g sin, m h cos.
struct FoldSum {
  double c[2] = {0, 0}, s[2] = {0, 0};  // terms with cos, with sin, [m odd]
  __device__ __forceinline__ void value(double* v) const {
    const double p = c[0] + c[1], m = c[0] - c[1], q = s[0] + s[1], n = s[0] - s[1];
    v[0] = p - q; v[1] = p + q; v[2] = m + n; v[3] = m - n;
  }
  __device__ __forceinline__ void dphi(double* v) const {
    const double p = c[0] + c[1], m = c[0] - c[1], q = s[0] + s[1], n = s[0] - s[1];
    v[0] = -(q + p); v[1] = q - p; v[2] = n - m; v[3] = -(n + m);
  }
};

}  // namespace
