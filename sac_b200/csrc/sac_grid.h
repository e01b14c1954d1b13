// sac_grid.h -- gridsetup1 (src/vacgrid.t:556-661) on the host: extrapolate the
// coordinates into the ghost layers and one layer beyond, then
// dx = (x(+1) - x(-1))/2 over the whole grid.  Shared by the single-grid and the
// batched contexts so that both see the same cell widths as the reference.
#pragma once
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace sacgpu {

// g: n, lo, hi, st, ncell, ndim set.  x: ndim blocks of g.ncell (mesh part read;
// the ghost part too when fullgridini).  Outputs the full-grid x and dx.
inline void gridsetup1(const int n[3], const int lo[3], const int hi[3], int ndim, long ncell, const double* x,
                       bool fullgridini, std::vector<double>& hx, std::vector<double>& hdx) {
  const long st1 = n[0], st2 = (long)n[0] * n[1];
  int qn[3], qo[3];
  for (int d = 0; d < 3; ++d) {
    qn[d] = (d < ndim) ? n[d] + 2 : 1;
    qo[d] = (d < ndim) ? 1 : 0;
  }
  const long qc = (long)qn[0] * qn[1] * qn[2];
  std::vector<double> qx((size_t)ndim * qc, 0.0);
  auto qid = [&](int i, int j, int k) { return (i + qo[0]) + (long)qn[0] * ((j + qo[1]) + (long)qn[1] * (k + qo[2])); };
  auto gid = [&](int i, int j, int k) { return i + st1 * j + st2 * k; };
  for (int jd = 0; jd < ndim; ++jd)
    for (int k = 0; k < n[2]; ++k)
      for (int j = 0; j < n[1]; ++j)
        for (int i = 0; i < n[0]; ++i) qx[jd * qc + qid(i, j, k)] = x[jd * ncell + gid(i, j, k)];
  for (int d = 0; d < ndim; ++d) {
    int lo3[3], hi3[3];
    for (int e = 0; e < 3; ++e) {
      lo3[e] = (e < ndim) ? -1 : 0;
      hi3[e] = (e < ndim) ? n[e] : 0;
    }
    for (int side = 0; side < 2; ++side) {
      int a, b, ixe, ixf;
      if (side == 0) {  // upper layers first
        b = n[d];
        a = fullgridini ? n[d] : hi[d] + 1;
        ixe = a - 1;
        ixf = ixe - 1;
      } else {
        a = -1;
        b = fullgridini ? -1 : lo[d] - 1;
        ixe = b + 1;
        ixf = ixe + 1;
      }
      for (int jd = 0; jd < ndim; ++jd)
        for (int q = a; q <= b; ++q) {
          int l2[3] = {lo3[0], lo3[1], lo3[2]}, h2[3] = {hi3[0], hi3[1], hi3[2]};
          l2[d] = h2[d] = q;
          for (int k = l2[2]; k <= h2[2]; ++k)
            for (int j = l2[1]; j <= h2[1]; ++j)
              for (int i = l2[0]; i <= h2[0]; ++i) {
                int ie[3] = {i, j, k}, iff[3] = {i, j, k};
                ie[d] = ixe;
                iff[d] = ixf;
                const int m = std::abs(ixe - q);
                qx[jd * qc + qid(i, j, k)] = (double)(1 + m) * qx[jd * qc + qid(ie[0], ie[1], ie[2])] -
                                             (double)m * qx[jd * qc + qid(iff[0], iff[1], iff[2])];
              }
        }
    }
  }
  hx.assign((size_t)ndim * ncell, 0.0);
  hdx.assign((size_t)ndim * ncell, 0.0);
  for (int jd = 0; jd < ndim; ++jd)
    for (int k = 0; k < n[2]; ++k)
      for (int j = 0; j < n[1]; ++j)
        for (int i = 0; i < n[0]; ++i) hx[jd * ncell + gid(i, j, k)] = qx[jd * qc + qid(i, j, k)];
  for (int d = 0; d < ndim; ++d)
    for (int k = 0; k < n[2]; ++k)
      for (int j = 0; j < n[1]; ++j)
        for (int i = 0; i < n[0]; ++i) {
          int p[3] = {i, j, k}, m[3] = {i, j, k};
          p[d] += 1;
          m[d] -= 1;
          hdx[d * ncell + gid(i, j, k)] = 0.5 * (qx[d * qc + qid(p[0], p[1], p[2])] - qx[d * qc + qid(m[0], m[1], m[2])]);
        }
}

// The rows of dimension d's table of widths: row 0 over the mesh, then one for each
// ghost layer next to the mesh across d (getcurrent reads the widths there, and
// gridsetup1's extrapolation rounds the coordinates along d in them), lower and upper
// of every other dimension in order.  Row r holds the cells with the coordinates
// a..b in the dimensions other than d.
inline void width_row(const int lo[3], const int hi[3], int d, int r, int a[3], int b[3]) {
  for (int e = 0; e < 3; ++e) a[e] = lo[e], b[e] = hi[e];
  if (r > 0) {
    const int k = (r - 1) / 2, e = k < d ? k : k + 1;
    a[e] = b[e] = (r - 1) % 2 ? hi[e] + 1 : lo[e] - 1;
  }
}

// Whether the width of every dimension varies along that dimension alone (bit for
// bit) in each of those rows, so that one entry per index and row holds it.
inline bool widths_on_axes(const int n[3], const int lo[3], const int hi[3], int ndim, long ncell,
                           const double* hdx) {
  const long st[3] = {1, n[0], (long)n[0] * n[1]};
  for (int d = 0; d < ndim; ++d)
    for (int r = 0; r < 2 * ndim - 1; ++r) {
      const double* q = hdx + (size_t)d * ncell;
      int a[3], b[3];
      width_row(lo, hi, d, r, a, b);
      const long first = a[0] + st[1] * a[1] + st[2] * a[2] - st[d] * a[d];  // index 0 along d
      a[d] = 0;
      b[d] = n[d] - 1;
      for (int k = a[2]; k <= b[2]; ++k)
        for (int j = a[1]; j <= b[1]; ++j) {
          const double* row = q + st[1] * j + st[2] * k;
          bool same = true;
          if (d == 0) {
            same = std::memcmp(row, q + first, sizeof(double) * n[0]) == 0;
          } else {
            const double v = q[first + st[d] * (d == 1 ? j : k)];
            for (int i = a[0]; i <= b[0]; ++i) same &= row[i] == v;
          }
          if (!same) return false;
        }
    }
  return true;
}

// (dx, 1/dx) pairs of S of the rows above, appended to out
template <typename S>
inline void append_width_pairs(std::vector<S>& out, const int n[3], const int lo[3], const int hi[3], int ndim,
                               const double* q, int d) {
  const long st[3] = {1, n[0], (long)n[0] * n[1]};
  for (int r = 0; r < 2 * ndim - 1; ++r) {
    int a[3], b[3];
    width_row(lo, hi, d, r, a, b);
    const long first = a[0] + st[1] * a[1] + st[2] * a[2] - st[d] * a[d];
    for (long i = 0; i < n[d]; ++i) {
      const double v = q[first + st[d] * i];
      out.push_back((S)v);
      out.push_back((S)(1.0 / v));
    }
  }
}

// whether the widths (every step-th value) are in the range of the stage's divisions
// through their reciprocals (qdiv, out_of_range)
inline bool widths_in_range(const double* v, long n, int step) {
  bool ok = true;
  for (long i = 0; i < n; i += step) ok &= v[i] >= 0x1p-40 && v[i] <= 0x1p40;
  return ok;
}

// Spatial profiles of the Gaussian velocity drivers on the full grid, two
// blocks of ncell: the stratified workload (user 4: horizontal Gaussian of width
// up[4] about (up[2], up[3]) times a vertical one of width up[6] about x1=up[5])
// and the flux tube (user 5: a Gaussian of width up[3] about x1=up[2] times one
// of width up[5] about x2=up[4]).  The time factor A sin(omega t) is applied in
// the stage update.
inline void gauss_driver_profiles(int user, int ndim, long ncell, const double* hx, const double* up,
                                  double* out) {
  for (long q = 0; q < ncell; ++q) {
    const double x1 = hx[q], x2 = ndim > 1 ? hx[ncell + q] : 0.0, x3 = ndim > 2 ? hx[2 * ncell + q] : 0.0;
    if (user == 4) {
      const double xx = ndim > 1 ? x2 - up[2] : 0.0, yy = ndim > 2 ? x3 - up[3] : 0.0, zz = x1 - up[5];
      out[q] = std::exp(-(xx * xx + yy * yy) / (up[4] * up[4]));
      out[ncell + q] = std::exp(-(zz * zz) / (up[6] * up[6]));
    } else {
      const double zz = x1 - up[2], xx = x2 - up[4];
      out[q] = std::exp(-(zz * zz) / (up[3] * up[3]));
      out[ncell + q] = std::exp(-(xx * xx) / (up[5] * up[5]));
    }
  }
}

}  // namespace sacgpu
