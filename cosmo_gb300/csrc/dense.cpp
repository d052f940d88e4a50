#include "dense.h"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace cg {

namespace {
// y += sum of four rows times their factors, then the rest one by one
inline void axpy_rows(int m, int rows, const double* f, const double* a, size_t lda, double* __restrict__ y) {
  int k = 0;
  for (; k + 4 <= rows; k += 4) {
    const double f0 = f[k], f1 = f[k + 1], f2 = f[k + 2], f3 = f[k + 3];
    const double *a0 = a + k * lda, *a1 = a0 + lda, *a2 = a1 + lda, *a3 = a2 + lda;
    for (int j = 0; j < m; ++j) y[j] += (f0 * a0[j] + f1 * a1[j]) + (f2 * a2[j] + f3 * a3[j]);
  }
  for (; k < rows; ++k) {
    const double f0 = f[k];
    const double* a0 = a + k * lda;
    for (int j = 0; j < m; ++j) y[j] += f0 * a0[j];
  }
}
// rows (x, y) <- (c x + s y, c y - s x)
inline void turn(int m, double c, double s, double* __restrict__ x, double* __restrict__ y) {
  for (int k = 0; k < m; ++k) {
    const double u = x[k], v = y[k];
    x[k] = c * u + s * v;
    y[k] = c * v - s * u;
  }
}
}  // namespace

namespace {
// Householder reduction to tridiagonal form: z (both triangles, row-major) is
// overwritten, row i keeping its Householder vector in columns 0 .. i - 1 and
// hs[i] half its squared norm (0: no reflection); d the diagonal, e[i] the
// element (i, i + 1).  A u is formed as a sum of rows and both triangles are
// updated, so that every inner loop runs along rows and vectorises.
void tridiagonal(int n, std::vector<double>& z, std::vector<double>& hs, std::vector<double>& d,
                 std::vector<double>& e) {
  const size_t ld = size_t(n);
  std::vector<double> p(n);
  for (int i = n - 1; i > 0; --i) {
    const int m = i;  // length of the vector
    double* zi = &z[i * ld];
    double scale = 0.0;
    if (m > 1)
      for (int k = 0; k < m; ++k) scale += std::fabs(zi[k]);
    if (m == 1 || scale == 0.0) {
      e[i - 1] = zi[m - 1];
      continue;
    }
    double h = 0.0;
    for (int k = 0; k < m; ++k) {
      zi[k] /= scale;
      h += zi[k] * zi[k];
    }
    const double f = zi[m - 1], g = f >= 0.0 ? -std::sqrt(h) : std::sqrt(h);
    e[i - 1] = scale * g;
    h -= f * g;
    zi[m - 1] = f - g;
    std::fill(p.begin(), p.begin() + m, 0.0);
    axpy_rows(m, m, zi, z.data(), ld, p.data());
    double up = 0.0;
    for (int j = 0; j < m; ++j) {
      p[j] /= h;
      up += p[j] * zi[j];
    }
    const double hh = up / (h + h);
    for (int j = 0; j < m; ++j) p[j] -= hh * zi[j];
    for (int j = 0; j < m; ++j) {
      double* zj = &z[j * ld];
      const double uj = zi[j], pj = p[j];
      for (int k = 0; k < m; ++k) zj[k] -= uj * p[k] + pj * zi[k];
    }
    hs[i] = h;
  }
  for (int i = 0; i < n; ++i) d[i] = z[i * ld + i];
  if (n > 0) e[n - 1] = 0.0;
}

// x <- (product of the reflections) x, x a vector of the tridiagonal frame
inline void reflect(int n, const std::vector<double>& z, const std::vector<double>& hs, double* x) {
  const size_t ld = size_t(n);
  for (int i = 0; i < n; ++i) {
    if (hs[i] == 0.0) continue;
    const double* v = &z[i * ld];
    double g0 = 0.0, g1 = 0.0, g2 = 0.0, g3 = 0.0;
    int k = 0;
    for (; k + 4 <= i; k += 4) {
      g0 += v[k] * x[k];
      g1 += v[k + 1] * x[k + 1];
      g2 += v[k + 2] * x[k + 2];
      g3 += v[k + 3] * x[k + 3];
    }
    for (; k < i; ++k) g0 += v[k] * x[k];
    const double g = ((g0 + g1) + (g2 + g3)) / hs[i];
    for (k = 0; k < i; ++k) x[k] -= g * v[k];
  }
}

// Diagonalises the tridiagonal (d, e) in place by implicitly shifted steps
// (Golub & Van Loan, Matrix Computations, section 8.3, upside down: the small
// eigenvalues of a projected problem come to the top and decouple first): the
// shift is the eigenvalue of the leading 2 x 2 block nearer to its first
// element, the first plane rotation is the one that T - shift asks for in the
// last two rows, and every further one chases the element left outside the band
// one row up.  The rotations act on the rows of q (n x n, nullptr: eigenvalues
// only).  d is not sorted.
void shifted_steps(int n, std::vector<double>& d, std::vector<double>& e, double* q) {
  const size_t ld = size_t(n);
  constexpr int kMaxSteps = 60;  // for one eigenvalue; two or three are usual
  const auto decoupled = [&](int i) { return std::fabs(e[i]) <= 1e-16 * (std::fabs(d[i]) + std::fabs(d[i + 1])); };
  int steps = 0;
  for (int first = 0; first + 1 < n;) {
    if (decoupled(first) || ++steps > kMaxSteps) {
      ++first;
      steps = 0;
      continue;
    }
    int last = first + 1;
    while (last + 1 < n && !decoupled(last)) ++last;
    const double half = 0.5 * (d[first + 1] - d[first]), off = e[first];
    const double shift = d[first] - off * (off / (half + std::copysign(std::hypot(half, off), half)));
    double in = d[last] - shift, out = e[last - 1];  // the pair whose second part the rotation removes
    for (int k = last; k > first; --k) {             // rows k and k - 1
      const double len = std::hypot(in, out);
      const double c = len > 0.0 ? in / len : 1.0, s = len > 0.0 ? out / len : 0.0;
      if (k < last) e[k] = len;
      // the 2 x 2 block [u b; b v] turned: u + s t, v - s t and c t - b with t = s (v - u) + 2 c b
      const double b = e[k - 1], t = s * (d[k - 1] - d[k]) + 2.0 * c * b;
      d[k] += s * t;
      d[k - 1] -= s * t;
      e[k - 1] = c * t - b;
      if (q) turn(n, c, s, q + k * ld, q + (k - 1) * ld);
      if (k - 1 > first) {
        in = e[k - 1];
        out = s * e[k - 2];
        e[k - 2] *= c;
      }
    }
  }
}

// Lowest eigenvectors of the tridiagonal (d, e) for the ascending eigenvalues
// w[0 .. need): inverse iteration (LU with row exchanges, Wilkinson &
// Reinsch, tristurm), each vector kept orthogonal to the earlier ones of its
// cluster.  Rows of v.  False when a residual or an overlap is not at rounding
// level; the caller then takes the full transformation.
bool inverse_iteration(int n, const std::vector<double>& d, const std::vector<double>& e,
                       const std::vector<double>& w, int need, std::vector<double>& v) {
  const size_t ld = size_t(n);
  const double eps = 2.2e-16;
  double norm = 0.0;
  for (int i = 0; i < n; ++i)
    norm = std::max(norm, std::fabs(d[i]) + std::fabs(e[i]) + (i ? std::fabs(e[i - 1]) : 0.0));
  if (!(norm > 0.0) || !std::isfinite(norm)) return false;
  std::vector<double> u0(n), u1(n), u2(n), l(n);
  std::vector<char> swap(n);
  v.assign(ld * need, 0.0);
  double last = 0.0;
  for (int s = 0; s < need; ++s) {
    double x = w[s];
    if (s && x - last < 4 * eps * norm) x = last + 4 * eps * norm;
    last = x;
    // U with two superdiagonals, L's multipliers and the exchanges
    double a = d[0] - x, b = n > 1 ? e[0] : 0.0;
    for (int i = 0; i + 1 < n; ++i) {
      const double c = e[i], dn = d[i + 1] - x, en = i + 2 < n ? e[i + 1] : 0.0;
      if (std::fabs(c) > std::fabs(a)) {
        swap[i] = 1;
        u0[i] = c; u1[i] = dn; u2[i] = en;
        l[i] = a / c;
        a = b - l[i] * dn;
        b = -l[i] * en;
      } else {
        swap[i] = 0;
        if (std::fabs(a) < eps * norm) a = eps * norm;
        u0[i] = a; u1[i] = b; u2[i] = 0.0;
        l[i] = c / a;
        a = dn - l[i] * b;
        b = en;
      }
    }
    u0[n - 1] = std::fabs(a) < eps * norm ? eps * norm : a;
    double* vs = &v[s * ld];
    unsigned r = 12345u + 977u * unsigned(s);
    for (int i = 0; i < n; ++i) {
      r = r * 1664525u + 1013904223u;
      vs[i] = 0.5 + double(r >> 8) * (1.0 / 16777216.0);
    }
    for (int it = 0; it < 3; ++it) {
      if (it)
        for (int i = 0; i + 1 < n; ++i) {
          if (swap[i]) std::swap(vs[i], vs[i + 1]);
          vs[i + 1] -= l[i] * vs[i];
        }
      for (int i = n - 1; i >= 0; --i) {
        double t = vs[i];
        if (i + 1 < n) t -= u1[i] * vs[i + 1];
        if (i + 2 < n) t -= u2[i] * vs[i + 2];
        vs[i] = t / u0[i];
      }
      double big = 0.0;
      for (int i = 0; i < n; ++i) big = std::max(big, std::fabs(vs[i]));
      if (!(big > 0.0) || !std::isfinite(big)) return false;
      for (int i = 0; i < n; ++i) vs[i] /= big;
      for (int q = s - 1; q >= 0 && w[s] - w[q] < 1e-3 * norm; --q) {
        double o = 0.0;
        for (int i = 0; i < n; ++i) o += v[q * ld + i] * vs[i];
        for (int i = 0; i < n; ++i) vs[i] -= o * v[q * ld + i];
      }
      double nn = 0.0;
      for (int i = 0; i < n; ++i) nn += vs[i] * vs[i];
      if (!(nn > 0.0)) return false;
      nn = 1.0 / std::sqrt(nn);
      for (int i = 0; i < n; ++i) vs[i] *= nn;
    }
    double res = 0.0;
    for (int i = 0; i < n; ++i) {
      double t = (d[i] - w[s]) * vs[i];
      if (i) t += e[i - 1] * vs[i - 1];
      if (i + 1 < n) t += e[i] * vs[i + 1];
      res = std::max(res, std::fabs(t));
    }
    if (!(res <= 64 * eps * norm)) return false;
    for (int q = 0; q < s; ++q) {
      double o = 0.0;
      for (int i = 0; i < n; ++i) o += v[q * ld + i] * vs[i];
      if (!(std::fabs(o) <= 1e-13)) return false;
    }
  }
  return true;
}
}  // namespace

// Householder reduction (Wilkinson & Reinsch, Handbook for Automatic Computation
// II) and shifted steps, the inner loops along rows.  need < n: only that many
// lowest eigenvectors are formed, by inverse iteration on the tridiagonal matrix
// (the steps then run without vectors); the other columns of zout are zero.  One such problem per Davidson
// iteration (up to 96 x 96): 24 -> 11 ms of a 46 -> 33 ms solve of 62 iterations
// (sd 4+4).
void sym_eig(int n, const std::vector<double>& a, std::vector<double>& w, std::vector<double>& zout, int need) {
  const size_t ld = size_t(n);
  std::vector<double> z(a), hs(n, 0.0), d(n), e(n);
  for (int i = 0; i < n; ++i)  // the lower triangle counts
    for (int j = i + 1; j < n; ++j) z[i * ld + j] = z[j * ld + i];
  tridiagonal(n, z, hs, d, e);
  w.resize(n);
  zout.assign(ld * n, 0.0);
  if (need >= 0 && 2 * need < n && n >= 16) {
    std::vector<double> dq(d), eq(e), v;
    shifted_steps(n, dq, eq, nullptr);
    std::sort(dq.begin(), dq.end());
    if (inverse_iteration(n, d, e, dq, need, v)) {
      w = dq;
      for (int k = 0; k < need; ++k) {
        reflect(n, z, hs, &v[k * ld]);
        for (int i = 0; i < n; ++i) zout[i * ld + k] = v[k * ld + i];
      }
      return;
    }
  }
  // rows of q: the columns of the product of the reflections, then the eigenvectors
  std::vector<double> q(ld * n, 0.0);
  for (int i = 0; i < n; ++i) q[i * ld + i] = 1.0;
  for (int i = 0; i < n; ++i) reflect(n, z, hs, &q[i * ld]);
  shifted_steps(n, d, e, q.data());
  std::vector<int> idx(n);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) { return d[x] < d[y]; });
  for (int k = 0; k < n; ++k) {
    w[k] = d[idx[k]];
    const double* qk = &q[idx[k] * ld];
    for (int i = 0; i < n; ++i) zout[i * ld + k] = qk[i];
  }
}

int cholesky(int n, std::vector<double>& a) {
  for (int j = 0; j < n; ++j) {
    double s = a[size_t(j) * n + j];
    for (int k = 0; k < j; ++k) s -= a[size_t(j) * n + k] * a[size_t(j) * n + k];
    if (!(s > 0.0)) return j;
    double l = std::sqrt(s);
    a[size_t(j) * n + j] = l;
    for (int i = j + 1; i < n; ++i) {
      double t = a[size_t(i) * n + j];
      for (int k = 0; k < j; ++k) t -= a[size_t(i) * n + k] * a[size_t(j) * n + k];
      a[size_t(i) * n + j] = t / l;
    }
  }
  return -1;
}

}  // namespace cg
