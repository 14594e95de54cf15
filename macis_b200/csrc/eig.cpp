// Lowest eigenpairs of a small symmetric matrix on the host: the syev step of
// lobpcgxx::rayleigh_ritz (src/lobpcgxx/include/lobpcgxx/rayleigh_ritz.hpp:
// 70-77). Davidson waits for it in every iteration, so the O(k^3) loops use
// four-wide vectors, with AVX2 code where the processor has it (k = 40, lowest
// pair: 87 us as plain scalar loops with one Sturm point at a time).
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <vector>

// the four-wide helpers are always inlined: no call passes such a vector
#pragma GCC diagnostic ignored "-Wpsabi"

namespace mb {
namespace {

typedef double v4 __attribute__((vector_size(32)));
inline __attribute__((always_inline)) v4 ld(const double* p) {
  v4 x;
  std::memcpy(&x, p, sizeof x);
  return x;
}
inline __attribute__((always_inline)) void st(double* p, v4 x) {
  std::memcpy(p, &x, sizeof x);
}

// Householder reduction of the symmetric a (lower triangle, column-major, ld
// k) to tridiagonal form: A <- H A H with H = I - 2 v v^T acting on rows and
// columns j+1.. The vectors v go to the columns of refl (zero: no reflection).
inline __attribute__((always_inline)) void tridiagonalise(int k, double* a,
                                                          double* refl,
                                                          double* p) {
  for(int j = 0; j + 2 < k; ++j) {
    double* v = refl + size_t(j) * k;
    const double* aj = a + size_t(j) * k;
    double nrm = 0;
    for(int i = j + 1; i < k; ++i) nrm += aj[i] * aj[i];
    nrm = std::sqrt(nrm);
    if(nrm == 0) continue;
    const double x0 = aj[j + 1];
    const double alpha = x0 > 0 ? -nrm : nrm;
    v[j + 1] = x0 - alpha;
    for(int i = j + 2; i < k; ++i) v[i] = aj[i];
    double vn = 0;
    for(int i = j + 1; i < k; ++i) vn += v[i] * v[i];
    vn = std::sqrt(vn);
    if(vn == 0) {
      std::fill(v, v + k, 0.0);
      continue;
    }
    for(int i = j + 1; i < k; ++i) v[i] /= vn;
    // p = A v ; K = v.p ; q = p - K v ; A <- A - 2 v q^T - 2 q v^T
    for(int r = j; r < k; ++r) p[r] = 0;
    for(int c = j; c < k; ++c) {  // column c below the diagonal, both ways
      const double* ac = a + size_t(c) * k;
      const double vc = v[c];
      const v4 vcv = {vc, vc, vc, vc};
      v4 s = {0, 0, 0, 0};
      double s0 = ac[c] * vc;
      int r = c + 1;
      for(; r + 3 < k; r += 4) {
        const v4 x = ld(ac + r);
        s += x * ld(v + r);
        st(p + r, ld(p + r) + x * vcv);
      }
      for(; r < k; ++r) {
        s0 += ac[r] * v[r];
        p[r] += ac[r] * vc;
      }
      p[c] += s0 + ((s[0] + s[1]) + (s[2] + s[3]));
    }
    double K = 0;
    for(int r = j + 1; r < k; ++r) K += v[r] * p[r];
    for(int r = j; r < k; ++r) p[r] -= K * v[r];
    for(int c = j; c < k; ++c) {
      double* ac = a + size_t(c) * k;
      const double vc = 2 * v[c], pc = 2 * p[c];
      const v4 vcv = {vc, vc, vc, vc}, pcv = {pc, pc, pc, pc};
      int r = c;
      for(; r + 3 < k; r += 4)
        st(ac + r, ld(ac + r) - (ld(v + r) * pcv + ld(p + r) * vcv));
      for(; r < k; ++r) ac[r] -= v[r] * pc + p[r] * vc;
    }
  }
}

// Sturm counts of eigenvalues below x at eight points: their division chains
// are independent, so eight cost little more than one. Counts come as the
// number of negative pivots.
constexpr int NP = 8;
inline __attribute__((always_inline)) void sturm(int k, const double* d,
                                                 const double* e2,
                                                 const double (&x)[NP],
                                                 int (&c)[NP]) {
  const v4 xa = ld(x), xb = ld(x + 4), zero = {0, 0, 0, 0},
           one = {1, 1, 1, 1}, tiny = {1e-300, 1e-300, 1e-300, 1e-300};
  const v4 d0 = {d[0], d[0], d[0], d[0]};
  v4 qa = d0 - xa, qb = d0 - xb;
  v4 ca = qa < zero ? one : zero, cb = qb < zero ? one : zero;
  for(int i = 1; i < k; ++i) {
    const v4 di = {d[i], d[i], d[i], d[i]};
    const v4 ei = {e2[i - 1], e2[i - 1], e2[i - 1], e2[i - 1]};
    qa = qa == zero ? tiny : qa;
    qb = qb == zero ? tiny : qb;
    qa = di - xa - ei / qa;
    qb = di - xb - ei / qb;
    ca += qa < zero ? one : zero;
    cb += qb < zero ? one : zero;
  }
  for(int t = 0; t < 4; ++t) {
    c[t] = int(ca[t]);
    c[t + 4] = int(cb[t]);
  }
}

inline __attribute__((always_inline)) void syev(int k, const double* lower,
                                                int nwant, double* W,
                                                double* Vec) {
  std::vector<double> a(lower, lower + size_t(k) * k);  // lower triangle used
  const size_t nr = size_t(k) * std::max(k - 2, 0);
  std::vector<double> refl(nr, 0.0), buf(size_t(k) * 8, 0.0);
  double *d = buf.data(), *e = d + k, *e2 = e + k, *p = e2 + k, *z = p + k,
         *w2 = z + k, *f = w2 + k, *rd = f + k;
  tridiagonalise(k, a.data(), refl.data(), p);
  for(int i = 0; i < k; ++i) d[i] = a[i + size_t(i) * k];
  for(int i = 0; i + 1 < k; ++i) {
    e[i] = a[i + 1 + size_t(i) * k];
    e2[i] = e[i] * e[i];
  }
  // Gershgorin bounds
  double lo = d[0], hi = d[0];
  for(int i = 0; i < k; ++i) {
    const double r = (i ? std::fabs(e[i - 1]) : 0) + (i + 1 < k ? std::fabs(e[i]) : 0);
    lo = std::min(lo, d[i] - r);
    hi = std::max(hi, d[i] + r);
  }
  const double span = std::max({hi - lo, std::fabs(lo), std::fabs(hi), 1e-30});
  lo -= 1e-12 * span;
  hi += 1e-12 * span;
  const double tiny = 1e-15 * span;  // pivot floor of the shifted solves
  nwant = std::min(nwant, k);
  std::vector<double> ztri(size_t(k) * nwant);  // of the tridiagonal matrix
  for(int m = 0; m < nwant; ++m) {
    double l = lo, h = hi;  // the m-th eigenvalue: count below x > m
    for(int it = 0; it < 200 && h - l > 4e-16 * std::max(std::fabs(l), std::fabs(h)) + 1e-300; ++it) {
      double x[NP];
      int c[NP];
      for(int t = 0; t < NP; ++t) x[t] = l + (h - l) * ((t + 1) / double(NP + 1));
      sturm(k, d, e2, x, c);
      double nl = l, nh = h;
      for(int t = NP - 1; t >= 0; --t)
        if(c[t] > m) nh = x[t];
      for(int t = 0; t < NP; ++t)
        if(c[t] <= m && x[t] < nh) nl = x[t];
      if(nl == l && nh == h) break;  // the last ulps (or not a number)
      l = nl;
      h = nh;
    }
    W[m] = 0.5 * (l + h);
    // inverse iteration on T - lambda I (tridiagonal LU with pivoting-free
    // elimination, shifted slightly to stay regular)
    const double lam = W[m] + 1e-14 * span;
    auto floor_piv = [&](double x) {
      return std::fabs(x) < tiny ? (x < 0 ? -tiny : tiny) : x;
    };
    rd[0] = 1.0 / floor_piv(d[0] - lam);
    for(int i = 1; i < k; ++i) {
      f[i] = e[i - 1] * rd[i - 1];
      rd[i] = 1.0 / floor_piv(d[i] - lam - f[i] * e[i - 1]);
    }
    // start vector: deterministic, different per wanted pair
    for(int i = 0; i < k; ++i)
      z[i] = 1.0 + 0.5 * std::sin(0.7 * (i + 1) * (m + 1) + 0.3 * m);
    for(int it = 0; it < 5; ++it) {
      w2[0] = z[0];
      for(int i = 1; i < k; ++i) w2[i] = z[i] - f[i] * w2[i - 1];
      w2[k - 1] *= rd[k - 1];
      for(int i = k - 2; i >= 0; --i) w2[i] = (w2[i] - e[i] * w2[i + 1]) * rd[i];
      // keep it orthogonal to the vectors of (nearly) equal eigenvalues
      for(int q = 0; q < m; ++q) {
        if(std::fabs(W[q] - W[m]) > 1e-7 * span) continue;
        const double* zq = ztri.data() + size_t(q) * k;
        double s2 = 0;
        for(int i = 0; i < k; ++i) s2 += zq[i] * w2[i];
        for(int i = 0; i < k; ++i) w2[i] -= s2 * zq[i];
      }
      double nn = 0;
      for(int i = 0; i < k; ++i) nn += w2[i] * w2[i];
      nn = std::sqrt(nn);
      if(!(nn > 0) || !std::isfinite(nn)) break;
      for(int i = 0; i < k; ++i) z[i] = w2[i] / nn;
    }
    std::copy(z, z + k, ztri.begin() + size_t(m) * k);
    // back-transform: y = H_0 H_1 ... H_{k-3} z
    for(int r = k - 3; r >= 0; --r) {
      const double* v = refl.data() + size_t(r) * k;
      double s2 = 0;
      for(int i = r + 1; i < k; ++i) s2 += v[i] * z[i];
      for(int i = r + 1; i < k; ++i) z[i] -= 2 * s2 * v[i];
    }
    double nn = 0;
    for(int i = 0; i < k; ++i) nn += z[i] * z[i];
    nn = std::sqrt(nn);
    for(int i = 0; i < k; ++i) Vec[i + size_t(m) * k] = z[i] / nn;
  }
}

#if defined(__x86_64__)
__attribute__((target("avx2,fma"))) void syev_avx2(int k, const double* lower,
                                                   int nwant, double* W,
                                                   double* Vec) {
  syev(k, lower, nwant, W, Vec);
}
#endif

}  // namespace

// Lowest nwant eigenpairs of the k x k symmetric matrix given by its lower
// triangle (column-major, ld k) as dsyev with Uplo::Lower reads it. Householder
// reduction to tridiagonal form, sections by Sturm counts for each wanted
// eigenvalue, inverse iteration on the tridiagonal matrix, back-transformation
// and Gram-Schmidt among nearly equal ones. W ascending; Vec columns.
void small_syev_lowest(int k, const double* lower, int nwant, double* W,
                       double* Vec) {
#if defined(__x86_64__)
  if(__builtin_cpu_supports("avx2") && __builtin_cpu_supports("fma"))
    return syev_avx2(k, lower, nwant, W, Vec);
#endif
  syev(k, lower, nwant, W, Vec);
}

}  // namespace mb
