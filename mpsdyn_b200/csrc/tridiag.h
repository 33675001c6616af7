// Lowest eigenpair of a real symmetric tridiagonal matrix (the projected
// Rayleigh-Ritz problem of the Lanczos iteration, kept in FP64 on the host:
// k <= 256, O(k) per step).
//
// Eigenvalue: Newton's iteration from below (solve_from), or bisection on the
// Gershgorin interval with Sturm-sequence counts (the number of negative pivots of the LDL^T factorisation of
// T - x I equals the number of eigenvalues below x; Wilkinson, "The
// Algebraic Eigenvalue Problem", 5.38).  Eigenvector: inverse iteration
// on T - theta I with a row-pivoted tridiagonal elimination.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace mpsgpu {

struct TridiagLowest {
  std::vector<double> d, u, u2, sub, y;
  std::vector<char> swp;

  static int count_below(const std::vector<double>& a, const std::vector<double>& b, int k, double x) {
    int cnt = 0;
    double q = a[0] - x;
    if (q < 0) cnt++;
    for (int i = 1; i < k; i++) {
      const double den = (q == 0.0) ? 1e-300 : q;
      q = a[i] - x - b[i - 1] * b[i - 1] / den;
      if (q < 0) cnt++;
    }
    return cnt;
  }

  // Newton's step for the characteristic polynomial p at x, -p(x)/p'(x), from
  // the pivots q_i of T - x I and their derivatives (p = prod q_i); negative
  // when a pivot is not positive (x is not below every eigenvalue).  From below
  // the lowest eigenvalue Newton's iterates rise to it without passing it, all
  // roots of p being real.
  static double newton_step(const std::vector<double>& a, const std::vector<double>& b, int k, double x) {
    double q = a[0] - x, dq = -1.0, sum = 0.0;
    for (int i = 0;;) {
      if (!(q > 0.0)) return -1.0;
      const double r = 1.0 / q;
      sum += dq * r;
      if (++i == k) break;
      const double t = b[i - 1] * b[i - 1] * r;
      q = a[i] - x - t;
      dq = t * r * dq - 1.0;
    }
    return -1.0 / sum;
  }

  // a: diagonal (k), b: off-diagonal (b[i] couples i and i+1; b[k-1] unused).
  void solve(const std::vector<double>& a, const std::vector<double>& b, int k, double& theta,
             std::vector<double>& s, double& normT) {
    double lo = a[0], hi = a[0];
    for (int i = 0; i < k; i++) {
      const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i < k - 1 ? std::fabs(b[i]) : 0.0);
      lo = std::min(lo, a[i] - r);
      hi = std::max(hi, a[i] + r);
    }
    normT = std::max(std::fabs(lo), std::fabs(hi));
    double l = lo, h = hi;
    for (int it = 0; it < 200; it++) {
      if (!(h - l > 4e-16 * std::max(std::fabs(l), std::fabs(h)) + 1e-300)) break;
      const double mid = 0.5 * (l + h);
      if (mid == l || mid == h) break;
      if (count_below(a, b, k, mid) >= 1) h = mid;
      else l = mid;
    }
    theta = 0.5 * (l + h);
    s.assign(k, 1.0);
    if (k == 1) return;
    invit(a, b, k, theta - 1e-14 * std::max(normT, 1e-300), 1e-15 * std::max(normT, 1e-300), s);
  }

  // As solve(), with the bracket started below an upper bound `ub` of the
  // lowest eigenvalue (the lowest Ritz value of the previous step: by
  // Cauchy interlacing the lowest eigenvalue of T_k is at most that of
  // T_{k-1}) at a guessed distance `step`, widened until the Sturm count
  // shows no eigenvalue below it; Newton from the lower end closes it in a few
  // steps (forty bisections, each a chain of k divisions, took most of this
  // function's time), and bisection settles the last digits.  Falls back to the
  // Gershgorin interval.
  void solve_from(const std::vector<double>& a, const std::vector<double>& b, int k, double ub, double step,
                  double& theta, std::vector<double>& s, double& normT) {
    double lo = a[0], hi = a[0];
    for (int i = 0; i < k; i++) {
      const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i < k - 1 ? std::fabs(b[i]) : 0.0);
      lo = std::min(lo, a[i] - r);
      hi = std::max(hi, a[i] + r);
    }
    normT = std::max(std::fabs(lo), std::fabs(hi));
    double h = std::min(hi, ub + 8e-16 * normT);
    if (!(std::isfinite(h) && count_below(a, b, k, h) >= 1)) h = hi;
    double st = std::max(std::fabs(step), 1e-15 * normT);
    double l = lo;
    for (int it = 0; it < 64; it++) {
      const double cand = h - st;
      if (!(cand > lo)) break;
      if (count_below(a, b, k, cand) == 0) {
        l = cand;
        break;
      }
      h = cand;  // still an upper bound
      st *= 16.0;
    }
    double x = l;
    for (int it = 0; it < 30; it++) {
      const double eps = 2e-16 * std::max(std::fabs(x), std::fabs(h));
      const double dx = newton_step(a, b, k, x);
      if (!(dx >= 0.0)) {  // passed it by rounding (or no pivot was positive at all)
        if (x > l && x < h && count_below(a, b, k, x) >= 1) h = x;
        break;
      }
      l = x;
      if (dx <= 4.0 * eps) {  // at the root: close the bracket around it
        const double cand = l + dx + 8.0 * eps;
        if (cand < h && count_below(a, b, k, cand) >= 1) h = cand;
        break;
      }
      x = l + dx;
      if (!(x < h)) break;
    }
    for (int it = 0; it < 200; it++) {
      if (!(h - l > 4e-16 * std::max(std::fabs(l), std::fabs(h)) + 1e-300)) break;
      const double mid = 0.5 * (l + h);
      if (mid == l || mid == h) break;
      if (count_below(a, b, k, mid) >= 1) h = mid;
      else l = mid;
    }
    theta = 0.5 * (l + h);
    s.assign(k, 1.0);
    if (k == 1) return;
    invit(a, b, k, theta - 1e-14 * std::max(normT, 1e-300), 1e-15 * std::max(normT, 1e-300), s);
  }

  // Three steps of inverse iteration on T - shift I from the start vector s
  // (overwritten by the normalised result); one row-pivoted elimination serves
  // all three (multipliers, row swaps and reciprocal pivots kept).
  void invit(const std::vector<double>& a, const std::vector<double>& b, int k, double shift, double tiny,
             std::vector<double>& s) {
    d.resize(k); u.resize(k); u2.resize(k); sub.resize(k); y.resize(k); swp.resize(k);
    for (int i = 0; i < k; i++) {
      d[i] = a[i] - shift;
      u[i] = (i < k - 1) ? b[i] : 0.0;
      u2[i] = 0.0;
    }
    for (int i = 0; i < k - 1; i++) {
      const double lo = b[i];
      swp[i] = std::fabs(lo) > std::fabs(d[i]);
      if (swp[i]) {
        // row i+1 becomes row i
        const double od = d[i], ou = u[i], ou2 = u2[i];
        d[i] = lo;
        u[i] = d[i + 1];
        u2[i] = (i + 1 < k - 1) ? u[i + 1] : 0.0;
        sub[i] = od / lo;
        d[i + 1] = ou - sub[i] * u[i];
        u[i + 1] = ou2 - sub[i] * u2[i];
      } else {
        sub[i] = lo / ((std::fabs(d[i]) < tiny) ? tiny : d[i]);
        d[i + 1] -= sub[i] * u[i];
        if (i + 1 < k - 1) u[i + 1] -= sub[i] * u2[i];
      }
    }
    for (int i = 0; i < k; i++) d[i] = 1.0 / ((std::fabs(d[i]) < tiny) ? tiny : d[i]);
    for (int rep = 0; rep < 3; rep++) {
      for (int i = 0; i < k; i++) y[i] = s[i];
      for (int i = 0; i < k - 1; i++) {
        if (swp[i]) std::swap(y[i], y[i + 1]);
        y[i + 1] -= sub[i] * y[i];
      }
      for (int i = k - 1; i >= 0; i--) {
        double acc = y[i];
        if (i + 1 < k) acc -= u[i] * y[i + 1];
        if (i + 2 < k) acc -= u2[i] * y[i + 2];
        y[i] = acc * d[i];
      }
      double nrm = 0.0;
      for (int i = 0; i < k; i++) nrm += y[i] * y[i];
      nrm = 1.0 / std::sqrt(nrm);
      for (int i = 0; i < k; i++) s[i] = y[i] * nrm;
    }
  }
};

// i-th smallest eigenvalue (0-based) of the k x k tridiagonal (a, b) by
// bisection on the Sturm counts.
inline double tridiag_eigenvalue(const std::vector<double>& a, const std::vector<double>& b, int k, int i) {
  double lo = a[0], hi = a[0];
  for (int r = 0; r < k; r++) {
    const double rad = (r > 0 ? std::fabs(b[r - 1]) : 0.0) + (r < k - 1 ? std::fabs(b[r]) : 0.0);
    lo = std::min(lo, a[r] - rad);
    hi = std::max(hi, a[r] + rad);
  }
  for (int it = 0; it < 200; it++) {
    if (!(hi - lo > 4e-16 * std::max(std::fabs(lo), std::fabs(hi)) + 1e-300)) break;
    const double mid = 0.5 * (lo + hi);
    if (mid == lo || mid == hi) break;
    if (TridiagLowest::count_below(a, b, k, mid) >= i + 1) hi = mid;
    else lo = mid;
  }
  return 0.5 * (lo + hi);
}

// All eigenvalues of the k x k tridiagonal (a, b), ascending, by implicit-shift
// QL (Dubrulle, Martin & Wilkinson, Numer. Math. 12, 1968; in the form of EISPACK's
// imtql1, which is in the public domain): O(k^2), where a bisection per value takes
// forty chains of k divisions each.  False when an
// off-diagonal element does not vanish within 60 sweeps.
inline bool tridiag_all_values(const std::vector<double>& a, const std::vector<double>& b, int k, double scale,
                               std::vector<double>& d, std::vector<double>& e) {
  d.resize(k);
  e.assign(k, 0.0);
  for (int i = 0; i < k; i++) d[i] = a[i] / scale;  // entries of order one: squares stay in range
  for (int i = 0; i + 1 < k; i++) e[i] = b[i] / scale;
  for (int l = 0; l < k; l++) {
    for (int it = 0;; it++) {
      int m = l;
      while (m + 1 < k && std::fabs(e[m]) > 1.1e-16 * (std::fabs(d[m]) + std::fabs(d[m + 1]))) m++;
      if (m == l) break;
      if (it == 60) return false;
      double g = (d[l + 1] - d[l]) / (2.0 * e[l]), r = std::sqrt(g * g + 1.0);
      g = d[m] - d[l] + e[l] / (g + std::copysign(r, g));
      double s = 1.0, c = 1.0, p = 0.0;
      int i = m - 1;
      for (; i >= l; i--) {  // chase the bulge up
        const double f = s * e[i], h = c * e[i];
        r = std::sqrt(f * f + g * g);
        e[i + 1] = r;
        if (r == 0.0) {  // the matrix splits here
          d[i + 1] -= p;
          e[m] = 0.0;
          break;
        }
        s = f / r;
        c = g / r;
        g = d[i + 1] - p;
        r = (d[i] - g) * s + 2.0 * c * h;
        p = s * r;
        d[i + 1] = g + p;
        g = c * r - h;
      }
      if (i >= l) continue;
      d[l] -= p;
      e[l] = g;
      e[m] = 0.0;
    }
  }
  for (int i = 0; i < k; i++) d[i] *= scale;
  std::sort(d.begin(), d.end());
  return true;
}

// sum_i x_i y_i in four chains
inline double dot4(const double* x, const double* y, int n) {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int i = 0;
  for (; i + 4 <= n; i += 4) {
    s0 += x[i] * y[i];
    s1 += x[i + 1] * y[i + 1];
    s2 += x[i + 2] * y[i + 2];
    s3 += x[i + 3] * y[i + 3];
  }
  for (; i < n; i++) s0 += x[i] * y[i];
  return (s0 + s1) + (s2 + s3);
}

// Thick restart of the Lanczos factorisation H V = V T + f e_m^T (Wu &
// Simon, "Thick-restart Lanczos method for large symmetric eigenvalue
// problems", SIAM J. Matrix Anal. Appl. 22, 2000), kept in tridiagonal form:
//   1. Y (m x keep): orthonormal approximations of the keep lowest Ritz
//      vectors of T (QL values + inverse iteration + modified Gram-Schmidt);
//   2. B = Y^T T Y and the coupling s = |f| Y^T e_m, both exact for this Y;
//   3. Lanczos on the small matrix B from s / |s| with full
//      reorthogonalisation gives Z with Z^T B Z tridiagonal and
//      Z^T s = |s| e_1; the order is reversed so that the last kept vector
//      carries the coupling.
// With G = Y Z (reversed), H (V G) = (V G) T' + (f / |f|) |s| e_r^T plus
// terms in span(V) that the continued reorthogonalised Lanczos absorbs; the
// relation holds for any orthonormal Y, so near-degenerate Ritz values only
// cost filtering quality, never consistency.  (Exact-shift implicit QR,
// the alternative, is not forward stable when converged Ritz values are
// used as shifts: Parlett & Le, SIAM J. Matrix Anal. Appl. 14, 1993.)
struct ThickRestart {
  TridiagLowest tri;
  std::vector<double> Y, TY, B, Z, w, s, v, vals, offd;

  // v -= Y[:, 0..i) Y[:, 0..i)^T v, twice
  void project_out(int m, int i) {
    for (int pass = 0; pass < 2; pass++)
      for (int q = 0; q < i; q++) {
        const double* yq = &Y[(size_t)q * m];
        const double dot = dot4(yq, v.data(), m);
        for (int r = 0; r < m; r++) v[r] -= dot * yq[r];
      }
  }

  double norm2(int m) const {
    double nrm = 0.0;
    for (int r = 0; r < m; r++) nrm += v[r] * v[r];
    return std::sqrt(nrm);
  }

  // a, b: T (m); fnorm = |f|.  Out: r kept vectors, a', b' (b'[r-1] = |s|,
  // the coupling to f / |f|), G (m x r, column-major).  Returns r.
  int compress(std::vector<double>& a, std::vector<double>& b, int m, int keep, double fnorm,
               std::vector<double>& G) {
    double lo = a[0], hi = a[0];
    for (int r = 0; r < m; r++) {
      const double rad = (r > 0 ? std::fabs(b[r - 1]) : 0.0) + (r < m - 1 ? std::fabs(b[r]) : 0.0);
      lo = std::min(lo, a[r] - rad);
      hi = std::max(hi, a[r] + rad);
    }
    const double normT = std::max(std::max(std::fabs(lo), std::fabs(hi)), 1e-300);
    Y.assign((size_t)m * keep, 0.0);
    v.assign(m, 0.0);
    const bool ql = tridiag_all_values(a, b, m, normT, vals, offd);
    double prev = 0.0;
    for (int i = 0; i < keep; i++) {
      double lam = ql ? vals[i] : tridiag_eigenvalue(a, b, m, i);
      // separate repeated values so that inverse iteration can tell them apart
      if (i > 0 && lam - prev < 1e-12 * normT) lam = prev + 1e-12 * normT;
      prev = lam;
      uint64_t z = 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1);
      for (int r = 0; r < m; r++) {  // deterministic, distinct start vectors
        z ^= z >> 31; z *= 0xBF58476D1CE4E5B9ull; z ^= z >> 29;
        v[r] = 1.0 + (double)(z >> 11) * (1.0 / 9007199254740992.0);
      }
      tri.invit(a, b, m, lam - 1e-14 * normT, 1e-15 * normT, v);
      project_out(m, i);
      double nrm = norm2(m);
      for (int e = 0; e < m && !(nrm > 1e-8); e++) {
        // lost to the previous vectors: take a unit vector instead
        for (int r = 0; r < m; r++) v[r] = (r == (e + i) % m) ? 1.0 : 0.0;
        project_out(m, i);
        nrm = norm2(m);
      }
      for (int r = 0; r < m; r++) Y[(size_t)i * m + r] = v[r] / nrm;
    }
    // B = Y^T T Y (symmetrised), s = |f| Y^T e_m
    TY.assign((size_t)m * keep, 0.0);
    for (int i = 0; i < keep; i++) {
      const double* y = &Y[(size_t)i * m];
      double* t = &TY[(size_t)i * m];
      for (int r = 0; r < m; r++) {
        double acc = a[r] * y[r];
        if (r > 0) acc += b[r - 1] * y[r - 1];
        if (r + 1 < m) acc += b[r] * y[r + 1];
        t[r] = acc;
      }
    }
    B.assign((size_t)keep * keep, 0.0);
    for (int i = 0; i < keep; i++)
      for (int j = 0; j < keep; j++) {
        B[(size_t)i * keep + j] = dot4(&Y[(size_t)i * m], &TY[(size_t)j * m], m);
      }
    for (int i = 0; i < keep; i++)
      for (int j = 0; j < i; j++)
        B[(size_t)i * keep + j] = B[(size_t)j * keep + i] = 0.5 * (B[(size_t)i * keep + j] + B[(size_t)j * keep + i]);
    s.assign(keep, 0.0);
    double snorm = 0.0;
    for (int i = 0; i < keep; i++) {
      s[i] = fnorm * Y[(size_t)i * m + (m - 1)];
      snorm += s[i] * s[i];
    }
    snorm = std::sqrt(snorm);
    // Lanczos on B from s / |s| (Z columns z_0 .. z_{r-1})
    std::vector<double> al, be;
    Z.assign((size_t)keep * keep, 0.0);
    int r = 0;
    if (snorm > 0.0) {
      for (int i = 0; i < keep; i++) Z[i] = s[i] / snorm;
      w.assign(keep, 0.0);
      for (r = 1;; r++) {
        const double* zc = &Z[(size_t)(r - 1) * keep];
        for (int i = 0; i < keep; i++) {
          w[i] = dot4(&B[(size_t)i * keep], zc, keep);
        }
        double alpha = 0.0;
        for (int i = 0; i < keep; i++) alpha += zc[i] * w[i];
        al.push_back(alpha);
        if (r == keep) break;
        for (int pass = 0; pass < 2; pass++)
          for (int q = 0; q < r; q++) {
            const double* zq = &Z[(size_t)q * keep];
            const double dot = dot4(zq, w.data(), keep);
            for (int i = 0; i < keep; i++) w[i] -= dot * zq[i];
          }
        double bn = 0.0;
        for (int i = 0; i < keep; i++) bn += w[i] * w[i];
        bn = std::sqrt(bn);
        if (!(bn > 1e-13 * normT)) break;  // the rest of Y is decoupled from f: dropped
        be.push_back(bn);
        for (int i = 0; i < keep; i++) Z[(size_t)r * keep + i] = w[i] / bn;
      }
    } else {
      // f is orthogonal to every kept vector: keep the lowest one alone
      Z[0] = 1.0;
      al.push_back(B[0]);
      r = 1;
    }
    // reversed order: u_p = z_{r-1-p}; G = Y u
    a.assign(r, 0.0);
    b.assign(r, 0.0);
    for (int p = 0; p < r; p++) {
      a[p] = al[r - 1 - p];
      if (p + 1 < r) b[p] = be[r - 2 - p];
    }
    b[r - 1] = snorm;
    G.assign((size_t)m * r, 0.0);
    for (int p = 0; p < r; p++) {
      const double* zc = &Z[(size_t)(r - 1 - p) * keep];
      double* g = &G[(size_t)p * m];
      for (int i = 0; i < keep; i++) {
        const double c = zc[i];
        if (c == 0.0) continue;
        const double* y = &Y[(size_t)i * m];
        for (int q = 0; q < m; q++) g[q] += c * y[q];
      }
    }
    return r;
  }
};

}  // namespace mpsgpu
