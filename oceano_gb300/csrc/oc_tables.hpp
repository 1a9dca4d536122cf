// 1D rules, Lagrange basis and per-degree tables of the GPU operator (host side).
//
// FE_DGQ(p) is the Lagrange basis on the p+1 Gauss-Lobatto points of [0,1]
// (deal.II FE_DGQ, lexicographic).  The operator uses three cell rules
// (OceanDG.h:448-450): QGauss(floor(1.5p)+1) for the L_h cell integrals,
// QGaussLobatto(p+2) for the zeta mass and inner faces, QGauss(p+1) for the
// discharge mass inverse; boundary faces use QGauss(floor(1.5p)+1).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>

#include "oc_layout.h"

namespace oc {

// Gauss-Legendre on [0,1] by Newton on the Legendre recurrence.
inline void gauss_rule(int n, double *x, double *w) {
  for (int i = 0; i < n; ++i) {
    double z = std::cos(M_PI * (i + 0.75) / (n + 0.5));
    double pn = 0, dpn = 1;
    for (int it = 0; it < 100; ++it) {
      double a = 1, b = z;
      for (int k = 2; k <= n; ++k) {
        double c = ((2 * k - 1) * z * b - (k - 1) * a) / k;
        a = b;
        b = c;
      }
      pn = b;
      dpn = n == 1 ? 1.0 : n * (z * b - a) / (z * z - 1);
      double dz = pn / dpn;
      z -= dz;
      if (std::fabs(dz) < 1e-17) break;
    }
    double a = 1, b = z;
    for (int k = 2; k <= n; ++k) {
      double c = ((2 * k - 1) * z * b - (k - 1) * a) / k;
      a = b;
      b = c;
    }
    dpn = n == 1 ? 1.0 : n * (z * b - a) / (z * z - 1);
    x[n - 1 - i] = z;
    w[n - 1 - i] = 2.0 / ((1 - z * z) * dpn * dpn);
  }
  for (int i = 0; i < n / 2; ++i) {
    double s = 0.5 * (x[n - 1 - i] - x[i]), ww = 0.5 * (w[i] + w[n - 1 - i]);
    x[i] = -s; x[n - 1 - i] = s; w[i] = ww; w[n - 1 - i] = ww;
  }
  if (n % 2) x[n / 2] = 0;
  for (int i = 0; i < n; ++i) { x[i] = 0.5 * (x[i] + 1); w[i] *= 0.5; }
}

// Gauss-Lobatto on [0,1]: Newton on (1-x^2)P'_{n-1} from Chebyshev-Lobatto nodes.
inline void lobatto_rule(int n, double *x, double *w) {
  const int m = n - 1;
  double P[16];
  for (int i = 0; i < n; ++i) {
    double z = std::cos(M_PI * i / m);
    for (int it = 0; it < 200; ++it) {
      P[0] = 1; P[1] = z;
      for (int k = 2; k <= m; ++k) P[k] = ((2 * k - 1) * z * P[k - 1] - (k - 1) * P[k - 2]) / k;
      double dz = (z * P[m] - P[m - 1]) / (n * P[m]);
      z -= dz;
      if (std::fabs(dz) < 1e-17) break;
    }
    P[0] = 1; P[1] = z;
    for (int k = 2; k <= m; ++k) P[k] = ((2 * k - 1) * z * P[k - 1] - (k - 1) * P[k - 2]) / k;
    x[m - i] = z;
    w[m - i] = 2.0 / (m * n * P[m] * P[m]);
  }
  x[0] = -1; x[m] = 1;
  for (int i = 0; i < n / 2; ++i) {
    double s = 0.5 * (x[m - i] - x[i]), ww = 0.5 * (w[i] + w[m - i]);
    x[i] = -s; x[m - i] = s; w[i] = ww; w[m - i] = ww;
  }
  if (n % 2) x[n / 2] = 0;
  for (int i = 0; i < n; ++i) { x[i] = 0.5 * (x[i] + 1); w[i] *= 0.5; }
}

inline double lag(int n, const double *xn, int i, double x) {
  double v = 1;
  for (int j = 0; j < n; ++j)
    if (j != i) v *= (x - xn[j]) / (xn[i] - xn[j]);
  return v;
}

inline double lag_d(int n, const double *xn, int i, double x) {
  double s = 0;
  for (int k = 0; k < n; ++k) {
    if (k == i) continue;
    double v = 1 / (xn[i] - xn[k]);
    for (int j = 0; j < n; ++j)
      if (j != i && j != k) v *= (x - xn[j]) / (xn[i] - xn[j]);
    s += v;
  }
  return s;
}

inline bool invert_small(int n, const double *a, double *ai) {
  double m[OC_MAXN][2 * OC_MAXN];
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < 2 * n; ++j) m[i][j] = j < n ? a[i * n + j] : (j - n == i);
  for (int c = 0; c < n; ++c) {
    int p = c;
    for (int r = c + 1; r < n; ++r)
      if (std::fabs(m[r][c]) > std::fabs(m[p][c])) p = r;
    if (m[p][c] == 0) return false;
    for (int j = 0; j < 2 * n; ++j) std::swap(m[c][j], m[p][j]);
    double d = m[c][c];
    for (int j = 0; j < 2 * n; ++j) m[c][j] /= d;
    for (int r = 0; r < n; ++r)
      if (r != c) {
        double f = m[r][c];
        for (int j = 0; j < 2 * n; ++j) m[r][j] -= f * m[c][j];
      }
  }
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) ai[i * n + j] = m[i][n + j];
  return true;
}

// Cyclic Jacobi eigen-decomposition of a small symmetric matrix: a = V diag(e) V^T.
inline void sym_eig(int n, const double *a_in, double *e, double *V) {
  double a[OC_MAXN * OC_MAXN];
  std::memcpy(a, a_in, sizeof(double) * n * n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) V[i * n + j] = i == j;
  for (int sweep = 0; sweep < 100; ++sweep) {
    double off = 0;
    for (int i = 0; i < n; ++i)
      for (int j = i + 1; j < n; ++j) off += a[i * n + j] * a[i * n + j];
    if (off < 1e-34) break;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) {
        if (std::fabs(a[p * n + q]) < 1e-300) continue;
        double th = 0.5 * (a[q * n + q] - a[p * n + p]) / a[p * n + q];
        double t = (th >= 0 ? 1 : -1) / (std::fabs(th) + std::sqrt(th * th + 1));
        double c = 1 / std::sqrt(t * t + 1), s = t * c;
        for (int k = 0; k < n; ++k) {  // columns
          double akp = a[k * n + p], akq = a[k * n + q];
          a[k * n + p] = c * akp - s * akq;
          a[k * n + q] = s * akp + c * akq;
        }
        for (int k = 0; k < n; ++k) {  // rows
          double apk = a[p * n + k], aqk = a[q * n + k];
          a[p * n + k] = c * apk - s * aqk;
          a[q * n + k] = s * apk + c * aqk;
        }
        for (int k = 0; k < n; ++k) {
          double vkp = V[k * n + p], vkq = V[k * n + q];
          V[k * n + p] = c * vkp - s * vkq;
          V[k * n + q] = s * vkp + c * vkq;
        }
      }
  }
  for (int i = 0; i < n; ++i) e[i] = a[i * n + i];
}

// Fill the tables of degree p (FP64; the FP32 copy is a cast).
inline void fill_tables(int p, DegTables<double> &t) {
  std::memset(&t, 0, sizeof(t));
  const int N = p + 1, Q = (3 * p) / 2 + 1, G = p + 2;
  double xN[OC_MAXN], wN[OC_MAXN], xQ[OC_MAXQ], wQ[OC_MAXQ], xG[OC_MAXF], wG[OC_MAXF];
  double xM[OC_MAXN], wM[OC_MAXN];
  lobatto_rule(N, xN, wN);
  gauss_rule(Q, xQ, wQ);
  lobatto_rule(G, xG, wG);
  gauss_rule(N, xM, wM);
  for (int q = 0; q < Q; ++q) {
    t.wQ[q] = wQ[q];
    t.xQ[q] = xQ[q];
    for (int i = 0; i < N; ++i) {
      t.BQ[q][i] = lag(N, xN, i, xQ[q]);
      t.DQ[q][i] = lag_d(N, xN, i, xQ[q]);
    }
  }
  double l1 = 0.;
  for (int q = 0; q < G; ++q) {
    t.wG[q] = wG[q];
    double s = 0.;
    for (int i = 0; i < N; ++i) {
      t.BG[q][i] = lag(N, xN, i, xG[q]);
      s += std::fabs(t.BG[q][i]);
    }
    l1 = s > l1 ? s : l1;
  }
  t.lebG = l1 * l1;  // tensor-product basis: the 2D sum factorises
  double S[OC_MAXN * OC_MAXN], Si[OC_MAXN * OC_MAXN];
  for (int q = 0; q < N; ++q) {
    t.wM[q] = wM[q];
    t.xM[q] = xM[q];
    for (int i = 0; i < N; ++i) {
      S[q * N + i] = lag(N, xN, i, xM[q]);
      t.BM[q][i] = S[q * N + i];
      t.DM[q][i] = lag_d(N, xN, i, xM[q]);
    }
  }
  invert_small(N, S, Si);
  for (int i = 0; i < N; ++i)
    for (int q = 0; q < N; ++q) t.Sinv[i][q] = Si[i * N + q];
  for (int nf = 2; nf <= OC_MAXF; ++nf) {
    double xf[OC_MAXF], wf[OC_MAXF];
    lobatto_rule(nf, xf, wf);
    for (int k = 0; k < nf; ++k) {
      t.wF[nf][k] = wf[k];
      for (int s = 0; s < 3; ++s) {
        const double par = s == 0 ? xf[k] : 0.5 * ((s - 1) + xf[k]);
        for (int i = 0; i < N; ++i) t.F[s][nf][k][i] = lag(N, xN, i, par);
      }
    }
  }
  // Closed form of max_iter sweeps u += ML^-1 (b - M u), u = 0 at first, of the lumped
  // iteration on a fully wet affine cell.  Gauss-Lobatto p+2 integrates the 1D mass M
  // exactly, its row sums are the Gauss-Lobatto p+1 weights l_i, and that rule differs
  // from the exact one on P_p^2 alone: L^-1 M = I - beta v w^T with v_i = P_p(x_i),
  // w_i = l_i v_i / sum_j l_j v_j^2 = p l_i v_i and beta = (p + 1) / (2p + 1).  With the
  // projections E1 = (v w^T) (x) I and E2 = I (x) (v w^T) the update of sweep k >= 1 is
  //   u_k = gamma^k E1 E2 u_0 + beta^k (E1 + E2 - 2 E1 E2) u_0,  gamma = 2 beta - beta^2,
  // and u_0 = b / (l_i l_j det).  Since |(w (x) w) . u_k| = gamma^k |s| for
  // s = (w (x) w) . u_0, the l1 norm of no update before sweep max_iter - 1 falls to the
  // stop rule's 1e-12 where gamma^(max_iter - 2) |s| > 1e-12 max_i w_i^2 (Sweeps::stop).
  const double beta = (p + 1.) / (2. * p + 1.), gamma = 2. * beta - beta * beta;
  for (int i = 0; i < N; ++i) {
    const double x = 2. * xN[i] - 1.;
    double v0 = 1., v1 = x;  // Legendre recurrence up to P_p
    for (int k = 2; k <= p; ++k) {
      const double v2 = ((2. * k - 1.) * x * v1 - (k - 1.) * v0) / k;
      v0 = v1;
      v1 = v2;
    }
    t.zi[i] = 1. / wN[i];
    t.zir[i] = t.zi[i] - (double)(float)t.zi[i];
    t.zv[i] = v1;
    t.zw[i] = p * wN[i] * v1;
  }
  for (int i = 0; i < N; ++i) {
    t.zl[i] = wN[i];
    for (int j = 0; j < N; ++j)
      for (int q = 0; q < N; ++q) t.GD[i][j] += wM[q] * t.DM[q][i] * t.BM[q][j];
  }
  auto lebesgue = [&](const double (*B)[OC_MAXN], int n) {
    double m = 0.;
    for (int q = 0; q < n; ++q) {
      double r = 0.;
      for (int i = 0; i < N; ++i) r += std::fabs(B[q][i]);
      m = std::max(m, r);
    }
    return m * m;
  };
  t.lebQ = lebesgue(t.BQ, Q);
  t.lebQ1 = lebesgue(t.BM, N);
  t.zbeta = beta;
  t.malpha = beta / (1. - beta);  // (I - beta v w^T)^-1 = I + malpha v w^T
  t.zgamma = gamma;
  // The same sweeps with dense 1D factors (the mixed reference-ABI stage):
  //   delta = (W2 (x) W2) diag(g(l_i l_j)) (W1 (x) W1) b / det,
  //   A = L^-1 M (1D), L^-1/2 M L^-1/2 = Qv diag(l) Qv^T, W1 = Qv^T L^-1/2, W2 = L^-1/2 Qv,
  //   g(mu) = sum_{k<K} (1-mu)^k.
  double M1[OC_MAXN * OC_MAXN] = {0}, L1[OC_MAXN] = {0};
  for (int q = 0; q < G; ++q)
    for (int i = 0; i < N; ++i) {
      L1[i] += wG[q] * t.BG[q][i];
      for (int j = 0; j < N; ++j) M1[i * N + j] += wG[q] * t.BG[q][i] * t.BG[q][j];
    }
  double Ms[OC_MAXN * OC_MAXN], ev[OC_MAXN], Qv[OC_MAXN * OC_MAXN];
  for (int i = 0; i < N; ++i) {
    for (int j = 0; j < N; ++j) Ms[i * N + j] = M1[i * N + j] / std::sqrt(L1[i] * L1[j]);
  }
  sym_eig(N, Ms, ev, Qv);
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      t.W1[i][j] = Qv[j * N + i] / std::sqrt(L1[j]);  // (Qv^T L^-1/2)[i][j]
      t.W2[i][j] = Qv[i * N + j] / std::sqrt(L1[i]);  // (L^-1/2 Qv)[i][j]
    }
  for (int i = 0; i < N; ++i) t.zev[i] = ev[i];
}

// What depends on max_iter in the sweeps of degree p (see fill_tables): the sums of their
// closed form, and the weights g(l_i l_j) of the dense one.
inline void fill_sweeps(int p, int max_iter, const DegTables<double> &t, Sweeps<double> &s,
                        double (*gk)[OC_MAXN]) {
  const int N = p + 1;
  double wmax = 0.;
  for (int i = 0; i < N; ++i) wmax = std::max(wmax, std::fabs(t.zw[i]));
  double pb = t.zbeta, pg = t.zgamma;
  s.sb = s.sg = 0.;
  for (int k = 1; k < max_iter; ++k) {
    s.sb += pb;
    s.sg += pg;
    pb *= t.zbeta;
    pg *= t.zgamma;
  }
  s.one = max_iter > 0 ? 1. : 0.;
  s.stop = max_iter < 2 ? -1. : 1.001e-12 * wmax * wmax / std::pow(t.zgamma, max_iter - 2);
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      const double mu = t.zev[i] * t.zev[j];
      double g = 0, pw = 1;
      for (int k = 0; k < max_iter; ++k) { g += pw; pw *= (1 - mu); }
      gk[i][j] = g;
    }
}

// The FP32 shape values at the cell Gauss points for cell_kernel: every entry moved by at most
// one unit, so that the values of a point add to 1 as nearly as they can (then: nearest to the
// FP64 entries), mirrored points mirrored.  Rounded one by one they add to 1 +- 3e-8, the same
// way in every cell and step (mixed against FP64, relative discharge difference of the 80x40
// vortex after 200 steps: degree 2 1.65e-9 -> 1.23e-9, 3 2.0e-9 -> 1.3e-9, 4 1.3e-9 -> 1.2e-9;
// derivatives to 0 as well changed little, and face rows by themselves no longer match the
// masses: 2.7e-10 -> 5.3e-10 on 8x4 cells).
inline void balance_rows(float (*B)[OC_MAXN], const double (*X)[OC_MAXN], int n, int N) {
  int combos = 1;
  for (int i = 0; i < N; ++i) combos *= 3;
  for (int q = 0; 2 * q < n; ++q) {
    float best[OC_MAXN] = {0};
    double best_sum = 1e300, best_err = 1e300;
    for (int c = 0; c < combos; ++c) {
      float t[OC_MAXN];
      double sum = -1., err = 0.;
      bool mirrored = true;
      for (int i = 0, k = c; i < N; ++i, k /= 3)
        t[i] = k % 3 == 0 ? B[q][i] : std::nextafterf(B[q][i], k % 3 == 1 ? 2.f : -2.f);
      for (int i = 0; i < N; ++i) {
        sum += t[i];
        err += (t[i] - X[q][i]) * (t[i] - X[q][i]);
        mirrored = mirrored && t[i] == t[N - 1 - i];
      }
      sum = std::fabs(sum);
      if ((2 * q + 1 == n && !mirrored) || sum > best_sum || (sum == best_sum && err >= best_err))
        continue;
      best_sum = sum;
      best_err = err;
      std::copy(t, t + N, best);
    }
    for (int i = 0; i < N; ++i) B[q][i] = B[n - 1 - q][N - 1 - i] = best[i];
  }
}

inline void balance_tables(int p, const DegTables<double> &d, DegTables<float> &t) {
  balance_rows(t.BQ, d.BQ, (3 * p) / 2 + 1, p + 1);
  balance_rows(t.BM, d.BM, p + 1, p + 1);
}

}  // namespace oc
