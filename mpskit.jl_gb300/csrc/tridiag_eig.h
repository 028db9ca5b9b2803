// Eigenvalues of the small projected matrices of the Krylov solvers, with as many rows of the
// eigenvector matrix as the caller looks at: a convergence test needs the last one only.
//
// Householder reflections bring the matrix to tridiagonal form, implicit QR steps with Wilkinson's
// shift make it diagonal (Golub & Van Loan, Matrix Computations, 4th ed., sections 8.3.1 and
// 8.3.4-8.3.5).  A step is written as what it is, rotations G T G' of neighbouring rows and columns,
// with the entries of the rotated 2 x 2 block spelled out.  It runs from the last row to the first,
// the mirror image of the book's: the first components of the eigenvectors, the ones that an
// exponential of a Krylov matrix multiplies with, then take part in the fewest rotations (error of
// exp(-i t T) e_1 at n = 8..30: 4.7e-16, in the other direction 1.1e-15).  4/3 n^3 operations for the
// last row, against some 50 n^3 of Jacobi sweeps.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

namespace gb {

// A row-major n x n, symmetric.  D ascending; Z[(i - i0) * n + j]: component i of eigenvector j, for
// the rows i0..n-1.  The signs of the eigenvectors are arbitrary.  False if an eigenvalue does not
// converge (NaN in A).
inline bool sym_eig_rows(int n, const std::vector<double>& Ain, int i0, std::vector<double>& D,
                         std::vector<double>& Z) {
  const int rows = n - i0;
  std::vector<double> A(Ain), Q((size_t)rows * n, 0.0), v(n), p(n);
  for (int i = 0; i < rows; ++i) Q[(size_t)i * n + i0 + i] = 1.0;

  // column k below the subdiagonal is reflected away by 1 - tau v v', v(k+1) = 1
  for (int k = 0; k + 2 < n; ++k) {
    double below = 0.0;
    for (int i = k + 2; i < n; ++i) below += A[i * n + k] * A[i * n + k];
    if (below == 0.0) continue;
    const double head = A[(k + 1) * n + k], len = std::sqrt(head * head + below);
    // head - len without cancellation
    const double first = head <= 0.0 ? head - len : -below / (head + len);
    const double tau = 2.0 * first * first / (below + first * first);
    v[k + 1] = 1.0;
    for (int i = k + 2; i < n; ++i) v[i] = A[i * n + k] / first;
    double vp = 0.0;
    for (int i = k + 1; i < n; ++i) {
      double sum = 0.0;
      for (int j = k + 1; j < n; ++j) sum += A[i * n + j] * v[j];
      p[i] = tau * sum;
      vp += p[i] * v[i];
    }
    for (int i = k + 1; i < n; ++i) p[i] -= 0.5 * tau * vp * v[i];
    for (int i = k + 1; i < n; ++i)
      for (int j = k + 1; j < n; ++j) A[i * n + j] -= v[i] * p[j] + p[i] * v[j];
    A[(k + 1) * n + k] = len;
    for (int r = 0; r < rows; ++r) {
      double* q = &Q[(size_t)r * n];
      double sum = 0.0;
      for (int i = k + 1; i < n; ++i) sum += q[i] * v[i];
      for (int i = k + 1; i < n; ++i) q[i] -= tau * sum * v[i];
    }
  }

  std::vector<double> d(n), e(std::max(n - 1, 0));  // diagonal, subdiagonal
  for (int i = 0; i < n; ++i) d[i] = A[i * n + i];
  for (int i = 0; i + 1 < n; ++i) e[i] = A[(i + 1) * n + i];
  auto negligible = [&](int i) {
    return std::fabs(e[i]) <= 0x1p-53 * (std::fabs(d[i]) + std::fabs(d[i + 1])) + 1e-300;
  };
  int steps = 0;
  for (int begin = 0; begin + 1 < n;) {
    if (negligible(begin)) {
      ++begin;
      steps = 0;
      continue;
    }
    if (++steps > 60) return false;
    int end = begin + 1;
    while (end + 1 < n && !negligible(end)) ++end;
    // the eigenvalue of the first 2 x 2 block closer to its first entry
    const double half = 0.5 * (d[begin + 1] - d[begin]), off = e[begin];
    const double shift = d[begin] - off * off / (half + std::copysign(std::hypot(half, off), half));
    // the first rotation leaves one entry of the shifted matrix's last column (y, x); the others
    // remove the entry y that the one before put beside the band
    double x = d[end] - shift, y = e[end - 1];
    for (int k = end - 1; k >= begin; --k) {
      const double len = std::hypot(x, y);
      const double c = len == 0.0 ? 1.0 : x / len, s = len == 0.0 ? 0.0 : y / len;
      if (k + 1 < end) e[k + 1] = len;
      const double a = d[k], b = e[k], g = d[k + 1];
      const double move = s * (2.0 * c * b + s * (a - g));  // the trace stays
      d[k] = a - move;
      d[k + 1] = g + move;
      e[k] = c * s * (a - g) + (c - s) * (c + s) * b;
      if (k > begin) {
        x = e[k];
        y = s * e[k - 1];
        e[k - 1] *= c;
      }
      for (int r = 0; r < rows; ++r) {
        double* q = &Q[(size_t)r * n + k];
        const double q0 = q[0], q1 = q[1];
        q[0] = c * q0 - s * q1;
        q[1] = c * q1 + s * q0;
      }
    }
  }

  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  std::sort(order.begin(), order.end(), [&](int i, int j) { return d[i] < d[j]; });
  D.resize(n);
  Z.resize((size_t)rows * n);
  for (int j = 0; j < n; ++j) {
    D[j] = d[order[j]];
    for (int r = 0; r < rows; ++r) Z[(size_t)r * n + j] = Q[(size_t)r * n + order[j]];
  }
  return true;
}

}  // namespace gb
