"""The small symmetric eigensolver of the Krylov solvers (csrc/tridiag_eig.h), built with the host
compiler, against LAPACK.  A backward stable method: eigenvalues and residuals within a few n eps of
the largest eigenvalue, orthogonal vectors within a few n eps."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mpskit.jl_gb300", "csrc")
EPS = np.finfo(np.float64).eps

PROGRAM = r"""
#include "tridiag_eig.h"
#include <cstdio>
int main() {
  int n, i0;
  while (std::scanf("%d %d", &n, &i0) == 2) {
    std::vector<double> A((size_t)n * n), D, Z;
    for (auto& a : A)
      if (std::scanf("%la", &a) != 1) return 1;
    std::printf("%d", (int)gb::sym_eig_rows(n, A, i0, D, Z));
    for (double v : D) std::printf(" %a", v);
    for (double v : Z) std::printf(" %a", v);
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("eig")
    (d / "eig.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(d / "eig.cpp"), "-o",
                    str(d / "eig")], check=True)
    return str(d / "eig")


def _run(exe, a, i0):
    n = len(a)
    text = f"{n} {i0}\n" + " ".join(float(v).hex() if np.isfinite(v) else str(v)
                                    for v in a.ravel()) + "\n"
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True, timeout=60)
    v = out.stdout.split()
    x = np.array([float.fromhex(t) for t in v[1:]])
    return v[0] == "1", x[:n], x[n:].reshape(n - i0, -1) if len(x) else None


def _matrices():
    rng = np.random.default_rng(0)
    for n in (1, 2, 3, 4, 13, 30, 64):
        a = rng.standard_normal((n, n))
        yield "full", a + a.T
        t = np.diag(rng.standard_normal(n)) + np.diag(rng.uniform(0.1, 1, n - 1), 1)
        yield "tridiagonal", np.triu(t) + np.triu(t, 1).T
        w = np.diag(np.sort(rng.standard_normal(n)))  # after a thick restart
        w[-1, :-1] = w[:-1, -1] = 1e-3 * rng.standard_normal(n - 1)
        yield "arrow", w
        s = 10.0 ** -rng.uniform(0, 12, n)
        yield "graded", (a + a.T) * np.outer(s, s)
        q = np.linalg.qr(a)[0]
        yield "degenerate", q @ np.diag(np.arange(n) // 3 * 1.0) @ q.T
        yield "zero", np.zeros((n, n))
        yield "large", 1e150 * (a + a.T)
    t = np.diag(np.zeros(20)) + np.diag(np.ones(19), 1)  # eigenvalues in pairs of opposite sign
    yield "chain", t + t.T


def test_against_lapack(exe):
    for name, a in _matrices():
        a = 0.5 * (a + a.T)
        n = len(a)
        ok, d, z = _run(exe, a, 0)
        ref = np.linalg.eigvalsh(a)
        top = max(np.abs(ref).max(), 1e-300)
        assert ok, (name, n)
        assert np.all(np.diff(d) >= 0), (name, n)
        assert np.abs(d - ref).max() <= 8 * n * EPS * top, (name, n)
        assert np.linalg.norm(z.T @ z - np.eye(n)) <= 8 * n * EPS, (name, n)
        assert np.linalg.norm((a / top) @ z - z * (d / top)) <= 8 * n * EPS, (name, n)
        ok, dl, zl = _run(exe, a, n - 1)  # the last row alone: the same numbers
        assert ok and np.array_equal(d, dl) and np.array_equal(z[-1:], zl), (name, n)


def test_not_a_number(exe):
    a = np.eye(6)
    a[2, 3] = a[3, 2] = np.nan
    ok, _, _ = _run(exe, a, 5)
    assert not ok
