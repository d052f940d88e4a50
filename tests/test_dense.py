"""The projected problem's eigensolver (csrc/dense.cpp) on the CPU: eigenvalues
against numpy, residuals and overlaps of the vectors, for all vectors and for
the lowest few (inverse iteration), on random, degenerate, decoupled and
graded matrices.  Tolerances: 1e-13 n of the largest element sum for
eigenvalues and residuals, 1e-12 for overlaps (both at rounding level)."""
import os
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cosmo_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include "dense.h"
int main(int argc, char** argv) {
  int n = 0, need = 0;
  FILE* f = std::fopen(argv[1], "rb");
  if (!f || std::fread(&n, 4, 1, f) != 1 || std::fread(&need, 4, 1, f) != 1) return 1;
  std::vector<double> a(size_t(n) * n), w, z;
  if (std::fread(a.data(), 8, a.size(), f) != a.size()) return 1;
  std::fclose(f);
  cg::sym_eig(n, a, w, z, need);
  f = std::fopen(argv[2], "wb");
  std::fwrite(w.data(), 8, w.size(), f);
  std::fwrite(z.data(), 8, z.size(), f);
  std::fclose(f);
}
"""


@pytest.fixture(scope="module")
def solver(tmp_path_factory):
    d = tmp_path_factory.mktemp("dense")
    (d / "m.cpp").write_text(MAIN)
    exe = str(d / "m")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O3", "-I", SRC, str(d / "m.cpp"),
                    os.path.join(SRC, "dense.cpp"), "-o", exe], check=True)

    def run(a, need):
        n = len(a)
        with open(d / "in", "wb") as f:
            f.write(np.array([n, need], np.int32).tobytes() + np.ascontiguousarray(a).tobytes())
        subprocess.run([exe, str(d / "in"), str(d / "out")], check=True)
        v = np.fromfile(d / "out")
        return v[:n], v[n:].reshape(n, n)
    return run


def _matrix(kind, n):
    r = np.random.default_rng(n)
    a = r.standard_normal((n, n))
    a = a + a.T
    if kind == "degenerate":
        q = np.linalg.qr(a)[0]
        a = (q * (np.arange(n) % 5)) @ q.T
        a = (a + a.T) / 2
    elif kind == "decoupled":
        a[:n // 2, n // 2:] = a[n // 2:, :n // 2] = 0
        a[n // 2:2 * (n // 2), n // 2:2 * (n // 2)] = a[:n // 2, :n // 2]
    elif kind == "restart":  # Ritz values on the diagonal, a border of new rows
        k = max(1, n - 8)
        a[:k, :k] = np.diag(np.sort(r.uniform(-50, -20, k)))
        a *= np.where(np.eye(n) > 0, 1.0, 1e-3)
    elif kind == "graded":
        s = 10.0 ** -np.linspace(0, 12, n)
        a = a * np.sqrt(s[:, None] * s[None])
    elif kind == "diagonal":
        a = np.diag(np.arange(n) % 3 * 1.0)
    return a


@pytest.mark.parametrize("kind", ["random", "degenerate", "decoupled", "restart", "graded", "diagonal"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 33, 96, 128])
def test_sym_eig(solver, kind, n):
    a = _matrix(kind, n)
    ref = np.linalg.eigvalsh(a)
    norm = max(np.abs(a).sum(1).max(), 1e-300)
    for need in (-1, min(10, n), min(32, n)):
        w, z = solver(a, need)
        k = n if need < 0 else need
        assert np.abs(w - ref).max() <= 1e-13 * n * norm
        v = z[:, :k]
        assert np.abs(a @ v - v * w[:k]).max() <= 1e-13 * n * norm
        assert np.abs(v.T @ v - np.eye(k)).max() <= 1e-12
