"""Scratch of the sorted move tables: bounded by the rows they serve.  The rule
itself on the CPU; on the GPU, ten protons alone in 30 states of one parity
(30e6 configurations, of which the basis has the M = 0 ones), whose tables
for every configuration would take more than the device's memory.  The matrix
is checked for the number of rows, ascending columns, a diagonal equal to the
sum of its terms (1e-12 relative) and x . H y = y . H x (1e-12 of the norms)."""
import os
import subprocess

import numpy as np
import pytest

import cosmo_gb300 as cg

SRC = os.path.join(os.path.dirname(cg.__file__), "csrc")
MAIN = r"""
#include "rowtab.h"
int main() {
  using cg::row_tables_worth;
  const uint64_t gib = 1ull << 30;
  bool ok = row_tables_worth(gib, 0) && !row_tables_worth(gib + 1, 0) && row_tables_worth(gib + 8, 1);
  ok = ok && !row_tables_worth(32 * 700000000ull, 700000000ull);  // one species: no list is shared
  ok = ok && row_tables_worth(32 * 700000000ull, 4 * 700000000ull);
  return ok ? 0 : 1;
}
"""


def test_rule(tmp_path):
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = str(tmp_path / "m")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", SRC, "-I", os.path.join(SRC, "..", "..", "include"),
                    "-I", "/usr/local/cuda/include", str(tmp_path / "m.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


@pytest.mark.gpu
def test_one_species_of_many_states(gpu_available):
    one = [(o, 2 * o + 2, j2, m2) for o, j2 in enumerate((13, 9, 5)) for m2 in range(-j2, j2 + 1, 2)]
    sps = np.array([(o, 0, l, j2, m2, 1, t, 0) for t in (1, -1) for o, l, j2, m2 in one], dtype=np.int32)
    rng = np.random.default_rng(9)
    k1 = np.array([(i, i) for i in range(60)], dtype=np.int32)
    v1 = rng.uniform(-4, 0, 60)
    pairs = [(a, b) for a in range(30, 60) for b in range(a + 1, 60)]
    by_m = {}
    for a, b in pairs:
        by_m.setdefault(sps[a, 4] + sps[b, 4], []).append((a, b))
    k2 = np.array([p + q for l in by_m.values() for i, p in enumerate(l) for q in l[i:]], dtype=np.int32)
    v2 = rng.standard_normal(len(k2))
    p = cg.Problem.from_terms(sps, 30, 0, 10, 0, 0, k1, v1, k2, v2)
    b = cg.ManyBodyStates(p)
    ways = np.zeros((11, 400))  # particles, 2m + 200
    ways[0, 200] = 1
    for _, _, _, m2 in one:
        ways[1:] += np.roll(ways[:-1], m2, axis=1)
    assert b.n == int(ways[10, 200])
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP64)
    rp, c, v = h.upper_rows(0, 64)
    rows = np.repeat(np.arange(64), np.diff(rp).astype(np.int64))
    assert np.all(np.diff(c.astype(np.int64))[np.diff(rows) == 0] > 0)
    pair = {tuple(k): x for k, x in zip(k2.tolist(), v2)}
    diag = np.array([sum(v1[i] for i in z) + sum(pair[(i, j, i, j)] for a, i in enumerate(z) for j in z[a + 1:])
                     for z in b.states(0, 64).tolist()])
    np.testing.assert_allclose(h.diagonal()[:64], diag, rtol=1e-12)
    np.testing.assert_allclose(v[c == rows], diag, rtol=1e-12)
    x = rng.standard_normal((b.n, 2))
    y = h.times_matrix(x)
    assert abs(x[:, 0] @ y[:, 1] - x[:, 1] @ y[:, 0]) <= 1e-12 * np.linalg.norm(x[:, 0]) * np.linalg.norm(y[:, 1])
