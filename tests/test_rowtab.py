"""Stored rows built from sorted move tables (4,096 rows and more) against the
oracle's rows: one species only, one particle beside several, more than half
filled.  Columns and row lengths equal, values within 1e-12 absolute (FP64
matrix) of the oracle's, FP32 hi + lo within 1e-12."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space,nv,zv,twom", [("fp", 0, 8, 0), ("fp", 8, 0, 0), ("fp", 1, 4, 1), ("fp", 4, 1, 1),
                                              ("sd", 3, 4, 1), ("sd", 9, 8, 3)])
def test_rows_match_oracle(gpu_available, space, nv, zv, twom, tmp_path):
    par = "-" if space == "fp" and (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem(space, nv, zv, twom, par, 0.5, 41))[1])
    b = cg.ManyBodyStates(p)
    assert b.n >= 4096
    k1, v1 = p.one_body()
    k2, v2 = p.two_body()
    rp, c, v = O.build_upper(p.info.n_sps, k1, v1, k2, v2, b.states())
    for prec in (cg.CG_PREC_FP64, cg.CG_PREC_FP32):
        h = cg.Hamiltonian(p, b, prec)
        grp, gc, gv = h.upper_rows()
        assert np.array_equal(grp, rp) and np.array_equal(gc, c)
        assert np.abs(gv - v).max() <= 1e-12
        rows = np.repeat(np.arange(b.n), np.diff(rp).astype(np.int64))
        d = np.zeros(b.n)
        d[rows[c == rows]] = v[c == rows]
        assert np.abs(h.diagonal() - d).max() <= 1e-12
