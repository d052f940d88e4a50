"""Infinities and NaN in x of the factored FP32 product: as in an element-wise
product they reach, in their own vector, the rows whose matrix element is not
zero, and no others (as infinity or NaN: the terms of an element may differ in
sign).  The rows are those of the stored FP64 matrix; the others
are held against its product without the entry, within 1e-5 of max |y| as the
other FP32 products.  One and several output tiles, both kinds of pairs."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space,nv,zv,twom", [("sd", 3, 3, 0), ("sd", 1, 4, 1), ("fp", 1, 1, 0), ("fp", 3, 2, 1),
                                              ("fp", 3, 3, 0)])
def test_rows_reached(gpu_available, space, nv, zv, twom, tmp_path):
    par = "-" if space == "fp" and (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem(space, nv, zv, twom, par, 0.5, 31))[1])
    b = cg.ManyBodyStates(p)
    hs = cg.Hamiltonian(p, b, cg.CG_PREC_FP64)
    hv = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=True)
    rng = np.random.default_rng(17)
    x = rng.standard_normal((b.n, 8))
    at = rng.integers(0, b.n, 8)
    bad = [np.inf, -np.inf, np.nan, None, np.inf, np.nan, None, -np.inf]
    clean, unit = x.copy(), np.zeros((b.n, 8))
    for k, v in enumerate(bad):
        if v is not None:
            x[at[k], k], clean[at[k], k], unit[at[k], k] = v, 0.0, 1.0
    reached = hs.times_matrix(unit) != 0
    ref = hs.times_matrix(clean)
    y = hv.times_matrix(x, cg.CG_PREC_FP32)
    assert np.array_equal(np.isfinite(y), ~reached)
    ok = ~reached
    np.testing.assert_allclose(y[ok], ref[ok], rtol=0, atol=1e-5 * np.abs(ref).max())
