"""FP64 operands are split into FP32 pairs from their bits between 2^-70 and
2^127 and by conversions outside: products of vectors of every scale around
those lines, and of numbers half way between two FP32 numbers.  Bound: the
REFINE product's 1e-11 of the largest result, per vector."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

pytestmark = pytest.mark.gpu

EXPS = [0, -66, -69, -70, -71, -72, -80, 60, 100]


@pytest.mark.parametrize("virtual", [False, True])
@pytest.mark.parametrize("m", [4, 8])
def test_scales(gpu_available, virtual, m, tmp_path):
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem("sd", 2, 2, 0, "+", 0.5, 31))[1])
    b = cg.ManyBodyStates(p)
    ref = cg.Hamiltonian(p, b, cg.CG_PREC_FP64)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=virtual)
    rng = np.random.default_rng(5)
    for e in EXPS:
        x = rng.standard_normal((b.n, m))
        x[::7] = 0.0
        x[1::7] = np.round(x[1::7] * 2**23) / 2**23 + 2.0**-25   # half way
        x[2::7] = np.ldexp(1.0, 0) - 2.0**-53                     # rounds up to a power of two
        x[3::7] *= np.ldexp(1.0, rng.integers(-4, 4, (len(x[3::7]), m)))
        y = np.ldexp(ref.times_matrix(x), e)
        z = h.times_matrix(np.ldexp(x, e), cg.CG_PREC_REFINE)
        assert np.max(np.abs(z - y) / np.max(np.abs(y), axis=0)) <= 1e-11


def test_not_finite(gpu_available, tmp_path):
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem("sd", 2, 2, 0, "+", 0.5, 31))[1])
    b = cg.ManyBodyStates(p)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32)
    x = np.random.default_rng(6).standard_normal((b.n, 8))
    x[5, 0], x[6, 1], x[7, 2], x[8, 3] = np.nan, np.inf, -np.inf, 1e300
    y = h.times_matrix(x, cg.CG_PREC_REFINE)
    assert not np.any(np.isfinite(np.diag(y[5:9, :4])))
    assert np.all(np.isfinite(y[:, 4:]))
