"""What FP32 products of up to 8 vectors read: the factored form is reported,
switched off and on again, on on-the-fly and on stored matrices.  Every format
within 1e-5 of max |y| of the FP64 product; the formats' own results come back
bit by bit when they are chosen again."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system
from test_factored import SYSTEMS

pytestmark = pytest.mark.gpu


def _problem(tmp_path, space, nv, zv, twom):
    par = "-" if space == "fp" and (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem(space, nv, zv, twom, par, 0.5, 31))[1])
    return p, cg.ManyBodyStates(p)


@pytest.mark.parametrize("space,nv,zv,twom", SYSTEMS)
def test_on_the_fly_formats(gpu_available, space, nv, zv, twom, tmp_path):
    p, b = _problem(tmp_path, space, nv, zv, twom)
    x = np.random.default_rng(3).standard_normal((b.n, 8))
    ref = cg.Hamiltonian(p, b, cg.CG_PREC_FP64).times_matrix(x)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=True)
    assert h.format_in_use() == cg.CG_FORMAT_FACTORED and h.format()[:2] == (cg.CG_FORMAT_FACTORED, False)
    y = h.times_matrix(x, cg.CG_PREC_FP32)
    h.set_format(cg.CG_FORMAT_ROWS)
    assert h.format_in_use() == cg.CG_FORMAT_ROWS
    z = h.times_matrix(x, cg.CG_PREC_FP32)
    for v in (y, z):
        np.testing.assert_allclose(v, ref, rtol=0, atol=1e-5 * np.abs(ref).max())
    assert b.n < 32 or not np.array_equal(y, z)  # another order of the sums
    with pytest.raises(cg.CosmoError):
        h.set_format(cg.CG_FORMAT_TILED)
    h.set_format(cg.CG_FORMAT_FACTORED)
    assert h.format_in_use() == cg.CG_FORMAT_FACTORED
    assert np.array_equal(h.times_matrix(x, cg.CG_PREC_FP32), y)


@pytest.fixture(scope="module")
def stored(tmp_path_factory):
    """fp 2+4, 2M = 0: 3.3e7 stored entries, factored by default."""
    p, b = _problem(tmp_path_factory.mktemp("fp24"), "fp", 2, 4, 0)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32)
    assert 2 ** 24 <= h.info.nnz_full < 2 ** 26 and h.format_in_use() == cg.CG_FORMAT_FACTORED
    return p, b, h


def test_autotune_of_wide_blocks_keeps_the_format(gpu_available, stored):
    h = stored[2]
    for fmt in (cg.CG_FORMAT_TILED, cg.CG_FORMAT_ROWS, cg.CG_FORMAT_FACTORED):
        h.set_format(fmt)
        r = h.autotune(16, reps=1)
        assert r["format"] == h.format_in_use() == fmt and all(c[1] > 0 for c in r["candidates"])
