"""What FP32 products of up to 8 vectors read: the factored form is reported,
switched off and on again, on on-the-fly and on stored matrices.  Every format
within 1e-5 of max |y| of the FP64 product; the formats' own results come back
bit by bit when they are chosen again."""
import json

import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system
from conftest import problem_for
from test_factored import SYSTEMS
from test_work_area import _full

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


def test_tuning_cache_and_the_factored_form(gpu_available, stored, tmp_path):
    """A cached choice is reused where it settles the matrix and timed again where it does not."""
    h, cache = stored[2], str(tmp_path / "tune.json")

    def edit(**kw):
        with open(cache) as f:
            db = json.load(f)
        (key, entry), = db.items()
        entry.update(kw)
        for k in [k for k, v in kw.items() if v is None]:
            del entry[k]
        with open(cache, "w") as f:
            json.dump({key: entry}, f)

    h.set_format(cg.CG_FORMAT_FACTORED)
    first = h.autotune(8, reps=1, cache=cache)
    assert first["cached"] is False and any(c[1] == -1 for c in first["candidates"])
    h.set_format(cg.CG_FORMAT_FACTORED)
    again = h.autotune(8, reps=1, cache=cache)
    assert again["cached"] is True and again["format"] == first["format"] == h.format_in_use()
    # an entry from before the factored form existed
    for fmt in (cg.CG_FORMAT_ROWS, cg.CG_FORMAT_TILED):
        h.set_format(cg.CG_FORMAT_FACTORED)
        edit(format=fmt, timed=None)
        assert h.autotune(8, reps=1, cache=cache)["cached"] is False
        assert h.autotune(8, reps=1, cache=cache)["cached"] is True
    # an entry whose factored form does not exist for this handle
    small = cg.Hamiltonian(*(lambda p: (p, cg.ManyBodyStates(p)))(problem_for("sd44m0s4", str(tmp_path))), cg.CG_PREC_FP32)
    cache = str(tmp_path / "small.json")
    assert small.autotune(8, reps=1, cache=cache)["cached"] is False
    edit(format=cg.CG_FORMAT_FACTORED)
    r = small.autotune(8, reps=1, cache=cache)
    assert r["cached"] is False and r["format"] == small.format_in_use() == cg.CG_FORMAT_ROWS
    # choices for wide blocks leave the format of narrow ones alone
    h.set_format(cg.CG_FORMAT_FACTORED)
    cache = str(tmp_path / "wide.json")
    for cached in (False, True):
        r = h.autotune(16, reps=1, cache=cache)
        assert r["cached"] is cached and r["format"] == h.format_in_use() == cg.CG_FORMAT_FACTORED


def test_query_on_a_full_device(gpu_available, tmp_path):
    """The block-tiled copy that a query would make (2.5e8 entries) does not fit: the answer is that there is none."""
    p, b = _problem(tmp_path, "fp", 3, 4, 1)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32)
    assert h.format_in_use() == cg.CG_FORMAT_FACTORED
    with _full(256 << 20):
        assert h.format()[:2] == (cg.CG_FORMAT_FACTORED, False)
    assert h.format()[:2] == (cg.CG_FORMAT_FACTORED, True)
