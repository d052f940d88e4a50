"""The factored form's work area on on-the-fly matrices (fp 3+4: 21 pairs of
particles x 483,887 rows x 32 bytes): only on handles made for FP32, taken with
the first FP32 product, given back by a solve and by another format, and not in
the way of anything when the device is full.  FP32 products within 1e-5 of max
|y| of FP64; residuals of solves <= 1e-5."""
import contextlib

import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

AREA = (3 * 4 + 3 + 6) * 483887 * 32


@pytest.fixture(scope="module")
def problem(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("fp34"))
    p = cg.Problem(make_system(d, SyntheticSystem("fp", 3, 4, 1, "-", 0.5, 31))[1])
    return p, cg.ManyBodyStates(p)


def _bytes(h):
    h.refresh_info()
    return int(h.info.device_bytes)


def _product(h, x, prec=cg.CG_PREC_FP32):
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    h.spmm_device(x.data_ptr(), 8, y.data_ptr(), 8, 8, prec)
    torch.cuda.synchronize()
    return y


@contextlib.contextmanager
def _full(leave):
    """All of the device's memory but `leave` bytes taken."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _solve(h):
    r = cg.davidson_diagonalization(h, 4, precision=cg.CG_PREC_FP32, tol_resid=1e-5, block=4, lim=24, algorithm=1)
    assert r.stats.converged == 4 and np.all(r.resid <= 1e-5)
    return r.eig


def test_taken_and_given_back(gpu_available, problem):
    b = problem[1]
    assert b.n * 21 * 32 == AREA
    x = torch.randn(b.n, 8, generator=torch.Generator().manual_seed(1)).cuda()
    h64 = cg.Hamiltonian(*problem, cg.CG_PREC_FP64, virtual=True)
    ref = _product(h64, x.double(), cg.CG_PREC_FP64)
    tol = 1e-5 * float(ref.abs().max())
    assert h64.format_in_use() == cg.CG_FORMAT_ROWS
    assert float((_product(h64, x) - ref).abs().max()) <= tol  # FP32 on a handle made for FP64
    h = cg.Hamiltonian(*problem, cg.CG_PREC_FP32, virtual=True)
    bare = _bytes(h)
    assert h.format_in_use() == cg.CG_FORMAT_FACTORED
    _solve(h)
    assert _bytes(h) == bare
    y = _product(h, x)
    assert float((y - ref).abs().max()) <= tol and _bytes(h) == bare + AREA
    _solve(h)
    assert _bytes(h) == bare + AREA
    h.set_format(cg.CG_FORMAT_ROWS)
    assert _bytes(h) == bare
    h.set_format(cg.CG_FORMAT_FACTORED)
    assert torch.equal(_product(h, x), y)


def test_full_device(gpu_available, problem):
    b = problem[1]
    x = torch.randn(b.n, 8, generator=torch.Generator().manual_seed(2)).cuda()
    h = cg.Hamiltonian(*problem, cg.CG_PREC_FP32, virtual=True)
    y = _product(h, x)
    eig = _solve(h)
    h.set_format(cg.CG_FORMAT_ROWS)
    rows = _product(h, x)
    h.set_format(cg.CG_FORMAT_FACTORED)
    h.set_format(cg.CG_FORMAT_ROWS)
    with _full(AREA - (64 << 20)):
        with pytest.raises(cg.CosmoError, match="CG_ERR_NOMEM"):
            h.set_format(cg.CG_FORMAT_FACTORED)
        assert h.format_in_use() == cg.CG_FORMAT_ROWS
    h = cg.Hamiltonian(*problem, cg.CG_PREC_FP32, virtual=True)
    with _full(AREA - (64 << 20)):
        assert torch.equal(_product(h, x), rows)  # the element-wise product serves
        assert h.format_in_use() == cg.CG_FORMAT_ROWS
    h.set_format(cg.CG_FORMAT_FACTORED)
    assert torch.equal(_product(h, x), y)
    # a solve whose FP64 phase needs the room that the area takes
    h = cg.Hamiltonian(*problem, cg.CG_PREC_FP32, virtual=True)
    with _full(AREA + (220 << 20)):
        np.testing.assert_allclose(_solve(h), eig, rtol=0, atol=1e-6)
        assert h.format_in_use() == cg.CG_FORMAT_ROWS


def test_host_buffers_are_counted(gpu_available, tmp_path):
    """Host products keep their device buffers with the handle (FP64, 4 vectors: the block and two operands)."""
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem("sd", 4, 4, 0, "+", 0.5, 31))[1])
    b = cg.ManyBodyStates(p)
    for virtual in (False, True):
        h = cg.Hamiltonian(p, b, cg.CG_PREC_FP64, virtual=virtual)
        bare = _bytes(h)
        h.times_matrix(np.ones((b.n, 4)))
        assert _bytes(h) - bare >= 3 * b.n * 4 * 8


def test_host_product_beside_the_area(gpu_available, problem):
    """An FP64 host product whose buffers fit only in place of the area that FP32 products left."""
    b = problem[1]
    h = cg.Hamiltonian(*problem, cg.CG_PREC_FP32, virtual=True)
    x = np.random.default_rng(4).standard_normal((b.n, 8))
    y32 = h.times_matrix(x, cg.CG_PREC_FP32)
    with _full(16 << 20):  # and the FP32 call's buffers, 62 MB; FP64 takes 93
        y = h.times_matrix(x, cg.CG_PREC_FP64)
        assert h.format_in_use() == cg.CG_FORMAT_ROWS
    assert np.abs(y32 - y).max() <= 1e-5 * np.abs(y).max()
    h.set_format(cg.CG_FORMAT_FACTORED)
    assert np.array_equal(h.times_matrix(x, cg.CG_PREC_FP32), y32)
