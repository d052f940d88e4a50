"""On-the-fly products whose result takes the place of their operand (y = x, or
overlapping it by all rows but one): bit-identical to the product into a buffer
of its own, also for operands that are packed already (FP64 4 vectors, FP32 8)
and would be read in place otherwise."""
import pytest

import cosmo_gb300 as cg
from conftest import problem_for

pytestmark = pytest.mark.gpu

CASES = [(cg.CG_PREC_FP64, 4, 4), (cg.CG_PREC_FP64, 3, 4), (cg.CG_PREC_FP64, 8, 8), (cg.CG_PREC_FP32, 8, 8),
         (cg.CG_PREC_FP32, 16, 16), (cg.CG_PREC_REFINE, 4, 4)]


# sd 6+6 keeps the element-wise kernel for FP32, sd 4+4 the factored form
@pytest.mark.parametrize("name", ["sd22m0s1", "sd44m0s4", "sd66m0s5"])
@pytest.mark.parametrize("prec,m,ld", CASES)
def test_on_the_fly_in_place(gpu_available, name, prec, m, ld, tmp_path):
    torch = pytest.importorskip("torch")
    p = problem_for(name, str(tmp_path))
    b = cg.ManyBodyStates(p)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=True)
    dt = torch.float32 if prec == cg.CG_PREC_FP32 else torch.float64
    x = torch.randn(b.n, ld, generator=torch.Generator().manual_seed(5), dtype=dt).cuda()

    def product(xp, yp):
        torch.cuda.synchronize()
        h.spmm_device(xp.data_ptr(), ld, yp.data_ptr(), ld, m, prec)
        torch.cuda.synchronize()

    y = torch.empty_like(x)
    product(x, y)
    z = x.clone()
    product(z, z)
    assert torch.equal(z[:, :m], y[:, :m])
    if m <= (8 if prec == cg.CG_PREC_FP32 else 4):  # one pass
        for shift in (0, 1):
            buf = torch.empty(b.n + 1, ld, dtype=dt, device="cuda")
            buf[shift:shift + b.n] = x
            product(buf[shift:], buf[1 - shift:])
            assert torch.equal(buf[1 - shift:][:b.n, :m], y[:, :m])
