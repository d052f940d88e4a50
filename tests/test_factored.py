"""Factored FP32 product (cores of two particles taken out) behind the on-the-fly
Hamiltonian against the stored FP64 matrix, at the edges of its tiles: one core
only, either species giving the spectators, 1 to 4 output tiles of a channel
(sd at most 28 pairs, fp up to 60), spectator groups of one and of many, rows
already packed (8 vectors, leading dimension 8) and packed by the call.
Tolerance: 1e-5 of max |y|, as for the other FP32 products."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

pytestmark = pytest.mark.gpu

SYSTEMS = [("sd", 1, 1, 0), ("sd", 2, 1, 1), ("sd", 1, 4, 1), ("sd", 4, 1, 1), ("sd", 3, 3, 0), ("sd", 2, 2, 4),
           ("fp", 1, 1, 0), ("fp", 2, 1, 3), ("fp", 1, 3, 0), ("fp", 3, 2, 1), ("fp", 2, 2, 14)]


@pytest.mark.parametrize("space,nv,zv,twom", SYSTEMS)
def test_factored_matches_stored(gpu_available, space, nv, zv, twom, tmp_path):
    torch = pytest.importorskip("torch")
    par = "-" if space == "fp" and (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem(space, nv, zv, twom, par, 0.5, 31))[1])
    b = cg.ManyBodyStates(p)
    hs = cg.Hamiltonian(p, b, cg.CG_PREC_FP64)
    hv = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=True)
    for m, ld in ((8, 8), (8, 12), (3, 8), (11, 11)):
        x = np.zeros((b.n, ld), dtype=np.float32)
        x[:, :m] = np.random.default_rng(m * ld).standard_normal((b.n, m))
        ref = hs.times_matrix(x[:, :m].astype(np.float64))
        xd = torch.from_numpy(x).cuda()
        yd = torch.full((b.n, ld), float("nan"), dtype=torch.float32, device="cuda")
        ys = []
        for _ in range(2):
            torch.cuda.synchronize()
            hv.spmm_device(xd.data_ptr(), ld, yd.data_ptr(), ld, m, cg.CG_PREC_FP32)
            torch.cuda.synchronize()
            ys.append(yd.cpu().numpy().copy())
        np.testing.assert_allclose(ys[0][:, :m], ref, rtol=0, atol=1e-5 * np.abs(ref).max())
        assert np.array_equal(ys[0][:, :m], ys[1][:, :m])  # fixed order of the sums
        assert np.isnan(ys[0][:, m:]).all()  # columns beyond m are left alone
