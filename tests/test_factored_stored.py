"""The factored FP32 product of stored matrices, the default from 2^24 entries
up, against the FP64-accurate product of the same matrix, and the branches of
the factored form that sd and fp on their own do not reach: species of both
parities, and more than 64 pairs a channel.

Bounds: 5e-6 of max |y| and 2e-6 in the RMS, as for the row-wise and the
block-tiled product; symmetry (x . H y = y . H x) 1e-6 of the norms."""
import itertools

import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _device(h, x, m, prec):
    y = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    h.spmm_device(x.data_ptr(), x.shape[1], y.data_ptr(), y.shape[1], m, prec)
    torch.cuda.synchronize()
    return y


def _within(y, ref):
    d = y.double() - ref
    assert float(d.abs().max()) <= 5e-6 * float(ref.abs().max())
    assert float(d.norm() / ref.norm()) <= 2e-6


# one and several spectator groups; either species the one with fewer cores; the largest stored matrix
@pytest.mark.parametrize("nv,zv,twom", [(2, 4, 0), (5, 2, 1), (4, 4, 0)])
def test_default_product(gpu_available, nv, zv, twom, tmp_path):
    par = "-" if (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem("fp", nv, zv, twom, par, 0.5, 7))[1])
    b = cg.ManyBodyStates(p)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32)
    assert h.info.nnz_full >= 2 ** 24 and h.format_in_use() == cg.CG_FORMAT_FACTORED
    gen = torch.Generator().manual_seed(nv)
    x = torch.randn(b.n, 8, generator=gen).cuda()
    ref = _device(h, x.double(), 8, cg.CG_PREC_REFINE)
    y = _device(h, x, 8, cg.CG_PREC_FP32)
    _within(y, ref)
    for m in range(1, 8):  # the vectors beyond m are zeros, their results are not stored
        xm = x.clone()
        xm[:, m:] = 0
        ym = _device(h, xm, m, cg.CG_PREC_FP32)
        assert torch.equal(ym[:, :m], y[:, :m]) and ym[:, m:].isnan().all()
    z = torch.randn(b.n, 8, generator=gen).cuda()
    hz = _device(h, z, 8, cg.CG_PREC_FP32)
    a, c = (z.double() * y.double()).sum(0), (x.double() * hz.double()).sum(0)
    assert float(((a - c).abs() / (z.double().norm(dim=0) * ref.norm(dim=0))).max()) <= 1e-6
    # more vectors than the form takes go to the rows
    x16 = torch.cat((x, z), 1)
    _within(_device(h, x16, 16, cg.CG_PREC_FP32)[:, :8], ref)


def _two_parities(orbits, nv, zv, twom, parity, seed):
    """Random terms that keep charge, M and parity in a space of (l, 2j) orbits, for both species."""
    one = [(o, l, j2, m2) for o, (l, j2) in enumerate(orbits) for m2 in range(-j2, j2 + 1, 2)]
    sps = np.array([(o, 0, l, j2, m2, 1, t, l & 1) for t in (1, -1) for o, l, j2, m2 in one], dtype=np.int32)
    rng = np.random.default_rng(seed)
    kind = [(s[4], s[7], s[6]) for s in sps.tolist()]
    k1 = [(i, j) for i in range(len(sps)) for j in range(i, len(sps)) if kind[i] == kind[j]]
    by = {}
    for i, j in itertools.combinations(range(len(sps)), 2):
        (m, q, t), (m2, q2, t2) = kind[i], kind[j]
        by.setdefault((m + m2, q ^ q2, t + t2), []).append((i, j))
    k2 = [a + c for l in by.values() for n, a in enumerate(l) for c in l[n:]]
    k1, k2 = np.array(k1, dtype=np.int32), np.array(k2, dtype=np.int32)
    return cg.Problem.from_terms(sps, len(one), nv, zv, twom, parity, k1, rng.uniform(-4, 0, len(k1)), k2,
                                 rng.standard_normal(len(k2)))


P_SD = [(1, 3), (1, 1), (2, 5), (0, 1), (2, 3)]
SD_FP = [(2, 5), (0, 1), (2, 3), (3, 7), (1, 3), (3, 5), (1, 1)]


# p + sd: 18 states; sd + fp: 32 states and channels of up to 88 pairs, which only one neutron and one proton can take
@pytest.mark.parametrize("orbits,nv,zv,twom,parity", [(P_SD, 2, 2, 0, 0), (P_SD, 2, 3, 1, 1), (P_SD, 1, 3, 2, 1),
                                                      (SD_FP, 1, 1, 0, 0), (SD_FP, 1, 1, 2, 1), (SD_FP, 1, 1, 0, 1)])
def test_two_parities(gpu_available, orbits, nv, zv, twom, parity):
    p = _two_parities(orbits, nv, zv, twom, parity, 5)
    b = cg.ManyBodyStates(p)
    h = cg.Hamiltonian(p, b, cg.CG_PREC_FP32, virtual=True)
    assert h.format_in_use() == cg.CG_FORMAT_FACTORED
    x = torch.randn(b.n, 8, generator=torch.Generator().manual_seed(6)).cuda()
    h64 = cg.Hamiltonian(p, b, cg.CG_PREC_FP64, virtual=True)  # element by element
    ref = torch.from_numpy(h64.times_matrix(x.double().cpu().numpy())).cuda()
    _within(_device(h, x, 8, cg.CG_PREC_FP32), ref)
