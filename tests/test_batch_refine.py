"""Batches of one to 160 problems: the cluster of CTAs that refines a problem's
projected eigenvectors has 8 down to 1 of them, with even and uneven column
splits; and single-particle energies with J-J+ alone, whose projected
matrices have clusters of equal eigenvalues.  A residual r bounds the distance
to the nearest eigenvalue by r (1e-5 here)."""
import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SMALL = [(2, 2, 0), (3, 1, 0), (4, 1, 1), (2, 3, 1)]


def _system(tmp, nv, zv, twom, seed, free=False):
    path, xml = make_system(str(tmp), SyntheticSystem("sd", nv, zv, twom, "+", 0.5, seed))
    if free:
        with open(path) as f:
            lines = f.read().splitlines(True)
        with open(path, "w") as f:
            for i, line in enumerate(lines):
                f.write(line if i < 2 else line[:-11] + "%10.4f\n" % 0.0)
    return cg.Problem(xml)


def _exact(p, k):
    inf = p.info
    z = O.basis(p.sps(), inf.nv + inf.zv, inf.twom, inf.nv - inf.zv, inf.parity)
    k1, v1 = p.one_body()
    k2, v2 = p.two_body()
    H = O.full_from_upper(*O.build_upper(inf.n_sps, k1, v1, k2, v2, z)).toarray()
    assert len(z) > 64
    return np.linalg.eigvalsh(H)[:k]


@pytest.mark.parametrize("count", [1, 2, 5, 30, 60, 160])
def test_batch_sizes(gpu_available, count, tmp_path):
    kinds = [_system(tmp_path, *s, 31) for s in SMALL]
    exact = [_exact(p, 5) for p in kinds]
    eig, res, nconv, _ = cg.Batch([kinds[i % len(kinds)] for i in range(count)]).solve(5)
    for i in range(count):
        assert nconv[i] == 5 and np.all(res[i, :5] <= 1e-5)
        np.testing.assert_allclose(eig[i, :5], exact[i % len(kinds)], rtol=0, atol=1e-5)


def test_batch_equal_eigenvalues(gpu_available, tmp_path):
    ps = [_system(tmp_path, *s, 31, free=True) for s in SMALL]
    eig, res, nconv, _ = cg.Batch(ps).solve(5)
    for i, p in enumerate(ps):
        # unit start vectors of a multiplet may miss a state: what counts is
        # that every value lies within its residual of an eigenvalue
        H = _exact(p, None)
        assert nconv[i] == np.sum(res[i, :5] <= 1e-5)
        for e, r in zip(eig[i, :5], res[i, :5]):
            assert np.min(np.abs(H - e)) <= r + 1e-9
