"""Host threads with handles of their own at the same time: kernels whose
dynamic shared memory depends on the handle (rows of a stored build, staged
blocks of the on-the-fly and the block-tiled products) must launch whatever the
other threads' sizes are.  Every result is bit-identical to the one of a thread
alone.  The window between another thread's setting and a launch is a few
microseconds, so the sources are read as well."""
import os
import re
import threading

import numpy as np
import pytest

import cosmo_gb300 as cg
from cosmo_gb300.synthetic import SyntheticSystem, make_system

SRC = os.path.join(os.path.dirname(cg.__file__), "csrc")

# short rows and blocks, for several threads; rows and blocks that take more
# than the 48 KB of shared memory a launch may always have
SMALL, LONG_ROWS, LONG_BLOCKS, LONG_TILES = ("sd", 3, 3, 0), ("fp", 3, 4, 1), ("fp", 1, 5, 0), ("fp", 2, 4, 0)


def test_attribute_is_the_same_for_every_handle():
    constants = re.compile(r"(kSmemMax|kSmemSort|int\(kRefineSmem\)|int\(jac_smem<(float|double)>\(\)\))$")
    found = 0
    for name in sorted(os.listdir(SRC)):
        with open(os.path.join(SRC, name)) as f:
            for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)\);", f.read()):
                assert constants.match(m.group(1)), (name, m.group(1))
                found += 1
    assert found >= 8


def _problem(tmp_path, system):
    space, nv, zv, twom = system
    par = "-" if space == "fp" and (nv + zv) & 1 else "+"
    p = cg.Problem(make_system(str(tmp_path), SyntheticSystem(space, nv, zv, twom, par, 0.5, 31))[1])
    return p, cg.ManyBodyStates(p)


def _beside(large, small, rounds):
    """large() `rounds` times while other threads call their own small() over and over."""
    want, others = large(), [(f, f()) for f in small]
    errors, stop = [], threading.Event()

    def work(f, ref):
        try:
            while not stop.is_set():
                assert all(map(np.array_equal, f(), ref))
        except BaseException as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=a) for a in others]
    for t in ts:
        t.start()
    try:
        for _ in range(rounds):
            assert all(map(np.array_equal, large(), want))
    finally:
        stop.set()
        for t in ts:
            t.join()
    assert not errors, errors


@pytest.mark.gpu
def test_builds(gpu_available, tmp_path):
    def build(pb):
        h = cg.Hamiltonian(*pb, cg.CG_PREC_FP64)
        return h.upper_rows(0, 64) + (h.diagonal(),)

    def call(system):
        pb = _problem(tmp_path, system)
        return lambda: build(pb)

    _beside(call(LONG_ROWS), [call(SMALL) for _ in range(6)], 200)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["on-the-fly fp64", "tiled"])
def test_products(gpu_available, kind, tmp_path):
    def call(system):
        prec = cg.CG_PREC_FP64 if kind != "tiled" else cg.CG_PREC_FP32
        h = cg.Hamiltonian(*_problem(tmp_path, system), prec, virtual=kind != "tiled")
        if kind == "tiled":
            h.set_format(cg.CG_FORMAT_TILED)
        x = np.random.default_rng(1).standard_normal((h.n, 8))
        return lambda: (h.times_matrix(x, prec),)

    _beside(call(LONG_TILES if kind == "tiled" else LONG_BLOCKS), [call(SMALL) for _ in range(6)], 100)
