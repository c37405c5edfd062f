"""The tag counter of the sweeps through L2 at its limit: the launch that
passes it clears the records and the next one starts from zero, with the bits
of a solver whose counter is far from it before, at and after it."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import block_mesh

pytestmark = pytest.mark.gpu

LIMIT = 2 ** 32 - 2 ** 29 - 1


def _sim(m, prec):
    it = XpbdLayer3D()
    it.setLayers([0])
    it.iterations = [5]
    sets = np.zeros((m.T, 1), np.int32, order="F")
    it.customRigidSets = sets
    v0 = np.random.default_rng(5).normal(0.0, 0.05, 3 * m.N)
    v0[m.pinnedDOFs - 1] = 0.0
    s = Solver(m, precision=prec)
    return s, ResidentSim(s, it, find_boundary_vertices(m, sets, [0]), 1.0 / 60.0, v0=v0)


@pytest.mark.parametrize("prec", [_lib.MLX_FP32, _lib.MLX_FP64])
@pytest.mark.parametrize("below", [0, 1, 40, 300])
def test_records_cleared_at_the_limit(gpu, monkeypatch, prec, below):
    m = block_mesh(dims=(9, 5, 4), energy=_lib.MLX_ENERGY_NEOHOOKEAN, seed=5)
    monkeypatch.setenv("MLXPBD_FLOW", "2")
    a, ref = _sim(m, prec)
    b, sim = _sim(m, prec)
    lib = _lib.load()
    for k in range(6):
        if k == 2:  # (tags only grow between two clears)
            _lib.check("mlx_sweep_tags_probe", lib.mlx_sweep_tags_probe(b.handle, LIMIT - below), lib)
        ref.step(1)
        sim.step(1)
        for x, y in zip(ref.state(), sim.state()):
            np.testing.assert_array_equal(x, y)
    a.close()
    assert lib.mlx_sweep_tags_probe(b.handle, 0) == 0
    b.close()


def test_refused_without_sweeps_through_l2(gpu, monkeypatch):
    monkeypatch.setenv("MLXPBD_FLOW", "1")
    s = Solver(block_mesh(dims=(2, 2, 2), seed=5))
    lib = _lib.load()
    assert lib.mlx_sweep_tags_probe(s.handle, 0) == _lib.MLX_ERR_UNSUPPORTED
    s.close()
