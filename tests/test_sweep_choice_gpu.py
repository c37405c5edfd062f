"""Which path a sweep takes and that the choice does not show in the results.

FP64: the sweep through L2 and the colour launches differ in their fused
multiply-adds, so every call of one shape takes the same of the two: the
first (stop rules on the host) and the replayed ones (rules on the device).
One iteration per launch: the colour launches where a CTA of the dataflow
sweep would have too many chunks."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import Case, block_mesh

pytestmark = pytest.mark.gpu

NH, STVK = _lib.MLX_ENERGY_NEOHOOKEAN, _lib.MLX_ENERGY_STVK_VOIGT


def _integ(hanging):
    integ = XpbdLayer3D()
    integ.computeResiduals = True
    integ.runUntilResSmallerThan = 1e-30
    integ.hangingStop = hanging
    return integ


def _three_calls(m, prec, layers, iterations, hanging, material="lame"):
    case = Case(m, layers, iterations, seed=7, integ=_integ(hanging), h=1.0 / 60.0)
    s = Solver(m, precision=prec, material=material)
    out = [case.product(prec, material, solver=s) for _ in range(3)]
    path = s.launch_path
    s.close()
    for xi, _, ra, ru, lam, it in out[1:]:
        assert it == out[0][5] and ru == out[0][3]
        np.testing.assert_array_equal(ra, out[0][2])
        np.testing.assert_array_equal(xi, out[0][0])
        np.testing.assert_array_equal(lam, out[0][4])
    return out[0], path


@pytest.mark.parametrize("energy", [NH, STVK])
@pytest.mark.parametrize("prec", [_lib.MLX_FP32, _lib.MLX_FP64])
@pytest.mark.parametrize("path", ["1", "2"])
@pytest.mark.parametrize("material,alpha1", [("lame", 0.0), ("blocks", 0.0), ("blocks", 0.01)])
def test_replays_of_a_forced_path(gpu, monkeypatch, energy, prec, path, material, alpha1):
    monkeypatch.setenv("MLXPBD_FLOW", path)
    m = block_mesh(dims=(9, 5, 4), energy=energy, seed=5, alpha1=alpha1)
    _three_calls(m, prec, [50, 0], [2, 3], 40, material)


@pytest.mark.parametrize("prec", [_lib.MLX_FP32, _lib.MLX_FP64])
def test_replays_of_a_large_mesh(gpu, monkeypatch, prec):
    m = block_mesh(dims=(48, 28, 28), energy=NH, seed=5)
    a, path = _three_calls(m, prec, [0], [3], 6)
    assert path.startswith("one launch per colour" if prec == _lib.MLX_FP64 else "version-ordered")
    monkeypatch.setenv("MLXPBD_FLOW", "0")
    b, _ = _three_calls(m, prec, [0], [3], 6)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[2], b[2])


@pytest.mark.parametrize("dims,colour_launches", [((16, 6, 6), False), ((48, 24, 24), True)])
def test_one_iteration_per_launch(gpu, monkeypatch, dims, colour_launches):
    m = block_mesh(dims=dims, energy=NH, seed=5)
    sets = np.zeros((m.T, 1), np.int32, order="F")
    ls = find_boundary_vertices(m, sets, [0])

    def run():
        integ = _integ(6)
        integ.setLayers([0])
        integ.iterations = [3]
        integ.customRigidSets = sets
        s = Solver(m, precision=_lib.MLX_FP32)
        sim = ResidentSim(s, integ, ls, 1.0 / 60.0)
        sim.step(2)
        out = sim.state() + (sim.monitor()[0],)
        n = sim.launches_per_step
        s.close()
        return out, n
    a, n = run()
    assert (n > m.numColors) == colour_launches
    monkeypatch.setenv("MLXPBD_FLOW", "1")
    b, n = run()
    assert n < m.numColors
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
