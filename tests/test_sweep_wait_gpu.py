"""A sweep whose bounded wait ran out ends its call with a status, promptly
also where the stop rules wait for a residual, and leaves the next call
alone.  No wait runs out here: mlx_sweep_wait_probe raises the flag that one
would raise."""
import time

import numpy as np
import pytest

from multilayersolver2024_b200 import _lib
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import Case, block_mesh

pytestmark = pytest.mark.gpu

NEVER = 8000  # iterations of a monitored solve whose residual target is out of reach


def _case(residuals):
    integ = XpbdLayer3D()
    integ.computeResiduals = residuals
    if residuals:
        integ.runUntilResSmallerThan = 1e-30
        integ.hangingStop = NEVER
    m = block_mesh(dims=(6, 3, 3), energy=_lib.MLX_ENERGY_NEOHOOKEAN, seed=5)
    return m, Case(m, [50, 0], [2, 3], seed=7, integ=integ, h=1.0 / 60.0)


def _probe(s):
    _lib.check("mlx_sweep_wait_probe", s._lib.mlx_sweep_wait_probe(s.handle), s._lib)


def _fails(call):
    t0 = time.perf_counter()
    with pytest.raises(_lib.MlxError) as e:
        call()
    assert e.value.code == _lib.MLX_ERR_LIMIT
    return time.perf_counter() - t0


@pytest.mark.parametrize("path", ["1", "2"])
@pytest.mark.parametrize("clean", [0, 2])
def test_fixed_iterations(gpu, monkeypatch, path, clean):
    """Issued (first call) and replayed (after two of the same shape)."""
    monkeypatch.setenv("MLXPBD_FLOW", path)
    m, case = _case(False)
    s = Solver(m, precision=_lib.MLX_FP32)
    want = Case.product(case, _lib.MLX_FP32)
    for _ in range(clean):
        case.product(solver=s)
    _probe(s)
    _fails(lambda: case.product(solver=s))
    got = case.product(solver=s)
    s.close()
    np.testing.assert_array_equal(got[0], want[0])


@pytest.mark.parametrize("clean", [0, 2])
def test_monitored_solve(gpu, monkeypatch, clean):
    """Host rules (first call) and the rules on the device (replayed)."""
    monkeypatch.setenv("MLXPBD_FLOW", "1")
    m, case = _case(True)
    s = Solver(m, precision=_lib.MLX_FP32)
    for _ in range(clean):
        case.product(solver=s)
    _probe(s)
    short = _fails(lambda: case.product(solver=s))
    t0 = time.perf_counter()
    got = case.product(solver=s)
    full = time.perf_counter() - t0
    s.close()
    assert got[5] > NEVER // 2 and np.isfinite(got[0]).all()
    assert short < 0.25 * full, (short, full)


@pytest.mark.parametrize("graph", [True, False])
def test_monitored_steps(gpu, monkeypatch, graph):
    monkeypatch.setenv("MLXPBD_FLOW", "1")
    m, case = _case(True)
    sets = np.asfortranarray(case.ls.rigidBodySetsPerLayer)
    ls = find_boundary_vertices(m, sets, case.ls.numRigids)

    def sim():
        return ResidentSim(Solver(m, precision=_lib.MLX_FP32), case.integ, ls, 1.0 / 60.0)
    a, b = sim(), sim()
    _probe(a.solver)
    _fails(lambda: a.step(1, graph=graph))
    if graph:
        ra, it, _, status = a.monitor()
        assert it == 1 and status == 3
    a = ResidentSim(a.solver, case.integ, ls, 1.0 / 60.0)
    a.step(0, graph=graph)
    for s in (a, b):
        s.step(1, graph=graph)
    for x, y in zip(a.state(), b.state()):
        np.testing.assert_array_equal(x, y)
    assert a.monitor()[1] == b.monitor()[1] > NEVER // 2
