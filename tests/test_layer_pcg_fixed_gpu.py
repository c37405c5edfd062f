"""The PCG in the layer solve with a fixed number of iterations: one
correction before the last layer's Gauss-Seidel and one after every `every`
of its iterations, on every launch path that runs several iterations in one
launch.  FP64 against the CPU restatement (the corrections of
oracle/pcg.py, the oracle's projectGS for the sweeps between them), within
1e-8 of the bounding-box diagonal as the residual-driven solve is; FP32
bit for bit against the colour launches, whose loop issues one iteration at
a time.  Intervals: a remainder, one dividing the count, longer than the
loop, and 0 (only the correction before the loop)."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib, scenes
from multilayersolver2024_b200.mesh3d import Mesh3D, to_lame
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import Case

pytestmark = pytest.mark.gpu

PATHS = {
    "default": {},
    "colours": {"MLXPBD_FLOW": "0", "MLXPBD_GROUPS": "0"},
    "flow": {"MLXPBD_FLOW": "1"},
    "sweep": {"MLXPBD_FLOW": "2"},
    "groups": {"MLXPBD_FLOW": "0", "MLXPBD_GROUPS": "1"},
    "cluster": {"MLXPBD_CLUSTER": "1"},
    "persistent": {"MLXPBD_PERSISTENT": "1"},
}
K_PCG = 60


def _block(dims=(8, 4, 4), seed=2):
    rng = np.random.default_rng(seed)
    V, T, _ = scenes.generate_beam(*dims, 0.1)
    n = T.shape[0]
    mu, lam = to_lame(rng.uniform(0.25, 0.45, n), np.exp(rng.uniform(np.log(1e4), np.log(1e7), n)))
    m = Mesh3D.from_arrays(V, T, mu, lam, rho=1000.0, energy_type=_lib.MLX_ENERGY_NEOHOOKEAN)
    m.pin(np.nonzero(np.isclose(V[:, 2], 0.0))[0] + 1)
    return m


def _case(m, iterations):
    return Case(m, [0], [iterations], seed=3, h=1.0 / 60.0, perturb=0.002, vel=0.5)


@pytest.fixture(scope="module")
def restated(oracle):
    """Positions after `iterations` sweeps with corrections, on the CPU."""
    from oracle import pcg as PCG
    known = {}

    def solve(iterations, every):
        if (iterations, every) in known:
            return known[iterations, every]
        m = _block()
        case = _case(m, iterations)
        h, x, lam = case.h, case.xi + case.h * case.resv, np.asfortranarray(case.lam.copy())
        free = np.setdiff1d(np.arange(3 * m.N), m.pinnedDOFs - 1)
        P = oracle.params(case.integ, h)
        done = 0
        while done < iterations:
            A, b, prec, J, W, C = PCG.nh_linearized_step(m, x, h, np.stack([lam[:, 0], lam[:, 1]], 1).ravel(), free)
            dx = np.zeros(3 * m.N)
            dx[free] = PCG.solve_pcg(K_PCG, A, b, np.zeros(free.size), prec)[0]
            ln = -(W @ (C + J @ dx))
            x, lam = x + dx, np.zeros_like(lam)
            lam[:, 0], lam[:, 1] = ln[0::2], ln[1::2]
            n = min(every, iterations - done) if every else iterations
            x, _, _, _, lam, its = oracle.layer_solve(m, case.ls, case.integ.layersMap, [n], P, oracle.ContactList(), x,
                                                      lam, case.oldp, case.oldOldp, case.f, np.zeros(3 * m.N),
                                                      case.pinnedx, np.array([0.0]), 0.0, "lame", True)
            done += n
        known[iterations, every] = x
        return x

    return solve


def _product(monkeypatch, path, precision, iterations, every):
    for k, v in PATHS[path].items():
        monkeypatch.setenv(k, v)
    m = _block()
    s = Solver(m, precision=precision, material="lame")
    s.layer_pcg(K_PCG, every)
    # the first call issues the loop, the second one records and replays it
    out = [_case(m, iterations).product(precision, "lame", solver=s) for _ in range(2)]
    s.close()
    for k in PATHS[path]:
        monkeypatch.delenv(k)
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][5] == out[1][5] == iterations
    return m, out[0]


@pytest.mark.parametrize("path", list(PATHS))
@pytest.mark.parametrize("iterations,every", [(7, 3), (6, 2), (4, 9), (4, 0)])
def test_fixed_iterations_against_the_cpu(gpu, monkeypatch, restated, path, iterations, every):
    m, res = _product(monkeypatch, path, _lib.MLX_FP64, iterations, every)
    assert np.abs(res[0] - restated(iterations, every)).max() / m.bbox_diagonal() <= 1e-8


@pytest.mark.parametrize("path", ["default", "flow", "sweep", "groups"])
@pytest.mark.parametrize("iterations,every", [(7, 3), (5, 1)])
def test_fixed_iterations_bits(gpu, monkeypatch, path, iterations, every):
    _, a = _product(monkeypatch, "colours", _lib.MLX_FP32, iterations, every)
    _, b = _product(monkeypatch, path, _lib.MLX_FP32, iterations, every)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[4], b[4])


@pytest.mark.parametrize("graph", [True, False])
def test_resident_steps(gpu, monkeypatch, graph):
    """The stepper's fixed loop, as a recorded step and issued call by call."""
    def run(path):
        for k, v in PATHS[path].items():
            monkeypatch.setenv(k, v)
        m = _block()
        it = XpbdLayer3D()
        it.setLayers([0])
        it.iterations = [7]
        sets = np.zeros((m.T, 1), np.int32, order="F")
        it.customRigidSets = sets
        s = Solver(m, precision=_lib.MLX_FP32, material="lame")
        s.layer_pcg(K_PCG, 3)
        sim = ResidentSim(s, it, find_boundary_vertices(m, sets, [0]), 1.0 / 60.0)
        sim.step(3, graph=graph)
        out = sim.state()
        s.close()
        for k in PATHS[path]:
            monkeypatch.delenv(k)
        return out
    for x, y in zip(run("colours"), run("default")):
        np.testing.assert_array_equal(x, y)
