"""Plans of the one-launch sweeps that the other tests do not reach: component
groups beside them, planned with the first obstacles; components whose
elements are not consecutive (one component for the plan); layers that change
between calls and grow, beside a recorded resident step."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib, scenes
from multilayersolver2024_b200.contacts import PlaneContactFinder3D
from multilayersolver2024_b200.mesh3d import Mesh3D, to_lame
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import Case, block_mesh

pytestmark = pytest.mark.gpu

NH, STVK = _lib.MLX_ENERGY_NEOHOOKEAN, _lib.MLX_ENERGY_STVK_VOIGT


def _blocks(dims, copies, shuffle=False, energy=NH):
    V, T, _ = scenes.generate_beam(*dims, 0.1)
    n, k = V.shape[0], np.arange(copies)
    V = (V[None] + np.stack([2.0 * k, 0 * k, 0 * k], 1)[:, None]).reshape(-1, 3)
    T = (T[None].astype(np.int64) + (n * k)[:, None, None]).reshape(-1, 4).astype(np.int32)
    rng = np.random.default_rng(4)
    if shuffle:
        T = T[rng.permutation(T.shape[0])]
    mu, lam = to_lame(0.3, np.exp(rng.uniform(np.log(2e4), np.log(2e5), T.shape[0])))
    return Mesh3D.from_arrays(V, T, mu, lam, rho=1000.0, energy_type=energy)


def _sim(m, prec=_lib.MLX_FP32, coloring=False, v0z=0.0):
    it = XpbdLayer3D()
    it.setLayers([0])
    it.iterations = [6]
    it.contactColoring = coloring
    sets = np.zeros((m.T, 1), np.int32, order="F")
    it.customRigidSets = sets
    s = Solver(m, precision=prec)
    v0 = np.random.default_rng(5).normal(0.0, 0.05, 3 * m.N)
    v0[2::3] += v0z
    return s, ResidentSim(s, it, find_boundary_vertices(m, sets, [0]), 1.0 / 60.0, v0=v0)


@pytest.mark.parametrize("coloring", [False, True])
def test_groups_planned_with_the_obstacles(gpu, monkeypatch, coloring):
    def run():
        s, sim = _sim(_blocks((4, 2, 2), 40), coloring=coloring, v0z=-1.0)
        before = s.launch_path
        if before.startswith("dataflow"):  # (switches count when a solver is created)
            monkeypatch.setenv("MLXPBD_GROUPS", "0")
        sim.set_obstacles([PlaneContactFinder3D([0.0, 0.0, 1.0], [0.0, 0.0, -0.005])])
        sim.step(4)
        assert sim.contact_count() > 0
        sim.set_obstacles([PlaneContactFinder3D([0.0, 0.0, 1.0], [0.0, 0.0, 0.001])])
        sim.step(4)
        out = sim.state(), before, s.launch_path
        s.close()
        return out
    a, before, after = run()
    assert before.startswith("dataflow") and "component groups" not in before
    assert "component groups for contacts" in after
    monkeypatch.setenv("MLXPBD_FLOW", "0")
    monkeypatch.setenv("MLXPBD_GROUPS", "0")
    for x, y in zip(a, run()[0]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("path", ["1", "2"])
@pytest.mark.parametrize("dims,copies", [((4, 2, 2), 3), ((9, 7, 6), 4)])
def test_elements_not_grouped_by_component(gpu, monkeypatch, path, dims, copies):
    out = []
    for flag in ("0", path):
        monkeypatch.setenv("MLXPBD_FLOW", flag)
        s, sim = _sim(_blocks(dims, copies, shuffle=True))
        sim.step(3)
        out.append(sim.state())
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("energy", [NH, STVK])
@pytest.mark.parametrize("coloring", [False, True])
def test_contacts_of_a_large_part(gpu, monkeypatch, energy, coloring):
    """More than 400 chunks of 32 tets in one CTA."""
    out = []
    for flag in ("0", "1"):
        monkeypatch.setenv("MLXPBD_FLOW", flag)
        monkeypatch.setenv("MLXPBD_GROUPS", "0")
        monkeypatch.setenv("MLXPBD_FLOW_CS", "1")
        s, sim = _sim(_blocks((20, 12, 12), 1, energy=energy), coloring=coloring, v0z=-1.0)
        sim.set_obstacles([PlaneContactFinder3D([0.0, 0.0, 1.0], [0.0, 0.0, 0.001])])
        sim.step(3)
        assert sim.contact_count() > 0
        assert s.launch_path.startswith("dataflow") == (flag == "1")
        out.append(sim.state())
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("energy,prec", [(NH, _lib.MLX_FP32), (STVK, _lib.MLX_FP32), (NH, _lib.MLX_FP64)])
@pytest.mark.parametrize("path", ["1", "2"])
def test_layers_that_grow(gpu, monkeypatch, energy, prec, path):
    """A resident step, recorded once, after every host call of the same
    solver (they share the vertex positions)."""
    m = block_mesh(dims=(9, 5, 4), energy=energy, seed=5)
    sims = []
    for flag in ("0", path):
        monkeypatch.setenv("MLXPBD_FLOW", flag)
        sims.append(_sim(m, prec))
    d = m.bbox_diagonal()

    def same(x, y):
        if prec == _lib.MLX_FP32:
            np.testing.assert_array_equal(x, y)
        assert np.abs(x - y).max() <= 1e-12 * d
    for k, pct in enumerate([95, 60, 80, 20, 5, 95, 0]):  # elastic tets: few, more, ..., all
        layers, its = ([0], [3]) if pct == 0 else ([pct, 0], [3, 2])
        case = Case(m, layers, its, seed=30 + k)
        a, b = (case.product(prec, solver=s) for s, _ in sims)
        same(a[0], b[0])
        for _, sim in sims:
            sim.step(1)
        same(*(sim.state()[0] for _, sim in sims))
    for s, _ in sims:
        s.close()
