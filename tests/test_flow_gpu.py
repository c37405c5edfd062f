"""The one-launch sweeps (flow.cuh: colours ordered by the vertices' chains,
records pushed through shared memory; sweep.cuh: versions through L2) against
one launch per colour: the same
arithmetic in the same order at every vertex, so FP32 results are equal bit
for bit (FP64 to the compiler's choice of fused multiply-adds), and against
the oracle.  Sizes: less than one chunk of 32 tets, ragged chunks, several
CTAs per cluster, several components per cluster and several clusters."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib, scenes
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import Case, block_mesh, rel_pos_err

pytestmark = pytest.mark.gpu

NH, STVK = _lib.MLX_ENERGY_NEOHOOKEAN, _lib.MLX_ENERGY_STVK_VOIGT


def _paths(monkeypatch, make, cs="", path="1"):
    """make() on the colour launches and on the dataflow path (or, "2", the
    sweep whose versions go through L2)."""
    out = []
    monkeypatch.setenv("MLXPBD_GROUPS", "0")
    for flag in ("0", path):
        monkeypatch.setenv("MLXPBD_FLOW", flag)
        if cs:
            monkeypatch.setenv("MLXPBD_FLOW_CS", cs)
        out.append(make())
    return out


def _resident(sc, steps, graph=True, precision=_lib.MLX_FP32, residuals=False, v0z=0.0):
    it = XpbdLayer3D()
    it.setLayers(sc.layers)
    it.iterations = list(sc.iterations)
    it.computeResiduals = residuals
    it.runUntilResSmallerThan = 2e-3 if residuals else -1.0
    it.contactResistance = sc.settings.get("contactResistance", it.contactResistance)
    it.contactColoring = bool(sc.settings.get("contactColoring", False))
    sets = sc.custom_sets
    ls = find_boundary_vertices(sc.mesh, sets, [int(sets[:, k].max(initial=0)) for k in range(sets.shape[1])])
    s = Solver(sc.mesh, precision=precision)
    v0 = np.zeros_like(sc.mesh.p)
    v0[2::3] = v0z
    sim = ResidentSim(s, it, ls, sc.h, v0=v0)
    if sc.impulse is not None:
        sim.add_velocity(*sc.impulse)
    if sc.contact_finders:
        sim.set_obstacles(sc.contact_finders)
    out = []
    for _ in range(steps):
        sim.step(1, graph=graph)
        out.append(sim.state() + ((sim.monitor()[0],) if residuals else ()))
    path = s.launch_path
    s.close()
    return out, path


def _same(runs):
    (a, pa), (b, pb) = runs
    assert "sweeps, one launch each" in pb and "sweeps, one launch each" not in pa
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("energy,alpha1,material", [(NH, 0.0, "blocks"), (STVK, 0.0, "blocks"), (STVK, 0.01, "blocks"),
                                                    (STVK, 0.01, "lame")])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 2), (9, 5, 4)])
@pytest.mark.parametrize("prec", [_lib.MLX_FP32, _lib.MLX_FP64])
@pytest.mark.parametrize("path", ["1", "2"])
def test_layer_solve(gpu, monkeypatch, energy, alpha1, material, dims, prec, path):
    def make():
        m = block_mesh(dims=dims, energy=energy, seed=5, alpha1=alpha1)
        c = Case(m, [50, 25, 0], [2, 3, 5], seed=6)
        c.integ.boundaryCompliance = 1e-7
        return c, c.product(prec, material)
    (c, a), (_, b) = _paths(monkeypatch, make, path=path)
    if prec == _lib.MLX_FP32:
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[4], b[4])
    assert rel_pos_err(a[0], b[0], c.mesh) <= 1e-13
    assert rel_pos_err(b[0], c.oracle(material)[0], c.mesh) <= (1e-9 if prec == _lib.MLX_FP64 else 2e-5)


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("residuals", [False, True])
@pytest.mark.parametrize("path", ["1", "2"])
def test_resident_steps(gpu, monkeypatch, graph, residuals, path):
    _same(_paths(monkeypatch, lambda: _resident(scenes.config2(nx=31, ny=13, nz=9), 4, graph, residuals=residuals),
                 path=path))


@pytest.mark.parametrize("cs", ["1", "2", "16"])
def test_components(gpu, monkeypatch, cs):
    """A batch of uneven blocks: components per group and CTAs per component."""
    _same(_paths(monkeypatch, lambda: _resident(scenes.config3(seed=7, n_scenes=9, tmin=600, tmax=6000), 3), cs))


@pytest.mark.parametrize("coloring,path,cs", [(False, "1", "1"), (False, "1", "4"), (True, "1", "1"), (True, "1", "4"),
                                              (False, "2", "")])
def test_device_contacts(gpu, monkeypatch, coloring, path, cs):
    """Contacts inside the sweep: after it (the reference's order) and
    coloured with the elastic constraints, below layers with bodies."""
    def make():
        sc = scenes.config4(seed=11, n_boxes=3, cubes=4, grid=(3, 1), spacing=1.5, n_spheres=1, coarse=2, mid=2,
                            drop=(0.005, 0.015), contact_coloring=coloring)
        return _resident(sc, 30, v0z=-1.0)
    _same(_paths(monkeypatch, make, cs, path))


@pytest.mark.parametrize("coloring", [False, True])
@pytest.mark.parametrize("boxes,cubes", [(2, 2), (6, 5)])
def test_device_contacts_default(gpu, monkeypatch, boxes, cubes, coloring):
    """The paths picked without switches: reference-order contacts of
    body-free layers on the component groups where those are planned, the
    rest on the dataflow sweeps; the same bits as with the
    colour launches."""
    def make():
        sc = scenes.config4(seed=12, n_boxes=boxes, cubes=cubes, grid=(boxes, 1), spacing=1.5, n_spheres=1, coarse=2,
                            mid=2, drop=(0.005, 0.015), contact_coloring=coloring)
        return _resident(sc, 30, v0z=-1.0)
    monkeypatch.setenv("MLXPBD_FLOW", "0")
    monkeypatch.setenv("MLXPBD_GROUPS", "0")
    a = make()
    monkeypatch.delenv("MLXPBD_FLOW")
    monkeypatch.delenv("MLXPBD_GROUPS")
    _same([a, make()])


@pytest.mark.parametrize("path", ["1", "2"])
def test_partial_pins(gpu, monkeypatch, path):
    """Pinned DOFs of one axis only, and on a vertex of every corner kind."""
    def make():
        m = block_mesh(dims=(5, 3, 2), energy=NH, seed=9)
        m.pinnedDOFs = np.sort(np.concatenate([m.pinnedDOFs[::2], [3 * m.N - 1]])).astype(np.int32)
        c = Case(m, [0], [4], seed=10)
        return c, c.product(_lib.MLX_FP32)
    (c, a), (_, b) = _paths(monkeypatch, make, path=path)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(b[0][c.mesh.pinnedDOFs - 1], c.pinnedx.astype(np.float32).astype(np.float64))
