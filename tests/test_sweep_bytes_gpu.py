"""mlx_sim_sweep_stats books the bytes of the kernel that ran: the chunk
planes and multipliers for the dataflow sweeps (vertex records stay in shared
memory, positions once per launch), every record for the sweeps through L2
and the colour launches."""
import numpy as np
import pytest

from multilayersolver2024_b200 import _lib, scenes
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim, Solver, XpbdLayer3D, find_boundary_vertices

from helpers import block_mesh

pytestmark = pytest.mark.gpu


# Neo-Hookean FP32: 12 words of planes, 32 bytes of corners, two multipliers
# read and written; vertex ids, 9 + 2 words, the multipliers, eight records
@pytest.mark.parametrize("path,per_tet", [("1", 48 + 32 + 16), ("2", 16 + 44 + 16 + 128), ("0", 16 + 44 + 16 + 128)])
def test_bytes_of_a_fixed_loop(gpu, monkeypatch, path, per_tet):
    monkeypatch.setenv("MLXPBD_FLOW", path)
    if path == "0":
        monkeypatch.setenv("MLXPBD_GROUPS", "0")
    m = block_mesh(dims=(6, 4, 4), energy=_lib.MLX_ENERGY_NEOHOOKEAN, seed=5)
    it = XpbdLayer3D()
    it.setLayers([0])
    it.iterations = [5]
    sets = np.zeros((m.T, 1), np.int32, order="F")
    it.customRigidSets = sets
    s = Solver(m, precision=_lib.MLX_FP32)
    sim = ResidentSim(s, it, find_boundary_vertices(m, sets, [0]), 1.0 / 60.0)
    sim.sweep_timing(True)
    sim.step(1)
    _, b, n = sim.sweep_stats()
    s.close()
    assert b == 5 * m.T * per_tet + (2 * m.N * 16 if path == "1" else 0)
    assert n == (1 if path != "0" else 5 * m.numColors)


@pytest.mark.parametrize("path,per_tet,launch", [("1", 96, 1), ("2", 204, 0)])
def test_bytes_with_bodies(gpu, monkeypatch, path, per_tet, launch):
    """One iteration per launch; a layer's list is read by the sweep through L2."""
    monkeypatch.setenv("MLXPBD_FLOW", path)
    sc = scenes.config2(nx=16, ny=6, nz=6)
    m = sc.mesh
    it = XpbdLayer3D()
    it.setLayers(sc.layers)
    it.iterations = list(sc.iterations)
    sets = sc.custom_sets
    ls = find_boundary_vertices(m, sets, [int(sets[:, k].max(initial=0)) for k in range(sets.shape[1])])
    s = Solver(m, precision=_lib.MLX_FP32)
    sim = ResidentSim(s, it, ls, sc.h)
    sim.sweep_timing(True)
    sim.step(1)
    _, b, n = sim.sweep_stats()
    s.close()
    want = 0
    columns = sorted(set(sc.layers))
    for layer, its in zip(sc.layers, sc.iterations):
        k = columns.index(layer)
        e = int((sets[:, k] == 0).sum())
        bodies = int(sets[:, k].max(initial=0)) > 0
        launches = its if bodies else 1
        want += its * e * (per_tet + (4 if path == "2" and e < m.T else 0)) + launch * launches * 2 * m.N * 16
    assert b == want
