"""The voxel grid where its rays' groups of lanes can go wrong: as many hits a
ray as are kept (64), one triangle, grids whose rays don't fill a block."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("sheets", [1, 2, 33, 63, 64])
@pytest.mark.parametrize("max_dim", [1, 7, 33, 64])
def test_sheets(gpu_ctx, oracle_mod, sheets, max_dim):
    from j3d_gb300 import Mesh, voxelize
    z = np.linspace(-1, 1, sheets)
    V = np.zeros((sheets, 3, 3), np.float32)
    V[:, :, 2] = z[:, None] + (np.array([0, 0.01, 0.02]) if sheets == 1 else 0)
    V[:, 0, :2], V[:, 1, :2], V[:, 2, :2] = (-1, -0.9), (1, -0.8), (0.1, 1)
    T = np.arange(3 * sheets, dtype=np.uint32).reshape(-1, 3)[::-1].copy()  # ids against the rays' direction
    C = np.random.default_rng(sheets).uniform(0, 1, size=(3 * sheets, 3)).astype(np.float32)
    V = V.reshape(-1, 3)
    mesh, om = Mesh(gpu_ctx, V, T), oracle_mod.Mesh(V, T)
    mesh.set_vertex_colors(C)
    om.set_vertex_colors(C)
    assert np.array_equal(voxelize(gpu_ctx, mesh, max_dim), oracle_mod.voxelize(om, max_dim))


@pytest.mark.gpu
@pytest.mark.parametrize("max_dim", [580, 600])  # about 970,000 and 1,040,000 rays
def test_many_rays(gpu_ctx, oracle_mod, max_dim):
    from j3d_gb300 import Mesh, voxelize, workloads as W
    V, T = W.icosphere(2)
    V = (V / np.abs(V).max(axis=0)).astype(np.float32)  # a cube of voxels
    g = voxelize(gpu_ctx, Mesh(gpu_ctx, V, T), max_dim)
    o = oracle_mod.voxelize(oracle_mod.Mesh(V, T), max_dim)
    assert g.shape == o.shape and np.array_equal(g, o)
