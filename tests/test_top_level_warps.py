"""Rays through a top level of objects: a warp's rays wait for one another at
leaves, so ray counts around whole warps, few and many objects, hits of all of
them and of none."""
import numpy as np
import pytest

FLT_MAX = np.float32(np.finfo(np.float32).max)


@pytest.mark.gpu
@pytest.mark.parametrize("n_obj", [2, 9, 33])
@pytest.mark.parametrize("n_rays", [1, 31, 33, 1000])
def test_rays_match_brute_force(gpu_ctx, oracle_mod, n_obj, n_rays):
    from j3d_gb300 import Mesh, SceneObject, find_closest
    from j3d_gb300._ffi import RAY_DTYPE
    O = oracle_mod
    rng = np.random.default_rng(100 * n_obj + n_rays)
    gpu, cpu = [], []
    for k in range(n_obj):
        nt = (1, 12, 700)[k % 3]
        V = (rng.uniform(-1, 1, size=(nt, 1, 3)) + rng.uniform(-0.3, 0.3, size=(nt, 3, 3))).reshape(-1, 3).astype(np.float32)
        T = np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)
        cs = np.eye(4, dtype=np.float32)
        cs[3, :3] = rng.uniform(-3, 3, size=3)
        gpu.append(SceneObject(Mesh(gpu_ctx, V, T), cs.reshape(16), k + 1))
        cpu.append((O.Mesh(V, T), cs.reshape(16), k + 1))
    rays = np.zeros(n_rays, RAY_DTYPE)
    o = rng.normal(size=(n_rays, 3))
    o = 9 * o / np.linalg.norm(o, axis=1, keepdims=True)
    rays["orig"][:, :3] = o
    rays["orig"][:, 3] = 1
    rays["dir"][:, :3] = rng.uniform(-3, 3, size=(n_rays, 3)) - o
    rays["dir"][::7, :3] *= -1  # away from everything
    rays["t_far"] = FLT_MAX
    hg = find_closest(gpu_ctx, gpu, rays)
    ho, _ = O.find_closest(cpu, rays, brute=True)
    assert np.array_equal(hg.view(np.uint8), ho.view(np.uint8))
