"""Ray batches on several objects with more rays than the device has lanes:
warps refill from a counter and their rays wait for one another at leaves
until none is left to refill with. (At most a lane each, as in
test_top_level_warps.py, every ray goes by itself.) The bound is taken from
the device, so no occupancy of the kernel lets the cases fall below it."""
import numpy as np
import pytest

FLT_MAX = np.float32(np.finfo(np.float32).max)


def _scene(ctx, O, n_obj, width):
    from j3d_gb300 import Mesh, SceneObject
    rng = np.random.default_rng(n_obj)
    gpu, cpu = [], []
    for k in range(n_obj):
        nt = (1, 12, 700)[k % 3]
        V = (rng.uniform(-1, 1, size=(nt, 1, 3)) + rng.uniform(-0.3, 0.3, size=(nt, 3, 3))).reshape(-1, 3).astype(np.float32)
        T = np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)
        cs = np.eye(4, dtype=np.float32)
        cs[3, :3] = rng.uniform(-3, 3, size=3)
        gpu.append(SceneObject(Mesh(ctx, V, T, width=width), cs.reshape(16), k + 1))
        cpu.append((O.Mesh(V, T), cs.reshape(16), k + 1))
    return gpu, cpu


@pytest.mark.gpu
@pytest.mark.parametrize("n_obj,width", [(2, 4), (9, 4), (33, 4), (9, 2), (9, 8)])
@pytest.mark.parametrize("times,more", [(1, 1), (1, 31), (2, 0), (3, 17)])
def test_more_rays_than_lanes(gpu_ctx, oracle_mod, n_obj, width, times, more):
    import torch
    from j3d_gb300 import find_closest
    from j3d_gb300._ffi import RAY_DTYPE
    p = torch.cuda.get_device_properties(0)
    n = times * p.multi_processor_count * p.max_threads_per_multi_processor + more
    gpu, cpu = _scene(gpu_ctx, oracle_mod, n_obj, width)
    rng = np.random.default_rng(n)
    rays = np.zeros(n, RAY_DTYPE)
    o = rng.normal(size=(n, 3))
    o = 9 * o / np.linalg.norm(o, axis=1, keepdims=True)
    rays["orig"][:, :3] = o
    rays["orig"][:, 3] = 1
    rays["dir"][:, :3] = rng.uniform(-3, 3, size=(n, 3)) - o
    rays["dir"][::7, :3] *= -1  # away from everything
    rays["t_far"] = FLT_MAX
    hg = find_closest(gpu_ctx, gpu, rays)
    ho, _ = oracle_mod.find_closest(cpu, rays)
    assert np.array_equal(hg.view(np.uint8), ho.view(np.uint8))
    any_hit = find_closest(gpu_ctx, gpu, rays, any_hit=True)
    assert np.array_equal(any_hit["found"], ho["found"])
    assert ho["found"].any() and not ho["found"].all()
