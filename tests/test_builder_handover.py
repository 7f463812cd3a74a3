"""Hits on both sides of the sizes where the builder hands over: a segment of
64 triangles, one block's task (480 triangles in builds below 130,000, 960
from there), and the sizes from which tasks, sort tiles and level items are
larger (130,000, 300,000, 600,000)."""
import numpy as np
import pytest

FLT_MAX = np.float32(np.finfo(np.float32).max)


def _soup(nt, size):
    rng = np.random.default_rng(nt)
    V = rng.uniform(-1, 1, size=(nt, 1, 3)) + rng.uniform(-size, size, size=(nt, 3, 3))
    return V.reshape(-1, 3).astype(np.float32), np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)


def _rays(V, n):
    from j3d_gb300._ffi import RAY_DTYPE
    rng = np.random.default_rng(n)
    rays = np.zeros(n, RAY_DTYPE)
    o = rng.normal(size=(n, 3))
    o = 3 * o / np.linalg.norm(o, axis=1, keepdims=True)
    rays["orig"][:, :3] = o
    rays["dir"][:, :3] = V[rng.integers(0, len(V), n)] + rng.normal(size=o.shape) * 0.02 - o
    rays["orig"][:, 3] = 1
    rays["t_far"] = FLT_MAX
    return rays


@pytest.mark.gpu
@pytest.mark.parametrize("width,leaf", [(4, 2), (2, 1), (8, 8)])
@pytest.mark.parametrize("nt,brute", [(n, True) for n in (63, 64, 65, 479, 480, 481, 959, 960, 961, 962, 1921)] +
                         [(n, False) for n in (129_999, 130_000, 299_999, 300_000, 599_999, 600_000)])
def test_hits(gpu_ctx, oracle_mod, nt, brute, width, leaf):
    from j3d_gb300 import Mesh, SceneObject, find_closest
    I16 = np.eye(4, dtype=np.float32).reshape(16)
    V, T = _soup(nt, 0.15 if brute else 0.02)
    rays = _rays(V, 2000)
    hg = find_closest(gpu_ctx, [SceneObject(Mesh(gpu_ctx, V, T, leaf, width=width), I16, 1)], rays)
    ho, _ = oracle_mod.find_closest([(oracle_mod.Mesh(V, T), I16, 1)], rays, brute=brute)
    assert np.array_equal(hg.view(np.uint8), ho.view(np.uint8))
    assert hg["found"].any()


@pytest.mark.gpu
@pytest.mark.parametrize("width,mixed", [(4, False), (4, True), (2, False), (8, False)])
def test_rebuilds_of_all_sizes_in_one_graph(gpu_ctx, width, mixed):
    """More meshes than lanes, the sizes of every regime among them: a lane's
    scratch, sized for its largest mesh, serves smaller ones that need more
    items, tasks and sort tiles; every rebuilt tree is the standalone build's."""
    from j3d_gb300 import Batch, Canvas, Matcap, Mesh, Scene, camera_for_vfov
    sizes = [700_000, 610_000, 599_000, 301_000, 299_000, 131_000, 129_000, 1000, 650_000, 305_000, 150_000, 40_000,
             600_001, 299_999, 129_999, 961, 481, 65, 9]
    mc, frames, meshes = Matcap.make(gpu_ctx, 0), [], []
    for k, nt in enumerate(sizes):
        V, T = _soup(nt, 0.02)
        meshes.append(Mesh(gpu_ctx, V, T, build="lbvh" if mixed and k % 3 == 1 else "ploc", width=width, rebuildable=True))
        sc = Scene()
        sc.add_object(meshes[-1], db_id=1)
        sc.prepare_scene()
        sc.unzoom()
        cv = Canvas(gpu_ctx, 32, 24)
        cv.set_camera(camera_for_vfov(60.0))
        cv.set_background_color()
        frames.append((cv, sc, mc))
    before = [m.nodes() for m in meshes]
    g = Batch(gpu_ctx, frames, rebuild=True)
    for _ in range(2):
        g.launch()
    gpu_ctx.synchronize()
    assert gpu_ctx.device_status() == 0
    for nt, m, b in zip(sizes, meshes, before):
        assert np.array_equal(m.nodes().view(np.uint32), b.view(np.uint32)), f"{nt} triangles"
    g.close()
    for cv, _, _ in frames:
        cv.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nt", [3, 40, 65, 481, 2500, 20000])
@pytest.mark.parametrize("kind", ["infinite", "huge"])
def test_boxes_without_an_area_are_refused(gpu_ctx, nt, kind):
    """No pair of clusters has a smallest area: the build says so, places
    nothing, and the next one is as ever."""
    from j3d_gb300 import J3dgError, Mesh
    V, T = _soup(nt, 0.02)
    good = Mesh(gpu_ctx, V, T, 1, width=2).nodes()
    W = V.copy()
    if kind == "infinite":
        W[1::3, 0] = np.inf
    else:
        W *= np.float32(3e38)
    with pytest.raises(J3dgError, match="malformed tree"):
        Mesh(gpu_ctx, W, T, 1, width=2)
    assert np.array_equal(Mesh(gpu_ctx, V, T, 1, width=2).nodes().view(np.uint32), good.view(np.uint32))
    assert gpu_ctx.device_status() == 0
