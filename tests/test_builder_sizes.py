"""Builds at the sizes where the builder changes how it splits: one cluster
list (at most 64 triangles), one block's task (at most 1024), level by level
above that; and meshes whose splits are lopsided or by position."""
import numpy as np
import pytest

I16 = np.eye(4, dtype=np.float32).reshape(16)
FLT_MAX = np.float32(np.finfo(np.float32).max)


def _mesh(kind, nt, rng):
    c = rng.uniform(-1, 1, size=(nt, 1, 3))
    V = c + rng.uniform(-0.15, 0.15, size=(nt, 3, 3))
    if kind == "scales":  # sizes over six magnitudes: splits far from the middle
        V = V * 10.0 ** rng.uniform(-6, 0, size=(nt, 1, 1))
    elif kind == "stacked":  # one centroid: every split is by position
        V = np.tile(V[:1], (nt, 1, 1))
    return V.reshape(-1, 3).astype(np.float32), np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nt,width,leaf",
                         [(k, n, w, l) for w, l in ((4, 2), (2, 1), (8, 8))
                          for k, n in (("soup", 9), ("soup", 64), ("soup", 65), ("soup", 66), ("soup", 1023),
                                       ("soup", 1024), ("soup", 1025), ("soup", 2049), ("soup", 20011),
                                       ("stacked", 1024), ("stacked", 3000))] +
                         # (trees deeper than the traversal stack's bound at widths 4 and 8 are refused)
                         [("scales", 1000, 2, 1), ("scales", 9000, 2, 1)])
def test_build_matches_brute_force(gpu_ctx, oracle_mod, kind, nt, width, leaf):
    from j3d_gb300 import Mesh, SceneObject, find_closest
    from j3d_gb300._ffi import RAY_DTYPE
    O = oracle_mod
    rng = np.random.default_rng(nt + len(kind))
    V, T = _mesh(kind, nt, rng)
    rays = np.zeros(2000, RAY_DTYPE)
    o = rng.normal(size=(len(rays), 3))
    o = 3 * o / np.linalg.norm(o, axis=1, keepdims=True)
    rays["orig"][:, :3] = o
    rays["dir"][:, :3] = V[rng.integers(0, len(V), len(rays))] + rng.normal(size=o.shape) * 0.02 - o
    rays["orig"][:, 3] = 1
    rays["t_far"] = FLT_MAX
    mesh = Mesh(gpu_ctx, V, T, leaf, width=width)
    info = mesh.info()
    assert 1 <= info.n_nodes < max(2, nt)
    hg = find_closest(gpu_ctx, [SceneObject(mesh, I16, 1)], rays)
    ho, _ = O.find_closest([(O.Mesh(V, T), I16, 1)], rays, brute=True)
    assert np.array_equal(hg.view(np.uint8), ho.view(np.uint8))
    assert hg["found"].any()
