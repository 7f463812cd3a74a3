"""The wide nodes of a build stand in depth-first order (a node's subtree is
the range that follows it) and their leaves in the order of the triangles."""
import numpy as np
import pytest

LEAF, EMPTY = 0x80000000, 0xffffffff


@pytest.mark.gpu
@pytest.mark.parametrize("width,leaf", [(4, 2), (2, 1), (8, 8)])
@pytest.mark.parametrize("nt", [9, 64, 65, 479, 480, 481, 959, 960, 961, 1921, 20011, 129_999, 130_000])
def test_depth_first(gpu_ctx, nt, width, leaf):
    from j3d_gb300 import Mesh
    rng = np.random.default_rng(nt)
    V = (rng.uniform(-1, 1, size=(nt, 1, 3)) + rng.uniform(-0.1, 0.1, size=(nt, 3, 3))).reshape(-1, 3)
    mesh = Mesh(gpu_ctx, V.astype(np.float32), np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3), leaf, width=width)
    nodes = mesh.nodes().reshape(mesh.info().n_nodes, -1)
    refs = nodes.view(np.uint32)[:, 6 * width:7 * width]
    order, tris, stack = [], 0, [0]
    while stack:
        r = stack.pop()
        if r & LEAF:
            assert ((r & 0x7fffffff) >> 3) == tris
            tris += (r & 7) + 1
            continue
        order.append(r)
        stack.extend(int(c) for c in refs[r][::-1] if c != EMPTY)
    assert order == list(range(len(nodes)))
    assert tris == nt


def _scales(nt):
    """Triangles over six magnitudes: the splits peel off small shares, so the
    tree is deeper than the levels that are launched without a look at it."""
    rng = np.random.default_rng(nt)
    V = rng.uniform(-1, 1, size=(nt, 1, 3)) + rng.uniform(-0.15, 0.15, size=(nt, 3, 3))
    V = V * 10.0 ** rng.uniform(-6, 0, size=(nt, 1, 1))
    return V.reshape(-1, 3).astype(np.float32), np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.gpu
def test_deep_tree_rebuilt_in_a_graph(gpu_ctx):
    from j3d_gb300 import Batch, Canvas, Matcap, Mesh, Scene, camera_for_vfov
    V, T = _scales(9000)
    built = Mesh(gpu_ctx, V, T, 1, width=2).nodes()
    mesh = Mesh(gpu_ctx, V, T, 1, width=2, rebuildable=True)
    assert np.array_equal(mesh.nodes().view(np.uint32), built.view(np.uint32))
    sc = Scene()
    sc.add_object(mesh, db_id=1)
    sc.prepare_scene()
    sc.unzoom()
    cv = Canvas(gpu_ctx, 64, 48)
    cv.set_camera(camera_for_vfov(60.0))
    cv.set_background_color()
    g = Batch(gpu_ctx, [(cv, sc, Matcap.make(gpu_ctx, 0))], rebuild=True)
    for _ in range(2):
        g.launch()
    gpu_ctx.synchronize()
    assert np.array_equal(mesh.nodes().view(np.uint32), built.view(np.uint32))
    g.close()
    cv.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nu,nv", [(1000, 500), (1100, 500)])  # the nodes' bound: 256 and 282 MB
def test_nodes_made_in_place(gpu_ctx, nu, nv):
    from j3d_gb300 import Mesh, workloads as W
    V, T = W.torus(nu, nv)
    a = Mesh(gpu_ctx, V, T, width=8)
    b = Mesh(gpu_ctx, V, T, width=8, rebuildable=True)
    assert np.array_equal(a.nodes().view(np.uint32), b.nodes().view(np.uint32))
