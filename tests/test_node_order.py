"""The wide nodes of a build stand in depth-first order (a node's subtree is
the range that follows it) and their leaves in the order of the triangles."""
import numpy as np
import pytest

LEAF, EMPTY = 0x80000000, 0xffffffff


@pytest.mark.gpu
@pytest.mark.parametrize("width,leaf", [(4, 2), (2, 1), (8, 8)])
@pytest.mark.parametrize("nt", [9, 64, 65, 959, 960, 961, 1921, 20011])
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
