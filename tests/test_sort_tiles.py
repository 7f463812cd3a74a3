"""The builder's radix sort at the edges of its tiles (1024 keys below 300,000
triangles, 4096 from there): the leaves of an LBVH of one triangle each stand
in the order of the triangles' Morton codes, equal codes in input order."""
import numpy as np
import pytest

LEAF, EMPTY = 0x80000000, 0xffffffff
F = np.float32


def _spread(x):
    r = np.zeros(len(x), np.uint64)
    for b in range(16):
        r |= ((x >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("nt", [2, 1023, 1024, 1025, 4097, 299_999, 300_000, 303_104, 303_105])
def test_leaves_in_morton_order(gpu_ctx, nt):
    from j3d_gb300 import Mesh
    rng = np.random.default_rng(nt)
    c = rng.uniform(-1, 1, size=(nt, 1, 3))
    c[: nt // 8] = np.round(c[: nt // 8] * 2) / 2  # many equal codes
    tri = (c + rng.uniform(-0.01, 0.01, size=(nt, 3, 3))).astype(F)
    tri[: nt // 16] = tri[0]
    V = tri.reshape(-1, 3)
    mesh = Mesh(gpu_ctx, V, np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3), 1, "lbvh")
    lo, hi = tri.min(axis=1), tri.max(axis=1)
    blo, bhi = V.min(axis=0), V.max(axis=0)
    f = ((lo + hi) * F(0.5) - blo) / (bhi - blo) * F(65536)
    q = np.clip(f, F(0), F(65535)).astype(np.uint64)
    code = (_spread(q[:, 0]) << np.uint64(2)) | (_spread(q[:, 1]) << np.uint64(1)) | _spread(q[:, 2])
    order = np.argsort(code, kind="stable")
    nodes = mesh.nodes().reshape(mesh.info().n_nodes, 32)
    refs = nodes.view(np.uint32)[:, 24:28]
    n, s = np.nonzero((refs & LEAF != 0) & (refs != EMPTY))
    ref = refs[n, s]
    assert np.array_equal(ref & 7, np.zeros(nt, np.uint32))
    slot = (ref & 0x7fffffff) >> 3
    assert np.array_equal(np.sort(slot), np.arange(nt))
    planes = nodes[:, :24].reshape(-1, 6, 4)[n, :, s]
    want = np.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1], lo[:, 2], hi[:, 2]], axis=1)[order[slot]]
    assert np.array_equal(planes, want)
