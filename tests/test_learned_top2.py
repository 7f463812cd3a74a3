"""The fused inference kernel's running top-2 where its groups can go wrong:
ties (the smaller cluster wins) and rows whose best logits come in every
group, in the first or in the last one. With all weights zero a row's logits
are the last layer's biases, small integers that bf16 holds exactly."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 257, 1000])
@pytest.mark.parametrize("pattern", ["rising", "falling", "ties", "all_equal", "last_two"])
def test_top2_of_the_biases(gpu_ctx, pattern, n):
    from j3d_gb300 import Mesh, workloads as W
    from j3d_gb300._ffi import RAY_DTYPE
    from j3d_gb300.learned import Learned, param_layout
    V, T = W.icosphere(5, W.SEED_BASE + 71)
    net = Learned(gpu_ctx, Mesh(gpu_ctx, V, T))
    K = net.n_clusters
    layout, total = param_layout()
    j = np.arange(4096)
    b = {"rising": j // 32, "falling": 128 - j // 32, "ties": (j * 37) % 8, "all_equal": 0 * j,
         "last_two": (j >= K - 2) * 3}[pattern].astype(np.float32)
    p = np.zeros(total, np.float32)
    p[layout[9][1]:layout[9][1] + 4096] = b
    net.set_params(p)
    rays = np.zeros(n, RAY_DTYPE)
    rng = np.random.default_rng(n)
    rays["orig"][:, :3] = rng.normal(size=(n, 3)) * 3
    rays["dir"][:, :3] = rng.normal(size=(n, 3))
    rays["orig"][:, 3], rays["t_far"] = 1, np.finfo(np.float32).max
    want = np.lexsort((j[:K], -b[:K]))[:2].astype(np.uint32)
    assert np.array_equal(net.predict(rays), np.tile(want, (n, 1)))
