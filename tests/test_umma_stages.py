"""The GEMM's shared-memory ring at the lengths of K where it can go wrong:
fewer chunks of 64 than its stages, exactly as many, one more, and many."""
import numpy as np
import pytest

from test_umma import _case, _run


@pytest.mark.gpu
@pytest.mark.parametrize("N", [128, 256, 512])
@pytest.mark.parametrize("K", [64, 128, 192, 256, 448, 1024])
@pytest.mark.parametrize("impl", [1, 0])
def test_gemm_at_ring_lengths(gpu_ctx, N, K, impl):
    A, Bt, ref, mag = _case(384, N, K, seed=N + K)
    C = _run(gpu_ctx, A, Bt, impl)
    assert np.isfinite(C).all()
    # fp32 accumulation of K exact products: every sum's error is below K 2^-24 of its terms' magnitudes
    assert (np.abs(C - ref) <= 2 * K * 2.0 ** -24 * mag + 1e-30).all()
