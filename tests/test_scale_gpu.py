"""The scale of a point set (its largest |x|) where one CTA finds it and where several do: sets of 32768 values and one
row more, strided rows on both sides of 256, the largest value first or last.  A wrong scale overflows fp16 or loses
the points' lo parts.  Tolerance: the split-fp16 kernel block's 2e-5 of the other kernel-block tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,ld", [(1, 1, 1), (1024, 32, 32), (1025, 32, 32), (255, 100, 104), (256, 100, 101),
                                    (257, 100, 104)])
@pytest.mark.parametrize("last", [False, True])
def test_scale(gpu_ctx, n, d, ld, last):
    import torch
    from darray_optimizer_b200 import _lib
    g = np.random.default_rng(n)
    X = (1e-3 * g.standard_normal((n, ld))).astype(np.float32)
    X[-1 if last else 0, d - 1 if last else 0] = 3.0e4
    y = torch.ones(n, device="cuda")
    dX, K = torch.from_numpy(X).cuda(), torch.zeros((n, n), device="cuda")
    gamma = 1e-9
    gpu_ctx.rbf_block(n, n, d, dX.data_ptr(), ld, dX.data_ptr(), ld, _lib.POINT_MAJOR, y.data_ptr(), y.data_ptr(),
                      K.data_ptr(), n, gamma)
    gpu_ctx.sync()
    Z = X[:, :d].astype(np.float64)
    s = (Z * Z).sum(1)
    ref = np.exp(-gamma * np.maximum(s[:, None] + s[None, :] - 2 * Z @ Z.T, 0.0))
    got = K.cpu().numpy()
    assert np.all(np.isfinite(got)) and np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)
