"""The FP64 sketch cut into ranges of the points j (partial products in slabs, summed in order): whole and ragged last
ranges, each tile width, a padded result, no labels.  Tolerance: an n-long FP64 sum in another order and the kernel
values' own error, 1e-12 relative, as for the uncut one."""
import numpy as np
import pytest

from oracle import oracle as O
from util import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,d,l,pad,labels", [
    (64, 512, 8, 16, 0, True), (65, 513, 16, 17, 3, True), (1, 1040, 7, 138, 1, False), (300, 2065, 33, 2, 0, False),
    (700, 1601, 16, 144, 5, True), (129, 1535, 24, 300, 0, True)])
def test_rbf_sketch_f64_ranges(gpu_ctx, m, n, d, l, pad, labels):
    import torch
    g = np.random.default_rng(m)
    Xi, Xj = (0.5 * g.standard_normal((k, d)).astype(np.float32) for k in (m, n))
    yi, yj = (np.where(g.random(k) < 0.5, -1.0, 1.0).astype(np.float32) for k in (m, n))
    Om = g.standard_normal((n, l))
    gamma = 1.0 / d
    ref = O.sketch(Xi, Xj, yi if labels else np.ones(m), yj if labels else np.ones(n), Om, gamma)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (Xi, Xj, yi, yj, Om.T)]
    Y = torch.full((l, m + pad), 7.0, dtype=torch.float64, device="cuda")
    gpu_ctx.rbf_sketch_f64(m, n, d, l, t[0].data_ptr(), d, t[1].data_ptr(), d, t[2].data_ptr() if labels else None,
                           t[3].data_ptr() if labels else None, t[4].data_ptr(), n, Y.data_ptr(), m + pad, gamma)
    gpu_ctx.sync()
    got = Y.cpu().numpy()
    assert rel_fro(got[:, :m].T, ref) <= 1e-12
    assert np.all(got[:, m:] == 7.0)
