"""Work items cut into ranges of the points j (few row blocks), kernel blocks stored through TMA, and the packs, at the
sizes where they can go wrong: one row, one past a tile or a row block, ranges whose last one is short, outputs whose
leading dimension TMA cannot write, point matrices with gaps and odd strides.

Tolerances are those of the unsplit paths (test_rbf_gpu.py): 2e-3 / 3e-6 relative Frobenius for the single and the
promoted product, 2e-5 elementwise for the block."""
import numpy as np
import pytest

from oracle import oracle as O
from util import rel_fro

pytestmark = pytest.mark.gpu


def points(n, d, ld, layout, seed):
    """(host n x d, device buffer, ld) of points with NaN in the gaps."""
    import torch
    g = np.random.default_rng(seed)
    X = (0.6 * g.standard_normal((n, d))).astype(np.float32)
    rows, cols = (n, d) if layout == 0 else (d, n)
    buf = np.full((rows, ld), np.nan, np.float32)
    buf[:, :cols] = X if layout == 0 else X.T
    y = np.where(g.random(n) < 0.5, 1.0, -1.0).astype(np.float32)
    return X, torch.from_numpy(buf).cuda(), y, torch.from_numpy(y).cuda()


@pytest.mark.parametrize("product,tol", [(0, 2e-3), (3, 3e-6)])
@pytest.mark.parametrize("m,n,d,l,gap,layout", [(1, 1, 1, 1, 0, 0), (256, 129, 5, 17, 3, 0), (257, 1025, 33, 64, 0, 1),
                                                (100, 4000, 54, 272, 1, 1), (1025, 3001, 128, 144, 4, 0)])
def test_split_sketch_edges(gpu_ctx, m, n, d, l, gap, layout, product, tol):
    import torch
    ldi = (d if layout == 0 else m) + gap
    ldj = (d if layout == 0 else n) + gap
    Xi, dXi, yi, dyi = points(m, d, ldi, layout, m + n)
    Xj, dXj, yj, dyj = points(n, d, ldj, layout, m + n + 1)
    g = np.random.default_rng(l)
    Om = g.standard_normal((n, l)).astype(np.float32)
    dOm = torch.from_numpy(np.ascontiguousarray(Om.T)).cuda()
    Y = torch.full((l, m + 1), 7.0, device="cuda")
    gpu_ctx.rbf_sketch_ex(m, n, d, l, dXi.data_ptr(), ldi, dXj.data_ptr(), ldj, layout, dyi.data_ptr(), dyj.data_ptr(),
                          dOm.data_ptr(), n, Y.data_ptr(), m + 1, 1.0 / d, product)
    gpu_ctx.sync()
    got = Y.cpu().numpy()
    assert rel_fro(got[:, :m].T, O.sketch(Xi, Xj, yi, yj, Om, 1.0 / d)) <= tol
    assert np.all(got[:, m] == 7.0)


@pytest.mark.parametrize("m,n,d,ldk", [(1, 1, 1, 4), (31, 33, 8, 32), (257, 129, 17, 260), (300, 300, 40, 301),
                                       (1000, 2050, 128, 1000), (4, 600, 3, 4)])
@pytest.mark.parametrize("layout", [0, 1])
def test_block_stores(gpu_ctx, m, n, d, ldk, layout):
    import torch
    ldi, ldj = (d, d) if layout == 0 else (m, n)
    Xi, dXi, yi, dyi = points(m, d, ldi, layout, 3 * m + n)
    Xj, dXj, yj, dyj = points(n, d, ldj, layout, 3 * m + n + 1)
    K = torch.full((n + 2, ldk), 7.0, device="cuda")
    gpu_ctx.rbf_block(m, n, d, dXi.data_ptr(), ldi, dXj.data_ptr(), ldj, layout, dyi.data_ptr(), dyj.data_ptr(),
                      K.data_ptr(), ldk, 0.5 / d)
    gpu_ctx.sync()
    got = K.cpu().numpy()
    want = O.rbf_block(Xi, Xj, yi, yj, 0.5 / d)
    assert np.abs(got[:n, :m].T - want).max() <= 2e-5
    assert np.all(got[n:] == 7.0) and np.all(got[:, m:] == 7.0)  # nothing beside the block is written


@pytest.mark.parametrize("n,d,s,k", [(9, 3, 9, 8), (257, 16, 130, 1), (300, 64, 300, 8), (5000, 128, 2049, 5), (700, 7, 129, 8)])
def test_knn_ranges(gpu_ctx, n, d, s, k):
    import torch
    g = np.random.default_rng(n + s)
    X = g.standard_normal((n, d)).astype(np.float32)
    X[1] = X[0]  # coincident points are neighbours at distance 0
    ref = np.sort(g.choice(n, s, replace=False)).astype(np.int32)
    dX, dref = torch.from_numpy(X).cuda(), torch.from_numpy(ref).cuda()
    out = torch.empty(n, device="cuda")
    gpu_ctx.knn_distance(n, d, dX.data_ptr(), d, s, dref.data_ptr(), k, out.data_ptr())
    gpu_ctx.sync()
    D2 = ((X[:, None, :].astype(np.float64) - X[None, ref, :]) ** 2).sum(2)
    D2[np.arange(n)[:, None] == ref[None, :]] = np.inf
    kth = np.sort(D2, axis=1)[:, k - 1]
    # k = s with the point itself among the references leaves fewer than k neighbours: infinite on both sides
    got = out.cpu().numpy().astype(np.float64) ** 2
    fin = np.isfinite(kth)
    assert np.array_equal(np.isfinite(got), fin)
    scale = 2 * (X.astype(np.float64) ** 2).sum(1).max()
    assert np.abs(got[fin] - kth[fin]).max() <= 2e-6 * scale  # a few fp32 roundings of |x|^2 + |y|^2
