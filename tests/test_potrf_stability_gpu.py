"""Backward stability of the FP64 Cholesky (csrc/potrf64.cuh: diagonal blocks of 16, two pivots a step) where neighbouring
columns are nearly collinear, points repeat, or the entries' range is wide: the one-launch factor (n <= 544), the blocked
one (n = 700 and block sizes below 64).

Tolerance: Cholesky in floating point gives |A - R^T R|(i, j) <= (n + 1) u sqrt(a_ii a_jj) (Higham, Accuracy and
Stability, thm 10.3 with |R^T||R| <= sqrt(a_ii a_jj)); eight times that leaves room for the blocks' corrected inverses and
for the product that forms R^T R here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
PATHS = [(3, 64), (16, 64), (64, 64), (138, 64), (528, 64), (700, 64), (138, 32), (90, 17)]


def check(ctx, A, nb):
    import torch
    n = A.shape[0]
    A = np.triu(A) + np.triu(A, 1).T
    np.linalg.cholesky(A)  # positive definite to working precision
    dA = torch.from_numpy(A).cuda()
    ctx.potrf(n, dA.data_ptr(), n, nb)
    ctx.sync()
    R = dA.cpu().numpy().T
    s = 1.0 / np.sqrt(np.diag(A))
    E = (R * s).T @ (R * s) - A * s[:, None] * s
    assert np.all(np.tril(R, -1) == 0.0)
    assert np.abs(E).max() <= 8 * (n + 1) * U


@pytest.mark.parametrize("noise", [1e-3, 1e-5, 1e-6])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n,nb", PATHS)
def test_nearly_collinear_neighbours(gpu_ctx, n, nb, off, noise):
    g = np.random.default_rng(n + nb + off)
    G = g.standard_normal((4 * n, n))
    cols = np.arange(off, n - 1, 6)
    G[:, cols + 1] = G[:, cols] + noise * g.standard_normal((4 * n, cols.size))
    check(gpu_ctx, G.T @ G, nb)


@pytest.mark.parametrize("nu", [1e-7, 1e-11])
@pytest.mark.parametrize("n,nb", PATHS)
def test_repeated_points_and_sorted_line(gpu_ctx, n, nb, nu):
    g = np.random.default_rng(n)
    P = np.repeat(g.random(((n + 1) // 2, 4)), 2, axis=0)[:n]  # every point twice
    D = ((P[:, None] - P) ** 2).sum(-1)
    check(gpu_ctx, np.exp(-D) + nu * np.eye(n), nb)
    x = np.sort(g.random(n))
    check(gpu_ctx, np.exp(-5 * (x[:, None] - x) ** 2) + nu * np.eye(n), nb)


@pytest.mark.parametrize("n,nb", PATHS)
def test_range_of_the_entries(gpu_ctx, n, nb):
    g = np.random.default_rng(n)
    B = g.standard_normal((n, 2 * n))
    A = B @ B.T / (2 * n) + 0.1 * np.eye(n)
    for e in (160, -160, 250, -250):
        check(gpu_ctx, A * 10.0 ** e, nb)
    s = 10.0 ** g.uniform(-120, 120, n)
    check(gpu_ctx, A * s[:, None] * s, nb)
    s = 10.0 ** np.linspace(9, -9, n)
    check(gpu_ctx, A * s[:, None] * s, nb)
