"""The pipelined FP64 tensor-core products (csrc/dmm64.cuh) behind gemm, gemm_tn, trsm_lutn, gram_weighted,
rbf_block_f64 and cholqr2, at the edges of their tiles: 16-row strips, 128-row and 32..88-column tiles, 16-long stages,
32-wide inverse blocks and shorter last pairs, operands that are not 16-byte aligned.

Tolerances: a p-long FP64 product sum differs from another summation order's by at most p u sum |a b|; 4 p u (2^-53)
of the absolute products is allowed.  Triangular solves: 8 l u cond(R), R well conditioned by construction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def dev(a, ld=None):
    """Column-major device copy with leading dimension ld (extra rows NaN); returns (tensor, ld)."""
    import torch
    m, n = a.shape
    ld = ld or m
    buf = np.full((n, ld), np.nan, a.dtype)
    buf[:, :m] = a.T
    return torch.from_numpy(buf).cuda(), ld


def host(t, m):
    return t.cpu().numpy()[:, :m].T


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N")])
@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (129, 33, 17, 1), (16, 88, 16, 0), (300, 89, 31, 3), (127, 72, 64, 2),
                                       (500, 177, 5, 1), (128, 528, 200, 0)])
def test_gemm_tile_edges(gpu_ctx, ta, tb, m, n, k, pad):
    g = np.random.default_rng(m * 31 + n)
    A = g.standard_normal((k, m) if ta == "T" else (m, k))
    B = g.standard_normal((n, k) if tb == "T" else (k, n))
    C = g.standard_normal((m, n))
    dA, lda = dev(A, A.shape[0] + pad)
    dB, ldb = dev(B, B.shape[0] + pad)
    dC, ldc = dev(C, m + pad)
    gpu_ctx.gemm(ta, tb, m, n, k, 1.5, dA.data_ptr(), lda, dB.data_ptr(), ldb, -0.5, dC.data_ptr(), ldc)
    gpu_ctx.sync()
    opA, opB = (A.T if ta == "T" else A), (B.T if tb == "T" else B)
    bound = 4 * (k + 2) * U * (1.5 * np.abs(opA) @ np.abs(opB) + 0.5 * np.abs(C))
    assert np.all(np.abs(host(dC, m) - (1.5 * opA @ opB - 0.5 * C)) <= bound)


@pytest.mark.parametrize("n,r,pad", [(1, 1, 0), (63, 5, 1), (1000, 88, 0), (4097, 138, 1), (777, 272, 0), (2500, 529, 2)])
@pytest.mark.parametrize("weighted", [False, True])
def test_gram_upper_edges(gpu_ctx, n, r, pad, weighted):
    import torch
    g = np.random.default_rng(n + r)
    Z = g.standard_normal((n, r))
    w = np.exp(g.uniform(-3, 3, n))
    dZ, ldz = dev(Z, n + pad)
    dw = torch.from_numpy(w).cuda()
    dM = torch.full((r, r), 7.0, dtype=torch.float64, device="cuda")
    gpu_ctx.gram_weighted(n, r, dZ.data_ptr(), ldz, dw.data_ptr() if weighted else None, dM.data_ptr(), r, 0)
    gpu_ctx.sync()
    ww = w if weighted else np.ones(n)
    M = host(dM, r)
    up = np.triu(np.ones((r, r), bool))
    bound = 4 * (n + 2) * U * (np.abs(Z).T * ww) @ np.abs(Z)
    assert np.all((np.abs(M - (Z.T * ww) @ Z) <= bound)[up])
    assert np.all(M[~up] == 7.0)  # the strictly lower part is not touched


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 64, 65, 95, 96, 97, 129, 191, 255, 257, 321, 545])
def test_trsm_inverse_block_edges(gpu_ctx, m):
    g = np.random.default_rng(m)
    R = np.triu(g.standard_normal((m, m))) / np.sqrt(m) + 2.0 * np.eye(m)
    B = g.standard_normal((m, 9))
    dR, ldr = dev(np.where(np.triu(np.ones((m, m), bool)), R, np.nan), m + m % 3)
    dB, ldb = dev(B, m + 1)
    gpu_ctx.trsm_lutn(m, 9, dR.data_ptr(), ldr, dB.data_ptr(), ldb)
    want = np.linalg.solve(R.T, B)
    tol = 8 * m * U * np.linalg.cond(R) * np.linalg.norm(want)
    assert np.linalg.norm(host(dB, m) - want) <= tol


@pytest.mark.parametrize("m,n,d,ldx", [(1, 1, 1, 1), (129, 90, 3, 5), (300, 88, 64, 64), (257, 177, 17, 20), (64, 33, 256, 257)])
def test_rbf_block_f64_edges(gpu_ctx, m, n, d, ldx):
    import torch
    g = np.random.default_rng(m + n + d)
    X = np.full((m + n, ldx), np.nan, np.float32)
    X[:, :d] = g.standard_normal((m + n, d)).astype(np.float32)
    y = np.where(g.random(m + n) < 0.5, 1.0, -1.0).astype(np.float32)
    gamma = 0.7 / d
    dX, dy = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    K = torch.full((n, m + 1), 7.0, dtype=torch.float64, device="cuda")
    gpu_ctx.rbf_block_f64(m, n, d, dX.data_ptr(), ldx, dX[m:].data_ptr(), ldx, dy.data_ptr(), dy[m:].data_ptr(),
                          K.data_ptr(), m + 1, gamma)
    gpu_ctx.sync()
    A, Bx = X[:m, :d].astype(np.float64), X[m:, :d].astype(np.float64)
    D = np.maximum((A * A).sum(1)[:, None] + (Bx * Bx).sum(1)[None, :] - 2 * A @ Bx.T, 0)
    want = np.exp(-gamma * D) * y[:m, None] * y[None, m:]
    # the distance's rounding (d terms of up to |a|^2 + |b|^2 each way) scales exp by gamma; exp itself 2 ulp
    size = (A * A).sum(1)[:, None] + (Bx * Bx).sum(1)[None, :]
    got = K.cpu().numpy()
    assert np.all(np.abs(got[:, :m].T - want) <= 8 * (d + 4) * U * gamma * 2 * size + 8 * U)
    assert np.all(got[:, m] == 7.0)
