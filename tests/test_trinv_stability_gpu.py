"""The triangular inverse by block doubling (csrc/la64.cu) on ill-conditioned factors: its right residual R X - I entry by
entry against |R| |X|, as column substitution keeps it.  trsm_lutn of the identity gives X^T; NaN below R's diagonal is
not read.

Tolerance: substitution gives |R X - I| <= n u |R| |X| (Higham, Accuracy and Stability, section 14.2); a corrected block
adds its own product's and correction's errors, 4 (n + 4) u in all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def factors(n):
    g = np.random.default_rng(n)
    x = np.sort(g.random(n))
    yield np.linalg.cholesky(np.exp(-5 * (x[:, None] - x) ** 2) + 1e-7 * np.eye(n)).T
    Q = np.linalg.qr(g.standard_normal((n, n)))[0]
    yield np.linalg.qr((Q * 10.0 ** -np.linspace(0, 8, n)) @ np.linalg.qr(g.standard_normal((n, n)))[0])[1]
    yield np.triu(g.standard_normal((n, n))) + 3 * np.sqrt(n) * np.eye(n)


@pytest.mark.parametrize("n,pad", [(31, 1), (33, 0), (64, 0), (97, 3), (138, 0), (321, 1), (528, 0), (1030, 2)])
def test_right_residual(gpu_ctx, n, pad):
    import torch
    for R in factors(n):
        buf = np.full((n, n + pad), np.nan)
        buf[:, :n] = np.where(np.tri(n, dtype=bool), R.T, np.nan)  # column j of R with NaN below the diagonal
        dR = torch.from_numpy(buf).cuda()
        dB = torch.eye(n, dtype=torch.float64, device="cuda")
        gpu_ctx.trsm_lutn(n, n, dR.data_ptr(), n + pad, dB.data_ptr(), n)
        X = dB.cpu().numpy()  # column j of R^-T as row j: R^-1
        assert np.all(np.tril(X, -1) == 0.0)
        E = np.abs((np.triu(R).astype(np.longdouble) @ X.astype(np.longdouble) - np.eye(n)).astype(float))
        assert np.all(E <= 4 * (n + 4) * U * (np.abs(np.triu(R)) @ np.abs(X)) + 1e-300)
