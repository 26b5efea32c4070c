"""The int8 Gram that the mixed solves use (seven base-256 digits per value, csrc/gram_tc.cu) against an extended-precision
one, entry by entry: odd sizes and leading dimensions, several scaling chunks, column counts off the tiles, columns of a
wide range, wide weights, entries at the digits' largest values.

Bound of an entry (p, q): an entry of column p is held to 2^-56 2^e <= 2.01 x 2^-56 m_p (m_p the chunk's largest), the
dropped digit groups add up to less than 6.1 x 2^-56 2^(e_p + e_q) a row, and the FP64 sums over the splits to a few u."""
import numpy as np
import pytest

from darray_optimizer_b200._lib import DB200Error

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
CHUNK = 16384


def columns(kind, g, n, r):
    """(Z, w): w None or powers of four, so that sqrt(w) z is exact."""
    Z, w = g.standard_normal((n, r)), None
    if kind == "decades":
        Z *= 10.0 ** g.uniform(-6, 0, (n, r))
    elif kind == "spikes":
        Z *= 1e-6
        Z[g.integers(0, n, r), np.arange(r)] = g.uniform(1.0, 1.9, r)
    elif kind == "weights":
        w = 4.0 ** g.integers(-15, 16, n)
    elif kind == "largest":
        Z = np.where(Z < 0, -1.0, 1.0) * np.where(np.arange(r) % 2, 1.0, 1.0 - 2.0 ** -53)
    return Z, w


def exact(Z, w):
    X = (Z if w is None else np.sqrt(w)[:, None] * Z).astype(np.longdouble)
    return X, np.stack([(X * X[:, [q]]).sum(0) for q in range(X.shape[1])], axis=1)


def grams(ctx, Z, w, pad, slices=None):
    import torch
    n, r = Z.shape
    buf = np.full((r, n + pad), np.nan)
    buf[:, :n] = Z.T
    dZ, dM = torch.from_numpy(buf).cuda(), torch.full((r, r), 7.0, dtype=torch.float64, device="cuda")
    dw = torch.from_numpy(w).cuda() if w is not None else None
    wp = dw.data_ptr() if w is not None else None
    if slices is None:
        ctx.check(ctx.lib.db200_selftest_solver_gram(ctx.h, n, r, dZ.data_ptr(), n + pad, wp, dM.data_ptr(), r))
    else:
        ctx.gram_weighted(n, r, dZ.data_ptr(), n + pad, wp, dM.data_ptr(), r, slices)
    ctx.sync()
    return dM.cpu().numpy().T


@pytest.mark.parametrize("kind", ["gauss", "decades", "spikes", "weights", "largest"])
@pytest.mark.parametrize("n,r,pad", [(1, 1, 0), (777, 5, 1), (4097, 64, 0), (16385, 70, 3), (40011, 33, 1)])
def test_entries(gpu_ctx, n, r, pad, kind):
    Z, w = columns(kind, np.random.default_rng(n + r), n, r)
    X, ref = exact(Z, w)
    A = np.abs(X).astype(float)
    bound = 32 * U * (A.T @ A)
    for c in range(0, n, CHUNK):
        B = A[c:c + CHUNK]
        m = B.max(0)
        bound += 6.1 * 2.0 ** -56 * B.shape[0] * 4.05 * m[:, None] * m
        bound += 2.01 * 2.0 ** -56 * (m[:, None] * B.sum(0) + B.sum(0)[:, None] * m)
    up = np.triu(np.ones((r, r), bool))
    err = np.abs(grams(gpu_ctx, Z, w, pad) - ref).astype(float)
    assert np.all((err <= bound)[up])


@pytest.mark.parametrize("kind", ["decades", "spikes", "weights"])
def test_no_further_off_than_eight_base128_digits(gpu_ctx, kind):
    n, r = 20011, 48
    Z, w = columns(kind, np.random.default_rng(3), n, r)
    X, ref = exact(Z, w)
    s = np.sqrt(np.diag(ref)).astype(float)
    up = np.triu(np.ones((r, r), bool), 1)  # the truncated digits' bias adds up on the diagonal: compare beside it
    rms = [np.sqrt(np.mean(((grams(gpu_ctx, Z, w, 1, k) - ref).astype(float) / s[:, None] / s)[up] ** 2)) for k in (None, 8)]
    assert rms[0] <= rms[1]


@pytest.mark.parametrize("slices", [9, 255, 256])
def test_unknown_slice_counts_are_refused(gpu_ctx, slices):
    with pytest.raises(DB200Error):
        grams(gpu_ctx, np.ones((64, 2)), None, 0, slices)
