"""The barrier's kernels at the edges of their tiles: the paired triangular solve (blocks of 16, panels of 256), the passes
over Z (64-row blocks, two rows per lane, four columns per warp, scalar loads where an odd stride or base leaves 16-byte
alignment) and the base-256 int8 capacity matrix.

Tolerances.  Terms: an n-long and an r-long FP64 sum, 4 (n + r) u (u = 2^-53) of the absolute products.  Solve: the
capacity matrix's error u cond(H) cond(D) <= 1e-16 * 520 * 400 = 2e-11 for these inputs, 1e-10 allowed.  Mixed barrier: its
steps are refined to a relative residual of 1e-10; objectives within 1e-8, as for the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def dev_z(Z, ld, shift=0):
    """Column-major device copy with leading dimension ld, `shift` doubles after an aligned base; unused entries NaN."""
    import torch
    n, r = Z.shape
    buf = np.full(shift + ld * r, np.nan)
    for k in range(r):
        buf[shift + k * ld:shift + k * ld + n] = Z[:, k]
    t = torch.from_numpy(buf).cuda()
    return t, t.data_ptr() + 8 * shift


def dev(a, dtype=np.float64):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=dtype)).cuda()


@pytest.mark.parametrize("r,n,ld,shift", [
    (1, 1, 1, 0), (1, 130, 130, 0), (15, 300, 300, 1), (16, 301, 301, 0), (17, 301, 302, 0), (255, 600, 600, 0),
    (256, 603, 605, 0), (257, 640, 640, 0), (273, 700, 702, 1), (529, 1100, 1100, 0), (545, 1101, 1102, 0),
    (4095, 601, 601, 0), (4096, 600, 600, 0)])
def test_woodbury_solve_edges(gpu_ctx, r, n, ld, shift):
    import torch
    g = np.random.default_rng(r)
    Z = g.standard_normal((n, r)) / np.sqrt(r)
    diag = np.exp(g.uniform(-3, 3, n))
    b = g.standard_normal(n)
    dZ, pz = dev_z(Z, ld, shift)
    dd, db, dx = dev(diag), dev(b), torch.zeros(n, dtype=torch.float64, device="cuda")
    gpu_ctx.woodbury_solve(n, r, pz, ld, dd.data_ptr(), db.data_ptr(), dx.data_ptr())
    ref = np.linalg.solve(Z @ Z.T + np.diag(diag), b)
    assert np.linalg.norm(dx.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("n,r,ld,shift", [(1, 1, 1, 0), (63, 3, 64, 0), (64, 4, 64, 0), (65, 5, 66, 0), (1025, 9, 1025, 0),
                                          (2050, 31, 2050, 1), (2051, 33, 2052, 0)])
def test_terms_edges(gpu_ctx, n, r, ld, shift):
    import torch
    g = np.random.default_rng(n)
    Z, a, C, t = g.standard_normal((n, r)), g.uniform(0.1, 0.9, n), 1.0, 10.0
    dZ, pz = dev_z(Z, ld, shift)
    da = dev(a)
    gf, gp, gr, D = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(4))
    gpu_ctx.barrier_terms(n, r, pz, ld, da.data_ptr(), C, t, gf.data_ptr(), gp.data_ptr(), gr.data_ptr(), D.data_ptr())
    room = 4 * (n + r) * U * (np.abs(Z) @ (np.abs(Z).T @ a) + 1.0)
    assert np.all(np.abs(gf.cpu().numpy() - (Z @ (Z.T @ a) - 1.0)) <= room)


@pytest.mark.parametrize("n,r", [(257, 1), (1024, 63), (1025, 64), (2048, 65), (3001, 129)])
def test_mixed_barrier_matches_fp64(gpu_ctx, n, r):
    import torch
    g = np.random.default_rng(r)
    y = np.where(g.random(n) < 0.5, -1.0, 1.0)
    Z = g.standard_normal((n, r)) * np.exp(g.uniform(-3, 0, r)) / np.sqrt(r)
    dZ, pz = dev_z(Z, n)
    dy, f = dev(y, np.float32), []
    for precision in (0, 1):
        da = torch.zeros(n, dtype=torch.float64, device="cuda")
        rep = gpu_ctx.svm_barrier(n, r, pz, n, dy.data_ptr(), 1.0, da.data_ptr(),
                                  params=gpu_ctx.barrier_params(precision=precision))
        assert rep.status == 0 and rep.fallbacks == 0
        f.append(rep.f)
    assert abs(f[0] - f[1]) <= 1e-8 * abs(f[1])
