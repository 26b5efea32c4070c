"""The scale of a point set with gaps (features of a larger matrix): long rows are scanned in pieces of 1024, whichever piece
the largest value is in.  The result is bit for bit the contiguous set's, whose scan is one list."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 1), (1023, 3), (1024, 2), (1025, 1), (4097, 8), (32768, 1), (40000, 5), (3000, 128)])
@pytest.mark.parametrize("gap,off", [(1, 0), (4, 0), (4096, 1)])
def test_gapped_feature_major_equals_contiguous(gpu_ctx, n, d, gap, off):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + d)
    X = torch.rand(d, n, device="cuda", generator=g)
    Om = torch.randn(n, device="cuda", generator=g)
    for at in {0, n // 2, n - 1, min(n - 1, 1023), min(n - 1, 1024)}:
        X[d // 2] = X[d // 2].clamp(max=1.0)
        X[d // 2, at] = 37.5  # alone sets the scale
        big = torch.full((d * (n + gap) + off,), float("nan"), device="cuda")
        wide = big[off:].view(d, n + gap)
        wide[:, n:] = 1e30  # beside the set: must not set it
        wide[:, :n] = X
        out = []
        for p, ld in ((X, n), (wide, n + gap)):
            Y = torch.empty(n, device="cuda")
            gpu_ctx.rbf_sketch(n, n, d, 1, p.data_ptr(), ld, p.data_ptr(), ld, 1, None, None, Om.data_ptr(), n, Y.data_ptr(),
                               n, 1e-4)
            out.append(Y)
        gpu_ctx.sync()
        assert torch.equal(out[0], out[1])
