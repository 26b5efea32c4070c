"""The FP64 sketch's scratch stays bounded where ranges of the points j would gain a part of a wave: the blocked test matrix
and at most 128 MB of partial products, with the result of plain FP64 sums."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,l", [(24296, 8, 528), (30011, 8, 144)])
def test_scratch_and_result(n, d, l):
    import torch
    from darray_optimizer_b200._lib import Context
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.rand(n, d, device="cuda", generator=g)
    Om = torch.randn(l, n, dtype=torch.float64, device="cuda", generator=g)
    Y = torch.empty(l, n, dtype=torch.float64, device="cuda")
    ctx = Context(0, torch.cuda.current_stream().cuda_stream)

    def call(m):
        ctx.rbf_sketch_f64(m, m, d, l, X.data_ptr(), d, X.data_ptr(), d, None, None, Om.data_ptr(), n, Y.data_ptr(), n, 0.5)
        ctx.sync()

    try:
        call(64)
        before = torch.cuda.mem_get_info()[0]
        call(n)
        assert before - torch.cuda.mem_get_info()[0] <= 8 * n * (l + 160) + (128 << 20) + (8 << 20)  # l padded to its tiles
        rows = torch.randperm(n, generator=g, device="cuda")[:256]
        P = X.double()
        K = torch.exp(-0.5 * torch.cdist(P[rows], P, compute_mode="donot_use_mm_for_euclid_dist") ** 2)
        ref = Om @ K.T
        # the tolerance of tests/test_rbf64_split_gpu.py
        assert float((Y[:, rows] - ref).norm() / ref.norm()) <= 1e-12
    finally:
        ctx.close()
