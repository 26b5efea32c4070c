"""Batched sketches of problems that alone are cut into ranges of the points j: bit for bit the single launches' results
whether the batch is small (ranges as work items, partial sums in slabs) or fills the GPU (ranges walked by their row
block), alone or beside problems of one range, with labels that are not +-1; and the memory such a batch takes."""
import numpy as np
import pytest

from tests.util import ptr

pytestmark = pytest.mark.gpu
FILL = [(1000, 16, 40), (2048, 64, 144), (4096, 128, 272), (600, 7, 330), (129, 3, 1), (3001, 100, 96)]


@pytest.mark.parametrize("copies,large", [(1, 0), (1, 2), (12, 0), (12, 2)])
def test_batch_equals_single_launches(gpu_ctx, copies, large):
    import torch
    from darray_optimizer_b200._lib import SketchJob
    g = torch.Generator(device="cuda").manual_seed(copies + large)
    jobs, keep = [], []
    for n, d, l in FILL * copies + [(6000, 32, 64), (9000, 128, 176)][:large]:
        X = torch.rand(n, d, device="cuda", generator=g)
        y = torch.randn(n, device="cuda", generator=g)
        Om = torch.randn(l, n, device="cuda", generator=g)
        Y = torch.full((l, n), 7.0, device="cuda")
        keep.append((n, d, l, X, y, Om, Y))
        jobs.append(SketchJob(n, n, d, l, ptr(X), d, ptr(X), d, ptr(y), ptr(y), ptr(Om), n, ptr(Y), n, 0.5 / d, 0, 0, 0))
    gpu_ctx.rbf_sketch_batched(jobs)
    for n, d, l, X, y, Om, Y in keep:
        one = torch.empty_like(Y)
        gpu_ctx.rbf_sketch(n, n, d, l, ptr(X), d, ptr(X), d, 0, ptr(y), ptr(y), ptr(Om), n, ptr(one), n, 0.5 / d)
        gpu_ctx.sync()
        assert torch.equal(one, Y)


def test_batch_memory_is_the_problems_own():
    """128 problems of 2048 points: the packed operands (about 140 MB) and at most 512 MB of partial sums."""
    import torch
    from darray_optimizer_b200._lib import Context, SketchJob
    n, d, l, count = 2048, 64, 144, 128
    X, Om = torch.rand(n, d, device="cuda"), torch.randn(l, n, device="cuda")
    Y = torch.empty(count, l, n, device="cuda")
    jobs = [SketchJob(n, n, d, l, ptr(X), d, ptr(X), d, None, None, ptr(Om), n, ptr(Y[k]), n, 0.5 / d, 0, 0, 0)
            for k in range(count)]
    ctx = Context(0, torch.cuda.current_stream().cuda_stream)
    try:
        ctx.rbf_sketch(256, 256, d, 16, ptr(X), d, ptr(X), d, 0, None, None, ptr(Om), n, ptr(Y), n, 0.5 / d)
        ctx.sync()
        before = torch.cuda.mem_get_info()[0]
        ctx.rbf_sketch_batched(jobs)
        ctx.sync()
        packed = count * (2 * n * d * 2 + n * 4 + l * n * 2)
        assert before - torch.cuda.mem_get_info()[0] <= 1.25 * (packed + (512 << 20)) + (4 << 20)
    finally:
        ctx.close()


def test_solve_groups_share_their_slabs():
    """64 instances whose ranges' partial sums take 20 MB or more each: the passes run in groups that share 512 MB of them, and
    the solves agree with single ones as tests/test_batch_gpu.py states."""
    import torch
    from darray_optimizer_b200 import datagen
    from darray_optimizer_b200._lib import Context, SvmInstance
    n, d, l, count = 6000, 64, 272, 64
    w = datagen.uniform_hyperplane(n=n, d=d, seed=5)
    X, y = torch.from_numpy(w.X).cuda(), torch.from_numpy(w.y).cuda()
    Om = torch.from_numpy(datagen.rng(6).standard_normal((l, n), dtype=np.float32)).cuda()
    Z = torch.zeros(count, l, n, dtype=torch.float64, device="cuda")
    a = torch.zeros(count, n, dtype=torch.float64, device="cuda")
    C = [0.5 + 0.125 * (k % 3) for k in range(count)]
    inst = [SvmInstance(n, d, l, ptr(X), d, ptr(y), 0.5 / d, C[k], ptr(Om), n, ptr(Z[k]), n, ptr(a[k]), 0, 0, 0)
            for k in range(count)]
    ctx = Context(0, torch.cuda.current_stream().cuda_stream)
    try:
        ctx.svm_solve_batched(inst[:1], q=1, use_graph=True, workers=1)
        ctx.sync()
        before = torch.cuda.mem_get_info()[0]
        reps, _ = ctx.svm_solve_batched(inst, q=1, use_graph=True, workers=1)
        ctx.sync()
        own = n * l * (4 + 4 + 8 + 4) + 2 * l * l * 8 + n * (4 * d + 8)  # outputs, factors, packed operands (bytes)
        assert before - torch.cuda.mem_get_info()[0] <= 1.25 * (count * own + (512 << 20)) + (4 << 20)
        for k in (0, 24, 25, 26, 50, 51, 63):
            one = ctx.svm_solve(n, d, l, 1, ptr(X), d, ptr(y), ptr(Om), n, 0.5 / d, C[k], ptr(a[0]), ptr(Z[0]), n)
            assert abs(one.f - reps[k].f) <= 1e-7 * abs(one.f)
    finally:
        ctx.close()


def test_more_problems_than_a_grid_dimension(gpu_ctx):
    import torch
    from darray_optimizer_b200._lib import SketchJob
    n, d, l, count = 520, 2, 1, 65600  # three row blocks, six ranges
    X, Om = torch.rand(n, d, device="cuda"), torch.randn(l, n, device="cuda")
    Y = torch.full((count, n), 7.0, device="cuda")
    jobs = [SketchJob(n, n, d, l, ptr(X), d, ptr(X), d, None, None, ptr(Om), n, Y.data_ptr() + 4 * n * k, n, 0.5, 0, 0, 0)
            for k in range(count)]
    gpu_ctx.rbf_sketch_batched(jobs)
    one = torch.empty(n, device="cuda")
    gpu_ctx.rbf_sketch(n, n, d, l, ptr(X), d, ptr(X), d, 0, None, None, ptr(Om), n, ptr(one), n, 0.5)
    gpu_ctx.sync()
    assert torch.equal(Y, one.expand(count, n))


@pytest.mark.parametrize("plan", [(1, 272, 1), (2, 144, 2), (3, 96, 2), (6, 48, 2)])
@pytest.mark.parametrize("n,copies", [(1500, 1), (2048, 1), (4096, 1), (2048, 24)])
def test_explicit_plans_keep_the_ranges(gpu_ctx, n, copies, plan):
    """An instance's tile plan (the autotuner's) does not change its ranges, so nor its bits."""
    import torch
    from darray_optimizer_b200._lib import SketchJob
    d, l = 64, 272
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.rand(n, d, device="cuda", generator=g)
    Om = torch.randn(l, n, device="cuda", generator=g)
    Y = torch.empty(copies, l, n, device="cuda")
    gpu_ctx.rbf_sketch_batched([SketchJob(n, n, d, l, ptr(X), d, ptr(X), d, None, None, ptr(Om), n, ptr(Y[k]), n, 0.5 / d,
                                          *plan) for k in range(copies)])
    one = torch.empty(l, n, device="cuda")
    gpu_ctx.rbf_sketch(n, n, d, l, ptr(X), d, ptr(X), d, 0, None, None, ptr(Om), n, ptr(one), n, 0.5 / d)
    gpu_ctx.sync()
    assert all(torch.equal(one, y) for y in Y)
