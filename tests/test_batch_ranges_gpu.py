"""Batched sketches of problems that alone are cut into ranges of the points j: bit for bit the single launches' results
whether the batch is small (ranges as work items, partial sums in slabs) or fills the GPU (ranges walked by their row
block), alone or beside problems of one range, with labels that are not +-1."""
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


def test_more_problems_than_a_grid_dimension(gpu_ctx):
    import torch
    from darray_optimizer_b200._lib import SketchJob
    n, d, l, count = 257, 2, 1, 65600
    X, Om = torch.rand(n, d, device="cuda"), torch.randn(l, n, device="cuda")
    Y = torch.full((count, n), 7.0, device="cuda")
    jobs = [SketchJob(n, n, d, l, ptr(X), d, ptr(X), d, None, None, ptr(Om), n, Y.data_ptr() + 4 * n * k, n, 0.5, 0, 0, 0)
            for k in range(count)]
    gpu_ctx.rbf_sketch_batched(jobs)
    one = torch.empty(n, device="cuda")
    gpu_ctx.rbf_sketch(n, n, d, l, ptr(X), d, ptr(X), d, 0, None, None, ptr(Om), n, ptr(one), n, 0.5)
    gpu_ctx.sync()
    assert torch.equal(Y, one.expand(count, n))
