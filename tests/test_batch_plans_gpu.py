"""The two kinds of kernel pass of a batched solve (range finder and final pass) take plans of their own: shapes whose final
pass needs less shared memory than the others, which are launched after both plans exist."""
import numpy as np
import pytest

from darray_optimizer_b200 import datagen
from tests.util import dev, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("d,l", [(16, 160), (64, 176), (90, 144), (128, 112), (128, 272)])
def test_passes_of_different_plans(gpu_ctx, d, l, use_graph):
    import torch
    from darray_optimizer_b200._lib import SvmInstance
    n = 2048
    w = datagen.uniform_hyperplane(n=n, d=d, seed=d + l)
    Om = datagen.rng(l).standard_normal((l, n), dtype=np.float32)
    dX, dy, dOm = dev(w.X), dev(w.y), torch.from_numpy(Om).cuda()
    Z = torch.zeros((l, n), dtype=torch.float64, device="cuda")
    a = torch.zeros(n, dtype=torch.float64, device="cuda")
    inst = [SvmInstance(n, d, l, ptr(dX), d, ptr(dy), 0.5 / d, 1.0, ptr(dOm), n, ptr(Z), n, ptr(a), 0, 0, 0)]
    reps, brep = gpu_ctx.svm_solve_batched(inst, q=1, use_graph=use_graph, workers=1)
    assert brep.kernel_passes == 3
    assert reps[0].gap_barrier < 1e-6 and reps[0].gap_primal_dual < 1e-6
    rep1 = gpu_ctx.svm_solve(n, d, l, 1, ptr(dX), d, ptr(dy), ptr(dOm), n, 0.5 / d, 1.0, ptr(a), ptr(Z), n)
    assert abs(rep1.f - reps[0].f) <= 1e-7 * abs(rep1.f)  # as test_batch_gpu.py: the same algorithm, not the same bits
