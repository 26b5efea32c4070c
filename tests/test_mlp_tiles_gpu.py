"""The leverage MLP's tiled products (csrc/landmarks.cu) at the edges of their 128 x 128 tiles, 16-long stages and
16-byte pieces, against an FP64 restatement with the network's bf16 roundings of weights and activations.

Tolerance: forward 5e-3 and gradients 2e-2 of the largest entry per layer, the ones of test_landmarks_gpu.py (a bf16
rounding that falls the other way moves an activation by 2^-8 of itself)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,inputs,width,hidden", [(1, 1, 1, 1), (127, 18, 128, 2), (129, 66, 136, 3), (300, 7, 33, 2),
                                                   (65, 130, 256, 1), (1000, 16, 8, 3)])
def test_mlp_tile_edges(gpu_ctx, m, inputs, width, hidden):
    import torch
    from darray_optimizer_b200._lib import Mlp
    net = Mlp(gpu_ctx, inputs, width, hidden, seed=m)
    g = np.random.default_rng(m + inputs)
    F = g.standard_normal((m, inputs)).astype(np.float32)
    t = g.standard_normal(m).astype(np.float32)
    dF, dt = torch.from_numpy(F).cuda(), torch.from_numpy(t).cuda()
    out = torch.empty(m, device="cuda")
    net.forward(m, dF.data_ptr(), out.data_ptr())
    grads = torch.empty(net.nparams, device="cuda")
    loss = net.gradients(m, dF.data_ptr(), dt.data_ptr(), grads.data_ptr())
    gpu_ctx.sync()
    params = net.get_params()
    want_out, want_loss, want = reference(params, F, t, inputs, width, hidden)
    scale = np.abs(want_out).max() + 1e-3
    assert np.abs(out.cpu().numpy() - want_out).max() <= 5e-3 * scale
    assert abs(loss - want_loss) <= 2e-2 * want_loss + 1e-6
    got = grads.cpu().numpy()
    for a, b in want:
        assert np.abs(got[a:a + b.size] - b).max() <= 2e-2 * (np.abs(b).max() + 1e-4)
    net.close()


def bf16(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).to(torch.bfloat16).float().numpy().astype(np.float64)


def reference(params, F, t, inputs, width, hidden):
    """Forward and backward in FP64 with the network's bf16 roundings."""
    sizes = [inputs] + [width] * hidden + [1]
    off, W, b, offs = 0, [], [], []
    for fi, fo in zip(sizes[:-1], sizes[1:]):
        W.append(bf16(params[off:off + fi * fo].reshape(fo, fi)))
        b.append(params[off + fi * fo:off + fi * fo + fo].astype(np.float64))
        offs.append((off, off + fi * fo))
        off += fi * fo + fo
    h = [bf16(F)]
    for k in range(hidden):
        h.append(bf16(np.maximum(h[-1] @ W[k].T + b[k], 0)))
    out = h[-1] @ W[-1][0] + b[-1][0]
    m = len(F)
    d = ((out - t) / m)[:, None]
    grads = []
    for k in range(hidden, -1, -1):
        grads += [(offs[k][0], (d.T @ h[k]).reshape(-1)), (offs[k][1], d.sum(0))]
        if k:
            d = (d @ W[k]) * (h[k] > 0)
    return out, 0.5 * np.mean((out - t) ** 2), grads
