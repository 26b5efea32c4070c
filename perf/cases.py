"""Performance cases of the kernel-SVM path: what a program that uses this library has it do, through the public
entry points (darray_optimizer_b200._lib.Context and Mlp), with the sizes of the repository's own workloads
(darray_optimizer_b200/datagen.py, batched.py, landmarks.py, bench.py) from the smallest call to the largest.

A case names a `kind` and its sizes.  `listed()` is the fixed list, `draw(rng)` one more case of the same ranges,
`prepare(case, seed)` the inputs on the GPU, `run(state)` one pass, `work(case)` the bytes and operations the pass
cannot do without, `exact(case, seed)` the same results in plain torch FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from darray_optimizer_b200 import _lib, datagen

_ctx = None


def context() -> _lib.Context:
    """The one library handle a program keeps, on torch's current stream."""
    global _ctx
    if _ctx is None:
        _ctx = _lib.Context(0, torch.cuda.current_stream().cuda_stream)
    return _ctx


def listed():
    return [
        # The smallest call: a kernel pass over a toy problem (the smoke test's shape); launches and host work count.
        dict(name="sketch_small", kind="sketch", data="gauss", m=1024, n=1024, d=32, l=64, layout=0, promoted=False),
        # The headline pass of the precision-form workload: Y = K Omega, single fp16 sketch product.
        dict(name="sketch_c2", kind="sketch", data="uniform", m=131072, n=131072, d=128, l=528, layout=0,
             promoted=False),
        # One rank's rows of a parity-grade kernel pass of the mixed solve (compensated product, 256-point chunks) at
        # a ragged size of the batched workload's range.
        dict(name="sketch_promoted_shard", kind="sketch", data="gauss", m=15005, n=30011, d=54, l=272, layout=0,
             promoted=True),
        # One materialised kernel block, the reference's rbf_kernel unit of work (feature-major points, 8192 x 8192).
        dict(name="kernel_block", kind="block", data="uniform", m=8192, n=8192, d=128, layout=1),
        # 8th-neighbour distances of the learned path's features, 16384 reference points.
        dict(name="knn_features", kind="knn", data="mixture", n=131072, d=64, s=16384, k=8),
        # The plain method in FP64 throughout, one whole solve: n = 4096, d = 32, rank 128 + 10, q = 1, C = 1.
        dict(name="solve_c1_fp64", kind="solve", data="gauss", n=4096, d=32, l=138, C=1.0),
        # Orthonormalisation of one kernel pass's output at the precision-form workload.
        dict(name="cholqr2_c2", kind="cholqr2", n=131072, l=528),
        # A dense Cholesky at the largest size the reference's own Cholesky benchmark runs on one rank.
        dict(name="potrf_4096", kind="potrf", n=4096),
        # The barrier solve (mixed precision) on a rank-528 factor of the precision-form workload.
        dict(name="barrier_c2", kind="barrier", data="uniform", n=131072, d=128, r=528, C=10.0),
        # The Nystrom factor on given landmarks, FP64 columns, as the learned solve takes it.
        dict(name="landmark_factor", kind="landmark", data="mixture", n=131072, d=64, r=1024),
        # One training step's forward and backward pass of the leverage MLP (66 -> 256 x 3 -> 1) over one instance.
        dict(name="mlp_gradients", kind="mlp", m=16384, inputs=66, width=256, hidden=3),
        # LIBSVM text of dense points already in device memory, parsed into float X and y.
        dict(name="libsvm_dense", kind="libsvm", n=16384, d=128, sparse=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sketch", "sketch", "block", "knn", "solve", "cholqr2", "potrf", "barrier", "landmark", "mlp",
                       "libsvm"])
    data = rng.choice(["gauss", "uniform"])
    if kind == "sketch":
        n = _log(rng, 1024, 131072)
        m = n if rng.random() < 0.6 else max(256, n // rng.randint(2, 8))
        return dict(kind=kind, data=data, m=m, n=n, d=_log(rng, 8, 128), l=_log(rng, 16, 528),
                    layout=rng.choice([0, 0, 1]), promoted=rng.random() < 0.5)
    if kind == "block":
        return dict(kind=kind, data=data, m=_log(rng, 256, 16384), n=_log(rng, 256, 16384), d=_log(rng, 8, 128),
                    layout=rng.choice([0, 1]))
    if kind == "knn":
        n = _log(rng, 4096, 131072)
        return dict(kind=kind, data="mixture", n=n, d=_log(rng, 8, 128), s=min(n, _log(rng, 1024, 16384)), k=8)
    if kind == "solve":
        n = _log(rng, 1024, 6000)
        return dict(kind=kind, data="gauss", n=n, d=_log(rng, 16, 64), l=_log(rng, 32, 144), C=1.0)
    if kind == "cholqr2":
        n = _log(rng, 4096, 131072)
        return dict(kind=kind, n=n, l=min(n // 8, _log(rng, 32, 528)))
    if kind == "potrf":
        return dict(kind=kind, n=_log(rng, 64, 6000))
    if kind == "barrier":
        n = _log(rng, 2048, 65536)
        return dict(kind=kind, data=data, n=n, d=rng.choice([16, 64, 128]), r=_log(rng, 48, 272),
                    C=2.0 ** rng.randint(-2, 3))
    if kind == "landmark":
        return dict(kind=kind, data="mixture", n=_log(rng, 8192, 131072), d=_log(rng, 16, 128), r=_log(rng, 128, 1024))
    if kind == "mlp":
        return dict(kind=kind, m=_log(rng, 1024, 16384), inputs=rng.choice([18, 66, 130]), width=256, hidden=3)
    return dict(kind=kind, n=_log(rng, 512, 16384), d=_log(rng, 8, 128), sparse=rng.random() < 0.4)


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _uniform(g, *shape, dtype=torch.float32):
    return torch.rand(*shape, generator=g, device="cuda", dtype=dtype)


def _points(data, n, d, seed):
    """(X n x d float32 point-major, y +-1 float32): the generators of darray_optimizer_b200/datagen.py on the GPU."""
    g = _gen(seed)
    if data == "gauss":  # two isotropic Gaussians N(+-0.5, I)
        y = torch.where(_uniform(g, n) < 0.5, 1.0, -1.0)
        return _normal(g, n, d) + 0.5 * y[:, None], y
    if data == "uniform":  # uniform cube, hyperplane labels, 5 % flipped
        X = _uniform(g, n, d)
        s = (X - X.mean(0)).double() @ _normal(g, d, dtype=torch.float64)
        y = torch.where(s >= 0, 1.0, -1.0)
        return X, torch.where(_uniform(g, n) < 0.05, -y, y)
    # 32 anisotropic Gaussians: means N(0, 16), random rotations, per-axis scales log-uniform in [0.1, 3]
    comps = 32
    means = 4.0 * _normal(g, comps, d)
    rot = torch.linalg.qr(_normal(g, comps, d, d))[0]
    scales = torch.exp(math.log(0.1) + (math.log(3.0) - math.log(0.1)) * _uniform(g, comps, d))
    labels = torch.where(_uniform(g, comps) < 0.5, 1.0, -1.0)
    comp = torch.randint(comps, (n,), generator=g, device="cuda")
    z = _normal(g, n, d) * scales[comp]
    X = torch.empty(n, d, device="cuda")
    for c in range(comps):
        rows = (comp == c).nonzero()[:, 0]
        X[rows] = means[c] + z[rows] @ rot[c].T
    return X, labels[comp]


def _gamma(case):
    return (0.5 if case["data"] == "uniform" else 1.0) / case["d"]


def _landmarks(n, r, seed):
    return torch.randperm(n, generator=_gen(seed + 17), device="cuda")[:r].sort()[0].to(torch.int32)


def _kernel64(A, B, ya, yb, gamma):
    """diag(ya) exp(-gamma |a - b|^2) diag(yb) in FP64."""
    A, B = A.double(), B.double()
    D = (A * A).sum(1)[:, None] + (B * B).sum(1)[None, :] - 2.0 * (A @ B.T)
    K = torch.exp_(D.clamp_(min=0.0).mul_(-gamma))
    return K.mul_(ya.double()[:, None]).mul_(yb.double()[None, :])


def _nystrom64(X, y, gamma, idx):
    """Z (n x r FP64) = C R^-1, R^T R = C(L, :) + nu I, nu = 1e-7 trace / r."""
    L = idx.long()
    C = _kernel64(X, X[L], y, y[L], gamma)
    W = C[L]
    W = 0.5 * (W + W.T)
    W += torch.eye(len(L), device="cuda", dtype=torch.float64) * (1e-7 * W.trace() / len(L))
    low = torch.linalg.cholesky(W)
    return torch.linalg.solve_triangular(low, C.T, upper=False).T


def _spd(n, seed):
    """I + G^T G / n: the capacity matrix's form."""
    G = _normal(_gen(seed), 2 * n, n, dtype=torch.float64)
    A = G.T @ G
    return A.div_(n).add_(torch.eye(n, device="cuda", dtype=torch.float64))


def _tall(n, l, seed):
    """l x n storage of an n x l FP64 sketch: Gaussian columns of decaying size plus one common direction."""
    g = _gen(seed)
    Y = _normal(g, l, n, dtype=torch.float64)
    Y *= torch.logspace(0, -2, l, device="cuda", dtype=torch.float64)[:, None]
    return Y + _normal(g, l, 1, dtype=torch.float64) * _normal(g, 1, n, dtype=torch.float64)


def _libsvm(case, seed):
    """(text bytes, X float64 n x d, y float64) of LIBSVM lines: dense six-decimal values, or sparse 0/1 features."""
    g = datagen.rng(seed)
    n, d = case["n"], case["d"]
    y = np.where(g.random(n) < 0.5, 1.0, -1.0)
    if case["sparse"]:
        X = (g.random((n, d)) < 0.11).astype(np.float64)
        lines = [("+1" if y[i] > 0 else "-1") + "".join(f" {k + 1}:1" for k in np.flatnonzero(X[i])) for i in range(n)]
        return ("\n".join(lines) + "\n").encode(), X, y
    X = np.rint(g.random((n, d)) * 1e6) / 1e6
    return datagen.libsvm_text(X, y), X, y


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "ctx": context()}
    if kind in ("sketch", "block"):
        m, n, d = case["m"], case["n"], case["d"]
        X, y = _points(case["data"], max(m, n), d, seed)
        X, y = X[:n], y[:n]
        if m > n:  # rows are another set than the columns
            Xi, yi = _points(case["data"], m, d, seed + 1)
        else:
            Xi, yi = X[:m], y[:m]  # the first rows of the same points (all of them when m = n)
        if case["layout"] == 1:
            same = m == n
            X = X.T.contiguous()
            Xi = X if same else Xi.T.contiguous()
        st.update(X=X, y=y.contiguous(), Xi=Xi, yi=yi.contiguous())
        if kind == "sketch":
            st["Om"] = _normal(_gen(seed + 2), case["l"], n)          # n x l column major
            st["Y"] = torch.empty(case["l"], m, device="cuda")        # m x l column major
        else:
            st["K"] = torch.empty(n, m, device="cuda")                # m x n column major
    elif kind == "knn":
        st["X"], _ = _points(case["data"], case["n"], case["d"], seed)
        st["ref"] = _landmarks(case["n"], case["s"], seed)
        st["out"] = torch.empty(case["n"], device="cuda")
    elif kind == "solve":
        n, l = case["n"], case["l"]
        st["X"], st["y"] = _points(case["data"], n, case["d"], seed)
        st["Om"] = _normal(_gen(seed + 2), l, n)
        st["a"] = torch.empty(n, device="cuda", dtype=torch.float64)
        st["Z"] = torch.empty(l, n, device="cuda", dtype=torch.float64)
        st["params"] = _lib.Context.barrier_params(precision=_lib.FP64)
    elif kind == "cholqr2":
        st["Y"] = _tall(case["n"], case["l"], seed)
        st["Q"] = torch.empty_like(st["Y"])
        st["R"] = torch.empty(case["l"], case["l"], device="cuda", dtype=torch.float64)
    elif kind == "potrf":
        st["A"] = _spd(case["n"], seed)
        st["R"] = torch.empty_like(st["A"])
    elif kind == "barrier":
        n, r = case["n"], case["r"]
        X, y = _points(case["data"], n, case["d"], seed)
        st["Z"] = _nystrom64(X, y, _gamma(case), _landmarks(n, r, seed)).T.contiguous()
        st["y"] = y
        st["a"] = torch.empty(n, device="cuda", dtype=torch.float64)
    elif kind == "landmark":
        n, r = case["n"], case["r"]
        st["X"], st["y"] = _points(case["data"], n, case["d"], seed)
        st["idx"] = _landmarks(n, r, seed)
        st["Z"] = torch.empty(r, n, device="cuda", dtype=torch.float64)
    elif kind == "mlp":
        st["net"] = _lib.Mlp(st["ctx"], case["inputs"], case["width"], case["hidden"], seed)
        st["F"], st["t"] = _training(case, seed)
        st["grads"] = torch.empty(st["net"].nparams, device="cuda")
    else:
        text, _, _ = _libsvm(case, seed)
        st["text"] = torch.from_numpy(np.frombuffer(text, np.uint8).copy()).cuda()
        st["X"] = torch.zeros(case["n"], case["d"], device="cuda")
        st["y"] = torch.zeros(case["n"], device="cuda")
    return st


def _training(case, seed):
    """Standardised features and centred log-leverage targets."""
    g = _gen(seed)
    F = _normal(g, case["m"], case["inputs"])
    w = _normal(g, case["inputs"]) / math.sqrt(case["inputs"])
    return F, torch.tanh(F @ w) + 0.1 * _normal(g, case["m"])


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind in ("sketch", "block"):
        m, n, d = case["m"], case["n"], case["d"]
        X, Xi, y, yi = st["X"], st["Xi"], st["y"], st["yi"]
        lx, lxi = X.stride(0), Xi.stride(0)
        if kind == "block":
            ctx.rbf_block(m, n, d, Xi.data_ptr(), lxi, X.data_ptr(), lx, case["layout"], yi.data_ptr(), y.data_ptr(),
                          st["K"].data_ptr(), m, _gamma(case))
            return st["K"]
        if case["promoted"]:
            ctx.rbf_sketch_ex(m, n, d, case["l"], Xi.data_ptr(), lxi, X.data_ptr(), lx, case["layout"], yi.data_ptr(),
                              y.data_ptr(), st["Om"].data_ptr(), n, st["Y"].data_ptr(), m, _gamma(case),
                              _lib.SKETCH_COMPENSATED_PROMOTED)
        else:
            ctx.rbf_sketch(m, n, d, case["l"], Xi.data_ptr(), lxi, X.data_ptr(), lx, case["layout"], yi.data_ptr(),
                           y.data_ptr(), st["Om"].data_ptr(), n, st["Y"].data_ptr(), m, _gamma(case))
        return st["Y"]
    if kind == "knn":
        ctx.knn_distance(case["n"], case["d"], st["X"].data_ptr(), case["d"], case["s"], st["ref"].data_ptr(),
                         case["k"], st["out"].data_ptr())
        return st["out"]
    if kind == "solve":
        n, l = case["n"], case["l"]
        rep = ctx.svm_solve(n, case["d"], l, 1, st["X"].data_ptr(), case["d"], st["y"].data_ptr(),
                            st["Om"].data_ptr(), n, _gamma(case), case["C"], st["a"].data_ptr(), st["Z"].data_ptr(),
                            n, st["params"])
        return {"a": st["a"], "Z": st["Z"], "f": rep.f}
    if kind == "cholqr2":
        st["Q"].copy_(st["Y"])
        ctx.cholqr2(case["n"], case["l"], st["Q"].data_ptr(), case["n"], st["R"].data_ptr(), case["l"])
        return {"Q": st["Q"], "R": st["R"]}
    if kind == "potrf":
        st["R"].copy_(st["A"])
        ctx.potrf(case["n"], st["R"].data_ptr(), case["n"])
        return st["R"]
    if kind == "barrier":
        rep = ctx.svm_barrier(case["n"], case["r"], st["Z"].data_ptr(), case["n"], st["y"].data_ptr(), case["C"],
                              st["a"].data_ptr())
        return {"a": st["a"], "f": rep.f}
    if kind == "landmark":
        nu = ctx.landmark_factor(case["n"], case["d"], st["X"].data_ptr(), case["d"], st["y"].data_ptr(), _gamma(case),
                                 case["r"], st["idx"].data_ptr(), st["Z"].data_ptr(), case["n"], _lib.FP64)
        return {"Z": st["Z"], "nu": nu}
    if kind == "mlp":
        loss = st["net"].gradients(case["m"], st["F"].data_ptr(), st["t"].data_ptr(), st["grads"].data_ptr())
        return {"grads": st["grads"], "loss": loss}
    lines = ctx.libsvm_parse(st["text"].data_ptr(), st["text"].numel(), case["n"], case["d"], _lib.F32,
                             st["X"].data_ptr(), case["d"], st["y"].data_ptr())
    return {"X": st["X"], "y": st["y"], "lines": lines}


# ------------------------------------------------------------------------------------------------ algorithmic work
def work(case):
    kind = case["kind"]
    if kind in ("sketch", "block"):
        m, n, d = case["m"], case["n"], case["d"]
        points = 4.0 * d * (n if m == n else m + n) + 4.0 * (m + n)
        if kind == "block":
            return {"bytes": points + 4.0 * m * n, "flops": 2.0 * m * n * d}
        l = case["l"]
        return {"bytes": points + 4.0 * l * (m + n), "flops": 2.0 * m * n * (d + l)}
    if kind == "knn":
        n, d, s = case["n"], case["d"], case["s"]
        return {"bytes": 4.0 * n * (d + 1) + 4.0 * s, "flops": 2.0 * n * s * d}
    if kind == "solve":
        # three kernel passes, two orthonormalisations, the core, and some 30 Newton steps over Z
        n, d, l = case["n"], case["d"], case["l"]
        return {"bytes": 4.0 * n * (d + l) + 8.0 * n * (l + 1),
                "flops": 6.0 * n * n * (d + l) + 12.0 * n * l * l + 30.0 * n * l * l}
    if kind == "cholqr2":
        n, l = case["n"], case["l"]
        return {"bytes": 16.0 * n * l + 8.0 * l * l, "flops": 4.0 * n * l * l}
    if kind == "potrf":
        n = case["n"]
        return {"bytes": 12.0 * n * n, "flops": n ** 3 / 3.0}
    if kind == "barrier":
        # some 50 Newton steps, each one pass over Z and one r x r capacity matrix (upper triangle)
        n, r = case["n"], case["r"]
        return {"bytes": 50 * 8.0 * n * r, "flops": 50 * (1.0 * n * r * r + r ** 3 / 3.0)}
    if kind == "landmark":
        n, d, r = case["n"], case["d"], case["r"]
        return {"bytes": 4.0 * n * d + 8.0 * n * r, "flops": 2.0 * n * r * d + 1.0 * n * r * r + r ** 3 / 3.0}
    if kind == "mlp":
        m, i, w, h = case["m"], case["inputs"], case["width"], case["hidden"]
        params = i * w + (h - 1) * w * w + w
        return {"bytes": 4.0 * m * (i + 1) + 8.0 * params, "flops": 6.0 * m * params - 2.0 * m * i * w}
    n, d = case["n"], case["d"]
    per_line = 15.0 if case["sparse"] else 3.0
    text = n * (per_line + (0.11 * d * 6 if case["sparse"] else d * 12.0))
    return {"bytes": text + 4.0 * n * (d + 1), "flops": 0.0}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _sketch64(Xi, X, yi, y, Om, gamma, rows=4096):
    """K Omega in FP64 by row blocks; Om n x l FP64."""
    return torch.cat([_kernel64(Xi[r:r + rows], X, yi[r:r + rows], y, gamma) @ Om for r in range(0, len(Xi), rows)])


def _qr64(Y):
    Q, R = torch.linalg.qr(Y)
    s = torch.sign(torch.diagonal(R))
    return Q * s[None, :], R * s[:, None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("barrier",):
        return None  # an iterative solve stopped at a gap: no closed form
    st = prepare(case, seed)
    if kind in ("sketch", "block"):
        X, Xi = (st["X"].T, st["Xi"].T) if case["layout"] == 1 else (st["X"], st["Xi"])
        if kind == "block":
            return _kernel64(Xi, X, st["yi"], st["y"], _gamma(case)).T.contiguous()
        return _sketch64(Xi, X, st["yi"], st["y"], st["Om"].T.double(), _gamma(case)).T.contiguous()
    if kind == "knn":
        X, ref = st["X"].double(), st["ref"].long()
        R, out = X[ref], []
        for r in range(0, case["n"], 4096):
            D = (X[r:r + 4096] ** 2).sum(1)[:, None] + (R * R).sum(1)[None, :] - 2.0 * (X[r:r + 4096] @ R.T)
            D[torch.arange(r, min(r + 4096, case["n"]), device="cuda")[:, None] == ref[None, :]] = math.inf
            near = torch.topk(D, case["k"], dim=1, largest=False)[1]
            diff = X[r:r + 4096][:, None, :] - R[near]
            out.append((diff * diff).sum(2).max(1)[0].sqrt())
        return torch.cat(out)
    if kind == "solve":
        X, y, g = st["X"], st["y"], _gamma(case)
        Q = _qr64(_sketch64(X, X, y, y, st["Om"].T.double(), g))[0]
        Q = _qr64(_sketch64(X, X, y, y, Q, g))[0]
        Cm = Q.T @ _sketch64(X, X, y, y, Q, g)
        Cm = 0.5 * (Cm + Cm.T)
        Cm += torch.eye(case["l"], device="cuda", dtype=torch.float64) * (1e-7 * Cm.trace() / case["l"])
        return {"a": None, "Z": (Q @ torch.linalg.cholesky(Cm)).T.contiguous(), "f": None}
    if kind == "cholqr2":
        Q, R = _qr64(st["Y"].T)
        return {"Q": Q.T.contiguous(), "R": R.T.contiguous()}
    if kind == "potrf":
        return torch.linalg.cholesky(st["A"])  # the storage of the upper factor, column major
    if kind == "landmark":
        Z = _nystrom64(st["X"], st["y"], _gamma(case), st["idx"])
        return {"Z": Z.T.contiguous(), "nu": 1e-7}  # K(i, i) = 1: the mean of W's diagonal is 1
    if kind == "mlp":
        flat = torch.from_numpy(st["net"].get_params()).cuda().double()
        h, off, layers = st["F"].double(), 0, []
        sizes = [case["inputs"]] + [case["width"]] * case["hidden"] + [1]
        for fi, fo in zip(sizes[:-1], sizes[1:]):
            W = flat[off:off + fi * fo].view(fo, fi).requires_grad_()
            b = flat[off + fi * fo:off + fi * fo + fo].clone().requires_grad_()
            off += fi * fo + fo
            layers += [W, b]
            h = h @ W.T + b
            h = torch.relu(h) if fo != 1 or len(layers) < 2 * len(sizes) - 2 else h
        loss = 0.5 * ((h[:, 0] - st["t"].double()) ** 2).mean()
        grads = torch.autograd.grad(loss, layers)
        return {"grads": torch.cat([v.reshape(-1) for v in grads]), "loss": float(loss.detach())}
    _, X, y = _libsvm(case, seed)
    return {"X": torch.from_numpy(X).cuda(), "y": torch.from_numpy(y).cuda(), "lines": None}
