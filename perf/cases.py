"""What the framework is timed on: the work its users have it do, through its public entry points.

Kinds of work
  dot       C = act(A . W + bias) through Context.gemm: one layer's forward product (the reference's ClusterNet::dot plus the
            elementwise passes behind it), in the fp32-accurate mode and in the single-pass TF32 mode
  dotmpi    the README's two-layer product through Context.dotmpi, the weights resident on the GPU
  backward  one layer's backward pass: weight gradient (Tdot), error for the layer below (dotT), unit derivative, RMSprop step
  train     a whole data-parallel training step of a three-layer network (dropout, softmax error, gradient exchange, update)
  codec     the 8-bit codec: scale, compress, decompress of one tensor
  packed    the codec over the gradients of several layers that lie back to back in one buffer
  batch     the batch allocator: stage, copy and swap in the next batch of a data set in pinned host memory

Matrices are column-major as everywhere in the framework: a rows x cols matrix is a tensor of shape (cols, rows).
"""
import ctypes
import math

import torch

import clusternet_b200 as cn
from clusternet_b200 import _lib

ACTS = {"linear": _lib.ACT_LINEAR, "relu": _lib.ACT_RELU, "logistic": _lib.ACT_LOGISTIC}
MODES = {"3xtf32": _lib.GEMM_3XTF32, "tf32": _lib.GEMM_TF32}

_context = None


def _ctx():
    """The one context a program keeps."""
    global _context
    if _context is None:
        _context = cn.Context(0)
    return _context


def listed():
    return [
        # one hidden layer's forward pass at the size of the single-layer configuration: the smallest call, bound by latency
        dict(name="dot_128x784x1024", kind="dot", M=128, K=784, N=1024, mode="3xtf32", act="relu", bias=True),
        # a layer whose sizes are no multiple of anything (a last, partial batch; an odd number of features and units)
        dict(name="dot_odd_203x4001x3001", kind="dot", M=203, K=4001, N=3001, mode="3xtf32", act="logistic", bias=True),
        # the smallest square product of the GEMM sweep: a large batch, bound by the tensor cores
        dict(name="dot_4096_cubed", kind="dot", M=4096, K=4096, N=4096, mode="3xtf32", act="linear", bias=False),
        # a wide layer of the sweep in the single-pass mode, bound by reading the weights
        dict(name="dot_tf32_128x40000x40000", kind="dot", M=128, K=40000, N=40000, mode="tf32", act="linear", bias=False),
        # the README's benchmark, on one GPU: the largest
        dict(name="dotmpi_readme", kind="dotmpi", M=128, K=100000, N1=40000, N2=20000),
        # backward pass of a wide layer
        dict(name="backward_128x4096x4096", kind="backward", M=128, K=4096, N=4096, act="relu"),
        # the training step of the network configuration, call by call as a program makes it
        dict(name="train_784_1200_1200_10", kind="train", M=128, n0=784, n1=1200, n2=1200, n3=10),
        # the gradient of that network's first layer through the codec: small, bound by launches
        dict(name="codec_784x1200", kind="codec", n=784 * 1200, scale="absmax", sigma=1e-3),
        # the codec configuration, the scale known beforehand
        dict(name="codec_4096x4096", kind="codec", n=4096 * 4096, scale="host", sigma=0.1),
        # the largest tensor of the codec benchmark: 1 GiB of floats
        dict(name="codec_1gib", kind="codec", n=1 << 28, scale="absmax", sigma=0.1),
        # gradients of a network with a bias column in every layer, packed: lengths and offsets that are not multiples of four
        dict(name="packed_785_1201_1201", kind="packed", n1=785 * 1201, n2=1201 * 1201, n3=1201 * 10, sigma=1e-3),
        # batches of 128 flattened 28 x 28 images
        dict(name="batch_128x784", kind="batch", rows=10000, cols=784, M=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A size between lo and hi, spread over the logarithm; half of them whole multiples of 8, as most layers are."""
    v = _log(rng, lo, hi)
    return min(hi, max(lo, (v + 4) // 8 * 8)) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["dot", "dot", "dot", "dot", "dotmpi", "backward", "backward", "train", "codec", "codec", "packed", "batch"])
    if kind == "dot":
        while True:
            M, K, N = _size(rng, 16, 4096), _size(rng, 64, 40000), _size(rng, 64, 40000)
            if M * K * N <= 4096 ** 3:
                break
        return dict(kind=kind, M=M, K=K, N=N, mode=rng.choice(["3xtf32", "3xtf32", "tf32"]), act=rng.choice(sorted(ACTS)),
                    bias=rng.random() < 0.7)
    if kind == "dotmpi":
        return dict(kind=kind, M=_size(rng, 32, 128), K=_size(rng, 2000, 100000), N1=_size(rng, 1000, 40000), N2=_size(rng, 500, 20000))
    if kind == "backward":
        return dict(kind=kind, M=_size(rng, 32, 512), K=_size(rng, 500, 6000), N=_size(rng, 500, 6000), act=rng.choice(["relu", "logistic"]))
    if kind == "train":
        return dict(kind=kind, M=_size(rng, 32, 512), n0=_size(rng, 64, 3000), n1=_size(rng, 64, 3000), n2=_size(rng, 64, 3000),
                    n3=rng.randint(2, 100))
    if kind == "codec":
        return dict(kind=kind, n=_size(rng, 10000, 1 << 28), scale=rng.choice(["absmax", "host"]), sigma=rng.choice([1e-3, 1e-2, 0.1, 1.0]))
    if kind == "packed":
        return dict(kind=kind, n1=_size(rng, 1000, 4000000), n2=_size(rng, 1000, 4000000), n3=_size(rng, 1000, 100000),
                    sigma=rng.choice([1e-3, 1e-2]))
    M, cols = _size(rng, 16, 512), _size(rng, 16, 2000)
    return dict(kind="batch", rows=_log(rng, 2 * M, 10000), cols=cols, M=M)


# ------------------------------------------------------------------------------------------------------- inputs
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _uniform(g, rows, cols, lo=-1.0, hi=1.0):
    return torch.rand((cols, rows), device="cuda", generator=g).mul_(hi - lo).add_(lo)


def _weight(g, rows, cols):
    """uniformSqrtWeight: uniform in +-4 sqrt(6 / (in + out))."""
    lim = 4.0 * math.sqrt(6.0 / (rows + cols))
    return _uniform(g, rows, cols, -lim, lim)


def _gradient(g, n, sigma):
    return torch.randn(n, device="cuda", generator=g).mul_(sigma)


def _empty(rows, cols):
    return torch.empty((cols, rows), device="cuda")


class _Batch:
    """A batch allocator and the host data set it reads, released with the state."""

    def __init__(self, ctx, X, y, M):
        self.X, self.y, self.lib = X, y, ctx.lib
        self.h = ctypes.c_void_p()
        cn.check(ctx.lib.cn_batch_create(ctx.h, X.data_ptr(), y.data_ptr(), X.shape[0], X.shape[1], 1, M, 0, ctypes.byref(self.h)))

    def __del__(self):
        self.lib.cn_batch_destroy(self.h)


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    g = _gen(seed)
    s = {"case": dict(case), "ctx": ctx}
    if kind == "dot":
        M, K, N = case["M"], case["K"], case["N"]
        s.update(A=_uniform(g, M, K), W=_weight(g, K, N), bias=_uniform(g, N, 1).view(-1) if case["bias"] else None, C=_empty(M, N))
    elif kind == "dotmpi":
        M, K, N1, N2 = case["M"], case["K"], case["N1"], case["N2"]
        s.update(A=_uniform(g, M, K, 0.0, 1.0), W1=_weight(g, K, N1), W2=_weight(g, N1, N2), out1=_empty(M, N1), out2=_empty(M, N2))
    elif kind == "backward":
        M, K, N = case["M"], case["K"], case["N"]
        act = torch.randn((K, M), device="cuda", generator=g)           # the activations the layer below handed up
        act = act.clamp_(min=0) if case["act"] == "relu" else act.sigmoid_()
        err = torch.randn((N, M), device="cuda", generator=g).mul_(1e-2)
        err.mul_(torch.rand((N, M), device="cuda", generator=g) < 0.5)  # half of the units above are off
        # a running mean of squared gradients as it stands in the middle of training
        s.update(act=act, err=err, W=_weight(g, K, N), grad=_empty(K, N), below=_empty(M, K), rms=_uniform(g, K, N, 5e-3, 2e-2).mul_(1e-1))
    elif kind == "train":
        M, sizes = case["M"], [case["n0"], case["n1"], case["n2"], case["n3"]]
        numel = [sizes[i] * sizes[i + 1] for i in range(3)]
        offs = [0, numel[0], numel[0] + numel[1]]
        X = torch.randn((sizes[0], M), device="cuda", generator=g)
        y = torch.randint(0, sizes[3], (M,), device="cuda", generator=g).float()
        Wp, gp = torch.empty(sum(numel), device="cuda"), torch.zeros(sum(numel), device="cuda")
        for i in range(3):
            Wp[offs[i]:offs[i] + numel[i]] = _weight(g, sizes[i], sizes[i + 1]).view(-1)
        views = [[t[offs[i]:offs[i] + numel[i]].view(sizes[i + 1], sizes[i]) for i in range(3)] for t in (Wp, gp)]
        s.update(X=X, y=y, Wp=Wp, gp=gp, rms=_uniform(g, sum(numel), 1, 0.5, 2.0).view(-1), W=views[0], grad=views[1], seg=(ctypes.c_int64 * 3)(*numel),
                 bias=[_uniform(g, sizes[i + 1], 1, -0.1, 0.1).view(-1) for i in range(3)],
                 act=[X] + [_empty(M, sizes[i + 1]) for i in range(3)], out=[_empty(M, n) for n in sizes],
                 err=[None] + [_empty(M, sizes[i + 1]) for i in range(3)], seed=torch.tensor([1000 + seed], dtype=torch.int64, device="cuda"))
    elif kind == "codec":
        x = _gradient(g, case["n"], case["sigma"])
        s.update(x=x, codes=torch.empty(case["n"], dtype=torch.uint8, device="cuda"), back=torch.empty_like(x),
                 scale=torch.empty(1, device="cuda") if case["scale"] == "absmax" else float(x.abs().max()))
    elif kind == "packed":
        sizes = [case["n1"], case["n2"], case["n3"]]
        x = _gradient(g, sum(sizes), case["sigma"])
        s.update(x=x, codes=torch.empty(sum(sizes), dtype=torch.uint8, device="cuda"), back=torch.empty_like(x), scales=torch.empty(3, device="cuda"))
        cut = [0, sizes[0], sizes[0] + sizes[1], sum(sizes)]
        s["parts"] = [tuple(t[cut[i]:cut[i + 1]] for t in (s["x"], s["codes"], s["back"])) + (s["scales"][i:i + 1],) for i in range(3)]
    elif kind == "batch":
        gh = _gen(seed, "cpu")
        X = torch.rand((case["rows"], case["cols"]), generator=gh, pin_memory=True)
        y = torch.randint(0, 10, (case["rows"], 1), generator=gh).float().pin_memory()
        s.update(batch=_Batch(ctx, X, y, case["M"]), px=ctypes.c_void_p(), py=ctypes.c_void_p(), rows=ctypes.c_int64())
    return s


# --------------------------------------------------------------------------------------------------------- work
def _run_backward(s):
    ctx, lib, h, c = s["ctx"], s["ctx"].lib, s["ctx"].h, s["case"]
    sp = ctx.stream_ptr()
    ctx.gemm(s["act"], s["err"], out=s["grad"], transA=True)
    ctx.gemm(s["err"], s["W"], out=s["below"], transB=True)
    cn.check(lib.cn_mul_activation_gradient(h, s["below"].data_ptr(), s["act"].data_ptr(), ACTS[c["act"]], None, s["below"].data_ptr(),
                                            s["below"].numel(), sp))
    cn.check(lib.cn_rmsprop_update(h, s["rms"].data_ptr(), s["grad"].data_ptr(), s["W"].data_ptr(), 0.9, 0.006, s["grad"].numel(), sp))
    return s["grad"], s["below"], s["W"], s["rms"]


def _run_train(s):
    """Forward with dropout, softmax error, backward, gradient exchange (one rank: the RMSprop step alone).  Logistic hidden units:
    with a unit that switches, two correct implementations differ wherever an input rounds to the other side of zero."""
    ctx, lib, h = s["ctx"], s["ctx"].lib, s["ctx"].h
    sp, seed = ctx.stream_ptr(), s["seed"].data_ptr()
    act, out, err, W, grad, bias = s["act"], s["out"], s["err"], s["W"], s["grad"], s["bias"]
    cn.check(lib.cn_dropout_dp(h, act[0].data_ptr(), out[0].data_ptr(), act[0].numel(), 0.2, seed, 0, sp))
    for l in range(3):
        last = l == 2
        ctx.gemm(out[l], W[l], out=out[3] if last else act[l + 1], bias=bias[l], activation=_lib.ACT_LINEAR if last else _lib.ACT_LOGISTIC)
        if not last:
            cn.check(lib.cn_dropout_dp(h, act[l + 1].data_ptr(), out[l + 1].data_ptr(), act[l + 1].numel(), 0.5, seed, 1 << (20 + l), sp))
    rows, classes = s["case"]["M"], s["case"]["n3"]
    cn.check(lib.cn_softmax_error(h, out[3].data_ptr(), s["y"].data_ptr(), out[3].data_ptr(), err[3].data_ptr(), rows, classes, sp))
    for l in (2, 1, 0):
        ctx.gemm(act[l], err[l + 1], out=grad[l], transA=True)
        if l > 0:
            ctx.gemm(err[l + 1], W[l], out=err[l], transB=True)
            cn.check(lib.cn_mul_activation_gradient(h, err[l].data_ptr(), act[l].data_ptr(), _lib.ACT_LOGISTIC, None, err[l].data_ptr(),
                                                    err[l].numel(), sp))
    cn.check(lib.cn_grad_sync_8bit_rmsprop(h, s["gp"].data_ptr(), s["seg"], 3, 0.0, s["rms"].data_ptr(), s["Wp"].data_ptr(), 0.9, 0.006, sp))
    cn.check(lib.cn_seed_advance(h, seed, sp))
    return out[3], s["gp"], s["Wp"], s["rms"], s["seed"]


class _Device:
    """Device memory of a batch allocator as torch.as_tensor takes it."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner   # the memory lives as long as a tensor shows it
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 2, "strides": None}


def _run_batch(s):
    ctx, b = s["ctx"], s["batch"]
    cn.check(ctx.lib.cn_batch_copy_next_async(b.h))
    cn.check(ctx.lib.cn_batch_swap(b.h, ctx.stream_ptr(), ctypes.byref(s["px"]), ctypes.byref(s["py"]), ctypes.byref(s["rows"])))
    n = s["rows"].value
    return (torch.as_tensor(_Device(b, s["px"].value, (s["case"]["cols"], n)), device="cuda"),
            torch.as_tensor(_Device(b, s["py"].value, (1, n)), device="cuda"))


def run(s):
    ctx, c = s["ctx"], s["case"]
    kind = c["kind"]
    if kind == "dot":
        return ctx.gemm(s["A"], s["W"], out=s["C"], bias=s["bias"], activation=ACTS[c["act"]], mode=MODES[c["mode"]])
    if kind == "dotmpi":
        ctx.dotmpi(s["A"], s["W1"], c["N1"], out=s["out1"])
        ctx.dotmpi(s["out1"], s["W2"], c["N2"], out=s["out2"])
        return s["out1"], s["out2"]
    if kind == "backward":
        return _run_backward(s)
    if kind == "train":
        return _run_train(s)
    if kind == "codec":
        if c["scale"] == "absmax":
            ctx.absmax_compress(s["x"], scale=s["scale"], out=s["codes"])
        else:
            ctx.compress(s["x"], s["scale"], out=s["codes"])
        ctx.decompress(s["codes"], s["scale"], out=s["back"])
        return s["codes"], s["back"], s["scale"]
    if kind == "packed":
        for x, codes, back, scale in s["parts"]:
            ctx.absmax_compress(x, scale=scale, out=codes)
        for x, codes, back, scale in s["parts"]:
            ctx.decompress(codes, scale, out=back)
        return s["codes"], s["back"], s["scales"]
    return _run_batch(s)


def work(case):
    kind = case["kind"]
    if kind == "dot":
        M, K, N = case["M"], case["K"], case["N"]
        return {"bytes": 4.0 * (M * K + K * N + M * N + (N if case["bias"] else 0)), "flops": 2.0 * M * K * N}
    if kind == "dotmpi":
        M, K, N1, N2 = case["M"], case["K"], case["N1"], case["N2"]
        return {"bytes": 4.0 * (M * K + K * N1 + 2 * M * N1 + N1 * N2 + M * N2), "flops": 2.0 * M * (K * N1 + N1 * N2)}
    if kind == "backward":
        M, K, N = case["M"], case["K"], case["N"]
        # read act, err, W, rms; write grad, the error below, W, rms
        return {"bytes": 4.0 * (2 * M * K + M * N + 5 * K * N), "flops": 4.0 * M * K * N}
    if kind == "train":
        M, n = case["M"], [case["n0"], case["n1"], case["n2"], case["n3"]]
        w = sum(n[i] * n[i + 1] for i in range(3))
        # the batch and the labels read; weights and RMS state read and written, gradients and probabilities written
        return {"bytes": 4.0 * (M * (n[0] + 1 + n[3]) + 5 * w), "flops": 2.0 * M * (3 * w - n[0] * n[1])}
    if kind == "codec":
        return {"bytes": 10.0 * case["n"], "flops": 0.0}   # compress: 4 bytes in, 1 out; decompress: 1 in, 4 out
    if kind == "packed":
        return {"bytes": 10.0 * (case["n1"] + case["n2"] + case["n3"]), "flops": 0.0}
    return {"bytes": 8.0 * case["M"] * (case["cols"] + 1), "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("codec", "packed", "batch"):
        return "exact"      # codes, decoded values and copied batches are the same bit for bit
    if kind == "dot" and case["mode"] == "tf32":
        return {"rel": 1e-3}   # both operands rounded to 11 significand bits: about 4e-4 of random rounding in each implementation
    return {"rel": 1e-5}    # sums of fp32 products, in another order
