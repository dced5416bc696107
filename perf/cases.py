"""What a user of this package has it do: the work whose time counts.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges, `prepare(case, seed)` makes what a
program holds before the call, `run(state)` is one pass through the public operators (luxlib_b200) and returns the
outputs whole, `work(case)` counts the bytes and operations that no implementation can do without, `tolerance(case)`
says how far another correct implementation of the same precision may be off, `exact(case, seed)` is what `run` returns
in 64-bit arithmetic.

Six kinds of work:
  mlp        two dense layers and the mean-squared error, forward + pullback (small, latency counts)
  dense      one fused dense layer: forward only (inference on small batches) or forward + pullback (training)
  conv_bn    one bias-free convolution + training-mode BatchNorm carrying relu, forward + pullback
  resnet18   the whole ResNet-18: a training step (loss, gradients, momentum update) or test-mode forward (logits)
  norm       layernorm / groupnorm / batchnorm, forward + pullback
  attention  scaled dot product attention, forward + pullback
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lux.jl_b200"))

import luxlib_b200 as L  # noqa: E402
from luxlib_b200 import distributed as D  # noqa: E402

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest training program: Dense(784 -> 256, relu) -> Dense(256 -> 10) on a batch of 128 images
        {"name": "mlp_f32", "kind": "mlp", "dtype": "f32", "d0": 784, "d1": 256, "d2": 10, "batch": 128},
        # a trained layer answering a handful of requests at a time: one pass over the weights
        {"name": "dense_infer_bf16", "kind": "dense", "mode": "infer", "dtype": "bf16", "act": "gelu", "M": 4096, "N": 8, "K": 4096},
        # the large fused dense layer in training: three full-size contractions
        {"name": "dense_train_bf16", "kind": "dense", "mode": "train", "dtype": "bf16", "act": "gelu", "M": 4096, "N": 8192, "K": 4096},
        # a layer whose sizes come from the data: nothing is a multiple of anything, Lux's default element type
        {"name": "dense_train_f32_ragged", "kind": "dense", "mode": "train", "dtype": "f32", "act": "tanh", "M": 1001, "N": 300, "K": 515},
        # the convolution of a ResNet basic block with its BatchNorm, in training
        {"name": "conv_bn_bf16", "kind": "conv_bn", "dtype": "bf16", "size": 56, "k": 3, "stride": 1, "pad": 1, "cin": 64, "cout": 64,
         "batch": 256},
        # the conv-net training step at the per-GPU batch of the data-parallel benchmark (the largest work here)
        {"name": "resnet18_train_bf16", "kind": "resnet18", "mode": "train", "dtype": "bf16", "size": 224, "batch": 256},
        # the same network in Lux's default element type, at a batch that fits a smaller budget
        {"name": "resnet18_train_f32", "kind": "resnet18", "mode": "train", "dtype": "f32", "size": 224, "batch": 32},
        # classifying a few images with the trained network
        {"name": "resnet18_infer_f32", "kind": "resnet18", "mode": "infer", "dtype": "f32", "size": 224, "batch": 4},
        # LayerNorm over the features of a large token batch, in training
        {"name": "layernorm_bf16", "kind": "norm", "op": "layernorm", "dtype": "bf16", "D": 4096, "R": 16384},
        # LayerNorm of a small token batch: launch-bound
        {"name": "layernorm_f32_small", "kind": "norm", "op": "layernorm", "dtype": "f32", "D": 768, "R": 197},
        # GroupNorm(32) on a feature map, in training
        {"name": "groupnorm_f32", "kind": "norm", "op": "groupnorm", "dtype": "f32", "size": 32, "channels": 512, "groups": 32, "batch": 128},
        # causal self-attention of a sequence model, in training
        {"name": "attention_bf16", "kind": "attention", "dtype": "bf16", "D": 64, "H": 8, "Hkv": 8, "L": 512, "S": 512, "batch": 8,
         "causal": True},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], uniform over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """As `_log`; half of the draws are rounded to a multiple of 8, as layer widths mostly are."""
    v = _log(rng, lo, hi)
    return max(lo, v // 8 * 8) if rng.random() < 0.5 and v >= 16 else v


def draw(rng):
    kind = rng.choice(["mlp", "dense", "dense", "conv_bn", "resnet18", "norm", "norm", "attention"])
    dtype = rng.choice(["f32", "bf16"])
    if kind == "mlp":
        return {"kind": kind, "dtype": dtype, "d0": _size(rng, 32, 1024), "d1": _size(rng, 32, 512), "d2": rng.randint(1, 100),
                "batch": _size(rng, 16, 512)}
    if kind == "dense":
        act = rng.choice(["identity", "relu", "gelu", "tanh", "sigmoid", "swish"])
        if rng.random() < 0.5:
            return {"kind": kind, "mode": "infer", "dtype": dtype, "act": act, "M": _size(rng, 256, 8192), "N": _log(rng, 1, 64),
                    "K": _size(rng, 256, 8192)}
        hi = 4096 if dtype == "bf16" else 2048
        return {"kind": kind, "mode": "train", "dtype": dtype, "act": act, "M": _size(rng, 128, hi), "N": _size(rng, 128, 2 * hi),
                "K": _size(rng, 128, hi)}
    if kind == "conv_bn":
        k, stride = rng.choice([(3, 1), (3, 1), (3, 2), (1, 1), (1, 2), (5, 1)])
        size = rng.randint(7, 64)
        cin, cout = _size(rng, 16, 256), _size(rng, 16, 256)
        most = (6e10 if dtype == "bf16" else 6e9) / (2.0 * (size / stride) ** 2 * cin * cout * k * k)
        return {"kind": kind, "dtype": dtype, "size": size, "k": k, "stride": stride, "pad": k // 2, "cin": cin, "cout": cout,
                "batch": max(2, min(_log(rng, 4, 256), int(most)))}
    if kind == "resnet18":
        if rng.random() < 0.5:
            return {"kind": kind, "mode": "infer", "dtype": dtype, "size": rng.randint(96, 256), "batch": _log(rng, 1, 32)}
        return {"kind": kind, "mode": "train", "dtype": dtype, "size": rng.randint(96, 224), "batch": _log(rng, 4, 128 if dtype == "bf16" else 32)}
    if kind == "norm":
        op = rng.choice(["layernorm", "groupnorm", "batchnorm"])
        if op == "layernorm":
            D = _size(rng, 64, 8192)
            return {"kind": kind, "op": op, "dtype": dtype, "D": D, "R": _log(rng, 64, min(32768, (1 << 26) // D))}
        size, channels = rng.choice([7, 14, 16, 28, 32, 56, rng.randint(5, 64)]), rng.choice([32, 64, 96, 128, 256, 512])
        batch = _log(rng, 2, max(2, min(256, (1 << 26) // (size * size * channels))))
        c = {"kind": kind, "op": op, "dtype": dtype, "size": size, "channels": channels, "batch": batch}
        return dict(c, groups=rng.choice([4, 8, 16, 32])) if op == "groupnorm" else c
    hkv, rep = rng.choice([1, 2, 4, 8, 12]), rng.choice([1, 1, 1, 2, 4])
    length = _size(rng, 16, 1024)
    causal = rng.random() < 0.5
    seen = length if causal or rng.random() < 0.5 else _size(rng, 16, 1024)
    most = int(2e8 / (4.0 * hkv * rep * length * seen))
    return {"kind": kind, "dtype": dtype, "D": rng.choice([32, 64, 64, 80, 128]), "H": hkv * rep, "Hkv": hkv, "L": length, "S": seen,
            "batch": max(1, min(_log(rng, 1, 16), most)), "causal": causal}


# ---------------------------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------------------------
class _Source:
    """Seeded device arrays in Julia's (column-major) layout."""

    def __init__(self, seed, dtype):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))
        self.dtype = dtype

    def _julia(self, t):
        t = t.to(self.dtype)
        return t.permute(*reversed(range(t.dim()))) if t.dim() > 1 else t

    def normal(self, *shape, std=1.0, mean=0.0):
        return self._julia(torch.randn(*reversed(shape), device="cuda", generator=self.g) * std + mean)

    def uniform(self, lo, hi, *shape):
        return self._julia(torch.rand(*reversed(shape), device="cuda", generator=self.g) * (hi - lo) + lo)

    def glorot(self, fan_out, fan_in):
        lim = math.sqrt(6.0 / (fan_out + fan_in))
        return self.uniform(-lim, lim, fan_out, fan_in)

    def kaiming(self, k, cin, cout):
        return self.normal(k, k, cin, cout, std=math.sqrt(2.0 / (k * k * cin)))

    def one_hot(self, classes, n):
        labels = torch.randint(0, classes, (n,), device="cuda", generator=self.g)
        return self._julia(torch.nn.functional.one_hot(labels, classes).float())


def _out(size, k, stride, pad):
    return (size + 2 * pad - k) // stride + 1


def _batchnorm_state(s, c):
    return {"scale": s.uniform(0.5, 1.5, c), "bias": s.normal(c, std=0.1), "mean": s.normal(c, std=0.1), "var": s.uniform(0.5, 1.5, c)}


def prepare(case, seed):
    s = _Source(seed, DTYPES[case["dtype"]])
    st = {"case": case}
    kind = case["kind"]
    if kind == "mlp":
        d0, d1, d2, n = case["d0"], case["d1"], case["d2"], case["batch"]
        st.update(W1=s.glorot(d1, d0), b1=s.normal(d1, std=0.01), W2=s.glorot(d2, d1), b2=s.normal(d2, std=0.01), x=s.normal(d0, n),
                  target=s.one_hot(d2, n))
    elif kind == "dense":
        M, N, K = case["M"], case["N"], case["K"]
        st.update(W=s.glorot(M, K), x=s.normal(K, N), b=s.uniform(-0.1, 0.1, M))
        if case["mode"] == "train":
            st["dy"] = s.normal(M, N)
    elif kind == "conv_bn":
        n, o = case["size"], _out(case["size"], case["k"], case["stride"], case["pad"])
        st.update(w=s.kaiming(case["k"], case["cin"], case["cout"]), x=s.normal(n, n, case["cin"], case["batch"]),
                  dy=s.normal(o, o, case["cout"], case["batch"]), bn=_batchnorm_state(s, case["cout"]),
                  dims=L.ConvDims.make(2, case["stride"], case["pad"]))
    elif kind == "resnet18":
        st.update(_resnet18_params(s), x=s.normal(case["size"], case["size"], 3, case["batch"]))
        if case["mode"] == "train":
            st["target"] = s.one_hot(1000, case["batch"])
            st["params"] = _resnet18_leaves(st)
            st["opt"] = D.FusedOptimizer(D.NCCLBackend, "momentum", eta=1e-2, rho=0.9)
            st["opt_state"] = st["opt"].init(st["params"])
    elif kind == "norm":
        if case["op"] == "layernorm":
            c, shape = case["D"], (case["D"], case["R"])
        else:
            c, shape = case["channels"], (case["size"], case["size"], case["channels"], case["batch"])
        st.update(_batchnorm_state(s, c), x=s.normal(*shape, std=1.3, mean=0.2), dy=s.normal(*shape))
    elif kind == "attention":
        b = case["batch"]
        st.update(q=s.normal(case["D"], case["H"], case["L"], b), k=s.normal(case["D"], case["Hkv"], case["S"], b),
                  v=s.normal(case["D"], case["Hkv"], case["S"], b), dx=s.normal(case["D"], case["H"], case["L"], b))
    return st


# ResNet-18: 7x7/2 stem, 3x3/2 max pool, four stages of two basic blocks (1x1/2 projections), global mean pool,
# Dense 512 -> 1000. The residual branches' last scales are those of a network that has trained for a while.
def _resnet18_params(s):
    conv = lambda k, cin, cout, stride, pad: {"w": s.kaiming(k, cin, cout), "bn": _batchnorm_state(s, cout),  # noqa: E731
                                              "dims": L.ConvDims.make(2, stride, pad)}
    blocks, cin = [], 64
    stem = conv(7, 3, 64, 2, 3)
    for cout in (64, 128, 256, 512):
        for j in range(2):
            stride = 2 if cout != 64 and j == 0 else 1
            blocks.append({"a": conv(3, cin, cout, stride, 1), "b": conv(3, cout, cout, 1, 1),
                           "skip": conv(1, cin, cout, stride, 0) if cin != cout else None})
            cin = cout
    return {"stem": stem, "blocks": blocks, "pool": L.PoolDims.make((3, 3), 2, 1), "Wd": s.glorot(1000, 512), "bd": s.normal(1000, std=0.01)}


def _resnet18_leaves(st):
    """The parameters in the order in which `_resnet18_step` collects their gradients."""
    leaves = [st["Wd"], st["bd"]]
    for blk in reversed(st["blocks"]):
        for layer in (blk["b"], blk["a"], blk["skip"]):
            if layer is not None:
                leaves += [layer["w"], layer["bn"]["scale"], layer["bn"]["bias"]]
    return leaves + [st["stem"]["w"], st["stem"]["bn"]["scale"], st["stem"]["bn"]["bias"]]


# ---------------------------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------------------------
def _conv_bn(act, layer, h):
    bn = layer["bn"]
    y, (bn["mean"], bn["var"]), pullback = L.rrule_conv_batchnorm(act, layer["w"], h, layer["dims"], bn["scale"], bn["bias"], bn["mean"],
                                                                  bn["var"], 0.1, 1e-5)
    return y, pullback


def _conv_bn_test(act, layer, h):
    bn = layer["bn"]
    u = L.fused_conv_bias_activation("identity", layer["w"], h, None, layer["dims"])
    return L.batchnorm(u, bn["scale"], bn["bias"], bn["mean"], bn["var"], False, act, 0.1, 1e-5)[0]


def _resnet18_forward(st):
    h = L.maxpool(_conv_bn_test("relu", st["stem"], st["x"]), st["pool"])
    for blk in st["blocks"]:
        a = _conv_bn_test("relu", blk["b"], _conv_bn_test("relu", blk["a"], h))
        h = L.add_activation("relu", a, h if blk["skip"] is None else _conv_bn_test("identity", blk["skip"], h))
    pooled = L.meanpool(h, L.PoolDims.global_(h))
    return L.fused_dense_bias_activation("identity", st["Wd"], pooled.reshape(512, h.shape[-1]), st["bd"])


def _resnet18_step(st):
    """One training step; the loss and the updated parameters."""
    grads = []
    h, pull_stem = _conv_bn("relu", st["stem"], st["x"])
    h, pull_pool = L.rrule_maxpool(h, st["pool"])
    tape = []
    for blk in st["blocks"]:
        skip, pull_skip = (h, None) if blk["skip"] is None else _conv_bn("identity", blk["skip"], h)
        a, pull_a = _conv_bn("relu", blk["a"], h)
        a, pull_b = _conv_bn("relu", blk["b"], a)
        h, pull_add = L.rrule_add_activation("relu", a, skip)
        tape.append((pull_a, pull_b, pull_skip, pull_add))
    n = h.shape[-1]
    pooled, pull_mean = L.rrule_meanpool(h, L.PoolDims.global_(h))
    y, pull_dense = L.rrule_fused_dense("identity", st["Wd"], pooled.reshape(512, n), st["bd"])
    loss, pull_loss = L.rrule_cross_entropy_loss(y, st["target"], logits=True)
    dW, dfeat, db = pull_dense(pull_loss())
    grads += [dW, db]
    dh = pull_mean(dfeat.reshape(1, 1, 512, n))
    for pull_a, pull_b, pull_skip, pull_add in reversed(tape):
        da, dskip = pull_add(dh)
        dw, da, dg, db = pull_b(da)
        grads += [dw, dg, db]
        dw, dmain, dg, db = pull_a(da)
        grads += [dw, dg, db]
        if pull_skip is not None:
            dw, dskip, dg, db = pull_skip(dskip)
            grads += [dw, dg, db]
        dh = L.add_activation("identity", dmain, dskip)
    dw, _, dg, db = pull_stem(pull_pool(dh), need_dx=False)
    st["opt"].update(st["opt_state"], st["params"], grads + [dw, dg, db])
    return [loss] + st["params"]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "mlp":
        h, pull1 = L.rrule_fused_dense("relu", st["W1"], st["x"], st["b1"])
        y, pull2 = L.rrule_fused_dense("identity", st["W2"], h, st["b2"])
        loss, pull_loss = L.rrule_mse_loss(y, st["target"])
        dW2, dh, db2 = pull2(pull_loss())
        dW1, dx, db1 = pull1(dh)
        return loss, dW1, db1, dW2, db2, dx
    if kind == "dense":
        if case["mode"] == "infer":
            return L.fused_dense_bias_activation(case["act"], st["W"], st["x"], st["b"])
        y, pullback = L.rrule_fused_dense(case["act"], st["W"], st["x"], st["b"])
        return (y,) + tuple(pullback(st["dy"]))
    if kind == "conv_bn":
        bn = st["bn"]
        y, stats, pullback = L.rrule_conv_batchnorm("relu", st["w"], st["x"], st["dims"], bn["scale"], bn["bias"], bn["mean"], bn["var"],
                                                    0.1, 1e-5)
        return (y,) + tuple(stats) + tuple(pullback(st["dy"]))
    if kind == "resnet18":
        return _resnet18_step(st) if case["mode"] == "train" else _resnet18_forward(st)
    if kind == "norm":
        if case["op"] == "layernorm":
            y, pullback = L.rrule_layernorm(st["x"], st["scale"], st["bias"], "identity", None, 1e-5)
            return (y,) + tuple(pullback(st["dy"]))
        if case["op"] == "groupnorm":
            y, pullback = L.rrule_groupnorm(st["x"], st["scale"], st["bias"], case["groups"], "identity", 1e-5)
            return (y,) + tuple(pullback(st["dy"]))
        y, stats, pullback = L.rrule_batchnorm(st["x"], st["scale"], st["bias"], st["mean"], st["var"], True, "identity", 0.1, 1e-5)
        return (y,) + tuple(stats) + tuple(pullback(st["dy"]))
    (x, w), pullback = L.rrule_scaled_dot_product_attention(st["q"], st["k"], st["v"], is_causal=True if case["causal"] else None)
    dq, dk, dv, _ = pullback(st["dx"])
    return x, w, dq, dk, dv


# ---------------------------------------------------------------------------------------------
# work, tolerance
# ---------------------------------------------------------------------------------------------
def _resnet18_macs(size, batch):
    """(multiply-adds of all convolutions and the dense layer, those of the stem, number of parameters)"""
    o = _out(size, 7, 2, 3)
    stem = o * o * 49 * 3 * 64
    macs, params = stem, 49 * 3 * 64 + 128
    h, cin = _out(o, 3, 2, 1), 64
    for cout in (64, 128, 256, 512):
        for j in range(2):
            stride = 2 if cout != 64 and j == 0 else 1
            o = _out(h, 3, stride, 1)
            macs += o * o * 9 * cout * (cin + cout)
            params += 9 * cout * (cin + cout) + 4 * cout
            if cin != cout:
                macs += o * o * cin * cout
                params += cin * cout + 2 * cout
            h, cin = o, cout
    return (macs + 512000) * batch, stem * batch, params + 513000


def work(case):
    es = 4 if case["dtype"] == "f32" else 2
    kind = case["kind"]
    if kind == "mlp":
        d0, d1, d2, n = case["d0"], case["d1"], case["d2"], case["batch"]
        return {"bytes": es * (2 * (d0 * d1 + d1 + d1 * d2 + d2) + 2 * d0 * n + d2 * n) + 4, "flops": 6.0 * n * (d0 * d1 + d1 * d2)}
    if kind == "dense":
        M, N, K = case["M"], case["N"], case["K"]
        if case["mode"] == "infer":
            return {"bytes": es * (M * K + K * N + M + M * N), "flops": 2.0 * M * N * K}
        return {"bytes": es * (2 * (M * K + K * N + M) + 2 * M * N), "flops": 6.0 * M * N * K}
    if kind == "conv_bn":
        o = _out(case["size"], case["k"], case["stride"], case["pad"])
        nx, ny = case["size"] ** 2 * case["cin"] * case["batch"], o * o * case["cout"] * case["batch"]
        nw = case["k"] ** 2 * case["cin"] * case["cout"]
        return {"bytes": es * (2 * nx + 2 * ny + 2 * nw + 8 * case["cout"]), "flops": 6.0 * ny * case["k"] ** 2 * case["cin"]}
    if kind == "resnet18":
        macs, stem, params = _resnet18_macs(case["size"], case["batch"])
        nx = case["size"] ** 2 * 3 * case["batch"]
        if case["mode"] == "infer":
            return {"bytes": es * (nx + params + 1000 * case["batch"]), "flops": 2.0 * macs}
        return {"bytes": es * (nx + 4 * params + 1000 * case["batch"]), "flops": 6.0 * macs - 2.0 * stem}   # no gradient of the images
    if kind == "norm":
        n = case["D"] * case["R"] if case["op"] == "layernorm" else case["size"] ** 2 * case["channels"] * case["batch"]
        c = case["D"] if case["op"] == "layernorm" else case["channels"]
        return {"bytes": es * (4 * n + (8 if case["op"] == "batchnorm" else 4) * c), "flops": 20.0 * n}
    D, H, hkv, b, ll, ss = case["D"], case["H"], case["Hkv"], case["batch"], case["L"], case["S"]
    pairs = H * b * (ll * (ll + 1) / 2 if case["causal"] else ll * ss)
    return {"bytes": es * b * (4 * D * H * ll + 4 * D * hkv * ss + H * ll * ss), "flops": 12.0 * D * pairs}


def tolerance(case):
    """Four times what the operators differ from another correct evaluation by (the CUDA-core kernels' summation order,
    or 64-bit arithmetic), over these ranges."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}       # the result's own rounding is 1.7e-3; 3.3e-3 after the 20 layers of a ResNet-18
    if case["kind"] == "resnet18" and case["mode"] == "train":
        return {"rel": 6e-4, "max": 1e-2}
    if case["kind"] in ("conv_bn", "mlp") or (case["kind"] == "dense" and case["act"] == "relu" and case["mode"] == "train"):
        # a pre-activation within rounding of zero may fall on the other side of relu: its cotangent comes or goes whole
        return {"rel": 6e-4, "max": 0.2}
    return {"rel": 1e-5}


# ---------------------------------------------------------------------------------------------
# exact: the same results from plain torch in 64 bits
# ---------------------------------------------------------------------------------------------
def _f64(t):
    """A double copy in row-major memory with the axes reversed: Julia's (W, H, C, N) is torch's (N, C, H, W)."""
    return t.permute(*reversed(range(t.dim()))).double().contiguous()


def _jl(t):
    t = t.detach()
    return t.permute(*reversed(range(t.dim()))) if t.dim() > 1 else t


_ACT64 = {"identity": lambda t: t, "relu": torch.relu, "tanh": torch.tanh, "sigmoid": torch.sigmoid,
          "swish": torch.nn.functional.silu, "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}


def _conv64(w, x, dims):
    """NNlib's convolution flips the filter; torch's does not."""
    return torch.nn.functional.conv2d(x, w.flip(2, 3), stride=dims.stride, padding=(dims.padding[0], dims.padding[2]))


def _norm64(x, mean, var, scale, bias):
    shape = (1, -1) + (1,) * (x.dim() - 2)
    return (x - mean) / torch.sqrt(var + 1e-5) * scale.view(shape) + bias.view(shape)


def _batch64(x, bn):
    """Training-mode BatchNorm and its updated running statistics."""
    over = [0] + list(range(2, x.dim()))
    n = x.numel() // x.shape[1]
    mean, var = x.mean(over, keepdim=True), x.var(over, unbiased=False, keepdim=True)
    y = _norm64(x, mean, var, bn["scale"], bn["bias"])
    return y, 0.9 * bn["mean"] + 0.1 * mean.flatten(), 0.9 * bn["var"] + 0.1 * var.flatten() * n / (n - 1)


def _classify64(st):
    def layer(act, l, h):
        bn = {k: v.double() for k, v in l["bn"].items()}
        shape = (1, -1, 1, 1)
        return act(_norm64(_conv64(_f64(l["w"]), h, l["dims"]), bn["mean"].view(shape), bn["var"].view(shape), bn["scale"], bn["bias"]))

    same = _ACT64["identity"]
    h = torch.nn.functional.max_pool2d(layer(torch.relu, st["stem"], _f64(st["x"])), 3, 2, 1)
    for blk in st["blocks"]:
        a = layer(torch.relu, blk["b"], layer(torch.relu, blk["a"], h))
        h = torch.relu(a + (h if blk["skip"] is None else layer(same, blk["skip"], h)))
    return h.mean((2, 3)) @ _f64(st["Wd"]) + st["bd"].double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "resnet18" and case["mode"] == "train":
        return None                # 62 layers of gradients in 64 bits take too long
    st = prepare(case, seed)
    if kind == "resnet18":
        with torch.no_grad():
            return _jl(_classify64(st))
    grad = lambda t: _f64(t).requires_grad_()  # noqa: E731
    if kind == "mlp":
        W1, b1, W2, b2, x = (grad(st[k]) for k in ("W1", "b1", "W2", "b2", "x"))
        y = torch.relu(x @ W1 + b1) @ W2 + b2
        loss = (y - _f64(st["target"])).square().mean()
        return [loss.detach().reshape(1)] + [_jl(g) for g in torch.autograd.grad(loss, (W1, b1, W2, b2, x))]
    if kind == "dense":
        W, x, b = (grad(st[k]) for k in ("W", "x", "b"))
        y = _ACT64[case["act"]](x @ W + b)
        if case["mode"] == "infer":
            return _jl(y)
        return [_jl(y)] + [_jl(g) for g in torch.autograd.grad(y, (W, x, b), _f64(st["dy"]))]
    if kind == "conv_bn" or (kind == "norm" and case["op"] == "batchnorm"):
        src = st["bn"] if kind == "conv_bn" else st
        bn = {k: src[k].double() for k in ("scale", "bias", "mean", "var")}
        bn["scale"].requires_grad_(), bn["bias"].requires_grad_()
        x = grad(st["x"])
        inputs = [x, bn["scale"], bn["bias"]]
        if kind == "conv_bn":
            w = grad(st["w"])
            inputs.insert(0, w)
            y, mean, var = _batch64(_conv64(w, x, st["dims"]), bn)
            y = torch.relu(y)
        else:
            y, mean, var = _batch64(x, bn)
        return [_jl(y), mean.detach(), var.detach()] + [_jl(g) for g in torch.autograd.grad(y, inputs, _f64(st["dy"]))]
    if kind == "norm":
        x, scale, bias = grad(st["x"]), st["scale"].double().requires_grad_(), st["bias"].double().requires_grad_()
        if case["op"] == "layernorm":
            y = torch.nn.functional.layer_norm(x, x.shape[1:], scale, bias, 1e-5)
        else:
            y = torch.nn.functional.group_norm(x, case["groups"], scale, bias, 1e-5)
        return [_jl(y)] + [_jl(g) for g in torch.autograd.grad(y, (x, scale, bias), _f64(st["dy"]))]
    q, k, v = (grad(st[n]) for n in "qkv")                       # (batch, tokens, heads, features)
    rep = case["H"] // case["Hkv"]
    k2, v2 = (t.repeat_interleave(rep, 2) for t in (k, v))
    logits = torch.einsum("bshd,blhd->bhls", k2, q) / math.sqrt(case["D"])
    if case["causal"]:
        logits = logits.masked_fill(torch.ones(case["L"], case["S"], device="cuda").triu(1).bool(), -math.inf)
    w = torch.softmax(logits, -1)
    y = torch.einsum("bshd,bhls->blhd", v2, w)
    return [_jl(y), _jl(w)] + [_jl(g) for g in torch.autograd.grad(y, (q, k, v), _f64(st["dx"]))]
