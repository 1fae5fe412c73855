"""Timed cases of the framework's public entry points: the calls its users make, over the range of sizes they make them at.

Families (`case["op"]`):
  net    one training step of a zoo net through the host layer: host image and labels in, forward, backward, update, loss and
         updated parameters out (dense prediction and classifier nets, bf16 tensor-core and fp32 arithmetic, 1 or 2 strips)
  conv   forward, data gradient, filter and bias gradient of one layer through the C ABI
  bn     batch normalisation (+ ReLU) of one activation, forward and backward
  halo   halo exchange and halo-gradient accumulate-back between the strips of one tensor
  head   the dense-prediction head: bilinear upsample, per-pixel softmax cross-entropy, both gradients
  pool   max or average pooling, forward and backward
"""
import ctypes as C
import math

import numpy as np
import torch

from arraydiff_cuda_b200 import abi, hostlib


def listed():
    return [
        # The dense-prediction configuration: dilated ResNet-50 on two 1024 x 2048 images, 19 classes.
        dict(name="net_segnet50_2x1024x2048_bf16", op="net", kind="segnet50", mode="bf16", N=2, H=1024, W=2048, strips=1),
        # Trunk of a partitioned net on one large image: many short launches.
        dict(name="net_stem_stage1_1024_bf16", op="net", kind="stem_stage1", mode="bf16", N=1, H=1024, W=1024, strips=1),
        # ImageNet training, 64 images per GPU cut into 2 strips each.
        dict(name="net_resnet50_64x224_2strips_bf16", op="net", kind="parallel_resnet50", mode="bf16", N=64, H=224, W=224, strips=2),
        # The default arithmetic of the training tools: fp32, NCHW.
        dict(name="net_resnet18_4x224_f32", op="net", kind="parallel_resnet18", mode="f32", N=4, H=224, W=224, strips=1),
        # The layer of the spatial convolution microbenchmark: 3x3, dilation 3, on a halo-3 strip.
        dict(name="conv_32x64x512x512_d3_bf16", op="conv", dtype="bf16", N=32, C=64, H=512, W=512, K=64, k=3, stride=1, dil=3),
        # A downsampling layer on an odd map.
        dict(name="conv_16x128x75x57_s2_bf16", op="conv", dtype="bf16", N=16, C=128, H=75, W=57, K=256, k=3, stride=2, dil=1),
        # One small fp32 layer: the smallest convolution anyone calls, latency and launches.
        dict(name="conv_1x64x64x64_f32", op="conv", dtype="f32", N=1, C=64, H=64, W=64, K=64, k=3, stride=1, dil=1),
        # Normalisation of the stage-1 block output of the 1024 x 2048 net.
        dict(name="bn_2x256x256x512_bf16", op="bn", dtype="bf16", N=2, C=256, H=256, W=512, relu=True),
        # Halo microbenchmark: 8 x 256 x 224 x 224 in 4 strips, 3 rows.
        dict(name="halo_4strips_8x256x224x224_p3_f32", op="halo", dtype="f32", R=4, p=3, N=8, C=256, H=224, W=224),
        # One-row halos of a small odd map in the tensor-core layout: the smallest exchange.
        dict(name="halo_2strips_1x64x56x57_p1_bf16", op="halo", dtype="bf16", R=2, p=1, N=1, C=64, H=56, W=57),
        # Head of the 1024 x 2048 net.
        dict(name="head_2x19x128x256_x8_bf16", op="head", dtype="bf16", N=2, C=19, H=128, W=256, scale=8),
        # The max pool behind the stem of the 1024 x 2048 net.
        dict(name="pool_max3s2_2x64x514x1026_bf16", op="pool", dtype="bf16", pooling="max", N=2, C=64, H=514, W=1026, k=3, stride=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["net", "net", "net", "conv", "conv", "conv", "bn", "halo", "head", "pool"])
    if op == "net":
        kind = rng.choice(["stem_stage1", "segnet50", "segnet_small", "parallel_resnet50", "parallel_resnet18"])
        mode = rng.choice(["bf16", "bf16", "bf16", "f32"])
        strips = rng.choice([1, 1, 2])
        unit = 64 * strips                          # rows: every stage of every strip keeps whole, wide enough strips
        side = 256 if mode == "f32" else 768 if kind == "stem_stage1" else 512
        H = unit * rng.randint(1, side // unit)
        W = _log(rng, 48, side)
        # enough images that the deepest maps still give the batch statistics a sample (1/32 of the rows and columns)
        most = (1 << 17 if mode == "f32" else 1 << 20) // (H * W)
        least = max(1, (1 << 16) // (H * W))
        N = _log(rng, least, max(least, min(32, most)))
        return dict(op=op, kind=kind, mode=mode, N=N, H=H, W=W, strips=strips)
    if op == "conv":
        while True:
            dtype = rng.choice(["bf16", "bf16", "f32"])
            k = rng.choice([1, 3, 3, 3])
            stride = rng.choice([1, 1, 1, 2])
            dil = rng.choice([1, 1, 2, 3, 4]) if k > 1 and stride == 1 else 1
            N, H, W = _log(rng, 1, 32), _log(rng, 7, 512), _log(rng, 7, 512)
            if dtype == "bf16":
                ch = rng.choice([64, 64, 128, 256, 512])
                K = rng.choice([64, 64, 128, 256, 512, 19])
            else:
                ch, K = _log(rng, 3, 256), _log(rng, 4, 256)
            case = dict(op=op, dtype=dtype, N=N, C=ch, H=H, W=W, K=K, k=k, stride=stride, dil=dil)
            if work(case)["flops"] <= (1.2e12 if dtype == "bf16" else 3e10):
                return case
    if op == "bn":
        while True:
            case = dict(op=op, dtype=rng.choice(["bf16", "bf16", "f32"]), N=_log(rng, 1, 64), C=8 * _log(rng, 2, 256), H=_log(rng, 7, 512),
                        W=_log(rng, 7, 512), relu=rng.random() < 0.8)
            if case["N"] * case["C"] * case["H"] * case["W"] <= 1 << 27:
                return case
    if op == "halo":
        while True:
            R, p = rng.choice([2, 4, 8]), rng.randint(1, 4)
            case = dict(op=op, dtype=rng.choice(["f32", "bf16"]), R=R, p=p, N=_log(rng, 1, 16), C=8 * _log(rng, 1, 64), H=R * _log(rng, 2 * p, 128),
                        W=_log(rng, 16, 512))
            if case["N"] * case["C"] * case["H"] * case["W"] <= 1 << 27:
                return case
    if op == "head":
        while True:
            case = dict(op=op, dtype=rng.choice(["bf16", "bf16", "f32"]), N=_log(rng, 1, 8), C=_log(rng, 2, 150), H=_log(rng, 8, 160), W=_log(rng, 8, 256),
                        scale=rng.choice([2, 4, 8]))
            if case["N"] * case["C"] * case["H"] * case["W"] * case["scale"] ** 2 <= 1 << 27:
                return case
    while True:
        pooling = rng.choice(["max", "max", "avg"])
        k, stride = rng.choice([(3, 2), (3, 2), (2, 2), (3, 1)]) if pooling == "max" else (0, 1)   # k 0: the whole map (global pool)
        side = (5, 512) if pooling == "max" else (4, 32)
        case = dict(op="pool", dtype=rng.choice(["bf16", "bf16", "f32"]), pooling=pooling, N=_log(rng, 1, 64), C=8 * _log(rng, 2, 256), H=_log(rng, *side),
                    W=_log(rng, *side), k=k, stride=stride)
        if case["N"] * case["C"] * case["H"] * case["W"] <= 1 << 27:
            return case


# ------------------------------------------------------------------ shared pieces
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _torch_dtype(name):
    return torch.float32 if name == "f32" else torch.bfloat16


def _uniform(g, shape, dtype=torch.float32):
    return torch.rand(shape, generator=g, device="cuda").mul_(2).sub_(1).to(dtype)


def _normal(g, shape, dtype=torch.float32, std=1.0):
    return torch.randn(shape, generator=g, device="cuda").mul_(std).to(dtype)


def _act(dtype, N, ch, H, W):
    """Shape of an activation: NCHW in fp32, NHWC in bf16."""
    return (N, ch, H, W) if dtype == "f32" else (N, H, W, ch)


def _view(t):
    f32 = t.dtype == torch.float32
    N, ch, H, W = t.shape if f32 else (t.shape[0], t.shape[3], t.shape[1], t.shape[2])
    if f32:
        sn, sc, sy, sx = t.stride()
    else:
        sn, sy, sx, sc = t.stride()
    return abi.Tensor4(t.data_ptr(), abi.AD_F32 if f32 else abi.AD_BF16, N, ch, H, W, sn, sc, sy, sx)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t):
    return C.c_void_p(t.data_ptr())


def _es(case):
    return 4 if case["dtype"] == "f32" else 2


# ------------------------------------------------------------------ net
# A program builds a net once and feeds it batches: nets are kept per configuration, a state is one batch.
_NETS = {}


def _arena_mb(case):
    px = case["N"] * case["H"] * case["W"] / case["strips"]
    # bytes per input pixel of the activations, gradients and working memory, and a constant for parameters and scratch
    per_px = dict(stem_stage1=2600, segnet50=9000, segnet_small=5200, parallel_resnet50=6400, parallel_resnet18=6400)[case["kind"]]
    fixed = dict(stem_stage1=400, segnet50=1600, segnet_small=900, parallel_resnet50=1800, parallel_resnet18=1100)[case["kind"]]
    return int(px * per_px * (2 if case["mode"] == "f32" else 1) / (1 << 20)) + fixed


def _net(case):
    key = (case["kind"], case["mode"], case["N"], case["H"], case["W"], case["strips"])
    if key not in _NETS:
        ctx = hostlib.Context([torch.cuda.current_device()] * case["strips"], hostlib.BF16_NHWC if case["mode"] == "bf16" else hostlib.F32_NCHW,
                              arena_mb=_arena_mb(case))
        net = hostlib.Net(ctx, case["kind"], case["H"], case["W"], 3, batch=case["N"], filters=1000 if "resnet" in case["kind"] else 64, seed=1)
        # no momentum: what one step leaves behind is the parameters alone.  The trunk has no loss, its objective <dy, y> is
        # unbounded: a small rate keeps its weights in range over thousands of steps.
        net.configure_sgd(1e-5 if case["kind"] == "stem_stage1" else 0.01, 0.0, l2=1e-4)
        first = net.params(0)
        x, labels = _batch(case, net, 0)
        net.forward(x)                              # call by call once: whatever is set up lazily exists afterwards
        if labels is None:
            dy = _normal(_gen(77), net.strip_shape).cpu().numpy()
            for r in range(case["strips"]):
                net.set_output_grad(r, dy)
        else:
            for r, lab in enumerate(labels):
                net.set_labels(r, lab)
        net.backward()
        net.sgd_step()
        net.step_graph(True)
        net.sync()
        _NETS[key] = (net, first, torch.empty(net.nparam).pin_memory().numpy())
    return _NETS[key]


def _batch(case, net, seed):
    g = _gen(1000 + seed)
    shape = (case["N"], 3, case["H"], case["W"])
    x = torch.randn(shape, generator=g, device="cuda") if "resnet" in case["kind"] else torch.rand(shape, generator=g, device="cuda")
    x = x.cpu().pin_memory().numpy()
    if case["kind"] == "stem_stage1":
        return x, None
    lshape = (case["N"],) + net.strip_shape[2:]
    classes = net.strip_shape[1]
    labels = []
    for r in range(case["strips"]):
        if "resnet" in case["kind"] and r:
            labels.append(labels[0])                # every strip's replica of the classifier scores the whole batch
            continue
        lab = torch.randint(0, classes, lshape, generator=g, device="cuda", dtype=torch.int32)
        labels.append(lab.cpu().pin_memory().numpy().view(np.uint32))
    return x, labels


def _prepare_net(case, seed):
    net, first, out = _net(case)
    net.set_params(first)
    x, labels = _batch(case, net, seed)
    return dict(net=net, x=x, labels=labels, params=out)


def _run_net(s):
    net = s["net"]
    net.load_input(s["x"])
    if s["labels"] is not None:
        for r, lab in enumerate(s["labels"]):
            net.set_labels(r, lab)
    net.step_graph(True)
    out = {}
    if s["labels"] is not None:
        total, n = net.loss()
        out["loss"] = total / n
    net.L.adh_net_get_params(net.h, 0, s["params"].ctypes.data_as(C.c_void_p))   # into pinned memory
    out["params"] = s["params"]
    return out


def _net_layers(case):
    """(C, K, k, P, Q, first) of every convolution of a net on the whole batch, and its activation elements and parameters."""
    N, H, W = case["N"], case["H"], case["W"]
    half = lambda v: (v - 1) // 2 + 1  # noqa: E731
    convs, acts = [], [0]

    def conv(ci, co, k, h, w, first=False):
        convs.append((ci, co, k, h, w, first))
        acts[0] += N * co * h * w

    kind = case["kind"]
    if kind == "parallel_resnet18":
        h, w = H, W
        conv(3, 64, 7, h, w, True)
        h, w = half(h), half(w)
        ci = 64
        for co, proj in [(64, 0), (64, 0), (128, 1), (128, 0), (256, 1), (256, 0), (512, 1), (512, 1)]:
            if proj:
                h, w = half(h), half(w)
                conv(ci, co, 1, h, w)
            conv(ci, co, 3, h, w)
            conv(co, co, 3, h, w)
            ci = co
        tail = 512 * 1000
    else:
        h, w = half(H), half(W)
        conv(3, 64, 7, h, w, True)
        h, w = half(h), half(w)
        ci = 64
        blocks = dict(stem_stage1=[3], segnet_small=[1, 1, 1, 1]).get(kind, [3, 4, 6, 3])
        strides = [1, 2, 1, 1] if kind.startswith("segnet") else [1, 2, 2, 2]
        for st, n in enumerate(blocks):
            b = 64 << st
            for i in range(n):
                ph, pw = h, w
                if i == 0:
                    if strides[st] == 2:
                        h, w = half(h), half(w)
                    conv(ci, 4 * b, 1, h, w)
                conv(ci, b, 1, ph, pw)
                conv(b, b, 3, h, w)
                conv(b, 4 * b, 1, h, w)
                ci = 4 * b
        tail = 0
        if kind.startswith("segnet"):
            conv(ci, 19, 1, h, w)
        elif kind == "parallel_resnet50":
            tail = 2048 * 1000
    flops = sum((2 if first else 3) * 2.0 * N * c * co * k * k * p * q for c, co, k, p, q, first in convs) + 6.0 * N * tail
    params = sum(c * co * k * k for c, co, k, _, _, _ in convs) + tail
    return flops, acts[0], params


def _work_net(case):
    flops, acts, params = _net_layers(case)
    es = 4 if case["mode"] == "f32" else 2
    # every convolution output written and read once forward, its gradient written and read once backward; parameters, gradients
    # and momentum read and written once; the host batch read once, the parameters returned once
    return dict(flops=flops, bytes=4.0 * acts * es + 6.0 * 4 * params + 4.0 * case["N"] * case["H"] * case["W"] * 4)


# ------------------------------------------------------------------ conv
def _conv_geo(case):
    """Input dims as the kernel reads them (a halo-padded strip for stride 1: pad rows and columns are in the buffer) and output dims."""
    p = case["dil"] * (case["k"] - 1) // 2
    H, W = case["H"] + 2 * p, case["W"] + 2 * p
    reach = case["dil"] * (case["k"] - 1) + 1
    return p, H, W, (H - reach) // case["stride"] + 1, (W - reach) // case["stride"] + 1


def _prepare_conv(case, seed):
    g = _gen(seed)
    dt = _torch_dtype(case["dtype"])
    f32 = case["dtype"] == "f32"
    N, ch, K, k = case["N"], case["C"], case["K"], case["k"]
    p, H, W, P, Q = _conv_geo(case)
    x = torch.zeros(_act(case["dtype"], N, ch, H, W), device="cuda", dtype=dt)
    inner = x[:, :, p:H - p, p:W - p] if f32 else x[:, p:H - p, p:W - p, :]
    inner.copy_(_uniform(g, tuple(inner.shape)))
    wshape = (K, ch, k, k) if f32 else (K, k, k, ch)
    s = dict(x=x, w=_normal(g, wshape, dt, math.sqrt(2.0 / (k * k * ch))), bias=_normal(g, (K,), std=0.1),
             dy=_uniform(g, _act(case["dtype"], N, K, P, Q), dt), y=torch.empty(_act(case["dtype"], N, K, P, Q), device="cuda", dtype=dt),
             dx=torch.zeros_like(x), dw=torch.empty(wshape, device="cuda"), db=torch.empty(K, device="cuda"))
    a = abi.Conv2dArgs()
    a.dtype, a.layout = (abi.AD_F32, abi.AD_NCHW) if f32 else (abi.AD_BF16, abi.AD_NHWC)
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, ch, H, W, K, k, k
    a.stride_h = a.stride_w = case["stride"]
    a.dil_h = a.dil_w = case["dil"]
    a.x, a.w = x.data_ptr(), s["w"].data_ptr()
    L = abi.lib()
    calls = []
    for i in range(3):
        b = abi.Conv2dArgs.from_buffer_copy(a)
        scratch = torch.zeros(max(16, L.ad_conv2d_scratch_bytes(C.byref(b), i)), dtype=torch.uint8, device="cuda")
        b.scratch, b.scratch_bytes = scratch.data_ptr(), scratch.numel()
        b.y = (s["y"] if i == 0 else s["dy"]).data_ptr()
        if i == 0:
            b.bias = s["bias"].data_ptr()
        elif i == 1:
            b.dx = s["dx"].data_ptr()
            if not f32 and p:                       # the pad columns of a gradient buffer are never read
                b.dx_col_begin, b.dx_col_count = p, case["W"]
        else:
            b.dw, b.db = s["dw"].data_ptr(), s["db"].data_ptr()
        calls.append((b, scratch))
    s["calls"] = calls
    return s


def _run_conv(s):
    L, st = abi.lib(), _stream()
    (f, _), (d, _), (w, _) = s["calls"]
    abi.check(L.ad_conv2d_fprop(C.byref(f), st))
    abi.check(L.ad_conv2d_dgrad(C.byref(d), st))
    abi.check(L.ad_conv2d_wgrad(C.byref(w), st))
    return [s["y"], s["dx"], s["dw"], s["db"]]


def _work_conv(case):
    _, H, W, P, Q = _conv_geo(case)
    N, ch, K, k = case["N"], case["C"], case["K"], case["k"]
    x, y, w = N * ch * H * W, N * K * P * Q, K * ch * k * k
    return dict(flops=6.0 * y * ch * k * k, bytes=_es(case) * (2.0 * x + 2.0 * y + w) + 4.0 * w + 8.0 * K)


# ------------------------------------------------------------------ bn
def _prepare_bn(case, seed):
    g = _gen(seed)
    dt = _torch_dtype(case["dtype"])
    ch = case["C"]
    shape = _act(case["dtype"], case["N"], ch, case["H"], case["W"])
    s = dict(x=_normal(g, shape, torch.float32).add_(0.3).to(dt), dy=_normal(g, shape, dt), gamma=_uniform(g, (ch,)).mul_(0.5).add_(1.0), beta=_normal(g, (ch,), std=0.2),
             relu=int(case["relu"]))
    s["y"], s["dx"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    for n in ("mean", "invstd", "var", "dgamma", "dbeta"):
        s[n] = torch.zeros(ch, device="cuda")
    s["scratch"] = torch.zeros(abi.lib().ad_bn_scratch_bytes(ch), dtype=torch.uint8, device="cuda")
    s["views"] = [_view(s[n]) for n in ("x", "y", "dy", "dx")]
    return s


def _run_bn(s):
    L, st = abi.lib(), _stream()
    x, y, dy, dx = s["views"]
    s["dgamma"].zero_()
    s["dbeta"].zero_()
    abi.check(L.ad_bn_fwd_train(C.byref(x), C.byref(y), _p(s["gamma"]), _p(s["beta"]), _p(s["mean"]), _p(s["invstd"]), _p(s["var"]), 1e-5, s["relu"],
                                _p(s["scratch"]), s["scratch"].numel(), st))
    abi.check(L.ad_bn_bwd(C.byref(x), C.byref(dy), C.byref(dx), _p(s["gamma"]), _p(s["beta"]), _p(s["mean"]), _p(s["invstd"]), _p(s["dgamma"]),
                          _p(s["dbeta"]), s["relu"], 0, _p(s["scratch"]), s["scratch"].numel(), st))
    return [s[n] for n in ("y", "mean", "invstd", "var", "dx", "dgamma", "dbeta")]


def _work_bn(case):
    n = case["N"] * case["C"] * case["H"] * case["W"]
    return dict(bytes=4.0 * n * _es(case) + 36.0 * case["C"], flops=14.0 * n)


# ------------------------------------------------------------------ halo
def _prepare_halo(case, seed):
    g = _gen(seed)
    dt = _torch_dtype(case["dtype"])
    R, p = case["R"], case["p"]
    shape = _act(case["dtype"], case["N"], case["C"], case["H"] // R + 2 * p, case["W"] + 2 * p)
    sides = []
    for _ in range(2):                              # the activations that are exchanged, the gradients that are summed back
        bufs = [_uniform(g, shape, dt) for _ in range(R)]
        a = abi.HaloArgs()
        a.dtype, a.layout = (abi.AD_F32, abi.AD_NCHW) if case["dtype"] == "f32" else (abi.AD_BF16, abi.AD_NHWC)
        a.halo_pad, a.base_width, a.base_height, a.num_channels, a.batch_size = p, case["W"], case["H"] // R, case["C"], case["N"]
        a.num_ranks, a.rank_first, a.rank_count, a.push = R, 0, R, 1
        for r in range(R):
            a.bufs[r] = bufs[r].data_ptr()
        sides.append((bufs, a))
    return dict(x=sides[0], g=sides[1])


def _run_halo(s):
    L, st = abi.lib(), _stream()
    abi.check(L.ad_halo_exchange(C.byref(s["x"][1]), st))
    abi.check(L.ad_halo_reduce(C.byref(s["g"][1]), st))
    return s["x"][0] + s["g"][0]


def _work_halo(case):
    rows = 2.0 * (case["R"] - 1) * case["N"] * case["C"] * case["p"] * case["W"]
    return dict(bytes=rows * _es(case) * 5, flops=rows)


# ------------------------------------------------------------------ head
def _prepare_head(case, seed):
    g = _gen(seed)
    dt = _torch_dtype(case["dtype"])
    N, ch, H, W, sc = (case[n] for n in ("N", "C", "H", "W", "scale"))
    low, full = _act(case["dtype"], N, ch, H, W), _act(case["dtype"], N, ch, H * sc, W * sc)
    s = dict(low=_normal(g, low, dt, 2.0), logits=torch.empty(full, device="cuda", dtype=dt), dlogits=torch.empty(full, device="cuda", dtype=dt),
             dlow=torch.empty(low, device="cuda", dtype=dt), loss=torch.empty(N, H * sc * W * sc, device="cuda"),
             labels=torch.randint(0, ch, (N, H * sc * W * sc), generator=g, device="cuda", dtype=torch.int32),
             dloss=torch.full((N, H * sc * W * sc), 1.0 / (N * H * sc * W * sc), device="cuda"), case=case)
    s["views"] = [_view(s[n]) for n in ("low", "logits", "dlogits", "dlow")]
    s["fmt"] = (abi.AD_F32, abi.AD_NCHW) if case["dtype"] == "f32" else (abi.AD_BF16, abi.AD_NHWC)
    return s


def _run_head(s):
    L, st = abi.lib(), _stream()
    case = s["case"]
    low, logits, dlogits, dlow = s["views"]
    dt, lay = s["fmt"]
    hw = s["loss"].shape[1]
    abi.check(L.ad_upsample_bilinear_fwd(C.byref(low), C.byref(logits), case["scale"], 0, case["H"], 0, st))
    abi.check(L.ad_softmax_ce_pixel_fwd(dt, lay, case["N"], case["C"], hw, _p(s["logits"]), _p(s["labels"]), _p(s["loss"]), None, st))
    abi.check(L.ad_softmax_ce_pixel_bwd(dt, lay, case["N"], case["C"], hw, _p(s["logits"]), _p(s["labels"]), _p(s["dloss"]), _p(s["dlogits"]), 0, st))
    abi.check(L.ad_upsample_bilinear_bwd(C.byref(dlogits), C.byref(dlow), case["scale"], 0, case["H"], 0, 0, st))
    return [s[n] for n in ("logits", "loss", "dlogits", "dlow")]


def _work_head(case):
    n = case["N"] * case["C"] * case["H"] * case["W"]
    px = case["N"] * case["H"] * case["W"] * case["scale"] ** 2
    # low-resolution logits in, full logits, losses, full gradients and low-resolution gradients out; labels and weights in
    return dict(bytes=_es(case) * (2.0 * n + 2.0 * n * case["scale"] ** 2) + 12.0 * px, flops=30.0 * n * case["scale"] ** 2)


# ------------------------------------------------------------------ pool
def _pool_window(case):
    kh, kw = (case["k"], case["k"]) if case["k"] else (case["H"], case["W"])
    return kh, kw, case["stride"], case["stride"]


def _prepare_pool(case, seed):
    g = _gen(seed)
    dt = _torch_dtype(case["dtype"])
    kh, kw, sh, sw = _pool_window(case)
    P, Q = (case["H"] - kh) // sh + 1, (case["W"] - kw) // sw + 1
    x = _normal(g, _act(case["dtype"], case["N"], case["C"], case["H"], case["W"]), dt).clamp_(min=0)      # after a ReLU
    y = torch.empty(_act(case["dtype"], case["N"], case["C"], P, Q), device="cuda", dtype=dt)
    s = dict(x=x, y=y, dy=_normal(g, tuple(y.shape), dt), dx=torch.empty_like(x), win=(kh, kw, sh, sw), avg=case["pooling"] == "avg")
    s["views"] = [_view(s[n]) for n in ("x", "y", "dy", "dx")]
    return s


def _run_pool(s):
    L, st = abi.lib(), _stream()
    x, y, dy, dx = s["views"]
    if s["avg"]:
        abi.check(L.ad_avgpool2d_fwd(C.byref(x), C.byref(y), *s["win"], st))
        abi.check(L.ad_avgpool2d_bwd(C.byref(dy), C.byref(dx), *s["win"], 0, st))
    else:
        abi.check(L.ad_maxpool2d_fwd(C.byref(x), C.byref(y), *s["win"], st))
        abi.check(L.ad_maxpool2d_bwd(C.byref(x), C.byref(dy), C.byref(dx), *s["win"], 0, st))
    return [s["y"], s["dx"]]


def _work_pool(case):
    kh, kw, sh, sw = _pool_window(case)
    n = case["N"] * case["C"] * case["H"] * case["W"]
    m = case["N"] * case["C"] * ((case["H"] - kh) // sh + 1) * ((case["W"] - kw) // sw + 1)
    return dict(bytes=_es(case) * (2.0 * n + 2.0 * m), flops=2.0 * m * kh * kw)


# ------------------------------------------------------------------ entry points
def prepare(case, seed):
    return dict(op=case["op"], state=globals()["_prepare_" + case["op"]](case, seed))


def run(state):
    return globals()["_run_" + state["op"]](state["state"])


def work(case):
    return globals()["_work_" + case["op"]](case)


def tolerance(case):
    op = case["op"]
    if op == "net":
        # loss and parameters after one or two updates through 10 to 50 normalised layers, each of which amplifies rounding
        return {"rel": 2e-4, "max": 0.05} if case["mode"] == "f32" else {"rel": 1e-2, "max": 0.5}
    if op == "halo":
        return "exact"
    if case["dtype"] == "f32":
        # fp32 sums over up to some millions of terms
        return {"rel": 2e-5, "max": 2e-3}
    return {"rel": 4e-3, "max": 0.2}                # bf16 results: a rounding step apart now and then
