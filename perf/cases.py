"""The work a user of this framework has it do, as timed cases over its public entry points.

Two ways in are covered. A *session* case is what a SOFIE user's program does: the model is parsed and generated once, the
emitted Session is constructed once, and every pass is one `infer()` from a host array to a host array, so the upload, the
kernels and the read-back all belong to the pass. A *device* case is what a program does that keeps its tensors on the GPU and
calls the operators of the C ABI one after the other through `sofie_b200.ops`.

Models, layer sizes and data come from `sofie_b200/configs.py` (the weights are seeded there and stay the same, as a trained
network's do; the inputs follow the seed of the state). Batches run from one event to the largest batch the benchmark uses.
"""
from __future__ import annotations

import functools
import hashlib
import os
import tempfile
from pathlib import Path

import numpy as np
import torch

from sofie_b200 import capi, configs, generated, ops

NHWC = capi.LAYOUT_NHWC
DYNAMIC_ROOM = 4096     # samples a Session with a run-time batch is constructed for
FP8_WIDTH, FP8_LAYERS = 4096, 4

# model -> (builder, smallest and largest batch a session case draws, floats returned per sample)
MODELS = {
    "mlp_f32": (configs.mlp_f32, 1, 1 << 18),
    "cnn_f32": (configs.cnn_f32, 1, 8192),
    "mlp_i8": (configs.mlp_i8, 1, 1 << 15),
    "cnn_i8": (configs.cnn_i8, 1, 16384),
    "fp8_chain": (configs.gemm_chain_fp8, 16, 8192),
    "resblock_f32": (configs.resblock_f32, 1, 4096),
    "upsample_f32": (functools.partial(configs.upsample_f32, channels=(32, 16)), 1, 1024),
}
DYNAMIC = ("mlp_f32", "cnn_f32", "mlp_i8", "cnn_i8")


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # event-by-event inference: one sample per call, the call SOFIE was written for; latency only
        dict(name="session mlp_f32 b1", kind="session", model="mlp_f32", batch=1, dynamic=False, pinned=False),
        # the fp32 perceptron at the batch of its configuration: still launch-latency sized
        dict(name="session mlp_f32 b1024", kind="session", model="mlp_f32", batch=1024, dynamic=False, pinned=False),
        # a program whose number of events per call varies: the run-time batch Session at an odd batch, from pinned memory
        dict(name="session cnn_f32 dyn b1003", kind="session", model="cnn_f32", batch=1003, dynamic=True, pinned=True),
        # a decoder: transposed convolutions and activations on a small batch
        dict(name="session upsample_f32 b64", kind="session", model="upsample_f32", batch=64, dynamic=False, pinned=False),
        # the quantised perceptron at the batch of its configuration
        dict(name="session mlp_i8 b8192", kind="session", model="mlp_i8", batch=8192, dynamic=False, pinned=False),
        # the quantised calorimeter CNN at the batch of its configuration: the benchmark's headline, 268 MB of floats per call
        dict(name="session cnn_i8 b16384", kind="session", model="cnn_i8", batch=16384, dynamic=False, pinned=False),
        # the FP8 chain from host to host: as many floats come back as go in
        dict(name="session fp8_chain b8192", kind="session", model="fp8_chain", batch=8192, dynamic=False, pinned=False),
        # the operators below are called on tensors that are on the device already
        # the fp32 CNN at the benchmark's large batch: convolutions with fused Relu and pooling, then the classifier
        dict(name="device cnn_f32 b8192", kind="cnn_f32", batch=8192),
        # the quantised CNN: QuantizeLinear, four fused convolutions, two products, DequantizeLinear
        dict(name="device cnn_i8 b16384", kind="cnn_i8", batch=16384),
        # the FP8 chain at the rows of its configuration: the largest contraction there is
        dict(name="device fp8_chain b65536", kind="fp8_chain", batch=65536),
        # one Gemm of ragged sizes with every option of the ONNX operator in use
        dict(name="device gemm_f32 ragged", kind="gemm_f32", M=1000, N=777, K=1333, transA=True, transB=False, bias=2, relu=True),
        # the memory-bound operators one after the other on an image tensor and a table of class scores
        dict(name="device pointwise", kind="pointwise", N=512, C=16, H=64, W=64, rows=32768, classes=1000),
    ]


def _log_int(rng, low, high):
    """An integer spread over the logarithm of [low, high]; every size in between can come, odd ones as often as even ones."""
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    kind = rng.choice(["session", "session", "session", "cnn_f32", "cnn_i8", "fp8_chain", "gemm_f32", "gemm_f32", "pointwise"])
    if kind == "session":
        model = rng.choice(sorted(MODELS))
        _, low, high = MODELS[model]
        dynamic = model in DYNAMIC and rng.random() < 0.4
        return dict(kind="session", model=model, batch=_log_int(rng, low, min(high, DYNAMIC_ROOM) if dynamic else high),
                    dynamic=dynamic, pinned=rng.random() < 0.3)
    if kind == "cnn_f32":
        return dict(kind=kind, batch=_log_int(rng, 1, 8192))
    if kind == "cnn_i8":
        return dict(kind=kind, batch=_log_int(rng, 1, 16384))
    if kind == "fp8_chain":
        return dict(kind=kind, batch=_log_int(rng, 16, 65536))
    if kind == "gemm_f32":
        while True:
            M, N, K = _log_int(rng, 1, 16384), _log_int(rng, 1, 4096), _log_int(rng, 8, 4096)
            if M * N * K <= 2 ** 35:
                break
        return dict(kind=kind, M=M, N=N, K=K, transA=rng.random() < 0.3, transB=rng.random() < 0.5, bias=rng.choice([0, 1, 1, 2]),
                    relu=rng.random() < 0.5)
    C, H, W = rng.choice([1, 3, 8, 16, 24, 32, 64]), _log_int(rng, 6, 96), _log_int(rng, 6, 96)
    classes = _log_int(rng, 2, 2000)
    return dict(kind=kind, N=_log_int(rng, 1, max(1, 2 ** 25 // (C * H * W))), C=C, H=H, W=W,
                rows=_log_int(rng, 1, max(1, 2 ** 25 // classes)), classes=classes)


# ------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _input(model, shape, seed):
    """N(0,1) for every network but the calorimeter CNN, which sees Exp(1) energies in 5 % of its cells and zeros elsewhere."""
    g = _generator(seed)
    if model != "cnn_i8":
        return torch.randn(shape, device="cuda", generator=g)
    x = torch.empty(shape, device="cuda").exponential_(1.0, generator=g)
    return x * (torch.rand(shape, device="cuda", generator=g) < 0.05)


def _to_host(x, pinned):
    """The array a program passes to infer(): ordinary memory, or memory it pinned itself."""
    if not pinned:
        return x.cpu().numpy()
    return torch.empty(x.shape, pin_memory=True).copy_(x).numpy()


# ------------------------------------------------------------------------------------ sessions
@functools.lru_cache(maxsize=None)
def _fp8_model():
    """The FP8 chain without its rows: the 67 million weights do not depend on them, and neither do the calibrated scales."""
    m, x = configs.gemm_chain_fp8(rows=512)
    return m, configs.calibrate_fp8_scales(m, x)


def _model(model, batch):
    if model == "fp8_chain":
        m, scales = _fp8_model()
        m.name, m.input_shape = f"gemm_chain_fp8_m{batch}", (batch, FP8_WIDTH)
        return m, scales
    return MODELS[model][0](batch=batch, with_input=False)[0], None


@functools.lru_cache(maxsize=None)
def _session(model, batch):
    """The Session a program constructs once; batch 0 is the one with a run-time batch."""
    written = (generated.ROOT, generated.LIBDIR, generated.LIBDIR / ".generator.lock")
    if not all(os.access(p, os.W_OK) for p in written if p.exists()):
        # an installation this user may only read: its generator is built, and what it emits goes to a temporary folder
        here = hashlib.sha1(str(generated.ROOT).encode()).hexdigest()[:12]
        generated._generator_built, generated.WORK = True, Path(tempfile.gettempdir()) / f"sofie_sessions_{os.getuid()}_{here}"
    if not batch:
        return generated.dynamic_session_from_model(_model(model, DYNAMIC_ROOM)[0], f"{model}_dyn", DYNAMIC_ROOM)
    m, scales = _model(model, batch)
    return generated.session_from_model(m, f"{model}_b{batch}", binary=model == "fp8_chain", fp8_scales=scales)


def _shape(model, batch):
    return (batch,) + {"mlp_f32": (64,), "cnn_f32": (3, 32, 32), "mlp_i8": (512,), "cnn_i8": (1, 64, 64), "fp8_chain": (FP8_WIDTH,),
                       "resblock_f32": (8, 16, 16), "upsample_f32": (3, 12, 12)}[model]


# ------------------------------------------------------------------------------------ weights of the device cases
def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@functools.lru_cache(maxsize=None)
def _cnn_f32_weights():
    m, _ = configs.cnn_f32(batch=1, with_input=False)
    w = {f"c{i}": (ops.conv2d_pack_f32(_dev(m.weights[f"cw{i}"])), _dev(m.weights[f"cb{i}"])) for i in range(3)}
    # the classifier reads the channel-last feature map: its columns are reordered once
    w["fc"] = (_dev(m.weights["fw"].reshape(10, 64, 8, 8).transpose(0, 2, 3, 1).reshape(10, 4096)), _dev(m.weights["fb"]))
    return w


@functools.lru_cache(maxsize=None)
def _cnn_i8_weights():
    m, _ = configs.cnn_i8(batch=1, with_input=False)
    s, w, x_scale = configs.CALO_SCALES, {}, configs.CALO_SCALES["x"]
    for i in range(4):
        W = m.weights[f"cw{i}"]
        mult, _ = ops.qlinear_prepare(W.reshape(W.shape[0], -1), True, x_scale, 0, m.weights[f"cs{i}"], s[f"c{i}"], None, "cuda")
        w[f"c{i}"] = (ops.qconv2d_pack_i8(_dev(W)), mult)
        x_scale = s[f"c{i}"]
    for i in range(2):
        W = m.weights[f"fw{i}"]
        if i == 0:  # the first product reads the channel-last feature map
            W = W.reshape(128, 4, 4, -1).transpose(1, 2, 0, 3).reshape(2048, -1)
        W = np.ascontiguousarray(W.T)
        w[f"f{i}"] = (_dev(W),) + ops.qlinear_prepare(W, True, x_scale, 0, m.weights[f"fs{i}"], s[f"f{i}"], None, "cuda")
        x_scale = s[f"f{i}"]
    return w


@functools.lru_cache(maxsize=None)
def _fp8_weights():
    g, layers = _generator(20260004), []
    sigma = 1.0
    for i in range(FP8_LAYERS):
        W = torch.randn((FP8_WIDTH, FP8_WIDTH), device="cuda", generator=g) * 0.02
        w_scale = 5.5 * 0.02 / 448
        bias = torch.randn(FP8_WIDTH, device="cuda", generator=g) * 0.02
        layers.append((ops.quantize_e4m3(W, w_scale), bias, w_scale, 6 * sigma / 448))
        # standard deviation of the next layer's input: 64 * 0.02 times this one's, and after Relu half the power
        sigma *= 64 * 0.02 * (1.0 if i == 0 else 0.5 ** 0.5)
    return layers


# ------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "session":
        model, batch = case["model"], case["batch"]
        x = _to_host(_input(model, _shape(model, batch), seed), case["pinned"])
        return dict(kind=kind, session=_session(model, 0 if case["dynamic"] else batch), x=x)
    if kind == "cnn_f32":
        return dict(kind=kind, x=_input(kind, (case["batch"], 3, 32, 32), seed), w=_cnn_f32_weights())
    if kind == "cnn_i8":
        return dict(kind=kind, x=_input(kind, (case["batch"], 1, 64, 64), seed), w=_cnn_i8_weights())
    if kind == "fp8_chain":
        return dict(kind=kind, x=_input(kind, (case["batch"], FP8_WIDTH), seed), w=_fp8_weights())
    g = _generator(seed)

    def rand(*shape):
        return torch.randn(shape, device="cuda", generator=g)
    if kind == "gemm_f32":
        M, N, K = case["M"], case["N"], case["K"]
        A = rand(K, M) if case["transA"] else rand(M, K)
        B = (rand(N, K) if case["transB"] else rand(K, N)) * K ** -0.5
        C = {0: None, 1: rand(N), 2: rand(M, N)}[case["bias"]]
        return dict(kind=kind, A=A, B=B, C=C, transA=int(case["transA"]), transB=int(case["transB"]), relu=case["relu"])
    N, C, H, W = case["N"], case["C"], case["H"], case["W"]
    return dict(kind=kind, x=rand(N, C, H, W), skip=rand(N, C, H, W), gain=rand(C, 1, 1), scale=rand(C).abs() + 0.5, shift=rand(C), mean=rand(C),
                scores=rand(case["rows"], case["classes"]))


# ------------------------------------------------------------------------------------ run
def run(state):
    return _RUN[state["kind"]](state)


def _run_session(s):
    return s["session"].infer(s["x"])


def _run_cnn_f32(s):
    w, n = s["w"], s["x"].shape[0]
    t = ops.conv2d_f32(s["x"], *w["c0"], pad=(1, 1), relu=True, y_layout=NHWC, w_packed=True, kernel=(3, 3))
    t = ops.conv2d_f32(t, *w["c1"], shape=(n, 16, 32, 32), pad=(1, 1), relu=True, pool=2, x_layout=NHWC, y_layout=NHWC, w_packed=True, kernel=(3, 3))
    t = ops.conv2d_f32(t, *w["c2"], shape=(n, 32, 16, 16), pad=(1, 1), relu=True, pool=2, x_layout=NHWC, y_layout=NHWC, w_packed=True, kernel=(3, 3))
    return ops.gemm_f32(t.view(n, 4096), *w["fc"], transB=1)


def _run_cnn_i8(s):
    w, n, hw, c = s["w"], s["x"].shape[0], 64, 1
    t = ops.quantize_u8(s["x"], configs.CALO_SCALES["x"], 0)
    for i, cout in enumerate((32, 64, 64, 128)):
        t = ops.qlinear_conv2d(t, *w[f"c{i}"], shape=(n, c, hw, hw), pad=(1, 1), relu=True, pool=2,
                               x_layout=NHWC, y_layout=NHWC, w_packed=True, kernel=(3, 3))
        hw, c = hw // 2, cout
    t = ops.qlinear_matmul(t.view(n, 2048), *w["f0"], relu=True)
    return ops.qlinear_matmul_f32(t, *w["f1"], configs.CALO_SCALES["f1"], y_zp=128)


def _run_fp8_chain(s):
    w = s["w"]
    q = ops.quantize_e4m3(s["x"], w[0][3])
    for i, (W, bias, w_scale, a_scale) in enumerate(w):
        last = i == len(w) - 1
        y, q = ops.gemm_e4m3(q, W, bias, a_scale=a_scale, w_scale=w_scale, relu=not last, q_scale=0.0 if last else w[i + 1][3], want_bf16=last)
    return y


def _run_gemm_f32(s):
    return ops.gemm_f32(s["A"], s["B"], s["C"], transA=s["transA"], transB=s["transB"], alpha=0.75, beta=1.5, relu=s["relu"])


def _run_pointwise(s):
    x = s["x"]
    N, C, H, W = x.shape
    q = ops.quantize_u8(x, 0.02, 128)
    return dict(relu=ops.relu_f32(x), sigmoid=ops.unary_f32(x, "Sigmoid"), add=ops.binary_f32(x, s["skip"], "Add"), mul=ops.binary_f32(x, s["gain"], "Mul"),
                norm=ops.batchnorm_f32(x, s["scale"], s["shift"], s["mean"], N, C, H * W), pool=ops.pool2d_f32(x), nhwc=ops.nchw_to_nhwc(x),
                q=q, dq=ops.dequantize_u8(q, 0.02, 128), e4m3=ops.quantize_e4m3(x, 0.01), softmax=ops.softmax_f32(s["scores"]))


_RUN = dict(session=_run_session, cnn_f32=_run_cnn_f32, cnn_i8=_run_cnn_i8, fp8_chain=_run_fp8_chain, gemm_f32=_run_gemm_f32,
            pointwise=_run_pointwise)


# ------------------------------------------------------------------------------------ work and tolerance
# per sample: floats in, floats out, operations of the contractions (2 x M x N x K); bytes of all weights
_NETWORKS = {
    "mlp_f32": (64, 10, 2 * (64 * 128 + 128 * 128 + 128 * 10), 4 * (64 * 128 + 128 * 128 + 128 * 10)),
    "cnn_f32": (3072, 10, 2 * (1024 * 16 * 27 + 1024 * 32 * 144 + 256 * 64 * 288 + 40960), 4 * (16 * 27 + 32 * 144 + 64 * 288 + 40960)),
    "mlp_i8": (512, 256, 2 * (512 * 1024 + 1024 * 1024 + 1024 * 256), 512 * 1024 + 1024 * 1024 + 1024 * 256),
    "cnn_i8": (4096, 2, 2 * (4096 * 32 * 9 + 1024 * 64 * 288 + 256 * 64 * 576 + 64 * 128 * 576 + 2048 * 256 + 512),
               32 * 9 + 64 * 288 + 64 * 576 + 128 * 576 + 2048 * 256 + 512),
    "fp8_chain": (FP8_WIDTH, FP8_WIDTH, 2 * FP8_LAYERS * FP8_WIDTH ** 2, FP8_LAYERS * FP8_WIDTH ** 2),
    "resblock_f32": (2048, 10, 2 * 256 * 16 * 9 * 24 + 20480, 4 * (16 * 9 * 24 + 10240)),
    "upsample_f32": (432, 3 * 48 * 48, 2 * 144 * (32 * 27 + 32 * 16 * 4 + 4 * 16 * 27), 4 * (32 * 27 + 32 * 16 * 4 + 16 * 27)),
}


def work(case):
    kind = case["kind"]
    if kind == "gemm_f32":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 4 * (M * K + K * N + M * N + (0, N, M * N)[case["bias"]]), "flops": 2 * M * N * K}
    if kind == "pointwise":
        n, scores = case["N"] * case["C"] * case["H"] * case["W"], case["rows"] * case["classes"]
        pooled = case["N"] * case["C"] * (case["H"] // 2) * (case["W"] // 2)
        # read and written by each operator: relu 8, sigmoid 8, add 12, mul 8, batch norm 8, layout 8, quantise 5, dequantise 5, e4m3 5, pool 4 + output
        return {"bytes": 71 * n + 4 * pooled + 8 * scores, "flops": 0}
    n_in, n_out, flops, weights = _NETWORKS[case["model"] if kind == "session" else kind]
    out_bytes = 2 if kind == "fp8_chain" else 4   # on the device the chain ends in bfloat16
    return {"bytes": case["batch"] * (4 * n_in + out_bytes * n_out) + weights, "flops": case["batch"] * flops}


def tolerance(case):
    network = case["model"] if case["kind"] == "session" else case["kind"]
    if network in ("mlp_i8", "cnn_i8"):
        return "exact"                      # int32 sums and a fixed rounding rule: one right answer
    if network == "fp8_chain":
        return {"rel": 1e-2}                # a sum in another order can land on the other side of an E4M3 step; bfloat16 result
    if network == "pointwise":
        return {"rel": 1e-6, "differ": 0.0}  # a few ulp of an exponential; bytes stay the same
    return {"rel": 1e-5}                    # float32 sums in another order
