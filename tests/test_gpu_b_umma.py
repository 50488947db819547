"""GPU parity of the tcgen05 / TMEM / TMA GEMM kernels (engine forced to the tensor-core family, so a
shape the kernel does not take fails instead of silently running on CUDA cores).
fp32 (3xTF32): tensor-relative error <= 1e-5 against the oracle; int8: bit-exact; FP8: <= 2e-2."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import rel_err
from oracle import cpu_oracle as o
from sofie_b200 import capi, ops

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def umma_engine(cuda_device):
    ops.set_engine(capi.ENGINE_TCGEN05)
    yield
    ops.set_engine(0)
    ctx = C.c_void_p()
    capi.call("sofie_cuda_ctx_create", C.byref(ctx), 0, 0)
    try:
        capi.call("sofie_cuda_ctx_check", ctx)  # no kernel gave up on a wait
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("M,N,K,bias,relu", [(128, 128, 32, 0, 0), (128, 128, 128, 1, 1), (1024, 128, 64, 1, 1),
                                             (1024, 10, 128, 1, 0), (300, 72, 260, 2, 1), (1, 7, 4, 0, 0),
                                             (256, 10, 4096, 1, 0), (513, 384, 1000, 1, 1), (4096, 256, 512, 1, 1)])
def test_gemm_f32_3xtf32(M, N, K, bias, relu):
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    Cb = None if bias == 0 else rng.standard_normal((N,) if bias == 1 else (M, N)).astype(np.float32)
    ref = o.gemm_f32(A, B, Cb, transB=1, alpha=1.25, beta=0.5, relu=bool(relu))
    y = ops.gemm_f32(dev(A), dev(B), None if Cb is None else dev(Cb), transB=1, alpha=1.25, beta=0.5, relu=bool(relu))
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert rel_err(y.cpu().numpy(), ref) <= 1e-5


# every way an operand can lie (rows of 16-byte multiples or not, K or the rows contiguous, an unaligned base) at the edges of the
# tiles (32 / 64 / 128 columns, 128 rows, 32 of K), one cluster rank to eight, several tiles per CTA, more than one promoted unit
@pytest.mark.parametrize("M,N,K,tA,tB,bias", [(129, 33, 31, 0, 1, 1), (127, 31, 33, 1, 0, 2), (128, 64, 32, 1, 1, 0), (200, 65, 4100, 0, 0, 1), (33, 1000, 2501, 1, 1, 1),
                                              (1, 130, 1025, 0, 1, 2), (1000, 777, 1333, 1, 0, 2), (2500, 1029, 289, 0, 0, 1), (5000, 512, 270, 0, 1, 1),
                                              (1300, 2050, 515, 1, 0, 1), (40000, 72, 64, 0, 1, 1), (64, 129, 257, 0, 1, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_gemm_f32_any_layout(M, N, K, tA, tB, bias, offset):
    rng = np.random.default_rng(M + N + K)

    def place(a):     # `offset` floats behind a 16-byte boundary
        buf = torch.empty(a.size + 4, device="cuda")
        v = buf[offset: offset + a.size].view(a.shape)
        v.copy_(torch.from_numpy(a))
        return v
    A = rng.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    Cb = None if bias == 0 else rng.standard_normal((N,) if bias == 1 else (M, N)).astype(np.float32)
    ref = o.gemm_f32(A, B, Cb, transA=tA, transB=tB, alpha=1.25, beta=0.5, relu=True)
    out = place(np.full((M, N), np.nan, np.float32))
    y = ops.gemm_f32(place(A), place(B), None if Cb is None else place(Cb), transA=tA, transB=tB, alpha=1.25, beta=0.5, relu=True, out=out)
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert rel_err(y.cpu().numpy(), ref) <= 1e-5


def test_gemm_f32_shape_outside_tensor_core_kernel_is_refused_when_forced():
    A, B = torch.zeros((8, 6), device="cuda"), torch.zeros((4, 6), device="cuda")   # K*4 not a multiple of 16
    with pytest.raises(capi.SofieCudaError) as e:
        ops.gemm_f32(A, B, transB=1)
    assert e.value.status == capi.ERR_UNSUPPORTED
    ops.set_engine(0)  # automatic: the CUDA-core kernel takes it
    ops.gemm_f32(A, B, transB=1)
    assert ops.last_engine() == capi.ENGINE_SIMT


@pytest.mark.parametrize("M,N,K,relu,zp", [(128, 32, 128, 0, 128), (8192 // 8, 1024, 512, 0, 128), (100, 40, 48, 1, 3),
                                           (700, 256, 2048, 1, 0), (257, 2, 256, 0, 128), (130, 1000, 1024, 0, 128)])
def test_qlinear_matmul_tcgen05_bit_exact(M, N, K, relu, zp):
    rng = np.random.default_rng(N + K)
    A = rng.integers(0, 256, (M, K)).astype(np.uint8)
    W = rng.integers(-127, 128, (N, K)).astype(np.int8)
    ws = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y_scale = 0.02 * np.sqrt(K) * 0.3
    ref = o.qlinear_matmul(A, 0.02, zp, W, ws, y_scale, 128, w_is_nk=True, relu=bool(relu))
    mult, corr = ops.qlinear_prepare(W, True, 0.02, zp, ws, y_scale, None, "cuda")
    y = ops.qlinear_matmul(dev(A), dev(W), mult, corr, w_is_nk=True, y_zp=128, relu=bool(relu)).cpu().numpy()
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert np.array_equal(y, ref)
    assert len(np.unique(ref)) > 20


# few tiles and a long K: four or two CTAs of a cluster share a tile of 64, 128 or 256 columns; ranks with uneven parts of K (17 and 33
# stages), with no columns of their own (64 columns, four ranks) and with columns beyond N
@pytest.mark.parametrize("M,N,K", [(5, 70, 2096), (257, 64, 4096), (130, 300, 4112), (128, 4096, 4096), (300, 4090, 4112),
                                   # rows that are stored value by value: K shared for the sake of the stores, two rounds of narrow tiles
                                   (1009, 131, 768), (340, 1919, 1744), (723, 1855, 96)])
def test_8_bit_products_that_share_k(M, N, K):
    rng = np.random.default_rng(M + N + K)
    A, W = rng.integers(0, 256, (M, K)).astype(np.uint8), rng.integers(-127, 128, (N, K)).astype(np.int8)
    acc = (A.astype(np.float64) @ W.astype(np.float64).T).astype(np.int64)     # exact: below 2^53
    ws = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y_scale = 0.02 * np.sqrt(K) * 0.3
    mult, corr = ops.qlinear_prepare(W, True, 0.02, 3, ws, y_scale, None, "cuda")
    ref = (acc - 3 * W.sum(1, dtype=np.int64)).astype(np.float32) * mult.cpu().numpy()
    ref = np.clip(np.rint(ref) + 128, 0, 255).astype(np.uint8)
    y = ops.qlinear_matmul(dev(A), dev(W), mult, corr, w_is_nk=True, y_zp=128)
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert np.array_equal(y.cpu().numpy(), ref) and len(np.unique(ref)) > 20
    Aq = o.quantize_e4m3(rng.standard_normal((M, K)).astype(np.float32), 0.01)
    Wq = o.quantize_e4m3(rng.standard_normal((N, K)).astype(np.float32), 0.01)
    bias = rng.standard_normal(N).astype(np.float32)
    Y, Yq = ops.gemm_e4m3(dev(Aq), dev(Wq), dev(bias), a_scale=0.01, w_scale=0.01, q_scale=0.05)
    table = torch.arange(256, dtype=torch.uint8).view(torch.float8_e4m3fn).double().numpy()
    a, w = table[Aq] * 0.01, table[Wq] * 0.01
    exact, size = a @ w.T + bias, np.abs(a) @ np.abs(w).T + np.abs(bias)
    # one rounding to bfloat16 of a sum whose tensor-core additions (32 of K each) truncate
    assert (np.abs(Y.double().cpu().numpy() - exact) <= 2.0 ** -8 * np.abs(exact) + (K / 32 + 8) * 2.0 ** -23 * size).all()
    assert np.array_equal(Yq.cpu().numpy(), o.quantize_e4m3(Y.float().cpu().numpy(), 0.05))


# up to 80 rows only those are copied: one, eight, a group of eight begun, the last count of the kind and the first beyond, at each tile width and cluster size
@pytest.mark.parametrize("M,N,K", [(1, 64, 4096), (8, 70, 2096), (9, 4090, 4112), (33, 4096, 4096), (80, 8190, 4096), (17, 16300, 4096), (81, 4096, 4096),
                                   (100, 4480, 2048), (130, 2176, 4096)])   # and 140 and 136 CTAs in fours, for which not every card has room at a time
def test_8_bit_products_of_few_rows_that_share_k(M, N, K):
    test_8_bit_products_that_share_k(M, N, K)


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (70, 45, 144), (1000, 512, 4096), (256, 4096, 512)])
def test_gemm_e4m3_tcgen05(M, N, K):
    rng = np.random.default_rng(K + M)
    X = rng.standard_normal((M, K)).astype(np.float32)
    Wf = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float32)
    sa, sw = float(np.abs(X).max() / 448), float(np.abs(Wf).max() / 448)
    Aq, Wq = o.quantize_e4m3(X, sa), o.quantize_e4m3(Wf, sw)
    ref = o.bf16_bits_to_f32(o.gemm_e4m3(Aq, sa, Wq, sw, bias, relu=True))
    Y, Yq = ops.gemm_e4m3(dev(Aq), dev(Wq), dev(bias), a_scale=sa, w_scale=sw, relu=True, q_scale=0.01)
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    y = Y.float().cpu().numpy()
    assert rel_err(y, ref) <= 2e-2
    assert rel_err(y, ref) <= 8e-3
    assert np.array_equal(Yq.cpu().numpy(), o.quantize_e4m3(y, 0.01))


def test_tensor_core_and_cuda_core_kernels_agree():
    rng = np.random.default_rng(11)
    A = rng.standard_normal((640, 256)).astype(np.float32)
    B = rng.standard_normal((192, 256)).astype(np.float32)
    y_tc = ops.gemm_f32(dev(A), dev(B), transB=1).cpu().numpy()
    ops.set_engine(capi.ENGINE_SIMT)
    y_cc = ops.gemm_f32(dev(A), dev(B), transB=1).cpu().numpy()
    assert rel_err(y_tc, y_cc) <= 1e-5


# Shapes with at least 296 tiles of 256 x 256 run on CTA pairs (cta_group::2); ragged M and N included.
@pytest.mark.parametrize("M,N,K,relu,zp", [(19000, 1000, 256, 1, 128), (2048 * 19, 512, 128, 0, 7)])
def test_qlinear_matmul_pair_kernel_bit_exact(M, N, K, relu, zp):
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(0, 256, (M, K)).astype(np.uint8)
    W = rng.integers(-127, 128, (N, K)).astype(np.int8)
    ws = rng.uniform(0.001, 0.01, N).astype(np.float32)
    y_scale = 0.02 * np.sqrt(K) * 0.3
    ref = o.qlinear_matmul(A, 0.02, zp, W, ws, y_scale, 128, w_is_nk=True, relu=bool(relu))
    mult, corr = ops.qlinear_prepare(W, True, 0.02, zp, ws, y_scale, None, "cuda")
    for _ in range(2):  # a second launch reuses the barriers' initial state and TMEM
        y = ops.qlinear_matmul(dev(A), dev(W), mult, corr, w_is_nk=True, y_zp=128, relu=bool(relu)).cpu().numpy()
        assert ops.last_engine() == capi.ENGINE_TCGEN05
        assert np.array_equal(y, ref)
    assert len(np.unique(ref)) > 20


def test_gemm_e4m3_pair_kernel():
    M, N, K = 19200, 1024, 256
    rng = np.random.default_rng(3)
    X = rng.standard_normal((M, K)).astype(np.float32)
    Wf = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float32)
    sa, sw = float(np.abs(X).max() / 448), float(np.abs(Wf).max() / 448)
    Aq, Wq = o.quantize_e4m3(X, sa), o.quantize_e4m3(Wf, sw)
    ref = o.bf16_bits_to_f32(o.gemm_e4m3(Aq, sa, Wq, sw, bias, relu=True))
    Y, Yq = ops.gemm_e4m3(dev(Aq), dev(Wq), dev(bias), a_scale=sa, w_scale=sw, relu=True, q_scale=0.01)
    y = Y.float().cpu().numpy()
    assert rel_err(y, ref) <= 8e-3
    assert np.array_equal(Yq.cpu().numpy(), o.quantize_e4m3(y, 0.01))


# The E4M3 output takes eight quotients at a time and divides only where one of them lies near a rounding boundary: with a scale of
# 0.01 or 0.25 many do, zeros (whole rows of them, some biases too) must not count as such nor change their sign, and 3e-39 has an
# infinite reciprocal. Sizes of the one-CTA kernel (ragged) and of the pair kernel.
@pytest.mark.parametrize("M,N,K", [(300, 72, 144), (18900, 1000, 128)])
@pytest.mark.parametrize("relu", [False, True])
def test_gemm_e4m3_output_bytes(relu, M, N, K):
    rng = np.random.default_rng(M + N)
    X = rng.standard_normal((M, K)).astype(np.float32)
    X[::7] = 0
    Wf = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    bias = np.where(rng.random(N) < 0.3, 0, rng.standard_normal(N) * 0.02).astype(np.float32)
    sa, sw = float(np.abs(X).max() / 448), float(np.abs(Wf).max() / 448)
    Aq, Wq = o.quantize_e4m3(X, sa), o.quantize_e4m3(Wf, sw)
    ref = o.bf16_bits_to_f32(o.gemm_e4m3(Aq, sa, Wq, sw, bias, relu=relu))
    for scale in (0.01, 0.01137, 0.25, 1e-6) + ((3e-39,) if M == 300 else ()):
        Y, Yq = ops.gemm_e4m3(dev(Aq), dev(Wq), dev(bias), a_scale=sa, w_scale=sw, relu=relu, q_scale=scale)
        y = Y.float().cpu().numpy()
        assert rel_err(y, ref) <= 8e-3
        assert np.array_equal(Yq.cpu().numpy(), o.quantize_e4m3(y, scale))


# ------------------------------------------------------------------------------------ implicit-GEMM convolution
CONV_TC = [
    # N, C, H, W, Cout, relu, pool
    (4, 16, 32, 32, 32, 1, 2), (6, 32, 16, 16, 64, 1, 2), (5, 64, 8, 8, 128, 1, 0), (5, 64, 8, 8, 128, 0, 2),
    (3, 8, 16, 24, 20, 1, 0), (2, 32, 64, 64, 64, 1, 2), (300, 16, 32, 32, 32, 1, 2), (1, 128, 8, 16, 16, 0, 0),
    # haloed-patch kernel: channels streamed in plane groups, partial channel chunks, wide tiles
    (2, 64, 16, 16, 32, 0, 0), (2, 16, 48, 40, 48, 1, 2), (2, 32, 32, 16, 128, 1, 2), (3, 16, 16, 8, 8, 0, 2),
]


@pytest.mark.parametrize("case", CONV_TC)
def test_conv3x3_f32_tcgen05(case):
    N, C, H, W, Cout, relu, pool = case
    rng = np.random.default_rng(sum(case))
    X = rng.standard_normal((N, C, H, W)).astype(np.float32)
    Wt = (rng.standard_normal((Cout, C, 3, 3)) * 0.2).astype(np.float32)
    b = rng.standard_normal(Cout).astype(np.float32)
    ref = o.conv2d_f32(X, Wt, b, pad=(1, 1), relu=bool(relu))
    if pool:
        ref = o.pool2d_f32(ref, 0, (2, 2), (2, 2))
    y = ops.conv2d_f32(dev(X.transpose(0, 2, 3, 1)), ops.conv2d_pack_f32(dev(Wt)), dev(b), shape=X.shape, pad=(1, 1),
                       relu=bool(relu), pool=pool, x_layout=1, y_layout=1, w_packed=True, kernel=(3, 3))
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert rel_err(y.cpu().numpy().transpose(0, 3, 1, 2), ref) <= 1e-5


# fp32 convolutions in half-precision parts: 16 and 32 channels, every width class of the output, odd tile counts, ragged channels
# (values that the parts hold, values that they do not -- scales that differ from channel to channel, in a pixel's neighbourhood, from tap
# to tap, beside weights that are zero or undo them --, filters that have died out, infinities and NaN)
@pytest.mark.parametrize("values", ["normal", "one sign", "image scales", "pixel scales", "tap scales", "channels 2^8", "channels 2^16", "channels 2^24", "channels 2^28",
                                    "channels 2^32", "channels 2^40", "channel blocks", "wide channel, no weights", "one place per image", "decayed channel", "dead filters",
                                    "sparse decades", "smallest", "specials"])
@pytest.mark.parametrize("N,C,H,W,Cout,relu,pool", [(3, 16, 16, 8, 20, 0, 0), (2, 16, 48, 24, 64, 1, 2), (150, 32, 16, 16, 64, 0, 2), (1, 32, 16, 40, 33, 1, 2),
                                                    (5, 32, 32, 16, 30, 0, 0), (3, 16, 32, 32, 100, 0, 2), (2, 16, 16, 16, 128, 1, 0), (1, 16, 16, 8, 1, 0, 2)])
def test_conv3x3_f32_in_half_precision_parts(N, C, H, W, Cout, relu, pool, values):
    rng = np.random.default_rng(N + C + H + W + Cout)
    x, w, b = rng.standard_normal((N, C, H, W)), rng.standard_normal((Cout, C, 3, 3)), rng.standard_normal(Cout)
    if values == "one sign":
        x, w = np.abs(x), np.abs(w)
    if values == "image scales":
        x *= 2.0 ** rng.integers(-40, 40, (N, 1, 1, 1))
    if values == "pixel scales":
        x *= 2.0 ** rng.integers(-30, 30, (N, 1, H, W))
    if values == "tap scales":
        w *= 2.0 ** rng.integers(-30, 30, (Cout, 1, 3, 3))
    if values.startswith("channels") or values == "channel blocks":      # every product of the size it would have without the scales
        e = float(values[values.find("^") + 1:]) if "^" in values else 30.0
        scale = 2.0 ** np.round(np.linspace(0, e, C) if "^" in values else np.repeat([0, e / 3, e], C)[::3])
        scale = (rng.permutation(scale) if "^" in values else scale)[:, None, None]
        x, w = x * scale, w / scale
    if values == "wide channel, no weights":
        x[:, 3] *= 2.0 ** 26
        x[N // 2:, 3] *= 2.0 ** 10
        w[:, 3] = 0
    if values == "one place per image":                                  # large there in every channel, and everywhere in a channel nobody reads
        d = np.abs(np.arange(H)[:, None] - rng.integers(0, H, (N, 1, 1, 1))) + np.abs(np.arange(W)[None] - rng.integers(0, W, (N, 1, 1, 1)))
        x *= 2.0 ** (-3.0 * d)
        x[:, 0], w[:, 0] = 1, 0
    if values == "decayed channel":                                      # weights of a channel that nobody used; half the images do
        w[:, 5] *= 2.0 ** -70
        w[:, 9:] *= rng.random((Cout, C - 9, 1, 1)) < 0.9
        x[N // 2:, np.arange(C) != 5] = 0
    if values == "dead filters":
        w[0] *= 2.0 ** -40
        w[Cout // 2] *= 2.0 ** -118
        w[Cout // 3] *= 2.0 ** -135
        w[Cout // 4] = 0
        b[[0, Cout // 2, Cout // 3, Cout // 4]] = 0
    if values == "sparse decades":
        x = 10.0 ** rng.uniform(-9, 0, x.shape) * (rng.random((N, 1, H, W)) < 0.05)
        x[:, :, : H // 2, : W // 2] = 0
    if values == "smallest":                                             # down to the smallest normal numbers and the subnormal ones
        x *= 2.0 ** rng.integers(-126, -90, (N, 1, H // 8, W // 8)).repeat(8, 2).repeat(8, 3)
        w *= 2.0 ** rng.integers(60, 90, (Cout, 1, 1, 1))
    if values == "specials":
        for v in (np.inf, -np.inf, np.nan, 3e38, 1e-39):
            x[rng.integers(N), rng.integers(C), rng.integers(H), rng.integers(W)] = v
    x, w, b = (a.astype(np.float32) for a in (x, w, b))
    y = ops.conv2d_f32(dev(x.transpose(0, 2, 3, 1)), ops.conv2d_pack_f32(dev(w)), dev(b), shape=x.shape, pad=(1, 1), relu=bool(relu), pool=pool,
                       x_layout=capi.LAYOUT_NHWC, y_layout=capi.LAYOUT_NHWC, w_packed=True, kernel=(3, 3))
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    y = y.cpu().double().view(N, H // max(pool, 1), W // max(pool, 1), Cout).permute(0, 3, 1, 2)
    xd, wd, bd = (torch.from_numpy(a).double() for a in (x, w, b))
    conv = torch.nn.functional.conv2d
    ref = conv(xd, wd, bd, padding=1)
    ref = ref.float().double()      # sums beyond fp32's range are infinite
    # every product is off by 2^-22 of itself, every MMA's sum by one truncation
    size = conv(xd.abs().nan_to_num(0, 0), wd.abs(), bd.abs(), padding=1)
    if relu:
        ref = torch.where(ref > 0, ref, 0.0)
    if pool:
        # a NaN is passed over, as a comparison with it is false, unless the window holds nothing else
        nan = -torch.nn.functional.max_pool2d(-ref.isnan().double(), 2) == 1
        ref = torch.where(ref.isnan(), -torch.inf, ref)
        ref, size = torch.nn.functional.max_pool2d(ref, 2), torch.nn.functional.max_pool2d(size, 2)
        ref[nan] = torch.nan
    finite = ref.isfinite()
    steps = 2 * 9 * C // 16 + 4
    assert ((y - ref).abs()[finite] <= steps * 2.0 ** -23 * size[finite] + 2.0 ** -149).all()
    assert torch.equal(y[~finite].float().nan_to_num(2.0, 1.0, -1.0), ref[~finite].float().nan_to_num(2.0, 1.0, -1.0))


# how a row of channels leaves: whole sectors, words of four, single values, the last of them partly, and every alignment of the result
@pytest.mark.parametrize("Cout", [1, 4, 6, 8, 12, 16, 17, 20, 24, 28, 31, 32, 36, 40, 56, 64, 72])
@pytest.mark.parametrize("C", [16, 32])
def test_conv3x3_f32_in_half_precision_parts_rows_of_channels(C, Cout):
    g = torch.Generator(device="cuda").manual_seed(C + Cout)
    N, H, W = 3, 32, 24
    x, w, b = (torch.randn(s, device="cuda", generator=g) for s in ((N, C, H, W), (Cout, C, 3, 3), (Cout,)))
    x[1, 3, 4, 5] = 2.0 ** 40                                            # a tile of the careful form, whose rows leave by sixteen channels
    ref, size = (torch.nn.functional.conv2d(f(x.double()), f(w.double()), f(b.double()), padding=1).permute(0, 2, 3, 1) for f in (lambda t: t, torch.abs))
    X, P = x.permute(0, 2, 3, 1).contiguous(), ops.conv2d_pack_f32(w)
    first = None
    for offset in (0, 1, 2, 4):                                          # floats past a 256-byte boundary
        whole = torch.full((N * H * W * Cout + 16,), 7.0, device="cuda")
        y = whole[offset: offset + N * H * W * Cout]
        ops.conv2d_f32(X, P, b, shape=x.shape, pad=(1, 1), x_layout=1, y_layout=1, w_packed=True, kernel=(3, 3), out=y.view(N, H, W, Cout))
        assert ops.last_engine() == capi.ENGINE_TCGEN05
        assert (whole[:offset] == 7).all() and (whole[offset + y.numel():] == 7).all()
        first = y.clone() if first is None else first
        assert torch.equal(y, first)
    assert ((first.view(ref.shape).double() - ref).abs() <= (2 * 9 * C // 16 + 4) * 2.0 ** -23 * size).all()


# many tiles a CTA, plain ones and such that take one pass, several or chains, in turn: their rings of slots, accumulators and patches come round
@pytest.mark.parametrize("wide_weights", [0, 1])
@pytest.mark.parametrize("N,C,H,W,Cout,pool", [(700, 16, 32, 32, 32, 2), (900, 32, 16, 32, 64, 0), (500, 16, 32, 32, 128, 2), (1700, 32, 16, 16, 24, 0)])
def test_conv3x3_f32_in_half_precision_parts_many_tiles(N, C, H, W, Cout, pool, wide_weights):
    g = torch.Generator(device="cuda").manual_seed(N + C + Cout)
    x, w = torch.randn(N, C, H, W, device="cuda", generator=g), torch.randn(Cout, C, 3, 3, device="cuda", generator=g)
    kind = torch.randint(0, 6, (N,), device="cuda", generator=g)
    scale = lambda low, high, *shape: 2.0 ** torch.randint(low, high, shape, device="cuda", generator=g).float()
    x = torch.where((kind == 1)[:, None, None, None], x * scale(-60, 60, N, 1, H, W), x)       # several passes
    x = torch.where((kind == 2)[:, None, None, None], x * scale(-35, 1, N, C, H, W), x)        # one value or the other is lost
    x[kind == 3, 3, 5, 5] = torch.inf
    x[kind == 4, 2, 9, 2] = torch.nan
    if wide_weights:
        w *= scale(-40, 1, Cout, C, 3, 3)
    y = ops.conv2d_f32(x.permute(0, 2, 3, 1).contiguous(), ops.conv2d_pack_f32(w), None, shape=x.shape, pad=(1, 1), pool=pool, x_layout=capi.LAYOUT_NHWC,
                       y_layout=capi.LAYOUT_NHWC, w_packed=True, kernel=(3, 3))
    y = y.double().view(N, H // max(pool, 1), W // max(pool, 1), Cout).permute(0, 3, 1, 2)
    conv, pool2 = torch.nn.functional.conv2d, torch.nn.functional.max_pool2d
    ref, size = conv(x.double(), w.double(), padding=1), conv(x.double().abs().nan_to_num(0, 0), w.double().abs(), padding=1)
    if pool:
        nan = -pool2(-ref.isnan().double(), 2) == 1
        ref, size = pool2(torch.where(ref.isnan(), -torch.inf, ref), 2), pool2(size, 2)
        ref[nan] = torch.nan
    finite = ref.isfinite()
    assert ((y - ref).abs()[finite] <= (2 * 9 * C // 16 + 4) * 2.0 ** -23 * size[finite]).all()
    assert torch.equal(y[~finite].nan_to_num(2.0, 1.0, -1.0), ref[~finite].nan_to_num(2.0, 1.0, -1.0))


@pytest.mark.parametrize("case", [(3, 32, 32, 32, 64, 1, 2), (7, 64, 16, 16, 64, 1, 2), (9, 64, 8, 8, 128, 1, 2), (2, 32, 16, 16, 40, 0, 0),
                                  (130, 32, 32, 32, 64, 1, 2), (3, 128, 16, 16, 128, 1, 2), (2, 256, 16, 16, 32, 0, 0),
                                  (2, 128, 32, 16, 64, 1, 0), (5, 32, 16, 16, 24, 1, 2),
                                  # pooled-window kernel (32 x 16 tiles, pooling in tensor memory): two K steps per tap, 32 and 48
                                  # output channels, no Relu, several tiles per image in both directions, more tiles than SMs
                                  (2, 64, 32, 32, 64, 1, 2), (2, 32, 64, 48, 32, 0, 2), (3, 64, 32, 16, 48, 1, 2), (40, 32, 64, 32, 16, 1, 2),
                                  # lines of eight pixels with more tiles than SMs (per-tap kernel with resident weights): two images per
                                  # tile, one image per tile, 32-byte pixels
                                  (301, 64, 8, 8, 128, 1, 2), (310, 64, 8, 8, 72, 0, 0), (160, 64, 16, 8, 64, 1, 2), (300, 32, 8, 8, 32, 1, 0)])
def test_qlinear_conv3x3_tcgen05_bit_exact(case):
    N, C, H, W, Cout, relu, pool = case
    rng = np.random.default_rng(sum(case))
    X = (rng.integers(0, 256, (N, C, H, W)) * (rng.random((N, C, H, W)) < 0.4)).astype(np.uint8)
    Wt = rng.integers(-127, 128, (Cout, C, 3, 3)).astype(np.int8)
    ws = rng.uniform(0.001, 0.01, Cout).astype(np.float32)
    bias = rng.integers(-1000, 1000, Cout).astype(np.int32)
    y_scale = 0.05 * 0.005 * 127 * 80 * np.sqrt(C * 9) / 100
    ref = o.qlinear_conv2d(X, 0.05, 0, Wt, ws, y_scale, 3, bias=bias, pad=(1, 1), relu=bool(relu))
    if pool:
        ref = o.maxpool2d_u8(ref)
    mult = dev(o.requant_multiplier(0.05, ws, y_scale))
    y = ops.qlinear_conv2d(dev(X.transpose(0, 2, 3, 1)), ops.qconv2d_pack_i8(dev(Wt)), mult, dev(bias), shape=X.shape, pad=(1, 1),
                           x_zp=0, y_zp=3, relu=bool(relu), pool=pool, x_layout=1, y_layout=1, w_packed=True, kernel=(3, 3))
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert np.array_equal(y.cpu().numpy().transpose(0, 3, 1, 2), ref)
    assert len(np.unique(ref)) > 20


@pytest.mark.parametrize("case", [(3, 64, 64, 32, 1, 0), (2, 32, 48, 16, 0, 7), (5, 96, 32, 64, 1, 0), (150, 64, 64, 32, 1, 3), (1, 32, 16, 48, 1, 200)])
def test_qlinear_first_layer_pooled_tcgen05_bit_exact(case):
    """One input channel, 3x3 / pad 1, Relu or not, MaxPool 2x2 fused: the tensor-core first-layer kernel (operand rows built
    from the staged image rows, pooling in tensor memory) against the oracle, NCHW input as the Session hands it over."""
    N, H, W, Cout, relu, y_zp = case
    ops.set_engine(0)
    rng = np.random.default_rng(sum(case))
    X = (rng.integers(0, 256, (N, 1, H, W)) * (rng.random((N, 1, H, W)) < 0.3)).astype(np.uint8)
    X[0, 0, 0, :] = 255
    X[0, 0, :, -1] = 255                       # bright borders next to the padding
    Wt = rng.integers(-127, 128, (Cout, 1, 3, 3)).astype(np.int8)
    ws = rng.uniform(0.001, 0.01, Cout).astype(np.float32)
    bias = rng.integers(-300, 300, Cout).astype(np.int32)
    y_scale = 0.03 * 0.005 * 127 * 6
    ref = o.maxpool2d_u8(o.qlinear_conv2d(X, 0.03, 0, Wt, ws, y_scale, y_zp, bias=bias, pad=(1, 1), relu=bool(relu)))
    mult = dev(o.requant_multiplier(0.03, ws, y_scale))
    y = ops.qlinear_conv2d(dev(X), dev(Wt), mult, dev(bias), shape=X.shape, pad=(1, 1), x_zp=0, y_zp=y_zp, relu=bool(relu), pool=2,
                           x_layout=0, y_layout=1, w_packed=False)
    assert ops.last_engine() == capi.ENGINE_TCGEN05
    assert np.array_equal(y.cpu().numpy().transpose(0, 3, 1, 2), ref)
    assert len(np.unique(ref)) > 20


@pytest.mark.parametrize("case", [(3, 32, 32, 32, 64), (2, 64, 16, 16, 64), (4, 1, 32, 32, 16), (2, 64, 8, 8, 128), (2, 64, 32, 32, 32)])
def test_qconv_pool_with_negative_multipliers(case):
    """A negative requantisation multiplier makes the requantisation decreasing in the accumulator, so the
    kernels must not pool the raw accumulators first; they detect it and pool the finished values."""
    N, C, H, W, Cout = case
    if C <= 4:
        ops.set_engine(0)  # the first-layer kernel is a CUDA-core kernel; this file forces tcgen05 otherwise
    rng = np.random.default_rng(sum(case))
    X = rng.integers(0, 256, (N, C, H, W)).astype(np.uint8)
    Wt = rng.integers(-127, 128, (Cout, C, 3, 3)).astype(np.int8)
    ws = (rng.uniform(0.001, 0.01, Cout) * rng.choice([-1.0, 1.0], Cout)).astype(np.float32)
    assert (ws < 0).any() and (ws > 0).any()
    y_scale = 0.02 * 0.005 * 128 * 3 * np.sqrt(C)
    ref = o.maxpool2d_u8(o.qlinear_conv2d(X, 0.02, 0, Wt, ws, y_scale, 100, pad=(1, 1), relu=False))
    mult = dev(o.requant_multiplier(0.02, ws, y_scale))
    y = ops.qlinear_conv2d(dev(X.transpose(0, 2, 3, 1)), ops.qconv2d_pack_i8(dev(Wt)), mult, None, shape=X.shape, pad=(1, 1),
                           x_zp=0, y_zp=100, relu=False, pool=2, x_layout=1, y_layout=1, w_packed=True, kernel=(3, 3)).cpu().numpy()
    assert np.array_equal(y.transpose(0, 3, 1, 2), ref)
    assert len(np.unique(ref)) > 20


@pytest.mark.parametrize("sign", ["both", "one"])
@pytest.mark.parametrize("M,N,K", [(300, 200, 8), (1024, 130, 17), (257, 333, 33), (700, 64, 96), (640, 250, 97), (512, 300, 128), (129, 260, 255), (300, 200, 256),
                                   (400, 70, 777), (600, 33, 1023), (260, 190, 1333), (100, 600, 4001)])
def test_gemm_f32_parts_are_no_further_from_float64_than_fma_chains(M, N, K, sign):
    """Products that run as chains of fp32 FMAs on the CUDA cores when the tensor cores are not used: their error (2-norm, against
    float64) is the bound for the tensor-core kernel, for every way the operands can lie, below and at the edges of its units of K."""
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    for tA, tB in ((1, 0), (1, 1), (0, 0)):
        A = torch.randn((K, M) if tA else (M, K), device="cuda", generator=g)
        B = torch.randn((N, K) if tB else (K, N), device="cuda", generator=g) * K ** -0.5
        if sign == "one":
            A, B = A.abs(), B.abs()
        exact = (A.double().t() if tA else A.double()) @ (B.double().t() if tB else B.double())

        def error(engine):
            ops.set_engine(engine)
            y = ops.gemm_f32(A, B, transA=tA, transB=tB)
            assert ops.last_engine() == engine
            return float((y.double() - exact).norm())
        assert error(capi.ENGINE_TCGEN05) <= error(capi.ENGINE_SIMT)


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("M,N,K,bias", [(130, 68, 40, 2), (131, 37, 41, 2), (300, 200, 64, 1), (90, 33, 1500, 0), (257, 130, 2047, 2), (20000, 64, 9, 1)])
def test_gemm_f32_of_values_the_parts_do_not_hold(M, N, K, bias, relu):
    """Infinities, NaNs, values that round up to infinity, products that overflow and rows near the bottom of the range: what the chain of
    FMAs gives (operands below bfloat16's denormals, row 21, count as zeros), for every layout, with one tile and with a cluster along K, whole words and single floats at the output."""
    rng = np.random.default_rng(M + N + K)
    for tA, tB in ((1, 0), (1, 1), (0, 0)):
        A = rng.standard_normal((M, K)).astype(np.float32)
        B = rng.standard_normal((N, K)).astype(np.float32)
        A[3, 5], A[7, K - 1], A[11, 0], B[2, 3], B[N - 1, K - 1] = np.inf, -np.inf, np.nan, np.inf, np.nan
        A[17, 2], A[18, 2], B[5, 7] = 3.4e38, -np.float32(3.4028235e38), 3.4028235e38
        A[20], A[21], B[9] = A[20] * 1e-35, A[21] * 1e-41, B[9] * 1e-30
        A[22], B[11] = 0., 0.
        A[23], B[12] = A[23] * 1e30, B[12] * 1e30
        a = dev(A.T if tA else A)
        b = dev(B if tB else B.T)
        c = {0: None, 1: dev(rng.standard_normal(N).astype(np.float32)), 2: dev(rng.standard_normal((M, N)).astype(np.float32))}[bias]

        def product(engine, in_place):
            ops.set_engine(engine)
            out = c.clone() if in_place else None      # the bias and the result may be the same memory
            y = ops.gemm_f32(a, b, out if in_place else c, transA=tA, transB=tB, alpha=1.5, beta=0.5, relu=relu, out=out)
            assert ops.last_engine() == engine
            return y.cpu().numpy()
        ref = product(capi.ENGINE_SIMT, False)
        assert relu or not np.isfinite(ref).all()
        for in_place in ([False, True] if bias == 2 else [False]):
            y = product(capi.ENGINE_TCGEN05, in_place)
            assert np.array_equal(np.isnan(y), np.isnan(ref))
            tiny = np.abs(ref) < 1e-29                 # 1.5 times a sum below 2^-96, as all of its parts are in a row this small
            tiny[:20], tiny[21:] = False, False
            assert np.array_equal(y[~np.isfinite(ref)], ref[~np.isfinite(ref)], equal_nan=True)
            if bias == 0:
                assert np.array_equal(y[tiny], ref[tiny])
            # the reference is a chain of K roundings of 2^-24 of a growing sum: a standard deviation of sqrt(K / 6) * 2^-24, of which the
            # largest of some ten thousand sums may show a dozen (1.1e-6 and 1.8e-5 at K = 2047)
            ok = np.isfinite(ref) & (np.abs(ref) < 1e6)
            bound = max(1e-5, 16 * np.sqrt(K / 6) * 2.0 ** -24)
            scale = np.maximum(np.abs(ref[ok]), np.sqrt(np.mean(ref[ok].astype(np.float64) ** 2)))    # some sums are a thousand times the others
            assert (np.abs(y[ok].astype(np.float64) - ref[ok]) / scale).max() <= bound


@pytest.mark.parametrize("M,N,K,tA,tB,bias,engine", [
    (16384, 1001, 9, 1, 0, 2, capi.ENGINE_SIMT), (4099, 2050, 8, 0, 0, 0, capi.ENGINE_SIMT), (8000, 777, 40, 1, 1, 2, capi.ENGINE_SIMT),   # output-bound
    (3190, 824, 9, 0, 1, 1, capi.ENGINE_SIMT), (290, 1431, 10, 0, 0, 1, capi.ENGINE_SIMT),
    (1000, 777, 1333, 1, 0, 2, capi.ENGINE_TCGEN05), (200, 200, 4000, 1, 1, 1, capi.ENGINE_TCGEN05), (4000, 1000, 500, 0, 0, 0, capi.ENGINE_TCGEN05),
    (43, 158, 3447, 0, 0, 1, capi.ENGINE_TCGEN05)])
def test_gemm_f32_takes_the_faster_kernel_where_tma_cannot_fetch(M, N, K, tA, tB, bias, engine):
    """The choice between the tensor-core kernel and the CUDA-core one, and the result of either."""
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn((K, M) if tA else (M, K), device="cuda", generator=g)
    B = torch.randn((N, K) if tB else (K, N), device="cuda", generator=g) * K ** -0.5
    C_ = {0: None, 1: torch.randn(N, device="cuda", generator=g), 2: torch.randn(M, N, device="cuda", generator=g)}[bias]
    exact = 0.75 * ((A.double().t() if tA else A.double()) @ (B.double().t() if tB else B.double())) + (0 if C_ is None else 1.5 * C_.double())
    ops.set_engine(0)
    y = ops.gemm_f32(A, B, C_, transA=tA, transB=tB, alpha=0.75, beta=1.5)
    assert ops.last_engine() == engine
    assert float((y.double() - exact).norm() / exact.norm()) <= 2e-6     # 24-bit chains of up to 4000 terms: sqrt(K / 6) * 2^-24 = 1.6e-6
    if engine == capi.ENGINE_SIMT:
        ops.set_engine(capi.ENGINE_SIMT)
        assert torch.equal(y, ops.gemm_f32(A, B, C_, transA=tA, transB=tB, alpha=0.75, beta=1.5))


# one tile and several per CTA, every tile width, K shared by 1, 2, 4 and 8 ranks, units of 3, 4 and 8 stages with remainders, ragged and whole rows of Y
@pytest.mark.parametrize("M,N,K,bias", [(2049, 513, 257, 1), (1000, 777, 1333, 2), (64, 60, 4100, 0), (5000, 330, 95, 2), (1024, 1024, 1024, 1), (390, 2052, 600, 0),
                                        (4200, 330, 2050, 1), (130, 1290, 3000, 2), (20000, 129, 65, 0), (12100, 520, 140, 1), (36, 3000, 3905, 2), (900, 2500, 64, 0)])
def test_gemm_f32_of_operands_split_beforehand(M, N, K, bias):
    """The workspace form against float64 and the chain of FMAs (whose 2-norm error is the bound), for every layout and an unaligned base; rows
    of values the parts do not hold give what the chain gives; without the workspace the call is the plain one."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lib = capi.load()

    def place(t, offset):
        buf = torch.empty(t.numel() + 4, device="cuda")
        return buf[offset: offset + t.numel()].view(t.shape).copy_(t)
    taken = 0
    for i, (tA, tB) in enumerate(((0, 0), (0, 1), (1, 0), (1, 1))):
        A = place(torch.randn((K, M) if tA else (M, K), device="cuda", generator=g), i % 2)
        B = place(torch.randn((N, K) if tB else (K, N), device="cuda", generator=g) * K ** -0.5, i // 2)
        C_ = {0: None, 1: torch.randn(N, device="cuda", generator=g), 2: torch.randn(M, N, device="cuda", generator=g)}[bias]
        a, b = (A.t() if tA else A), (B.t() if tB else B)
        a[5, 7], a[6, K - 1], a[9] = float("inf"), float("nan"), a[9] * 1e-35
        d = capi.GemmF32Desc(M, N, K, tA, tB, 0.75, 1.5, bias, i % 2)
        nbytes = lib.sofie_cuda_gemm_f32_workspace(C.byref(d))
        taken += nbytes > 0

        def product(engine, size):
            ops.set_engine(engine)
            w = torch.empty(max(size, 1), dtype=torch.uint8, device="cuda")
            Y = torch.full((M, N), 7.0, device="cuda")
            capi.call("sofie_cuda_gemm_f32_ws", ops._stream(), C.byref(d), *[C.c_void_p(0 if t is None else t.data_ptr()) for t in (A, B, C_, Y)], C.c_void_p(w.data_ptr()), size)
            return Y
        chain, plain = product(capi.ENGINE_SIMT, nbytes), product(capi.ENGINE_TCGEN05, nbytes - 1 if nbytes else 0)
        y = product(capi.ENGINE_TCGEN05, nbytes)
        assert ops.last_engine() == capi.ENGINE_TCGEN05
        exact = 0.75 * (a.double() @ b.double()) + (0 if C_ is None else 1.5 * C_.double())
        if i % 2:
            exact = torch.where(exact > 0, exact, 0.)
        for odd in (5, 6):
            assert torch.equal(y[odd].nan_to_num(1.), chain[odd].nan_to_num(1.)) and torch.equal(y[odd].isnan(), chain[odd].isnan())
        if bias == 0:
            assert torch.equal(y[9], chain[9])
        rows = [r for r in range(M) if r not in (5, 6, 9)]
        off = [float((t[rows].double() - exact[rows]).norm()) for t in (y, chain, plain)]
        assert off[0] <= off[1] * 1.02 and off[2] <= off[1] * 1.02      # K = 64 .. 95: all of them round a handful of times
    assert taken == 4


@pytest.mark.parametrize("M,N,K,bias", [(1000, 777, 1333, 2), (64, 60, 4100, 0), (2049, 513, 257, 1), (36, 3000, 3905, 2)])
@pytest.mark.parametrize("tA,tB", [(0, 0), (1, 1)])
def test_gemm_f32_workspace_and_without(M, N, K, bias, tA, tB):
    """The workspace is written as far as it was asked for and no further, under the automatic dispatch too; one byte less, none, a base that is not aligned,
    workspace=False and no memory left are the plain call, bit for bit, and take nothing."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lib = capi.load()
    A, B = torch.randn((K, M) if tA else (M, K), device="cuda", generator=g), torch.randn((N, K) if tB else (K, N), device="cuda", generator=g)
    C_ = {0: None, 1: torch.randn(N, device="cuda", generator=g), 2: torch.randn(M, N, device="cuda", generator=g)}[bias]
    d = capi.GemmF32Desc(M, N, K, tA, tB, 0.75, 1.5, bias, 0)
    pointers = [C.c_void_p(0 if t is None else t.data_ptr()) for t in (A, B, C_)]
    for engine in (0, capi.ENGINE_TCGEN05):
        ops.set_engine(engine)
        nbytes = lib.sofie_cuda_gemm_f32_workspace(C.byref(d))
        assert nbytes > 0
        whole = torch.full((nbytes + 8192,), 0xA5, dtype=torch.uint8, device="cuda")

        def product(offset, size):
            Y = torch.full((M, N), 7.0, device="cuda")
            capi.call("sofie_cuda_gemm_f32_ws", ops._stream(), C.byref(d), *pointers, C.c_void_p(Y.data_ptr()), C.c_void_p(whole.data_ptr() + offset), size)
            return Y
        plain = torch.full((M, N), 7.0, device="cuda")
        capi.call("sofie_cuda_gemm_f32", ops._stream(), C.byref(d), *pointers, C.c_void_p(plain.data_ptr()))
        for short in (product(4096, nbytes - 1), product(4096, 0), product(4096 + 64, nbytes)):
            assert torch.equal(short, plain) and (whole == 0xA5).all()
        exact = 0.75 * ((A.t() if tA else A).double() @ (B.t() if tB else B).double()) + (0 if C_ is None else 1.5 * C_.double())
        y = product(4096, nbytes)
        assert float((y.double() - exact).norm() / exact.norm()) <= 2.5e-7
        assert (whole[:4096] == 0xA5).all() and (whole[4096 + nbytes:] == 0xA5).all() and not (whole[4096:4096 + nbytes] == 0xA5).all()
        call = lambda **kw: ops.gemm_f32(A, B, C_, transA=tA, transB=tB, alpha=0.75, beta=1.5, **kw)
        assert torch.equal(call(), y)
        out = torch.empty(M, N, device="cuda")
        taken = torch.cuda.memory_stats()["allocation.all.allocated"]
        call(out=out, workspace=False)
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == taken
        assert torch.equal(out, plain)
        del y, whole
        torch.cuda.empty_cache()
        out.fill_(7.0)
        hold = []
        try:                                                             # no more than there is now, and that is held
            torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)
            for size in (1 << 24, 1 << 21, 1 << 18):
                with pytest.raises(torch.OutOfMemoryError):
                    while True:
                        hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            call(out=out)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        del hold
        assert torch.equal(out, plain)
    ops.set_engine(0)


# the form without conversions (zero point 0; one input channel without bias, and 32 with one): multipliers of zero, subnormal and far below one,
# such that most products are ties, that saturate everything, the largest that stay with it (2^20) and larger ones
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("C,Cout", [(1, 32), (1, 64), (1, 16), (32, 64)])
def test_qconv_pooled_requantisation_at_its_edges(C, Cout, bias):
    g = torch.Generator(device="cuda").manual_seed(C + Cout)
    N, H, W = 3, 64, 32
    X = torch.randint(0, 256, (N, C, H, W), device="cuda", generator=g, dtype=torch.uint8)
    X[0] = 255
    Wt = torch.randint(-128, 128, (Cout, C, 3, 3), device="cuda", generator=g, dtype=torch.int8)
    Wt[1], Wt[2] = 127, -128                                    # the largest sums there are
    exact = torch.nn.functional.conv2d(X.double(), Wt.double(), padding=1)
    b = torch.randint(-2000, 2000, (Cout,), device="cuda", generator=g, dtype=torch.int32) if bias else None
    if bias:
        exact = exact + b.double()[:, None, None]
    for values in ([0.0, 2.0 ** -140, 2.0 ** -126, 1e-30, 2.0 ** -24, 3e-5], [0.5, 0.25, 0.125, 1.5, 0.0625, 2.0 ** -9], [1e-3, 7.3e-4, 255.5 / 291465, 1.0, 2.0 ** 20, 1000.0],
                   [1e-3, 2.0 ** 20 + 1, 2.0 ** 40, 3e38, 0.0, 0.02]):
        mult = torch.tensor(values, device="cuda").repeat(Cout // 6 + 1)[:Cout].contiguous()
        q = (exact.float() * mult[:, None, None]).round().clamp(0, 255)      # one rounding to fp32, then to the nearest even integer
        ref = torch.nn.functional.max_pool2d(q, 2).permute(0, 2, 3, 1).to(torch.uint8)
        ops.set_engine(0)
        y = ops.qlinear_conv2d(X.permute(0, 2, 3, 1).contiguous(), ops.qconv2d_pack_i8(Wt), mult, b, shape=X.shape, pad=(1, 1), relu=True, pool=2,
                               x_layout=capi.LAYOUT_NHWC, y_layout=capi.LAYOUT_NHWC, w_packed=True, kernel=(3, 3))
        assert ops.last_engine() == capi.ENGINE_TCGEN05
        assert torch.equal(y.view(ref.shape), ref)
