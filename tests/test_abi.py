"""The C-ABI library loads without a GPU and exports exactly what include/sofie_cuda.h declares."""
import ctypes as C
import re
from pathlib import Path

import pytest

from sofie_b200 import capi

ROOT = Path(__file__).resolve().parents[1]


def declared_symbols():
    text = (ROOT / "include" / "sofie_cuda.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(sofie_cuda_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound():
    lib = capi.load()
    names = declared_symbols()
    assert len(names) >= 40
    for n in names:
        assert hasattr(lib, n), f"{n} declared in sofie_cuda.h but not exported by libSOFIE_cuda.so"
    bound = set(capi.SIGNATURES) | set(capi.STRING_GETTERS) | set(capi.SIZE_GETTERS)
    assert bound == set(names), sorted(bound ^ set(names))


def test_struct_sizes_match_header():
    # all descriptor fields are 4 bytes wide, so the size is 4 * number of fields
    assert C.sizeof(capi.GemmF32Desc) == 9 * 4
    assert C.sizeof(capi.Conv2dDesc) == 19 * 4
    assert C.sizeof(capi.Pool2dDesc) == 15 * 4
    assert C.sizeof(capi.QGemmDesc) == 6 * 4
    assert C.sizeof(capi.QConv2dDesc) == 18 * 4
    assert C.sizeof(capi.Fp8GemmDesc) == 7 * 4
    assert C.sizeof(capi.MlpDesc) == (2 + 9 + 8 + 8) * 4


def test_fused_mlp_shared_memory_arithmetic():
    from sofie_b200 import ops
    # 64 -> 128 -> 128 -> 10: padded weight rows (68, 132, 132 floats), biases, one input tile and two activation tiles of 32 rows
    d = ops.mlp_desc(0, [64, 128, 128, 10], [1, 1, 0], [1, 1, 1])
    want = 4 * (128 * 68 + 128 + 128 * 132 + 128 + 32 * 132 + 32 + 32 * 68 + 2 * 32 * 132)
    assert capi.load().sofie_cuda_mlp_f32_smem(C.byref(d)) == want
    assert ops.mlp_fits([64, 128, 128, 10]) and ops.mlp_fits([256, 96, 1])
    assert not ops.mlp_fits([256, 256, 8]) and not ops.mlp_fits([300, 8]) and not ops.mlp_fits([8] * 10)


def test_status_strings_and_argument_errors():
    lib = capi.load()
    assert lib.sofie_cuda_strerror(0) == b"success"
    assert lib.sofie_cuda_strerror(1) == b"invalid argument"
    assert lib.sofie_cuda_abi_version() == 1
    # NULL descriptor: rejected before anything touches a device
    rc = lib.sofie_cuda_gemm_f32(None, None, None, None, None, None)
    assert rc == capi.ERR_INVALID
    assert b"NULL" in lib.sofie_cuda_last_error()
    d = capi.GemmF32Desc(0, 4, 4, 0, 0, 1.0, 1.0, 0, 0)   # an empty batch is not an error
    assert lib.sofie_cuda_gemm_f32(None, C.byref(d), None, None, None, None) == capi.OK
    d = capi.GemmF32Desc(4, 0, 4, 0, 0, 1.0, 1.0, 0, 0)
    rc = lib.sofie_cuda_gemm_f32(None, C.byref(d), C.c_void_p(16), C.c_void_p(16), None, C.c_void_p(16))
    assert rc == capi.ERR_INVALID
    with pytest.raises(capi.SofieCudaError):
        capi.call("sofie_cuda_set_engine", 7)


@pytest.mark.parametrize("M,N,K,taken", [(41, 17142, 180, 0), (17142, 41, 255, 0), (36, 3000, 3905, 1), (172, 33, 3880, 1), (48, 17142, 180, 1), (31, 3000, 3905, 0),
                                         (1000, 777, 1333, 1), (16384, 4093, 8, 0), (64, 64, 64, 0), (8192, 8192, 8192, 1), (65536, 65536, 4096, 0)])
def test_workspace_is_asked_for_where_the_split_was_measured_to_pay(M, N, K, taken):
    """Six bytes a value of whole tiles of A and B, 1 GiB at most; from 32 rows and columns on, below 48 from K = 256 on."""
    d = capi.GemmF32Desc(M, N, K, 1, 0, 1.0, 1.0, 2, 0)
    nbytes = capi.load().sofie_cuda_gemm_f32_workspace(C.byref(d))
    assert (nbytes > 0) == bool(taken) and nbytes <= 1 << 30
    assert not taken or 6 * K * (M + N) <= nbytes <= 6 * (K + 31) * (M + 127 + N + 127)


def test_no_gpu_means_loud_failure_not_cpu_fallback():
    """Without a device the context cannot be created; nothing computes on the CPU instead."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    lib = capi.load()
    ctx = C.c_void_p()
    rc = lib.sofie_cuda_ctx_create(C.byref(ctx), 0, 1 << 20)
    assert rc != capi.OK and not ctx.value
    import mirror_session as runner
    from sofie_b200 import configs
    m, _ = configs.mlp_f32(batch=4)
    with pytest.raises(RuntimeError):
        runner.Session(m)


@pytest.mark.parametrize("threads", [1, 2, 4, 7])
def test_threaded_host_copy_moves_every_byte(threads):
    """The copy that carries pageable inputs into the staging ring, run on plain host memory: chunk sizes below and above the 4 MB
    from which the helper threads join in, lengths that are no multiple of a page or of the thread count, many chunks in a row
    (the helpers spin between chunks, then sleep), and a pool that is created and destroyed per call."""
    import numpy as np
    capi.load()
    rng = np.random.default_rng(threads)
    for nbytes, chunk, repeats in ((0, 1 << 20, 1), (1, 8 << 20, 1), (4095, 8 << 20, 2), ((4 << 20) - 1, 8 << 20, 1), (4 << 20, 8 << 20, 1),
                                   ((4 << 20) + 1, 8 << 20, 3), ((33 << 20) + 7, 8 << 20, 2), ((24 << 20) + 4097, (5 << 20) + 13, 1)):
        src = rng.integers(0, 256, nbytes, dtype=np.uint8)
        dst = np.zeros(nbytes + 64, np.uint8)
        dst[nbytes:] = 0xA5                                     # canary behind the destination
        capi.call("sofie_cuda_selftest_host_copy", dst.ctypes.data, src.ctypes.data, nbytes, chunk, threads, repeats)
        assert np.array_equal(dst[:nbytes], src), (nbytes, chunk)
        assert (dst[nbytes:] == 0xA5).all()
    with pytest.raises(RuntimeError):
        capi.call("sofie_cuda_selftest_host_copy", 0, 0, 16, 1 << 20, 1, 1)
    with pytest.raises(RuntimeError):
        capi.call("sofie_cuda_selftest_host_copy", dst.ctypes.data, src.ctypes.data, 16, 1 << 20, 0, 1)


@pytest.mark.parametrize("kind,zp", [(1, 0), (1, 128), (1, 255), (2, 0)])
def test_host_quantisation_gives_the_operators_bytes(kind, zp):
    """What the host makes of a pageable input while it stages it, against the oracle's QuantizeLinear: every tie and its neighbours, both
    saturations, infinities, subnormals, lengths around the vector width. A NaN takes the lower bound / the E4M3 NaN."""
    import numpy as np
    from oracle import cpu_oracle as o
    rng = np.random.default_rng(kind)
    for scale in (0.02, 1.0, 8.0 / 255.0, 3e-3, 1e-30):
        if kind == 1:
            ties = (np.arange(-300, 300) + 0.5).astype(np.float32) * np.float32(scale)
        else:
            codes = o.e4m3_table()[:127].astype(np.float32)
            ties = np.concatenate([codes, (codes[1:] + codes[:-1]) / 2]) * np.float32(scale)
            ties = np.concatenate([ties, -ties])
        x = np.concatenate([ties, np.nextafter(ties, np.float32(np.inf)), np.nextafter(ties, np.float32(-np.inf)),
                            np.array([0.0, -0.0, np.inf, -np.inf, 3e38, -3e38, 1e-45, 1e-39], np.float32), (rng.standard_normal(5000) * 100 * scale).astype(np.float32)])
        want = o.quantize_u8(x, scale, zp) if kind == 1 else o.quantize_e4m3(x, scale)
        for n in (x.size, 0, 1, 15, 16, 17, 63, 65):
            y = np.full(n + 64, 0xA5, np.uint8)
            capi.call("sofie_cuda_selftest_host_quantize", y.ctypes.data, x.ctypes.data, n, kind, scale, zp)
            assert np.array_equal(y[:n], want[:n]) and (y[n:] == 0xA5).all()
    nan = np.full(1, np.nan, np.float32)
    y = np.zeros(1, np.uint8)
    capi.call("sofie_cuda_selftest_host_quantize", y.ctypes.data, nan.ctypes.data, 1, kind, 1.0, zp)
    assert y[0] == (0 if kind == 1 else 0x7F)
    with pytest.raises(RuntimeError):
        capi.call("sofie_cuda_selftest_host_quantize", y.ctypes.data, nan.ctypes.data, 1, kind, 0.0, zp)


def test_operator_calls_refuse_what_they_refused():
    """Tensors of another rank, short sequences and a missing scale are refused before anything is launched (or a device is needed)."""
    import torch
    from sofie_b200 import ops
    image, weights, row = torch.zeros(2, 3, 4, 4, 1), torch.zeros(2, 3, 3, 3), torch.zeros(4)
    bytes3, wi = torch.zeros(2, 3, 4, dtype=torch.uint8), torch.zeros(4, 3, dtype=torch.int8)
    for call in (lambda: ops.conv2d_f32(image, weights), lambda: ops.conv2d_f32(torch.zeros(2, 3, 4, 4), weights, shape=(2, 3, 4)),
                 lambda: ops.qlinear_conv2d(image, weights, row), lambda: ops.pool2d_f32(image), lambda: ops.maxpool2d_u8(image),
                 lambda: ops.pool2d_f32(torch.zeros(2, 3, 4, 4), pads=(0, 0, 0)), lambda: ops.qlinear_matmul(bytes3, wi, row, row),
                 lambda: ops.gemm_e4m3(bytes3, wi.view(torch.uint8)), lambda: ops.gemm_e4m3_f32(bytes3, wi.view(torch.uint8))):
        with pytest.raises(ValueError):
            call()
    with pytest.raises(IndexError):
        ops.conv2d_f32(torch.zeros(2, 3, 4, 4), weights, pad=(1,))
    for call in (ops.relu_f32, ops.softmax_f32, lambda t: ops.unary_f32(t, "Exp")):
        with pytest.raises(AssertionError):
            call(torch.zeros(4, dtype=torch.bfloat16))
    for call in (lambda: ops.qlinear_matmul_f32(bytes3[0], wi, row, row, None), lambda: ops.conv2d_f32(torch.zeros(2, 3, 4, 4), weights, pad=(1.5, 1.0))):
        with pytest.raises(TypeError):
            call()


@pytest.mark.parametrize("a,b", [((2, 3, 4, 5), (3, 1, 1)), ((7,), (4, 1)), ((1, 6), (5, 1, 6)), ((), (2, 2)), ((0, 3), (1,))])
def test_strides_of_a_broadcast_operand(a, b):
    import torch
    from sofie_b200 import ops
    out, shape4, sa, sb = ops.binary_strides(a, b)
    assert out == tuple(torch.broadcast_shapes(a, b)) and shape4 == [1] * (4 - len(out)) + list(out)
    for operand, strides in ((a, sa), (b, sb)):
        full = (1,) * (4 - len(operand)) + tuple(operand)
        want = torch.empty(operand).reshape(full).stride()
        assert all(s == (0 if n == 1 else w) for n, s, w in zip(full, strides, want) if 0 not in operand)
    with pytest.raises(ValueError):
        ops.binary_strides((1, 1, 1, 1, 2), (1,))
    with pytest.raises(RuntimeError):
        ops.binary_strides((2,), (3,))


def test_transfers_share_the_helper_threads_of_the_process():
    """One transfer may have all cores but two (at most fourteen threads with the caller); transfers at the same time get what is left,
    three helpers at least; one after the other they use the same threads, and none is left when the last context is gone."""
    import os
    import subprocess
    import sys
    script = (
        "import ctypes as C, os, sys\n"
        "sys.path.insert(0, sys.argv[1])\n"
        "from sofie_b200 import capi\n"
        "capi.load()\n"
        "threads = lambda: len(os.listdir('/proc/self/task'))\n"
        "before = threads()\n"
        "h = (C.c_int * 5)()\n"
        "for n in (1, 1, 5, 1):\n"
        "    capi.call('sofie_cuda_selftest_host_pools', n, h)\n"
        "    print(*h[:n])\n"
        "    assert threads() == before, (threads(), before)\n")
    r = subprocess.run([sys.executable, "-c", script, str(ROOT)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    one, again, five, last = [[int(v) for v in line.split()] for line in r.stdout.strip().splitlines()[-4:]]
    cores = len(os.sched_getaffinity(0))
    first = max(min(cores - 2, 14), 1) - 1
    assert one == again == last == [first] and five[0] == first
    assert all(h == min(first, 3) for h in five[1:]) or cores > 17
    assert sum(five) <= max(cores - 2, first + 3 * 4)


def test_helper_threads_that_cannot_be_started_are_done_without(tmp_path):
    """A process at its limit of threads (here: of address space, which their stacks need) copies with the threads it gets."""
    import subprocess
    import sys
    script = (
        "import ctypes as C, resource, sys\n"
        "sys.path.insert(0, sys.argv[1])\n"
        "from sofie_b200 import capi\n"
        "capi.load()\n"
        "used = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()\n"
        "n = 8 << 20\n"
        "libc, src, dst = C.CDLL(None), (C.c_char * n)(*[7] * 64), (C.c_char * n)()\n"
        "used = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()\n"
        "resource.setrlimit(resource.RLIMIT_AS, (used + (20 << 20), used + (20 << 20)))\n"
        "rc = capi.load().sofie_cuda_selftest_host_copy(dst, src, n, 1 << 20, 16, 3)\n"
        "assert rc == 0 and libc.memcmp(dst, src, n) == 0\n"
        "print('ok')\n")
    r = subprocess.run([sys.executable, "-c", script, str(ROOT)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stdout[-2000:])


@pytest.mark.parametrize("nbytes,dst_at,src_at,threads", [(1 << 20, 0, 0, 4), ((1 << 20) + 1, 1, 0, 3), ((5 << 20) - 63, 63, 17, 4), (98304, 16, 3, 2), (300001, 40, 40, 6)])
def test_host_copy_past_the_caches(nbytes, dst_at, src_at, threads):
    """Large results are carried with stores past the caches: any size and any alignment of either side, no byte beyond the end."""
    import numpy as np
    src = np.random.default_rng(nbytes).integers(0, 256, nbytes + 64, dtype=np.uint8)
    dst = np.full(nbytes + 128, 7, np.uint8)
    capi.call("sofie_cuda_selftest_host_copy", dst.ctypes.data + dst_at, src.ctypes.data + src_at, nbytes, 1 << 22, threads, 2)
    assert np.array_equal(dst[dst_at:dst_at + nbytes], src[src_at:src_at + nbytes])
    assert (dst[:dst_at] == 7).all() and (dst[dst_at + nbytes:] == 7).all()


def test_the_cut_of_a_product_does_not_depend_on_the_card():
    """The last bits of a product's sums follow from how it is cut along K: no launcher asks the card it runs on how many clusters it has room for."""
    for p in sorted((ROOT / "sofie_b200" / "csrc").glob("*.cu*")):
        for query in ("cudaOccupancyMaxActive", "cudaDeviceGetAttribute", "cudaGetDeviceProperties"):
            assert query not in p.read_text(), f"{p.name}: {query}"


def test_what_an_earlier_kernel_wrote_is_read_behind_the_wait_for_it():
    """A load through a restrict pointer of a kernel may move before griddep_wait(), unless the pointer is one of its arguments; so may __ldg of a pointer that the kernel did not wait with."""
    weights = {"umma_qconv3x3_first_pool_kernel": {"W"}}   # read before the wait, on purpose
    waiting = 0
    for p in sorted((ROOT / "sofie_b200" / "csrc").glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", p.read_text())
        for m in re.finditer(r"__global__", text):
            start = text.index("{", m.end())
            depth, end = 0, start
            while end == start or depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            head, body = text[m.end():start], text[start:end]
            waits = re.findall(r"griddep_wait\(([^)]*)\)", body)
            if not waits:
                continue
            waiting += 1
            name = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)+", "", head))[0]
            read = {q for q in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s*(\w+)", head)} - weights.get(name, set())
            named = {a.strip() for a in ",".join(waits).split(",")}
            assert read <= named, f"{p.name}: {name} reads {sorted(read - named)} through a restrict pointer behind its wait"
    assert waiting > 30
