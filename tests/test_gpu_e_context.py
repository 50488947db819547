"""Context services on the GPU: the per-context status word with a bounded wait that is made to run out (the kernel
ends by itself, reports once, and the context keeps computing), the per-operator device timers of the emitted
Launch(), Session::RunResident, and two Sessions that do not see each other's failures."""
import ctypes as C
import re

import numpy as np
import pytest
import torch

from oracle import run_model
from sofie_b200 import capi, configs, generated

pytestmark = pytest.mark.gpu


def _ctx(arena=1 << 20):
    ctx = C.c_void_p()
    capi.call("sofie_cuda_ctx_create", C.byref(ctx), 0, arena)
    stream = C.c_void_p()
    capi.call("sofie_cuda_ctx_stream", ctx, C.byref(stream))
    return ctx, stream


def test_bounded_wait_runs_out_reports_once_and_the_context_stays_usable(cuda_device):
    a, sa = _ctx()
    b, sb = _ctx()
    try:
        flag = torch.zeros(1, dtype=torch.int32, device=cuda_device)
        # a barrier nothing arrives on, a limit of 200 000 SM clocks (about 0.1 ms): the kernel gives up and returns
        capi.call("sofie_cuda_selftest_wait_timeout", sa, 200_000, C.c_void_p(flag.data_ptr()))
        with pytest.raises(capi.SofieCudaError) as e:
            capi.call("sofie_cuda_ctx_check", a)
        assert e.value.status == capi.ERR_DEVICE and "0x1ff" in str(e.value) and "0x7e57" in str(e.value)
        assert int(flag.item()) == 1                    # the kernel went through its normal exit (tensor memory released)
        capi.call("sofie_cuda_ctx_check", a)            # reported once, then clear
        capi.call("sofie_cuda_ctx_check", b)            # the other context never saw it
        # the context still computes: a tensor-core GEMM on the same stream, then a clean check
        rng = np.random.default_rng(3)
        A = rng.standard_normal((256, 512)).astype(np.float32)
        B = rng.standard_normal((64, 512)).astype(np.float32)
        dA, dB = torch.from_numpy(A).to(cuda_device), torch.from_numpy(B).to(cuda_device)
        dY = torch.empty(256, 64, device=cuda_device)
        d = capi.GemmF32Desc(256, 64, 512, 0, 1, 1.0, 0.0, 0, 0)
        torch.cuda.synchronize()
        capi.call("sofie_cuda_gemm_f32", sa, C.byref(d), C.c_void_p(dA.data_ptr()), C.c_void_p(dB.data_ptr()), None, C.c_void_p(dY.data_ptr()))
        capi.call("sofie_cuda_ctx_check", a)
        ref = A.astype(np.float64) @ B.astype(np.float64).T
        assert np.abs(dY.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
        # a limit outside the self test's range is refused before anything is launched
        with pytest.raises(capi.SofieCudaError):
            capi.call("sofie_cuda_selftest_wait_timeout", sa, 10**12, None)
    finally:
        capi.call("sofie_cuda_ctx_destroy", a)
        capi.call("sofie_cuda_ctx_destroy", b)


@pytest.mark.parametrize("role,copied,detail", [(0, 8, None), (1, 5, "0x7e5c"), (2, 3, "0x7e59")])
def test_waits_of_whole_warps_run_out(cuda_device, role, copied, detail):
    """A warp whose wait ran out hands nothing on: the copying role gets no slot back from it (stages 0 to 4 of eight fit before that), the
    reading role no accumulator; both leave at once, and the kernel ends behind the last copy and reports."""
    ctx, stream = _ctx()
    try:
        src, out = torch.full((4096,), 3, dtype=torch.uint8, device=cuda_device), torch.zeros(5, dtype=torch.int32, device=cuda_device)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        external = torch.cuda.ExternalStream(stream.value)
        a.record(external)
        capi.call("sofie_cuda_selftest_warp_waits", stream, role, 200_000, C.c_void_p(src.data_ptr()), C.c_void_p(out.data_ptr()))
        b.record(external)
        if role:
            with pytest.raises(capi.SofieCudaError) as e:
                capi.call("sofie_cuda_ctx_check", ctx)
            assert e.value.status == capi.ERR_DEVICE and "0x1ff" in str(e.value) and detail in str(e.value)
        capi.call("sofie_cuda_ctx_check", ctx)
        assert out.tolist() == [1, copied, 0 if role else 1, 1 if role else 0, 1]
        assert a.elapsed_time(b) < (800 if role == 2 else 100)  # ms; the other roles' own limits: a second, and a quarter for the issuer
        for args in ((3, 1000, src, out), (1, 10**12, src, out), (1, 1000, src[1:], out)):
            with pytest.raises(capi.SofieCudaError):
                capi.call("sofie_cuda_selftest_warp_waits", stream, args[0], args[1], *[C.c_void_p(t.data_ptr()) for t in args[2:]])
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


def test_fetch_reports_a_kernel_that_gave_up(cuda_device):
    ctx, stream = _ctx()
    try:
        buf = C.c_void_p()
        capi.call("sofie_cuda_ctx_arena", ctx, 0, 1024, C.byref(buf))
        capi.call("sofie_cuda_selftest_wait_timeout", stream, 100_000, None)
        host = C.c_void_p()
        with pytest.raises(capi.SofieCudaError) as e:   # what the emitted infer() turns into std::runtime_error
            capi.call("sofie_cuda_ctx_fetch", ctx, buf, 1024, C.byref(host))
        assert e.value.status == capi.ERR_DEVICE
        capi.call("sofie_cuda_ctx_fetch", ctx, buf, 1024, C.byref(host))
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


def test_copies_are_refused_during_a_graph_capture(cuda_device):
    ctx, _ = _ctx()
    try:
        buf = C.c_void_p()
        capi.call("sofie_cuda_ctx_arena", ctx, 0, 1024, C.byref(buf))
        src = np.zeros(256, np.float32)
        capi.call("sofie_cuda_ctx_graph_begin", ctx)
        for name, args in (("sofie_cuda_ctx_h2d", (ctx, buf, src.ctypes.data_as(C.c_void_p), 1024)),
                           ("sofie_cuda_ctx_d2h", (ctx, src.ctypes.data_as(C.c_void_p), buf, 1024)),
                           ("sofie_cuda_ctx_check", (ctx,))):
            with pytest.raises(capi.SofieCudaError) as e:
                capi.call(name, *args)
            assert e.value.status == capi.ERR_INVALID
        capi.call("sofie_cuda_ctx_graph_end", ctx)
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


def test_operator_timers_and_run_resident_of_the_emitted_session(cuda_device, monkeypatch):
    m, x = configs.cnn_f32(batch=32)
    ref = run_model.run(m, x).ravel()
    plain = generated.session_from_model(m, "c2_b32_timers")
    y0 = plain.infer(x)
    n = C.c_int(-1)
    capi.call("sofie_cuda_ctx_timers_read", plain.ctx, None, 0, C.byref(n))
    assert n.value == 0                                     # timers are off unless asked for
    monkeypatch.setenv("SOFIE_CUDA_TIMERS", "1")
    timed = generated.session_from_model(m, "c2_b32_timers")
    monkeypatch.delenv("SOFIE_CUDA_TIMERS")
    plan = generated.launch_plan(timed.hxx)
    assert [p["calls"] for p in plan] == [["sofie_cuda_conv2d_f32"]] * 3 + [[], ["sofie_cuda_gemm_f32"]]   # Flatten is an alias
    assert sum(p["flops"] for p in plan) == m.flops_per_sample * 32
    ms = (C.c_float * len(plan))()
    for _ in range(3):                                      # eager pass, capturing pass, graph replay
        y = timed.infer(x)
        capi.call("sofie_cuda_ctx_timers_read", timed.ctx, ms, len(plan), C.byref(n))
        assert n.value == len(plan) and all(0.0 <= t < 50.0 for t in ms)
        assert np.array_equal(y, y0)
    assert np.abs(y0 - ref).max() <= 1e-5 * np.abs(ref).max()
    # RunResident: the kernels again on the input the last infer() left on the device, no copies
    stream = C.c_void_p()
    capi.call("sofie_cuda_ctx_stream", plain.ctx, C.byref(stream))
    plain.run_resident()
    plain.run_resident()
    capi.call("sofie_cuda_ctx_check", plain.ctx)
    assert np.array_equal(plain.infer(x), y0)


def test_shared_memory_allowed_for_one_network_survives_a_smaller_one_on_another_thread(cuda_device):
    """The allowance of a kernel's dynamic shared memory belongs to the process: a thread whose network needs less must not take it away
    from one whose network needs more, neither for operator calls nor for the replay of a captured Session of one kernel."""
    import threading
    from sofie_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(5)

    def net(width):
        w = [torch.randn(width, 64, device="cuda", generator=g), torch.randn(10, width, device="cuda", generator=g)]
        x = torch.randn(40, 64, device="cuda", generator=g)
        return lambda: ops.mlp_f32(x, w, [None, None], [1, 0], [1, 1]).cpu()
    large, small = net(240), net(96)
    sessions = {}
    for width in (240, 96):
        m, x = configs.mlp_f32(batch=40, dims=(64, width, 10))
        s = generated.session_from_model(m, f"c1_smem_{width}")
        sessions[width] = (s, x)
    first = {}

    def elsewhere(f):
        box = []
        t = threading.Thread(target=lambda: box.append(f()))
        t.start()
        t.join()
        assert box, "the call on the other thread failed"
        return box[0]
    first["large"] = large()
    s, x = sessions[240]
    first[240] = [s.infer(x) for _ in range(3)][-1]      # the third is a replay
    for _ in range(2):
        elsewhere(small)
        s2, x2 = sessions[96]
        elsewhere(lambda: s2.infer(x2))
        assert torch.equal(large(), first["large"])
        assert np.array_equal(s.infer(x), first[240])


@pytest.mark.parametrize("kind", ["u8", "u8 ranges", "e4m3"])
def test_run_resident_after_an_input_the_host_quantised(kind, cuda_device):
    """RunResident() runs every kernel of one inference, QuantizeLinear too, on the last infer()'s input -- also when that input was
    pageable and only its quantised form is on the device. The result of every repetition is the one infer() gave."""
    if kind == "e4m3":
        m, x = configs.gemm_chain_fp8(rows=64, width=256, layers=4)
        x[0, :8] = [0., -0., 1e9, -1e9, 1e-9, -1e-9, np.nan, 3.]
        s = generated.session_from_model(m, "c4_resident", fp8_scales=configs.calibrate_fp8_scales(m, np.nan_to_num(x)))
    else:
        m, x = configs.mlp_i8(batch=4096 if "ranges" in kind else 100, dims=(512, 256, 128, 64, 10))
        x[0, :6] = [0., 1e9, -1e9, np.nan, np.inf, -np.inf]
        s = generated.session_from_model(m, f"c3_resident_{m.batch()}")
    y = s.infer(x)
    text = s.hxx.read_text()
    where = re.search(r"sofie_cuda_ctx_(arena|host_output)\(fCtx, (\d+)[^&]*&dev_" + m.output_name + r"\)", text)
    out = C.c_void_p()
    if where.group(1) == "arena":
        capi.call("sofie_cuda_ctx_arena", s.ctx, int(where.group(2)), y.nbytes, C.byref(out))
    for _ in range(3):
        s.run_resident()
        capi.call("sofie_cuda_ctx_check", s.ctx)
        if where.group(1) == "arena":
            again = np.empty_like(y)
            capi.call("sofie_cuda_ctx_d2h", s.ctx, again.ctypes.data_as(C.c_void_p), out, y.nbytes)
            assert np.array_equal(again.view(np.uint32), y.view(np.uint32))
    for _ in range(2):
        assert np.array_equal(s.infer(x).view(np.uint32), y.view(np.uint32))


def test_e4m3_codes_and_their_values(cuda_device):
    from sofie_b200 import ops
    codes = torch.arange(256, dtype=torch.uint8, device="cuda")
    for scale in (1.0, 0.0123, 3.7e5):
        v = torch.empty(256, device="cuda")
        capi.call("sofie_cuda_dequantize_e4m3_f32", None, C.c_void_p(codes.data_ptr()), C.c_void_p(v.data_ptr()), 256, scale)
        torch.cuda.synchronize()
        want = codes.view(torch.float8_e4m3fn).float() * scale
        assert torch.equal(v.nan_to_num(-7.), want.nan_to_num(-7.))
        back = ops.quantize_e4m3(v, scale)
        number = (codes & 127) != 127
        assert torch.equal(back[number], codes[number]) and bool((back[~number] & 127 == 127).all())


def test_pinned_and_pageable_inputs_in_turn(cuda_device):
    """Each kind of input has a graph of its own (with and without QuantizeLinear); results are the same bytes, and so after another batch."""
    m, x = configs.mlp_i8(batch=96, dims=(512, 256, 128, 64, 10))
    pinned = torch.from_numpy(x).pin_memory().numpy()
    s = generated.session_from_model(m, "c3_turns")
    want = s.infer(pinned)
    ready = C.c_int()
    for i in range(9):
        assert np.array_equal(s.infer(x if i % 2 else pinned).view(np.uint32), want.view(np.uint32))
        if i == 1:
            capi.call("sofie_cuda_ctx_graph_swap", s.ctx)
            capi.call("sofie_cuda_ctx_graph_ready", s.ctx, C.byref(ready))
            assert ready.value                    # the pinned input's graph is still there
            capi.call("sofie_cuda_ctx_graph_swap", s.ctx)
    d = generated.dynamic_session_from_model(m, "c3_turns_dyn", 96)
    for n in (96, 50, 96):
        for source in (x, pinned, x):
            assert np.array_equal(d.infer(source[:n]).view(np.uint32), want.view(np.uint32)[:n * 10])


def test_operator_timers_of_a_session_that_cuts_its_batch(cuda_device, monkeypatch):
    """With the timers on a batch that would be cut into ranges, from memory whose quantisation the host would take over, is launched
    operator by operator: one interval for each, QuantizeLinear's among them, and the same result."""
    m, x = configs.mlp_i8(batch=4099)
    y0 = generated.session_from_model(m, "c3_b4099_timed").infer(x)
    monkeypatch.setenv("SOFIE_CUDA_TIMERS", "1")
    timed = generated.session_from_model(m, "c3_b4099_timed")
    monkeypatch.delenv("SOFIE_CUDA_TIMERS")
    plan = generated.launch_plan(timed.hxx)
    assert plan[0]["calls"] == ["sofie_cuda_quantize_u8"]
    n, ms = C.c_int(-1), (C.c_float * len(plan))()
    for _ in range(3):
        assert np.array_equal(timed.infer(x).view(np.uint32), y0.view(np.uint32))
        capi.call("sofie_cuda_ctx_timers_read", timed.ctx, ms, len(plan), C.byref(n))
        assert n.value == len(plan) and all(0.0 <= t < 50.0 for t in ms) and ms[0] > 0.0


_READ_AFTER_FAILURE = r"""
import ctypes as C, mmap, sys, time
sys.path.insert(0, sys.argv[1])
from sofie_b200 import capi
libc = C.CDLL(None, use_errno=True)
libc.mprotect.argtypes = [C.c_void_p, C.c_size_t, C.c_int]
ctx, dst, size = C.c_void_p(), C.c_void_p(), 64 << 20
capi.call("sofie_cuda_ctx_create", C.byref(ctx), -1, size)
capi.call("sofie_cuda_ctx_arena", ctx, 0, size, C.byref(dst))
m = mmap.mmap(-1, size)
src = C.addressof(C.c_char.from_buffer(m))
C.memset(src, 1, size)
lib = capi.load()
for i in range(40):
    capi.call("sofie_cuda_selftest_fail_copy", ctx, 1 + i % 5)
    rc = (lib.sofie_cuda_ctx_h2d(ctx, dst, src, size) if i % 2 else lib.sofie_cuda_ctx_h2d_quantized(ctx, dst, src, size // 4, 1, 0.1, 3, -1))
    assert libc.mprotect(src, size, 0) == 0          # the caller's memory goes away: a reader would be killed
    assert rc == capi.ERR_CUDA, rc
    time.sleep(0.002)
    assert libc.mprotect(src, size, 3) == 0
capi.call("sofie_cuda_ctx_h2d", ctx, dst, src, size)
capi.call("sofie_cuda_ctx_sync", ctx)
capi.call("sofie_cuda_ctx_destroy", ctx)
print("ok")
"""


def test_no_helper_reads_the_source_of_a_copy_that_failed(cuda_device, tmp_path):
    import subprocess
    import sys
    from pathlib import Path
    script = tmp_path / "read_after_failure.py"
    script.write_text(_READ_AFTER_FAILURE)
    r = subprocess.run([sys.executable, str(script), str(Path(__file__).resolve().parents[1])], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stdout[-2000:])


def test_no_copy_writes_the_result_of_an_inference_that_failed(cuda_device):
    """infer() into pinned memory of the caller that fails between two ranges: earlier ranges' results are not on their way any more."""
    import time
    m, x = configs.mlp_i8(batch=16387)
    s = generated.session_from_model(m, "c3_b16387")
    want = s.infer(x)
    out = torch.empty(want.size, pin_memory=True).numpy()
    for nth in (5, 6, 8, 10):                   # the first range is copied in four pieces, each later one in one
        capi.call("sofie_cuda_selftest_fail_copy", s.ctx, nth)
        with pytest.raises(RuntimeError):
            s.infer(x, out)
        out.fill(-12345.)
        time.sleep(0.02)
        assert (out == -12345.).all()
        assert s.infer(x, out) is out and np.array_equal(out.view(np.uint32), want.view(np.uint32))


def test_a_part_nobody_waited_for_keeps_its_staging_slots(cuda_device):
    """An input part that is still on its way when a result ends: its bytes in the staging ring are not overwritten by the next copy."""
    ctx, _ = _ctx(64 << 20)
    try:
        n = 24 << 20
        first, second, result, host = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p()
        for p, off, size in ((first, 0, n), (second, n, n), (result, 2 * n, 256)):
            capi.call("sofie_cuda_ctx_arena", ctx, off, size, C.byref(p))
        a, b = np.full(n, 1, np.uint8), np.full(n, 2, np.uint8)
        for _ in range(60):
            capi.call("sofie_cuda_ctx_result_begin", ctx, None, 256)
            capi.call("sofie_cuda_ctx_h2d_part", ctx, first, a.ctypes.data_as(C.c_void_p), n, 0)
            capi.call("sofie_cuda_ctx_result_part", ctx, result, 0, 256)
            capi.call("sofie_cuda_ctx_result_end", ctx, C.byref(host))
            capi.call("sofie_cuda_ctx_h2d_part", ctx, second, b.ctypes.data_as(C.c_void_p), n, 1)
            capi.call("sofie_cuda_ctx_wait_part", ctx, 0)
            capi.call("sofie_cuda_ctx_wait_part", ctx, 1)
            got = np.zeros(n, np.uint8)
            capi.call("sofie_cuda_ctx_d2h", ctx, got.ctypes.data_as(C.c_void_p), first, n)
            assert (got == 1).all()
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


def test_sessions_share_the_helper_threads(cuda_device):
    """Sessions called one after the other add no threads; called at the same time from several threads they give the same results."""
    import os
    import threading
    m, x = configs.mlp_i8(batch=2048)
    sessions = [generated.session_from_model(m, "c3_b2048_threads") for _ in range(6)]
    want = sessions[0].infer(x)
    threads = len(os.listdir("/proc/self/task"))
    for s in sessions:
        assert np.array_equal(s.infer(x).view(np.uint32), want.view(np.uint32))
    assert len(os.listdir("/proc/self/task")) <= threads + 2        # the driver's own, at most
    wrong = []

    def work(s):
        for _ in range(50):
            if not np.array_equal(s.infer(x).view(np.uint32), want.view(np.uint32)):
                wrong.append(1)
    workers = [threading.Thread(target=work, args=(s,)) for s in sessions]
    for t in workers:
        t.start()
    for t in workers:
        t.join()
    assert not wrong


@pytest.mark.parametrize("nbytes", [(5 << 19) - 4, 5 << 19, (4 << 20) + 12, (17 << 20) + 4100, (70 << 20) + 1])
def test_results_land_in_pieces(cuda_device, nbytes):
    """A result for pageable memory, as one part: it lands whole or in two to eight pieces, the same bytes and nothing beside them; a second part
    after it (the same bytes again) is refused or lands too, and an abandoned result leaves the context usable."""
    x = torch.randint(0, 256, (nbytes,), dtype=torch.uint8, device=cuda_device)
    torch.cuda.synchronize()
    ctx, _ = _ctx()
    host = C.c_void_p()
    try:
        out = np.full(nbytes + 64, 7, np.uint8)
        for _ in range(2):
            out[:] = 7
            capi.call("sofie_cuda_ctx_result_begin", ctx, C.c_void_p(out.ctypes.data), C.c_size_t(nbytes))
            capi.call("sofie_cuda_ctx_result_part", ctx, C.c_void_p(x.data_ptr()), C.c_size_t(0), C.c_size_t(nbytes))
            capi.call("sofie_cuda_ctx_result_end", ctx, C.byref(host))
            assert host.value == out.ctypes.data and np.array_equal(out[:nbytes], x.cpu().numpy()) and (out[nbytes:] == 7).all()
        capi.call("sofie_cuda_ctx_result_begin", ctx, C.c_void_p(out.ctypes.data), C.c_size_t(nbytes))
        for _ in range(8):
            try:
                capi.call("sofie_cuda_ctx_result_part", ctx, C.c_void_p(x.data_ptr()), C.c_size_t(0), C.c_size_t(nbytes))
            except capi.SofieCudaError as e:
                assert e.status == capi.ERR_INVALID
        capi.call("sofie_cuda_ctx_result_abort", ctx)
        capi.call("sofie_cuda_ctx_check", ctx)
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


@pytest.mark.parametrize("nbytes", [3, 524288, 524288 + 19, 700001, 1 << 20, (1 << 20) + 1, 3 << 20])
def test_inputs_from_pageable_memory(cuda_device, nbytes):
    """One kernel's fetch, two of them with a ragged end, and the copies above: the same bytes, nothing beside them, twice with other bytes."""
    rng = np.random.default_rng(nbytes)
    dst = torch.zeros(nbytes + 64, dtype=torch.uint8, device=cuda_device)
    torch.cuda.synchronize()
    ctx, _ = _ctx()
    try:
        for _ in range(2):
            x = rng.integers(1, 256, nbytes, dtype=np.uint8)
            capi.call("sofie_cuda_ctx_h2d", ctx, C.c_void_p(dst.data_ptr()), C.c_void_p(x.ctypes.data), C.c_size_t(nbytes))
            capi.call("sofie_cuda_ctx_check", ctx)
            got = dst.cpu().numpy()
            assert np.array_equal(got[:nbytes], x) and not got[nbytes:].any()
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


@pytest.mark.parametrize("part", [None, 0])
@pytest.mark.parametrize("ahead,nbytes", [(1, 4096), (1001, 4096), (1001, 300000), (4096, 300000), (4100, 700001), (16, 17), (2 << 20, 3 << 20)])
def test_a_fill_ahead_that_is_shorter_than_its_copy(cuda_device, ahead, nbytes, part):
    """The helpers were started on fewer bytes than the copy takes, on whatever number the caller named: the pieces behind it begin on no boundary."""
    rng = np.random.default_rng(ahead + nbytes)
    dst = torch.zeros(nbytes + 64, dtype=torch.uint8, device=cuda_device)
    torch.cuda.synchronize()
    ctx, _ = _ctx()
    try:
        for _ in range(2):
            x = rng.integers(1, 256, nbytes, dtype=np.uint8)
            capi.call("sofie_cuda_ctx_stage_ahead", ctx, C.c_void_p(x.ctypes.data), C.c_size_t(ahead), 0, 1.0, 0)
            args = (ctx, C.c_void_p(dst.data_ptr()), C.c_void_p(x.ctypes.data), C.c_size_t(nbytes))
            if part is None:
                capi.call("sofie_cuda_ctx_h2d", *args)
            else:
                capi.call("sofie_cuda_ctx_h2d_part", *args, part)
                capi.call("sofie_cuda_ctx_wait_part", ctx, part)
            capi.call("sofie_cuda_ctx_check", ctx)
            got = dst.cpu().numpy()
            assert np.array_equal(got[:nbytes], x) and not got[nbytes:].any()
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)


@pytest.mark.parametrize("nbytes", [(5 << 19) - 4, 5 << 19, (4 << 20) + 12, (17 << 20) + 4100, (70 << 20) + 1])
def test_parts_after_a_whole_result(cuda_device, nbytes):
    """A result for pageable memory whose first part is all of it, in one piece or several: seven more parts are taken after it, whole or not, and a ninth is refused."""
    x = torch.randint(0, 256, (nbytes,), dtype=torch.uint8, device=cuda_device)
    torch.cuda.synchronize()
    ctx, _ = _ctx()
    host = C.c_void_p()
    try:
        out = np.full(nbytes + 64, 7, np.uint8)
        third = nbytes // 3
        for again in ((0, nbytes), (third, nbytes - third)):
            out[:] = 7
            capi.call("sofie_cuda_ctx_result_begin", ctx, C.c_void_p(out.ctypes.data), C.c_size_t(nbytes))
            for offset, count in ((0, nbytes),) + 7 * (again,):
                capi.call("sofie_cuda_ctx_result_part", ctx, C.c_void_p(x.data_ptr() + offset), C.c_size_t(offset), C.c_size_t(count))
            with pytest.raises(capi.SofieCudaError) as e:
                capi.call("sofie_cuda_ctx_result_part", ctx, C.c_void_p(x.data_ptr()), C.c_size_t(0), C.c_size_t(nbytes))
            assert e.value.status == capi.ERR_INVALID
            capi.call("sofie_cuda_ctx_result_end", ctx, C.byref(host))
            assert np.array_equal(out[:nbytes], x.cpu().numpy()) and (out[nbytes:] == 7).all()
    finally:
        capi.call("sofie_cuda_ctx_destroy", ctx)
