"""The library's host code on a fake CUDA runtime (fake_cudart.cpp): its own objects, linked against functions that copy with
memcpy and write launches down. What goes wrong with threads, streams, contexts and captures shows here without a GPU."""
import ctypes
import glob
import os
import subprocess
import sys
import threading

import pytest

import cabi

MB = 1 << 20
PER_THREAD_STREAM = 2        # cudaStreamPerThread


def build_fake(directory):
    import importlib.util
    spec = importlib.util.spec_from_file_location("ttb_build", os.path.join(cabi.ROOT, "tt-metal_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build_libttb()
    so = os.path.join(directory, "libttb_fake.so")
    # (-Bsymbolic: its own copies of the runtime, whatever else the process has loaded)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wno-attributes", "-I/usr/local/cuda/include",
                    os.path.join(cabi.ROOT, "tests", "fake_cudart.cpp")] + sorted(glob.glob(os.path.join(build.OBJ, "*.o"))) +
                   ["-o", so, "-lpthread", "-ldl"], check=True)
    return so


@pytest.fixture(scope="module")
def fake_so(tmp_path_factory):
    return build_fake(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture(scope="module")
def fake(fake_so):
    lib = cabi.Lib(fake_so)
    lib.cdll.fake_log.restype = ctypes.c_char_p
    return lib


def round_trip(lib, nbytes, stream=None):
    """Host to device and back; both host buffers are pageable, the device's is plain memory here."""
    src, dev, dst = os.urandom(nbytes), ctypes.create_string_buffer(nbytes), ctypes.create_string_buffer(nbytes)
    lib.check(lib.cdll.ttb_memcpy_h2d(dev, src, nbytes, stream))
    lib.check(lib.cdll.ttb_memcpy_d2h(dst, dev, nbytes, stream))
    assert dst.raw == src


def test_copies_on_the_per_thread_stream_stay_on_the_callers_thread(fake):
    """The handle names another stream on every thread: whoever enqueues on it elsewhere is not ordered after the caller's work."""
    fake.cdll.fake_stream_users()
    round_trip(fake, 9 * MB + 5, PER_THREAD_STREAM)
    assert fake.cdll.fake_stream_users() == 1
    round_trip(fake, 9 * MB + 5)
    assert fake.cdll.fake_stream_users() > 1      # the legacy stream is the same on all of them


@pytest.mark.parametrize("nbytes,to_device,to_host", [(4 * MB - 1, False, False), (4 * MB, False, True), (5 * MB - 1, False, True), (5 * MB, True, True)])
def test_copies_are_staged_from_the_size_that_measured_faster(fake, nbytes, to_device, to_host):
    dev, host = ctypes.create_string_buffer(nbytes), ctypes.create_string_buffer(nbytes)
    for copy, dst, src, staged in ((fake.cdll.ttb_memcpy_h2d, dev, host, to_device), (fake.cdll.ttb_memcpy_d2h, host, dev, to_host)):
        fake.cdll.fake_stream_users()
        fake.check(copy(dst, src, nbytes, None))
        assert (fake.cdll.fake_stream_users() > 1) == staged


def test_a_stream_of_another_context_takes_the_plain_copy(fake):
    """Handle 0x300 belongs to a context that is not current (another device's, for instance): events of the current one cannot be
    recorded there."""
    fake.cdll.fake_stream_users()
    round_trip(fake, 8 * MB, 0x300)
    assert fake.cdll.fake_stream_users() == 1


def test_a_callers_own_context_stays_current_and_is_the_helpers(fake):
    """A context made through the driver API, not the device's primary one: the helper threads work in it, and it stays current."""
    def work():
        fake.cdll.fake_context(1)
        before = fake.cdll.fake_set_device_calls()
        round_trip(fake, 8 * MB + 1, 0x300)                                  # a stream of that context
        result.extend([fake.cdll.fake_context_is_other(), fake.cdll.fake_set_device_calls() - before])

    result = []
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert result == [1, 0]


def test_a_first_large_copy_leaves_another_threads_capture_intact(fake):
    """While some thread captures in global mode, allocations and waits of the others are forbidden calls that end its capture,
    unless they declare themselves relaxed. The plain copy made none; its pinned buffers, allocated by the first copy, may not either."""
    fake.cdll.fake_reset_device()
    fake.cdll.fake_capture(1)
    try:
        round_trip(fake, 8 * MB)
        assert fake.cdll.fake_violations() == 0
        assert fake.cdll.ttb_stream_synchronize(None) != 0 and fake.cdll.fake_violations() == 1   # the caller's own mode is as it was
    finally:
        fake.cdll.fake_capture(0)


def test_pinned_buffers_are_allocated_again_once_their_context_is_gone(fake):
    """cudaDeviceReset and a destroyed context take the pinned buffers with them."""
    round_trip(fake, 8 * MB)
    assert fake.cdll.fake_pinned() == 1
    fake.cdll.fake_reset_device()
    round_trip(fake, 8 * MB)
    assert fake.cdll.fake_pinned() == 1


@pytest.mark.parametrize("failing", range(4))
def test_a_thread_that_cannot_be_made_is_done_without(fake, failing):
    """std::thread's own allocation fails (std::bad_alloc, not std::system_error): no exception leaves the C entry point, the threads
    that did start are joined, and the bytes are right."""
    src, dev = os.urandom(16 * MB + 3), ctypes.create_string_buffer(16 * MB + 3)
    fake.cdll.fake_fail_new(failing)
    try:
        rc = fake.cdll.ttb_memcpy_h2d(dev, src, len(src), None)
    finally:
        fake.cdll.fake_fail_new(-1)
    assert rc == 0 and dev.raw == src


@pytest.mark.parametrize("w_dtype", [cabi.BFLOAT16, cabi.BFLOAT8_B, cabi.BFLOAT4_B])
def test_first_calls_of_several_threads_set_a_kernel_up_once(fake_so, w_dtype):
    """The launch reads what the set-up of its device counted: a second thread waits until that is there. (A process of its own: the
    set-up is done once.)"""
    code = """if True:
        import ctypes, sys, threading
        sys.path.insert(0, %r)
        import cabi
        lib = cabi.Lib(%r)
        lib.cdll.fake_log.restype = ctypes.c_char_p
        lib.cdll.fake_slow_us(20000)
        go, codes = threading.Barrier(4), []
        def work():
            go.wait()
            codes.append(lib.cdll.ttb_matmul(4096, 0, 8192, %d, None, 16384, 0, 1, 128, 4096, 256, 0, 8, None, 0, None))
        threads = [threading.Thread(target=work) for _ in range(4)]
        [t.start() for t in threads]; [t.join() for t in threads]
        log = lib.cdll.fake_log().decode().split()
        assert codes == [0] * 4 and len(log) == 4 and len(set(log)) == 1, (codes, log)
        print(lib.cdll.fake_most_configured())
    """ % (os.path.join(cabi.ROOT, "tests"), fake_so, w_dtype)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "1", r.stdout + r.stderr


KERNEL_NAMES = {cabi.KERNEL_GENERIC: "matmul_generic_kernel", cabi.KERNEL_ROWS: "matmul_rows_kernel", cabi.KERNEL_BF16: "matmul_bf16_kernel"}


@pytest.mark.parametrize("out_dtype", [cabi.BFLOAT16, cabi.FLOAT32])
@pytest.mark.parametrize("w_dtype", [cabi.BFLOAT16, cabi.BFLOAT8_B, cabi.BFLOAT4_B])
@pytest.mark.parametrize("flags", [0, cabi.MM_DETERMINISTIC, cabi.MM_FORCE_GENERIC])
def test_matmul_kernel_names_the_kernel_that_is_launched(fake, w_dtype, out_dtype, flags):
    """ttb_matmul_kernel against the launches that ttb_matmul makes, and the launches of row ranges against ttb_matmul_plan."""
    seen = set()
    for M in (32, 64, 96, 256, 320, 512, 544, 2048):
        for K, N in ((32, 96), (512, 512), (1024, 4672), (4096, 4096), (8192, 9472)):
            kind = fake.cdll.ttb_matmul_kernel(w_dtype, out_dtype, 1, M, K, N, flags)
            fake.cdll.fake_log()
            rc = fake.cdll.ttb_matmul(4096, cabi.BFLOAT16, 8192, w_dtype, None, 1 << 20, out_dtype, 1, M, K, N, 0, flags | cabi.MM_WORKSPACE_ZEROED, 1 << 21, 1 << 40, None)
            log = fake.cdll.fake_log().decode().split()
            assert rc == 0 and log, (M, K, N, rc)
            if kind == cabi.KERNEL_RANGES:
                plan = (ctypes.c_int64 * 33)()
                assert fake.cdll.ttb_matmul_plan(w_dtype, 1, M, K, N, flags, plan, 33) == 0
                decode = sum("matmul_decode" in k for k in log)
                assert decode == list(plan)[2:2 + 2 * plan[0]:2].count(0) and not any(n in k for k in log for n in KERNEL_NAMES.values()), (M, K, N, log)
            else:
                assert all(KERNEL_NAMES[kind] in k for k in log), (M, K, N, kind, log)
            seen.add(kind)
    block_float = {cabi.KERNEL_RANGES, cabi.KERNEL_ROWS} if out_dtype == cabi.BFLOAT16 and not flags else {cabi.KERNEL_RANGES}
    bf16 = {cabi.KERNEL_BF16, cabi.KERNEL_GENERIC}
    assert seen == ({cabi.KERNEL_GENERIC} if flags & cabi.MM_FORCE_GENERIC else bf16 if w_dtype == cabi.BFLOAT16 else block_float)
    assert fake.cdll.ttb_matmul_kernel(w_dtype, out_dtype, 1, 32, 48, 64, flags) == -1


def kernel(lib, M, K, N, w_dtype=cabi.BFLOAT8_B):
    return lib.cdll.ttb_matmul_kernel(w_dtype, cabi.BFLOAT16, 1, M, K, N, 0)


@pytest.mark.parametrize("w_dtype", [cabi.BFLOAT8_B, cabi.BFLOAT4_B])
def test_96_to_256_rows_take_the_kernel_that_measured_faster(fake, w_dtype):
    """Shapes on either side of the line between the decode and the middling-rows kernel, each faster on its side; as one
    weight, and as several that together have its column tiles. (Timings in the comments of the rules.)"""
    decode = [(224, 128, 1024), (224, 512, 1024), (160, 256, 1024), (160, 512, 3072), (96, 640, 4096), (96, 1024, 3072), (224, 1024, 2048), (160, 768, 2048),
              (96, 28672, 256), (96, 12288, 512), (160, 20480, 512), (224, 28672, 384), (256, 20480, 128), (128, 28672, 512), (192, 28672, 256), (192, 28672, 1024)]
    rows = [(96, 256, 1024), (160, 256, 4096), (96, 1024, 1024), (192, 512, 1024), (128, 512, 128), (224, 512, 3072), (160, 1536, 512), (96, 512, 6144),
            (96, 8192, 512), (128, 12288, 256), (160, 28672, 768), (256, 12288, 256), (96, 28672, 1536), (224, 20480, 512), (256, 4096, 128)]
    for want, shapes in ((cabi.KERNEL_RANGES, decode), (cabi.KERNEL_ROWS, rows)):
        for M, K, N in shapes:
            assert kernel(fake, M, K, N, w_dtype) == want, (M, K, N)
            Ns = (N // 2, N - N // 2) if N % 256 == 0 else (N,)
            P = lambda at: (ctypes.c_void_p * len(Ns))(*[at + (j << 30) for j in range(len(Ns))])   # noqa: E731
            fake.cdll.fake_log()
            fake.check(fake.cdll.ttb_matmul_multi(4096, cabi.BFLOAT16, len(Ns), P(1 << 34), w_dtype, None, P(1 << 38), cabi.BFLOAT16, 1, M, K,
                                                  (ctypes.c_int64 * len(Ns))(*Ns), 0, cabi.MM_WORKSPACE_ZEROED, 1 << 40, 1 << 40, None, None, None))
            log = fake.cdll.fake_log().decode().split()
            assert log and all(("matmul_decode" if want == cabi.KERNEL_RANGES else "matmul_rows") in k for k in log), (M, K, Ns, log)


@pytest.mark.parametrize("shape,w_dtype,prefill", [
    # short K ranges: nearly full last rounds, then broken ones and blocks that are not 256 x 256
    ((1024, 256, 9472), cabi.BFLOAT8_B, True), ((1024, 1024, 18944), cabi.BFLOAT8_B, True), ((1024, 512, 16384), cabi.BFLOAT4_B, True),
    ((2048, 512, 28672), cabi.BFLOAT4_B, True), ((1536, 512, 28672), cabi.BFLOAT8_B, True), ((768, 512, 12544), cabi.BFLOAT4_B, True),
    ((512, 1024, 28416), cabi.BFLOAT8_B, False), ((640, 1024, 14336), cabi.BFLOAT4_B, False), ((512, 1024, 14208), cabi.BFLOAT8_B, False),
    ((1024, 2048, 9472), cabi.BFLOAT8_B, False), ((2048, 512, 16384), cabi.BFLOAT8_B, False), ((512, 512, 9472), cabi.BFLOAT8_B, False),
    # long ones
    ((1024, 8192, 18944), cabi.BFLOAT8_B, True), ((1024, 8192, 28416), cabi.BFLOAT8_B, True), ((1024, 28672, 8192), cabi.BFLOAT8_B, True),
    ((2048, 8192, 28672), cabi.BFLOAT8_B, True), ((2048, 12288, 18944), cabi.BFLOAT4_B, True), ((2048, 8192, 28416), cabi.BFLOAT4_B, True),
    ((2048, 8192, 4096), cabi.BFLOAT8_B, False), ((2048, 8192, 8192), cabi.BFLOAT8_B, False), ((1024, 8192, 18944), cabi.BFLOAT4_B, False),
    ((2048, 4096, 28672), cabi.BFLOAT8_B, False), ((2048, 8192, 28672), cabi.BFLOAT4_B, False), ((1024, 4096, 9472), cabi.BFLOAT8_B, False)])
def test_512_rows_and_more_take_the_kernel_that_measured_faster(fake, shape, w_dtype, prefill):
    """Shapes on either side of the line between the prefill and the middling-rows kernel."""
    assert kernel(fake, *shape, w_dtype) == (cabi.KERNEL_RANGES if prefill else cabi.KERNEL_ROWS)


@pytest.mark.parametrize("batch,M,K,N,tensor_cores", [
    (1, 32, 32, 32, False), (1, 128, 32, 512, False), (1, 512, 32, 512, False), (1000, 32, 32, 32, False), (4000, 32, 64, 32, False), (32, 64, 32, 64, False),
    (1, 1024, 32, 1024, True), (32, 128, 32, 128, True), (500, 32, 64, 32, True), (1, 32, 64, 1024, True), (1000, 32, 64, 128, True), (1, 32, 96, 32, True)])
def test_small_bfloat16_products_take_the_kernel_that_measured_faster(fake, batch, M, K, N, tensor_cores):
    """Batched (ttb_bmm) and, for one matrix, also as a linear: shapes on either side of the line between CUDA and tensor cores."""
    fake.cdll.fake_log()
    fake.check(fake.cdll.ttb_bmm(4096, cabi.BFLOAT16, 8192, cabi.BFLOAT16, 16384, cabi.BFLOAT16, batch, M, K, N, None))
    log = fake.cdll.fake_log().decode().split()
    assert len(log) == 1 and ("matmul_bf16_kernel" in log[0]) == tensor_cores, log
    if batch == 1:
        assert kernel(fake, M, K, N, cabi.BFLOAT16) == (cabi.KERNEL_BF16 if tensor_cores else cabi.KERNEL_GENERIC)


@pytest.mark.parametrize("M,K,N", [(96, 28672, 256), (256, 20480, 128), (1024, 8192, 9472), (512, 512, 18944)])
@pytest.mark.parametrize("workspace,nbytes", [(None, 0), (1 << 40, 16), ((1 << 40) + 16, 1 << 40)])
def test_calls_without_scratch_get_the_kernel_that_needs_none(fake, M, K, N, workspace, nbytes):
    """Shapes that go to the decode or prefill kernel with the workspace they ask for: with none, too little or a misaligned one they
    are served all the same; under MM_DETERMINISTIC, which only those kernels serve, they are refused."""
    assert kernel(fake, M, K, N) == cabi.KERNEL_RANGES and fake.matmul_workspace_bytes(cabi.BFLOAT8_B, 1, M, K, N, 0) > 0
    run = lambda flags: fake.cdll.ttb_matmul(4096, cabi.BFLOAT16, 8192, cabi.BFLOAT8_B, None, 1 << 20, cabi.BFLOAT16, 1, M, K, N, 0, flags, workspace, nbytes, None)   # noqa: E731
    fake.cdll.fake_log()
    assert run(0) == 0
    log = fake.cdll.fake_log().decode().split()
    assert log and all("matmul_rows" in k for k in log), log
    assert run(cabi.MM_DETERMINISTIC) in (-1, -4) and not fake.cdll.fake_log()
    if M <= 256:
        assert fake.cdll.ttb_matmul_multi(4096, cabi.BFLOAT16, 1, (ctypes.c_void_p * 1)(1 << 34), cabi.BFLOAT8_B, None, (ctypes.c_void_p * 1)(1 << 35), cabi.BFLOAT16, 1,
                                          M, K, (ctypes.c_int64 * 1)(N), 0, 0, workspace, nbytes, None, None, None) == 0
        assert "matmul_rows" in fake.cdll.fake_log().decode()
