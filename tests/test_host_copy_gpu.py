"""Copies of pageable host memory through the pinned staging buffers (csrc/host_copy.cu): sizes around the chunk and the threshold,
unaligned host addresses, several threads at once, pinned memory - the same bytes."""
import threading

import pytest

import cabi

pytestmark = pytest.mark.gpu
MB = 1 << 20


def round_trip(ttb, bytes_, skip, pinned=False):
    import torch
    src = torch.randint(0, 256, (bytes_ + skip,), dtype=torch.uint8)
    dst = torch.zeros(bytes_ + skip + 64, dtype=torch.uint8)
    if pinned:
        src, dst = src.pin_memory(), dst.pin_memory()
    dev = torch.empty(bytes_, dtype=torch.uint8, device="cuda")
    ttb.check(ttb.cdll.ttb_memcpy_h2d(dev.data_ptr(), src.data_ptr() + skip, bytes_, None))
    ttb.check(ttb.cdll.ttb_memcpy_d2h(dst.data_ptr() + skip, dev.data_ptr(), bytes_, None))
    ttb.check(ttb.cdll.ttb_stream_synchronize(None))
    assert torch.equal(dst[skip:skip + bytes_], src[skip:]) and not dst[:skip].any() and not dst[skip + bytes_:].any()


@pytest.mark.parametrize("bytes_,skip", [(4 * MB - 1, 0), (4 * MB, 0), (4 * MB + 1, 3), (5 * MB, 1), (16 * MB, 0), (16 * MB + 12345, 7), (40 * MB - 5, 0)])
def test_round_trip(ttb, bytes_, skip):
    round_trip(ttb, bytes_, skip)
    round_trip(ttb, bytes_, skip, pinned=True)


@pytest.mark.parametrize("stream", [None, 2, "own"])
def test_copies_are_ordered_after_the_streams_work(ttb, stream):
    """A kernel's worth of copies writes what is read back, and reads what is overwritten, on the default stream, the per-thread
    default stream (handle 2) and one of the caller's."""
    import torch
    n, own = 24 * MB, torch.cuda.Stream()
    s = own.cuda_stream if stream == "own" else stream
    big = torch.zeros(2, 512 * MB, dtype=torch.uint8, device="cuda")
    dev, old = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")
    src, dst = torch.full((n,), 3, dtype=torch.uint8), torch.zeros(n, dtype=torch.uint8)
    torch.cuda.synchronize()
    for _ in range(20):                                        # about 4 ms ahead of what the copy has to wait for
        ttb.check(ttb.cdll.ttb_memcpy_d2d(big[0].data_ptr(), big[1].data_ptr(), 512 * MB, s))
    ttb.check(ttb.cdll.ttb_memset(dev.data_ptr(), 7, n, s))
    ttb.check(ttb.cdll.ttb_memcpy_d2h(dst.data_ptr(), dev.data_ptr(), n, s))
    ttb.check(ttb.cdll.ttb_stream_synchronize(s))
    assert bool((dst == 7).all())
    for _ in range(20):
        ttb.check(ttb.cdll.ttb_memcpy_d2d(big[0].data_ptr(), big[1].data_ptr(), 512 * MB, s))
    ttb.check(ttb.cdll.ttb_memcpy_d2d(old.data_ptr(), dev.data_ptr(), n, s))
    ttb.check(ttb.cdll.ttb_memcpy_h2d(dev.data_ptr(), src.data_ptr(), n, s))
    ttb.check(ttb.cdll.ttb_stream_synchronize(s))
    assert bool((old == 7).all()) and bool((dev == 3).all())


def test_several_threads(ttb):
    failures = []

    def work(n):
        try:
            import torch
            torch.cuda.set_device(0)
            for _ in range(3):
                round_trip(ttb, 9 * MB + n, n)
        except BaseException as e:   # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_copies_beside_another_threads_capture():
    """The first large copies of a process, on a stream of their own, while another thread captures in global mode: both succeed, and the
    graph replays. (A process of its own, so that the pinned buffers are not there yet.)"""
    import os
    import subprocess
    import sys
    code = """if True:
        import sys, threading
        sys.path.insert(0, %r)
        import torch, cabi
        lib, n = cabi.load(), 24 << 20
        src, dst, dev = torch.randint(0, 256, (n,), dtype=torch.uint8), torch.zeros(n, dtype=torch.uint8), torch.empty(n, dtype=torch.uint8, device="cuda")
        x, own, side = torch.zeros(1024, device="cuda"), torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        codes, graph = [], torch.cuda.CUDAGraph()

        def work():
            codes.append(lib.cdll.ttb_memcpy_h2d(dev.data_ptr(), src.data_ptr(), n, own.cuda_stream))
            codes.append(lib.cdll.ttb_memcpy_d2h(dst.data_ptr(), dev.data_ptr(), n, own.cuda_stream))

        with torch.cuda.graph(graph, stream=side, capture_error_mode="global"):
            x.add_(1)
            t = threading.Thread(target=work)
            t.start()
            t.join()
            x.add_(1)
        graph.replay()
        torch.cuda.synchronize()
        assert codes == [0, 0], (codes, lib.cdll.ttb_last_error())
        assert torch.equal(src, dst) and bool((x == 2).all())
    """ % os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
