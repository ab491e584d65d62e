"""Middling row counts of block-float weights (csrc/matmul_rows.cu) at the edges of its tiling, against 64-bit torch.

Tolerance, per element: one rounding to bfloat16 (2^-9 of the result, doubled for the activations) and 2^-15 of sum |x||w|: at most
K / 16 = 256 additions of 16 products in a row, each cutting off at most 2^-23 of the magnitudes added."""
import pytest

import cabi

pytestmark = pytest.mark.gpu

# rows, K, N: one tile row more than the decode kernels' blocks; a K range of fewer than four blocks and of one more than a group;
# unequal row chunks; a partial column tile; clusters of 8, 3 and 2 blocks; whole rounds of tiles with a remainder launch, and more
# tiles than SMs without one; chunks of 256 rows
SHAPES = [(96, 32, 32), (96, 160, 96), (64, 4096, 128), (352, 992, 672), (544, 1056, 608), (224, 288, 4672), (1056, 512, 4672), (416, 96, 7168),
          (512, 4096, 4096)]


def reference(x, w, bias, act):
    import torch
    y, mag = x.double() @ w.double(), x.double().abs() @ w.double().abs()
    if bias is not None:
        y, mag = y + bias.double(), mag + bias.double().abs()
    return {cabi.ACT_NONE: lambda v: v, cabi.ACT_RELU: torch.relu, cabi.ACT_GELU: torch.nn.functional.gelu, cabi.ACT_SILU: torch.nn.functional.silu}[act](y), mag


def close(y, want, mag, K=4096):
    bound = 2.0 ** -8 * want.abs() + K / 16 * 2.0 ** -23 * mag
    assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())


def weight(ttb, fmt, K, N, scale, seed):
    """Packed by the (bit-exact, separately tested) device packer, and the values it stands for."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    packed = ttb.pack(torch.randn(K, N, generator=g, device="cuda") * scale, fmt, 1, K, N)
    return packed, ttb.unpack(packed, fmt, 1, K, N).reshape(K, N)


@pytest.mark.parametrize("fmt", [cabi.BFLOAT8_B, cabi.BFLOAT4_B])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_against_64_bits(ttb, fmt, M, K, N):
    import torch
    for scale, act, with_bias, flags in ((0.02, cabi.ACT_NONE, False, 0), (3.0, cabi.ACT_GELU, True, 0), (0.02, cabi.ACT_SILU, True, cabi.MM_A_ROW_MAJOR | cabi.MM_OUT_ROW_MAJOR),
                                         (0.02, cabi.ACT_RELU, False, cabi.MM_WEIGHTS_RESIDENT)):
        packed, values = weight(ttb, fmt, K, N, scale, 3)   # (3.0: exponents above 127)
        x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").bfloat16()
        bias = torch.randn(1, N, device="cuda").bfloat16() if with_bias else None
        bt = ttb.tilize(torch.cat([bias, bias.new_zeros(31, N)]), 1, 32, N) if with_bias else None
        a = x.reshape(-1).contiguous() if flags & cabi.MM_A_ROW_MAJOR else ttb.tilize(x, 1, M, K)
        buf = torch.full((8 + M * N + 512,), 7.0, dtype=torch.bfloat16, device="cuda")   # 16-byte aligned, a guard on both sides
        out = buf[8:8 + M * N]
        nbytes = ttb.matmul_workspace_bytes(fmt, 1, M, K, N, flags)
        ws = torch.zeros(max(nbytes, 16), dtype=torch.uint8, device="cuda")
        ttb.check(ttb.cdll.ttb_matmul(a.data_ptr(), cabi.BFLOAT16, packed.data_ptr(), fmt, bt.data_ptr() if with_bias else None, out.data_ptr(), cabi.BFLOAT16,
                                      1, M, K, N, act, flags | cabi.MM_WORKSPACE_ZEROED, ws.data_ptr(), nbytes, None))
        ttb.check(ttb.check_status(None))
        assert bool((buf[:8] == 7.0).all()) and bool((buf[8 + M * N:] == 7.0).all()) and int(ws.count_nonzero()) == 0
        y = out.reshape(M, N) if flags & cabi.MM_OUT_ROW_MAJOR else ttb.untilize(out.clone(), 1, M, N).reshape(M, N)
        close(y, *reference(x, values, bias, act))


# long K ranges with and without a cluster, row counts far above one chunk (whole rounds with and without a remainder launch)
@pytest.mark.parametrize("fmt", [cabi.BFLOAT8_B, cabi.BFLOAT4_B])
@pytest.mark.parametrize("M,K,N", [(96, 28672, 1152), (320, 12288, 160), (352, 8192, 18976), (1888, 512, 4544), (2048, 2048, 2048), (4096, 288, 1184)])
def test_long_k_ranges_and_many_rows(ttb, fmt, M, K, N):
    import torch
    assert ttb.cdll.ttb_matmul_kernel(fmt, cabi.BFLOAT16, 1, M, K, N, 0) == cabi.KERNEL_ROWS
    packed, values = weight(ttb, fmt, K, N, 0.02, 5)
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda").bfloat16()
    y = ttb.untilize(ttb.matmul(ttb.tilize(x, 1, M, K), packed, fmt, 1, M, K, N), 1, M, N).reshape(M, N)
    close(y, *reference(x, values, None, cabi.ACT_NONE), K=K)


@pytest.mark.parametrize("fmt", [cabi.BFLOAT8_B, cabi.BFLOAT4_B])
@pytest.mark.parametrize("M,K,N", [(96, 160, 96), (320, 4096, 160)])
def test_infinities_and_nan_stay_in_their_rows(ttb, fmt, M, K, N):
    """Rows share tiles and, with a K range in pieces, partial sums; a non-finite activation reaches its own row only."""
    import torch
    packed, values = weight(ttb, fmt, K, N, 0.02, 7)
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(8), device="cuda").bfloat16()
    x[5, 33], x[40, 100], x[M - 1, K - 1] = float("inf"), float("nan"), float("-inf")
    y = ttb.untilize(ttb.matmul(ttb.tilize(x, 1, M, K), packed, fmt, 1, M, K, N), 1, M, N).reshape(M, N)
    want = x.double() @ values.double()
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isposinf(y), torch.isposinf(want)) and torch.equal(torch.isneginf(y), torch.isneginf(want))


@pytest.mark.parametrize("fmt", [cabi.BFLOAT8_B, cabi.BFLOAT4_B])
@pytest.mark.parametrize("M,K,Ns", [(96, 512, (512, 96, 160)), (96, 768, (512, 96, 160)), (128, 1024, (1024, 128)), (256, 288, (96, 4672, 32, 4096))])
def test_several_weights_in_one_launch(ttb, fmt, M, K, Ns):
    import ctypes
    import torch
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").bfloat16()
    a, n = ttb.tilize(x, 1, M, K), len(Ns)
    ws = [weight(ttb, fmt, K, N, 0.02, 20 + j) for j, N in enumerate(Ns)]
    biases = [torch.randn(1, N, device="cuda").bfloat16() if j != 1 else None for j, N in enumerate(Ns)]
    tiled = [ttb.tilize(torch.cat([b, b.new_zeros(31, N)]), 1, 32, N) if b is not None else None for b, N in zip(biases, Ns)]
    outs = [torch.full((M * N + 64,), 7.0, dtype=torch.bfloat16, device="cuda") for N in Ns]
    ptrs = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() if t is not None else None for t in ts])   # noqa: E731
    arr_n = (ctypes.c_int64 * n)(*Ns)
    nbytes = ttb.matmul_multi_workspace_bytes(fmt, 1, M, K, n, arr_n)
    wsp = torch.zeros(max(nbytes, 16), dtype=torch.uint8, device="cuda")
    ttb.check(ttb.cdll.ttb_matmul_multi(a.data_ptr(), cabi.BFLOAT16, n, ptrs([p for p, _ in ws]), fmt, ptrs(tiled), ptrs(outs), cabi.BFLOAT16, 1, M, K, arr_n,
                                        cabi.ACT_SILU, cabi.MM_WORKSPACE_ZEROED | cabi.MM_WEIGHTS_RESIDENT, wsp.data_ptr(), nbytes, None, None, None))
    ttb.check(ttb.check_status(None))
    for (_, values), b, o, N in zip(ws, biases, outs, Ns):
        assert bool((o[M * N:] == 7.0).all())
        close(ttb.untilize(o[:M * N].clone(), 1, M, N).reshape(M, N), *reference(x, values, b, cabi.ACT_SILU))


def test_launches_that_follow_each_other_give_the_same_bytes(ttb):
    """Overlapped launches (resident weights), each reading what the one before wrote; twice."""
    import torch
    M, K, fmt = 352, 1024, cabi.BFLOAT8_B
    packed, _ = weight(ttb, fmt, K, K, 0.03, 9)
    x = ttb.tilize(torch.randn(M, K, device="cuda").bfloat16(), 1, M, K)
    results = []
    for _ in range(2):
        cur, outs = x, [torch.empty(M * K, dtype=torch.bfloat16, device="cuda") for _ in range(20)]
        for o in outs:
            ttb.check(ttb.cdll.ttb_matmul(cur.data_ptr(), cabi.BFLOAT16, packed.data_ptr(), fmt, None, o.data_ptr(), cabi.BFLOAT16, 1, M, K, K, 0,
                                          cabi.MM_WEIGHTS_RESIDENT, None, 0, None))
            cur = o
        ttb.check(ttb.check_status(None))
        results.append(outs)
    assert all(torch.equal(a, b) for a, b in zip(*results)) and bool(torch.isfinite(results[0][-1].float()).all())
