"""bfloat16 weights on the tensor cores (csrc/matmul_bf16.cu) at the edges of its tiling, against 64-bit torch.

Tolerance, per element: one rounding of the result (2^-9 of it for bfloat16, 2^-24 for fp32, doubled for the activations), and
2^-18 of sum |x||w|: at most 16 additions of 16 products in a tensor-memory chain and K / 64 chains, each cutting or rounding off
at most 2^-23 of the magnitudes added (K <= 2048: (16 + 32) * 2^-23 < 2^-17.4, of which the sum reaches half at most)."""
import pytest

import cabi

pytestmark = pytest.mark.gpu

# rows, K, N: one tile of each kind (CUDA cores, then many tiles of it); partial row tiles, partial column tiles, a last K stage of 32; K ranges shared by clusters
# of 8, 4 and 2 blocks; more tiles than SMs
SHAPES = [(32, 32, 32), (1024, 32, 1056), (64, 96, 160), (160, 64, 96), (96, 2048, 96), (128, 1056, 1024), (512, 544, 1120), (1312, 160, 2080)]


def expect(x, w, bias, act):
    import torch
    y = x.double() @ w.double()
    mag = x.double().abs() @ w.double().abs()
    if bias is not None:
        y, mag = y + bias.double(), mag + bias.double().abs()
    return {cabi.ACT_NONE: lambda v: v, cabi.ACT_RELU: torch.relu, cabi.ACT_GELU: torch.nn.functional.gelu, cabi.ACT_SILU: torch.nn.functional.silu}[act](y), mag


def check(y, want, mag, fp32):
    bound = 2 * (2.0 ** -24 if fp32 else 2.0 ** -9) * want.abs() + 2.0 ** -18 * mag
    assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())


def operands(batch, M, K, N, batched, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(batch, M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(batch if batched else 1, K, N, generator=g, device="cuda") * 0.02).bfloat16()
    return x, w


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_linear(ttb, M, K, N, fp32):
    import torch
    x, w = operands(1, M, K, N, False, 3)
    bias = torch.randn(1, N, device="cuda").bfloat16()
    wt, bt = ttb.tilize(w, 1, K, N), ttb.tilize(torch.cat([bias, bias.new_zeros(31, N)]), 1, 32, N)
    for act, b in ((cabi.ACT_NONE, None), (cabi.ACT_RELU, bias), (cabi.ACT_GELU, bias), (cabi.ACT_SILU, None)):
        want, mag = expect(x[0], w[0], b, act)
        kw = dict(bias=bt if b is not None else None, act=act, out_fp32=fp32)
        y = ttb.untilize(ttb.matmul(ttb.tilize(x, 1, M, K), wt, cabi.BFLOAT16, 1, M, K, N, **kw), 1, M, N).reshape(M, N)
        check(y, want, mag, fp32)
        y = ttb.matmul(x.contiguous(), wt, cabi.BFLOAT16, 1, M, K, N, flags=cabi.MM_A_ROW_MAJOR | cabi.MM_OUT_ROW_MAJOR, **kw).reshape(M, N)
        check(y, want, mag, fp32)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("batch,M,K,N", [(3, 160, 96, 224), (2, 32, 2048, 64), (200, 32, 64, 32), (8, 256, 128, 512)])
def test_batched(ttb, batch, M, K, N, fp32):
    import torch
    x, w = operands(batch, M, K, N, True, 5)
    a, wt = ttb.tilize(x, batch, M, K), ttb.tilize(w, batch, K, N)
    # a guard on both sides, and an output that starts 16 but not 32 bytes into a line
    skip = 4 if fp32 else 8
    buf = torch.full((batch * M * N + skip + 64,), 7.0, dtype=torch.float32 if fp32 else torch.bfloat16, device="cuda")
    out = buf[skip:skip + batch * M * N]
    ttb.check(ttb.cdll.ttb_bmm(a.data_ptr(), cabi.BFLOAT16, wt.data_ptr(), cabi.BFLOAT16, out.data_ptr(), cabi.FLOAT32 if fp32 else cabi.BFLOAT16, batch, M, K, N,
                               None))
    ttb.check(ttb.check_status(None))
    assert bool((buf[:skip] == 7.0).all()) and bool((buf[skip + batch * M * N:] == 7.0).all())
    want, mag = expect(x, w, None, cabi.ACT_NONE)
    check(ttb.untilize(out.clone(), batch, M, N).reshape(batch, M, N), want, mag, fp32)


def test_infinities_and_nan_stay_in_their_rows_and_columns(ttb):
    """Rows and columns beyond the matrix share tiles with garbage, and a non-finite input reaches its own row and column only."""
    import torch
    M, K, N = 96, 160, 96
    x, w = operands(1, M, K, N, False, 7)
    x[0, 5, 33], w[0, 40, 70] = float("inf"), float("nan")
    y = ttb.untilize(ttb.matmul(ttb.tilize(x, 1, M, K), ttb.tilize(w, 1, K, N), cabi.BFLOAT16, 1, M, K, N), 1, M, N).reshape(M, N)
    want = x[0].double() @ w[0].double()
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
