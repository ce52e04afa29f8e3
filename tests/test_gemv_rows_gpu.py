"""Single-token products of Q4_K, Q6_K and Q8_0 rows in groups (csrc/gemv_stream.cu), against the decoded weights in double precision."""
import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.quant.qweight import QuantWeight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# The activations are whole numbers up to 127 with a 127 in every group of 32 (times a power of two), which int8 groups hold exactly: what
# is left is the rounding of float sums, at most some 300 additions of terms as large as the result's parts (1e-5 with room).
@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0])
@pytest.mark.parametrize("blocks", [1, 2, 3, 6, 10, 11, 12, 13, 16, 18, 24, 25, 26, 30, 38, 46, 50, 56, 64, 84, 93, 96])
@pytest.mark.parametrize("N,kind", [(64, "plain"), (67, "joined"), (2370, "joined"), (2372, "gated"), (130, "gated")])
def test_rows_of_every_length(t, blocks, N, kind):
    if t == GGMLType.Q6_K and (blocks % 2 or kind == "gated") or t != GGMLType.Q8_0 and blocks > 64:
        pytest.skip("the general kernels' form")
    from tensorsharp_b200.ops import kernels as k
    torch.manual_seed(blocks * 7 + N)
    Kd = blocks * 256
    w = QuantWeight.from_float(torch.randn(N, Kd, device=DEV) * 0.05 * torch.rand(N, 1, device=DEV), t)
    x = torch.randint(-127, 128, (1, Kd // 32, 32), device=DEV)
    x[..., 5] = torch.where(x[..., 5] < 0, -127, 127)
    x = (x.reshape(1, Kd).float() / 64).bfloat16()
    xq, xds = k.quantize_q8(x)
    assert torch.equal(xq.reshape(-1).float() * xds.reshape(-1, 2)[:, 0].repeat_interleave(32), x.float().reshape(-1))
    n_out = N // 2 if kind == "gated" else N
    bias = torch.randn(N, device=DEV) if kind != "plain" else None
    res = torch.randn(1, n_out, device=DEV) if kind == "joined" else None
    scale = torch.tensor([0.75], device=DEV) if kind == "joined" else None
    got = k.gemv(w, xq=xq, xds=xds, xb=x, M=1, bias=bias, residual=res, row_scale=scale, act="swiglu" if kind == "gated" else None)
    y = x.double() @ w.dequantize().double().t()
    parts = x.double().abs() @ w.dequantize().double().abs().t()
    if kind == "gated":
        # the derivative of silu(g) * u by either is below 1.1 times the other, or itself
        tol = 1e-5 * (parts[:, :n_out] * (y[:, n_out:] + bias[n_out:]).abs() * 1.1 + parts[:, n_out:] * (y[:, :n_out] + bias[:n_out]).abs()) + 1e-5
        y = y + bias
        want = torch.nn.functional.silu(y[:, :n_out]) * y[:, n_out:]
        tol = tol + 1e-5 * want.abs()                                  # the gate's exponential
    else:
        want = y if bias is None else (y + bias) * 0.75 + res
        tol = 1e-5 * parts + 1e-6
    assert ((got.double() - want).abs() <= tol).all(), ((got.double() - want).abs() / tol).max().item()
    half = k.gemv(w, xq=xq, xds=xds, xb=x, M=1, bias=bias, residual=res.bfloat16() if res is not None else None, row_scale=scale,
                  act="swiglu" if kind == "gated" else None, out_dtype=torch.bfloat16)
    assert torch.allclose(half.float(), got, rtol=2 ** -7, atol=0.02)


@pytest.mark.parametrize("blocks", [2, 8, 10, 12, 14, 18, 24])
@pytest.mark.parametrize("rows", [(61, 3), (512, 130, 131), (4096, 1024, 1024)])
@pytest.mark.parametrize("last", [GGMLType.Q4_K, GGMLType.Q6_K])
def test_matrices_side_by_side(blocks, rows, last):
    from tensorsharp_b200.ops import kernels as k
    torch.manual_seed(blocks)
    Kd = blocks * 256
    ws = [QuantWeight.from_float(torch.randn(n, Kd, device=DEV) * 0.05, last if i == len(rows) - 1 else GGMLType.Q4_K) for i, n in enumerate(rows)]
    x = torch.randn(1, Kd, device=DEV).bfloat16()
    xq, xds = k.quantize_q8(x)
    want = torch.cat([k.gemv(w, xq=xq, xds=xds, M=1) for w in ws], 1)
    parts = torch.cat([x.float().abs() @ w.dequantize().abs().t() for w in ws], 1)
    got = k.gemv_multi(ws, xq=xq, xds=xds, M=1)
    assert ((got - want).abs() <= 1e-5 * parts).all()                  # the same whole-number sums, joined in another order
    half = k.gemv_multi(ws, xq=xq, xds=xds, M=1, out_dtype=torch.bfloat16)
    assert torch.equal(half, got.bfloat16())
