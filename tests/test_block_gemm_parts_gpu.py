"""Tensor-core products of GGUF blocks where tiles and slabs are not whole, and what F.linear gives for two to eight rows."""
import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.ops import functional as F
from tensorsharp_b200.ops import reference as ref
from tensorsharp_b200.quant.qweight import QuantWeight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from tensorsharp_b200.ops import kernels
    return kernels


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def tiles_of(counts, rows):
    out, at = [], 0
    for e, n in enumerate(counts):
        out += [(e, at + i, min(rows, n - i), 0) for i in range(0, n, rows)]
        at += n
    return torch.tensor(out + [(0, 0, 0, 0)], dtype=torch.int32, device=DEV), torch.tensor([len(out), at], dtype=torch.int32, device=DEV)


# f32 sums of exact bf16 products in another order: far below 1e-5; a bf16 result is rounded once, 2^-9 at most: 3e-3
@pytest.mark.parametrize("rows", [16, 32, 64])
@pytest.mark.parametrize("E,F_,Kd,counts", [(2, 112, 480, [1, 33]), (3, 80, 224 * 2, [64, 0, 65]), (2, 48, 96, [7, 2])])
def test_gated_experts_of_partial_tiles(rows, E, F_, Kd, counts):
    """Halves that are no whole tiles of 64 rows, rows that are no whole slabs of 64 values."""
    torch.manual_seed(1)
    w = QuantWeight.from_float(torch.randn(E, 2 * F_, Kd, device=DEV) * 0.2, GGMLType.MXFP4)
    assert K().gemm_experts_takes(w, "swiglu") >= rows
    P = sum(counts)
    x, b = torch.randn(P, Kd, device=DEV).bfloat16(), torch.randn(E, 2 * F_, device=DEV)
    tiles, meta = tiles_of(counts, rows)
    of = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    y = torch.einsum("pk,pnk->pn", x.double(), w.dequantize().view(E, 2 * F_, Kd).double()[of]) + b[of]
    for act in ("swiglu_oai", "swiglu"):
        got = K().gemm_experts(w, x, tiles, meta, rows, out_dtype=torch.bfloat16, bias=b, act=act)
        assert rel(got, ref.glu(act, y[:, :F_], y[:, F_:])) < 3e-3
    assert int(K().gemm_status(DEV).item()) == 0


@pytest.mark.parametrize("rows", [16, 32, 64])
@pytest.mark.parametrize("E,N,Kd,counts", [(2, 208, 480, [1, 33]), (2, 16, 32, [3, 70])])
def test_experts_of_partial_tiles(rows, E, N, Kd, counts):
    torch.manual_seed(2)
    w = QuantWeight.from_float(torch.randn(E, N, Kd, device=DEV) * 0.05, GGMLType.MXFP4)
    assert K().gemm_experts_takes(w) >= rows
    P = sum(counts)
    x, s = torch.randn(P, Kd, device=DEV).bfloat16(), torch.rand(P, device=DEV)
    tiles, meta = tiles_of(counts, rows)
    of = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    want = torch.einsum("pk,pnk->pn", x.double(), w.dequantize().view(E, N, Kd).double()[of]) * s[:, None]
    assert rel(K().gemm_experts(w, x, tiles, meta, rows, out_dtype=torch.float32, row_scale=s), want) < 1e-5
    assert int(K().gemm_status(DEV).item()) == 0


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0])
@pytest.mark.parametrize("T", [3, 5, 8])
@pytest.mark.parametrize("N,Kd", [(4096, 4096), (6144, 2560)])
@pytest.mark.parametrize("wild", [False, True])
def test_few_rows_are_no_further_from_64_bits_than_the_gemv(t, T, N, Kd, wild):
    """Weights rounded to bf16 by rows as they are, where the GEMV has weights as they are by rows rounded to eight bits."""
    torch.manual_seed(3)
    w = QuantWeight.from_float(torch.randn(N, Kd, device=DEV) * 0.05 * torch.rand(N, 1, device=DEV), t)
    x = torch.randn(T, Kd, device=DEV)
    if wild:
        x[:, torch.randint(0, Kd, (40,), device=DEV)] *= 30
    x = x.bfloat16()
    assert T > F.gemv_rows(w)
    want = x.double() @ w.dequantize().double().t()
    xq, xds = K().quantize_q8(x)
    assert rel(F.linear(F.Act(x), w), want) <= rel(K().gemv(w, xq=xq, xds=xds, M=T), want)
