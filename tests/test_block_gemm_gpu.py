"""Products of few rows with weights in GGUF blocks on the tensor cores (csrc/gemm_blocks.cu), against the same products of the decoded weights."""
import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.ops import reference as ref
from tensorsharp_b200.quant.qweight import QuantWeight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = [GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0]


def K():
    from tensorsharp_b200.ops import kernels
    return kernels


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def status():
    return int(K().gemm_status(DEV).item())


def weight(t, *shape, scale=0.05):
    return QuantWeight.from_float(torch.randn(*shape, device=DEV) * scale * torch.rand(*shape[:-1], 1, device=DEV), t)


# one product per output value: the decoded weight itself, which is the value that the bf16 copy holds (Q4_K: where the offset of a
# sub-block is as large as its scale, as in these, it is exact too)
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("N,Kd", [(3, 256), (300, 512), (2000, 768)])
def test_decoded_values_are_those_of_the_copy(t, N, Kd):
    torch.manual_seed(1)
    w = weight(t, N, Kd)
    copy = K().gather_rows(w, None, 1.0)
    eye = torch.eye(Kd, device=DEV, dtype=torch.bfloat16)
    for k in range(0, Kd, 64):
        assert torch.equal(K().gemm_blocks(w, eye[k:k + 64]), copy[:, k:k + 64].t().float())
    assert status() == 0


# f32 sums of exact bf16 products in another order: far below 1e-5; a bf16 result is rounded once, 2^-9 at most: 2e-3
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("T", [1, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,Kd", [(1, 256), (129, 1024), (1000, 4864), (19000, 512)])
def test_dense(t, T, N, Kd):
    torch.manual_seed(2)
    w, x = weight(t, N, Kd), torch.randn(T, Kd, device=DEV).bfloat16()
    want = x.double() @ K().gather_rows(w, None, 1.0).double().t()
    assert rel(K().gemm_blocks(w, x), want) < 1e-5
    bias, res = torch.randn(N, device=DEV), torch.randn(T, N, device=DEV)
    assert rel(K().gemm_blocks(w, x, bias=bias, residual=res), want + bias + res) < 1e-5
    assert rel(K().gemm_blocks(w, x, out_dtype=torch.bfloat16, bias=bias, residual=res.bfloat16()), want + bias + res.bfloat16()) < 3e-3
    assert status() == 0


# the result is rounded to bf16 once: 2^-9 at most
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("act", ["swiglu", "geglu", "swiglu_oai", "silu", "relu2"])
@pytest.mark.parametrize("T,F,Kd", [(9, 40, 256), (64, 320, 1280), (30, 9728, 512)])
def test_activations(t, act, T, F, Kd):
    torch.manual_seed(3)
    gated = act not in ("silu", "relu2")
    w, x = weight(t, 2 * F if gated else F, Kd, scale=0.2), torch.randn(T, Kd, device=DEV).bfloat16()
    y = x.double() @ K().gather_rows(w, None, 1.0).double().t()
    want = ref.glu(act, y[:, :F], y[:, F:]) if gated else ref.glu(act, y, None)
    assert rel(K().gemm_blocks(w, x, act=act), want) < 1e-5
    assert rel(K().gemm_blocks(w, x, act=act, out_dtype=torch.bfloat16), want) < 3e-3
    assert status() == 0


def test_launched_back_to_back():
    """Hundreds of launches with nothing between them: tensor memory and clusters of one while the next ones start."""
    torch.manual_seed(4)
    a, b, x = weight(GGMLType.Q4_K, 2560, 4096), weight(GGMLType.Q6_K, 1300, 4096), torch.randn(40, 4096, device=DEV).bfloat16()
    want = K().gemm_blocks(a, x), K().gemm_blocks(b, x[:12])
    outs = [(K().gemm_blocks(a, x), K().gemm_blocks(b, x[:12])) for _ in range(150)]
    assert all(torch.equal(o[0], want[0]) and torch.equal(o[1], want[1]) for o in outs) and status() == 0


def tiles_of(counts, rows):
    out, at = [], 0
    for e, n in enumerate(counts):
        for i in range(0, n, rows):
            out.append((e, at + i, min(rows, n - i), 0))
        at += n
    return torch.tensor(out + [(0, 0, 0, 0)] * 3, dtype=torch.int32, device=DEV), torch.tensor([len(out), at], dtype=torch.int32, device=DEV)


# every code under the scales whose values are normal in bf16: exact there, and in the product with one
def test_mxfp4_values():
    e = (4 + torch.arange(256) % 249).to(torch.uint8)[:, None]
    blocks = torch.cat([e, ((torch.arange(16) * 17 + 16 * e.long()) % 256).to(torch.uint8)], 1)
    blocks = torch.cat([blocks, blocks.flip(0)], 1)                              # two blocks of a row
    w = QuantWeight.from_raw(blocks.contiguous().view(-1), GGMLType.MXFP4, (1, 256, 64), device=DEV)
    tiles, meta = tiles_of([64], 64)
    got = K().gemm_experts(w, torch.eye(64, device=DEV, dtype=torch.bfloat16), tiles, meta, 64, out_dtype=torch.float32)
    assert torch.equal(got, w.dequantize().view(256, 64).t().float()) and status() == 0


@pytest.mark.parametrize("rows", [16, 32, 64])
@pytest.mark.parametrize("E,N,Kd,counts", [(3, 128, 64, [5, 0, 70]), (2, 200, 480, [1, 33]), (8, 2880, 2880, [0, 16, 17, 1, 64, 65, 9, 0]),
                                           (40, 640, 1056, [3] * 40)])
def test_experts(rows, E, N, Kd, counts):
    torch.manual_seed(5)
    P = sum(counts)
    w, x = weight(GGMLType.MXFP4, E, N, Kd), torch.randn(P, Kd, device=DEV).bfloat16()
    if K().gemm_experts_takes(w) < rows:
        pytest.skip("scales of a tile that are no whole pieces of 16 bytes")
    b, s = torch.randn(E, N, device=DEV), torch.rand(P, device=DEV)
    tiles, meta = tiles_of(counts, rows)
    of = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    full = w.dequantize().view(E, N, Kd).double()
    want = torch.stack([x[p].double() @ full[of[p]].t() for p in range(P)])
    assert rel(K().gemm_experts(w, x, tiles, meta, rows, out_dtype=torch.float32), want) < 1e-5
    got = K().gemm_experts(w, x, tiles, meta, rows, out_dtype=torch.float32, bias=b, row_scale=s)
    assert rel(got, (want + b[of]) * s[:, None]) < 1e-5
    assert status() == 0


@pytest.mark.parametrize("rows", [16, 32, 64])
@pytest.mark.parametrize("E,F,Kd,counts", [(3, 64, 64, [5, 0, 70]), (2, 104, 480, [1, 33]), (8, 2880, 2880, [0, 16, 17, 1, 64, 65, 9, 0])])
def test_gated_experts(rows, E, F, Kd, counts):
    torch.manual_seed(6)
    P = sum(counts)
    w, x = weight(GGMLType.MXFP4, E, 2 * F, Kd, scale=0.2), torch.randn(P, Kd, device=DEV).bfloat16()
    if K().gemm_experts_takes(w, "swiglu_oai") < rows:
        pytest.skip("scales of a tile that are no whole pieces of 16 bytes")
    b = torch.randn(E, 2 * F, device=DEV)
    tiles, meta = tiles_of(counts, rows)
    of = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    full = w.dequantize().view(E, 2 * F, Kd).double()
    y = torch.stack([x[p].double() @ full[of[p]].t() + b[of[p]] for p in range(P)])
    for act in ("swiglu_oai", "swiglu"):
        got = K().gemm_experts(w, x, tiles, meta, rows, out_dtype=torch.bfloat16, bias=b, act=act)
        assert rel(got, ref.glu(act, y[:, :F], y[:, F:])) < 3e-3
    assert status() == 0
