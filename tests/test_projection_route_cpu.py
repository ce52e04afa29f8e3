"""Which kernel a projection goes to, and what that kernel is given: F.linear and F.linear_multi over kernels that run on the CPU and refuse what the real ones
refuse."""
import subprocess
import sys

import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.ops import functional as F
from tensorsharp_b200.ops import kernels
from tensorsharp_b200.quant.qweight import QuantWeight


class OnGpu(QuantWeight):
    device = property(lambda self: torch.device("cuda", 0))


class Kernels:
    def __init__(self):
        self.calls, self.asked = [], 0

    def gemm_blocks_takes(self, w, act=None):
        self.asked += 1
        return kernels.gemm_blocks_takes(w, act)

    @staticmethod
    def quantize_q8(x):
        assert x.is_contiguous()
        return x, x                                        # the recorder multiplies the rows themselves

    def gemv(self, w, *, xq=None, xds=None, xb=None, M, out_dtype, bias=None, residual=None, act=None):
        x = xq if w.uses_q8_activations else xb
        assert x.is_contiguous() and x.shape == (M, w.K)
        return self.product("gemv", w, x, out_dtype)

    def gemv_multi(self, ws, *, xq=None, xds=None, xb=None, M, out_dtype):
        x = xq if ws[0].uses_q8_activations else xb
        self.calls.append("gemv_multi")
        return torch.cat([x.float() @ w.dequantize().float().t() for w in ws], 1).to(out_dtype)

    def gemm_blocks(self, w, x, *, out_dtype, bias=None, residual=None, act=None):
        assert x.shape[0] <= 64 and self.gemm_blocks_takes(w, act)
        return self.product("gemm_blocks", w, self.tma(x), out_dtype)

    def gemm_bf16(self, wb, x, *, out_dtype, bias=None, residual=None):
        self.calls.append("gemm_bf16")
        return (self.tma(x).float() @ wb.float().t()).to(out_dtype)

    @staticmethod
    def gather_rows(w, ids, scale, out):
        return out.copy_(w.dequantize().view(out.shape))

    @staticmethod
    def tma(x):
        assert x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0
        return x

    def product(self, name, w, x, out_dtype):
        self.calls.append(name)
        return (x.float() @ w.dequantize().float().t()).to(out_dtype)


@pytest.fixture
def recorder(monkeypatch):
    k = Kernels()
    monkeypatch.setattr(F, "_kernels", k)
    monkeypatch.setattr(F, "_bf16_budget", lambda dev: 1 << 40)
    real = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **kw: real(*a, **{n: v for n, v in kw.items() if n != "device"}))
    return k


def weight(t, N, K):
    w = QuantWeight.from_float(torch.randn(N, K, generator=torch.Generator().manual_seed(N + K)) * 0.05, t)
    w.__class__ = OnGpu
    return w


def route(k, w, T, act=None):
    k.calls.clear()
    F.linear(F.Act(torch.randn(T, w.K).bfloat16()), w, act=act)
    return k.calls[0]


LARGE = {t: weight(t, 4096, 4096) for t in (GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.BF16)}


@pytest.mark.parametrize("rows", [0, 1, 5, 16])
def test_the_number_of_rows_that_is_given_holds(recorder, monkeypatch, rows):
    """TSB_GEMV_MAX_M: up to so many rows go to the GEMV, of every type; none with 0."""
    monkeypatch.setattr(F, "DENSE_GEMV_MAX_M", rows)
    monkeypatch.setattr(F, "GEMV_ROWS_GIVEN", True, raising=False)
    for t, w in LARGE.items():
        for T in (1, 2, 5, 6, 16, 17):
            assert (route(recorder, w, T) == "gemv") == (T <= rows), (t, T)
            recorder.calls.clear()
            F.linear_multi(F.Act(torch.randn(T, w.K).bfloat16()), [w, w])
            assert (recorder.calls == ["gemv_multi"]) == (T <= rows), (t, T)


def test_the_switch_is_read():
    out = subprocess.run([sys.executable, "-c", "from tensorsharp_b200.ops import functional as F; print(F.DENSE_GEMV_MAX_M, F.GEMV_ROWS_GIVEN)"], capture_output=True,
                         text=True, env={**__import__("os").environ, "TSB_GEMV_MAX_M": "12"})
    assert out.stdout.split() == ["12", "True"]
    assert not F.GEMV_ROWS_GIVEN or "TSB_GEMV_MAX_M" in __import__("os").environ


def test_rows_without_a_bf16_form(recorder):
    """An activation that is there in 8 bits only stays with the GEMV up to sixteen rows, as its caller gives it."""
    x = torch.randn(9, 4096).bfloat16()
    F.linear(F.Act(None, x, x), LARGE[GGMLType.Q4_K])
    assert recorder.calls == ["gemv"]


def forms(T, K):
    """The same rows dense, with a stride that is no multiple of 16 bytes, off 16 bytes, transposed, and behind one another at any distance."""
    x = torch.randn(T, K).bfloat16()
    out = [x]
    for stride, off in ((K + 3, 0), (K + 8, 5), (K + 1, 1)):
        buf = torch.zeros(T * stride + off + 8, dtype=torch.bfloat16)
        y = buf[off:].as_strided((T, K), (stride, 1))
        out.append(y.copy_(x))
    out.append(x.t().contiguous().t())
    flat = torch.zeros(T * K + 1, dtype=torch.bfloat16)
    flat[1:] = x.reshape(-1)
    return out + [flat[1:].view(T, K)]


@pytest.mark.parametrize("t", list(LARGE))
@pytest.mark.parametrize("T", [1, 2, 3, 8])
@pytest.mark.parametrize("act", [None, "relu2"])
def test_few_rows_in_any_form(recorder, monkeypatch, t, T, act):
    """Rows that the GEMV took in any form are made what the tensor cores read where they go there."""
    w = weight(t, 2048, 2048) if t != GGMLType.BF16 else LARGE[t]
    monkeypatch.setattr(Kernels, "glu", lambda self, y, up, act, n, s0, s1, T: (y.float().clamp(min=0).square(), None, None), raising=False)
    monkeypatch.setattr(F, "gemv_rows", lambda *a: 1)
    seen = set()
    for x in forms(T, w.K):
        recorder.calls.clear()
        y = F.linear(F.Act(x), w, act=act)
        seen.add(recorder.calls[-1])
        assert y.shape == (T, w.N)
        if act is None:
            assert torch.allclose(y.float(), x.float() @ w.dequantize().float().t(), atol=1e-4, rtol=1e-5)
    assert seen == {"gemv" if T == 1 else "gemm_bf16" if t == GGMLType.BF16 else "gemm_blocks"}
