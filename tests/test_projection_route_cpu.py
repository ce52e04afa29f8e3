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


# (type, N, K, activation) -> us with 2, 3, 4, 8, 16 and 64 rows: the GEMV (more than eight: the bf16 copy), and the tensor cores on the weight as it is
ROWS = (2, 3, 4, 8, 16, 64)
MEASURED = {
    ("Q4_K", 256, 256, None): [(1.5, 2.7), (2.3, 2.8), (2.6, 2.9), (1.7, 3.2), (3.5, 3.9), (4.7, 8.2)],
    ("Q4_K", 512, 512, None): [(1.7, 3.4), (2.4, 3.6), (2.6, 3.6), (2.2, 4.0), (5.4, 4.4), (6.7, 8.3)],
    ("Q4_K", 512, 1024, None): [(1.7, 3.6), (2.5, 3.6), (2.7, 3.6), (3.1, 3.7), (5.4, 4.3), (6.8, 6.5)],
    ("Q4_K", 1024, 1024, None): [(1.7, 3.7), (2.6, 3.6), (2.8, 3.7), (4.5, 3.8), (5.5, 4.4), (7.0, 6.5)],
    ("Q4_K", 2048, 2048, None): [(2.7, 5.0), (4.6, 5.1), (4.9, 5.1), (7.2, 5.2), (7.5, 5.3), (9.3, 6.6)],
    ("Q4_K", 1024, 2560, None): [(2.8, 4.9), (5.0, 4.8), (5.8, 4.9), (9.5, 4.9), (6.4, 5.7), (8.2, 8.0)],
    ("Q4_K", 6144, 2560, None): [(8.6, 7.7), (13.9, 7.7), (15.6, 7.7), (10.2, 7.9), (10.7, 8.5), (13.3, 11.0)],
    ("Q4_K", 2560, 9728, None): [(8.7, 10.9), (16.1, 11.0), (17.6, 11.0), (31.2, 11.1), (13.5, 11.3), (15.6, 13.7)],
    ("Q4_K", 1536, 512, "swiglu"): [(2.3, 3.8), (2.8, 3.8), (3.1, 3.8), (3.9, 3.8), (7.2, 4.3), (8.7, 7.0)],
    ("Q6_K", 1024, 1024, None): [(1.9, 3.5), (3.1, 3.5), (3.3, 3.5), (5.2, 3.6), (5.5, 4.2), (7.0, 6.4)],
    ("Q6_K", 2560, 1024, None): [(2.5, 4.2), (3.8, 4.5), (4.0, 4.5), (10.7, 4.5), (6.0, 5.2), (8.0, 7.3)],
    ("Q6_K", 2560, 9728, None): [(12.5, 11.9), (20.6, 12.1), (20.9, 12.1), (59.8, 12.2), (13.7, 12.4), (15.7, 14.8)],
    ("Q8_0", 1024, 1024, None): [(1.7, 3.5), (1.9, 3.6), (1.9, 3.6), (2.8, 3.7), (5.5, 4.2), (7.0, 6.5)],
    ("Q8_0", 1024, 2560, None): [(2.8, 4.9), (3.1, 4.9), (3.2, 4.9), (4.7, 4.9), (6.4, 5.7), (8.2, 8.0)],
    ("Q8_0", 2560, 4096, None): [(4.2, 6.6), (5.8, 6.7), (5.8, 6.7), (13.6, 6.9), (9.5, 7.0), (11.5, 8.9)],
    ("Q8_0", 4096, 4096, None): [(7.4, 8.4), (10.0, 8.5), (10.2, 8.5), (15.5, 8.6), (11.2, 8.8), (13.1, 10.7)],
    ("Q8_0", 4096, 2048, "swiglu"): [(4.7, 6.7), (6.9, 6.9), (7.4, 7.0), (10.0, 7.1), (10.0, 7.3), (12.2, 9.1)],
    ("BF16", 2048, 2048, None): [(4.1, 6.4), (5.1, 6.5), (6.3, 6.5), (11.2, 7.1), (7.6, 7.6), (9.3, 9.3)],
    ("BF16", 4096, 4096, None): [(9.6, 10.7), (13.0, 10.8), (13.5, 10.9), (23.1, 11.2), (11.4, 11.4), (13.3, 13.3)],
    ("BF16", 19456, 2560, "swiglu"): [(21.6, 32.0), (29.2, 31.9), (30.3, 32.2), (57.3, 32.3), (32.7, 32.7), (36.3, 36.3)],
}


@pytest.mark.parametrize("name,N,K,act", list(MEASURED))
def test_no_slower_than_the_general_kernels(name, N, K, act):
    t = GGMLType[name]
    w = QuantWeight(t, N, K, [torch.empty(0, dtype=torch.uint8)] * 4)
    for T, (general, blocks) in zip(ROWS, MEASURED[name, N, K, act]):
        takes = t != GGMLType.BF16
        on_blocks = T > F.gemv_rows(w, act, takes) if T <= 8 else takes and T <= F.block_rows(w, act)
        assert (blocks if on_blocks else general) <= 1.03 * general, T
        assert T > 2 or not on_blocks or blocks <= general


def test_the_route_is_worked_out_once(recorder):
    for T, most in ((1, 0), (2, 1), (5, 1), (9, 1), (64, 1), (65, 0), (300, 0)):
        for t in (GGMLType.Q4_K, GGMLType.Q8_0):
            recorder.asked = 0
            w = LARGE[t]
            F.linear(F.Act(torch.randn(T, w.K).bfloat16()), w)
            ours = recorder.calls.count("gemm_blocks")             # the recorder's own check of what it is given
            recorder.calls.clear()
            assert recorder.asked - ours <= most, (t, T)
