"""Single-token rows around the sizes where a second round of groups would leave most warps idle (csrc/gemv_stream.cu), against the decoded weights in double precision."""
import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.quant.qweight import QuantWeight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# Whole numbers up to 127 with a 127 in every group of 32 are exact in int8 groups: what is left is the rounding of float sums, at most some 200 additions of terms
# as large as the result's parts (1e-5 with room); silu(g) * u moves by less than 1.1 of either's error times the other.
@pytest.mark.parametrize("t", [GGMLType.Q6_K, GGMLType.Q8_0])
@pytest.mark.parametrize("N,Kd", [(3552, 512), (3553, 512), (4096, 1024), (4262, 1024), (4264, 1024), (4096, 4096), (7104, 2048), (8192, 2048), (8526, 2048), (2400, 4096)])
@pytest.mark.parametrize("act", [None, "swiglu"])
def test_rows_of_one_and_a_bit_rounds(t, N, Kd, act):
    from tensorsharp_b200.ops import kernels as k
    if act and N % 2:
        pytest.skip("two halves")
    torch.manual_seed(N)
    w = QuantWeight.from_float(torch.randn(N, Kd, device=DEV) * 0.05 * torch.rand(N, 1, device=DEV), t)
    x = torch.randint(-127, 128, (1, Kd // 32, 32), device=DEV)
    x[..., 5] = 127
    x = (x.reshape(1, Kd).float() / 64).bfloat16()
    xq, xds = k.quantize_q8(x)
    got = k.gemv(w, xq=xq, xds=xds, M=1, act=act).double()
    y, parts = x.double() @ w.dequantize().double().t(), x.double().abs() @ w.dequantize().double().abs().t()
    if act is None:
        assert ((got - y).abs() <= 1e-5 * parts + 1e-6).all()
        return
    n = N // 2
    want = torch.nn.functional.silu(y[:, :n]) * y[:, n:]
    tol = 1e-5 * (1.1 * parts[:, :n] * y[:, n:].abs() + parts[:, n:] * y[:, :n].abs() + want.abs()) + 1e-5
    assert ((got - want).abs() <= tol).all()
