"""Kernels of the prompt path and of batched experts against plain tensor arithmetic, at the sizes where their tiles end."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

from tensorsharp_b200.gguf.constants import GGMLType
from tensorsharp_b200.ops import reference as ref
from tensorsharp_b200.quant.qweight import QuantWeight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from tensorsharp_b200.ops import kernels
    return kernels


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def status():
    return int(K().gemm_status(DEV).item())


# f32 sums of exact bf16 products in another order: far below 1e-5; a bf16 result is rounded once, 2^-9 at most: 2e-3
@pytest.mark.parametrize("T", [65, 80, 129, 600, 2050])
@pytest.mark.parametrize("N,Kd", [(1, 64), (40, 72), (255, 320), (257, 128), (640, 2048), (4104, 512)])
def test_gemm_pairs(T, N, Kd):
    torch.manual_seed(1)
    W, X = (torch.randn(N, Kd, device=DEV) * 0.05).bfloat16(), torch.randn(T, Kd, device=DEV).bfloat16()
    want = X.double() @ W.double().t()
    assert rel(K().gemm_bf16(W, X, out_dtype=torch.float32), want) < 1e-5
    bias, res = torch.randn(N, device=DEV), torch.randn(T, N, device=DEV)
    assert rel(K().gemm_bf16(W, X, out_dtype=torch.float32, bias=bias, residual=res), want + bias + res) < 1e-5
    assert rel(K().gemm_bf16(W, X, bias=bias, residual=res.bfloat16()), want + bias + res.bfloat16()) < 3e-3
    assert status() == 0


def test_gemm_pairs_launched_back_to_back():
    """Hundreds of launches with nothing between them, each with the tensor memory that the one before gives back."""
    torch.manual_seed(2)
    W, X = (torch.randn(700, 192, device=DEV) * 0.05).bfloat16(), torch.randn(300, 192, device=DEV).bfloat16()
    want = K().gemm_bf16(W, X, out_dtype=torch.float32)
    outs = [K().gemm_bf16(W, X, out_dtype=torch.float32) for _ in range(300)]
    assert all(torch.equal(o, want) for o in outs) and status() == 0


# each of gate and up is rounded to bf16 ahead of the activation and the result once more; swiglu's slope is at most about 1.1
@pytest.mark.parametrize("act", ["swiglu", "geglu", "geglu_erf", "swiglu_oai"])
@pytest.mark.parametrize("T,F,Kd", [(65, 40, 64), (300, 129, 200), (1000, 576, 512), (2050, 4104, 72)])      # the last: several tiles a pair
def test_gemm_glu(act, T, F, Kd):
    torch.manual_seed(3)
    W, X, b = (torch.randn(2 * F, Kd, device=DEV) * 0.1).bfloat16(), torch.randn(T, Kd, device=DEV).bfloat16(), torch.randn(2 * F, device=DEV)
    y = (X.double() @ W.double().t() + b).float().bfloat16()
    want = ref.glu(act, y[:, :F], y[:, F:])
    for _ in range(3):
        assert rel(K().gemm_bf16_glu(W, X, act, bias=b), want) < 6e-3
    assert status() == 0


@pytest.mark.parametrize("T,E,k,bn", [(70, 8, 1, 80), (500, 7, 3, 112), (1000, 32, 4, 256), (33, 300, 8, 32)])
@pytest.mark.parametrize("e0", [0, 2])
def test_moe_spread_and_grouped(T, E, k, bn, e0):
    torch.manual_seed(4)
    Kd, N = 128, 264
    x = torch.randn(T, Kd, device=DEV).bfloat16()
    ids = torch.stack([torch.randperm(E + 3, device=DEV)[:k] for _ in range(T)]).to(torch.int32)       # some of other ranks
    xs, pos, tiles = K().moe_spread(x, ids, e0, E, bn)
    e = ids.reshape(-1).long() - e0
    ok = (e >= 0) & (e < E)
    p = pos.long()
    assert torch.equal(p < 0, ~ok) and torch.equal(p[ok].sort().values, torch.arange(int(ok.sum()), device=DEV))
    assert torch.equal(xs[p[ok]], x.repeat_interleave(k, 0)[ok])
    owner = torch.full((T * k,), -1, device=DEV)
    for g, a, b in tiles.tolist():
        if g >= 0:
            assert 0 < b - a <= bn
            assert (owner[a:b] == -1).all()
            owner[a:b] = g
    assert torch.equal(owner[p[ok]], e[ok])
    W = (torch.randn(E * N, Kd, device=DEV) * 0.1).bfloat16()
    bias = torch.randn(E, N, device=DEV)
    y = K().gemm_bf16_grouped(W, E, xs, tiles, bn, out_dtype=torch.float32, bias=bias, zero=False)
    want = torch.einsum("pk,pnk->pn", x.repeat_interleave(k, 0)[ok].double(), W.view(E, N, Kd)[e[ok]].double()) + bias[e[ok]]
    assert rel(y[p[ok]], want) < 1e-5
    if bn > 64:
        h = K().gemm_bf16_glu(W, xs, "swiglu", bias=bias, E=E, tiles=tiles, bn=bn)
        yb = want.float().bfloat16()
        assert rel(h[p[ok]], ref.glu("swiglu", yb[:, :N // 2], yb[:, N // 2:])) < 6e-3
    w, s, g, r = torch.rand(T, k, device=DEV), torch.randn(T, N, device=DEV), torch.randn(T, 1, device=DEV), torch.randn(T, N, device=DEV)
    full = torch.zeros(T * k, N, device=DEV, dtype=torch.float64)
    full[ok] = want * w.reshape(-1)[ok].unsqueeze(1)
    got = K().moe_combine(y, pos, w.reshape(-1), T, k, (s, g), r)
    assert rel(got, full.view(T, k, N).sum(1) + s * torch.sigmoid(g) + r) < 1e-5
    assert status() == 0


# tiles of 1 .. 16 pairs, rows that end inside a 64-row block, 9 blocks of K (one stage and a bit), both 4-bit types
@pytest.mark.parametrize("t", [GGMLType.MXFP4, GGMLType.Q4_0])
@pytest.mark.parametrize("T,k,E,Kd,Fd", [(40, 2, 3, 288, 160), (70, 1, 4, 2880, 96), (33, 4, 9, 64, 256),
                                           # gate and up once on an SM: 255 pairs tiles of eight, 256 pairs of sixteen; beyond the ring's K; an odd number of blocks there
                                           (255, 1, 32, 4096, 64), (256, 1, 32, 4096, 64), (40, 2, 3, 12288, 64), (40, 2, 3, 12320, 32)])
def test_moe_tiles_of_sixteen(t, T, k, E, Kd, Fd):
    torch.manual_seed(5)
    gu = QuantWeight.from_float(torch.randn(E, 2 * Fd, Kd, device=DEV) * 0.1, t)
    dn = QuantWeight.from_float(torch.randn(E, Kd, Fd, device=DEV) * 0.1, t)
    gb, db = torch.randn(E, 2 * Fd, device=DEV) * 0.1, torch.randn(E, Kd, device=DEV) * 0.1
    x = torch.randn(T, Kd, device=DEV).bfloat16()
    ids = torch.stack([torch.randperm(E, device=DEV)[:k] for _ in range(T)]).to(torch.int32)
    w = torch.rand(T, k, device=DEV)
    xq, xds = K().quantize_q8(x)
    got = K().moe_grouped(xq=xq, xds=xds, ids=ids, weights=w.reshape(-1), gate_up=gu, down=dn, act="swiglu", gate_up_bias=gb, down_bias=db)
    # the activations as the kernel sees them: int8 groups of 32 with one scale; between the projections bf16, then int8 again
    xd = (xq.view(T, -1, 32).double() * xds[..., :1].double()).view(T, Kd)
    G, D = gu.dequantize().view(E, 2 * Fd, Kd).double(), dn.dequantize().view(E, Kd, Fd).double()
    want = torch.zeros(T, Kd, dtype=torch.float64, device=DEV)
    for j in range(k):
        e = ids[:, j].long()
        y = torch.einsum("tk,tnk->tn", xd, G[e]) + gb[e]
        h = ref.glu("swiglu", y[:, :Fd].float(), y[:, Fd:].float()).bfloat16()
        hq, hds = K().quantize_q8(h)
        hd = (hq.view(T, -1, 32).double() * hds[..., :1].double()).view(T, Fd)
        want += (torch.einsum("tk,tnk->tn", hd, D[e]) + db[e]) * w[:, j:j + 1].double()
    # a bf16 value on a rounding edge may fall the other way (2^-8 of it) and its int8 code with it (1 / 127 of its group's largest)
    assert rel(got, want) < 5e-3


def test_moe_tiles_without_matrix_instructions():
    """The same with TSB_MOE_MMA=0, which the library reads once per process: every tile then goes to a kernel of eight rows."""
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", f"{__file__}::test_moe_tiles_of_sixteen"], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, TSB_MOE_MMA="0"))
    assert r.returncode == 0, r.stdout[-3000:]


def test_moe_tile_height_is_checked():
    lib, w = K()._lib(), QuantWeight.from_float(torch.randn(1, 64, 64, device=DEV), GGMLType.Q8_0)
    none = C.c_void_p(0)
    some = K()._p(torch.zeros(1 << 12, dtype=torch.int8, device=DEV))

    def call(rows, max_tiles=0):
        return lib.tsb_moe_gemv_tiles(*K()._planes(w), C.c_int(int(w.ggml_type)), C.c_int(64), C.c_int(64), some, some, none, some, none, none, some, some,
                                      C.c_int(max_tiles), C.c_int(rows), C.c_int(1), C.c_int(0), K()._stream())
    assert call(8) == 0 and call(16) != 0 and call(0) != 0


@pytest.mark.parametrize("Hq,Hkv,Dh,rot", [(8, 2, 64, 64), (5, 1, 128, 128), (4, 2, 256, 64), (3, 3, 128, 32), (16, 8, 128, 0), (14, 2, 256, 128)])
@pytest.mark.parametrize("T", [64, 65, 374, 375, 700])             # 374 / 375: either side of the line of the first heads
@pytest.mark.parametrize("f32", [False, True])
def test_rope_rows(Hq, Hkv, Dh, rot, T, f32):
    from tensorsharp_b200.ops import functional as F
    torch.manual_seed(6)
    H = Hq + 2 * Hkv
    qkv = torch.randn(T, H * Dh, device=DEV).to(torch.float32 if f32 else torch.bfloat16)
    q, k, v = qkv[:, :Hq * Dh].view(T, Hq, Dh), qkv[:, Hq * Dh:(Hq + Hkv) * Dh].view(T, Hkv, Dh), qkv[:, (Hq + Hkv) * Dh:].view(T, Hkv, Dh)
    qn, kn = torch.rand(Dh, device=DEV) + 0.5, torch.rand(Dh, device=DEV) + 0.5
    pos = torch.randint(0, 5000, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(T + 9, device=DEV)[:T]
    kc, vc = (torch.zeros(T + 9, Hkv, Dh, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    batch = F.Batch(tokens=pos, positions=pos, slots=slots, cu_q=None, kv_lens=pos, block_table=None, last_idx=None, seq_slots=None, max_q_len=T,
                    max_kv_len=T, is_decode=False, page_size=64)
    spec = F.RopeSpec(rot_dim=rot, theta_base=1e4) if rot else None
    out = F.qkv_rope_cache(q, k, v, Hq=Hq, Hkv=Hkv, Dh=Dh, batch=batch, k_cache=kc, v_cache=vc, rope=spec, qn=qn, kn=kn, v_norm=True, q_scale=0.5)
    qf, kf, vf = ref.rmsnorm(q.float(), qn, 1e-6), ref.rmsnorm(k.float(), kn, 1e-6), ref.rmsnorm(v.float(), None, 1e-6)
    if rot:
        c, s = ref.rope_cos_sin(pos, rot, 1e4)
        qf, kf = ref.apply_rope(qf, c, s, rot, 0), ref.apply_rope(kf, c, s, rot, 0)
    # one bf16 rounding of the result; angles up to 5000 in f32, 3e-4 off at most
    for got, want in ((out, qf * 0.5), (kc[slots], kf), (vc[slots], vf)):
        assert rel(got, want) < 3e-3


@pytest.mark.parametrize("C", [4, 132, 1024, 1124, 1128, 2052])           # five prompts of at most 64 tokens: from 1128 channels on the kernel for prompts
@pytest.mark.parametrize("f32", [False, True])
def test_conv_over_prompts(C, f32):
    torch.manual_seed(7)
    lens = [16, 1, 23, 2, 64]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    x = torch.randn(sum(lens), C + 8, device=DEV).to(torch.float32 if f32 else torch.bfloat16)[:, :C]
    w, bias, state = torch.randn(C, 4, device=DEV), torch.randn(C, device=DEV), torch.randn(7, 3, C, device=DEV)
    slots = torch.tensor([4, 0, 6, 1, 3], device=DEV)
    want, tail = [], state.clone()
    for i, s in enumerate(slots.tolist()):
        o, t = ref.causal_conv1d(x[cu[i]:cu[i + 1]].float().cpu(), w.cpu(), bias.cpu(), state[s].cpu(), True)
        want.append(o.to(DEV))
        tail[s] = t.to(DEV)
    got = K().causal_conv1d(x, w, bias, state, cu, slots, max(lens))
    assert rel(got, torch.cat(want)) < 1e-5 and torch.equal(state, tail)


@pytest.mark.parametrize("n", [65535 * 8, 65535 * 8 + 1])
def test_conv_over_the_longest_prompts(n):
    """Either side of the 65535 groups of eight tokens that a grid dimension takes."""
    torch.manual_seed(9)
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    x, w, state = torch.randn(n, 4, device=DEV), torch.randn(4, 4, device=DEV), torch.randn(1, 3, 4, device=DEV)
    want, tail = (t.to(DEV) for t in ref.causal_conv1d(x.cpu(), w.cpu(), None, state[0].cpu(), True))
    got = K().causal_conv1d(x, w, None, state, cu, torch.zeros(1, dtype=torch.int64, device=DEV), n)
    assert rel(got, want) < 1e-5 and torch.equal(state[0], tail)


@pytest.mark.parametrize("D", [32, 2048, 5376, 8192])
@pytest.mark.parametrize("rows", [1, 16, 300])
def test_rms_seam(D, rows):
    torch.manual_seed(8)
    y, h = torch.randn(rows, D, device=DEV) * 3, torch.randn(rows, D, device=DEV)
    post, pre = torch.rand(D, device=DEV) + 0.5, torch.rand(D, device=DEV) + 0.5
    h1, a, q, ds = K().rms_seam(y, post, h, pre, 1e-6, want_q8=True)
    want = h.double() + ref.rmsnorm(y.double(), post, 1e-6).double()
    assert rel(h1, want) < 1e-6
    assert rel(a, ref.rmsnorm(want.float(), pre, 1e-6)) < 3e-3
    wq, wds = K().quantize_q8(ref.rmsnorm(want.float(), pre, 1e-6).contiguous())
    assert (q.int() - wq.int()).abs().max() <= 1 and rel(ds[..., 0], wds[..., 0]) < 1e-5


# either side of the lines of the Q8_0 pair loop (K 1024, and 8192 rows for several activation rows), K with a group that ends early
@pytest.mark.parametrize("N,Kd", [(8192, 1024), (8192, 1056), (8196, 1056), (8196, 2080), (6, 1056), (6, 32)])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_q8_pairs(N, Kd, M):
    torch.manual_seed(10)
    w = QuantWeight.from_float(torch.randn(N, Kd, device=DEV) * 0.1, GGMLType.Q8_0)
    xq, xds = K().quantize_q8(torch.randn(M, Kd, device=DEV))
    got = K().gemv(w, xq=xq, xds=xds, M=M, act="swiglu")
    y = (xq.view(M, -1, 32).double() * xds[..., :1].double()).view(M, Kd) @ w.dequantize().double().t()
    # whole-number products of blocks, scaled and added in f32
    assert rel(got, torch.nn.functional.silu(y[:, :N // 2]) * y[:, N // 2:]) < 1e-5


@pytest.mark.parametrize("D,dtype,plain", [(2048, torch.float32, False), (2048, torch.bfloat16, False), (8224, torch.float32, False), (2056, torch.float32, False),
                                           (2048, torch.float32, True)])
def test_norm_add_norm(D, dtype, plain):
    """The seam of two norms in one kernel and, for a bf16 sublayer, wide or odd rows or a missing weight, as two."""
    from tensorsharp_b200.ops import functional as F
    torch.manual_seed(11)
    y, h, post, pre = torch.randn(20, D, device=DEV).to(dtype), torch.randn(20, D, device=DEV), torch.rand(D, device=DEV) + 0.5, torch.rand(D, device=DEV) + 0.5
    post = None if plain else post
    out, a = F.norm_add_norm(y, post, h, pre, 1e-6)
    want = h.double() + ref.rmsnorm(y.double(), post, 1e-6).double()
    assert rel(out, want) < 1e-6 and rel(a.b, ref.rmsnorm(want.float(), pre, 1e-6)) < 3e-3
