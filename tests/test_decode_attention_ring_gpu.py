"""Decode attention that loads ahead (csrc/attention_decode_mma.cu: attn_decode_ring_kernel) against plain attention in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from tensorsharp_b200.ops import kernels
    return kernels


def want(q, k, v, table, lens, page, scale, window, sinks, softcap):
    B, Hq, Dh = q.shape
    out = torch.empty(B, Hq, Dh, dtype=torch.float64, device=DEV)
    for b in range(B):
        j = torch.arange(max(0, lens[b] - window) if window else 0, lens[b], device=DEV)
        slots = table[b, j // page].long() * page + j % page
        kb, vb = (x[slots].double().repeat_interleave(Hq // k.shape[1], 1) for x in (k, v))
        s = torch.einsum("hd,nhd->hn", q[b].double(), kb) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        p = torch.softmax(s, 1)[:, :len(j)]
        out[b] = torch.einsum("hn,nhd->hd", p, vb)
    return out


# softmax weights and values in bf16: 2^-9 each, sums in f32: below 5e-3 of the result.  Lengths at the ends of chunks (16), of a warp's
# stride (64), of pages; windows that start inside a chunk; rows outside the range are NaN and must not reach the sums
@pytest.mark.parametrize("Hq,Hkv,Dh", [(32, 8, 128), (64, 8, 64), (4, 4, 128), (16, 1, 64)])
@pytest.mark.parametrize("page", [16, 64])
@pytest.mark.parametrize("window,sink,softcap", [(0, False, 0.0), (50, True, 0.0), (128, False, 20.0)])
@pytest.mark.parametrize("splits,split_len", [(1, 0), (3, 0), (5, 64), (7, -128)])
def test_against_plain_attention(Hq, Hkv, Dh, page, window, sink, softcap, splits, split_len):
    if window and split_len > 0:
        pytest.skip("a fixed split length goes with no window")
    torch.manual_seed(1)
    lens = [1, 15, 16, 17, 64, 65, 129, 300]
    B, pages = len(lens), (320 + page - 1) // page
    table = torch.randperm(B * pages, device=DEV).int().view(B, pages)
    k, v = (torch.full((B * pages * page, Hkv, Dh), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(2))
    for b, n in enumerate(lens):
        j = torch.arange(max(0, n - window) if window else 0, n, device=DEV)
        slots = table[b, j // page].long() * page + j % page
        k[slots], v[slots] = (torch.randn(len(j), Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(B, Hq, Dh, device=DEV).bfloat16()
    sinks = torch.randn(Hq, device=DEV) if sink else None
    kl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got, gq, gds = K().attn_decode(q, k, v, table, kl, scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=page, splits=splits, split_len=split_len,
                                   window=window, sinks=sinks, softcap=softcap, want_q8=True)
    ref = want(q, k, v, table, lens, page, Dh ** -0.5, window, sinks, softcap)
    assert ((got.double() - ref).norm() / ref.norm()).item() < 5e-3
    back = gq.view(B, -1, 32).double() * gds.view(B, -1, 2)[..., :1].double()
    assert ((back.view_as(ref) - got.double()).norm() / ref.norm()).item() < 1e-2            # 8 bits of a group's largest value


def test_a_sequence_is_cut_alike_whatever_the_bucket():
    """A captured step has splits for its bucket, an eager one for the longest sequence: the same parts, the same bits."""
    torch.manual_seed(2)
    lens, page, Hq, Hkv, Dh = [70, 300, 129], 64, 8, 2, 128
    table = torch.arange(15, device=DEV).int().view(3, 5)
    k, v = (torch.randn(15 * page, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    q, kl = torch.randn(3, Hq, Dh, device=DEV).bfloat16(), torch.tensor(lens, dtype=torch.int32, device=DEV)
    a, b = (K().attn_decode(q, k, v, table, kl, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=page, splits=s, split_len=-128) for s in (3, 8))
    assert torch.equal(a, b)
