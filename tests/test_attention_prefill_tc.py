"""Prompt attention on tcgen05 (csrc/attention_prefill_tc.cu) against the float32 softmax, at the sizes where its tiles end."""
import pytest
import torch

from tensorsharp_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _paged(lens, Hkv, Dh, ps):
    """Caches whose pages are dealt out in a shuffled order; slots that no sequence owns, and those past each end, hold NaN."""
    need = [(n + ps - 1) // ps for n in lens]
    pages = torch.randperm(sum(need) + 2)
    kc, vc = (torch.full(((sum(need) + 2) * ps, Hkv, Dh), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    table, rows, at = torch.zeros(len(lens), max(need), dtype=torch.int32), [], 0
    for b, (n, c) in enumerate(zip(lens, need)):
        table[b, :c] = pages[at:at + c]
        at += c
        idx = (table[b, :c].long()[:, None] * ps + torch.arange(ps)).reshape(-1)[:n].to(DEV)
        kc[idx], vc[idx] = torch.randn(n, Hkv, Dh, device=DEV).bfloat16(), torch.randn(n, Hkv, Dh, device=DEV).bfloat16()
        rows.append(idx)
    return kc, vc, table.to(DEV), rows


def _check(Hq, Hkv, Dh, qlens, lens, ps=64, window=0, sinks=False, softcap=0.0, gate=False, scale=None, peak=1.0):
    from tensorsharp_b200.ops import kernels as K
    torch.manual_seed(3)
    scale = scale or Dh ** -0.5
    kc, vc, table, rows = _paged(lens, Hkv, Dh, ps)
    q = (torch.randn(sum(qlens), Hq, Dh, device=DEV) * peak).bfloat16()
    sk = torch.randn(Hq, device=DEV) if sinks else None
    gt = torch.randn(sum(qlens), Hq, device=DEV) if gate else None
    cu = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32, device=DEV)
    kl = torch.tensor(lens, dtype=torch.int32, device=DEV)

    def run():
        return K.attn_prefill(q, kc, vc, table, kl, cu, max(qlens), scale=scale, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=ps, sinks=sk, softcap=softcap,
                              window=window, gate=gt)
    got = run()
    assert all(torch.equal(got, run()) for _ in range(20))              # no atomics, one order of sums: the same bits every time
    assert int(K.gemm_status(DEV).item()) == 0
    at = 0
    for ql, n, r in zip(qlens, lens, rows):
        want = ref.attention(q[at:at + ql], kc[r], vc[r], torch.arange(n - ql, n, device=DEV), scale=scale, window=window, sinks=sk, softcap=softcap)
        if gate:
            want = want * torch.sigmoid(gt[at:at + ql])[..., None]
        # the weights and the result are rounded to bf16 once each, at most 2^-9 of a term: errors add over a row as the
        # terms themselves do, so the 2-norm is off by at most 2 * 2^-9 = 0.4 % where nothing cancels
        err = ((got[at:at + ql].float() - want).norm() / want.norm()).item()
        assert err < 6e-3, (ql, n, err)
        at += ql


HEADS = [(8, 1, 64), (8, 2, 128), (3, 3, 128), (12, 2, 128), (16, 1, 256), (6, 6, 64)]


@pytest.mark.parametrize("Hq,Hkv,Dh", HEADS)
def test_edges(Hq, Hkv, Dh):
    # one token, tile edges of 64 and 128 keys, prompts on top of a cache, the last token of a long sequence
    _check(Hq, Hkv, Dh, [1, 63, 64, 65, 129, 1, 17, 200], [1, 63, 64, 65, 129, 400, 145, 713])


@pytest.mark.parametrize("Hq,Hkv,Dh", HEADS)
@pytest.mark.parametrize("window", [1, 70, 128])
def test_windows(Hq, Hkv, Dh, window):
    _check(Hq, Hkv, Dh, [5, 300, 130], [5, 300, 900], window=window, sinks=True)


@pytest.mark.parametrize("Hq,Hkv,Dh", HEADS[:2] + HEADS[4:5])
def test_forms(Hq, Hkv, Dh):
    _check(Hq, Hkv, Dh, [70, 9], [70, 333], ps=128, softcap=20.0, gate=True)
    _check(Hq, Hkv, Dh, [257], [1000], sinks=True, peak=30.0)            # row maxima that grow: O is rescaled
    _check(Hq, Hkv, Dh, [2300], [2300])                                  # 144 CTAs: just below one per SM at head sizes 64 and 128


# on the GPU's 148 SMs: grids on either side of one CTA per SM (head size 64) and two (128), where the tiles change from 128 to 64 keys
@pytest.mark.parametrize("Hq,Hkv,Dh,qlens,lens", [
    (64, 8, 64, [288], [700]), (64, 8, 64, [304], [700]), (64, 8, 64, [1000, 17, 333], [1000, 500, 333]),
    (32, 8, 128, [1184], [1500]), (32, 8, 128, [1185], [1500]), (32, 8, 128, [2048], [2048]), (32, 8, 128, [900, 5, 700], [2000, 400, 700])])
@pytest.mark.parametrize("window,sinks,peak", [(0, False, 1.0), (300, True, 1.0), (0, True, 20.0)])
def test_grids_of_one_and_two_blocks_per_sm(Hq, Hkv, Dh, qlens, lens, window, sinks, peak):
    _check(Hq, Hkv, Dh, qlens, lens, window=window, sinks=sinks, peak=peak)


def test_window_over_a_ring_of_pages():
    """A table whose pages come round again: only the pages that the window reaches hold their own keys."""
    from tensorsharp_b200.ops import kernels as K
    torch.manual_seed(8)
    Hq, Hkv, Dh, window, n, ql, ring = 8, 2, 128, 200, 1500, 180, 7
    k, v = (torch.randn(n, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    kc, vc = (torch.zeros(ring * 64, Hkv, Dh, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    for j in range(n):                                                       # the newest keys stay, as a ring keeps them
        kc[j % (ring * 64)], vc[j % (ring * 64)] = k[j], v[j]
    table = (torch.arange((n + 63) // 64, dtype=torch.int32, device=DEV) % ring)[None].contiguous()
    q = torch.randn(ql, Hq, Dh, device=DEV).bfloat16()
    cu, kl = torch.tensor([0, ql], dtype=torch.int32, device=DEV), torch.tensor([n], dtype=torch.int32, device=DEV)
    got = K.attn_prefill(q, kc, vc, table, kl, cu, ql, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=64, window=window)
    want = ref.attention(q, k, v, torch.arange(n - ql, n, device=DEV), scale=0.1, window=window)
    assert ((got.float() - want).norm() / want.norm()).item() < 6e-3


@pytest.mark.parametrize("Hq,Hkv,Dh", [(16, 2, 64), (8, 2, 128)])
@pytest.mark.parametrize("qlens,lens,window,softcap", [([600], [700], 0, 20.0), ([256, 255, 3], [256, 256, 250], 0, 0.0), ([400, 257], [900, 257], 256, 0.0),
                                                      ([400, 257], [900, 257], 257, 0.0), ([600, 9], [700, 9], 100, 20.0)])
def test_both_sides_of_the_tile_rule(Hq, Hkv, Dh, qlens, lens, window, softcap):
    # grids below one CTA per SM: 64-key tiles with a soft cap and where a row sees at most 256 keys, 128-key tiles otherwise
    _check(Hq, Hkv, Dh, qlens, lens, window=window, softcap=softcap, gate=softcap > 0 and window > 0)


@pytest.mark.parametrize("qlens,lens", [([64], [128]), ([65], [65]), ([128, 3], [128, 120]), ([65] * 7, [70] * 7), ([65] * 8, [70] * 8), ([10] * 29, [100] * 29),
                                        ([64] * 30, [128] * 30), ([10] * 30, [129] * 30)])
def test_both_sides_of_the_rule_for_single_heads(qlens, lens):
    # ten heads in groups of five: one head per row tile
    _check(10, 2, 64, qlens, lens, sinks=True)


@pytest.mark.parametrize("Hq,Hkv,Dh,ql,n,peak", [(32, 8, 128, 300, 2000, 3.0), (32, 8, 128, 1100, 1100, 6.0), (16, 2, 64, 1024, 1024, 4.0), (16, 2, 256, 200, 900, 3.0)])
def test_as_exact_as_the_mma_kernel(Hq, Hkv, Dh, ql, n, peak):
    """Both kernels round each weight, taken relative to the running maximum, and the result to bf16 and keep the rest in f32, so
    their errors against 64 bits are two samples of one size: over the 10^5 and more values here they differ by well below 3 %."""
    from tensorsharp_b200.ops import kernels as K
    torch.manual_seed(5)
    kc, vc, table, (r,) = _paged([n], Hkv, Dh, 64)
    q = (torch.randn(ql, Hq, Dh, device=DEV) * peak).bfloat16()
    cu, kl = torch.tensor([0, ql], dtype=torch.int32, device=DEV), torch.tensor([n], dtype=torch.int32, device=DEV)
    s = torch.einsum("thd,nhd->htn", q.double(), kc[r].double().repeat_interleave(Hq // Hkv, 1)) * Dh ** -0.5
    s = s.masked_fill(torch.arange(n, device=DEV) > torch.arange(n - ql, n, device=DEV)[:, None], float("-inf"))
    want = torch.einsum("htn,nhd->thd", s.softmax(-1), vc[r].double().repeat_interleave(Hq // Hkv, 1))
    err = []
    for pos0 in (None, torch.tensor([n - ql], dtype=torch.int32, device=DEV)):             # first positions given: the kernel of attention.cu
        got = K.attn_prefill(q, kc, vc, table, kl, cu, ql, scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=64, q_pos0=pos0)
        err.append(((got.double() - want).norm() / want.norm()).item())
    assert err[0] < 1.03 * err[1], err


def test_output_off_sixteen_bytes():
    """A caller's output that starts on 8 bytes only: 16-byte stores may not reach it."""
    from tensorsharp_b200.ops import kernels as K
    torch.manual_seed(6)
    kc, vc, table, (r,) = _paged([200], 2, 128, 64)
    q = torch.randn(70, 8, 128, device=DEV).bfloat16()
    cu, kl = torch.tensor([0, 70], dtype=torch.int32, device=DEV), torch.tensor([200], dtype=torch.int32, device=DEV)
    buf = torch.zeros(4 + 70 * 8 * 128 + 4, dtype=torch.bfloat16, device=DEV)
    K.attn_prefill(q, kc, vc, table, kl, cu, 70, scale=0.1, Hq=8, Hkv=2, Dh=128, page_size=64, out=buf[4:-4].view(70, 8, 128))
    want = ref.attention(q, kc[r], vc[r], torch.arange(130, 200, device=DEV), scale=0.1)
    assert ((buf[4:-4].view(70, 8, 128).float() - want).norm() / want.norm()).item() < 6e-3 and not buf[:4].any() and not buf[-4:].any()


def test_gate_through_the_public_call():
    """F.attention names every form, at its neutral value: the route follows the values, and the bits those of the plain call."""
    from tensorsharp_b200.ops import functional as F
    from tensorsharp_b200.ops import kernels as K
    torch.manual_seed(7)
    T, n, Hq, Hkv, Dh = 90, 300, 8, 2, 128
    kc, vc, table, (r,) = _paged([n], Hkv, Dh, 64)
    q, gate = torch.randn(T, Hq, Dh, device=DEV).bfloat16(), torch.randn(T, Hq, device=DEV)
    cu, kl = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.tensor([n], dtype=torch.int32, device=DEV)
    pos = torch.arange(n - T, n, device=DEV, dtype=torch.int32)
    batch = F.Batch(tokens=pos, positions=pos, slots=pos.long(), cu_q=cu, kv_lens=kl, block_table=table, last_idx=None, seq_slots=None, max_q_len=T,
                    max_kv_len=n, is_decode=False, page_size=64, h_cu_q=(0, T), h_kv_lens=(n,))
    got = F.attention(q, kc, vc, batch, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh, gate=gate)
    plain = K.attn_prefill(q, kc, vc, table, kl, cu, T, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=64, gate=gate)
    want = ref.attention(q, kc[r], vc[r], pos, scale=0.1) * torch.sigmoid(gate)[..., None]
    assert ((plain.float() - want).norm() / want.norm()).item() < 6e-3 and torch.equal(got.view_as(plain), plain)
