"""Decode attention through F.attention: caches whose rows are slices of wider rows, keys written just ahead, lengths far apart."""
import pytest
import torch

from tensorsharp_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def decode_batch(lens, page, positions=None):
    """A batch of one new token per sequence, the last of its ``lens`` positions; pages in a random order."""
    need = [-(-n // page) for n in lens]
    order, at = torch.randperm(sum(need)).tolist(), 0
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    for b, n in enumerate(need):
        table[b, :n] = torch.tensor(order[at:at + n])
        at += n
    slots = [int(table[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(lens)]
    B = len(lens)
    return F.Batch(tokens=i32([0] * B), positions=i32([n - 1 for n in lens]), slots=torch.tensor(slots, device=DEV), cu_q=i32(list(range(B + 1))),
                   kv_lens=i32(lens), block_table=table.to(DEV), last_idx=torch.arange(B, device=DEV), seq_slots=torch.arange(B, device=DEV), max_q_len=1,
                   max_kv_len=max(lens), is_decode=True, page_size=page, h_cu_q=tuple(range(B + 1)), h_kv_lens=tuple(lens), rows_in_order=True), sum(need) * page


def exact(q, k, v, batch, scale, window=0, sinks=None):
    """Attention in 64 bits."""
    B, Hq, Dh = q.shape
    out = torch.empty(B, Hq, Dh, dtype=torch.float64, device=DEV)
    for b, n in enumerate(batch.h_kv_lens):
        j = torch.arange(max(0, n - window) if window else 0, n, device=DEV)
        rows = batch.block_table[b, j // batch.page_size].long() * batch.page_size + j % batch.page_size
        kb, vb = (x[rows].double() for x in (k, v))
        qb = q[b].double().view(kb.shape[1], -1, Dh)
        s = torch.einsum("kgd,nkd->kgn", qb, kb) * scale
        if sinks is not None:
            s = torch.cat([s, sinks.double().view(s.shape[0], s.shape[1], 1)], 2)
        out[b] = torch.einsum("kgn,nkd->kgd", torch.softmax(s, 2)[..., :len(j)], vb).reshape(Hq, Dh)
    return out


def worst(got, want):
    """Largest relative error of a (sequence, head)."""
    got, want = got.double().view_as(want), want
    return ((got - want).norm(dim=-1) / want.norm(dim=-1)).max().item()


# weights and the result in bf16, 2^-9 each at most: of a head 5e-3 at most, whatever the lengths
@pytest.mark.parametrize("as_act", [False, True])
@pytest.mark.parametrize("window", [0, 50])
def test_rows_that_are_slices(window, as_act):
    torch.manual_seed(1)
    Hq, Hkv, Dh, page = 8, 2, 64, 64
    batch, rows = decode_batch([1, 40, 130, 700], page)
    wide = torch.randn(rows, 3 * Hkv * Dh, device=DEV).bfloat16()
    k, v = (wide[:, i * Hkv * Dh:(i + 1) * Hkv * Dh].unflatten(1, (Hkv, Dh)) for i in (0, 2))
    q = torch.randn(4, Hq, Dh, device=DEV).bfloat16()
    got = F.attention(q, k, v, batch, scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, window=window, as_act=as_act)
    assert worst(got.b if as_act else got, exact(q, k, v, batch, Dh ** -0.5, window)) < 5e-3


def stepped(batch, rows, Hq, Hkv, Dh, ahead):
    """Rows of this step through the rotary kernel and the attention right behind it, over a cache that holds everything older."""
    k, v = (torch.randn(rows, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    k[batch.slots], v[batch.slots] = float("nan"), float("nan")           # not yet there
    q, kn, vn = (torch.randn(batch.B, h, Dh, device=DEV) for h in (Hq, Hkv, Hkv))
    outs = []
    for _ in range(20):                                                   # launched in a row: rotary, attention, rotary, ...
        k[batch.slots], v[batch.slots] = float("nan"), float("nan")
        qr = F.qkv_rope_cache(q, kn, vn, Hq=Hq, Hkv=Hkv, Dh=Dh, batch=batch, k_cache=k, v_cache=v, rope=None)
        outs.append(F.attention(qr, k, v, batch, scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, ahead=ahead))
    want = exact(qr, k, v, batch, Dh ** -0.5)
    assert torch.equal(k[batch.slots], kn.bfloat16())
    return max(worst(o, want) for o in outs)


# newest keys at the start, in the middle and at the end of a chunk of 16; bounds as above
@pytest.mark.parametrize("ahead", [False, True])
@pytest.mark.parametrize("lens", [[1], [17, 300, 64], [2049], [33, 32, 31, 1000, 1, 1217, 640, 16]])
def test_newest_rows_written_just_ahead(lens, ahead):
    torch.manual_seed(2)
    batch, rows = decode_batch(lens, 64)
    batch.rows_apart = True
    assert stepped(batch, rows, 32, 8, 128, ahead) < 5e-3


def test_a_sequence_twice():
    """Two tokens of one sequence as two entries: the second sees the first's key, which the rotary kernel writes in the same launch, in the chunk before its own."""
    torch.manual_seed(3)
    n, page = 1025, 64
    batch, rows = decode_batch([n], page)
    t = batch.block_table[0]
    batch.cu_q, batch.h_cu_q, batch.kv_lens, batch.h_kv_lens = i32([0, 1, 2]), (0, 1, 2), i32([n - 1, n]), (n - 1, n)
    batch.tokens, batch.positions, batch.block_table = i32([0, 0]), i32([n - 2, n - 1]), torch.stack([t, t])
    batch.slots = torch.tensor([int(t[p // page]) * page + p % page for p in (n - 2, n - 1)], device=DEV)
    assert not batch.rows_apart
    assert stepped(batch, rows, 32, 8, 128, True) < 5e-3


# one long sequence among short ones, whose parts are then cut by all positions together; bounds as above
@pytest.mark.parametrize("Hq,Hkv,Dh", [(32, 8, 128), (64, 8, 64), (8, 1, 128)])
@pytest.mark.parametrize("lens", [[300, 9000, 17, 1], [3000, 2500, 600, 1023, 1024, 1025, 500, 64], [129] * 40, [1] * 33 + [20000], [16000, 16000]])
@pytest.mark.parametrize("window,sink", [(0, False), (700, True)])
def test_lengths_far_apart(Hq, Hkv, Dh, lens, window, sink):
    torch.manual_seed(4)
    batch, rows = decode_batch(lens, 64)
    k, v = (torch.randn(rows, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    q, sinks = torch.randn(len(lens), Hq, Dh, device=DEV).bfloat16(), torch.randn(Hq, device=DEV) if sink else None
    kw = dict(scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, window=window, sinks=sinks)
    got = F.attention(q, k, v, batch, as_act=True, **kw)
    assert worst(got.b, exact(q, k, v, batch, Dh ** -0.5, window, sinks)) < 5e-3
    back = got.q.view(len(lens), -1, 32).double() * got.ds.view(len(lens), -1, 2)[..., :1].double()
    assert (back.view_as(got.b.double()) - got.b.double()).abs().max() <= got.b.abs().max().double() / 254 * 1.01       # half a step of 127ths of a group's largest value
    batch.max_kv_len = 32768                                             # a captured step's bucket: the same parts, the same bits
    assert torch.equal(F.attention(q, k, v, batch, **kw), got.b)


@pytest.mark.parametrize("Hq,Hkv,Dh,lens", [(32, 8, 128, [2048 - 64 * i for i in range(16)]), (64, 8, 64, [1024 - 8 * i for i in range(64)]), (32, 8, 128, [700, 400])])
def test_even_lengths_are_cut_as_each_alone(Hq, Hkv, Dh, lens):
    """Where no sequence is far longer than the others the plan changes nothing: the bits of a launch that cuts each sequence into the same number of parts."""
    torch.manual_seed(5)
    batch, rows = decode_batch(lens, 64)
    k, v = (torch.randn(rows, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(len(lens), Hq, Dh, device=DEV).bfloat16()
    got = F.attention(q, k, v, batch, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh)
    assert any(key[0] == "attn_plan" for key in batch.cache)
    each = F.decode_parts(batch, Hkv, 0)[1]
    alone = F._k().attn_decode(q, k, v, batch.block_table, batch.kv_lens, scale=0.1, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=64, splits=each, split_len=-128)
    assert torch.equal(got.view_as(alone), alone)


# every warp goes round its ring of three chunks many times; bounds as above, for each sequence and head
@pytest.mark.parametrize("Hq,Hkv,Dh", [(32, 8, 128), (64, 8, 64), (16, 1, 64)])
@pytest.mark.parametrize("page", [16, 64])
@pytest.mark.parametrize("window", [0, 900])
@pytest.mark.parametrize("splits,split_len", [(1, 0), (2, 0), (2, -128), (1, 3072)])
def test_long_parts(Hq, Hkv, Dh, page, window, splits, split_len):
    if window and split_len > 0:
        pytest.skip("a fixed split length goes with no window")
    torch.manual_seed(6)
    batch, rows = decode_batch([500, 777, 1023, 1024, 1025, 2048, 3000], page)
    k, v = (torch.randn(rows, Hkv, Dh, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(7, Hq, Dh, device=DEV).bfloat16()
    got = F._k().attn_decode(q, k, v, batch.block_table, batch.kv_lens, scale=Dh ** -0.5, Hq=Hq, Hkv=Hkv, Dh=Dh, page_size=page, splits=splits, split_len=split_len,
                             window=window)
    assert worst(got, exact(q, k, v, batch, Dh ** -0.5, window)) < 5e-3
