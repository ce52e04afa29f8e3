"""The chunked delta rule over states and rows that are slices of wider ones: the bits of the dense call."""
import pytest
import torch

from tensorsharp_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lens", [[70], [65, 1, 130]])
@pytest.mark.parametrize("form", ["state of a layer among others", "state off 16 bytes", "rows off 16 bytes", "rows of a wider product", "every second row"])
def test_slices(monkeypatch, lens, form):
    monkeypatch.setenv("TSB_GDN_CHUNKED", "1")
    monkeypatch.setenv("GDN_CHUNK_PREFILL_MIN_SEQ_LEN", "2")
    torch.manual_seed(1)
    Hk, Hv, Dk, Dv, T, B = 2, 4, 64, 64, sum(lens), len(lens)
    W = 2 * Hk * Dk + Hv * Dv
    qkv, z = torch.randn(T, W, device=DEV), torch.randn(T, Hv * Dv, device=DEV)
    beta, alpha, state0 = torch.randn(T, Hv, device=DEV), torch.randn(T, Hv, device=DEV), torch.randn(B + 2, Hv, Dv, Dk, device=DEV) * 0.1
    weights = torch.randn(Hv, device=DEV) * 0.5, -torch.rand(Hv, device=DEV), torch.rand(Dv, device=DEV) + 0.5
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    slots = list(range(B + 1, 1, -1))
    i32 = dict(dtype=torch.int32, device=DEV)
    none = torch.zeros(T, **i32)

    def run(rows, state):
        batch = F.Batch(tokens=none, positions=none, slots=none.long(), cu_q=torch.tensor(cu, **i32), kv_lens=torch.tensor(lens, **i32), block_table=None, last_idx=None,
                        seq_slots=torch.tensor(slots, device=DEV), max_q_len=max(lens), max_kv_len=max(lens), is_decode=False, page_size=16, h_cu_q=tuple(cu),
                        h_kv_lens=tuple(lens), h_seq_slots=tuple(slots))
        return F.gdn(rows, z, beta, alpha, *weights, state, batch, Hk=Hk, Hv=Hv, Dk=Dk, Dv=Dv, eps=1e-6)

    want_s = state0.clone()
    want = run(qkv, want_s)
    state, rows = state0.clone(), qkv
    if form == "state of a layer among others":
        others = torch.randn(B + 2, 3, Hv, Dv, Dk, device=DEV)
        state = others[:, 1]
        state.copy_(state0)
        kept = others[:, 0].clone()
    elif form == "state off 16 bytes":
        state = torch.zeros(state0.numel() + 1, device=DEV)[1:].view(state0.shape).copy_(state0)
    elif form == "rows off 16 bytes":
        rows = torch.zeros(T * W + 1, device=DEV)[1:].view(T, W).copy_(qkv)
    elif form == "rows of a wider product":
        rows = torch.zeros(T, W + 37, device=DEV)[:, 5:5 + W].copy_(qkv)
    else:
        rows = torch.zeros(2 * T, W, device=DEV)[::2].copy_(qkv)
    got = run(rows, state)
    assert torch.equal(got, want) and torch.equal(state, want_s)
    if form == "state of a layer among others":
        assert torch.equal(others[:, 0], kept)
