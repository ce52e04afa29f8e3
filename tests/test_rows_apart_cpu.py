"""Batches say whether a sequence is in them twice; decode attention reads ahead of the launch before it only where none is, and only where it is told to."""
import ctypes as C

import pytest
import torch

from tensorsharp_b200.models import synth
from tensorsharp_b200.models.base import ModelBase
from tensorsharp_b200.ops import functional as F
from tensorsharp_b200.ops import kernels
from tensorsharp_b200.runtime.engine import BatchGraphStepper, DecodeGraph


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("rows") / "m.gguf")
    synth.write_qwen3(path, device="cpu")
    return ModelBase.create(path, "cpu", max_context=64, max_seqs=4)


def test_batches_that_hold_a_sequence_twice(model):
    s, t = model.new_sequence(), model.new_sequence()
    assert model.kv.build_batch([s, t], [[1], [2]]).rows_apart
    twice = model.kv.build_batch([s, t, s], [[1], [2], [3]])
    assert twice.is_decode and not twice.rows_apart
    assert DecodeGraph(model, [s, t], 4).batch.rows_apart and BatchGraphStepper(model, 2)._make_batch(2, 64).rows_apart
    for x in (s, t):
        model.free_sequence(x)


@pytest.mark.parametrize("apart", [False, True])
@pytest.mark.parametrize("told", [None, False, True])
@pytest.mark.parametrize("as_act", [False, True])
def test_who_reads_ahead(monkeypatch, apart, told, as_act):
    """What the library gets, without a GPU: the arguments of the call."""
    seen = []

    class Lib:
        def tsb_attn_decode(self, args, stream):
            seen.append(args._obj.ahead)
            return 0

        def tsb_attn_decode_is_one_launch(self, args):
            return 0
    monkeypatch.setattr(kernels, "_lib", lambda: Lib())
    monkeypatch.setattr(kernels, "_stream", lambda: C.c_void_p(0))

    class OnDevice(torch.Tensor):
        is_cuda = True
    q = torch.zeros(2, 4, 64, dtype=torch.bfloat16).as_subclass(OnDevice)
    cache = torch.zeros(128, 2, 64, dtype=torch.bfloat16)
    z = torch.zeros(2, dtype=torch.int32)
    batch = F.Batch(tokens=z, positions=z, slots=z.long(), cu_q=torch.arange(3, dtype=torch.int32), kv_lens=z + 5, block_table=z.view(2, 1), last_idx=z.long(),
                    seq_slots=z.long(), max_q_len=1, max_kv_len=5, is_decode=True, page_size=64, h_cu_q=(0, 1, 2), h_kv_lens=(5, 5), rows_apart=apart)
    F.attention(q, cache, cache, batch, scale=0.1, Hq=4, Hkv=2, Dh=64, as_act=as_act, **({} if told is None else dict(ahead=told)))
    kernels.attn_decode(q, cache, cache, batch.block_table, batch.kv_lens, scale=0.1, Hq=4, Hkv=2, Dh=64, page_size=64, splits=1)
    assert seen == [int(bool(told) and apart), 0]


@pytest.mark.skipif(not kernels.native.available(), reason="the kernel library is not built here")
@pytest.mark.parametrize("kw,one", [(dict(), True), (dict(splits=2), False), (dict(page_size=24), False), (dict(Dh=256, Dv=256), False), (dict(gate=64), False),
                                    (dict(k_ld=1024), False), (dict(plan=64, parts=9, each=1), False)])
def test_launches_of_a_step(kw, one):
    """The launch count asks the library, by a host function that follows no pointer."""
    a = kernels.AttnArgs()
    for k, v in {**dict(B=2, Hq=8, Hkv=2, Dh=128, Dv=128, page_size=64, splits=1), **kw}.items():
        setattr(a, k, v)
    assert bool(kernels._lib().tsb_attn_decode_is_one_launch(C.byref(a))) is one
