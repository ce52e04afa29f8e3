"""Logits of places asked for out of order, twice, or not at all: as many wanted places as tokens are not the tokens in their order."""
import pytest
import torch

from tensorsharp_b200.models import synth
from tensorsharp_b200.models.base import ModelBase
from tensorsharp_b200.runtime.batching import StepEngine

FILES = {"qwen3": synth.write_qwen3, "gemma3": lambda p, **kw: synth.write_gemma(p, arch="gemma3", **kw), "nemotron_h": synth.write_nemotron_h,
         "qwen35": synth.write_qwen35, "gptoss": synth.write_gptoss}
FOLDERS = {"fobolorn": synth.write_fobolorn, "sogulix": synth.write_sogulix, "kegetar": synth.write_kegetar, "lisorax": synth.write_lisorax}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    d, made = tmp_path_factory.mktemp("rows"), {}

    def get(name):
        if name not in made:
            path = str(d / (name + (".gguf" if name in FILES else "")))
            (FILES.get(name) or FOLDERS[name])(path, device="cpu")
            made[name] = ModelBase.create(path, "cpu", max_context=64, max_seqs=4)
        return made[name]
    return get


def every_place(m, portions):
    """Logits of each place of fresh sequences' tokens, asked for one at a time."""
    out = []
    for ids in portions:
        for r in range(len(ids)):
            s = m.new_sequence()
            out.append(m.forward_batch(m.kv.build_batch([s], [ids[:r + 1]]))[0])
            m.free_sequence(s)
    return torch.stack(out)


# Each case: tokens per sequence, wanted places per sequence.  The sums of a place run over other row counts in the two computations: 2e-3 of
# the largest logit, where two places' logits are far apart.
@pytest.mark.parametrize("name", list(FILES) + list(FOLDERS))
@pytest.mark.parametrize("lens,rows", [((3,), [[2, 1, 0]]), ((3,), [[2, 2, 2]]), ((3,), [[1, 0, 2]]), ((1, 1), [[0, 0], []]), ((2, 1), [[1, 1], [0]]), ((2, 2), [[], [1, 0, 1, 0]]),
                                       ((3,), [[0, 1, 2]]), ((1, 1), [[0], [0]])])
def test_logits_come_in_the_order_asked_for(models, monkeypatch, name, lens, rows):
    monkeypatch.setenv("TSB_GATHER_GRAPH", "0")          # packed batches throughout: a step engine's single tokens as well
    m = models(name)
    g = torch.Generator().manual_seed(3)
    portions = [torch.randint(1, min(500, m.cfg.vocab), (n,), generator=g).tolist() for n in lens]
    each = every_place(m, portions)
    at = [sum(lens[:i]) + r for i, want in enumerate(rows) for r in want]
    assert (each[1:] - each[:-1]).abs().amax() > 0.02 * each.abs().max()
    seqs = [m.new_sequence() for _ in lens]
    got = m.forward_batch(m.kv.build_batch(seqs, portions, rows=rows))
    for s in seqs:
        m.free_sequence(s)
    e = StepEngine(m, 4)
    step = e.step([(i, t, r) for i, (t, r) in enumerate(zip(portions, rows))])
    for i in range(len(lens)):
        e.end(i)
    for y in (got, step):
        assert y.shape == each[at].shape
        assert (y - each[at]).abs().max() < 2e-3 * each.abs().max()
