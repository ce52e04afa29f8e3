"""Generation loops: eager token loop, CUDA-graph decode, and the throughput benchmark.

The reference's hot loop is the host token loop of ModelService / Program.RunBenchmark
(TensorSharp.Cli/Program.cs:1515-1607): one native call per token, logits downloaded,
arg-max on the host.  Here a decode step is one CUDA-graph replay that ends with the
sampled ids on the device and the batch bookkeeping (positions, cache lengths, KV slots)
advanced by a kernel, so consecutive steps need no host work at all; the host only reads
ids when a caller wants them.
"""
from __future__ import annotations

import gc
import time
from dataclasses import dataclass
from typing import Callable, Iterable, List, Optional, Sequence

import torch

from ..ops import functional as F
from ..ops.functional import Batch
from .paged_kv import SeqState
from .sampling import SamplingConfig, TokenSampler


def capture_graph(body: Callable[[], None]) -> "torch.cuda.CUDAGraph":
    """Capture ``body`` into a CUDA graph.  Python's cycle collector is kept out of the capture: objects it would free there
    (another model's graphs or events) issue CUDA calls that invalidate it."""
    gc.collect()
    on = gc.isenabled()
    gc.disable()
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            body()
    finally:
        if on:
            gc.enable()
    return graph


class DecodeGraph:
    """Greedy batched decode of ``seqs`` captured as one CUDA graph."""

    def __init__(self, model, seqs: Sequence[SeqState], max_new_tokens: int, use_graph: bool = True, sampling=None):
        """``sampling`` (a SamplingConfig the device sampler supports) replaces the arg-max by a draw
        inside the captured step; penalties see the tokens generated by this object."""
        self.model = model
        self.sampling = sampling
        self.seqs = list(seqs)
        kv = model.kv
        for s in self.seqs:
            kv.reserve(s, s.length + max_new_tokens + 1)
        B = len(self.seqs)
        dev = model.device
        ps = kv.page_size
        width = max(len(s.pages) for s in self.seqs)
        table = torch.zeros((B, width), dtype=torch.int32)
        for i, s in enumerate(self.seqs):
            table[i, :len(s.pages)] = torch.tensor(s.pages, dtype=torch.int32)
        max_len = max(s.length for s in self.seqs) + max_new_tokens + 1
        ring = {}
        if kv.ring:                             # window layers: logical page -> ring page, for every page up to the limit
            ring = dict(slots_w=torch.zeros(B, dtype=torch.int64, device=dev),
                        block_table_w=torch.tensor([kv.wtable_row(s, width) for s in self.seqs], dtype=torch.int32).to(dev))
        self.batch = Batch(**ring,
            tokens=torch.zeros(B, dtype=torch.int32, device=dev),
            positions=torch.zeros(B, dtype=torch.int32, device=dev),
            slots=torch.zeros(B, dtype=torch.int64, device=dev),
            cu_q=torch.arange(B + 1, dtype=torch.int32, device=dev),
            kv_lens=torch.zeros(B, dtype=torch.int32, device=dev),
            block_table=table.to(dev),
            last_idx=torch.arange(B, dtype=torch.int64, device=dev), rows_in_order=True, rows_apart=len(set(map(id, self.seqs))) == B,
            seq_slots=torch.tensor([s.slot for s in self.seqs], dtype=torch.int64, device=dev),
            max_q_len=1, max_kv_len=max_len, is_decode=True, page_size=ps,
            h_cu_q=tuple(range(B + 1)), h_kv_lens=tuple(s.length + 1 for s in self.seqs))
        self.sampled = torch.zeros(B, dtype=torch.int32, device=dev)
        self.ngen = torch.zeros(B, dtype=torch.int32, device=dev)
        self.counts = None
        if sampling is not None and dev.type == "cuda":
            from ..ops import kernels
            if not kernels.device_sampler_supports(sampling):
                raise ValueError("these sampling settings need the host sampler (top_p without top_k, or top_k > 1024)")
            if sampling.has_penalties:
                self.counts = torch.zeros((B, model.cfg.vocab), dtype=torch.int32, device=dev)
            self.seed = sampling.seed if sampling.seed >= 0 else int.from_bytes(__import__("os").urandom(7), "little")
        self.h_tokens = torch.zeros(B, dtype=torch.int32).pin_memory() if dev.type == "cuda" else torch.zeros(B, dtype=torch.int32)
        self.h_sampled = torch.zeros(B, dtype=torch.int32).pin_memory() if dev.type == "cuda" else torch.zeros(B, dtype=torch.int32)
        self.graph: Optional[torch.cuda.CUDAGraph] = None
        self.use_graph = use_graph and dev.type == "cuda"
        self.launches_per_step = 0

    # ------------------------------------------------------------------ state
    def set_tokens(self, tokens: Sequence[int]) -> None:
        """Load the next input token of every sequence and the matching positions / slots."""
        ps = self.batch.page_size
        pos = [s.length for s in self.seqs]
        slots = [s.pages[p // ps] * ps + p % ps for s, p in zip(self.seqs, pos)]
        dev = self.model.device
        self.h_tokens.copy_(torch.tensor(list(tokens), dtype=torch.int32))
        self.batch.tokens.copy_(self.h_tokens, non_blocking=True)
        self.batch.positions.copy_(torch.tensor(pos, dtype=torch.int32), non_blocking=False)
        self.batch.kv_lens.copy_(torch.tensor([p + 1 for p in pos], dtype=torch.int32))
        self.batch.slots.copy_(torch.tensor(slots, dtype=torch.int64))
        if self.batch.slots_w is not None:
            kv = self.model.kv
            self.batch.slots_w.copy_(torch.tensor([kv.wslot(s, p) for s, p in zip(self.seqs, pos)], dtype=torch.int64))

    def _step_body(self) -> None:
        self.batch.cache.clear()
        logits = self.model.forward_batch(self.batch, True)
        self.logits = logits                    # inside a captured graph this buffer is rewritten by every replay
        if self.sampling is not None and self.model.device.type == "cuda":
            from ..ops import kernels
            c = self.sampling
            lg = logits[:, :self.model.cfg.vocab].contiguous()
            kernels.sample(lg, self.ngen, temperature=c.temperature, top_k=c.top_k, top_p=c.top_p, min_p=c.min_p,
                           repetition_penalty=c.repetition_penalty, presence_penalty=c.presence_penalty,
                           frequency_penalty=c.frequency_penalty, seed=self.seed, counts=self.counts, out=self.sampled)
        else:
            self.sampled.copy_(F.argmax(logits))
        if self.model.device.type == "cuda":
            from ..ops import kernels
            kernels.decode_advance(self.sampled, self.batch)
        else:
            self._advance_host()
        b = self.batch
        if b.slots_w is not None:               # the ring's slot of the new position (tensor ops: capturable)
            ps = b.page_size
            page = torch.div(b.positions, ps, rounding_mode="floor").long()
            b.slots_w.copy_(b.block_table_w.gather(1, page.unsqueeze(1)).squeeze(1).long() * ps + (b.positions % ps).long())

    def _advance_host(self) -> None:
        b, ps = self.batch, self.batch.page_size
        b.tokens.copy_(self.sampled)
        b.positions.add_(1)
        b.kv_lens.copy_(b.positions + 1)
        page = (b.positions // ps).long()
        b.slots.copy_(b.block_table.gather(1, page.unsqueeze(1)).squeeze(1).long() * ps + (b.positions % ps).long())
        b.h_kv_lens = tuple(int(x) for x in b.kv_lens.tolist())

    def capture(self) -> None:
        """Warm up once (eagerly, without advancing) and capture the step."""
        if not self.use_graph:
            return
        from ..ops import kernels
        snap = [t.clone() for t in (self.batch.tokens, self.batch.positions, self.batch.kv_lens, self.batch.slots)]
        ring_snap = self.batch.slots_w.clone() if self.batch.slots_w is not None else None
        # the warm-up step below really runs: a K / V row it writes is written again by the first real step, but the
        # recurrent state of linear-attention / SSM layers would have advanced by one token, so it is put back
        state_slots = torch.tensor([s.slot for s in self.seqs], dtype=torch.long, device=self.model.device)
        state_snap = [(t, t[state_slots].clone()) for t in self.model.recurrent_state_tensors()]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            n0 = kernels.LAUNCHES
            self._step_body()
            self.launches_per_step = kernels.LAUNCHES - n0
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        for dst, src in zip((self.batch.tokens, self.batch.positions, self.batch.kv_lens, self.batch.slots), snap):
            dst.copy_(src)
        if ring_snap is not None:
            self.batch.slots_w.copy_(ring_snap)
        for t, saved in state_snap:
            t[state_slots] = saved
        self.ngen.zero_()                       # the warm-up draw is not part of the run
        if self.counts is not None:
            self.counts.zero_()
        self.graph = capture_graph(self._step_body)

    # ------------------------------------------------------------------ stepping
    def step(self) -> torch.Tensor:
        """One decode step for every sequence; returns the sampled ids (device int32 [B])."""
        # the pages reserved at construction and the attention split length fixed at capture both end at
        # ``max_kv_len``; a step beyond it would write into the last reserved page again and attend to a cut context
        if max(s.length for s in self.seqs) + 1 > self.batch.max_kv_len:
            raise RuntimeError(f"DecodeGraph was sized for a context of {self.batch.max_kv_len} tokens; make a new one to go on")
        if self.graph is not None:
            self.graph.replay()
        else:
            self._step_body()
        for s in self.seqs:
            s.length += 1
        return self.sampled

    def step_host(self, tokens: Sequence[int]) -> List[int]:
        """End-to-end step: token ids in from pinned host memory, sampled ids back out."""
        self.h_tokens.copy_(torch.tensor(list(tokens), dtype=torch.int32))
        self.batch.tokens.copy_(self.h_tokens, non_blocking=True)
        out = self.step()
        self.h_sampled.copy_(out, non_blocking=True)
        if self.model.device.type == "cuda":
            torch.cuda.current_stream().synchronize()
        return self.h_sampled.tolist()


class GraphStepper:
    """Single-token steps of one sequence through a captured graph, for hosts that pick the token themselves
    (the server's and the CLI's token loops sample on the host and call ``model.forward([t])``).  An eager step
    costs the host about 20 us per kernel launch, several times what the GPU needs for the step; a replay costs
    one launch.  The graph is captured for a context bucket (a power of two of positions, pages reserved up to
    it) and re-captured when the sequence outgrows the bucket; prefill, truncation and reset happen outside and
    are picked up before the next step (positions, slots and the block table are rewritten when they changed)."""

    MIN_BUCKET = 1024

    def __init__(self, model, seq: SeqState):
        self.model, self.seq = model, seq
        self.dg: Optional[DecodeGraph] = None
        self.bucket = 0
        self.expect_len = -1
        self.pages: List[int] = []

    def _bucket_for(self, length: int) -> int:
        b = self.MIN_BUCKET
        while b < length + 1:
            b *= 2
        return min(b, self.model.max_context)

    def _sync(self, token: int) -> bool:
        """Make the graph's inputs describe the sequence as it is now; False when the context is exhausted."""
        seq, m = self.seq, self.model
        if seq.length + 1 > m.max_context:
            return False
        if self.dg is None or seq.length + 1 > self.bucket:
            bucket = self._bucket_for(seq.length)
            need = (bucket + m.kv.page_size - 1) // m.kv.page_size - len(seq.pages)
            if need > m.kv.free_pages:                      # other sequences hold the pages: stay on the eager path
                return False
            self.bucket = bucket
            self.dg = DecodeGraph(m, [seq], self.bucket - seq.length - 1)
            self.dg.set_tokens([token])
            self.dg.capture()
            self.pages = list(seq.pages)
            self.expect_len = seq.length
            return True
        if seq.length != self.expect_len or seq.pages != self.pages:
            need = (self.bucket + m.kv.page_size - 1) // m.kv.page_size - len(seq.pages)
            if need > m.kv.free_pages:
                return False
            m.kv.reserve(seq, self.bucket)                  # a truncate or reset gave pages back
            table = self.dg.batch.block_table
            row = torch.zeros(table.shape[1], dtype=torch.int32)
            row[:len(seq.pages)] = torch.tensor(seq.pages, dtype=torch.int32)
            table[0].copy_(row)
            self.dg.set_tokens([token])
            self.pages = list(seq.pages)
            self.expect_len = seq.length
        return True

    def step(self, token: int) -> Optional[torch.Tensor]:
        """Append ``token`` and return the next-token logits (a private copy), or None when the caller has to
        take the eager path (context exhausted)."""
        if not self._sync(int(token)):
            return None
        dg = self.dg
        dg.batch.tokens.fill_(int(token))                  # by value: a caller need not wait for one step before it asks for the next
        dg.step()
        self.expect_len = self.seq.length
        return dg.logits[0].clone()


class BatchGraphStepper:
    """Single-token steps of several sequences at once through captured graphs: what ``GraphStepper`` does for one
    sequence, for the merged steps of concurrent requests (runtime/gather.py).  The batch's metadata lives in static
    device tensors that are rewritten before every step (tokens, positions, cache slots, lengths, block-table rows), so
    which sequences take part may change from step to step; one graph is captured per (batch size, context bucket) and
    replayed while the longest sequence fits the bucket.  Pages are reserved one step ahead only.  Without a GPU the
    same static batch runs eagerly, which is how the bookkeeping is tested."""

    MIN_BUCKET = 1024

    def __init__(self, model, max_batch: int):
        self.model, self.max_batch = model, int(max_batch)
        kv = model.kv
        self.width = (model.max_context + kv.page_size - 1) // kv.page_size
        self._state = {}                  # (B, bucket) -> (Batch, graph or None, static logits holder)
        self.replays = 0
        self.captures = 0

    def _bucket_for(self, length: int) -> int:
        b = self.MIN_BUCKET
        while b < length:
            b *= 2
        return min(b, self.model.max_context)

    def _make_batch(self, B: int, bucket: int) -> Batch:
        dev = self.model.device
        return Batch(tokens=torch.zeros(B, dtype=torch.int32, device=dev), positions=torch.zeros(B, dtype=torch.int32, device=dev),
                     slots=torch.zeros(B, dtype=torch.int64, device=dev), cu_q=torch.arange(B + 1, dtype=torch.int32, device=dev),
                     kv_lens=torch.ones(B, dtype=torch.int32, device=dev),
                     block_table=torch.zeros((B, self.width), dtype=torch.int32, device=dev),
                     last_idx=torch.arange(B, dtype=torch.int64, device=dev), rows_in_order=True, rows_apart=True,
                     seq_slots=torch.zeros(B, dtype=torch.int64, device=dev),
                     max_q_len=1, max_kv_len=bucket, is_decode=True, page_size=self.model.kv.page_size,
                     h_cu_q=tuple(range(B + 1)), h_kv_lens=tuple([1] * B))

    def _fill(self, batch: Batch, seqs: Sequence[SeqState], tokens: Sequence[int]) -> None:
        ps = batch.page_size
        B = len(seqs)
        pos = [s.length for s in seqs]
        i32 = torch.tensor([list(map(int, tokens)), pos, [p + 1 for p in pos]], dtype=torch.int32)
        i64 = torch.tensor([[s.pages[p // ps] * ps + p % ps for s, p in zip(seqs, pos)], [s.slot for s in seqs]], dtype=torch.int64)
        table = torch.zeros((B, self.width), dtype=torch.int32)
        for i, s in enumerate(seqs):
            table[i, :len(s.pages)] = torch.tensor(s.pages, dtype=torch.int32)
        dev = self.model.device
        if dev.type == "cuda":
            i32, i64, table = i32.pin_memory(), i64.pin_memory(), table.pin_memory()
        batch.tokens.copy_(i32[0], non_blocking=True)
        batch.positions.copy_(i32[1], non_blocking=True)
        batch.kv_lens.copy_(i32[2], non_blocking=True)
        batch.slots.copy_(i64[0], non_blocking=True)
        batch.seq_slots.copy_(i64[1], non_blocking=True)
        batch.block_table.copy_(table, non_blocking=True)
        batch.h_kv_lens = tuple(p + 1 for p in pos)

    def supports(self) -> bool:
        m = self.model
        return ((m.supports_kv_truncation or m.graphs_with_state) and m.tp_size == 1 and m.pp_size == 1 and not m._pending_embeddings and not m.kv.ring)

    def step(self, seqs: Sequence[SeqState], tokens: Sequence[int]) -> Optional[torch.Tensor]:
        """Append one token to every sequence and return the next-token logits ``[B, vocab...]`` (a private copy);
        None when this step has to take the eager path (too many sequences, context exhausted, no page left)."""
        m, kv = self.model, self.model.kv
        B = len(seqs)
        if B == 0 or B > self.max_batch or getattr(self, "disabled", False) or not self.supports():
            return None
        longest = max(s.length for s in seqs) + 1
        if longest > m.max_context:
            return None
        ps = kv.page_size
        need = sum(max(0, (s.length + 1 + ps - 1) // ps - len(s.pages)) for s in seqs)
        if need > kv.free_pages:
            return None
        for s in seqs:
            kv.reserve(s, s.length + 1)
        bucket = self._bucket_for(longest)
        key = (B, bucket)
        st = self._state.get(key)
        on_gpu = m.device.type == "cuda"
        if st is None:
            batch = self._make_batch(B, bucket)
            self._fill(batch, seqs, tokens)
            holder = {}

            def body():
                batch.cache.clear()
                holder["logits"] = m.forward_batch(batch, True)
            graph = None
            if on_gpu:
                # the warm-up step really runs: it writes the K / V rows that the replay writes again, but it would
                # advance recurrent state by one token, so that is put back
                slots = torch.tensor([s.slot for s in seqs], dtype=torch.long, device=m.device)
                state = [(t, t[slots].clone()) for t in m.recurrent_state_tensors()]
                side = torch.cuda.Stream()
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    body()
                torch.cuda.current_stream().wait_stream(side)
                torch.cuda.synchronize()
                for t, saved in state:
                    t[slots] = saved
                try:
                    graph = capture_graph(body)
                except Exception:
                    # a step that cannot be captured (an operator that synchronises, for one): the merged steps of this
                    # model stay eager from here on; the warm-up above only wrote rows the eager step writes again
                    self.disabled = True
                    torch.cuda.synchronize()
                    return None
                self.captures += 1
            st = self._state[key] = (batch, graph, holder, body)
        batch, graph, holder, body = st
        self._fill(batch, seqs, tokens)
        if graph is not None:
            graph.replay()
            self.replays += 1
        else:
            batch.max_kv_len = longest
            body()
        for s in seqs:
            s.length += 1
        return holder["logits"].clone()


def generate(model, prompt: Sequence[int], max_tokens: int, sampler: Optional[TokenSampler] = None,
             eos_ids: Iterable[int] = (), on_token: Optional[Callable[[int], bool]] = None,
             prefill_chunk: int = 2048) -> List[int]:
    """Single-sequence generation on the model's default sequence (prefix already cached is
    the caller's business: pass only the suffix that still has to be prefilled)."""
    sampler = sampler or TokenSampler(SamplingConfig.greedy())
    eos = set(int(e) for e in eos_ids)
    logits = model.forward_refill(list(prompt), prefill_chunk)
    out: List[int] = []
    for _ in range(max_tokens):
        t = sampler.sample(logits, out)
        if t in eos:
            break
        out.append(t)
        if on_token is not None and on_token(t) is False:
            break
        logits = model.forward([t])
    return out


@dataclass
class BenchResult:
    prefill_tokens: int
    decode_tokens: int
    prefill_ms: float
    decode_ms: float

    @property
    def prefill_tps(self) -> float:
        return self.prefill_tokens / (self.prefill_ms / 1e3) if self.prefill_ms > 0 else 0.0

    @property
    def decode_tps(self) -> float:
        return self.decode_tokens / (self.decode_ms / 1e3) if self.decode_ms > 0 else 0.0

    @property
    def ms_per_token(self) -> float:
        return self.decode_ms / max(1, self.decode_tokens)


def synthetic_prompt(n: int, vocab: int) -> List[int]:
    """The reference benchmark's prompt ids: min(100, vocab-1) + (i % 17) (Program.cs:1515-1607)."""
    base = min(100, vocab - 1)
    return [min(vocab - 1, base + (i % 17)) for i in range(n)]


def run_benchmark(model, prefill: int = 32, decode: int = 64, runs: int = 1, chunked: bool = False,
                  use_graph: bool = True) -> List[BenchResult]:
    """``--benchmark``: per run reset the cache, time one prefill, then ``decode`` greedy
    steps.  Timed with CUDA events on a CUDA device (host clock on the CPU)."""
    cuda = model.device.type == "cuda"
    ids = synthetic_prompt(prefill, model.cfg.vocab)
    results = []
    for _ in range(runs):
        model.reset_kv_cache()
        if cuda:
            torch.cuda.synchronize()
            e0, e1, e2, e3 = (torch.cuda.Event(enable_timing=True) for _ in range(4))
            e0.record()
        t0 = time.perf_counter()
        logits = model.forward_refill(ids) if chunked else model.forward(ids)
        nxt = int(F.argmax(logits.view(1, -1))[0])
        if cuda:
            e1.record()
        t1 = time.perf_counter()
        seq = model._seq()
        if cuda and use_graph and decode > 0:
            dg = DecodeGraph(model, [seq], decode + 1)
            dg.set_tokens([nxt])
            dg.capture()
            torch.cuda.synchronize()
            e3.record()
            for _ in range(decode):
                dg.step()
            e2.record()
            torch.cuda.synchronize()
            pre_ms = e0.elapsed_time(e1)
            dec_ms = e3.elapsed_time(e2)
        else:
            for _ in range(decode):
                logits = model.forward([nxt])
                nxt = int(F.argmax(logits.view(1, -1))[0])
            if cuda:
                e2.record()
                torch.cuda.synchronize()
                pre_ms, dec_ms = e0.elapsed_time(e1), e1.elapsed_time(e2)
            else:
                t2 = time.perf_counter()
                pre_ms, dec_ms = 1e3 * (t1 - t0), 1e3 * (t2 - t1)
        results.append(BenchResult(prefill, decode, pre_ms, dec_ms))
    return results
