"""Fused tensor-parallel exchange (peer-memory mailboxes inside the GEMV and norm kernels) on real
GPUs: equality with the NCCL all-reduce path and with a single GPU, CUDA-graph replay, and the
bounded wait (a flag that nothing sets must end in a status code, not a hang)."""
import json
import os
import socket
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _free_port():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _run_ranks(n, *model_paths, **extra_env):
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", **extra_env)
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}", "--master-addr", "127.0.0.1",
           "--master-port", str(_free_port()), os.path.join(HERE, "tp_worker.py"), *model_paths]
    p = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    lines = [l for l in p.stdout.splitlines() if l.startswith("TPCHECK ")]
    assert p.returncode == 0 and lines, f"rc={p.returncode}\nstdout:\n{p.stdout[-3000:]}\nstderr:\n{p.stderr[-3000:]}"
    assert len(lines) == len(model_paths), p.stdout[-3000:]
    cp = [json.loads(l[8:]) for l in p.stdout.splitlines() if l.startswith("CPCHECK ")]
    assert cp and cp[0]["status"] == 0 and cp[0]["max_err"] < 3e-2, cp          # context-parallel attention
    return [json.loads(l[8:]) for l in lines]


@pytest.fixture(scope="module")
def kv8_model_path(tmp_path_factory):
    """A small Qwen3-shaped model with 8 KV heads so it can be cut 2, 4 and 8 ways."""
    from tensorsharp_b200.models import synth
    p = str(tmp_path_factory.mktemp("tp") / "qwen3_kv8.gguf")
    synth.write_qwen3(p, n_layers=3, hidden=512, n_heads=16, n_kv_heads=8, head_dim=64, ffn=2048, vocab=4096, scheme="Q8_0",
                      device="cpu")
    return p


@pytest.fixture(scope="module")
def moe_model_path(tmp_path_factory):
    """A small GPT-OSS-shaped model (sinks, sliding window, 8 experts top-2, MXFP4 experts) with 8 KV heads."""
    from tensorsharp_b200.models import synth
    p = str(tmp_path_factory.mktemp("tp") / "gptoss_kv8.gguf")
    synth.write_gptoss(p, n_layers=2, hidden=512, n_heads=16, n_kv_heads=8, head_dim=64, n_experts=8, top_k=2, device="cpu")
    return p


@pytest.mark.parametrize("n", [2, 4, 8])
def test_fused_exchange_matches_nccl_and_single_gpu(n, kv8_model_path, moe_model_path):
    """Dense (Qwen3) and mixture-of-experts (GPT-OSS, experts sharded over the ranks) models: the
    in-kernel exchanges give the NCCL path's and a single GPU's logits, for decode-sized batches
    (mailbox exchange, CUDA-graph replay) and for a 300-token prefill (sequence-parallel path)."""
    if torch.cuda.device_count() < n:
        pytest.skip(f"needs {n} GPUs")
    for r in _run_ranks(n, kv8_model_path, moe_model_path):
        check_result(r)


def check_result(r):
    assert r["status"] == 0 and r["exchanges"] > 0, r
    # different summation orders, int8 activations with one scale per 256 (fused decode step) or per 32 (mailbox GEMV)
    # against bf16 activations on the tensor-core GEMM for the 9-token prompt of the NCCL path
    assert r["fused_vs_nccl"] <= 1.5e-2 * max(1.0, r["scale"]), r
    assert r["fused_vs_single"] <= 2e-2 * max(1.0, r["scale"])
    assert r["graph_tokens"] == r["eager_tokens"]
    # sequence-parallel prefill: same logits as the NCCL path and as one GPU (bf16 GEMMs on both sides)
    assert r["seq_status"] == 0
    assert r["seq_vs_nccl"] <= 3e-2 * max(1.0, r["scale"]) and r["seq_next_vs_nccl"] <= 3e-2 * max(1.0, r["scale"])
    # mixture of experts: rows sent only to the ranks that hold their experts give what rows sent to every rank give
    # (the skipped partial sums are zeros)
    if r.get("routed_vs_allgather") is not None:
        assert r["routed_vs_allgather"] <= 1e-5 * max(1.0, r["scale"]), r
    assert r["seq_vs_single"] <= 3e-2 * max(1.0, r["scale"])


def test_wait_without_sender_times_out_with_status():
    """Nothing ever raises the flag: the kernel must give up after its time limit, record which
    rank it waited for and leave the context usable."""
    from tensorsharp_b200.parallel.dist import Communicator
    from tensorsharp_b200.parallel.fused import TpExchange
    dev = torch.device("cuda", 0)
    tpx = TpExchange(Communicator(0, 1, dev), 4, 256)
    h = torch.ones((2, 256), dtype=torch.float32, device=dev)
    w = torch.full((256,), 2.0, dtype=torch.float32, device=dev)
    a = tpx.reduce_norm(h, w, 1e-6)
    assert tpx.status() == 1                      # 1 + rank 0
    torch.cuda.synchronize()
    assert torch.allclose(h, torch.ones_like(h))  # empty mailbox: nothing was added
    assert torch.allclose(a.b.float(), torch.full_like(h, 2.0), atol=2e-2)
    assert float((torch.ones(4, device=dev) * 2).sum()) == 8.0          # context still works
    tpx.close()


def test_single_rank_push_then_reduce_round_trip():
    from tensorsharp_b200.ops import functional as F
    from tensorsharp_b200.gguf.constants import GGMLType
    from tensorsharp_b200.parallel.dist import Communicator
    from tensorsharp_b200.parallel.fused import TpExchange
    from tensorsharp_b200.quant.qweight import QuantWeight
    dev = torch.device("cuda", 0)
    torch.manual_seed(0)
    N, K, T = 512, 1024, 5
    w = QuantWeight.from_float(torch.randn(N, K) * 0.05, GGMLType.Q8_0, dev)
    x = (torch.randn(T, K, device=dev)).to(torch.bfloat16)
    h0 = torch.randn(T, N, device=dev)
    nw = torch.rand(N, device=dev) + 0.5
    tpx = TpExchange(Communicator(0, 1, dev), 16, N)
    for rep in range(6):                           # several epochs: slots and counters wrap
        h = h0.clone()
        tpx.linear_push(F.as_act(x), w)
        a = tpx.reduce_norm(h, nw, 1e-6)
        ref_h = F.linear(F.as_act(x), w, residual=h0.clone())
        ref = F.norm(ref_h.clone(), nw, 1e-6, want_q8=True)
        assert torch.allclose(h, ref_h, atol=1e-4, rtol=1e-4)
        assert torch.allclose(a.b.float(), ref.b.float(), atol=2e-2, rtol=2e-2)
        assert (a.q.int() - ref.q.int()).abs().max() <= 1
        assert torch.allclose(a.ds, ref.ds, atol=1e-3, rtol=1e-3)
    assert tpx.status() == 0
    tpx.close()


@pytest.mark.parametrize("T", [3000, 2900, 300])
def test_sequence_parallel_gemms_of_a_single_rank(T):
    """Gather, gather -> GEMM, GEMM -> reduce-scatter and the reducing norm with one rank, every wait already met by the launch before it.
    3000 tokens: a shard of 3072 rows, the persistent kernel with tiles of 256 rows; 2900: of 2944 and 128; 300: one tile per CTA."""
    from tensorsharp_b200.gguf.constants import GGMLType
    from tensorsharp_b200.ops import reference as ref
    from tensorsharp_b200.parallel.dist import Communicator
    from tensorsharp_b200.parallel.fused import TpSeqParallel
    from tensorsharp_b200.quant.qweight import QuantWeight
    dev = torch.device("cuda", 0)
    torch.manual_seed(1)
    hidden, N, K = 2048, 2568, 328
    sp = TpSeqParallel(Communicator(0, 1, dev), T, hidden)
    wq = QuantWeight.from_float(torch.randn(N, hidden, device=dev) * 0.02, GGMLType.BF16)
    wo = QuantWeight.from_float(torch.randn(hidden, K, device=dev) * 0.05, GGMLType.BF16)
    nw, bias = torch.rand(hidden, device=dev) + 0.5, torch.randn(N, device=dev)
    h = torch.zeros(sp.shard, hidden, device=dev)
    h[:T] = torch.randn(T, hidden, device=dev)
    x = torch.randn(T, K, device=dev).bfloat16()
    rel = lambda a, b: ((a.double() - b.double()).norm() / b.double().norm()).item()               # noqa: E731
    sp.norm_gather(h, nw, 1e-6, False)
    for rep in range(3):                            # counters and accumulators of several exchanges
        a = ref.rmsnorm(h[:T], nw, 1e-6).bfloat16()
        # the gathered rows are rounded to bf16 once, as those are: a value on an edge may fall the other way
        assert rel(sp.gemm_ag(wq, T, bias=bias, out_dtype=torch.float32), a.double() @ wq.dequantize().double().t() + bias) < 2e-3
        want = h[:T].double() + (x.double() @ wo.dequantize().double().t()).float().bfloat16().double()
        sp.gemm_rs(x, wo)
        sp.norm_gather(h, nw, 1e-6, True)
        assert rel(h[:T], want) < 2e-4 and not h[T:].any()
    assert sp.status() == 0
    sp.close()


def test_pipeline_stages_over_nccl(kv8_model_path):
    """Two pipeline stages on two GPUs (NCCL send / recv of the residual stream, token broadcast back)
    generate what one GPU generates."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", TSB_WORKER_MODE="pipeline")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", str(_free_port()), os.path.join(HERE, "tp_worker.py"), kv8_model_path]
    p = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    lines = [l for l in p.stdout.splitlines() if l.startswith("PPCHECK ")]
    assert p.returncode == 0 and lines, f"rc={p.returncode}\nstdout:\n{p.stdout[-3000:]}\nstderr:\n{p.stderr[-3000:]}"
    r = json.loads(lines[0][8:])
    assert r["ranks_agree"] == 2 and r["tokens"] == r["want"], r


def test_context_parallel_prefill_over_peer_memory(kv8_model_path):
    """A prompt dealt to two GPUs (keys and values of the earlier slice pulled from the peer inside the attention
    kernels, caches completed by an all-gather per layer) gives the logits of one GPU, for the prompt, a decode
    step and a second prompt on the same sequence."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", TSB_WORKER_MODE="cp_model")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", str(_free_port()), os.path.join(HERE, "tp_worker.py"), kv8_model_path]
    p = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    lines = [l for l in p.stdout.splitlines() if l.startswith("CPMODEL ")]
    assert p.returncode == 0 and lines, f"rc={p.returncode}\nstdout:\n{p.stdout[-3000:]}\nstderr:\n{p.stderr[-3000:]}"
    r = json.loads(lines[0][8:])
    assert r["status"] == 0 and max(r["rel_err"]) < 5e-2, r


@pytest.mark.parametrize("n", [2, 4, 8])
def test_fused_decode_step_with_tensor_parallel_ranks(n, tmp_path_factory):
    """The one-kernel decode step on N ranks: partial sums of o_proj / down cross NVLink as tagged words written by
    the kernel itself.  Same logits as one GPU (fused step and per-op path), identical on all ranks, no wait ran out,
    and a captured graph reproduces the eager tokens."""
    if torch.cuda.device_count() < n:
        pytest.skip(f"needs {n} GPUs")
    from tensorsharp_b200.models import synth
    path = str(tmp_path_factory.mktemp("mega") / "qwen3_q4km.gguf")
    synth.write_qwen3(path, n_layers=2, hidden=1024, n_heads=32, n_kv_heads=8, head_dim=64, ffn=4096, vocab=8192, scheme="Q4_K_M",
                      device="cpu")
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", TSB_WORKER_MODE="mega")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}", "--master-addr", "127.0.0.1",
           "--master-port", str(_free_port()), os.path.join(HERE, "tp_worker.py"), path]
    p = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    lines = [l for l in p.stdout.splitlines() if l.startswith("MEGACHECK ")]
    assert p.returncode == 0 and lines, f"rc={p.returncode}\nstdout:\n{p.stdout[-3000:]}\nstderr:\n{p.stderr[-3000:]}"
    r = json.loads(lines[0][10:])
    print(r)
    assert r["engaged"] and r["status"] == 0, r
    assert r["spread"] == 0.0, r
    assert r["tp_vs_single_mega"] < 0.05 and r["tp_vs_single_plain"] < 0.12, (r["tp_vs_single_mega"], r["tp_vs_single_plain"], r["mega_vs_plain"])
    assert r["graph_tokens"] == r["eager_tokens"], r


@pytest.mark.parametrize("n", [2, 4])
def test_mailbox_all_reduce_in_gemma_qwen35_nemotron(n, tmp_path_factory):
    """The families without a fused projection + norm pair sum their row-parallel projections (attention output, MLP,
    experts) with the mailbox all-reduce kernel for decode-sized batches: same logits as the NCCL path and as one GPU,
    and the captured decode graph follows the eager tokens."""
    if torch.cuda.device_count() < n:
        pytest.skip(f"needs {n} GPUs")
    from tensorsharp_b200.models import synth
    d = tmp_path_factory.mktemp("tpfam")
    paths = [str(d / "gemma3.gguf"), str(d / "qwen35.gguf"), str(d / "nemotron.gguf")]
    synth.write_gemma(paths[0], arch="gemma3", n_heads=8, n_kv_heads=4, device="cpu")
    synth.write_qwen35(paths[1], device="cpu") if n == 2 else synth.write_qwen35(paths[1], n_heads=8, n_kv_heads=4, device="cpu")
    synth.write_nemotron_h(paths[2], device="cpu")
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", TSB_WORKER_MODE="families")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}", "--master-addr", "127.0.0.1",
           "--master-port", str(_free_port()), os.path.join(HERE, "tp_worker.py"), *paths]
    p = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    res = [json.loads(l[8:]) for l in p.stdout.splitlines() if l.startswith("TPCHECK ")]
    assert p.returncode == 0 and len(res) == 3, f"rc={p.returncode}\nstdout:\n{p.stdout[-3000:]}\nstderr:\n{p.stderr[-3000:]}"
    for r in res:
        assert r["status"] == 0 and r["exchanges"] > 0, r
        # two ranks: a + b in either order, the same bits as NCCL; more ranks: rank order against NCCL's order, then int8
        # re-quantisation of the activations (Gemma's sandwich norms amplify the last bit the most)
        assert r["fused_vs_nccl"] <= (1e-2 if n == 2 else 2.5e-2) * max(1.0, r["scale"]), r
        assert r["fused_vs_single"] <= 3e-2 * max(1.0, r["scale"]), r
        assert r["graph_tokens"] == r["eager_tokens"], r


@pytest.mark.parametrize("n", [2, 4])
def test_sequence_parallel_prefill_through_the_persistent_gemm(n, kv8_model_path, moe_model_path):
    """The same checks with every GEMM forced onto the persistent kernel (TSB_GEMM_PERSISTENT=2; by default only GEMMs
    with more tiles than SMs take it, which these small models never have): all-gather wait in its producer, reduce-
    scatter epilogue with whole-row peer stores, arrival counting per tile."""
    if torch.cuda.device_count() < n:
        pytest.skip(f"needs {n} GPUs")
    for r in _run_ranks(n, kv8_model_path, moe_model_path, TSB_GEMM_PERSISTENT="2"):
        check_result(r)
