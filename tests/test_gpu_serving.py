"""Serving on the GPU: greedy tokens from the paged engine against the CPU reference engine on the same weights."""
import pytest
import torch

from rustral_b200.models.config import preset
from rustral_b200.runtime.fused_gpt import FlatParams
from rustral_b200.serve import ModelRunner, ServingEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["gpt2-test", "llama-test"])
def test_gpu_engine_logits_match_cpu(name, cuda_status):
    cfg = preset(name)
    gpu = ModelRunner(cfg, device="cuda", num_blocks=64, seed=4)
    cpu = ModelRunner(cfg, device="cpu", num_blocks=64, seed=4)
    cpu.params.master.copy_(gpu.params.lowp.float().cpu())
    cpu.params.sync_lowp()
    g = torch.Generator().manual_seed(0)
    prompt = torch.randint(0, cfg.vocab_size, (37,), generator=g).tolist()
    for r in (gpu, cpu):
        assert r.cache.allocate(1, len(prompt) + 4)
    lg, lc = gpu.prefill(1, prompt), cpu.prefill(1, prompt)
    assert (lg.float().cpu() - lc).abs().max() < 0.05 * lc.abs().max() + 0.02
    tok = int(lc[:cfg.vocab_size].argmax())
    for step in range(3):
        n = len(prompt) + step + 1
        dg, dc = gpu.decode([1], [tok], [n]), cpu.decode([1], [tok], [n])
        assert (dg.float().cpu() - dc).abs().max() < 0.05 * dc.abs().max() + 0.02
        tok = int(dc[0, :cfg.vocab_size].argmax())


def test_gpu_engine_continuous_batching_completes(cuda_status):
    cfg = preset("llama-test")
    eng = ServingEngine(ModelRunner(cfg, device="cuda", num_blocks=128), max_batch_size=8)
    g = torch.Generator().manual_seed(1)
    ids = [eng.submit(torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist(), 8) for n in (3, 30, 64, 17, 5)]
    done = eng.run_to_completion()
    assert len(done) == 5 and all(len(r.generated) == 8 for r in done)
    assert eng.runner.cache.free_blocks == 128


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
@pytest.mark.parametrize("transport", ["peer", "nvls"])
def test_tensor_parallel_serving_matches_single_gpu(transport):
    """`nvls`: the per-layer all-reduces are summed inside the NVSwitch (multimem.ld_reduce); all ranks must still hold
    bit-identical logits, or their samplers would part ways."""
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ)
    env["TP_TRANSPORT"] = transport
    if transport == "peer":
        env["NCCL_NVLS_ENABLE"] = "0"
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", "29681" if transport == "peer" else "29683", os.path.join(root, "tests", "mp_serve_worker.py")]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600, env=env, cwd=root)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    out = json.loads([l for l in res.stdout.splitlines() if l.startswith("{")][-1])
    assert out["status_max"] == 0 and out["ranks_identical"] and out["transport"] == transport
    assert out["prefill_rel_err"] < 3e-2, out
    # greedy decoding of random-init logits can flip on near ties; the first tokens must agree
    assert out["tokens_ref"][:4] == out["tokens_tp"][:4], out


def test_steps_keep_their_host_memory(cuda_status):
    """Steps that are issued one behind another share two page-locked blocks, whatever their batch size, and what they copy is theirs: a
    block is not written again before its copy has been made."""
    cfg = preset("llama-test")
    r = ModelRunner(cfg, device="cuda", num_blocks=128, seed=3)
    for i in range(5):
        assert r.cache.allocate(i, 40)
    prompts = torch.arange(5 * 8).view(5, 8).tolist()

    def steps():
        got = {}
        for B in (1, 3, 5):
            for n in (1, 8, 20):
                got[B, n] = r.decode(list(range(B)), [7 * n + i for i in range(B)], [n] * B).clone()
        got["prompts"] = torch.stack(r.step_mixed([(i, t, 20, True) for i, t in enumerate(prompts)], [], [], [])[0])
        return got

    steps()                                                    # graphs are captured, every slot that is seen below is written
    want = steps()
    torch.cuda.synchronize()
    before = torch.cuda.host_memory_stats()["num_host_alloc"]
    rounds = []
    for _ in range(30):
        torch.cuda._sleep(200000)                              # the copies below wait in the stream
        rounds.append(steps())
    assert len(r._memory.free) <= 2
    assert torch.cuda.host_memory_stats()["num_host_alloc"] == before
    for got in rounds:
        for key, logits in want.items():
            assert torch.equal(got[key], logits), key


@pytest.mark.parametrize("H,G,D,lens", [(4, 2, 64, [(1, 1), (129, 129)]), (8, 8, 128, [(257, 600), (128, 128), (33, 2000), (256, 256)]),
                                        (6, 2, 64, [(40 * i + 1, 60 * i + 1) for i in range(11)])])
def test_portions_in_one_launch_are_those_alone(H, G, D, lens, cuda_status):
    """Portions (queries, keys) of several sequences, whole and later ones, more than fit one launch: the same bits as a launch each, and nothing of the
    rows between and behind them (NaN) enters."""
    from rustral_b200 import _native as N
    from rustral_b200.ops import attention as A
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    parts, alone = [], []
    for L, S in lens:
        q = torch.full((L + 3, (H + 2 * G) * D), float("nan"), device="cuda").bfloat16()
        kv = torch.full((S + 3, 2 * G * D), float("nan"), device="cuda").bfloat16()
        q[:L], kv[:S] = torch.randn(L, q.shape[1], device="cuda", generator=g).bfloat16(), torch.randn(S, kv.shape[1], device="cuda", generator=g).bfloat16()
        view = (q[:L, :H * D].view(1, L, H, D), kv[:S, :G * D].view(1, S, G, D), kv[:S, G * D:].view(1, S, G, D))
        parts.append((*view, torch.zeros(1, L, H, D, device="cuda").bfloat16()))
        alone.append(A.prompt_attention(*view, 0.2, torch.zeros(1, L, H, D, device="cuda").bfloat16()))
    before = N.launch_count
    A.prompt_attention_many(parts, 0.2)
    assert N.launch_count - before == -(-len(parts) // 8)
    assert all(torch.equal(p[3], o) and torch.isfinite(o).all() for p, o in zip(parts, alone))
