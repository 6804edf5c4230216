"""The fused engine on the GPU against the same engine on the CPU reference path."""
import pytest
import torch

from rustral_b200.models.config import preset
from rustral_b200.runtime.fused_gpt import FusedGPTEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["gpt2-test", "llama-test"])
def test_engine_gpu_matches_cpu(name, cuda_status):
    cfg = preset(name)
    cpu = FusedGPTEngine(cfg, "cpu", micro_batch=2, seed=5, max_grad_norm=1.0)
    gpu = FusedGPTEngine(cfg, "cuda", micro_batch=2, seed=5, max_grad_norm=1.0)
    # same starting point: the GPU works on the bf16 rounding of the weights, give the CPU engine the same values
    cpu.params.master.copy_(gpu.params.lowp.float().cpu())
    cpu.params.sync_lowp()
    g = torch.Generator().manual_seed(2)
    ids = torch.randint(0, cfg.vocab_size, (4, cfg.seq_len), generator=g)
    tg = torch.randint(0, cfg.vocab_size, (4, cfg.seq_len), generator=g)
    lc = cpu.train_step(ids, tg, do_step=False)
    lg = gpu.train_step(ids.cuda(), tg.cuda(), do_step=False)
    assert abs(float(lc) - float(lg)) < 2e-2, (float(lc), float(lg))
    gc, gg = cpu.params.grad, gpu.params.grad.cpu()
    for s in cpu.params.specs:
        a, b = gc[s.offset:s.offset + s.numel], gg[s.offset:s.offset + s.numel]
        rel = (a - b).norm() / (a.norm() + 1e-8)
        assert rel < 6e-2, f"{s.name}: relative gradient error {rel:.3g}"
    # a few optimizer steps keep the two trajectories together
    for _ in range(3):
        lc = cpu.train_step(ids, tg)
        lg = gpu.train_step(ids.cuda(), tg.cuda())
    assert abs(float(lc) - float(lg)) < 5e-2, (float(lc), float(lg))


def test_trainer_public_api_loss_decreases(cuda_status):
    from rustral_b200.runtime.lm_trainer import LMTrainer, TrainConfig
    cfg = preset("gpt2-test")
    tr = LMTrainer(cfg, TrainConfig(global_batch=8, micro_batch=4, lr=1e-3), torch.device("cuda"))
    tokens = torch.randint(0, cfg.vocab_size, (8, cfg.seq_len + 1), dtype=torch.int64).pin_memory()
    losses = [tr.step(tokens) for _ in range(8)]
    assert losses[-1] < losses[0] - 0.5, losses


@pytest.mark.parametrize("name", ["gpt2-test", "llama-test"])
def test_weight_gradients_beside_the_chain_are_those_in_line(name, cuda_status):
    """The same kernels on the same operands on another stream: equal bits, in line for the eager calls (the first two of a shape) and replayed, with
    two micro-batches, from a stream that is not the default one, while freed memory is handed out again and overwritten."""
    cfg = preset(name)
    g = torch.Generator().manual_seed(3)
    grads = []
    for beside in (False, True):
        e = FusedGPTEngine(cfg, "cuda", micro_batch=2, seed=5, max_grad_norm=1.0)
        assert e._beside(2 * cfg.seq_len) is not None
        if not beside:
            e._beside = lambda tokens: None
        g.manual_seed(3)
        out = []
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(5):
                ids, tg = (torch.randint(0, cfg.vocab_size, (4, cfg.seq_len), generator=g).cuda() for _ in range(2))
                e.train_step(ids, tg, do_step=False)
                junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 10, 1 << 14, 1 << 18)]  # noqa: F841
                out.append(e.params.grad.clone())
        torch.cuda.synchronize()
        grads.append(torch.stack(out))
    assert torch.equal(grads[0], grads[1])


def test_split_weight_gradients_and_joins_beside_the_chain(monkeypatch, cuda_status):
    """Enough tokens for split contractions, whose slabs and column sums then lie on the other stream, and limits on what is held that make the main stream
    wait after every gradient, after a few and not before the end: equal bits."""
    from rustral_b200 import _native as N
    from rustral_b200.models.config import GPTConfig
    from rustral_b200.ops import matmul
    from rustral_b200.runtime import fused_gpt
    cfg = GPTConfig(vocab_size=1000, seq_len=512, n_layer=3, n_head=6, n_kv_head=6, d_model=384, ffn_dim=1536, arch="gpt2")
    T = 4 * cfg.seq_len
    a = N.RbGemmArgs()
    a.M, a.N, a.K, a.a_mn_major, a.b_mn_major, a.out_f32, a.alpha, a.col_sum = 384, 384, T, 1, 1, 1, 1.0, 256
    assert N.kernels().rb_gemm_workspace(a, matmul.WORKSPACE_BYTES) > 0
    g = torch.Generator().manual_seed(4)
    batches = [[torch.randint(0, cfg.vocab_size, (4, cfg.seq_len), generator=g).cuda() for _ in range(2)] for _ in range(5)]
    grads = []
    for limit in (None, 1, 8 << 20, 1 << 40):
        e = FusedGPTEngine(cfg, "cuda", micro_batch=4, seed=5, max_grad_norm=1.0)
        if limit is None:
            e._beside = lambda tokens: None
        else:
            monkeypatch.setattr(fused_gpt._Beside, "MOST_HELD", limit)
        out = []
        for ids, tg in batches:
            e.train_step(ids, tg, do_step=False)
            out.append(e.params.grad.clone())
        grads.append(torch.stack(out))
    assert all(torch.equal(grads[0], x) for x in grads[1:])
