"""Performance cases of the framework's main paths, through its public entry points.

Five kinds of work, each over the range of sizes that users of the framework give it:

* "train":   `LMTrainer.step` of GPT-2 style and Llama style decoders (forward, backward, clipping, AdamW, token ids from pinned host
             memory, loss back on the host);
* "decode":  `ModelRunner.decode`, one new token for every sequence of a batch against the paged cache;
* "prompt":  `ModelRunner.step_mixed`, prompts (whole ones and later portions) beside sequences that decode;
* "experts": forward and backward of the routed expert layer (`ops.moe.moe_mlp`);
* "encoder": forward and backward of `nn` encoder layers over padded batches.

`listed` names the standing cases, `draw` gives more of the same ranges, `exact` restates each in 64 bits with plain tensor operations.
"""
from __future__ import annotations

import math
import random

import torch

from rustral_b200.core import ForwardCtx
from rustral_b200.core.backend import B200Backend
from rustral_b200.models.config import GPTConfig
from rustral_b200.nn.attention import KeyPaddingMask
from rustral_b200.nn.transformer import TransformerEncoderConfig, TransformerEncoderLayer
from rustral_b200.ops.moe import moe_mlp
from rustral_b200.runtime.lm_trainer import LMTrainer, TrainConfig
from rustral_b200.serve.model_runner import ModelRunner
from rustral_b200.serve.weights import InferenceWeights

GPT2_SMALL = dict(arch="gpt2", layers=12, d=768, heads=12, kv=12, ffn=3072, vocab=50257)
WIDE = dict(arch="llama", layers=4, d=4096, heads=32, kv=8, ffn=14336, vocab=65536)          # layers of the 8B decoder
MIDDLE = dict(arch="llama", layers=8, d=2048, heads=16, kv=4, ffn=8192, vocab=32768)
HEADS64 = dict(arch="llama", layers=8, d=2048, heads=32, kv=8, ffn=8192, vocab=32768)


def listed() -> list:
    return [
        # one user of a small model: every launch and every gap between launches counts
        dict(name="decode_one_gpt2", kind="decode", **GPT2_SMALL, batch=1, low=300, high=300),
        # one user of a larger model: the weights are read once per token
        dict(name="decode_one_llama", kind="decode", **MIDDLE, batch=1, low=2047, high=2047),
        # a busy server: a full batch with contexts of all lengths
        dict(name="decode_64_ragged", kind="decode", **MIDDLE, batch=64, low=100, high=4000),
        # layers of the 8B decoder under the prompt and output lengths of the serving workload
        dict(name="decode_24_wide", kind="decode", **WIDE, batch=24, low=128, high=2560),
        # one long prompt
        dict(name="prompt_8192_wide", kind="prompt", **WIDE, prompts=1, short=8192, long=8192, resumed=False, batch=0, low=0, high=0),
        # continuous batching: portions of several prompts of odd lengths, one of them a later portion, beside decoding sequences
        dict(name="prompt_mixed", kind="prompt", **HEADS64, prompts=4, short=129, long=1500, resumed=True, batch=21, low=64, high=2000),
        # the headline training configuration, one micro-batch and the optimizer
        dict(name="train_gpt2_small", kind="train", **GPT2_SMALL, seq=1024, batch=32, micro=32),
        # the smallest training step, as in tests and examples
        dict(name="train_gpt2_tiny", kind="train", arch="gpt2", layers=2, d=256, heads=4, kv=4, ffn=1024, vocab=1000, seq=128, batch=8,
             micro=8),
        # Llama style layers with grouped heads of 128, two micro-batches
        dict(name="train_llama", kind="train", arch="llama", layers=4, d=2048, heads=16, kv=4, ffn=8192, vocab=32768, seq=2048, batch=4,
             micro=2),
        # a sequence length and vocabulary that fit no tile
        dict(name="train_odd", kind="train", arch="gpt2", layers=6, d=384, heads=6, kv=6, ffn=1536, vocab=5003, seq=333, batch=6, micro=6),
        # one layer of the mixture-of-experts decoder over one sequence of 2048 tokens and a part of a second
        dict(name="experts_train", kind="experts", tokens=3000, d=2048, experts=8, top=2, ffn=8192, act="swiglu"),
        # fine-tuning of an encoder on padded sentences
        dict(name="encoder_train", kind="encoder", layers=2, d=768, heads=12, ffn=3072, batch=16, seq=384),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("train", "decode", "decode", "prompt", "experts", "encoder"))
    if kind == "train":
        if rng.random() < 0.5:
            heads = rng.choice((4, 6, 8, 12))
            m = dict(arch="gpt2", layers=rng.randint(2, 12), d=64 * heads, heads=heads, kv=heads, ffn=256 * heads, vocab=_log(rng, 1000, 50257))
        else:
            kv, size = rng.choice((2, 4)), rng.choice((64, 128))
            m = dict(arch="llama", layers=rng.randint(2, 4), d=4 * kv * size, heads=4 * kv, kv=kv, ffn=256 * rng.randint(2 * kv, 8 * kv),
                     vocab=_log(rng, 1000, 32768))
        seq = _log(rng, 100, 2048)
        most = 32768 if m["arch"] == "gpt2" else 8192
        micro = max(1, min(32, _log(rng, 1000, most) // seq))
        return dict(kind=kind, **m, seq=seq, batch=2 * micro if 2 * micro * seq <= most and rng.random() < 0.5 else micro, micro=micro)
    if kind in ("decode", "prompt"):
        m = dict(rng.choice((GPT2_SMALL, WIDE, MIDDLE, HEADS64)))
        m["layers"] = rng.randint(2, m["layers"])
        most = 1024 if m["arch"] == "gpt2" else 4000
        if kind == "decode":
            low = _log(rng, 1, most)
            return dict(kind=kind, **m, batch=_log(rng, 1, 64), low=low, high=rng.randint(low, most))
        prompts = rng.randint(1, 4)
        short = _log(rng, 16, most // 4)
        batch = rng.choice((0, _log(rng, 1, 48)))
        return dict(kind=kind, **m, prompts=prompts, short=short, long=rng.randint(short, most // 2), resumed=rng.random() < 0.3, batch=batch,
                    low=min(batch, 16), high=rng.randint(64, most) if batch else 0)
    if kind == "experts":
        return dict(kind=kind, tokens=_log(rng, 100, 4096), d=rng.choice((1024, 2048)), experts=rng.choice((8, 16)), top=rng.choice((1, 2)),
                    ffn=256 * rng.randint(4, 16), act=rng.choice(("swiglu", "gelu")))
    heads = rng.choice((4, 8, 12, 16))
    return dict(kind=kind, layers=rng.randint(1, 3), d=64 * heads, heads=heads, ffn=256 * heads, batch=_log(rng, 1, 32), seq=_log(rng, 30, 512))


# ---- sizes ---------------------------------------------------------------------------------------------------------------------
def _config(c) -> GPTConfig:
    train = c["kind"] == "train"
    # a served model takes any position up to its configured length; GPT-2 has a table of 1024
    seq = c["seq"] if train else 1024 if c["arch"] == "gpt2" else 16384
    return GPTConfig(vocab_size=c["vocab"], seq_len=seq, n_layer=c["layers"], n_head=c["heads"], n_kv_head=c["kv"], d_model=c["d"],
                     ffn_dim=c["ffn"], arch=c["arch"])


def _between(count, low, high, salt) -> list:
    """`count` lengths from low to high: a property of the case, not of its seed."""
    if count == 1:
        return [high]
    r = random.Random(salt)
    return [low, high] + [r.randint(low, high) for _ in range(count - 2)]


def _decoding(c) -> list:
    return _between(c["batch"], c["low"], c["high"], 1) if c["batch"] else []


def _portions(c) -> list:
    """(first position, tokens) of every prompt portion; with `resumed` the last one follows as many tokens as it has."""
    n = _between(c["prompts"], c["short"], c["long"], 2)
    at = [0] * len(n)
    if c["resumed"]:
        at[-1] = n[-1]
    return list(zip(at, n))


def _padded(c) -> list:
    return _between(c["batch"], max(1, c["seq"] // 8), c["seq"], 3)


def work(c) -> dict:
    """Each input read once, each output written once; matrix products and attention of the positions that are seen."""
    if c["kind"] == "experts":
        gates = 2 if c["act"] == "swiglu" else 1
        weights = c["experts"] * c["d"] * c["ffn"] * (gates + 1)
        flops = 6.0 * c["tokens"] * c["top"] * c["d"] * c["ffn"] * (gates + 1)
        return dict(bytes=2.0 * (2 * weights + 4 * c["tokens"] * c["d"]), flops=flops)
    if c["kind"] == "encoder":
        T, layer = c["batch"] * c["seq"], 4 * c["d"] ** 2 + 2 * c["d"] * c["ffn"]
        flops = c["layers"] * (6.0 * T * layer + 12.0 * c["d"] * c["seq"] * sum(_padded(c)))
        return dict(bytes=2.0 * (2 * c["layers"] * layer + 4 * T * c["d"]), flops=flops)
    cfg = _config(c)
    d, hd = c["d"], cfg.head_dim
    layer = cfg.qkv_dim * d + d * d + (2 if c["arch"] == "gpt2" else 3) * d * c["ffn"]
    if c["kind"] == "train":
        T = c["batch"] * c["seq"]
        # fp32 master weights and both moments are read and written; the fp32 gradient and the bf16 copy are results
        return dict(bytes=cfg.num_parameters() * (2.0 + 24 + 4 + 2) + 8.0 * T, flops=float(T) * cfg.flops_per_token())
    decoding, portions = _decoding(c), _portions(c) if c["kind"] == "prompt" else []
    rows = len(decoding) + sum(n for _, n in portions)
    heads = len(decoding) + len(portions)
    seen = sum(decoding) + sum(at * n + n * (n + 1) // 2 for at, n in portions)
    cached = sum(decoding) + sum(at + n for at, n in portions)
    flops = c["layers"] * (2.0 * rows * layer + 4.0 * seen * d) + 2.0 * heads * d * cfg.vocab_padded
    weights = c["layers"] * layer + cfg.vocab_padded * d
    return dict(bytes=2.0 * (weights + c["layers"] * 2 * c["kv"] * hd * cached + rows * d + heads * cfg.vocab_padded), flops=flops)


def tolerance(c) -> dict:
    """bf16 activations.  Distance of one pass from 64-bit arithmetic: 0.007 to 0.019 behind 2 to 12 decoder layers (logits, cached keys
    of the last layers, gradients), 0.004 to 0.007 behind one or two layers; about four times that, and 0.03 at most."""
    return {"rel": 0.02 if c["kind"] in ("experts", "encoder") else 0.03}


# ---- what a program holds before the call -----------------------------------------------------------------------------------------
def prepare(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *shape, std=1.0: torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, std, generator=g).bfloat16()  # noqa: E731
    if c["kind"] == "experts":
        f1 = c["ffn"] * (2 if c["act"] == "swiglu" else 1)
        s = dict(x=rand(c["tokens"], c["d"]), router=rand(c["experts"], c["d"], std=0.02), w1=rand(c["experts"], f1, c["d"], std=0.02),
                 w2=rand(c["experts"], c["d"], c["ffn"], std=0.02), dy=rand(c["tokens"], c["d"], std=0.01))
        for k in ("x", "router", "w1", "w2"):
            s[k].requires_grad_()
        return dict(case=c, **s)
    if c["kind"] == "encoder":
        backend = B200Backend()
        layers = [TransformerEncoderLayer.new(backend, TransformerEncoderConfig(c["d"], c["heads"], c["layers"], c["ffn"], dropout=0.0),
                                              seed + 100 * i) for i in range(c["layers"])]
        params = [p.tensor for layer in layers for p in layer.parameters()]
        for p in params:
            p.requires_grad_()
        return dict(case=c, layers=layers, params=params, x=rand(c["batch"], c["seq"], c["d"]).requires_grad_(),
                    dy=rand(c["batch"], c["seq"], c["d"], std=0.01), ctx=ForwardCtx.train(backend),
                    mask=KeyPaddingMask(torch.tensor(_padded(c), dtype=torch.int32, device="cuda")))
    cfg = _config(c)
    if c["kind"] == "train":
        trainer = LMTrainer(cfg, TrainConfig(global_batch=c["batch"], micro_batch=c["micro"], seed=seed), "cuda")
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g, device="cuda")
        return dict(case=c, trainer=trainer, tokens=ids.cpu().pin_memory())
    decoding, portions = _decoding(c), _portions(c) if c["kind"] == "prompt" else []
    lengths = decoding + [at + n for at, n in portions]
    weights = InferenceWeights.random_llama(cfg, "cuda", seed=seed) if c["arch"] == "llama" else None
    runner = ModelRunner(cfg, params=weights, device="cuda", num_blocks=sum(-(-n // 16) for n in lengths) + 8, block_size=16, seed=seed)
    # sequences grow side by side, so their pages lie interleaved as in a running server
    for end in range(256, max(lengths) + 256, 256):
        for i, n in enumerate(lengths):
            assert runner.cache.allocate(i, min(n, end))
    for l in range(c["layers"]):
        runner.cache.k[l].normal_(0.0, 0.9, generator=g)
        runner.cache.v[l].normal_(0.0, 0.9, generator=g)
    ids = torch.randint(0, c["vocab"], (len(decoding) + sum(n for _, n in portions),), generator=g, device="cuda").tolist()
    chunks, r = [], len(decoding)
    for i, (at, n) in enumerate(portions):
        chunks.append((len(decoding) + i, ids[r:r + n], at, True))
        r += n
    return dict(case=c, runner=runner, chunks=chunks, ids=list(range(len(decoding))), tokens=ids[:len(decoding)], lengths=decoding)


def _without_key_bias(s, grads) -> list:
    """A softmax does not change when all its scores move together, so the gradient of the keys' bias is zero up to rounding: it is
    computed with the others, and nothing can be said about its digits."""
    names = ["x"] + [n for layer in s["layers"] for n, _ in layer.named_parameters()]
    return [g for n, g in zip(names, grads) if n != "self_attn.k_proj.bias"]


# ---- one pass ------------------------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["case"]["kind"]
    if kind == "experts":
        y, aux = moe_mlp(s["x"], s["router"], s["w1"], s["w2"], s["case"]["top"], s["case"]["act"], True)
        grads = torch.autograd.grad((y, aux * 0.01), (s["x"], s["router"], s["w1"], s["w2"]), (s["dy"], torch.ones_like(aux)))
        return dict(y=y, aux=aux, grads=grads)
    if kind == "encoder":
        y = s["x"]
        for layer in s["layers"]:
            y = layer.forward(y, s["ctx"], s["mask"])
        grads = torch.autograd.grad(y, [s["x"], *s["params"]], s["dy"])
        return dict(y=y, grads=_without_key_bias(s, grads))
    if kind == "train":
        t = s["trainer"]
        loss = t.step(s["tokens"])
        return dict(loss=loss, grads=t.engine.params.grad, weights=t.engine.params.master)
    r = s["runner"]
    if kind == "decode":
        return dict(logits=r.decode(s["ids"], s["tokens"], s["lengths"]), k=r.cache.k, v=r.cache.v)
    first, decoded = r.step_mixed(s["chunks"], s["ids"], s["tokens"], s["lengths"])
    return dict(first=first, decoded=decoded, k=r.cache.k, v=r.cache.v)


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------------
def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _rotate(x, pos, theta):
    """x [rows, heads, size]: number i turns with number i + size / 2."""
    half = x.shape[-1] // 2
    a = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    cos, sin = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def _attend(q, k, v, causal, real=None):
    """q [rows, H, D], k and v [keys, G, D]; the rows are the last of the keys' positions.  `real`: keys that are no padding."""
    H, G = q.shape[1], k.shape[1]
    hidden = torch.ones(q.shape[0], k.shape[0], dtype=torch.bool, device=q.device)
    hidden = hidden.triu(k.shape[0] - q.shape[0] + 1) if causal else ~hidden
    if real is not None:
        hidden = hidden | (torch.arange(k.shape[0], device=q.device) >= real)[None]
    out = []
    for h in range(H):
        kk, vv = k[:, h * G // H], v[:, h * G // H]
        score = (q[:, h] @ kk.T / math.sqrt(q.shape[2])).masked_fill(hidden, -math.inf)
        out.append(torch.softmax(score, -1) @ vv)
    return torch.stack(out, 1)


def _decoder(cfg, w, ids, pos, attend):
    """The stream behind the last norm; w: name -> weights in 64 bits, attend(layer, q, k, v) -> [rows, heads * size]."""
    rms, H, G, D = cfg.arch == "llama", cfg.n_head, cfg.n_kv_head, cfg.head_dim

    def norm(x, name):
        if rms:
            return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + cfg.norm_eps) * w(name + ".weight")
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w(name + ".weight"), w(name + ".bias"), cfg.norm_eps)

    def product(x, name):
        y = x @ w(name + ".weight").T
        return y if rms else y + w(name + ".bias")

    x = w("tok_embed.embed")[ids]
    if not rms:
        x = x + w("pos_embed.embed")[pos]
    for l in range(cfg.n_layer):
        p = f"layers.{l}."
        q, k, v = product(norm(x, p + "ln1"), p + "attn.wqkv").split((H * D, G * D, G * D), -1)
        q, k, v = q.reshape(-1, H, D), k.reshape(-1, G, D), v.reshape(-1, G, D)
        if rms:
            q, k = _rotate(q, pos, cfg.rope_theta), _rotate(k, pos, cfg.rope_theta)
        x = x + product(attend(l, q, k, v).reshape(x.shape[0], H * D), p + "attn.wo")
        h = norm(x, p + "ln2")
        if rms:
            gate, up = product(h, p + "ffn.gate_up").chunk(2, -1)
            x = x + product(torch.nn.functional.silu(gate) * up, p + "ffn.down")
        else:
            x = x + product(_gelu(product(h, p + "ffn.fc1")), p + "ffn.fc2")
    return norm(x, "final_norm")


def _head_name(cfg) -> str:
    return "tok_embed.embed" if cfg.tie_embeddings else "head.weight"


def _exact_train(c, s):
    t = s["trainer"]
    cfg, P, tc = t.model_cfg, t.engine.params, t.cfg
    flat = P.lowp.double().requires_grad_()
    views = {p.name: flat[p.offset:p.offset + p.numel].view(p.shape) for p in P.specs}
    tokens = s["tokens"].cuda()
    loss, S, N = 0.0, c["seq"], c["batch"]
    step = max(1, min(N, 4096 // S))
    for b in range(0, N, step):
        part = tokens[b:b + step]
        n = part.shape[0]

        def attend(l, q, k, v):
            heads = lambda a: a.view(n, S, a.shape[1], a.shape[2]).transpose(1, 2)  # noqa: E731
            q, k, v = heads(q), *(heads(a).repeat_interleave(cfg.n_head // cfg.n_kv_head, 1) for a in (k, v))
            score = (q @ k.transpose(-1, -2) / math.sqrt(cfg.head_dim)).masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -math.inf)
            return (torch.softmax(score, -1) @ v).transpose(1, 2).reshape(n * S, -1)

        pos = torch.arange(S, device="cuda").repeat(n)
        logits = _decoder(cfg, views.__getitem__, part[:, :-1].reshape(-1), pos, attend) @ views[_head_name(cfg)].T
        e = torch.nn.functional.cross_entropy(logits[:, :cfg.vocab_size], part[:, 1:].reshape(-1), reduction="sum") / (N * S)
        e.backward()
        loss += float(e.detach())
        del logits, e
    with torch.no_grad():
        grad, master = flat.grad, P.master.double()
        gs = grad * min(1.0, tc.max_grad_norm / (float(grad.norm()) + 1e-6))
        update = gs / (gs.abs() + tc.eps)                       # the first step: both moments are the gradient's own
        update[:P.decay_end] += tc.weight_decay * master[:P.decay_end]
        return dict(loss=torch.tensor(loss, dtype=torch.float64), grads=grad, weights=master - tc.lr * update)


@torch.no_grad()
def _exact_serve(c, s):
    r = s["runner"]
    cfg, D, G = r.cfg, r.cfg.head_dim, r.cfg.n_kv_head
    kc, vc = ([t.double().view(-1, G, D) for t in a] for a in (r.cache.k, r.cache.v))
    place = lambda seq, n: (torch.tensor(r.cache.block_table(seq), device="cuda")[:, None] * 16 + torch.arange(16, device="cuda")).view(-1)[:n]  # noqa: E731
    parts = [(i, ids, at) for i, ids, at, _ in s["chunks"]] + [(i, [t], n - 1) for i, t, n in zip(s["ids"], s["tokens"], s["lengths"])]
    ids = torch.tensor([t for _, p, _ in parts for t in p], device="cuda")
    pos = torch.tensor([at + j for _, p, at in parts for j in range(len(p))], device="cuda")
    where = [place(i, at + len(p)) for i, p, at in parts]
    ends = [0]
    for _, p, _ in parts:
        ends.append(ends[-1] + len(p))

    def attend(l, q, k, v):
        out = []
        for (_, p, at), slots, r0, r1 in zip(parts, where, ends, ends[1:]):
            kc[l][slots[at:]], vc[l][slots[at:]] = k[r0:r1], v[r0:r1]
            out.append(_attend(q[r0:r1], kc[l][slots], vc[l][slots], True))
        return torch.cat(out)

    x = _decoder(cfg, lambda name: r.params.w(name).double(), ids, pos, attend)
    logits = x[[e - 1 for e in ends[1:]]] @ r.params.w(_head_name(cfg)).double().T
    cache = [torch.stack(a).view(c["layers"], -1, 16, G, D) for a in (kc, vc)]
    n = len(s["chunks"])
    if c["kind"] == "decode":
        return dict(logits=logits, k=cache[0], v=cache[1])
    return dict(first=list(logits[:n]), decoded=logits[n:] if s["ids"] else None, k=cache[0], v=cache[1])


def _exact_experts(c, s):
    x, router, w1, w2 = (s[k].detach().double().requires_grad_() for k in ("x", "router", "w1", "w2"))
    p = torch.softmax(x @ router.T, -1)
    top, idx = p.topk(c["top"], -1)
    weight = top / top.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(c["experts"]):
        rows, j = (idx == e).nonzero(as_tuple=True)
        h = x[rows] @ w1[e].T
        if c["act"] == "swiglu":
            gate, up = h.chunk(2, -1)
            h = torch.nn.functional.silu(gate) * up
        else:
            h = _gelu(h)
        y = y.index_add(0, rows, (h @ w2[e].T) * weight[rows, j][:, None])
    share = torch.bincount(idx.reshape(-1), minlength=c["experts"]).double() / idx.numel()
    aux = (share * p.mean(0)).sum() * c["experts"]
    grads = torch.autograd.grad((y, aux * 0.01), (x, router, w1, w2), (s["dy"].double(), torch.ones_like(aux)))
    return dict(y=y, aux=aux, grads=grads)


def _exact_encoder(c, s):
    B, S, d, H = c["batch"], c["seq"], c["d"], c["heads"]
    params = [p.detach().double().requires_grad_() for p in s["params"]]
    names = [n for layer in s["layers"] for n, _ in layer.named_parameters()]
    per = len(names) // c["layers"]
    x = s["x"].detach().double().requires_grad_()
    y = x
    for l in range(c["layers"]):
        w = dict(zip(names[l * per:(l + 1) * per], params[l * per:(l + 1) * per]))
        norm = lambda t, n: torch.nn.functional.layer_norm(t, (d,), w[n + ".weight"], w[n + ".bias"], 1e-5)  # noqa: E731
        lin = lambda t, n: t @ w[n + ".weight"].T + w[n + ".bias"]  # noqa: E731
        h = norm(y, "norm1")
        q, k, v = (lin(h, f"self_attn.{n}_proj").view(B, S, H, d // H) for n in "qkv")
        a = torch.stack([_attend(q[b], k[b], v[b], False, n).reshape(S, d) for b, n in enumerate(_padded(c))])
        y = y + lin(a, "self_attn.out_proj")
        y = y + lin(_gelu(lin(norm(y, "norm2"), "ff_linear1")), "ff_linear2")
    return dict(y=y, grads=_without_key_bias(s, torch.autograd.grad(y, [x, *params], s["dy"].double())))


def exact(c, seed):
    s = prepare(c, seed)
    return {"train": _exact_train, "experts": _exact_experts, "encoder": _exact_encoder}.get(c["kind"], _exact_serve)(c, s)
