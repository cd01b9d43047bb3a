"""The work whose speed is watched: optimizer steps of LoRA fine-tuning through `Trainer.train_step`, and requests served by every
model family through `LLMEngine.replay_step`, which packs, schedules and runs a step as the server does and returns logits.

A serving pass is one batch of requests from their prompts to their end: one step over all prompts, then `new` steps of one
token per request, then the pages go back. `new = 0` is the prompt alone. Weights are random, in the layer sizes of the presets
(`models/config.py`, `models/sigosun.py`, ...), with fewer layers so that a pass is short. `exact` restates all of it in double
precision on plain torch.
"""
from __future__ import annotations

import math
import random

import torch

VOCAB = 32000
FAMILIES = ("llama", "sigosun", "logozen", "latanex", "ridazen")
#: Layers of one unit of a family's pattern; a Ridazen has at least four layers, of which the second and third run twice.
PATTERN = {"llama": 1, "sigosun": 4, "logozen": 2, "latanex": 2, "ridazen": 1}


def serve(family, width, units, seqs, prompt, new, dtype="bfloat16", spread=0, **more):
    """`seqs` requests; the longest prompt has `prompt` tokens, the shortest about `spread` percent fewer."""
    return {**more, "kind": "serve", "family": family, "width": width, "units": units, "seqs": seqs, "prompt": prompt, "new": new,
            "dtype": dtype, "spread": spread}


def train(width, layers, groups, micro, seqs, length, dtype="bfloat16", spread=0, zero=3, recompute=True, dropout=0.05, **more):
    """`micro` micro-batches of `seqs` rows of up to `length` tokens; `groups` query heads share a key/value head."""
    return {**more, "kind": "train", "width": width, "layers": layers, "groups": groups, "micro": micro, "seqs": seqs, "length": length,
            "dtype": dtype, "spread": spread, "zero": zero, "recompute": recompute, "dropout": dropout}


def listed():
    return [
        # the headline: layers of Llama-2-7B, an accumulation window of 4 x 2 x 2048 tokens, recompute, dropout, ZeRO-3
        train(4096, 4, 1, 4, 2, 2048, name="train window 7b"),
        # fine-tuning on short rows of unequal length with grouped heads, fp16 with loss scaling, nothing recomputed
        train(2048, 4, 4, 1, 8, 700, dtype="float16", spread=70, zero=1, recompute=False, name="train ragged fp16"),
        # one user of a Llama-2-7B shaped model: a short prompt, then tokens one at a time; weights and launches are all there is
        serve("llama", 4096, 6, 1, 100, 32, groups=1, name="llama one user"),
        # a full batch of short chats
        serve("llama", 2048, 12, 64, 120, 16, dtype="float16", spread=50, groups=4, name="llama batch 64"),
        # a batch of long prompts of unequal length
        serve("llama", 4096, 4, 4, 2048, 0, spread=20, groups=4, name="llama prompts"),
        # one long document
        serve("sigosun", 2048, 2, 1, 8192, 0, name="sigosun long prompt"),
        # a small batch answering
        serve("sigosun", 2048, 2, 16, 100, 32, spread=50, name="sigosun batch 16"),
        # several prompts of ordinary length
        serve("logozen", 2048, 3, 4, 2048, 0, spread=10, name="logozen prompts"),
        # a full batch answering
        serve("logozen", 2048, 3, 64, 100, 16, spread=50, name="logozen batch 64"),
        # many short prompts
        serve("latanex", 2048, 2, 16, 512, 0, spread=30, name="latanex prompts"),
        # a small batch answering: every step reads most experts
        serve("latanex", 2048, 2, 16, 60, 24, spread=50, name="latanex batch 16"),
        # few requests with longer context, prompt and answer together
        serve("ridazen", 2048, 4, 4, 1000, 24, spread=25, name="ridazen chat"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of these ranges: 1 - 64 requests, prompts of 2 - 8192 tokens with at most 8192 in a step, up to 32 answered tokens,
    widths of 1024 - 4096; optimizer steps over 100 - 16384 tokens."""
    most = max(_cost(c) for c in listed())
    while True:
        if rng.random() < 0.2:
            width = rng.choice((1024, 2048, 4096))
            length = _log(rng, 20, 2048)
            c = train(width, rng.randint(2, 4), rng.choice((1, 4)), rng.choice((1, 1, 2, 4)), rng.randint(1, 8), length,
                      rng.choice(("bfloat16", "bfloat16", "float16")), rng.choice((0, 40, 70)), rng.choice((1, 2, 3)), rng.random() < 0.7,
                      rng.choice((0.0, 0.05)))
            tokens = sum(_lengths(c["seqs"], length, c["spread"])) * c["micro"]
            if not 100 <= tokens <= 16384:
                continue
        else:
            family = rng.choice(FAMILIES)
            width = rng.choice((1024, 2048, 2048, 4096))
            units = {"llama": rng.randint(2, 12), "sigosun": rng.randint(1, 2), "logozen": rng.randint(1, 3), "latanex": rng.randint(1, 2),
                     "ridazen": rng.randint(4, 5)}[family]
            seqs, new = _log(rng, 1, 64), rng.choice((0, 0, _log(rng, 4, 32)))
            prompt = _log(rng, 2, 8192)
            more = {"groups": rng.choice((1, 4))} if family == "llama" else {}
            c = serve(family, width, units, seqs, prompt, new, "float16" if family == "llama" and rng.random() < 0.5 else "bfloat16",
                      rng.choice((0, 30, 60)), **more)
            if sum(_lengths(seqs, prompt, c["spread"])) > 8192:
                continue
        if _cost(c) <= most:
            return c


def _cost(c):
    w = work(c)
    return max(w["bytes"] / 6e12, w["flops"] / 1e15)


def _lengths(n, longest, spread):
    return [max(1, longest - longest * spread * i // (100 * n)) for i in range(n)]


def _llama_sizes(width, groups, layers):
    heads = width // 128
    return dict(hidden_size=width, intermediate_size=width * 43 // 16 // 256 * 256, num_hidden_layers=layers, num_attention_heads=heads,
                num_key_value_heads=heads // groups, vocab_size=VOCAB, max_position_embeddings=8448)


def _model(c):
    """config.json of a layer-stack model."""
    width, n = c["width"], c["units"]
    heads = width // 128
    kv = max(1, heads // 4)
    head = dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5)
    base = {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}}
    if c["family"] == "sigosun":
        ff = {"kind": "dense", "ff": 4 * width}
        att = dict(head, mask={"size": 2048}, rot={"base": 5e5, "dims": 128})
        layers = []
        for b in range(n):
            layers += [{"type": "attention", "mixer": att, "mlp": ff}, {"type": "attention", "mixer": dict(att, kv_from=4 * b), "mlp": ff},
                       {"type": "mamba2", "mixer": dict(heads=width // 32, vdim=64, state=128, groups=1, conv=4, norm_groups=1), "mlp": None},
                       {"type": "lightning", "mixer": dict(heads=heads, dim=128, vdim=128, decay=[1 - 2.0 ** (-4 - 5 * h / heads) for h in range(heads)]),
                        "mlp": None}]
        return {"architecture": "Sigosun", **base, "layers": layers}
    if c["family"] == "logozen":
        ff = {"kind": "dense", "ff": 4 * width}
        att = dict(heads=heads, dim=64, rot_dim=64, vdim=128, kv_rank=512, scale=128 ** -0.5, rot={"base": 1e6, "dims": 64})
        mem = dict(heads=heads // 2, dim=128, vdim=256, gate_cap=15.0)
        return {"architecture": "Logozen", **base, "streams": 4, "canon": {"taps": 4}, "embedding": {"scale": 45.0},
                "layers": [{"type": "mlstm", "mixer": mem, "mlp": ff}, {"type": "latent_attention", "mixer": att, "mlp": ff}] * n}
    if c["family"] == "latanex":
        moe = {"kind": "moe", "expert": {"ff": width // 4, "limit": 7.0}, "shared": {"ff": width // 2, "limit": 7.0},
               "router": {"experts": 64, "top": 8, "scale": 2.5, "groups": {"count": 8, "keep": 4}}}
        att = dict(head, softcap=30.0, mask={"size": 2048}, v_mix=True)
        mem = dict(heads=heads, kv_heads=heads, dim=128, vdim=128, conv=4)
        return {"architecture": "Latanex", **base, "embedding": {"scale": 4.0}, "logit_scale": 0.5,
                "layers": [{"type": "delta", "mixer": mem, "mlp": moe}, {"type": "attention", "mixer": att, "mlp": moe}] * n}
    moe = {"kind": "moe", "expert": {"ff": width // 4}, "shared": {"ff": width // 2}, "router": {"experts": 64, "top": 8}}
    att = dict(head, conv=4, q_temp={"coef": 0.1, "every": 1024}, bias_max=128, bias_rows=32)
    return {"architecture": "Ridazen", **base, "residual_mult": 0.7, "logit_scale": 0.5, "logit_softcap": 30.0, "token_side": {"dim": 128},
            "loop": {"start": 1, "stop": 3, "times": 2}, "layers": [{"type": "attention", "mixer": att, "mlp": moe}] * n}


# ---- inputs ------------------------------------------------------------------------------------------------
def _tokens(seed, n):
    return torch.randint(3, VOCAB, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def prepare(case, seed):
    return _prepare_train(case, seed) if case["kind"] == "train" else _prepare_serve(case, seed)


def _prepare_serve(c, seed):
    from dlti_b200.models.config import LlamaConfig
    from dlti_b200.models.llama import ResidentWeights
    from dlti_b200.models.registry import FAMILIES as KNOWN
    from dlti_b200.serve.engine import LLMEngine
    from dlti_b200.serve.model_runner import TPContext, TPWeights
    from dlti_b200.serve.tokenizer import ByteTokenizer

    if c["family"] == "llama":
        dtype = getattr(torch, c["dtype"])
        cfg = LlamaConfig(**_llama_sizes(c["width"], c["groups"], c["units"]), name="llama")
        source = ResidentWeights.random_init(cfg, "cuda", dtype, seed)
        weights = TPWeights(cfg, 0, 1, "cuda", dtype).load_from_full(source)
    else:
        from dlti_b200.models import latanex, logozen, ridazen, sigosun
        design = {"sigosun": sigosun, "logozen": logozen, "latanex": latanex, "ridazen": ridazen}[c["family"]]
        d = _model(c)
        cfg = KNOWN[d["architecture"]].config_cls.from_dict(d, name=c["family"])
        source = design.random_state(cfg, seed, "cuda")
        weights = design.from_state(cfg, source, "cuda", torch.bfloat16)
    lengths = _lengths(c["seqs"], c["prompt"], c["spread"])
    prompts = [_tokens(seed * 1000 + i, n) for i, n in enumerate(lengths)]
    answers = [_tokens(seed * 1000 + 500 + i, c["new"]) for i in range(c["seqs"])]
    longest = c["prompt"] + c["new"]
    engine = LLMEngine(cfg, weights, TPContext(), ByteTokenizer(VOCAB), num_blocks=sum(-(-(n + c["new"]) // 16) for n in lengths) + 8,
                       max_num_seqs=c["seqs"], max_num_batched_tokens=8192, max_model_len=-(-longest // 64) * 64)
    if c["new"]:
        engine.warmup(c["seqs"])                  # as a server does before its first request
    state = {"engine": engine, "prompts": prompts, "answers": answers}
    if c.get("source"):
        state["source"] = source
    return state


def _prepare_train(c, seed):
    from dlti_b200.config.args import TrainingArgs
    from dlti_b200.engine.trainer import Trainer
    from dlti_b200.models.config import LlamaConfig
    from dlti_b200.models.llama import pack_batch
    from dlti_b200.models.lora import LoraConfig

    cfg = LlamaConfig(**_llama_sizes(c["width"], c["groups"], c["layers"]), name="llama")
    args = TrainingArgs(output_dir="/tmp/dlti_cases", per_device_train_batch_size=c["seqs"], gradient_accumulation_steps=c["micro"],
                        precision="fp16" if c["dtype"] == "float16" else "bf16", gradient_checkpointing=c["recompute"],
                        deepspeed=f"configs/ds_config_zero{c['zero']}.json", no_offload=True, max_steps=1000)
    trainer = Trainer(cfg, LoraConfig(r=16, lora_alpha=32, lora_dropout=c["dropout"]), args, init_seed=seed)
    # fine-tuning that goes on from an adapter: B is no longer zero
    g = torch.Generator().manual_seed(seed)
    adapter = {}
    for name, t in trainer.lora.state_dict().items():
        adapter[name] = torch.empty_like(t).normal_(0.0, 0.02 if "lora_B" in name else t.shape[1] ** -0.5 / 2, generator=g)
    trainer.lora.load_state_dict(adapter)
    batches = []
    lengths = _lengths(c["seqs"], c["length"], c["spread"])
    for _ in range(c["micro"]):
        ids = torch.randint(3, VOCAB, (c["seqs"], c["length"]), generator=g)
        mask = (torch.arange(c["length"])[None, :] < torch.tensor(lengths)[:, None]).long()
        labels = ids.masked_fill(mask == 0, -100)
        labels[:, :c["length"] // 8] = -100       # instructions are not learned
        batches.append(pack_batch(ids, labels, mask, pin=True))
    return {"trainer": trainer, "batches": batches}


def run(state):
    if "trainer" in state:
        trainer = state["trainer"]
        loss = trainer.train_step(state["batches"])
        return {"loss": loss, "adapters": trainer.lora.master, "momentum": trainer.optimizer.m}
    from dlti_b200.serve.params import Request, SamplingParams
    engine, prompts, answers = state["engine"], state["prompts"], state["answers"]
    steps = len(answers[0])
    requests = [Request(str(i), [], SamplingParams(temperature=0.0)) for i in range(len(prompts))]
    logits = engine.replay_step([(r, p, [] if steps else [len(p) - 1]) for r, p in zip(requests, prompts)])
    for k in range(steps):
        logits = engine.replay_step([(r, [a[k]], [0] if k == steps - 1 else []) for r, a in zip(requests, answers)])
    for r in requests:
        engine.replay_end(r)
    return logits


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _parts(c):
    """Per layer run: (parameters every token uses, parameters that a step of few rows may skip and the share that a token
    uses, key/value elements a token caches, state elements of a sequence, scores of a (query, key) pair, furthest key)."""
    width = c["width"]
    heads, kv = width // 128, max(1, width // 512)
    if c["family"] == "llama":
        kv = heads // c["groups"]
        s = _llama_sizes(width, c["groups"], 1)
        return [(width * 128 * (2 * heads + 2 * kv) + 3 * width * s["intermediate_size"], 0, 1, 2 * 128 * kv, 0, 4 * 128 * heads, 1 << 30)] * c["units"]
    out = []
    if c["family"] == "sigosun":
        ff, attn = 8 * width * width, width * 128 * (2 * heads)
        inner, n = 2 * width, width // 32
        out = [(ff + attn + width * 256 * kv, 0, 1, 256 * kv, 0, 4 * 128 * heads, 2048), (ff + attn, 0, 1, 0, 0, 4 * 128 * heads, 2048),
               (width * (3 * inner + 256 + n), 0, 1, 0, n * 128 * 64, 0, 0), (5 * width * width, 0, 1, 0, heads * 128 * 128, 0, 0)] * c["units"]
    elif c["family"] == "logozen":
        ff = 8 * width * width
        out = [(ff + 4 * width * width, 0, 1, 0, heads // 2 * 128 * 256, 0, 0),
               (ff + width * (2 * 128 * heads + 576) + 512 * heads * 192, 0, 1, 576, 0, 4 * 128 * heads, 1 << 30)] * c["units"]
    else:
        gated = 3 if c["family"] == "latanex" else 2
        moe, shared = 64 * gated * width * width // 4, gated * width * width // 2 + 64 * width
        if c["family"] == "latanex":
            out = [(shared + 5 * width * width, moe, 1 / 8, 0, heads * 128 * 128, 0, 0),
                   (shared + width * 128 * (2 * heads + 2 * kv), moe, 1 / 8, 256 * kv, 0, 4 * 128 * heads, 2048)] * c["units"]
        else:
            out = [(shared + width * 128 * (3 * heads + 2 * kv) + 256 * width, moe, 1 / 8, 256 * kv, 0, 4 * 128 * heads, 1 << 30)] * (c["units"] + 2)
    return out


def work(case):
    c = case
    if c["kind"] == "train":
        s = _llama_sizes(c["width"], c["groups"], c["layers"])
        d, ff, kv = s["hidden_size"], s["intermediate_size"], s["num_key_value_heads"] * 128
        per_layer = d * (2 * d + 2 * kv) + 3 * d * ff
        matrices = c["layers"] * per_layer + VOCAB * d
        adapters = c["layers"] * 16 * (d * 4 + 2 * d + 2 * kv)
        lengths = _lengths(c["seqs"], c["length"], c["spread"]) * c["micro"]
        pairs = sum(n * (n + 1) // 2 for n in lengths)
        tokens = sum(lengths)
        # forward, and backward to the inputs; scores forward and (four products of six) backward; adapters three ways
        flops = 4 * tokens * matrices + 6 * tokens * adapters + pairs * c["layers"] * 4 * d * 3.0
        return {"bytes": 2 * 2 * matrices + 16 * adapters + 24 * tokens, "flops": flops}
    parts = _parts(c)
    lengths = _lengths(c["seqs"], c["prompt"], c["spread"])
    head = VOCAB * c["width"]
    flops = nbytes = 0.0
    for k in range(c["new"] + 1):
        rows = sum(lengths) if k == 0 else c["seqs"]
        asked = c["seqs"] if k == c["new"] else 0
        nbytes += 2 * head * (asked > 0) + 4 * VOCAB * asked + 2 * rows * c["width"]
        flops += 2 * asked * head
        for dense, moe, share, cached, state, score, reach in parts:
            nbytes += 2 * (dense + moe * (1 - (1 - share) ** rows)) + 2 * cached * rows
            flops += 2 * rows * (dense + share * moe)
            if state:
                nbytes += 4 * state * c["seqs"] * (1 if k == 0 else 2)
                flops += 4 * state * rows
            if score and k == 0:
                flops += score * sum(m * (m + 1) // 2 + (n - m) * m for n in lengths for m in (min(n, reach),))
            elif score:
                seen = sum(min(n + k, reach) for n in lengths)
                flops += score * seen
                nbytes += 2 * cached * seen
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # 16-bit activations between the layers; a router that tips at a near tie exchanges one of a token's eight experts. The same
    # inputs twice (sums of split products come in any order) differ by up to 0.012 in bf16 and 0.002 in fp16
    return {"rel": 0.01, "max": 0.1} if case["dtype"] == "float16" else {"rel": 0.03, "max": 0.3}


# ---- the same in double precision ---------------------------------------------------------------------------
def exact(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        return _exact_train(c, seed)
    state = prepare({**c, "new": 0, "source": True}, seed)     # the weights and tokens; `new` only adds graphs
    w, prompts = state["source"], state["prompts"]
    answers = [_tokens(seed * 1000 + 500 + i, c["new"]) for i in range(c["seqs"])]
    del state["engine"]
    rows = [p + a for p, a in zip(prompts, answers)]
    last = torch.tensor([len(r) - 1 for r in rows], device="cuda")
    ids = torch.zeros(len(rows), int(last.max()) + 1, dtype=torch.long)       # padded on the right: nothing looks ahead
    for i, r in enumerate(rows):
        ids[i, :len(r)] = torch.tensor(r)
    ids = ids.cuda()
    pick = lambda x: x[torch.arange(len(rows), device="cuda"), last]
    with torch.no_grad():
        if c["family"] == "llama":
            return _llama_logits(_llama_sizes(c["width"], c["groups"], c["units"]), w, ids, pick)
        return {"sigosun": _sigosun, "logozen": _logozen, "latanex": _latanex, "ridazen": _ridazen}[c["family"]](_model(c), _Weights(w), ids, pick)


class _Weights:
    """Checkpoint tensors in double precision, made when they are used."""

    def __init__(self, state, prefix=""):
        self.state, self.prefix = state, prefix

    def __getitem__(self, name):
        return self.state[self.prefix + name].double()

    def __contains__(self, name):
        return self.prefix + name in self.state

    def at(self, prefix):
        return _Weights(self.state, self.prefix + prefix)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _heads(x, n):
    return x.view(*x.shape[:-1], n, -1)


def _turn(x, base, dims):
    """x [B, T, heads, dim]: coordinates (2i, 2i + 1) of the first `dims` turn by position * base^(-2i / dims)."""
    a = torch.arange(x.shape[1], device=x.device).double()[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device).double() / dims)
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    out = x.clone()
    out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, chunk=0, window=0, cap=0.0, sink=None, bias=None):
    """q [B, T, H, d], k and v [B, T, G, .]; chunk, window: what a query sees; bias [T, H]: added at that distance."""
    B, T, H, _ = q.shape
    rep = H // k.shape[2]
    out = torch.empty(B, T, H, v.shape[3], dtype=q.dtype, device=q.device)
    for t0 in range(0, T, 2048):
        t1 = min(T, t0 + 2048)
        lo = t0 // chunk * chunk if chunk else max(0, t0 - window + 1) if window else 0
        i, j = torch.arange(t0, t1, device=q.device)[:, None], torch.arange(lo, t1, device=q.device)[None, :]
        hidden = j > i
        if chunk:
            hidden = hidden | (j // chunk != i // chunk)
        if window:
            hidden = hidden | (i - j >= window)
        for h in range(H):
            s = q[:, t0:t1, h] @ k[:, lo:t1, h // rep].transpose(1, 2) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if bias is not None:
                s = s + bias[(i - j).clamp(min=0), h]
            s = s.masked_fill(hidden, -math.inf)
            top = s.amax(2, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[h])
            e = torch.exp(s - top)
            total = e.sum(2, keepdim=True)
            if sink is not None:
                total = total + torch.exp(sink[h] - top)
            out[:, t0:t1, h] = e @ v[:, lo:t1, h // rep] / total
    return out


def _conv(x, weight):
    """Per channel: y_t = sum_j weight[:, j] x_(t - taps + 1 + j)."""
    taps = weight.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    return sum(weight[:, j] * padded[:, j:j + x.shape[1]] for j in range(taps))


def _memory(q, k, v, decay):
    """S <- decay_t S + k_t v_t^T, o_t = S^T q_t; q, k [B, T, H, d], v [B, T, H, e], decay [B, T, H]."""
    S = torch.zeros(*q.shape[:1], *q.shape[2:], v.shape[3], dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        S.mul_(decay[:, t, :, None, None])
        S.addcmul_(k[:, t, :, :, None].expand_as(S), v[:, t, :, None, :].expand_as(S))
        out[:, t] = torch.einsum("bhd,bhde->bhe", q[:, t], S)
    return out


def _sigosun(cfg, w, ids, pick):
    eps = cfg["norm"]["eps"]
    x = w["embed"][ids]
    cache = {}
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], w.at(f"l{i}.mix.")
        if layer["type"] == "attention":
            norm = lambda y, s, n: _turn(_rms(_heads(y, n), eps) * p[s + ".norm"], m["rot"]["base"], m["rot"]["dims"])
            if "kv_from" not in m:
                cache[i] = norm(x @ p["k"].T, "k", m["kv_heads"]), _heads(x @ p["v"].T, m["kv_heads"])
            y = _attend(norm(x @ p["q"].T, "q", m["heads"]), *cache[m.get("kv_from", i)], m["scale"], chunk=m["mask"]["size"])
            y = (y * torch.sigmoid(x @ p["g"].T)[..., None]).flatten(2)
        elif layer["type"] == "mamba2":
            H, N, G = m["heads"], m["state"], m["groups"]
            inner = H * m["vdim"]
            z, xbc, dt = torch.split(x @ p["in"].T, [inner, inner + 2 * G * N, H], -1)
            u, b, r = torch.split(_silu(_conv(xbc, p["conv"]) + p["conv.b"]), [inner, G * N, G * N], -1)
            dt = torch.nn.functional.softplus(dt + p["dt_bias"], threshold=1e9)
            u, b, r = _heads(u, H), (_heads(b, G).repeat_interleave(H // G, 2)), (_heads(r, G).repeat_interleave(H // G, 2))
            y = _memory(r, b, u * dt[..., None], torch.exp(-torch.exp(p["A_log"]) * dt)) + p["D"][:, None] * u
            y = _rms(_heads(y.flatten(2) * _silu(z), m["norm_groups"]), eps).flatten(2) * p["norm"]
        else:
            q, k, v = (_heads(_silu(x @ p[s].T), m["heads"]) for s in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=ids.device).expand(*ids.shape, -1)
            y = _rms(_memory(q, k, v, decay).flatten(2), eps) * p["norm"] * torch.sigmoid(x @ p["g"].T)
        x = x + _rms(y @ p["o"].T, eps) * (1 + w[f"l{i}.norm1"])
        if layer["mlp"]:
            y = torch.relu(x @ w[f"l{i}.mlp.up"].T).square() @ w[f"l{i}.mlp.down"].T
            x = x + _rms(y, eps) * (1 + w[f"l{i}.norm2"])
    return (_rms(pick(x), eps) * (1 + w["final.norm"])) @ w["head"].T


def _logozen(cfg, w, ids, pick):
    eps, n = cfg["norm"]["eps"], cfg["streams"]

    def norm(y, weight):
        y = y - y.mean(-1, keepdim=True)
        return _rms(y, eps) * weight

    xs = [w["embed"][ids] * cfg["embedding"]["scale"]] * n

    def latent(h, p, m):
        H, r = m["heads"], m["kv_rank"]
        q, down = _heads(h @ p["q"].T, H), h @ p["dkv"].T
        c = _rms(down[..., :r], eps) * p["dkv.norm"]
        turn = lambda y: _turn(y, m["rot"]["base"], m["rot"]["dims"])
        q = torch.cat([q[..., :m["dim"]], turn(q[..., m["dim"]:])], -1)
        k = torch.cat([_heads(c @ p["uk"].T, H), turn(down[..., None, r:]).expand(-1, -1, H, -1)], -1)
        y = _attend(q, k, _heads(c @ p["uv"].T, H), m["scale"], sink=p["sink"])
        return (y * torch.sigmoid(h @ p["g"].T)[..., None]).flatten(2)

    def mlstm(h, p, m):
        H = m["heads"]
        cap = lambda z: m["gate_cap"] * torch.tanh(z / m["gate_cap"])
        q, k, v = _heads(h @ p["q"].T, H) * m["dim"] ** -0.5, _heads(h @ p["k"].T, H), _heads(h @ p["v"].T, H)
        log_in, log_keep = cap(h @ p["i"].T + p["i.b"]), torch.nn.functional.logsigmoid(cap(h @ p["f"].T + p["f.b"]))
        S = torch.zeros(len(q), H, q.shape[3], v.shape[3] + 1, dtype=q.dtype, device=q.device)       # last column: the normaliser
        v1 = torch.cat([v, torch.ones_like(v[..., :1])], -1)
        top = torch.zeros(len(q), H, dtype=q.dtype, device=q.device)
        y = torch.empty_like(v)
        for t in range(q.shape[1]):
            new = torch.maximum(log_keep[:, t] + top, log_in[:, t])
            S.mul_(torch.exp(log_keep[:, t] + top - new)[..., None, None])
            S.addcmul_((torch.exp(log_in[:, t] - new)[..., None] * k[:, t])[..., None].expand_as(S), v1[:, t, :, None, :].expand_as(S))
            top = new
            o = torch.einsum("bhd,bhde->bhe", q[:, t], S)
            y[:, t] = o[..., :-1] / (torch.maximum(o[..., -1].abs(), torch.exp(-top)) + 1e-6)[..., None]
        return _rms(y, eps).flatten(2) * p["norm"] * torch.sigmoid(h @ p["g"].T)

    def between(i, s, f):
        p = w.at(f"l{i}.")
        a, b, mix = p[f"hc{s}.in"], p[f"hc{s}.out"], p[f"hc{s}.mix"]
        h = norm(sum(a[j] * xs[j] for j in range(n)), p[f"norm{s}"])
        y = f(h + _conv(h, p[f"canon{s}"]))
        return [sum(mix[j, t] * xs[j] for j in range(n)) + b[t] * y for t in range(n)]

    for i, layer in enumerate(cfg["layers"]):
        p, mixer = w.at(f"l{i}."), latent if layer["type"] == "latent_attention" else mlstm
        xs = between(i, 1, lambda h: mixer(h, p.at("mix."), layer["mixer"]) @ p["mix.o"].T)

        def forward(h):
            z, (a, b, e, f) = h @ p["mlp.up"].T, p["mlp.act"]
            return (a * _rms(z, eps) + b * _rms(z * z, eps) + e * _rms(z * z * z, eps) + f) @ p["mlp.down"].T
        xs = between(i, 2, forward)
    return norm(pick(sum(xs)), w["final.norm"]) @ w["head"].T


def _experts(h, p, chosen, weight, one):
    """Sum of the chosen experts' outputs; chosen, weight [rows, top]; one(rows, expert's tensors)."""
    out = torch.zeros_like(h)
    for e in range(64):
        rows, slot = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, weight[rows, slot][:, None] * one(h[rows], p.at(f"e{e}.")))
    return out


def _latanex(cfg, w, ids, pick):
    eps = cfg["norm"]["eps"]
    norm = lambda y, p, name: torch.tanh(p[name + ".alpha"] * y) * p[name] + p[name + ".b"]
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    first = None

    def clipped(limit):
        def one(h, p):
            g, u = (h @ p["gate"].T).clamp(max=limit), (h @ p["up"].T).clamp(-limit, limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ p["down"].T
        return one

    def moe(h, p, m):
        r = m["router"]
        s = torch.sigmoid(h @ p["router"].T)
        c = s + p["correction"]
        n = r["groups"]["count"]
        best = _heads(c, n).topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
        closed = torch.ones(len(h), n, dtype=torch.bool, device=h.device).scatter_(1, best, False).repeat_interleave(c.shape[1] // n, 1)
        chosen = c.masked_fill(closed, -math.inf).topk(r["top"], -1).indices
        weight = s.gather(1, chosen)
        weight = weight / weight.sum(1, keepdim=True) * r["scale"]
        return _experts(h, p, chosen, weight, clipped(m["expert"]["limit"])) + clipped(m["shared"]["limit"])(h, p.at("shared."))

    for i, layer in enumerate(cfg["layers"]):
        m, q_ = layer["mixer"], w.at(f"l{i}.")
        p, h, H = q_.at("mix."), norm(x, q_, "norm1"), m["heads"]
        if layer["type"] == "attention":
            q, k, v = (h @ p[s].T + p[s + ".b"] for s in "qkv")
            q, k = _heads(_rms(q, eps) * p["q.norm"], H), _heads(_rms(k, eps) * p["k.norm"], m["kv_heads"])
            if first is None:
                first = v
            else:
                v = (1 - p["vmix"]) * v + p["vmix"] * first
            y = _attend(q, k, _heads(v, m["kv_heads"]), m["scale"], window=m["mask"]["size"], cap=m["softcap"], sink=p["sink"]).flatten(2)
        else:
            q, k, v = (_heads(_silu(_conv(h @ p[s].T, p[s + ".conv"])), H) for s in "qkv")
            unit = lambda y: y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)
            q, k = unit(q) * m["dim"] ** -0.5, unit(k)
            beta = torch.sigmoid(h @ p["b"].T)
            decay = torch.exp(-torch.exp(p["A_log"]) * torch.nn.functional.softplus(h @ p["a"].T + p["dt_bias"], threshold=1e9))
            S = torch.zeros(len(q), H, q.shape[3], v.shape[3], dtype=q.dtype, device=q.device)
            y = torch.empty_like(v)
            for t in range(q.shape[1]):
                S.mul_(decay[:, t, :, None, None])
                u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhd,bhde->bhe", k[:, t], S))
                S.addcmul_(k[:, t, :, :, None].expand_as(S), u[:, :, None, :].expand_as(S))
                y[:, t] = torch.einsum("bhd,bhde->bhe", q[:, t], S)
            y = (_rms(y, eps) * p["norm"] * _silu(_heads(h @ p["g"].T, H))).flatten(2)
        x = x + norm(y @ p["o"].T, q_, "norm1b")
        h = norm(x, q_, "norm2")
        x = x + norm(moe(h.flatten(0, 1), q_.at("mlp."), layer["mlp"]).view_as(x), q_, "norm2b")
    return norm(pick(x), w, "final.norm") @ w["head"].T * cfg["logit_scale"]


def _ridazen(cfg, w, ids, pick):
    eps, mult, side = cfg["norm"]["eps"], cfg["residual_mult"], cfg["token_side"]["dim"]
    loop, T = cfg["loop"], ids.shape[1]
    order = [(i, False) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, t > 0 and i == loop["start"]) for i in range(loop["start"], loop["stop"])]
    order += [(i, False) for i in range(loop["stop"], len(cfg["layers"]))]
    embed = w["embed"][ids]
    vectors = w.state["side.embed"][ids]
    x = embed

    def bucket(n, rows, far):
        half = rows // 2
        return n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(far / half) * (rows - half)))

    def relu2(h, p):
        return torch.relu(h @ p["up"].T).square() @ p["down"].T

    for i, again in order:
        m, e, q_ = cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"], w.at(f"l{i}.")
        p, H = q_.at("mix."), m["heads"]
        if again:
            x = x + embed
        h = _rms(x, eps) * q_["norm1"]
        q, k, v = (_conv(h @ p[s].T, p[s + ".conv"]) for s in "qkv")
        t = m["q_temp"]
        temp = torch.tensor([1 + t["coef"] * math.log((j + 1) // t["every"] + 1) for j in range(T)], dtype=torch.float64, device=ids.device)
        q = _rms(_heads(q, H), eps) * p["q.norm"] * temp[:, None, None]
        k = _rms(_heads(k, m["kv_heads"]), eps) * p["k.norm"]
        bias = p["rel"][torch.tensor([bucket(n, m["bias_rows"], m["bias_max"]) for n in range(T)], device=ids.device)]
        y = _attend(q, k, _heads(v, m["kv_heads"]), m["scale"], bias=bias).flatten(2)
        x = x + mult * ((y * torch.sigmoid(h @ p["g"].T)) @ p["o"].T)
        h, p = (_rms(x, eps) * q_["norm2"]).flatten(0, 1), q_.at("mlp.")
        z, chosen = (h @ p["router"].T + p["router.b"]).topk(e["router"]["top"], -1)
        y = _experts(h, p, chosen, torch.softmax(z, -1), relu2) + relu2(h, p.at("shared.")) * torch.sigmoid(h @ p["shared.sg"].T)
        x = x + mult * y.view_as(x)
        p = q_.at("side.")
        y = torch.nn.functional.gelu(x @ p["gate"].T, approximate="tanh") * vectors[..., i * side:(i + 1) * side].double()
        x = x + mult * _rms(y @ p["proj"].T, eps) * p["norm"]
    z = (_rms(pick(x), eps) * w["final.norm"]) @ w["head"].T * cfg["logit_scale"]
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _half_turn(x, theta):
    """x [B, T, heads, dim]: coordinates (i, i + dim / 2) turn by position * theta^(-2i / dim)."""
    half = x.shape[-1] // 2
    a = torch.arange(x.shape[1], device=x.device).double()[:, None] * theta ** (-torch.arange(half, device=x.device).double() / half)
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _llama_block(s, lw, x, extra=lambda name, h: 0.0):
    """One decoder layer; extra(name, input): what an adapter adds to a projection."""
    H, G = s["num_attention_heads"], s["num_key_value_heads"]
    eps, q_, kv_ = 1e-5, H * 128, G * 128
    h = _rms(x, eps) * lw.ln1.double()
    q, k, v = (h @ t.double().T + extra(n, h) for n, t in zip("qkv", torch.split(lw.w_qkv, [q_, kv_, kv_])))
    q, k, v = _half_turn(_heads(q, H), 1e4), _half_turn(_heads(k, G), 1e4), _heads(v, G)
    if x.requires_grad:
        wide = lambda y: y.transpose(1, 2)
        k, v = (y.repeat_interleave(H // G, 2) for y in (k, v))
        later = torch.ones(x.shape[1], x.shape[1], dtype=torch.bool, device=x.device).triu(1)
        a = torch.softmax((wide(q) @ wide(k).transpose(2, 3) * 128 ** -0.5).masked_fill(later, -math.inf), -1)
        y = wide(a @ wide(v)).flatten(2)
    else:
        y = _attend(q, k, v, 128 ** -0.5).flatten(2)
    x = x + y @ lw.w_o.double().T + extra("o", y)
    gate, up = (_rms(x, eps) * lw.ln2.double() @ lw.w_gu.double().T).chunk(2, -1)
    return x + (_silu(gate) * up) @ lw.w_down.double().T


def _llama_logits(s, w, ids, pick):
    x = w.embed[ids].double()
    for lw in w.layers:
        x = _llama_block(s, lw, x)
    return (_rms(pick(x), 1e-5) * w.final_norm.double()) @ w.lm_head.double().T


def _keep(rows, cols, p, seed, stream, device):
    """Which elements a dropout mask of the counter-based generator Philox-4x32-10 keeps: element e takes word e % 4 of counter
    (e // 4, stream) under the key `seed`."""
    mask = 0xFFFFFFFF

    def product(m, x):
        low, high = m * (x & 0xFFFF), m * (x >> 16)
        return (high + (low >> 16)) >> 16, (m * x) & mask

    at = torch.arange(-(-rows * cols // 4), device=device)
    c0, c1, c2, c3 = at & mask, at >> 32, torch.full_like(at, stream & mask), torch.full_like(at, stream >> 32)
    k0, k1 = seed & mask, seed >> 32
    for _ in range(10):
        h0, l0 = product(0xD2511F53, c0)
        h1, l1 = product(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    threshold = int(torch.tensor(p, dtype=torch.float32) * 4294967296.0)
    return (torch.stack([c0, c1, c2, c3], 1).flatten()[:rows * cols] >= threshold).view(rows, cols)


def _exact_train(c, seed):
    state = _prepare_train(c, seed)
    trainer, batches = state["trainer"], state["batches"]
    s = _llama_sizes(c["width"], c["groups"], c["layers"])
    w = trainer.weights
    layers = [w.layer(i) for i in range(c["layers"])]
    names = list(trainer.lora.state_dict())
    leaf = {n: t.cuda().double().requires_grad_() for n, t in trainer.lora.state_dict().items()}
    padded, drop = trainer.lora.padded_numel, c["dropout"]
    valid = sum(b.n_valid for b in batches)
    total = 0.0
    for k, b in enumerate(batches):
        cu = b.cu_seqlens.tolist()
        n = len(cu) - 1
        T = max(y - x for x, y in zip(cu, cu[1:]))
        ids, labels = torch.zeros(n, T, dtype=torch.long), torch.full((n, T), -100)
        place = torch.cat([torch.arange(y - x) + i * T for i, (x, y) in enumerate(zip(cu, cu[1:]))]).cuda()
        for i, (x, y) in enumerate(zip(cu, cu[1:])):
            ids[i, :y - x], labels[i, :y - x] = b.input_ids[x:y], b.labels[x:y]
        ids, labels = ids.cuda(), labels.cuda()
        x = w.get_embed()[ids].double().requires_grad_()
        for li, lw in enumerate(layers):
            masks = {}

            def extra(name, h):
                site = 1 if name == "o" else 0
                if drop and site not in masks:             # the generator counts the rows without padding
                    m = _keep(cu[-1], h.shape[2], drop, 42, (k << 20) | (li << 4) | site, h.device).double() / (1 - drop)
                    masks[site] = torch.zeros(n * T, h.shape[2], dtype=torch.float64, device=h.device).index_copy_(0, place, m).view_as(h)
                key = f"base_model.model.model.layers.{li}.self_attn.{name}_proj.lora_%s.weight"
                return 2.0 * ((h * masks[site] if drop else h) @ leaf[key % "A"].T) @ leaf[key % "B"].T
            x = _llama_block(s, lw, x, extra)
        z = (_rms(x, 1e-5) * w.get_final_norm().double()) @ w.get_lm_head().double().T
        loss = torch.nn.functional.cross_entropy(z.flatten(0, 1), labels.flatten(), ignore_index=-100, reduction="sum") / valid
        loss.backward()
        total += float(loss.detach())
        del x, z, loss
    flat = lambda ts: torch.nn.functional.pad(torch.cat([t.flatten() for t in ts]), (0, padded - sum(t.numel() for t in ts)))
    grad = flat([leaf[n].grad for n in names])
    grad = grad * min(1.0, 1.0 / (float(grad.norm()) + 1e-6))
    # the warm-up schedule begins with a step of rate zero: the moments move, the adapters do not
    return {"loss": total, "adapters": flat([leaf[n].detach() for n in names]), "momentum": 0.1 * grad}
