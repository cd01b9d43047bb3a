"""Decode attention of query heads that share key / value heads, one kernel for a group, beside the kernel that takes every head by itself
(reached with the shared heads written out)."""
import pytest
import torch

from dlti_b200.ops import serving as S

pytestmark = pytest.mark.gpu
BF16, F16 = torch.bfloat16, torch.float16


def _paged(rows, bs=16):
    """Contexts [ctx, KV, 128] (pairs of keys and values) as pages in a shuffled order."""
    g = torch.Generator().manual_seed(len(rows))
    need = [-(-k.shape[0] // bs) for k, _ in rows]
    perm, at = torch.randperm(sum(need), generator=g), 0
    kc, vc = (torch.zeros(sum(need), bs, *rows[0][0].shape[1:], dtype=rows[0][0].dtype) for _ in range(2))
    tables = torch.zeros(len(rows), max(need), dtype=torch.int32)
    for i, (k, v) in enumerate(rows):
        own = perm[at:at + need[i]]
        at += need[i]
        tables[i, :need[i]] = own.int()
        for cache, x in ((kc, k), (vc, v)):
            pad = torch.zeros(need[i] * bs, *x.shape[1:], dtype=x.dtype)
            pad[:len(x)] = x
            cache[own] = pad.view(need[i], bs, *x.shape[1:])
    return kc.cuda(), vc.cuda(), tables.cuda(), torch.tensor([len(k) for k, _ in rows], dtype=torch.int32).cuda()


@pytest.fixture(autouse=True)
def together(monkeypatch):
    """At every size, not where it pays alone."""
    monkeypatch.setattr(S, "heads_together", lambda batch, H, KV, reach: H > KV)


def _run(q, rows, H, max_ctx, alone=False):
    kc, vc, tables, ctx = _paged(rows)
    KV = kc.shape[2]
    if alone:
        kc, vc = (x.repeat_interleave(H // KV, 2) for x in (kc, vc))
    return S.paged_decode(q.cuda(), kc, vc, tables, ctx, H, H if alone else KV, 128, max_ctx=max_ctx).double().cpu().view(-1, H, 128)


def _exact(q, rows, H):
    out = []
    for x, (k, v) in zip(q.double().view(len(rows), H, 128), rows):
        k, v = (t.double().repeat_interleave(H // t.shape[1], 1) for t in (k, v))
        out.append(torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", x, k) * 128 ** -0.5, 1), v))
    return torch.stack(out)


@pytest.mark.parametrize("dtype", [BF16, F16])
@pytest.mark.parametrize("max_ctx", [64, 400, 4096])                       # one CTA, a cluster, more than a cluster
def test_weights_keep_their_24_bits(dtype, max_ctx):
    """Three values per column that cancel for the first head of a group leave the errors of the weights: those of fp32 (scores and
    exponentials to about 2^-22), far below those of 16 bits (2^-19)."""
    B, H, KV = 24, 8, 2
    g = torch.Generator().manual_seed(max_ctx)
    q = (torch.randn(B, H * 128, generator=g) * 0.1).to(dtype)
    rows, scale = [], []
    for x in q.double().view(B, KV, H // KV, 128)[:, :, 0]:
        k = torch.randn(3, KV, 128, generator=g).to(dtype)
        p = torch.softmax(torch.einsum("gd,tgd->tg", x, k.double()) * 128 ** -0.5, 0)[..., None]
        v = torch.zeros(3, KV, 128, dtype=dtype)
        v[0] = (1 + torch.rand(KV, 128, generator=g)).to(dtype)
        v[1] = (-p[0] * v[0].double() / p[1]).to(dtype)
        v[2] = (-(p[0] * v[0].double() + p[1] * v[1].double()) / p[2]).to(dtype)
        scale.append(p[0] * v[0].double())
        rows.append((k, v))
    first = lambda y: y.view(B, KV, H // KV, 128)[:, :, 0]
    for alone in (False, True):
        error = first(_run(q, rows, H, max_ctx, alone) - _exact(q, rows, H)) / torch.stack(scale)
        assert error.square().mean().sqrt() < 2 ** -20.5


@pytest.mark.parametrize("dtype", [BF16, F16])
@pytest.mark.parametrize("H,KV,longest", [(8, 4, 90), (16, 4, 1000), (20, 1, 400), (32, 2, 4000)])
def test_no_further_from_64_bits_than_head_by_head(dtype, H, KV, longest):
    g = torch.Generator().manual_seed(H + longest)
    rows = [tuple(torch.randn(n, KV, 128, generator=g).to(dtype) for _ in range(2)) for n in [longest - longest * i // 12 for i in range(8)]]
    q = (2 * torch.randn(8, H * 128, generator=g)).to(dtype)
    want = _exact(q, rows, H)
    error, by_head = ((_run(q, rows, H, longest, alone) - want).norm() for alone in (False, True))
    assert error <= 1.002 * by_head                   # both are the rounding of the output, fp32 errors move a few ties


@pytest.mark.parametrize("dtype", [BF16, F16])
@pytest.mark.parametrize("max_ctx", [64, 400, 4096])
def test_infinite_values(dtype, max_ctx):
    B, H, KV = 16, 8, 2
    g = torch.Generator().manual_seed(1)
    rows = [tuple(torch.randn(n, KV, 128, generator=g).to(dtype) for _ in range(2)) for n in [50 + i for i in range(B)]]
    q = (0.5 * torch.randn(B, H * 128, generator=g)).to(dtype)
    for _, v in rows:
        v[7, :, 3], v[-1, :, 9], v[11, :, 20], v[12, :, 20] = torch.inf, -torch.inf, torch.inf, -torch.inf
    want, got = _exact(q, rows, H), _run(q, rows, H, max_ctx)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    ok = want.isfinite()
    assert (got - want)[ok].norm() <= (4e-3 if dtype == BF16 else 6e-4) * want[ok].norm()      # outputs rounded to 8 and 11 bits


@pytest.mark.parametrize("dtype", [BF16, F16])
@pytest.mark.parametrize("H,KV,splits", [(8, 4, 1), (16, 4, 3), (32, 2, 16)])
def test_the_entry_for_single_heads_stays_itself(dtype, H, KV, splits):
    """dlti_paged_decode gives shared heads the arithmetic of heads with keys and values of their own, at any number of rows."""
    g = torch.Generator().manual_seed(H)
    rows = [tuple(torch.randn(n, KV, 128, generator=g).to(dtype) for _ in range(2)) for n in [700 - 40 * i for i in range(16)]]
    q = torch.randn(16, H * 128, generator=g).to(dtype).cuda()
    got = []
    for share in (H // KV, 1):
        kc, vc, tables, ctx = _paged(rows)
        kc, vc = (x.repeat_interleave(H // KV // share, 2).contiguous() for x in (kc, vc))
        out, ws = torch.empty_like(q), torch.empty(16 * H * splits * 130, device="cuda")
        V, I, L = S._V, S._I, S._L
        f = S._lib.fn("dlti_paged_decode", [V, L, V, V, V, I, V, I, I, I, I, I, S._F, I, V, V, L, I, V])
        p = S._lib.ptr
        S._lib.check(f(p(q), q.stride(0), p(kc), p(vc), p(tables), tables.shape[1], p(ctx), 16, 16, H, kc.shape[2], 128, 128 ** -0.5, splits, p(ws), p(out),
                       out.stride(0), S._lib.dtype_code(dtype), S._lib.stream_ptr()), "paged_decode")
        got.append(out.cpu())
    assert torch.equal(*got)


def test_a_whole_model_either_way(monkeypatch):
    """A bf16 model answering through the engine, its heads together and apart, beside the whole sequences run as prompts: what two ways of
    rounding 16-bit activations differ by."""
    from dlti_b200.models.config import PRESETS
    from dlti_b200.models.llama import ResidentWeights
    from dlti_b200.serve.engine import LLMEngine
    from dlti_b200.serve.model_runner import TPContext, TPWeights
    from dlti_b200.serve.params import Request, SamplingParams
    from dlti_b200.serve.tokenizer import ByteTokenizer
    cfg, rows, calls = PRESETS["tiny-gqa"], 40, []
    full = ResidentWeights.random_init(cfg, "cuda", BF16, seed=3)
    for t in full.all_matrices():
        t.mul_(4.0)
    w = TPWeights(cfg, 0, 1, "cuda", BF16).load_from_full(full)
    g = torch.Generator().manual_seed(2)
    toks = [torch.randint(3, cfg.vocab_size, (20 + 9 * i,), generator=g).tolist() for i in range(rows)]
    request = lambda i: Request(str(i), [], SamplingParams(temperature=0.0))
    got = []
    for way in (True, False, None):
        monkeypatch.setattr(S, "heads_together", lambda *a: calls.append(way) or way)
        eng = LLMEngine(cfg, w, TPContext(), ByteTokenizer(cfg.vocab_size), num_blocks=1200, max_model_len=512, max_num_seqs=rows, max_num_batched_tokens=8192)
        if way is None:
            got.append(eng.replay_step([(request(i), t, list(range(len(t) - 6, len(t)))) for i, t in enumerate(toks)]).view(rows, 6, -1))
            break
        reqs = [request(i) for i in range(rows)]
        eng.replay_step([(r, t[:-6], []) for r, t in zip(reqs, toks)])
        got.append(torch.stack([eng.replay_step([(r, [t[k - 6]], [0]) for r, t in zip(reqs, toks)]) for k in range(6)], 1))
    assert {True, False} <= set(calls) and cfg.num_key_value_heads < cfg.num_attention_heads
    error = lambda a, b: (a - b).double().norm() / b.double().norm()
    apart = error(got[1], got[2])
    assert apart < 0.05 and error(got[0], got[2]) < 1.3 * apart + 2 ** -9 and error(got[0], got[1]) < 0.05
