"""Kernels of decode rows whose work is cut by the sizes of a step: recurrent states moved several columns a lane, each against the
op's restatement in plain PyTorch."""
import pytest
import torch

from dlti_b200.ops import delta as D
from dlti_b200.ops import stack as K

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def _rows(n, device):
    """n decode rows; every fifth sequence is new (nothing carried), every seventh has no state slot (padding)."""
    i = torch.arange(n, dtype=torch.int32)
    ctx = torch.where(i % 5 == 0, torch.ones_like(i), i + 2)
    state = torch.where(i % 7 == 3, torch.full_like(i, -1), n - 1 - i)
    t = lambda x: x.to(device)
    return K.Rows(t(ctx - 1), t(i), t(i.long()), t(ctx), None, torch.zeros(n, 1, dtype=torch.int32, device=device), t(state), n, 0, 64)


def _act(x, device, dtype):
    out = K.act(x.shape[0], x.shape[1], dtype, device)
    return out.copy_(x)


# two columns and one per lane, on both sides of a wave of CTAs; last blocks and last rows partly filled; every row count of a warp
SIZES = [(8, 128, 70, 40), (4, 20, 44, 160), (8, 60, 33, 80), (4, 200, 100, 27), (4, 200, 100, 28), (2, 128, 64, 148), (2, 128, 64, 149), (4, 128, 128, 40), (4, 128, 256, 40), (8, 30, 132, 40), (4, 72, 64, 40), (4, 20, 44, 80), (4, 128, 70, 40), (8, 256, 96, 40), (3, 64, 33, 60),
         (2, 300, 40, 80), (2, 128, 128, 3)]


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("heads,N,P,n", SIZES)
@pytest.mark.parametrize("kind", ["mamba2", "lightning", "mlstm", "delta"])
def test_recurrences_of_decode_rows(kind, heads, N, P, n, dtype):
    g = torch.Generator().manual_seed(N + P)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k, v, z = (rnd(n, w).to(BF16).float() for w in (heads * N, heads * N, heads * P, 2 * heads))
    state, vec = rnd(n, heads, N, P), rnd(n, heads, 1, N + 1).repeat(1, 1, -(-P // 32), 1).flatten(2)
    bias, A_log, skip, fall = rnd(heads), rnd(heads) * 0.5, rnd(heads), torch.rand(heads, generator=g)
    got = {}
    for device in ("cpu", "cuda"):
        t = lambda x: x.to(device)
        rows, st, vc, dt = _rows(n, device), state.to(device, copy=True), vec.to(device, copy=True), F32 if device == "cpu" else dtype
        a = [_act(x, device, dt) for x in (q, k, v)]
        if kind == "delta":
            out = D.delta_scan(*a, _act(z, device, F32), t(A_log), t(bias), st, rows, heads, heads, N, P)
        elif kind == "mlstm":
            out = K.mlstm_scan(*a, _act(z, device, F32), t(torch.cat([bias, bias])), 15.0, st, vc, rows, heads, N, P)
        else:
            dec = K.Decay(const=t(fall)) if kind == "lightning" else K.Decay(dt=_act(z[:, :heads], device, dt), dt_bias=t(bias), A_log=t(A_log), D=t(skip))
            out = K.linear_scan(*a, dec, st, rows, heads, heads, N, P, silu=kind == "lightning" and dtype == F32)
        got[device] = out.float().cpu(), st.cpu(), vc.cpu()
    live = (_rows(n, "cpu").state >= 0)
    for x, y, tol in zip(got["cuda"], got["cpu"], (1e-5 if dtype == F32 else 4e-3, 1e-5, 1e-5)):     # fp32 sums; outputs rounded to 8 bits
        x, y = (x[live], y[live]) if x.shape[0] == n and x.dim() == 2 else (x, y)                     # rows without a slot: no result
        assert (x.double() - y.double()).norm() <= tol * y.double().norm()


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
def test_fed_ids(n):
    from dlti_b200.ops import serving as S
    g = torch.Generator().manual_seed(n)
    ids, sampled = torch.randint(0, 1 << 40, (n,), generator=g), torch.randint(0, 1 << 40, (300,), generator=g)
    src = torch.randint(-1, 300, (n,), generator=g, dtype=torch.int32)
    assert torch.equal(S.feed_ids(ids.cuda(), src.cuda(), sampled.cuda()).cpu(), S.feed_ids(ids, src, sampled))


@pytest.mark.parametrize("kind", ["mamba2", "lightning", "mlstm"])
@pytest.mark.parametrize("lens,carried", [((1024,), 0), ((1025,), 7), ((1600, 30, 700), 5), ((512, 1537), 0)])
@pytest.mark.parametrize("N,P", [(64, 32), (128, 40), (200, 24)])
def test_prompts_in_segments(kind, N, P, lens, carried, monkeypatch):
    """Segments of a prompt side by side give what the chain of all chunks gives; both have the same products, in another order."""
    heads, T, dev = 2, 2 + sum(lens), "cuda"
    g = torch.Generator().manual_seed(N + T)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k, v = (_act(x, dev, BF16) for x in (rnd(T, heads * N), rnd(T, heads * N) * 0.2, rnd(T, heads * P)))
    z = rnd(T, 2 * heads)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    n = 2 + len(lens)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    rows = K.Rows(i32([0] * T), i32([0] * T), i32([0] * T).long(), i32([9, 1] + [x + carried for x in lens]), i32(cu), i32([[0]] * n),
                  i32(list(range(n, 0, -1))), 2, max(lens), 4096)
    assert K._scan_workspace(rows, len(lens), heads, N, P, dev) is not None
    state, vec = rnd(n + 1, heads, N, P).to(dev), rnd(n + 1, heads, 1, N + 1).repeat(1, 1, -(-P // 32), 1).flatten(2).to(dev)
    bias, A_log = torch.linspace(-4, 0, heads, device=dev), torch.linspace(-1, 1, heads, device=dev)
    out = []
    for split in (True, False):
        if not split:
            monkeypatch.setattr(K, "_scan_workspace", lambda *a: None)
        st, vc = state.clone(), vec.clone()
        if kind == "mlstm":
            y = K.mlstm_scan(q, k, v, _act(z, dev, F32), torch.cat([bias, 4 - bias]), 15.0, st, vc, rows, heads, N, P)
        elif kind == "lightning":
            y = K.linear_scan(q, k, v, K.Decay(const=torch.tensor([0.999, 0.9], device=dev)), st, rows, heads, heads, N, P)
        else:
            dec = K.Decay(dt=_act(z[:, :heads], dev, BF16), dt_bias=bias, A_log=A_log, D=bias)
            y = K.linear_scan(q, k, v, dec, st, rows, heads, heads, N, P)
        out.append((y.double(), st.double(), vc.double()))
    for a, b, tol in zip(*out, (2e-3, 2e-5, 2e-5)):              # outputs rounded to 8 bits; states: 16 bits and more in every product
        assert bool(torch.isfinite(a).all()) and (a - b).norm() <= tol * b.norm()
    assert torch.equal(out[0][1][0], state[0].double())


@pytest.mark.parametrize("dtype,tol", [(BF16, 4e-3), (torch.float16, 6e-4)])       # outputs rounded to 8 and 11 bits
@pytest.mark.parametrize("max_ctx", [64, 400, 4096])                               # one CTA, a cluster, more than a cluster
@pytest.mark.parametrize("H,KV,bs", [(4, 2, 16), (8, 2, 16), (16, 1, 24), (20, 1, 16), (51, 3, 16)])
def test_decode_attention_of_shared_heads(H, KV, bs, max_ctx, dtype, tol, monkeypatch):
    from dlti_b200.ops import serving as S
    monkeypatch.setattr(S, "heads_together", lambda *a: True)        # also at sizes that go head by head
    g = torch.Generator().manual_seed(H)
    ctx = [c for c in (1, 15, 63, 64, 65, 129, 400, 700, 4096) if c <= max_ctx]
    ctx += [37] * (-(-64 // H) - len(ctx))
    nb = [-(-c // bs) for c in ctx]
    tables, kc, vc = torch.zeros(len(ctx), max(nb), dtype=torch.int32), *(torch.randn(sum(nb), bs, KV, 128, generator=g).to(dtype) for _ in range(2))
    perm, at = torch.randperm(sum(nb), generator=g).int(), 0
    for i, n in enumerate(nb):
        tables[i, :n] = perm[at:at + n]
        at += n
    q, lens = torch.randn(len(ctx), H * 128, generator=g).to(dtype) * 2, torch.tensor(ctx, dtype=torch.int32)
    want = S.paged_decode_ref(q.float(), kc.float(), vc.float(), tables, lens, H, KV, 128, 128 ** -0.5)
    got = S.paged_decode(q.cuda(), kc.cuda(), vc.cuda(), tables.cuda(), lens.cuda(), H, KV, 128, max_ctx=max_ctx).cpu()
    assert bool(((got.float() - want).norm(dim=1) <= tol * want.norm(dim=1)).all())


@pytest.mark.parametrize("n,d", [(1, 8), (5, 40), (300, 2048), (7, 4104)])
def test_embedded_rows_by_pieces(n, d):
    from dlti_b200.ops import streams as H
    g = torch.Generator().manual_seed(d)
    table, ids = torch.randn(50, d, generator=g).to(BF16), torch.randint(0, 50, (n,), generator=g)
    x, h = K.embed_rows(ids.cuda(), table.cuda())
    assert torch.equal(x.cpu(), table[ids].float()) and torch.equal(h.cpu(), table[ids])
    assert torch.equal(H.embed_streams(ids.cuda(), table.cuda(), 3, 2.5).cpu(), (table[ids].float() * 2.5)[:, None].expand(n, 3, d))


@pytest.mark.parametrize("n,w", [(1, 8), (5, 2048), (6, 2056), (131, 6144)])
def test_silu_of_rows(n, w):
    x = torch.randn(n, w + 16, generator=torch.Generator().manual_seed(w)).to(BF16).cuda()
    want = x.clone()
    want[:, :w] = torch.nn.functional.silu(x[:, :w].float()).to(BF16)
    K.silu_rows_(x[:, :w])
    assert torch.equal(x[:, w:], want[:, w:]) and (x.float() - want.float()).abs().max() <= 2 ** -8 * want.float().abs().max()
