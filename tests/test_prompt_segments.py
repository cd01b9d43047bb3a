"""Long prompts through the recurrences, cut into segments that run side by side: the same bits as without segments."""
import pytest
import torch

from dlti_b200.ops import _lib
from dlti_b200.ops import stack as K

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def _act(x, dtype):
    return K.act(x.shape[0], x.shape[1], dtype, "cuda").copy_(x)


def _whole(monkeypatch):
    """Calls of the split forms go to those that never cut."""
    get, plain = _lib.fn, {"dlti_linear_scan_split": "dlti_linear_scan_chunked", "dlti_mlstm_scan_split": "dlti_mlstm_scan"}

    def fn(name, types, *a, **kw):
        if name not in plain:
            return get(name, types, *a, **kw)
        f = get(plain[name], types[:-3] + types[-1:], *a, **kw)
        return lambda *args: f(*args[:-3], args[-1])
    monkeypatch.setattr(K._lib, "fn", fn)


# two segments and sixteen, sequences too short for any, a carried state, sizes that are no multiple of a tile, one and more slices
SHAPES = [(2, 64, 32, (1024,), 0), (2, 64, 32, (9000,), 3), (2, 128, 40, (1600, 30, 700), 5), (3, 200, 24, (512, 1537), 0), (2, 256, 32, (2049,), 1),
          (16, 128, 128, (4096,), 0), (64, 128, 64, (1030,), 2), (36, 128, 128, (1024,), 0)]


@pytest.mark.parametrize("kind", ["mamba2", "lightning", "mlstm"])
@pytest.mark.parametrize("heads,N,P,lens,carried", SHAPES)
def test_segments_change_no_bit(kind, heads, N, P, lens, carried, monkeypatch):
    T = 2 + sum(lens)
    g = torch.Generator().manual_seed(N + T)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k, v = (_act(x, BF16) for x in (rnd(T, heads * N), rnd(T, heads * N) * 0.2, rnd(T, heads * P)))
    z = rnd(T, 2 * heads)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    n = 2 + len(lens)
    rows = K.Rows(i32([0] * T), i32([0] * T), i32([0] * T).long(), i32([9, 1] + [x + carried for x in lens]), i32([sum(lens[:i]) for i in range(len(lens) + 1)]),
                  i32([[0]] * n), i32(list(range(n, 0, -1))), 2, max(lens), 1 << 14)
    state = rnd(n + 1, heads, N, P).cuda()
    vec = rnd(n + 1, heads, 1, N + 1).repeat(1, 1, -(-P // 32), 1).flatten(2).cuda()
    bias, A_log = torch.linspace(-4, 0, heads, device="cuda"), torch.linspace(-1, 1, heads, device="cuda")
    out = []
    for _ in range(2):
        st, vc = state.clone(), vec.clone()
        if kind == "mlstm":
            y = K.mlstm_scan(q, k, v, _act(z, F32), torch.cat([bias, 4 - bias]), 15.0, st, vc, rows, heads, N, P)
        elif kind == "lightning":
            y = K.linear_scan(q, k, v, K.Decay(const=torch.linspace(0.9, 0.999, heads, device="cuda")), st, rows, heads, heads, N, P)
        else:
            y = K.linear_scan(q, k, v, K.Decay(dt=_act(z[:, :heads], BF16), dt_bias=bias, A_log=A_log, D=bias), st, rows, heads, heads, N, P)
        out.append((y, st, vc))
        _whole(monkeypatch)
    assert bool(torch.isfinite(out[0][0].float()).all())
    for a, b in zip(*out):
        assert torch.equal(a, b)
