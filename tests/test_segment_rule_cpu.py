"""How many segments a long prompt is cut into for the recurrences: a rule of sizes alone, which needs no GPU."""
import ctypes as C

import pytest

from dlti_b200.ops import _lib


def _segments(longest, nseq, heads, N, P):
    """How many segments the workspace is for."""
    floats = _lib.fn("dlti_scan_workspace", [C.c_int] * 5, restype=C.c_longlong)(longest, nseq, heads, N, P)
    rows = next((r for r in (64, 128, 256) if N <= r), 1)
    per = nseq * heads * -(-P // 32) * (rows * 34 + 4)
    assert floats % per == 0
    return max(1, floats // per)


# (longest, sequences, heads, N, P) -> segments on 148 SMs: by the room of the SMs, by the length, whole where two fit no SM of their own and are short
RULE = [((8192, 1, 16, 128, 128), 4), ((8192, 1, 24, 128, 128), 3), ((5119, 1, 32, 128, 128), 1), ((5120, 1, 64, 128, 64), 2), ((1024, 1, 16, 128, 128), 2),
        ((1024, 1, 24, 128, 128), 1), ((1023, 1, 4, 64, 64), 1), ((1 << 20, 1, 1, 64, 32), 16), ((8192, 2, 8, 256, 256), 1), ((8192, 1, 8, 256, 256), 2),
        ((8192, 1, 12, 256, 256), 1), ((8192, 1, 4, 200, 256), 4), ((8192, 1, 4, 300, 64), 1)]


@pytest.mark.parametrize("sizes,segments", RULE)
def test_segments_where_they_pay(sizes, segments):
    if _lib.gpu_lib().dlti_sm_count() != 148:
        pytest.skip("the rule's lines lie at the number of SMs")
    assert _segments(*sizes) == segments
