"""Token ids that a caller gives, as arrays."""
import numpy as np
import pytest

from dlti_b200.serve.engine import _id_array


@pytest.mark.parametrize("toks", [[], [3], list(range(1000)), tuple(range(5)), [np.int64(7), np.int32(2)], np.arange(4), [2.0, True], b"abc", range(3)])
def test_ids_as_they_were_given(toks):
    a = _id_array(toks)
    assert a.dtype == np.int64 and a.tolist() == [int(t) for t in toks]


@pytest.mark.parametrize("t", [-1, -(1 << 70), 1 << 70, (1 << 63) - 1])
def test_ids_outside_stay_outside(t):
    a = _id_array([1, t])
    assert a.min() < 0 or a.max() >= 1 << 62
