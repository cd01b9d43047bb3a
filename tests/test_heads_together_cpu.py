"""Which decode attention a step's sizes get."""
import pytest

from dlti_b200.ops.serving import heads_together


# rows, heads, key / value heads, keys that a context may have
@pytest.mark.parametrize("sizes,together", [((64, 16, 16, 4096), False), ((1, 32, 8, 4096), False), ((3, 16, 4, 4096), False), ((4, 16, 4, 256), True),
                                            ((4, 16, 4, 255), False), ((16, 16, 4, 192), False), ((64, 16, 4, 192), True), ((64, 16, 8, 192), False),
                                            ((32, 32, 8, 192), True), ((31, 32, 8, 192), False), ((64, 16, 8, 512), True), ((2, 32, 1, 1024), True)])
def test_rule(sizes, together):
    assert heads_together(*sizes) == together
