"""When 32-bit portions are taken by one group of threads a block (CPU: the rule alone)."""

import pytest

from edgerag_b200.ops import kernels


@pytest.mark.parametrize("lens,past,reach,heads,one", [
    ([32] * 16, 0, 0, 32, True), ([32] * 8, 0, 0, 32, True), ([32] * 16, 100, 0, 32, True), ([333] * 2, 0, 0, 32, True), ([40] * 4, 0, 0, 32, True),
    ([333], 0, 0, 9, False), ([96], 500, 0, 32, False), ([2048], 0, 0, 9, False), ([333] * 2, 500, 0, 32, True), ([32] * 16, 0, 0, 9, False),
    ([2048], 0, 0, 32, True), ([333], 500, 0, 32, False), ([40] * 4, 500, 0, 32, False), ([512], 4000, 64, 16, False)])
def test_where_one_group_pays(lens, past, reach, heads, one):
    lasts = tuple(past + n - 1 for n in lens)
    assert kernels.one_group_pays(tuple(lens), lasts, reach, heads, 148) is one
