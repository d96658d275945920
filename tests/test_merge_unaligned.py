"""GPU parity of the merge with inputs off the 16-byte boundaries, one array or
all of them: one tile, ragged tiles, few tiles a CTA and many."""
from __future__ import annotations

import pytest

from tests.test_merge_order import CASES, SMS, check_merge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,value", CASES)
def test_unaligned_inputs(cuda, key, value):
    tile = 4096 if key[1:] == "32" else 2048
    sizes = [(3, 5), (tile - 1, 2), (tile, tile + 1), (5 * tile + 7, 11), (20 * tile + 1, 21 * tile),
             (tile * SMS * 10, tile * SMS * 9 + 1), (tile * SMS * 25 + 3, tile * SMS * 26)]
    where = [(1, 0, 0, 0, 0), (0, 1, 0, 0, 0), (1, 1, 1, 1, 0), (1, 0, 0, 1, 1)]
    if value is not None:
        where += [(0, 0, 1, 0, 0), (0, 0, 0, 1, 0)]
    for na, nb in sizes:
        for offsets in where if na < 40 * tile else where[2:3]:
            check_merge(key, value, na, nb, 1 << 30, cuda, offsets)
            check_merge(key, value, na, nb, 9, cuda, offsets)
