"""The form of a key sort: one launch whose blocks all have to be resident, or
a launch per pass where they cannot be."""
import ctypes

import pytest

from hostcheck import build as hb


@pytest.mark.parametrize("n,cooperative,sms,per_sm,blocks", [
    (1, 1, 152, 2, 1), (2048, 1, 152, 2, 1), (2049, 1, 152, 2, 2), (1 << 22, 1, 152, 2, 152),
    ((1 << 22) + 1, 1, 152, 2, 0),   # beyond the line between the forms
    (100_000, 0, 152, 2, 0),         # no cooperative launches
    (100_000, 1, 152, 0, 0),         # a block does not fit an SM
    (100_000, 1, 8, 1, 8), (1 << 20, 1, 400, 4, 256), (0, 1, 152, 2, 0),
])
def test_blocks_are_resident_or_the_passes_are_launched(n, cooperative, sms, per_sm, blocks):
    lib = ctypes.CDLL(hb._build("hc_sort", "hostcheck_sort.cpp"))
    assert lib.hc_sort_blocks(ctypes.c_int64(n), cooperative, sms, per_sm) == blocks
