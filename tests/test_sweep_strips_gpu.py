"""Strips of the uneven sweep cut to fill the last wave of blocks: heights that do not divide the
members' rows, a last strip of one row, and more items than blocks.  The cut changes no bits, so the
oracle is the same set of members under the shortest tiling, and one member stepped alone."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_sweep_gpu import _members, _scales, _sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,rows", [([(512, 333)] * 18 + [(256, 129)] * 6 + [(128, 77)] * 5, (64, 333)),
                                        ([(512, 41)], (16, 40)), ([(128, 9), (64, 8), (256, 5)], (8, 1024)),
                                        ([(512, 512)] * 40, (48, 512))])
def test_cut_strips_change_no_bits(cuda_lib, sizes, rows):
    members = _members(sizes=sizes)
    for m in members:  # _members scales its physics with the index: keep it moderate for many members
        m["physics"] = members[0]["physics"]
    steps = 3
    ref = _sweep(members)
    ref.set_tiling(512, 8)
    ref.advance(0, steps, _scales(members, steps))
    want = ref.get_state()
    ref.close()
    eng = _sweep(members)
    for r in rows:
        eng.set_tiling(512, r)
        tiling = eng.tiling
        assert tiling["strip_rows"] == r
        whole = sum(-(-m["ny"] // r) for m in members)
        assert tiling["items"] <= -(-whole // tiling["blocks"]) * tiling["blocks"]
        eng.set_state([m["psi"] for m in members], [m["res"] for m in members])
        eng.advance(0, steps, _scales(members, steps))
        got = eng.get_state()
        for m in range(len(members)):
            assert np.array_equal(got[0][m], want[0][m]) and np.array_equal(got[1][m], want[1][m]), (r, m)
    eng.close()
