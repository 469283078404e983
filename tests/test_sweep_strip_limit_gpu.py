"""``set_tiling`` takes strip heights that are not multiples of the kernel's 8-row turn as the most rows of
a work item: no item is taller, and the cut changes no bits."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_sweep_gpu import _members, _scales, _sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9, 12, 23, 100])
def test_strips_are_at_most_strip_rows(cuda_lib, rows):
    members = _members(sizes=[(512, 512)] * 20 + [(512, 101)] * 3)
    for m in members:
        m["physics"] = members[0]["physics"]
    outs = []
    for r in (8, rows):
        eng = _sweep(members)
        eng.set_tiling(512, r)
        # one strip an item, as the members are as wide as a block
        assert eng.tiling["items"] >= sum(-(-m["ny"] // r) for m in members)
        eng.advance(0, 2, _scales(members, 2))
        outs.append(eng.get_state())
        eng.close()
    for got, want in zip(outs[1], outs[0]):
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
