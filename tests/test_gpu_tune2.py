"""The 2-D mixed tuner on few tiles (needs a GPU): the 16x16 variants launch one
kernel there, so they get one time and the default stands for them, not whichever
of them noise made the fastest: the batch may grow under the choice."""
from __future__ import annotations

import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Batch, problems

pytestmark = pytest.mark.gpu

SQUARE = (0, 4, 6, 8)  # the 16x16 variants, by occupancy target


@pytest.mark.parametrize("precision,side,alike", [(PREC_MIXED, 64, True), (PREC_MIXED, 640, False),
                                                  (PREC_FP64, 64, False)])
def test_square_tiles_on_few_tiles_are_one_variant(need_gpu, precision, side, alike):
    b = Batch(2, precision=precision, arena_bytes=512 << 20, max_sims=2)
    b.add(problems.orszag_tang(side, seed=1), 2)
    variant, ms = b.tune(3)
    assert len(ms) == 11 and all(m > 0 for m in ms)
    assert (len({ms[v] for v in SQUARE}) == 1) == alike
    assert not alike or variant not in (0, 4, 8)
    b.step(2)
    b.sync()
    b.close()
