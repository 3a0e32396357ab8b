"""The 3-D tuner times each tile shape once: variants that launch the same get one
time, and the choice among them is the first (needs a GPU)."""
from __future__ import annotations

import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Batch, problems

pytestmark = pytest.mark.gpu

ALIKE = [(0, 3, 5), (1, 4), (2,), (6, 8), (7, 9)]


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_variants_alike_are_timed_once(need_gpu, precision):
    b = Batch(3, precision=precision, arena_bytes=256 << 20, max_sims=2)
    b.add(problems.blast_wave(40, seed=1), 2)
    variant, ms = b.tune(3)
    assert len(ms) == 10 and all(m > 0 for m in ms)
    for group in ALIKE:
        assert len({ms[v] for v in group}) == 1
    assert variant in [g[0] for g in ALIKE] and ms[variant] == min(ms)
    for v in range(10):  # every number stays valid
        b.set_variant(v)
    b.step(2)
    b.sync()
    b.close()
