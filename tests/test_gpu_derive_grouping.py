"""The 3-D derive pass loads the state of one or of four cells at a time,
depending on how many blocks it has: a small simulation gives the same bits
alone (few blocks) and beside a large one (many) (needs a GPU)."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Batch, problems

from test_gpu_passes import alone

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_small_simulation_alone_and_beside_a_large_one(need_gpu, precision):
    probs = [problems.blast_wave(64, seed=1), problems.blast_wave(6, seed=2), problems.blast_wave(17, seed=3),
             problems.atmosphere(21, 9, 6, noise=1e-3, seed=4)]
    b = Batch(3, precision=precision, arena_bytes=1 << 30, max_sims=4)
    kws = [dict(dt_mode=0, dt0=1e-2) if p.name == "atmosphere" else dict(dt_mode=0, dt0=2e-4) for p in probs]
    slots = [b.add(p, 2, **kw) for p, kw in zip(probs, kws)]
    b.step(2)
    b.sync()
    for p, s, kw in list(zip(probs, slots, kws))[1:]:
        assert np.array_equal(b.state(s), alone(p, 2, precision, **kw)), p.n
    b.close()
