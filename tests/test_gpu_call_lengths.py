"""A context's calls of any length give the bits of its stages one by one: the
graphs of 1 and of 16 steps are captured when a call first needs them (needs a
GPU)."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Engine, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: problems.orszag_tang(40, seed=3), lambda: problems.blast_wave(16, seed=4)],
                         ids=["2d", "3d"])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("calls", [(4, 16, 3), (16, 1), (19,), (0, 32, 5), (1, 18)], ids=str)
def test_calls_of_any_length(need_gpu, make, prec, calls):
    import torch
    a, b = (Engine(make(), precision=prec) for _ in range(2))
    s = torch.cuda.Stream()
    for k, n in enumerate(calls):
        l0 = a.launches
        if k % 2:
            a.step_on(n, s.cuda_stream)
        else:
            a.step(n)
        l1 = b.launches
        for _ in range(n):
            for stage in (1, 2, 3, 4):
                b.stage(stage)
        # inside a graph one kernel ends a step and opens the next
        assert a.launches - l0 == (b.launches - l1) - 15 * (n // 16)
    a.sync()
    b.sync()
    assert np.array_equal(a.state(), b.state())
    assert a.scalars() == b.scalars()
    a.close()
    b.close()
