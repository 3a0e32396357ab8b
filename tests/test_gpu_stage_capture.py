"""A step captured stage by stage from the context's own stream into a caller's
graph, with the caller's copies between the stages, replays to the same bits as
smaug_step (needs a GPU).  The stage kernels carry a dependent-launch attribute,
which behind a copy has to fall back to a full dependency."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Engine, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("make", [lambda: problems.orszag_tang(40, seed=3), lambda: problems.blast_wave(12, seed=4)],
                         ids=["2d", "3d"])
def test_captured_stages_with_copies_between(need_gpu, make, prec):
    import torch
    a, b = (Engine(make(), precision=prec, dt_mode=0, dt0=1e-4) for _ in range(2))
    for _ in range(4):
        a.step(1)
    s = torch.cuda.ExternalStream(b.stream)
    x = torch.arange(4096.0, device="cuda")
    y = torch.zeros_like(x)
    b.step(1)  # the kernels are loaded before the capture
    b.sync()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        for k in (1, 2, 3, 4):
            y.copy_(x)
            b.stage(k)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    b.sync()
    a.sync()
    assert np.array_equal(a.state(), b.state())
    assert torch.equal(x, y)
    a.close()
