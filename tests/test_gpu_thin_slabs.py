"""A 3-D context on a device with little memory left gets a small workspace, in
slabs of one plane, and the bits of a context with plenty (needs a GPU; most of
its memory is set aside, untouched, while the second context is made)."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_MIXED, Engine, footprint, problems

pytestmark = pytest.mark.gpu


def test_one_plane_slabs_give_the_same_bits(need_gpu):
    import torch
    # 120 000 cells a plane: four planes and their halos take 156 MB of
    # workspace, one plane with its halos 95 MB
    prob = problems.atmosphere(396, 296, 8, noise=1e-3, seed=3)
    kw = dict(precision=PREC_MIXED, dt_mode=0, dt0=1e-2)
    e = Engine(prob, **kw)
    e.step(3)
    e.sync()
    want, scalars = e.state(), e.scalars()
    e.close()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    try:
        filler = torch.empty(free - footprint(prob, PREC_MIXED) - (125 << 20), dtype=torch.uint8, device="cuda")
    except torch.cuda.OutOfMemoryError:
        pytest.skip("the device's memory is in use")
    e = Engine(prob, **kw)
    left, _ = torch.cuda.mem_get_info()
    del filler
    torch.cuda.empty_cache()
    assert left < 60 << 20  # the workspace of whole slabs would not have fitted
    e.step(3)
    e.sync()
    assert np.array_equal(e.state(), want)
    assert e.scalars() == scalars
    e.close()
