"""A batch that outgrows its work lists does not wait for the steps queued before
(needs a GPU): an admission in a served stream must not drain the GPU."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_MIXED, Batch, footprint, problems

pytestmark = pytest.mark.gpu


def admit_into_running_batch(ndim, small, large, steps):
    """`small` runs `steps` steps (a few hundred ms); `large`, admitted
    meanwhile, is stepped without waiting for them."""
    import torch
    b = Batch(ndim, precision=PREC_MIXED, arena_bytes=1 << 30, max_sims=4)
    b.add(small, steps, dt_mode=0, dt0=1e-7)
    b.step(1)
    b.sync()
    b.step(steps - 1)
    queued = torch.cuda.Event()
    queued.record(torch.cuda.ExternalStream(b.stream))
    slot = b.add(large, 1, dt_mode=0, dt0=1e-7)
    assert slot is not None
    assert not queued.query(), "the queue ran out before the admission: queue more steps"
    b.step(1)
    assert not queued.query(), "the step call waited for the queued steps"
    b.sync()
    b.close()


def test_growing_lists_do_not_wait_for_queued_steps(need_gpu):
    admit_into_running_batch(2, problems.orszag_tang(128), problems.orszag_tang(1536, ny=1400), 8000)


def test_growing_workspace_does_not_wait_for_queued_steps(need_gpu):
    admit_into_running_batch(3, problems.blast_wave(40, seed=1), problems.blast_wave(120, seed=2), 2500)


def test_lists_of_many_tiny_simulations(need_gpu):
    """Simulations so small that their items outgrow the room that the lists
    start with, before and while steps are queued."""
    from test_gpu_passes import alone
    kw = dict(dt_mode=0, dt0=1e-4)
    probs = [problems.orszag_tang(6 + k % 5, seed=k) for k in range(8)]
    count = 4200
    size = max(footprint(p, PREC_MIXED) for p in probs)
    b = Batch(2, precision=PREC_MIXED, arena_bytes=count * size, max_sims=count)
    slots = [b.add(probs[k % 8], 3, **kw) for k in range(1000)]
    b.step(1)
    slots += [b.add(probs[k % 8], 3, **kw) for k in range(1000, count)]
    b.step(3)
    b.sync()
    want = [alone(p, 3, PREC_MIXED, **kw) for p in probs]
    for k in (0, 999, 1000, 2501, 4199):
        assert np.array_equal(b.state(slots[k]), want[k % 8]), k
    b.close()
