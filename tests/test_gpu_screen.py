"""The FP64 wave-speed screen keeps a NaN of the exact speeds (needs a GPU).

Where sound and Alfven speed along a dimension agree, the discriminant of the
fast speed is zero but for rounding, and where rounding makes it negative the
speed is NaN: the step reports SMAUG_ERR_NONFINITE.  That must not depend on
what the thread has seen before: the state here is a layer of such cells behind
layers whose speeds are ten times theirs, deep enough that every thread of the
advance pass meets a fast cell first, and the same layer by itself.
"""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, Batch, Engine, SmaugError, problems

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0
NX = 128        # with ghosts: a divisor of any block count times 256, so a thread keeps its column
FAST = 5120     # rows before the layer: more than twice the cells that are in flight at once


def layers(fast: int, slow: int, aligned: bool = True):
    """A static equilibrium, uniform along x: `fast` rows of thin hot gas
    without field, then `slow` rows of dense gas whose field along x gives it a
    sound speed equal to its Alfven speed (aligned=False: four times it)."""
    prob = problems.orszag_tang(NX - 4, ny=fast + slow)
    rng = np.random.default_rng(7)
    rho = np.full(fast + slow, 0.01)
    rho[fast:] = 1.0 + rng.random(slow)
    b = np.zeros(fast + slow)
    # p + B^2 / 2 = 1 everywhere, gamma p = B^2 (or 16 B^2) in the slow rows
    b[fast:] = np.sqrt(1.0 / ((1.0 if aligned else 16.0) / GAMMA + 0.5))
    p = 1.0 - 0.5 * b * b
    row = np.r_[fast + slow - 2:fast + slow, 0:fast + slow, 0:2]  # periodic ghosts
    w = np.zeros_like(prob.w)
    w[0] = rho[row][:, None]
    w[3] = (p / (GAMMA - 1.0) + 0.5 * b * b)[row][:, None]
    w[4] = b[row][:, None]
    prob.w = w
    prob.gamma = GAMMA
    prob.hyperdif = 0
    return prob


def stepped(prob):
    e = Engine(prob, rk4=True, precision=PREC_FP64, dt_mode=0, dt0=1e-6)
    e.step(2)
    try:
        e.sync()
    finally:
        e.close()


def test_negative_discriminant_is_reported_behind_faster_cells(need_gpu):
    with pytest.raises(SmaugError, match="non-finite"):
        stepped(layers(8, 128))
    with pytest.raises(SmaugError, match="non-finite"):
        stepped(layers(FAST, 128))
    stepped(layers(FAST, 128, aligned=False))  # the same layers without the coincidence are an ordinary state


def test_negative_discriminant_is_reported_in_a_batch(need_gpu):
    b = Batch(2, precision=PREC_FP64, arena_bytes=1 << 30, max_sims=3)
    good = b.add(layers(FAST, 128, aligned=False), 2, dt_mode=0, dt0=1e-6)
    bad = b.add(layers(FAST, 128), 2, dt_mode=0, dt0=1e-6)
    b.step(2)
    rc, slot, _ = b.status()
    assert rc != 0 and slot == bad != good
    b.close()
