"""What the FP64 3-D passes add to a state, field by field, against the oracle
(needs a GPU).

The state's own norm hides a small field behind a large one and a small change
behind a large value, so the increments over three steps are compared, each
field over its own norm.  The bar is rounding alone: 1e-12 of the increment,
and 256 units of 2^-53 of what the field's increments are formed from (the
field, and per step the largest flux along each dimension times dt / dx).  The
same bar refuses every field that was left as it was, and every field without
its hyperdiffusion: both are asserted on the oracle, so that the bar is known to
hold the terms it is meant to hold.
"""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, Engine, problems

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
STEPS = 3
INNER = (slice(2, -2),) * 3


def norm(a):
    return float(np.linalg.norm(a[INNER]))


def oracle_state(prob, dt, hyperdif):
    keep = prob.hyperdif
    prob.hyperdif = hyperdif
    o = Oracle(prob, dt_fixed=dt)
    o.step(STEPS, rk4=True, dt_mode=0)
    prob.hyperdif = keep
    return o.w.copy()


def rounding_scale(prob, w, dt):
    """Per evolved field: what its increments are formed from (norms)."""
    rho = w[0] + w[9]
    v = [w[1 + k] / rho for k in range(3)]
    b, bb = w[5:8], w[10:13]
    bt = [b[k] + bb[k] for k in range(3)]
    e = np.abs(w[4]) + np.abs(w[8])
    press = (prob.gamma + 1.0) * (e + sum(x * x for x in bt) + sum(w[1 + k] * v[k] for k in range(3)))
    speed = np.sqrt(press / rho) + sum(np.abs(x) for x in v)  # at least every wave speed
    c = STEPS * dt * sum(1.0 / d for d in prob.dx)
    field = sum(np.abs(x) for x in bt)
    scale = [np.abs(w[0]) + c * rho * speed]
    scale += [np.abs(w[1 + k]) + c * (press + rho * speed * speed) for k in range(3)]
    scale += [e + c * speed * (press + field * field)]
    scale += [np.abs(b[k]) + c * speed * field for k in range(3)]
    return [norm(s) for s in scale]


@pytest.mark.parametrize("make", [
    lambda: problems.blast_wave(6, seed=2),
    lambda: problems.blast_wave(33, seed=2),
    lambda: problems.atmosphere(37, 9, 6, noise=1e-3, seed=3),
    lambda: problems.atmosphere(12, 34, 13, noise=1e-3, seed=4),
], ids=["blast6", "blast33", "atmosphere37x9x6", "atmosphere12x34x13"])
def test_3d_increments_against_the_oracle(need_gpu, make):
    prob = make()
    dt = 1e-2 if prob.name == "atmosphere" else 2e-4
    w0 = prob.w.copy()
    ref = {h: oracle_state(prob, dt, h) for h in (1, 0)}
    scale = rounding_scale(prob, w0, dt)
    held = {"left": 0, "hyperdif": 0}
    for hyperdif in (1, 0):
        prob.hyperdif = hyperdif
        e = Engine(prob, rk4=True, precision=PREC_FP64, dt_mode=0, dt0=dt)
        e.step(STEPS)
        e.sync()
        w = e.state()
        e.close()
        for f in range(8):
            inc = ref[hyperdif][f] - w0[f]
            bar = 1e-12 * norm(inc) + 256 * EPS * scale[f]
            err = norm(w[f] - ref[hyperdif][f])
            assert err <= bar, (f, hyperdif, err, bar)
            if hyperdif:
                held["left"] += norm(inc) > 10 * bar
                held["hyperdif"] += norm(ref[1][f] - ref[0][f]) > 10 * bar
    assert held == {"left": 8, "hyperdif": 8}
