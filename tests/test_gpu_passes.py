"""The stage kernels' routes at the sizes where they change (needs a GPU).

2-D mixed: up to two tiles per SM run one cell per thread, larger batches pairs
of cells; both give the same bits, on tiles cut anywhere.  3-D: the derive,
faces and terms passes on the smallest grids, on ragged tiles and face runs,
with and without live backgrounds and hyperdiffusion, against the oracle; and a
batch whose workspace needs more than one group of slabs against its members
alone.  Bars as in test_gpu_parity (FP64 1e-6) and test_gpu_mixed (1e-5),
relative L2 per field; a field below 1e-3 of the largest counts against that.
"""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import PREC_FP64, PREC_MIXED, Batch, Engine, problems

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def field_errors(w, ref, nw):
    sl = (slice(None),) + tuple(slice(2, -2) for _ in range(w.ndim - 1))
    a, b = w[sl][:nw], ref[sl][:nw]
    norms = np.array([np.linalg.norm(b[f]) for f in range(nw)])
    scale = np.where(norms > 1e-3 * norms.max(), norms, norms.max())
    return np.array([np.linalg.norm(a[f] - b[f]) for f in range(nw)]) / scale


def alone(prob, steps, precision, **kw):
    e = Engine(prob, rk4=True, precision=precision, **kw)
    e.step(steps)
    e.sync()
    w = e.state()
    e.close()
    return w


def test_pairs_and_single_cells_give_the_same_bits(need_gpu):
    """The filler's 400 tiles send the batch through pairs; each small member
    alone has at most nine tiles."""
    probs = [problems.orszag_tang(320, seed=1), problems.orszag_tang(6), problems.orszag_tang(17, ny=31),
             problems.orszag_tang(33, ny=24), problems.orszag_tang(16, ny=40),
             problems.atmosphere(39, 23, noise=1e-3, seed=4), problems.atmosphere(16, 9, noise=1e-3, seed=5)]
    probs[5].btype, probs[6].btype = (4, 3), (6, 5)
    probs[2].divb = 1
    b = Batch(2, precision=PREC_MIXED, arena_bytes=512 << 20, max_sims=8)
    fixed = [dict(dt_mode=0, dt0=1e-2) if p.name == "atmosphere" else dict(dt_mode=0, dt0=2e-4) for p in probs]
    slots = [b.add(p, 3, **kw) for p, kw in zip(probs, fixed)]
    b.step(3)
    b.sync()
    for p, s, kw in zip(probs, slots, fixed):
        assert np.array_equal(b.state(s), alone(p, 3, PREC_MIXED, **kw)), p.n
    b.close()


@pytest.mark.parametrize("precision,tol", [(PREC_FP64, 1e-6), (PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("make", [
    lambda: problems.blast_wave(6, seed=2),
    lambda: problems.blast_wave(33, seed=2),
    lambda: problems.atmosphere(37, 9, 6, noise=1e-3, seed=3),
    lambda: problems.atmosphere(12, 34, 13, noise=1e-3, seed=4),
], ids=["blast6", "blast33", "atmosphere37x9x6", "atmosphere12x34x13"])
def test_3d_passes_against_the_oracle(need_gpu, make, precision, tol):
    for hyperdif in (1, 0):
        prob = make()
        prob.hyperdif = hyperdif
        dt0 = 1e-2 if prob.name == "atmosphere" else 2e-4
        o = Oracle(prob, dt_fixed=dt0)
        o.step(3, rk4=True, dt_mode=0)
        err = field_errors(alone(prob, 3, precision, dt_mode=0, dt0=dt0), o.w, 8)
        assert np.all(err < tol), (hyperdif, err)


def test_3d_batch_over_several_groups_of_slabs(need_gpu):
    probs = [problems.blast_wave(98, seed=k) for k in (1, 2, 3)]  # 178 MB of workspace each, 512 MB per group
    b = Batch(3, precision=PREC_MIXED, arena_bytes=3 << 30, max_sims=4)
    slots = [b.add(p, 1) for p in probs]
    b.step(1)
    b.sync()
    for p, s in zip(probs, slots):
        assert np.array_equal(b.state(s), alone(p, 1, PREC_MIXED))
    b.close()
