"""What smaug_step_noalloc shares with a context (needs a GPU): the same bits in
2-D (RK4 and single step) and for 3-D single steps, which run the same kernels;
3-D RK4 runs without the workspace of the context's passes and agrees to
rounding."""
from __future__ import annotations

import numpy as np
import pytest

from smaug_b200 import problems

from test_zz_no_alloc import _lib, _noalloc, _regular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rk4", [True, False])
@pytest.mark.parametrize("make", [lambda: problems.orszag_tang(48), lambda: problems.orszag_tang(97, ny=33),
                                  lambda: problems.blast_wave(14, seed=5)], ids=["48x48", "97x33", "14x14x14"])
def test_noalloc_and_context(need_gpu, make, rk4):
    prob = make()
    a, s = _noalloc(_lib(), prob, prob.w, 5, rk4=rk4)
    b, t = _regular(prob, prob.w, 5, rk4=rk4)
    if prob.ndim == 2 or not rk4:
        assert np.array_equal(a, b) and s[0] == t["dt"]
    else:
        inner = (slice(2, -2),) * 3
        for f in range(8):
            assert np.linalg.norm((a[f] - b[f])[inner]) <= 1e-12 * np.linalg.norm(b[f][inner]), f
        assert s[0] == pytest.approx(t["dt"], rel=1e-12)
