"""The kernels of a stage start while the kernel before them still runs
(programmatic dependent launch) and wait inside.  Non-coherent loads are defined
for data that nothing writes during a kernel's whole life, so in those kernels
they may reach only what is fixed between steps: the backgrounds and the metric.
The state, the sources and the workspace take ordinary loads.  (A source check:
a violation is a race, which no run has to show.)"""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "smaug-all_b200" / "csrc"
FIXED = ("bg", "a.bg", "g.dxlast", "g.dx1", "g.rdx1")


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name", ["batch_kernels.inc", "smaug_pass3.cuh", "smaug_pairs2.cuh", "smaug_tile.cuh",
                                  "smaug_tile2.cuh"])
def test_non_coherent_loads_reach_fixed_data_only(name):
    text = code(name)
    assert ".nc" not in text
    bases = [re.match(r"[\w.]+", m).group(0) for m in re.findall(r"__ldg\(\s*([^)]*)", text)]
    assert all(b in FIXED for b in bases), sorted(set(bases) - set(FIXED))
