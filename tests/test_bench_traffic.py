"""bench.py finds the DRAM traffic of the kernels that it times in the committed
ncu summary (a renamed key left the line's `traffic` null)."""
from __future__ import annotations

import bench


def test_committed_traffic_is_found_under_the_timed_kernels():
    entry = bench.load_traffic()[bench.STAGE_KERNELS]
    # at least the algorithm's bytes, at most a few times this design's
    alg = bench.BYTES_PER_CELL_UPDATE_MIXED_2D / 4
    assert alg <= entry["dram_bytes_per_inner_cell"] <= 4 * bench.DESIGN_BYTES_MIXED[2] / 4
