"""The bench's phase tables on made-up counts (no GPU): the accounting of the
sections that print them, and what a rate may be formed of."""

import os
import sys
import types

import numpy as np

from conftest import ROOT

sys.path.insert(0, ROOT)

import bench  # noqa: E402

PHASES = ("preprocess", "depth_sort", "emit", "tile_sort", "ranges", "raster")


def test_sort_beside_the_vertex_stage_has_no_rate_of_its_own():
    """The sort's ms is what it takes beyond the vertex stage, down to 0: bytes
    over it are no rate. The two together have one."""
    ms = dict(zip(PHASES, (0.3, 0.0, 0.4, 0.2, 0.0, 0.5)))
    rows = bench.phase_rows(ms, lambda k: 6_000_000, {"measured": 6000.0, "nominal": 8000.0})
    for k in ("preprocess", "depth_sort"):
        assert set(rows[k]) == {"ms", "bytes"}
    both = rows["preprocess_depth_sort"]
    assert both["ms"] == 0.3 and both["bytes"] == 12_000_000
    assert abs(both["gbs"] - 40.0) < 1e-9
    assert abs(both["frac_measured"] - 40.0 / 6000) < 1e-12
    assert abs(both["frac_nominal"] - 40.0 / 8000) < 1e-12
    assert rows["ranges"]["gbs"] is None and rows["ranges"]["frac_measured"] is None
    assert abs(rows["raster"]["gbs"] - 12.0) < 1e-9


def test_raster_bytes_do_not_grow_with_the_tiles_a_splat_covers():
    """A frame whose splats cover many tiles is opaque early: pairs are no
    bound on what the raster reads, drawn records and the image are."""
    few, many = (types.SimpleNamespace(visible=100, drawn=90, tile_keys=k) for k in (200, 10**9))
    assert bench.algorithmic_bytes("raster", few, 120, 12, 64, 32, 1) == \
        bench.algorithmic_bytes("raster", many, 120, 12, 64, 32, 1) == 90 * 48 + 64 * 32 * 4


def test_batched_rows_sum_the_views():
    """Two groups: 1,200 bins (two passes) and 4 (one)."""
    specs = [(0, None, 1920, 2560), (0, None, 100, 100)]
    stats = [types.SimpleNamespace(group=g, visible_count=50, drawn_count=40, tile_pairs=1600)
             for g in (0, 1)]
    scenes = [{"positions": np.zeros((60, 3))}]
    rows = bench.batched_phase_rows({k: 1.0 for k in PHASES}, specs, stats, scenes, 12, 6000.0)
    assert rows["tile_sort"]["bytes"] == (2 + 1) * 100 * 16
    assert rows["preprocess"]["bytes"] == bench.batched_preprocess_bytes(specs, stats, scenes, 12)
    assert rows["raster"]["bytes"] == 2 * 40 * 48 + 4 * (1920 * 2560 + 100 * 100)
    assert abs(rows["raster"]["frac_measured"] - rows["raster"]["bytes"] / 6e9) < 1e-12
