"""The benchmark's kernel names and their DRAM traffic, without a GPU."""
from __future__ import annotations

import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402

DEFAULT = dict(leaf_dmma=0, b_staging=0, dmma_pair_cutoff=0, fused_csr_output=1, keep_tiles=0,
               global_rows=0, segment_walk=0, persistent_rows=0, split_target=0)


@pytest.mark.parametrize("cfg,split,increasing,want", [
    ({}, 0, True, "k_numeric_tilerow"), ({}, 9, True, "k_numeric_rowwin"),
    ({}, 9, False, "k_numeric_flat"), ({}, 0, False, "k_numeric_flat"),
    (dict(fused_csr_output=0), 9, True, "k_numeric_flat"),
    (dict(global_rows=2), 9, True, "k_numeric_glob2"), (dict(global_rows=2), 0, True, "k_numeric_tilerow"),
    (dict(split_target=-1), 0, True, "k_numeric_flat"), (dict(b_staging=1), 0, True, "k_numeric_rows"),
    (dict(leaf_dmma=1), 0, True, "k_numeric_leaf"), (dict(segment_walk=1), 0, True, "k_numeric_flat")])
def test_kernel_names(cfg, split, increasing, want):
    stats = dict(split_windows=split, dmma_pairs=0)
    assert bench.numeric_kernel({**DEFAULT, **cfg}, stats, increasing) == want


def test_traffic_is_the_named_kernels():
    assert bench.load_traffic("stencil27_80", "k_numeric_tilerow") == 948715776
    assert bench.load_traffic("stencil27_96", "k_numeric_flat") is None
    assert bench.load_traffic("rmat16_aat", "k_numeric_rowwin") is None
