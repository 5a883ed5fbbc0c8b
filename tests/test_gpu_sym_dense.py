"""Symbolic steps of dense C tile rows (bitmaps of B's tile rows, row masks
directly addressed: csrc/symbolic.cu) at the ends of their 1024-tile windows,
with tiles of the union that hold no entry, long and short B rows and a ragged
last tile row.  Equal to the slot-table form (sym_window_slots = -1) and the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

import rtt_spgemm as R
from conftest import assert_csr_close
from rtt_spgemm import generators as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = torch.device("cuda:0")


def _random(m, n, per, seed):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(m), rng.integers(0, 2 * per + 1, m))
    return G.from_coo(m, n, rows, rng.integers(0, n, rows.size), rng.uniform(-1, 1, rows.size))


# (rows of A, inner, columns, entries per row of A, of B); the columns lie
# around one, two and three windows of 1024 tiles
CASES = {
    "one": (70, 300, 16 * 1023 + 5, 40, 60),
    "exact": (64, 300, 16 * 1024, 40, 60),
    "two": (33, 300, 16 * 1025, 60, 60),
    "three": (50, 400, 16 * 2049 + 1, 90, 90),
    "sparse_tiles": (48, 2000, 16 * 1100, 20, 40),  # many empty tiles in the union
    "short_rows": (160, 9000, 16 * 700, 50, 4),
}


@pytest.mark.parametrize("case", list(CASES))
def test_dense_rows(case, orc):
    m, k, n, pa, pb = CASES[case]
    a, b = _random(m, k, pa, 1), _random(k, n, pb, 2)
    runs = []
    for slots in (0, -1):
        ctx = R.Context(0, dict(sym_window_slots=slots))
        t = [(x.m, x.n, *(torch.from_numpy(v).to(DEV) for v in (x.rowptr, x.col, x.val)))
             for x in (a, b)]
        nnz, tiles = ctx.symbolic(t[0], t[1])
        heat = ctx.tile_heatmap("C", 8)
        out = (torch.empty(m + 1, dtype=torch.int32, device=DEV),
               torch.empty(nnz, dtype=torch.int32, device=DEV),
               torch.empty(nnz, dtype=torch.float64, device=DEV))
        ctx.numeric(*out)
        runs.append([np.array([tiles]), heat] + [x.cpu().numpy() for x in out])
        ctx.close()
    for x, y in zip(*runs):
        assert np.array_equal(x.view(np.int32), y.view(np.int32)), case
    assert_csr_close(*runs[0][2:], *orc.spgemm_csr(a, b), case)
