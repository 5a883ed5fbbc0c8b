"""The one-window tile-row kernel (csrc/numeric_tilerow.cu) at its edges: exactly
128 C tiles and 2048 entries, one tile, tile columns beyond its slot table,
B rows of 0, 1, 32, 33 and more entries, a ragged last tile row, empty rows.
Bitwise equal to the kernel that also keeps the tiles, and within the bound of
the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import rtt_spgemm as R
from conftest import assert_csr_close
from rtt_spgemm import generators as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = torch.device("cuda:0")


def _rows(lists, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum([len(c) for c in lists])]).astype(np.int32)
    col = np.concatenate([np.sort(np.asarray(c)) for c in lists]).astype(np.int32)
    return G.CSR(len(lists), n, rp, col, rng.uniform(-1, 1, col.size))


def _pick(m, per, k, seed):
    rng = np.random.default_rng(seed)
    return _rows([rng.choice(k, per, replace=False) for _ in range(m)], k, seed)


def _ends(w):
    """Rows with entries in tile columns 7, 7 + w and one between."""
    return _rows([16 * np.array([7, 8 + w // 2 + i, 7 + w]) + i for i in range(16)],
                 16 * (w + 9), 8)


CASES = {
    # a tile row of 16 x 128 = 2048 entries in 128 tiles
    "full": lambda: (_pick(32, 3, 8, 1), _rows([16 * np.arange(128) + 5] * 8, 2048, 2)),
    "dense": lambda: (_pick(40, 5, 8, 3), _rows([np.arange(128)] * 8, 128, 4)),  # 2048 in 8 tiles
    "one_tile": lambda: (_pick(5, 2, 4, 5), _rows([[3, 9]] * 4, 16, 6)),
    "far": lambda: (_pick(37, 4, 16, 7),
                    _rows([16 * np.arange(i % 2, 80000 // 16, 1250) + i for i in range(16)], 80000, 8)),
    # 4,095 tile columns from a tile row's first to its last: the slot table's
    # most; 4,096 and more: no table
    **{f"span{w}": (lambda w=w: (_pick(37, 4, 16, 7), _ends(w))) for w in (4095, 4096, 9000)},
    "lengths": lambda: (_pick(50, 6, 8, 9),
                        _rows([np.arange(k) for k in (0, 1, 31, 32, 33, 64, 65, 100)], 110, 10)),
    "empty_rows": lambda: (_rows([[0, 1]] + [[]] * 20 + [[2]] + [[]] * 30, 3, 11),
                           _rows([[1, 40], [], [5]], 60, 12)),
}


@pytest.mark.parametrize("case", list(CASES))
def test_tile_rows(case, orc):
    a, b = CASES[case]()
    runs = []
    for cfg in (None, dict(keep_tiles=1)):
        ctx = R.Context(0, cfg)
        t = [(x.m, x.n, *(torch.from_numpy(v).to(DEV) for v in (x.rowptr, x.col, x.val)))
             for x in (a, b)]
        nnz, _ = ctx.symbolic(t[0], t[1])
        out = (torch.full((a.m + 1,), -1, dtype=torch.int32, device=DEV),
               torch.full((nnz,), -1, dtype=torch.int32, device=DEV),
               torch.full((nnz,), float("nan"), dtype=torch.float64, device=DEV))
        ctx.numeric(*out)
        runs.append([x.cpu().numpy() for x in out] + [np.array([ctx.stats()["nnz_cub"]])])
        ctx.close()
    for x, y in zip(*runs):
        assert np.array_equal(x.view(np.int32), y.view(np.int32)), case
    assert_csr_close(*runs[0][:3], *orc.spgemm_csr(a, b), case)
    if case.startswith("span"):
        rp, col = runs[0][:2]
        for i in range(0, a.m, 16):
            tiles = col[rp[i]:rp[min(i + 16, a.m)]] // 16
            assert tiles.max() - tiles.min() == int(case[4:])
