"""Heavy C tile rows, one scalar row per warp (csrc/numeric_rowwin.cu), where
its windows, pieces and cursors can go wrong: rows of exactly one window's
entries or tiles and one more or less, tile columns further apart than one
column index spans, rows with more A entries than the kept places, rows cut
into pieces.  Bitwise equal to the tile-row kernel's windows
(split_target = -1), and within the bound of the oracle."""
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
    """CSR whose row i has the columns lists[i]."""
    rng = np.random.default_rng(seed)
    cnt = [len(c) for c in lists]
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    col = np.concatenate([np.sort(np.asarray(c)) for c in lists]).astype(np.int32)
    return G.CSR(len(lists), n, rp, col, rng.uniform(-1, 1, col.size))


def _pick(m, per, k, seed):
    rng = np.random.default_rng(seed)
    return _rows([rng.choice(k, min(per, k), replace=False) for _ in range(m)], k, seed)


def _entries():
    # C rows of 511 .. 1025 entries (windows of 512), two B rows each
    sizes = [511, 512, 513, 1023, 1024, 1025, 600, 1] * 4
    b = _rows([np.arange(7 * i, 7 * i + s) for i, s in enumerate(sizes)] +
              [np.arange(7 * i, 7 * i + s, 3) for i, s in enumerate(sizes)], 1300, 1)
    return _rows([[i, i + 32] for i in range(32)], 64, 2), b


def _tiles():
    # C rows of 255 .. 513 tiles with one entry each (windows of 256)
    sizes = [255, 256, 257, 511, 512, 513, 8, 7] * 4
    b = _rows([16 * np.arange(i, i + s) + i % 16 for i, s in enumerate(sizes)], 16 * 700, 3)
    return _rows([[i] for i in range(32)], 32, 4), b


def _spans():
    # a cluster of tiles, then tiles further apart than 512 * 32 tile columns
    # span 8 of them; and single entries around the end of one span
    n = 16 * 300000
    far = [np.concatenate([np.arange(0, 1600, 16), 16 * np.arange(1000 + i, 290000, 8700)])
           for i in range(30)]
    edge = 16 * 32 * 512
    far += [[0, edge - 1, edge, edge + 1, 2 * edge], list(range(edge - 800, edge + 800))]
    return _pick(40, 6, 32, 5), _rows(far, n, 6)


def _long():
    # 3,000 A entries per row, places kept for all; C rows of many windows
    rng = np.random.default_rng(7)
    b = _rows([rng.choice(9000, 40, replace=False) for _ in range(6000)], 9000, 8)
    return _pick(20, 3000, 6000, 9), b


def _over():
    # 9,000 A entries per row, places kept for 4,096: the others are searched,
    # and take the places of those whose B rows end early
    rng = np.random.default_rng(20)
    b = _rows([rng.choice(9000, 30, replace=False) if k % 3 else rng.choice(2000, 5, replace=False)
               for k in range(12000)], 9000, 21)
    return _pick(20, 9000, 12000, 22), b


def _hub():
    # power-law rows: pieces cut by weight
    a = G.rmat(12, 16, seed=3)
    return a, a


def _entries_long():
    # more than 1,024 entries a row: windows of 1024, rows of one and two of them
    sizes = [1023, 1024, 1025, 2047, 2048, 2049, 600, 1] * 4
    b = _rows([np.arange(7 * i, 7 * i + s) for i, s in enumerate(sizes)] +
              [np.arange(7 * i, 7 * i + s, 3) for i, s in enumerate(sizes)], 2400, 14)
    return _rows([[i, i + 32] for i in range(32)], 64, 15), b


def _tiles_long():
    # the same windows, of 512 tiles: rows of 511 .. 1025 tiles with one entry
    # each between rows of 3,000 entries
    sizes = [511, 512, 513, 1023, 1024, 1025, 8, 7] * 4
    b = _rows([16 * np.arange(i, i + s) + i % 16 for i, s in enumerate(sizes)] +
              [np.arange(9 * i, 9 * i + 3000) for i in range(32)], 16 * 1100, 16)
    return _rows([[i // 2 + 32 * (i % 2)] for i in range(64)], 64, 17), b


def _groups(m, n):
    # rows of little work, in tasks of neighbours: two from 9,472 rows (64 an SM),
    # four from 37,888
    return _pick(m, 3, 48, 18), _pick(48, 40, n, 19)


CASES = {"entries": _entries, "tiles": _tiles, "spans": _spans, "long": _long, "hub": _hub,
         "over": _over,
         "entries_long": _entries_long, "tiles_long": _tiles_long,
         "groups2": lambda: _groups(9473, 20000),
         # (and columns further apart than one column index spans)
         "groups4": lambda: _groups(38001, 16 * 300000)}


def _run(a, b, cfg):
    ctx = R.Context(0, cfg)
    t = [(x.m, x.n, *(torch.from_numpy(v).to(DEV) for v in (x.rowptr, x.col, x.val)))
         for x in (a, b)]
    nnz, _ = ctx.symbolic(t[0], t[1])
    out = (torch.full((a.m + 1,), -1, dtype=torch.int32, device=DEV),
           torch.full((nnz,), -1, dtype=torch.int32, device=DEV),
           torch.full((nnz,), float("nan"), dtype=torch.float64, device=DEV))
    ctx.numeric(*out)
    st = ctx.stats()
    ctx.close()
    return [x.cpu().numpy() for x in out], st


@pytest.mark.parametrize("case", list(CASES))
def test_row_windows(case, orc):
    a, b = CASES[case]()
    want, st0 = _run(a, b, dict(split_target=-1))
    for target in (0, 1, 1 << 16):
        got, st = _run(a, b, dict(split_target=target))
        assert st["split_windows"] > 0 and st["nnz_cub"] == st0["nnz_cub"]
        assert target or not case.startswith("groups") or \
            st["split_windows"] == -(-a.m // int(case[6:]))
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.int32), w.view(np.int32)), (case, target)
    assert_csr_close(*want, *orc.spgemm_csr(a, b), case)
    if case.endswith("_long"):
        assert want[1].size > 1024 * a.m


def test_last_columns(orc):
    """B's columns at the end of the int range: cuts and windows that end past
    the last tile column."""
    width, n = 40000, 2**31 - 1
    b0 = _pick(400, 3000, width, 10)
    b = G.CSR(b0.m, n, b0.rowptr, b0.col + (n - width), b0.val)
    a = _pick(64, 200, 400, 11)
    want, _ = _run(a, b0, dict(split_target=1))
    for cfg in (dict(split_target=1), dict(split_target=-1), dict(keep_tiles=1),
                dict(sym_window_slots=-1), dict(global_rows=2)):
        got, st = _run(a, b, cfg)
        if cfg.get("split_target") == 1:
            assert st["split_windows"] > a.m  # cut into pieces
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1] + (n - width)), cfg
        if "global_rows" in cfg:
            # atomic adds, in any order: two sums of at most 200 products of
            # magnitude below 1, each within 200 * 200 * 2^-53 of the exact one
            assert np.abs(got[2] - want[2]).max() <= 2 * 200 * 200 * 2.0**-53
        else:
            assert np.array_equal(got[2].view(np.int64), want[2].view(np.int64)), cfg
    assert_csr_close(*want, *orc.spgemm_csr(a, b0), "last columns")


def test_pieces_without_the_table(orc):
    """B of more rows than the table of its parts holds: pieces find their part
    of a B row by searching it."""
    rows, width = 2_100_000, 6000
    rng = np.random.default_rng(12)
    long = set(rng.choice(rows, 3000, replace=False).tolist())
    counts = np.ones(rows, np.int64)
    counts[list(long)] = 900
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    col = rng.integers(0, width, rp[-1]).astype(np.int32)
    for k in long:
        col[rp[k]:rp[k + 1]] = np.sort(rng.choice(width, 900, replace=False))
    b = G.CSR(rows, width, rp, col, rng.uniform(-1, 1, col.size))
    picks = np.array(sorted(long))
    a = _rows([np.union1d(rng.choice(picks, 1500, replace=False), rng.choice(rows, 15000))
               for _ in range(24)], rows, 13)
    want, _ = _run(a, b, dict(split_target=-1))
    for target in (0, 1):
        got, st = _run(a, b, dict(split_target=target))
        assert st["split_windows"] > 8 * a.m  # cut into pieces
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.int32), w.view(np.int32)), target
    assert_csr_close(*want, *orc.spgemm_csr(a, b), "no table")


def test_split_target_counts_tile_rows():
    """A task of one scalar row gets a sixteenth of split_target, at most 2^17:
    2^18 is this product's default."""
    a = G.rmat(14, 16, seed=3)
    want, st0 = _run(a, a, {})
    _, whole = _run(a, a, dict(split_target=-1))
    assert whole["split_windows"] == 0
    tasks = {}
    for target in (1 << 18, 1 << 22, 1 << 30):
        got, st = _run(a, a, dict(split_target=target))
        tasks[target] = st["split_windows"]
        assert np.array_equal(got[2].view(np.int64), want[2].view(np.int64))
    assert tasks[1 << 18] == st0["split_windows"]
    assert tasks[1 << 22] == tasks[1 << 30]  # 2^18 and 2^26 a row: both 2^17
