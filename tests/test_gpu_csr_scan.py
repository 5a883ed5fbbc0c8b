"""The entry-wise CSR passes of the device path (checks, row segments, tile
index: csrc/csr2tile.cu) at the ends of their 256-entry blocks, 8-block CTAs
and warps' chunks: entry counts around them, runs of one tile column and rows
that cross them, long rows, thousands of empty rows, an unaligned column array,
and errors in the last entry.  C = A * B against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import rtt_spgemm as R
from conftest import assert_csr_close
from rtt_spgemm import generators as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = torch.device("cuda:0")


def _csr(counts, n, seed, runs=False):
    """Rows of the given lengths: random columns, or runs of neighbours."""
    rng = np.random.default_rng(seed)
    cols = []
    for k in counts:
        if runs:
            cols.append(np.arange(k) + int(rng.integers(0, n - k + 1)))
        else:
            cols.append(np.sort(rng.choice(n, k, replace=False)))
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32) if cols else np.zeros(0, np.int32)
    return G.CSR(len(counts), n, rp, col, rng.uniform(-1, 1, col.size))


def _dev(a, shift=0):
    col = torch.zeros(a.nnz + shift, dtype=torch.int32, device=DEV)
    col[shift:] = torch.from_numpy(a.col)
    return (a.m, a.n, torch.from_numpy(a.rowptr).to(DEV), col[shift:],
            torch.from_numpy(a.val).to(DEV))


def _tiles(a):
    rows = np.repeat(np.arange(a.m), np.diff(a.rowptr))
    return np.unique((rows // 16).astype(np.int64) * (a.n // 16 + 1) + a.col // 16).size


CASES = {
    # entry counts around a block, a CTA of blocks and twice it
    **{f"nnz{k}": (lambda k=k: _csr([7] * (k // 7) + [k % 7], 300, k))
       for k in (1, 255, 256, 257, 2047, 2048, 2049, 4097)},
    "runs": lambda: _csr([37] * 200, 400, 3, runs=True),       # runs across every block end
    "one_row": lambda: _csr([5000], 9000, 4),                   # one row over many warps
    "long_run": lambda: _csr([0, 900, 0, 1100, 3], 1200, 5, runs=True),
    "empty": lambda: _csr([3] + [0] * 4000 + [5] * 60 + [0] * 3000, 500, 6),
    # empty rows: walked, and past 2,080 of them among 256 entries looked up
    "gap40": lambda: _csr(([3] + [0] * 40) * 300, 500, 9),
    "gap600": lambda: _csr(([2] + [0] * 600) * 40 + [5] * 100, 500, 10),
    "gap5000": lambda: _csr(([37] + [0] * 5000 + [1]) * 9, 400, 11, runs=True),
    "front": lambda: _csr([0] * 30000 + [7] * 100, 300, 12),
    "back": lambda: _csr([8] * 64 + [0] * 30000, 300, 13),     # 512 entries: the last word is full
    "middle": lambda: _csr([4] * 100 + [0] * 30000 + [9] * 100, 300, 14),
    # two blocks to a warp (more than 2 * 1200 CTAs of 8 warps' blocks): runs over
    # their ends, rows longer than both, empty rows among them
    "many": lambda: _csr([24] * 100000 + [5000] + [0] * 9000 + [37] * 3000 + [24] * 105000 + [3],
                         9000, 7, runs=True),
}


# (payload: segments beside the tiles, without the tile index from them)
@pytest.mark.parametrize("shift,cfg", [(0, {}), (1, {}), (0, dict(dmma_pair_cutoff=4000))])
@pytest.mark.parametrize("case", list(CASES))
def test_scan(case, shift, cfg, orc):
    a = CASES[case]()
    assert case != "many" or a.nnz > 2 * 1200 * 8 * 256
    b = _csr([2] * a.n, 200, 8)
    if cfg:  # the segments that step 2 reads are B's
        filled = np.flatnonzero(np.diff(a.rowptr))
        pick = _csr([min(2, filled.size)] * 50, filled.size, 8)
        a, b = G.CSR(50, a.m, pick.rowptr, filled[pick.col].astype(np.int32), pick.val), a
    ctx = R.Context(0, cfg)
    da, db = _dev(a, shift), _dev(b)
    nnz, _ = ctx.symbolic(da, db)
    out = (torch.empty(a.m + 1, dtype=torch.int32, device=DEV),
           torch.empty(nnz, dtype=torch.int32, device=DEV),
           torch.empty(nnz, dtype=torch.float64, device=DEV))
    ctx.numeric(*out)
    st = ctx.stats()
    assert st["tiles_a"] == _tiles(a) and st["tiles_b"] == _tiles(b)
    assert_csr_close(*(x.cpu().numpy() for x in out), *orc.spgemm_csr(a, b), case)
    # the last entry's column, or the row pointer's end, out of range
    for bad in () if cfg else ("col", "rowptr"):
        a2 = G.CSR(a.m, a.n, a.rowptr.copy(), a.col.copy(), a.val)
        if bad == "col":
            a2.col[-1] = a.n
        else:
            a2.rowptr[-1] += 1
        for args in ((_dev(a2, shift), db), (_dev(a2, shift), None, R.RTT_OP_AAT)):
            with pytest.raises(R.RttError) as e:
                ctx.symbolic(*args)
            assert e.value.status == 2
    # the context is as good as before
    assert ctx.symbolic(da, db)[0] == nnz
    ctx.close()


# (rows of A, columns, rows' lengths): tile rows of few segments over one, two
# and many windows of 8192 tile columns, merged or not; of many segments over a
# few; runs of one tile column
WIDE = {
    "two_windows": (200, 16 * 8192 + 5, 6),
    "merge_few": (200, 5_000_000, 5),
    "merge_one": (100, 100_000_000, 1),
    "merge_more": (40, 200_000_000, 120),
    "windows": (40, 600_000, 900),
    "last": (60, 2**31 - 1, 7),
}


@pytest.mark.parametrize("case", list(WIDE))
def test_wide_tile_index(case):
    """The tile index of wide, nearly empty rows: tiles counted and binned."""
    m, n, per = WIDE[case]
    rng = np.random.default_rng(m + per)
    cols = rng.integers(0, n, (m, per))
    cols[:, -1] = np.minimum(cols[:, 0] + rng.integers(0, 16, m), n - 1)  # runs of one tile
    rows = [np.unique(r) for r in cols]
    rows[m // 2] = np.zeros(0, np.int64)
    rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    b = G.CSR(m, n, rp, np.concatenate(rows).astype(np.int32), np.ones(rp[-1]))
    a = _csr([3] * 10, m, 1)
    ctx = R.Context(0)
    dev = (_dev(a), _dev(b))  # borrowed
    ctx.symbolic(*dev)
    assert ctx.stats()["tiles_b"] == _tiles(b)
    tilem, tilen = -(-m // 16), -(-n // 16)
    tiles = np.unique((np.repeat(np.arange(m), np.diff(rp)) // 16).astype(np.int64) * tilen +
                      b.col // 16)
    want = np.zeros((64, 64), np.int64)
    np.add.at(want, (tiles // tilen * 64 // tilem, tiles % tilen * 64 // tilen), 1)
    assert np.array_equal(np.asarray(ctx.tile_heatmap("B", 64)).reshape(64, 64), want)
    ctx.close()


@pytest.mark.parametrize("cfg", [{}, dict(keep_tiles=1), dict(fused_csr_output=0), dict(b_staging=1),
                                 dict(dmma_pair_cutoff=1), dict(leaf_dmma=1)],
                         ids=lambda c: "_".join(c) or "default")
@pytest.mark.parametrize("empty", ["rows", "product"])
def test_empty_product(empty, cfg):
    """C without entries, its columns and values NULL: the row pointer is
    written all the same.  No entries at all, or tiles that meet where no row
    and column do."""
    a = _csr([0] * 500, 300, 15) if empty == "rows" else _csr([1] * 500, 300, 15)
    if empty == "product":
        a.col[:] = 16 * (a.col // 16)  # first rows of B's tiles, which are empty
    b = _csr([0 if k % 16 == 0 else 3 for k in range(300)], 200, 16)
    ctx = R.Context(0, cfg)
    dev = (_dev(a), _dev(b))
    nnz, tiles = ctx.symbolic(*dev)
    assert nnz == 0 and (tiles > 0) == (empty == "product")
    out = (torch.full((501,), -1, dtype=torch.int32, device=DEV),
           torch.empty(0, dtype=torch.int32, device=DEV),
           torch.empty(0, dtype=torch.float64, device=DEV))
    for _ in range(3):  # the third replays a graph
        ctx.numeric(*out)
        assert not out[0].any()
        out[0].fill_(-1)
    if empty == "product":
        ctx.numeric_values(dev[0][4], dev[1][4], *out)
        assert not out[0].any()
    ctx.close()


@pytest.mark.parametrize("tiles", [4096, 5120, 5121, 10240, 10241, 16384, 16385])
def test_scan_lengths(tiles):
    """Sums of as many tile rows and C tiles as one CTA scans, and one more: a
    diagonal matrix, squared."""
    m = 16 * tiles - 3
    v = torch.rand(m, dtype=torch.float64, device=DEV)
    i = torch.arange(m + 1, dtype=torch.int32, device=DEV)
    a = (m, m, i, i[:m].contiguous(), v)
    for wide in (False, True):
        ctx = R.Context(0)
        nnz = ctx.symbolic64(a) if wide else ctx.symbolic(a)[0]
        assert nnz == m
        out = (torch.empty(m + 1, dtype=torch.int64 if wide else torch.int32, device=DEV),
               torch.empty(m, dtype=torch.int32, device=DEV),
               torch.empty(m, dtype=torch.float64, device=DEV))
        (ctx.numeric64 if wide else ctx.numeric)(*out)
        assert torch.equal(out[0], i.to(out[0].dtype)) and torch.equal(out[1], i[:m])
        assert torch.equal(out[2], v * v)
        ctx.close()
