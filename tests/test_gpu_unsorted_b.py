"""C = A * B where A's rows are sorted and B's are not: B then lists no row
segments, and symbolic step 2 walks B's rows for A's entries.  One and several windows per tile row, hub rows, the 64-bit products
in chunks, batches, another B for the same A, and new values."""
from __future__ import annotations

import numpy as np
import pytest

import rtt_spgemm as R
from conftest import assert_csr_close
from rtt_spgemm import generators as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = torch.device("cuda:0")


def _dev(a):
    return (a.m, a.n, torch.from_numpy(a.rowptr).to(DEV), torch.from_numpy(a.col).to(DEV),
            torch.from_numpy(a.val).to(DEV))


def _shuffled(a, seed):
    """The entries of every row in random order."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(a.m), np.diff(a.rowptr))
    order = np.lexsort((rng.random(a.nnz), rows))
    return G.CSR(a.m, a.n, a.rowptr, a.col[order].copy(), a.val[order].copy())


def _out(m, nnz, wide=False):
    return (torch.full((m + 1,), -1, dtype=torch.int64 if wide else torch.int32, device=DEV),
            torch.full((nnz,), -1, dtype=torch.int32, device=DEV),
            torch.full((nnz,), float("nan"), dtype=torch.float64, device=DEV))


def _close(out, a, b, orc, tag):
    assert_csr_close(*(x.cpu().numpy() for x in out), *orc.spgemm_csr(a, b), tag)


CASES = {
    "small": lambda: (G.random_csr(500, 300, 0.02, seed=51), G.random_csr(300, 700, 0.015, seed=52)),
    "windows": lambda: (G.random_csr(300, 900, 0.03, seed=53), G.random_csr(900, 30000, 0.01, seed=54)),
    "hubs": lambda: (G.rmat(12, 16, seed=3), G.rmat(12, 16, seed=4)),
    "grid": lambda: (G.stencil_27(9, 1), G.stencil_27(9, 2)),
}


@pytest.mark.parametrize("case", list(CASES))
def test_sorted_a_unsorted_b(case, orc):
    a, b = CASES[case]()
    bs = _shuffled(b, 7)
    da, db, dbs = _dev(a), _dev(b), _dev(bs)
    ctx = R.Context(0)
    nnz, _ = ctx.symbolic(da, dbs)
    out = _out(a.m, nnz)
    ctx.numeric(*out)
    _close(out, a, bs, orc, case)
    # new values of both, the structure kept
    va, vb = a.val[::-1].copy(), bs.val[::-1].copy()
    ctx.numeric_values(torch.from_numpy(va).to(DEV), torch.from_numpy(vb).to(DEV), *out)
    _close(out, G.CSR(a.m, a.n, a.rowptr, a.col, va), G.CSR(b.m, b.n, b.rowptr, bs.col, vb), orc, case)
    # the same A with one B after the other
    nnz, _ = ctx.symbolic(da, db)
    for d, h in ((dbs, bs), (db, b), (dbs, bs)):
        nnz, _ = ctx.update_b(d)
        out = _out(a.m, nnz)
        ctx.numeric(*out)
        _close(out, a, h, orc, case + " update_b")
    ctx.close()


@pytest.mark.parametrize("case", ["windows", "hubs"])
def test_in_chunks(case, orc):
    a, b = CASES[case]()
    bs = _shuffled(b, 8)
    ctx = R.Context(0, dict(chunk_tiles=3000))
    da, db = _dev(a), _dev(bs)
    nnz = ctx.symbolic64(da, db)
    out = _out(a.m, nnz, wide=True)
    ctx.numeric64(*out)
    _close(out, a, bs, orc, case)
    ctx.close()


@pytest.mark.parametrize("op", ["A2", "AB", "AAT"])
def test_set_up_once(op, orc):
    """Unsorted rows are checked and transposed once: one synchronisation for
    the operands, one per tiled operand, two for steps 1 and 2."""
    a, b = CASES["grid"]()
    s = _shuffled(a, 11)
    args = {"A2": (s, None, R.RTT_OP_AB), "AB": (s, _shuffled(b, 12), R.RTT_OP_AB),
            "AAT": (s, None, R.RTT_OP_AAT)}[op]
    ctx = R.Context(0)
    dev = (_dev(args[0]), _dev(args[1]) if args[1] else None, args[2])  # borrowed until numeric
    nnz, _ = ctx.symbolic(*dev)
    out = _out(s.m, nnz)
    ctx.numeric(*out)
    assert ctx.stats()["host_syncs"] <= (6 if op == "AB" else 5)
    _close(out, s, {"A2": s, "AB": args[1], "AAT": a.transpose()}[op], orc, op)
    ctx.close()


def test_batched(orc):
    pairs = [CASES[c]() for c in ("small", "grid", "small")]
    hosts = [(a, _shuffled(b, 9 + i)) for i, (a, b) in enumerate(pairs)]
    ctx = R.Context(0)
    As, Bs = [_dev(a) for a, _ in hosts], [_dev(b) for _, b in hosts]
    for (a, b), c in zip(hosts, R.spgemm_batched(ctx, As, Bs)):
        _close(c, a, b, orc, "batched")
    ctx.close()


@pytest.mark.parametrize("cfg", [{}, dict(b_staging=1), dict(dmma_pair_cutoff=1)],
                         ids=lambda c: "_".join(c) or "default")
@pytest.mark.parametrize("which", ["A", "A sorted", "B"])
@pytest.mark.parametrize("n", [40, 60000])
def test_tiles_of_repeated_columns(n, which, cfg, orc):
    """Rows that repeat columns until a tile holds more than 255 entries, which a
    tile's byte offsets cannot count: unsorted or not, one window and several."""
    rng = np.random.default_rng(20)
    a_cols = [np.concatenate([rng.integers(0, 16, 40), rng.integers(0, 300, 5)]) for _ in range(50)]
    rp = np.arange(51, dtype=np.int32) * 45
    a = G.CSR(50, 300, rp, np.concatenate(a_cols).astype(np.int32), rng.uniform(-1, 1, 50 * 45))
    b = _shuffled(G.random_csr(300, n, min(0.2, 1200 / n), seed=21), 22)
    if which == "A sorted":
        order = np.lexsort((a.col, np.repeat(np.arange(50), 45)))
        a = G.CSR(50, 300, rp, a.col[order].copy(), a.val[order].copy())
    elif which == "B":
        a, b = G.random_csr(70, 50, 0.2, seed=23), a
    ctx = R.Context(0, cfg)
    dev = (_dev(a), _dev(b))
    nnz, _ = ctx.symbolic(*dev)
    out = _out(a.m, nnz)
    for _ in range(3):  # the third replays a graph
        out[2].fill_(float("nan"))
        ctx.numeric(*out)
        _close(out, a, b, orc, "repeated columns")
    ctx.close()
