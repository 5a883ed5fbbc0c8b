"""Products on a nearly full device: a product that fits without the scratch of
the faster forms (row windows of heavy tile rows, the table of B's parts,
bitmaps of tile rows) runs without it, with bitwise the same C."""
from __future__ import annotations

import numpy as np
import pytest

import rtt_spgemm as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = torch.device("cuda:0")
MB = 1 << 20


def _csr(m, n, per, seed):
    """Rows of at most `per` random columns, made on the device."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    key = torch.randint(0, n, (m, per), device=DEV, generator=g)
    key = torch.unique(key + torch.arange(m, device=DEV)[:, None] * n)
    rp = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(key // n, minlength=m), 0)
    val = torch.rand(key.numel(), dtype=torch.float64, device=DEV, generator=g) - 0.5
    return m, n, rp.int(), (key % n).int(), val


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _product(a, b, wide, out=None, cfg=None, keep=None):
    """C and the device memory that the context took for it."""
    ctx = R.Context(0, cfg)
    before = torch.cuda.mem_get_info()[0]
    nnz = ctx.symbolic64(a, b) if wide else ctx.symbolic(a, b)[0]
    if out is None:
        out = (torch.empty(a[0] + 1, dtype=torch.int64 if wide else torch.int32, device=DEV),
               torch.empty(nnz, dtype=torch.int32, device=DEV),
               torch.empty(nnz, dtype=torch.float64, device=DEV))
        before -= sum(t.numel() * t.element_size() for t in out)
    (ctx.numeric64 if wide else ctx.numeric)(*out)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    return out, used


# what is refused: (A's rows, columns, entries per row; B's columns, entries per
# row; 64-bit; room in MB beside what the product takes without it)
CASES = {
    # 1 GiB: the table of B's parts
    "parts": (24, 2_000_000, 8000, 6000, 1, False, 300),
    # 512 MB each: B's bitmaps, and the table
    "bitmaps": (48, 1 << 20, 2000, 1 << 20, 9, True, 200),
    # 290 MB: the masks row by row, so the row windows as a whole
    "rows": (20000, 50000, 10, 1 << 20, 40, False, 200),
}


@pytest.mark.parametrize("case", list(CASES))
def test_nearly_full_device(case):
    m, k, pa, n, pb, wide, room = CASES[case]
    a, b = _csr(m, k, pa, 1), _csr(k, n, pb, 2)
    out, full = _product(a, b, wide)
    want = [t.clone() for t in out]
    # the slot tables and the tile-row windows take none of that scratch
    _, least = _product(a, b, wide, out, dict(sym_window_slots=-1, split_target=-1))
    hog_bytes = _free() - least - room * MB
    assert full > least + room * MB, (full // MB, least // MB)
    hog = torch.empty(hog_bytes, dtype=torch.uint8, device=DEV)
    for t in out:
        t.fill_(-1)
    try:
        _product(a, b, wide, out)
    finally:
        del hog
        torch.cuda.empty_cache()
    for x, y in zip(out, want):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32)), case
