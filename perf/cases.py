"""The work that programs have this library do, as cases that can be timed.

``listed()`` names twelve products over the whole range of use: the smallest
calls, where launches and host round trips count, the benchmark's own
workloads, and products whose C is several gigabytes.  ``draw()`` gives more
cases of the same kinds, with sizes over the whole of each range.

Matrices are made on the GPU from the seed with the shapes and distributions of
``rtt_spgemm.generators`` (which makes them on the host).  The 2-D and 3-D
grids have a fixed structure; an R-MAT or banded case names its graph by a
seed of its own (``graph``), so that the values alone follow the seed.

The kinds:

``lap2d``     C = A^2 of a 5-point operator on an nx x ny grid: coarse levels
              of a multigrid hierarchy, served requests of small matrices.
``stencil``   C = A^2 of a 27-point operator on a g^3 grid (the headline at 96).
``rmat_sq``, ``rmat_aat``  power-law graphs: A^2 (two-hop neighbours) and A*A^T.
``rmat_wide``  A*A^T through the 64-bit products (nnz(C) may pass INT32_MAX).
``banded``    C = A^2 of a banded matrix with a few scattered entries per row.
``batched``   many independent banded A_i^2 in one call.
``values``    the values-only update of a product whose structure is kept (time
              steps, Newton iterations): new values of A every pass.
``galerkin``  the triple product P^T A P of a 27-point operator and trilinear
              interpolation: transpose and general rectangular products.
``host``      host CSR in, host CSR out.
``tiles``     the drop-in entry points of the tiled path on host data:
              csr2tile (both layouts), tile SpGEMM, tile2csr.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "rtt-spgemm_b200"))
import rtt_spgemm as R  # noqa: E402

DEV = torch.device("cuda", 0)
_CTX = []


def listed():
    return [
        # a coarse multigrid level or a small served request, ragged tiles
        {"name": "lap2d_61x67", "kind": "lap2d", "nx": 61, "ny": 67},
        # the plain configuration: 256^2 grid
        {"name": "lap2d_256", "kind": "lap2d", "nx": 256, "ny": 256},
        # the headline configuration: 27-point stencil on 96^3
        {"name": "stencil27_96", "kind": "stencil", "g": 96},
        # two-hop neighbours of a mid-size power-law graph
        {"name": "rmat14_sq", "kind": "rmat_sq", "scale": 14, "edges": 16, "graph": 1},
        # the power-law configuration's generator at a scale whose C is 32-bit
        {"name": "rmat16_aat", "kind": "rmat_aat", "scale": 16, "edges": 16, "graph": 1},
        # the power-law configuration's own entry points (64-bit row pointer)
        {"name": "rmat17_aat_wide", "kind": "rmat_wide", "scale": 17, "edges": 16, "graph": 1},
        # the largest instance of the batched configuration, on its own
        {"name": "banded_200k", "kind": "banded", "n": 200000, "hb": 32, "graph": 1},
        # sixteen instances of the batched configuration's shapes
        {"name": "batched_16", "kind": "batched", "count": 16, "n_lo": 2000, "n_hi": 50000,
         "graph": 1},
        # time steps on a 64^3 grid: the structure stays, the values change
        {"name": "values_64", "kind": "values", "g": 64},
        # one coarsening step of a geometric multigrid, odd grid
        {"name": "galerkin_49", "kind": "galerkin", "g": 49},
        # a host program's one call
        {"name": "host_stencil_40", "kind": "host", "g": 40},
        # a program of the tiled reference path
        {"name": "tiles_lap2d_256", "kind": "tiles", "nx": 256, "ny": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lap2d", "stencil", "rmat_sq", "rmat_aat", "rmat_wide", "banded", "batched",
                       "values", "galerkin", "host", "tiles"])
    if kind in ("lap2d", "tiles"):
        hi = 512 if kind == "lap2d" else 300
        return {"kind": kind, "nx": _log(rng, 16, hi), "ny": _log(rng, 16, hi)}
    if kind in ("stencil", "values"):
        return {"kind": kind, "g": _log(rng, 7, 96)}
    if kind in ("rmat_sq", "rmat_aat", "rmat_wide"):
        return {"kind": kind, "scale": rng.randint(10, 15 if kind == "rmat_sq" else 16),
                "edges": rng.randint(4, 16), "graph": rng.randrange(1 << 20)}
    if kind == "banded":
        return {"kind": kind, "n": _log(rng, 2000, 200000), "hb": rng.randint(8, 64),
                "graph": rng.randrange(1 << 20)}
    if kind == "batched":
        return {"kind": kind, "count": rng.randint(2, 16), "n_lo": 2000, "n_hi": _log(rng, 5000, 50000),
                "graph": rng.randrange(1 << 20)}
    if kind == "galerkin":
        return {"kind": kind, "g": 2 * _log(rng, 4, 32) + 1}
    return {"kind": kind, "g": _log(rng, 7, 48)}


# ---------------------------------------------------------------- matrices
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _csr(m, n, rows, cols, vals):
    """(m, n, rowptr, col, val) of entries already in row-major order."""
    rp = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return (m, n, rp.int(), cols.int().contiguous(), vals.contiguous())


def _lap2d(nx, ny, seed):
    """5-point operator with coefficients that vary: diagonal 4, off-diagonals
    -1, each scaled by a seeded factor in [0.5, 1.5)."""
    n = nx * ny
    i = torch.arange(n, device=DEV)
    x, y = i % nx, i // nx
    cols = torch.stack([i - nx, i - 1, i, i + 1, i + nx], 1)
    keep = torch.stack([y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1], 1)
    base = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], dtype=torch.float64, device=DEV)
    vals = base * (0.5 + torch.rand(n, 5, dtype=torch.float64, device=DEV, generator=_gen(seed)))
    return _csr(n, n, i[:, None].expand(n, 5)[keep], cols[keep], vals[keep])


def _stencil(g, seed):
    """27-point operator: off-diagonals U[-1, 1), diagonal 1 + the row's sum of
    their magnitudes."""
    n = g ** 3
    i = torch.arange(n, device=DEV)
    x, y, z = i % g, (i // g) % g, i // (g * g)
    d = torch.arange(27, device=DEV)
    dx, dy, dz = d % 3 - 1, (d // 3) % 3 - 1, d // 9 - 1
    keep = torch.ones(n, 27, dtype=torch.bool, device=DEV)
    for p, dp in ((x, dx), (y, dy), (z, dz)):
        q = p[:, None] + dp[None, :]
        keep &= (q >= 0) & (q < g)
    cols = i[:, None] + (dx + g * dy + g * g * dz)[None, :]
    vals = 2.0 * torch.rand(n, 27, dtype=torch.float64, device=DEV, generator=_gen(seed)) - 1.0
    vals = torch.where(keep, vals, 0.0)
    vals[:, 13] = 0.0
    vals[:, 13] = 1.0 + vals.abs().sum(1)
    return _csr(n, n, i[:, None].expand(n, 27)[keep], cols[keep], vals[keep])


def _rmat(scale, edges, graph, seed):
    n, e, g = 1 << scale, edges << scale, _gen(graph)
    r = torch.zeros(e, dtype=torch.int64, device=DEV)
    c = torch.zeros_like(r)
    for _ in range(scale):
        u = torch.rand(e, device=DEV, dtype=torch.float64, generator=g)
        r = 2 * r + (u >= 0.76)
        c = 2 * c + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    key = torch.unique(r * n + c)
    vals = torch.rand(key.numel(), dtype=torch.float64, device=DEV, generator=_gen(seed))
    return _csr(n, n, key // n, key % n, vals)


def _banded(n, hb, graph, seed):
    """Band entries kept with probability 0.5, 0..4 scattered entries a row."""
    g = _gen(graph)
    i = torch.arange(n, device=DEV)
    cols = i[:, None] + torch.arange(-hb, hb + 1, device=DEV)[None, :]
    keep = (torch.rand(cols.shape, device=DEV, generator=g) < 0.5) & (cols >= 0) & (cols < n)
    band = (i[:, None] * n + cols)[keep]
    ns = torch.randint(0, 5, (n,), device=DEV, generator=g)
    srow = torch.repeat_interleave(i, ns)
    scol = torch.randint(0, n, (srow.numel(),), device=DEV, generator=g)
    key = torch.unique(torch.cat([band, srow * n + scol]))
    vals = 2.0 * torch.rand(key.numel(), dtype=torch.float64, device=DEV,
                            generator=_gen(seed)) - 1.0
    return _csr(n, n, key // n, key % n, vals)


def _interpolation(g):
    """Trilinear interpolation from every second point of a g^3 grid (g odd)."""
    h = (g + 1) // 2
    i = torch.arange(g ** 3, device=DEV)
    row, col, w = i, torch.zeros_like(i), torch.ones(g ** 3, dtype=torch.float64, device=DEV)
    for step in (1, g, g * g):  # each axis: the point itself, or its two neighbours at half weight
        p = (row // step) % g
        odd = (p % 2).bool()
        low = col + (p // 2) * (1, h, h * h)[(1, g, g * g).index(step)]
        up = low[odd] + (1, h, h * h)[(1, g, g * g).index(step)]
        w = torch.where(odd, 0.5 * w, w)
        row, col, w = torch.cat([row, row[odd]]), torch.cat([low, up]), torch.cat([w, w[odd]])
    key, order = torch.sort(row * h ** 3 + col)
    return _csr(g ** 3, h ** 3, key // h ** 3, key % h ** 3, w[order])


def _shapes(case):
    r = random.Random(case["graph"])
    return [(_log(r, case["n_lo"], case["n_hi"]), r.randint(8, 64)) for _ in range(case["count"])]


def _operands(case, seed):
    """The case's matrices on the GPU."""
    k = case["kind"]
    if k in ("lap2d", "tiles"):
        return [_lap2d(case["nx"], case["ny"], seed)]
    if k in ("stencil", "values", "host"):
        return [_stencil(case["g"], seed)]
    if k == "galerkin":
        return [_stencil(case["g"], seed), _interpolation(case["g"])]
    if k == "banded":
        return [_banded(case["n"], case["hb"], case["graph"], seed)]
    if k == "batched":
        return [_banded(n, hb, case["graph"] + i, 1000 * seed + i)
                for i, (n, hb) in enumerate(_shapes(case))]
    return [_rmat(case["scale"], case["edges"], case["graph"], seed)]


def _host(a):
    return R.CSR(a[0], a[1], a[2].cpu().numpy(), a[3].cpu().numpy(), a[4].cpu().numpy())


# ------------------------------------------------------------------- cases
def _context():
    """The one handle that a program keeps for all its products."""
    if not _CTX:
        _CTX.append(R.Context(0))
    return _CTX[0]


def prepare(case, seed):
    k = case["kind"]
    ops = _operands(case, seed)
    s = {"kind": k, "ctx": _context(), "ops": ops}
    if k in ("host", "tiles"):
        s["ops"] = [_host(a) for a in ops]
    if k == "values":
        # a time stepper: its own handle, whose structure stays, its output
        # buffers, and the next step's values
        s["ctx"] = R.Context(0)
        a = ops[0]
        nnz, _ = s["ctx"].symbolic(a)
        s["out"] = _empty(a[0], nnz)
        s["ctx"].numeric(*s["out"])
        s["new"] = a[4] * (0.5 + torch.rand(a[4].shape, dtype=torch.float64, device=DEV,
                                            generator=_gen(seed + 7)))
    return s


def _empty(m, nnz, wide=False):
    return (torch.empty(m + 1, dtype=torch.int64 if wide else torch.int32, device=DEV),
            torch.empty(nnz, dtype=torch.int32, device=DEV),
            torch.empty(nnz, dtype=torch.float64, device=DEV))


def _multiply(ctx, a, b=None, op=R.RTT_OP_AB):
    nnz, _ = ctx.symbolic(a, b, op)
    out = _empty(a[0], nnz)
    ctx.numeric(*out)
    return out


def run(s):
    k, ctx, ops = s["kind"], s["ctx"], s["ops"]
    if k == "rmat_aat":
        return _multiply(ctx, ops[0], op=R.RTT_OP_AAT)
    if k == "rmat_wide":
        out = _empty(ops[0][0], ctx.symbolic64(ops[0], op=R.RTT_OP_AAT), wide=True)
        ctx.numeric64(*out)
        return out
    if k == "batched":
        return R.spgemm_batched(ctx, ops)
    if k == "values":
        ctx.numeric_values(s["new"], None, *s["out"])
        return s["out"]
    if k == "galerkin":
        a, p = ops
        ap = _multiply(ctx, a, p)
        pt = ctx.transpose(p)
        rap = _multiply(ctx, pt, (a[0], p[1], *ap))
        return {"ap": ap, "pt": pt[2:], "rap": rap}
    if k == "host":
        c = ctx.spgemm_csr_host(ops[0])
        return c.rowptr, c.col, c.val
    if k == "tiles":
        c = R.spgemm_tile(R.csr2tile_row_major(ops[0]), R.csr2tile_col_major(ops[0]))
        o = R.tile2csr(c, tile_dim=16)
        return {"csr": (o.rowptr, o.col, o.val),
                "tiles": [c["tile_ptr"], c["tile_columnidx"], c["tile_nnz"], c["tile_csr_Ptr"],
                          c["tile_csr_Col"], c["tile_csr_Value"], c["mask"]]}
    return _multiply(ctx, ops[0])


def tolerance(case):
    # FP64 sums in another order, about four times what the path measures
    # against exact(): grids and bands add up to some hundred terms (1.2e-16 to
    # 1.8e-16 in the 2-norm, 2.5e-15 at the worst entry), the hub rows of a
    # power-law graph many thousands (5.2e-15 in the 2-norm of a sample).
    if case["kind"].startswith("rmat"):
        return {"rel": 2e-14}
    return {"rel": 1e-15, "max": 2e-14}


# ------------------------------------------------- products in plain torch
def _rows_of(a):
    return torch.repeat_interleave(torch.arange(a[0], device=DEV), a[2].long().diff())


def _transposed(a):
    rows = _rows_of(a)
    key, order = torch.sort(a[3].long() * a[0] + rows)
    return _csr(a[1], a[0], key // a[0], key % a[0], a[4][order])


def _products(a, b):
    """Products of each row of a * b."""
    blen = b[2].long().diff()
    per = torch.zeros(a[0], dtype=torch.int64, device=DEV)
    return per.index_add_(0, _rows_of(a), blen[a[3].long()])


def _plain(a, b, step=1, most=1 << 27):
    """a * b by expanding all products, sorting them by (row, column) and adding
    the equal ones; every step-th row only, in blocks of about `most` products."""
    n, brp, blen = b[1], b[2].long(), b[2].long().diff()
    rows = _rows_of(a)
    if step > 1:
        take = rows % step == 0
        rows, acol, aval = rows[take], a[3].long()[take], a[4][take]
    else:
        acol, aval = a[3].long(), a[4]
    cnt = blen[acol]
    ends = torch.cumsum(cnt, 0)
    per_row = torch.zeros(a[0], dtype=torch.int64, device=DEV).index_add_(0, rows, cnt)
    rend = torch.cumsum(per_row, 0).cpu()
    at, r0, col, val, counts = 0, 0, [], [], torch.zeros(a[0], dtype=torch.int64, device=DEV)
    rptr = torch.searchsorted(rows, torch.arange(a[0] + 1, device=DEV)).cpu()
    while r0 < a[0]:
        done = int(rend[r0 - 1]) if r0 else 0
        r1 = max(r0 + 1, int(torch.searchsorted(rend, done + most, right=True)))
        e0, e1 = int(rptr[r0]), int(rptr[r1])
        c = cnt[e0:e1]
        own = torch.repeat_interleave(torch.arange(e0, e1, device=DEV), c)
        src = torch.arange(own.numel(), device=DEV) - (ends[own] - cnt[own] - at) + brp[acol[own]]
        key, order = torch.sort((rows[own] - r0) * n + b[3].long()[src])
        v = (aval[own] * b[4][src])[order]
        uniq, inv = torch.unique_consecutive(key, return_inverse=True)
        val.append(torch.zeros(uniq.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, v))
        col.append((uniq % n).int())
        counts[r0:r1] = torch.bincount(uniq // n, minlength=r1 - r0)
        at += own.numel()
        r0 = r1
    rp = torch.zeros(a[0] + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(counts, 0)
    return rp, torch.cat(col), torch.cat(val)


def exact(case, seed):
    k, ops = case["kind"], _operands(case, seed)
    if k == "batched":
        return [(c[0].int(), c[1], c[2]) for c in (_plain(a, a) for a in ops)]
    if k == "galerkin":
        a, p = ops
        ap, pt = _plain(a, p), _transposed(p)
        rap = _plain(pt, (a[0], p[1], *ap))
        return {"ap": (ap[0].int(), *ap[1:]), "pt": pt[2:], "rap": (rap[0].int(), *rap[1:])}
    a = ops[0]
    if k == "values":
        a = (*a[:4], a[4] * (0.5 + torch.rand(a[4].shape, dtype=torch.float64, device=DEV,
                                              generator=_gen(seed + 7))))
        rp, col, val = _plain(a, (*ops[0][:4], a[4]))
    else:
        rp, col, val = _plain(a, _transposed(a) if k in ("rmat_aat", "rmat_wide") else a)
    c = (rp if k == "rmat_wide" else rp.int(), col, val)
    if k == "tiles":
        return {"csr": c, "tiles": [None] * 7}
    return c


def work(case):
    """Operands read once, C written once (12 bytes an entry and the row
    pointers), two operations a product.  nnz(C) is counted on a sample of
    rows where the product is large."""
    k, ops = case["kind"], _operands(case, 0)
    size = lambda m, nnz: 4.0 * (m + 1) + 12.0 * nnz  # noqa: E731
    total = {"bytes": 0.0, "flops": 0.0}

    def product(a, b):
        per = float(_products(a, b).sum())
        step = max(1, int(per // 3e7))
        c = _plain(a, b, step)
        total["flops"] += 2.0 * per
        total["bytes"] += size(a[0], step * c[1].numel())
        return c

    def read(*mats):
        for a in mats:
            total["bytes"] += size(a[0], a[3].numel())

    read(*ops)
    if k == "galerkin":
        a, p = ops
        ap, pt = _plain(a, p), _transposed(p)
        ap = (a[0], p[1], *ap)
        product(a, p)
        product(pt, ap)
        read(p, pt)
    else:
        for a in ops:
            product(a, _transposed(a) if k in ("rmat_aat", "rmat_wide") else a)
    if k == "values":
        total["bytes"] -= 4.0 * (ops[0][3].numel() + ops[0][0] + 1)  # the values alone are new
    return total
