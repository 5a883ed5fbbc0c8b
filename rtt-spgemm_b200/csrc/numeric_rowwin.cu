// numeric_rowwin.cu - numeric step of heavy C tile rows, one scalar row of C
// per warp.
//
// A tile row whose C tiles need several windows of the tile-row kernel
// (numeric_flat.cu: at most 128 tiles and 2048 entries of all 16 rows
// together) walks all its A entries once per window, and a window then holds
// only a few entries of each row: on R-MAT 2^16 A*A^T that kernel set up 90
// million (A entry, window) pairs for 4.5 products each, and the set-up, not
// the products, was its time.  Here a warp owns one scalar row, so a window
// holds EW entries of that row alone: about 18 million pairs on the same
// product (6 of whole rows, 12 of pieces), and a banded row with scattered entries (about 256 entries in 80
// tiles, among 1,200 tiles of its tile row) is one window and one walk.
//
// A window lives in the warp's shared memory:
//   acc, ccol   the row's C entries of the window in CSR order: value, column
//   word        per non-empty C tile (slot): column mask << 16 | first entry
//   bm          tile column -> slot, as 32-tile words {bits, slot of the first}
// so a product at column c costs two shared loads to find its entry and a
// read-modify-write; no table spans the row's whole column range, and there
// are no probes.  The row's masks come from a row-by-row copy of the C tile
// masks: a lane reads 8 tiles' masks at once, a warp 256, since most tiles of
// the tile row have nothing in the row (one tile per lane took a third of all
// instructions on banded rows).  A's entries are taken in CSR order, 32 to a
// batch.  A row of one window cuts its B rows into items of 32 entries;
// otherwise a B row is walked in steps of 32 entries until a column lies past
// the window, and where it stopped is kept for the next window.  Every C entry
// is summed by one warp in the order of its row's A entries with fma: bitwise
// the tile-row kernel's value.
//
// Work is queued by k_row_plan: rows of little work in groups (neighbouring
// rows share B rows in L1), rows of much work cut into pieces, taken first.
// The cuts are tile columns that split B's entries into parts of like weight
// (the low columns of an R-MAT matrix hold most of them: cut into as many
// tiles each, one piece ran as long as all the rest), the same for all rows,
// so that k_row_prepare can list where every B row passes them and a piece finds
// its part of a B row by one load.  A piece finds its place in C's row by
// counting the masks before it, so no piece waits for another.
//
// What bounds it: issue and shared-memory latency at 14 to 20 warps per SM
// (about 5 warp instructions per product, 0.42 issued per cycle and scheduler
// on R-MAT 2^16; DRAM under 6 %).  The whole numeric step against the windows of
// the tile-row kernel (B200): R-MAT 2^16 A*A^T 20.3 -> 5.2 ms (this kernel 4.75),
// banded 200k with half-band 32 4.6 -> 2.2 ms (this kernel 1.9).
#include "rtt_internal.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

namespace rtt
{
namespace
{

constexpr int RW_WARPS = 2;      // warps per CTA (independent of each other)
constexpr int RW_CTAS = 10;      // CTAs per SM the registers leave room for
// C entries of a window (EW; half as many C tiles): 512, or 1024 for products
// of more than EW_LONG entries per row of C on average.  Longer windows walk
// the A entries less often, shorter ones leave room for more warps: whole
// products with 512 against 1024: 16 banded instances (500 entries per row)
// 3.55 and 3.82 ms, R-MAT 2^16 A*A^T (2,500 per row) 19.9 and 18.2 ms.
constexpr long long EW_LONG = 1024;
constexpr int RW_SPAN_MAX = 512; // 32-tile words of bm, at most
constexpr int RW_UNROLL = 4;     // B rows whose first 32 entries are loaded together
constexpr int RW_GROUP = 4;      // rows of one task, at most
// The table of B's parts is made up to this size (2 million rows of B); past it, or
// where it cannot be had, pieces search: the 4,000 longest rows of R-MAT 2^20 (6
// edges a row) times the matrix 41 ms with it, of 2^21 168 ms without.
constexpr size_t PART_BYTES_MAX = size_t(1) << 30;
constexpr int CUTS = 128; // parts of like weight that B's columns are cut into
// A entries of a row whose places in B are kept from one window to the next, by the
// longest row of A (in segments, a power of two between these; the least where it
// is not known).
constexpr int CURSORS_MIN = 256, CURSORS_MAX = 4096;
// Rows of more A entries than this drop those whose B rows end; shorter ones keep
// every entry's place in its own position, half the bytes (16 banded instances 3.36
// ms, 3.39 with lists for all rows).
constexpr int LIST_MIN = 2 * CURSORS_MIN;
constexpr int PLAN_WARPS = 8;
// Work of one task (products, and 4 for each pair of an A entry and a
// window): rows with more are cut.  Between these by nnz(C) / 2048, so that
// the row tasks of a product number some thousands: 2^14 against 2^16 took
// R-MAT 2^14 A^2 from 4.36 to 3.80 ms, 2^16 A*A^T from 18.2 to 19.5 ms.
// rtt_config.split_target counts a whole tile row's products, as for its
// window tasks: a task of one of its 16 rows gets a sixteenth, and no more than
// TARGET_MAX.
constexpr long long TARGET_MIN = 1ll << 14, TARGET_MAX = 1ll << 17;

struct RowTask
{
    int row0, rows; // rows: bit r = row row0 + r is part of the task; a
                    // piece's first part (low half) and end part (high half)
    int t0, t1;     // one row's piece: C tiles [t0, t1); t0 < 0: whole rows
};

// cut_tile[g]: first tile column of part g (g = CUTS: tilen).  The parts hold
// about as many of B's entries each, from about WEIGHT_SAMPLES of them counted
// per bin of tile columns (one bin per tile column up to WEIGHT_BINS): the
// columns of a power-law matrix differ by orders of magnitude.  One CTA.
constexpr int WEIGHT_SAMPLES = 1 << 15, WEIGHT_BINS = 8192, CUT_THREADS = 1024;
__global__ void __launch_bounds__(CUT_THREADS)
    k_cut_tiles(DevTiles B, int tilen, int *__restrict__ cut_tile)
{
    __shared__ int bins[WEIGHT_BINS], wtot[CUT_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int PER = WEIGHT_BINS / CUT_THREADS;
    for (int i = tid; i < WEIGHT_BINS; i += CUT_THREADS)
        bins[i] = 0;
    __syncthreads();
    const int per_bin = ceil_div(max(tilen, 1), WEIGHT_BINS);
    const int step = max(1, B.nnz / WEIGHT_SAMPLES);
#pragma unroll 8
    for (long long e = (long long)tid * step; e < B.nnz; e += (long long)CUT_THREADS * step)
    {
        const int J = __ldg(B.csr_col + e) >> 4;
        atomicAdd(&bins[min((unsigned)(J / per_bin), (unsigned)(WEIGHT_BINS - 1))], 1);
    }
    __syncthreads();
    // exclusive prefix sums of the bins, PER to a thread
    int v[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        v[i] = sum;
        sum += bins[tid * PER + i];
    }
    const int incl = warp_incl_scan(sum);
    if (lane == 31)
        wtot[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32)
    {
        const int w = wtot[tid], wi = warp_incl_scan(w);
        wtot[tid] = wi - w;
    }
    __syncthreads();
    const int before = wtot[tid >> 5] + incl - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i)
        bins[tid * PER + i] = before + v[i];
    __syncthreads();
    if (tid <= CUTS)
    {
        const int total = ceil_div(B.nnz, step); // samples taken
        int J = (int)((long long)tilen * tid / CUTS); // too few: as many tiles each
        if (total >= 4 * CUTS)
            J = (int)min((long long)tilen,
                         (long long)per_bin *
                             lower_bound(bins, 0, WEIGHT_BINS, (int)((long long)total * tid / CUTS)));
        cut_tile[tid] = tid == 0 ? 0 : tid == CUTS ? tilen : J;
    }
}

// One warp per C tile row: is it heavy (several windows of the tile-row
// kernel), and if so its rows' tasks.
template <int EW, int TW>
__global__ void __launch_bounds__(PLAN_WARPS * 32)
    k_row_plan(int tilem, int m, DevTiles A, DevTiles B,
               const int *__restrict__ c_tile_ptr, const int *__restrict__ c_tile_col,
               const int *__restrict__ c_tile_nnz, const int *__restrict__ csr_rowptr,
               const int *__restrict__ cut_tile, uint8_t *__restrict__ heavy,
               RowTask *__restrict__ big, int big_cap, RowTask *__restrict__ normal, int group,
               long long target, TaskQueue *q, long long *counters)
{
    const int lane = lane_id();
    const int I = blockIdx.x * PLAN_WARPS + (threadIdx.x >> 5);
    if (I >= tilem)
        return;
    const int cs0 = __ldg(c_tile_ptr + I), cs1 = __ldg(c_tile_ptr + I + 1);
    const int nrows = min(TD, m - I * TD);
    const int nt = cs1 - cs0;
    // lane r < 16: row r's C entries
    int nC = 0, e0 = 0, nA = 0;
    if (lane < nrows)
    {
        nC = __ldg(csr_rowptr + I * TD + lane + 1) - __ldg(csr_rowptr + I * TD + lane);
        e0 = __ldg(A.csr_rowptr + I * TD + lane);
        nA = __ldg(A.csr_rowptr + I * TD + lane + 1) - e0;
    }
    bool multi = false;
    if (nt > 0)
    {
        const int E = __ldg(c_tile_nnz + cs1) - __ldg(c_tile_nnz + cs0);
        multi = nt > FLAT_SLOT_CAP || E > FLAT_ACC;
        if (multi && nt <= FLAT_SLOT_CAP)
        {
            // the tile-row kernel's row windows: every row pair fits
            const int pair = nC + __shfl_xor_sync(FULL, nC, 1);
            multi = __any_sync(FULL, pair > FLAT_ACC);
        }
    }
    if (lane == 0)
        heavy[I] = multi;
    if (!multi)
        return;
    // products of every row (lane r: row r's)
    long long P = 0;
    for (int r = 0; r < nrows; ++r)
    {
        const int eb = __shfl_sync(FULL, e0, r), en = eb + __shfl_sync(FULL, nA, r);
        long long p = 0;
#pragma unroll 4
        for (int e = eb + lane; e < en; e += 32)
        {
            const int k = __ldg(A.csr_col + e);
            if ((unsigned)k < (unsigned)B.m)
                p += __ldg(B.csr_rowptr + k + 1) - __ldg(B.csr_rowptr + k);
        }
        p = warp_sum(p);
        if (lane == r)
            P = p;
    }
    // windows the row needs, and its work: products, (entry, window) pairs
    // and the tiles it reads
    const int nwin = max(1, max((nC + EW - 1) / EW, (min(nt, nC) + TW - 1) / TW));
    const long long work = P + 4ll * nA * nwin + nt;
    const bool live = lane < nrows && nC > 0;
    // a piece walks all the row's A entries, so it takes at least as much
    // work as finding its part of their B rows; `parts` cuts to a piece
    const long long size = max(target, 4ll * nA);
    int parts = 0;
    if (live && work > size + size / 2)
        for (parts = CUTS / 2; parts > 1 && work * parts > size * CUTS; parts /= 2)
            ;
    const int pieces = parts > 0 ? CUTS / parts : 0;
    // room for the pieces, row by row (a row that finds none stays whole)
    int pbase = -1;
    if (pieces > 0)
    {
        pbase = atomicAdd(&q->want, pieces);
        if (pbase + pieces > big_cap)
            pbase = -1;
        else
            atomicMax(&q->big, pbase + pieces);
    }
    const unsigned cutrows = __ballot_sync(FULL, pbase >= 0);
    for (unsigned rows = cutrows; rows != 0u; rows &= rows - 1u)
    {
        const int r = __ffs(rows) - 1;
        const int n = __shfl_sync(FULL, pieces, r), base = __shfl_sync(FULL, pbase, r);
        const int per = CUTS / n;
        for (int g = lane; g < n; g += 32)
        {
            const int g0 = g * per, g1 = g0 + per;
            big[base + g] = RowTask{I * TD + r, g0 | (g1 << 16),
                                    lower_bound(c_tile_col, cs0, cs1, __ldg(cut_tile + g0)),
                                    lower_bound(c_tile_col, cs0, cs1, __ldg(cut_tile + g1))};
        }
    }
    // the other rows: groups of `group` neighbours, or single rows when a
    // group would be more than a task's work
    const bool rest = live && pbase < 0;
    const unsigned rmask = __ballot_sync(FULL, rest);
    long long gwork = rest ? work : 0;
    for (int o = 1; o < group; o <<= 1)
        gwork += __shfl_xor_sync(FULL, gwork, o);
    const int g0 = lane & ~(group - 1);
    const bool single = gwork > target;
    const unsigned gmask = single ? (rest ? 1u : 0u)
                                  : (rmask >> g0) & ((1u << group) - 1u);
    const bool lead = single ? rest : (lane == g0 && gmask != 0u);
    const unsigned leads = __ballot_sync(FULL, lead);
    int nbase = 0;
    if (lane == 0 && leads != 0u)
        nbase = atomicAdd(&q->normal, __popc(leads)); // at most a task per row of C
    nbase = __shfl_sync(FULL, nbase, 0);
    if (lead)
        normal[nbase + __popc(leads & ((1u << lane) - 1u))] =
            RowTask{I * TD + (single ? lane : g0), (int)gmask, -1, 0};
    const bool several = lead && (__popc(gmask) > 1 || nwin > 1);
    const int ptot = warp_sum(pbase >= 0 ? pieces : 0);
    const int wide = __popc(__ballot_sync(FULL, several)) +
                     warp_sum(pbase >= 0 ? min(pieces, max(0, nwin - pieces)) : 0);
    P = warp_sum(P);
    if (lane == 0 && counters != nullptr)
    {
        // every product once; tasks; tasks of two or more windows
        atomicAdd((unsigned long long *)&counters[1], (unsigned long long)P);
        atomicAdd((unsigned long long *)&counters[2], (unsigned long long)(ptot + __popc(leads)));
        if (wide > 0)
            atomicAdd((unsigned long long *)&counters[3], (unsigned long long)wide);
    }
}

// Row-by-row copy of a heavy tile row's C tile masks: row r's masks start at
// row_masks(cs0, I, nt, r), 16-byte aligned and padded with zeroes to 8 tiles.
__host__ __device__ __forceinline__ size_t row_masks(int cs0, int I, int nt, int r)
{
    return (size_t)cs0 * TD + (size_t)I * 8 * TD + (size_t)r * ((nt + 7) & ~7);
}

// Where B's rows pass the cuts: part[k * (CUTS + 1) + g] = first entry of row
// k at or past part g's first column.  Long rows of C are cut at the same
// columns, so their pieces find their part of every B row by one load.  (No
// table for B's of more than PART_BYTES_MAX: their pieces search.)
//
// One launch for both: CTAs [0, tilem) copy a tile row's masks, the others list
// B's parts when some row of C was cut.
constexpr int PREP_THREADS = 128;
__global__ void __launch_bounds__(PREP_THREADS)
    k_row_prepare(int tilem, const int *__restrict__ c_tile_ptr,
                  const uint16_t *__restrict__ c_mask, const uint8_t *__restrict__ heavy,
                  uint16_t *__restrict__ maskt, DevTiles B, const int *__restrict__ cut_tile,
                  const TaskQueue *q, int *__restrict__ part)
{
    const int I = blockIdx.x;
    if (I >= tilem)
    {
        __shared__ int s_cut[CUTS + 1]; // first columns
        if (*(volatile const int *)&q->big == 0)
            return;
        for (int g = threadIdx.x; g <= CUTS; g += PREP_THREADS)
            s_cut[g] = first_column(cut_tile[g]);
        __syncthreads();
        constexpr int WARPS = PREP_THREADS / 32;
        const int warps = (int)(gridDim.x - tilem) * WARPS;
        for (int k = (I - tilem) * WARPS + (threadIdx.x >> 5); k < B.m; k += warps)
        {
            const int fs = min(max(__ldg(B.csr_rowptr + k), 0), B.nnz);
            const int fe = min(max(__ldg(B.csr_rowptr + k + 1), fs), B.nnz);
            for (int g = lane_id(); g <= CUTS; g += 32)
                part[(size_t)k * (CUTS + 1) + g] =
                    g == 0 ? fs : g == CUTS ? fe : lower_bound(B.csr_col, fs, fe, s_cut[g]);
        }
        return;
    }
    if (!heavy[I])
        return;
    const int cs0 = __ldg(c_tile_ptr + I), nt = __ldg(c_tile_ptr + I + 1) - cs0;
    const int ns = (nt + 7) & ~7;
    uint16_t *out = maskt + row_masks(cs0, I, nt, 0);
    // two neighbouring tiles per thread: 32-bit stores
    for (int i = threadIdx.x * 2; i < ns; i += 2 * PREP_THREADS)
    {
        uint4 u[2][2] = {};
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (i + x < nt)
            {
                const uint4 *mp = reinterpret_cast<const uint4 *>(c_mask + (size_t)(cs0 + i + x) * TD);
                u[x][0] = __ldg(mp);
                u[x][1] = __ldg(mp + 1);
            }
        const uint32_t w0[8] = {u[0][0].x, u[0][0].y, u[0][0].z, u[0][0].w,
                                u[0][1].x, u[0][1].y, u[0][1].z, u[0][1].w};
        const uint32_t w1[8] = {u[1][0].x, u[1][0].y, u[1][0].z, u[1][0].w,
                                u[1][1].x, u[1][1].y, u[1][1].z, u[1][1].w};
#pragma unroll
        for (int p = 0; p < 8; ++p)
        {
            *reinterpret_cast<uint32_t *>(out + (size_t)(2 * p) * ns + i) =
                __byte_perm(w0[p], w1[p], 0x5410);
            *reinterpret_cast<uint32_t *>(out + (size_t)(2 * p + 1) * ns + i) =
                __byte_perm(w0[p], w1[p], 0x7632);
        }
    }
}

template <int EW, int TW>
struct RowSmem // one warp's; bm (span words) follows
{
    double acc[EW];
    int4 ent[32]; // B row's start and length, a_ik
    int ccol[EW];
    uint32_t word[TW];
};

template <int EW, int TW>
constexpr size_t row_smem_bytes(int span)
{
    return (sizeof(RowSmem<EW, TW>) + sizeof(uint2) * (size_t)span + 15) / 16 * 16;
}

// TABLE: B's parts are listed (a kernel of its own: deciding at run time took 2 to 3 %
// of R-MAT 2^14 A^2 and 2^16 A*A^T).
template <int EW, int TW, bool TABLE>
__global__ void __launch_bounds__(RW_WARPS * 32, RW_CTAS)
    k_numeric_rowwin(DevTiles A, DevTiles B, long long nnzC, const int *__restrict__ c_tile_ptr,
                     const int *__restrict__ c_tile_col, const uint16_t *__restrict__ maskt,
                     const int *__restrict__ csr_rowptr, int *__restrict__ csr_col,
                     double *__restrict__ csr_val, const RowTask *__restrict__ big,
                     const RowTask *__restrict__ normal, TaskQueue *q, int span,
                     const int *__restrict__ part, const int *__restrict__ cut_tile, int4 *cursors,
                     int ncursors, int *err)
{
    static_assert(EW <= 65535, "entry offsets are 16 bits");
    extern __shared__ __align__(16) unsigned char rw_raw[];
    const int lane = lane_id();
    RowSmem<EW, TW> &S = *reinterpret_cast<RowSmem<EW, TW> *>(
        rw_raw + (size_t)(threadIdx.x >> 5) * row_smem_bytes<EW, TW>(span));
    uint2 *bm = reinterpret_cast<uint2 *>(&S + 1);
    const unsigned lt = (1u << lane) - 1u;
    int4 *cur = cursors + (size_t)(blockIdx.x * RW_WARPS + (threadIdx.x >> 5)) * ncursors;
    const int nbig = *(volatile int *)&q->big, ntask = nbig + *(volatile int *)&q->normal;
    for (;;)
    {
        int u = 0;
        if (lane == 0)
            u = atomicAdd(&q->head, 1);
        u = __shfl_sync(FULL, u, 0);
        if (u >= ntask)
            break;
        const int4 tk = __ldg(reinterpret_cast<const int4 *>(u < nbig ? big + u : normal + (u - nbig)));
        if (tk.z >= 0 && tk.z >= tk.w)
            continue; // a piece without tiles
        const bool piece = tk.z >= 0;
        for (unsigned rows = piece ? 1u : (unsigned)tk.y; rows != 0u; rows &= rows - 1u)
        {
            const int i = tk.x + __ffs(rows) - 1;
            const int I = i / TD, r = i % TD;
            const int cs0 = __ldg(c_tile_ptr + I), cs1 = __ldg(c_tile_ptr + I + 1);
            const int nt = cs1 - cs0;
            // the task's tiles of the row, counted from the tile row's first
            int t = piece ? tk.z - cs0 : 0;
            const int tend = piece ? tk.w - cs0 : nt;
            const uint16_t *mrow = maskt + row_masks(cs0, I, nt, r);
            const int *crow = c_tile_col + cs0;
            const int ea = __ldg(A.csr_rowptr + i), ee = __ldg(A.csr_rowptr + i + 1);
            int dst = __ldg(csr_rowptr + i);
            const int row_end = __ldg(csr_rowptr + i + 1);
            if (t > 0)
            {
                int before = 0;
                for (int x = lane; x < t; x += 32)
                    before += __popc((unsigned)__ldg(mrow + x));
                dst += warp_sum(before);
            }
            int lo = 0; // first column of the row's window (not its first in the task)
            bool first = true; // the row's first window in this task
            // A entries whose B rows go on past the window: the first of them in
            // cur (place, end, a_ik), then all from e_over on
            int kept = 0, e_over = ea;
            const bool lists = ee - ea > LIST_MIN;
            int2 *places = reinterpret_cast<int2 *>(cur); // (rows without lists: place, end)
            // a whole row ends with its last entry, a piece with its last tile
            while (t < tend && dst < row_end)
            {
                // ---- the window: tiles from t on, while they fit
                for (int x = lane; x < span; x += 32)
                    bm[x] = make_uint2(0u, 0xFFFFFFFFu);
                __syncwarp();
                int E = 0, T = 0, wlo = -1;
                bool full = false;
                auto put = [&](int x, uint32_t mk, int slot, int off) {
                    const int J = __ldg(crow + x);
                    const int w = ((J >> 5) - wlo) & (span - 1);
                    atomicOr(&bm[w].x, 1u << (J & 31));
                    atomicMin(&bm[w].y, (unsigned)slot);
                    S.word[slot] = (mk << 16) | (unsigned)off;
                };
                while (t < tend && !full && dst + E < row_end)
                {
                    // lane l: tiles x0 .. x0 + 7
                    const int x0 = (t & ~7) + 8 * lane;
                    uint32_t mk[8] = {};
                    if (x0 < tend)
                    {
                        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(mrow + x0));
                        const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int b = 0; b < 8; ++b)
                            mk[b] = (h[b >> 1] >> (16 * (b & 1))) & 0xFFFFu;
                        if (x0 < t || x0 + 8 > tend)
#pragma unroll
                            for (int b = 0; b < 8; ++b)
                                if (x0 + b < t || x0 + b >= tend)
                                    mk[b] = 0u;
                    }
                    int pc = 0, cnt = 0, fb = 0, lb = 0;
#pragma unroll
                    for (int b = 0; b < 8; ++b)
                    {
                        pc += __popc(mk[b]);
                        cnt += mk[b] != 0u;
                        lb = mk[b] != 0u ? b : lb;
                        fb = mk[7 - b] != 0u ? 7 - b : fb;
                    }
                    const unsigned ne = __ballot_sync(FULL, cnt > 0);
                    if (ne == 0u)
                    {
                        t = (t & ~7) + 256;
                        continue;
                    }
                    if (wlo < 0)
                        wlo = __shfl_sync(FULL, cnt > 0 ? __ldg(crow + x0 + fb) >> 5 : 0, __ffs(ne) - 1);
                    const int incl = warp_incl_scan(pc | (cnt << 16));
                    const int e1 = E + (incl & 0xFFFF), c1 = T + (incl >> 16);
                    const bool fits = cnt == 0 || (e1 <= EW && c1 <= TW &&
                                                   (__ldg(crow + x0 + lb) >> 5) - wlo < span);
                    const unsigned bad = __ballot_sync(FULL, !fits);
                    const int take = bad ? __ffs(bad) - 1 : 32;
                    if (take == 0 && T == 0)
                    {
                        // 8 tiles that do not lie in one span (they always
                        // hold few enough entries): one by one
#pragma unroll
                        for (int b = 0; b < 8; ++b)
                        {
                            const uint32_t m0 = __shfl_sync(FULL, mk[b], 0);
                            const int x = (t & ~7) + b;
                            if (m0 == 0u || full)
                                continue;
                            if ((__ldg(crow + x) >> 5) - wlo >= span)
                            {
                                t = x; // the next window's first tile
                                full = true;
                                continue;
                            }
                            if (lane == 0)
                                put(x, m0, T, E);
                            E += __popc(m0);
                            ++T;
                        }
                        break;
                    }
                    if (lane < take && cnt > 0)
                    {
                        int slot = c1 - cnt, off = e1 - pc;
#pragma unroll
                        for (int b = 0; b < 8; ++b)
                            if (mk[b] != 0u)
                            {
                                put(x0 + b, mk[b], slot, off);
                                ++slot;
                                off += __popc(mk[b]);
                            }
                    }
                    if (take > 0)
                    {
                        E = __shfl_sync(FULL, e1, take - 1);
                        T = __shfl_sync(FULL, c1, take - 1);
                        t = (t & ~7) + 8 * take;
                    }
                    full = bad != 0u && T > 0;
                }
                if (E == 0)
                    break; // no entries left in the piece
                // columns of the window: [lo, hi); the task's last window of
                // the row takes all that is left of the B rows
                const bool more = t < tend && dst + E < row_end;
                const int hi = more ? __ldg(crow + t) * TD : INT_MAX;
                for (int p = lane; p < E; p += 32)
                    S.acc[p] = 0.0;
                // the entry of column c in the window (the masks on the indexes
                // keep inconsistent operands inside this warp's shared memory)
                auto find = [&](int c) -> int {
                    const int J = c >> 4;
                    const uint2 bw = bm[((J >> 5) - wlo) & (span - 1)];
                    const unsigned slot = bw.y + __popc(bw.x & ((1u << (J & 31)) - 1u));
                    const uint32_t w = S.word[slot & (TW - 1)];
                    return (int)((w & 0xFFFFu) + __popc(__funnelshift_rc(w, 0u, 32 - (c & 15)))) &
                           (EW - 1);
                };
                // (no branch around the loads: those of other lanes stay in
                // bounds and are dropped)
                auto add = [&](bool ok, int pos, int c, double a, double b) {
                    const double sum = fma(a, b, S.acc[pos]);
                    if (ok)
                    {
                        S.acc[pos] = sum;
                        S.ccol[pos] = c; // every structural entry receives a product
                    }
                };
                // the first 32 entries of RW_UNROLL listed B rows
                struct Ahead
                {
                    int4 g[RW_UNROLL];
                    int c[RW_UNROLL];
                    double b[RW_UNROLL];
                };
                auto fetch = [&](Ahead &x, int j, int n) {
#pragma unroll
                    for (int v = 0; v < RW_UNROLL; ++v)
                    {
                        x.g[v] = S.ent[(j + v) & 31];
                        if (j + v >= n)
                            x.g[v].y = 0; // past the list: the word holds anything
                        x.c[v] = INT_MAX;
                        x.b[v] = 0.0;
                        if (lane < x.g[v].y)
                        {
                            x.c[v] = __ldg(B.csr_col + x.g[v].x + lane);
                            x.b[v] = __ldg(B.csr_val + x.g[v].x + lane);
                        }
                    }
                };
                // list entries [0, n), in order: their places are looked up
                // together, the adds follow one B row after the other.
                // WALK: a B row goes on until a column lies past the window;
                // where it stopped is left in the list.
                auto products = [&](int n, auto walk) {
                    constexpr bool WALK = decltype(walk)::value;
                    for (int j = 0; j < n; j += RW_UNROLL)
                    {
                        Ahead x;
                        fetch(x, j, n);
                        int pos[RW_UNROLL];
#pragma unroll
                        for (int v = 0; v < RW_UNROLL; ++v)
                            pos[v] = find(x.c[v]);
#pragma unroll
                        for (int v = 0; v < RW_UNROLL; ++v)
                        {
                            const double av = __hiloint2double(x.g[v].w, x.g[v].z);
                            add(x.c[v] < hi, pos[v], x.c[v], av, x.b[v]);
                            __syncwarp();
                            if (!WALK)
                                continue;
                            int done = __popc(__ballot_sync(FULL, x.c[v] < hi));
                            if (done == 32 && x.g[v].y > 32)
                                // the rest of a long B row, 128 entries at a time
                                for (unsigned f = 32 + lane, len = x.g[v].y;;
                                     f += 32 * RW_UNROLL)
                                {
                                    int lc[RW_UNROLL], lp[RW_UNROLL];
                                    double lb[RW_UNROLL];
#pragma unroll
                                    for (int u = 0; u < RW_UNROLL; ++u)
                                    {
                                        lc[u] = INT_MAX;
                                        lb[u] = 0.0;
                                        if (f + 32 * u < len)
                                        {
                                            lc[u] = __ldg(B.csr_col + x.g[v].x + (f + 32 * u));
                                            lb[u] = __ldg(B.csr_val + x.g[v].x + (f + 32 * u));
                                        }
                                    }
#pragma unroll
                                    for (int u = 0; u < RW_UNROLL; ++u)
                                        lp[u] = find(lc[u]);
                                    int got = 0;
#pragma unroll
                                    for (int u = 0; u < RW_UNROLL; ++u)
                                    {
                                        add(lc[u] < hi, lp[u], lc[u], av, lb[u]);
                                        got += __popc(__ballot_sync(FULL, lc[u] < hi));
                                    }
                                    __syncwarp();
                                    done += got;
                                    if (got < 32 * RW_UNROLL)
                                        break;
                                }
                            if (lane == 0 && j + v < n)
                                S.ent[j + v].x = x.g[v].x + done;
                        }
                    }
                };
                // ---- products: the row's A entries, 32 to a batch.  A B row
                // starts at its head, or at the piece's part of it; what the
                // window leaves is kept for the next one, and exhausted entries
                // leave the list (three hub rows of 200,000 entries with 3 products
                // each, walked in all of 128 pieces' 7 windows, took 156 ms, now 43;
                // R-MAT 2^16 A*A^T 7.44 -> 7.28 ms, 2^14 A^2 1.34 -> 1.32).  Entries past the list's room are searched again.
                //
                // entry e of A's row: its part of the B row from the window's first
                // column on
                auto entry = [&](int e, int &fs, int &fe, double &a) {
                    fs = fe = 0;
                    a = 0.0;
                    if (e >= ee)
                        return;
                    a = __ldg(A.csr_val + e);
                    const int k = __ldg(A.csr_col + e);
                    if ((unsigned)k < (unsigned)B.m)
                    {
                        // (parts lie in the row: k_row_prepare)
                        const bool listed = TABLE && piece;
                        const int *p = listed ? part + (size_t)k * (CUTS + 1) : B.csr_rowptr + k;
                        fs = __ldg(p + (listed ? tk.y & 0xFFFF : 0));
                        fe = __ldg(p + (listed ? tk.y >> 16 : 1));
                        fs = min(max(fs, 0), B.nnz);
                        fe = min(max(fe, fs), B.nnz);
                        if (!TABLE && piece)
                        {
                            fs = lower_bound(B.csr_col, fs, fe,
                                             first_column(__ldg(cut_tile + (tk.y & 0xFFFF))));
                            fe = lower_bound(B.csr_col, fs, fe,
                                             first_column(__ldg(cut_tile + (tk.y >> 16))));
                        }
                    }
                    if (!first)
                        fs = lower_bound(B.csr_col, fs, fe, lo);
                };
                int used = 0, e_next = e_over;
                if (first && !more)
                {
                    // one window: items of at most 32 B entries, in order
                    for (int q0 = ea; q0 < ee; q0 += 32)
                    {
                        int fs, fe;
                        double a;
                        entry(q0 + lane, fs, fe, a);
                        const int nch = (fe - fs + 31) >> 5;
                        const int cincl = warp_incl_scan(nch);
                        const int items = __shfl_sync(FULL, cincl, 31);
                        for (int i0 = 0; i0 < items; i0 += 32)
                        {
                            // item i0 + lane: its entry by shuffle search
                            const int qi = i0 + lane;
                            int own = 0;
#pragma unroll
                            for (int b = 16; b > 0; b >>= 1)
                                if (__shfl_sync(FULL, cincl, own + b - 1) <= qi)
                                    own += b;
                            own = min(own, 31);
                            const int k = qi - __shfl_sync(FULL, cincl - nch, own);
                            const int of = __shfl_sync(FULL, fs, own);
                            const int ol = __shfl_sync(FULL, fe - fs, own);
                            const double oa = __shfl_sync(FULL, a, own);
                            __syncwarp(); // the previous items are done
                            S.ent[lane] = make_int4(of + 32 * k, qi < items ? min(32, ol - 32 * k) : 0,
                                                    __double2loint(oa), __double2hiint(oa));
                            __syncwarp();
                            products(min(32, items - i0), std::false_type());
                        }
                    }
                }
                else
                {
                    bool room = true;
                    for (int q0 = -kept, qa = e_over; q0 < 0 || qa < ee;)
                    {
                        const bool listed_entry = q0 < 0;
                        int fs = 0, fe = 0;
                        double a = 0.0;
                        if (listed_entry)
                        {
                            const int at = kept + q0 + lane;
                            if (at < kept && lists)
                            {
                                const int4 c = cur[at];
                                fs = c.x;
                                fe = c.y;
                                a = __hiloint2double(c.w, c.z);
                            }
                            else if (at < kept)
                            {
                                const int2 c = places[at];
                                fs = c.x;
                                fe = c.y;
                                a = __ldg(A.csr_val + ea + at);
                            }
                            q0 += 32;
                        }
                        else
                        {
                            entry(qa + lane, fs, fe, a);
                            qa += 32;
                        }
                        // entries whose B row has nothing in the window leave the list
                        const bool has = fs < fe && (!more || __ldg(B.csr_col + fs) < hi);
                        const unsigned list = __ballot_sync(FULL, has);
                        const int at = __popc(list & lt);
                        __syncwarp(); // the previous batch (or the zeroes) is done
                        if (has)
                            S.ent[at] = make_int4(fs, fe - fs, __double2loint(a), __double2hiint(a));
                        __syncwarp();
                        products(__popc(list), std::true_type());
                        __syncwarp();
                        if (more && !lists)
                        {
                            const int i = (listed_entry ? kept + q0 : qa - ea) - 32 + lane;
                            if (i < ee - ea)
                                places[i] = make_int2(has ? S.ent[at].x : fs, fe);
                            used = ee - ea;
                            e_next = ee;
                        }
                        else if (more)
                        {
                            const int rest = has ? S.ent[at].x : fs;
                            const unsigned live = __ballot_sync(FULL, rest < fe);
                            room = room && used + __popc(live) <= ncursors; // (a list never grows)
                            if (room)
                            {
                                if (rest < fe)
                                    cur[used + __popc(live & lt)] =
                                        make_int4(rest, fe, __double2loint(a), __double2hiint(a));
                                used += __popc(live);
                                if (!listed_entry)
                                    e_next = min(qa, ee);
                            }
                        }
                    }
                }
                kept = used;
                e_over = e_next;
                first = false;
                __syncwarp();
                // ---- the window's entries into C
                if (dst < 0 || (long long)dst + E > nnzC || dst + E > row_end)
                {
                    if (lane == 0)
                        set_error(err, DERR_NUM_BOUNDS);
                    break;
                }
                for (int p = lane; p < E; p += 32)
                {
                    csr_val[(size_t)dst + p] = S.acc[p];
                    csr_col[(size_t)dst + p] = S.ccol[p];
                }
                __syncwarp(); // before the next window overwrites them
                dst += E;
                lo = hi;
            }
        }
    }
}

template <int EW, int TW>
int rowwin_run(Workspace &ws, const DevTiles &A, const DevTiles &B, SymbolicOut &S,
               const NumericConfig &cfg)
{
    cudaStream_t s = ws.stream;
    // 32-tile words of the column index: a power of two
    int span = 32;
    while (span < RW_SPAN_MAX && span * 32 < S.tilen)
        span *= 2;
    const size_t smem = RW_WARPS * row_smem_bytes<EW, TW>(span);
    // one wave of warps that take tasks from the queue
    const int sms = ws.sms;
    int per_sm = 0;
    for (auto k : {k_numeric_rowwin<EW, TW, true>, k_numeric_rowwin<EW, TW, false>})
        RTT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    RTT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_numeric_rowwin<EW, TW, true>,
                                                           RW_WARPS * 32, smem));
    const int grid = std::max(1, per_sm * sms);
    // scratch, before anything is enqueued: without it the caller runs the
    // windows of the tile-row kernel
    const int big_cap = (int)std::min<long long>(S.nnz / 128 + (1 << 16), 1 << 24);
    RTT_CHECK(S.r_normal.ensure(sizeof(RowTask) * ((size_t)S.m + 16), s));
    RTT_CHECK(S.r_big.ensure(sizeof(RowTask) * (size_t)big_cap, s));
    RTT_CHECK(S.r_mask.ensure(sizeof(uint16_t) * row_masks(S.numtile, S.tilem, 0, 0), s));
    RTT_CHECK(S.r_cut.ensure(sizeof(int) * (CUTS + 1), s));
    int ncursors = CURSORS_MIN;
    while (ncursors < CURSORS_MAX && ncursors < A.max_row_segs)
        ncursors *= 2;
    RTT_CHECK(S.r_cursor.ensure(sizeof(int4) * (size_t)grid * RW_WARPS * ncursors, s));
    RTT_CHECK(S.w_queue.ensure(sizeof(TaskQueue), s));
    // the table of B's parts where it is small enough and can be had
    const size_t part_bytes = sizeof(int) * (size_t)B.m * (CUTS + 1) + 16;
    bool table = part_bytes <= PART_BYTES_MAX;
    if (table)
    {
        const int st = S.r_part.ensure(part_bytes, s);
        table = st == RTT_OK;
        if (!table && st != RTT_ERR_OUT_OF_MEMORY)
            return st;
    }
    int *part = table ? S.r_part.as<int>() : nullptr;
    RTT_CUDA(cudaMemsetAsync(S.w_queue.p, 0, sizeof(TaskQueue), s));
    int *cut_tile = S.r_cut.as<int>();
    k_cut_tiles<<<1, CUT_THREADS, 0, s>>>(B, S.tilen, cut_tile);
    // a task per row when the groups would leave warps without work: from 64 rows an
    // SM two, from 256 four (a quarter of that: banded 20k numeric step 244 us
    // against 234; four times: 224, and 306 against 318 on banded 50k, half-band 8)
    const int group = S.m >= 64 * RW_GROUP * sms ? RW_GROUP : S.m >= 64 * sms ? 2 : 1;
    const long long target =
        cfg.split_target > 0 ? std::max(1ll, std::min(TARGET_MAX, (long long)cfg.split_target / TD))
                             : std::max(TARGET_MIN, std::min(TARGET_MAX, S.nnz / 2048));
    k_row_plan<EW, TW><<<ceil_div(S.tilem, PLAN_WARPS), PLAN_WARPS * 32, 0, s>>>(
        S.tilem, S.m, A, B, S.c_tile_ptr.as<int>(), S.c_tile_col.as<int>(),
        S.c_tile_nnz.as<int>(), cfg.csr_rowptr, cut_tile, S.w_heavy.as<uint8_t>(),
        S.r_big.as<RowTask>(), big_cap, S.r_normal.as<RowTask>(), group,
        target, S.w_queue.as<TaskQueue>(), cfg.counters);
    k_row_prepare<<<S.tilem + (table ? 8 * sms : 0), PREP_THREADS, 0, s>>>(
        S.tilem, S.c_tile_ptr.as<int>(), S.c_mask.as<uint16_t>(), S.w_heavy.as<uint8_t>(),
        S.r_mask.as<uint16_t>(), B, cut_tile, S.w_queue.as<TaskQueue>(), part);
    ws.launches += 3;
    auto kern = table ? k_numeric_rowwin<EW, TW, true> : k_numeric_rowwin<EW, TW, false>;
    // on the side stream, beside the tile-row CTAs of the other tile rows
    RTT_CUDA(cudaEventRecord(ws.fork_ev, s));
    RTT_CUDA(cudaStreamWaitEvent(ws.side, ws.fork_ev, 0));
    kern<<<grid, RW_WARPS * 32, smem, ws.side>>>(
        A, B, S.nnz, S.c_tile_ptr.as<int>(), S.c_tile_col.as<int>(), S.r_mask.as<uint16_t>(),
        cfg.csr_rowptr, cfg.csr_col, cfg.csr_val, S.r_big.as<RowTask>(), S.r_normal.as<RowTask>(),
        S.w_queue.as<TaskQueue>(), span, part, cut_tile, S.r_cursor.as<int4>(), ncursors, ws.err.as<int>());
    ws.launches++;
    RTT_CUDA(cudaEventRecord(ws.join_ev, ws.side));
    return RTT_OK;
}

} // namespace

int numeric_rowwin_device(Workspace &ws, const DevTiles &A, const DevTiles &B, SymbolicOut &S,
                          const NumericConfig &cfg)
{
    const int st = S.nnz > EW_LONG * S.m ? rowwin_run<1024, 512>(ws, A, B, S, cfg)
                                         : rowwin_run<512, 256>(ws, A, B, S, cfg);
    if (st == RTT_ERR_OUT_OF_MEMORY) // leave the room to what runs instead
        for (DevBuf *b : {&S.r_normal, &S.r_big, &S.r_mask, &S.r_cursor, &S.r_part})
            b->release();
    return st;
}

} // namespace rtt
