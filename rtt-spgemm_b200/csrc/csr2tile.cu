// csr2tile.cu - CSR -> 16x16 tile CSR on sm_100a.
//
// Semantics follow csr2tile_row_major (reference src/csr2tile.h:196-259):
// tiles of a tile row in ascending column order, per-tile exclusive row
// offsets (u8), entries of a (tile, row) in CSR order, packed column byte
// (row << 4) | col, mask bit (15 - col); and csr2tile_col_major (:261-478):
// the same tiles with per-tile data in tile-CSC order and plain column bytes.
//
// Fast path (every row's tile column index non-decreasing, i.e. sorted CSR):
// a half-warp owns one tile row, one lane per scalar row.  Each lane walks
// its row with a cursor; the half-warp takes the minimum pending tile column
// (4 xor-shuffles), every lane consumes its entries of that tile, a
// half-warp scan turns per-row counts into the tile's row offsets, and the
// lanes write their entries at tile base + row offset.  Reads of col/val are
// sequential per lane and the 16 rows of a tile row are contiguous in
// memory, so the half-warp streams one contiguous CSR slice.
// Generic path (unsorted rows): a warp per tile row extracts tile columns in
// ascending order and places entries with match_any ranking, which keeps CSR
// order inside each (tile, row).
#include "rtt_internal.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <algorithm>
#include <climits>

namespace rtt
{
namespace
{

// ------------------------------------------------------------ validation
// The checks and the row segments go over the entries, not the rows: a warp
// takes a chunk of consecutive entries, 256 at a time, whatever rows they
// belong to, so a hub row costs what its entries cost.  (A warp
// per 32 rows left the 32 hub rows of an R-MAT matrix to one warp: 460 us for
// the checks of R-MAT 2^16's 1M entries and 1 ms for its segments; now 14 and
// 19 us.  96^3 stencil, 23.4M entries: 45 us and 110 us before, 42 and 126 us.)  The
// row starts among the 256 entries are marked in a shared bitmap.
constexpr int CS_WARPS = 8, CS_THREADS = CS_WARPS * 32;
constexpr int CS_BLOCK = 256, CS_WORDS = CS_BLOCK / 32;
constexpr int CS_CTAS_MAX = 4096; // CTAs of entries, at most

// First index in [0, n) with a[i] >= key, by one warp 32 probes at a time (a
// need not be sorted: then some index).
__device__ __forceinline__ int warp_lower_bound(const int *__restrict__ a, int n, long long key)
{
    int lo = 0, hi = n; // the answer lies in [lo, hi]
    while (hi - lo > 0)
    {
        const int step = (hi - lo + 31) / 32;
        const long long i = lo + (long long)lane_id() * step;
        const unsigned less = __ballot_sync(FULL, i < hi && __ldg(a + min(i, (long long)n - 1)) < key);
        const int k = __popc(less); // probes below key, the first k of a sorted list
        if (k == 0)
            return lo;
        const long long nlo = lo + (long long)(k - 1) * step + 1;
        hi = (int)min((long long)hi, lo + (long long)k * step);
        lo = (int)min(nlo, (long long)hi);
    }
    return lo;
}

// The rest of mark_rows where many rows are empty: every entry is looked up in the
// row pointer.
__device__ __forceinline__ int look_up_rows(uint32_t *bits, const int *__restrict__ rowptr, int rows,
                                         int cursor, long long s0, long long end)
{
    const int lane = lane_id();
    const int last = cursor + warp_lower_bound(rowptr + cursor, rows - cursor, end);
    __syncwarp();
    for (int i = 0; i < CS_WORDS; ++i)
    {
        const long long j = s0 + i * 32 + lane;
        bool start = false;
        if (j < end)
        {
            const int r = lower_bound(rowptr, cursor, last, (int)j);
            start = r < last && __ldg(rowptr + r) == (int)j;
        }
        const unsigned st = __ballot_sync(FULL, start);
        if (lane == 0)
            bits[i] |= st;
    }
    return last;
}

// Marks the rows that start in [s0, end), from row `cursor` on (the first that
// starts at or past s0), in the warp's cleared bitmap; returns the first row
// that starts at or past end.  The rows are walked, 32 and then 128 at a time;
// past WALK_STEPS of those, among empty rows, the entries are looked up in the row
// pointer instead (the walk alone left the 18 million empty rows of a matrix of 5
// million entries to two warps: 276 ms of symbolic step, now 3.0).
constexpr int WALK_STEPS = 16;
__device__ __forceinline__ int mark_rows(uint32_t *bits, const int *__restrict__ rowptr, int rows,
                                         int cursor, long long s0, long long end)
{
    const int lane = lane_id();
    if (lane < CS_WORDS)
        bits[lane] = 0u;
    __syncwarp();
    // (unsigned: rows may number INT_MAX)
    auto mark = [&](unsigned r) -> bool {
        const long long x = r < (unsigned)rows ? (long long)__ldg(rowptr + r) : LLONG_MAX;
        const bool in = x < end;
        if (in && x >= s0)
            atomicOr(&bits[(x - s0) >> 5], 1u << ((x - s0) & 31));
        return in;
    };
    int n = __popc(__ballot_sync(FULL, mark((unsigned)cursor + lane)));
    cursor += n;
    if (n == 32)
    {
        for (int step = 0; step < WALK_STEPS; ++step)
        {
            bool in[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                in[q] = mark((unsigned)cursor + q * 32 + lane);
            n = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                n += __popc(__ballot_sync(FULL, in[q]));
            cursor += n;
            if (n < 128)
                break;
        }
        if (n == 128)
            cursor = look_up_rows(bits, rowptr, rows, cursor, s0, end);
    }
    __syncwarp();
    return cursor;
}

// Row pointer and column checks, the flags, and how many row segments start in
// each warp's chunk (warp_cnt) and each CTA's (cta_cnt), when not null.
// flags[0]: some row's tile column decreases (needs the generic path)
// flags[1]: some row's column decreases (entries not sorted inside rows)
// flags[2]: some row repeats a column
// unmade (one of two words beside the error word): set for errors and flags[0];
// what follows then makes no segments and no index.  A word of its own beside the error word, which is hardly ever written:
// flags[0], cleared for every matrix, took the small products' kernels 0.5 us each.
__global__ void __launch_bounds__(CS_THREADS, 4)
    k_csr_scan(int m, int n, int nnz, const int *__restrict__ rowptr, const int *__restrict__ col,
               int ctas, int blocks, int *__restrict__ cta_cnt, int *__restrict__ warp_cnt,
               int *err, int *flags, int *unmade)
{
    __shared__ uint32_t s_bits[CS_WARPS][CS_WORDS];
    __shared__ int s_total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    bool bad = false;
    for (long long r = blockIdx.x * (long long)CS_THREADS + tid; r < m;
         r += (long long)gridDim.x * CS_THREADS)
    {
        const int b = rowptr[r], e = rowptr[r + 1];
        bad |= b < 0 || e < b || e > nnz || (r == 0 && b != 0) || (r == m - 1 && e != nnz);
    }
    if (tid == 0)
        s_total = 0;
    if (__syncthreads_or(bad))
    {
        if (tid == 0)
        {
            set_error(err, DERR_CSR_ROWPTR);
            if (unmade != nullptr)
                atomicOr(unmade, 1);
        }
        return;
    }
    if ((int)blockIdx.x >= ctas)
        return;
    const long long span = (long long)blocks * CS_BLOCK;
    const long long c0 = (blockIdx.x * (long long)CS_WARPS + warp) * span;
    const long long c1 = min((long long)nnz, c0 + span);
    int segs = 0;
    bool col_bad = false, tile_dec = false, col_dec = false, col_dup = false;
    if (c0 < c1)
    {
        uint32_t *bits = s_bits[warp];
        const bool vec = (reinterpret_cast<uintptr_t>(col) & 15) == 0;
        int cursor = warp_lower_bound(rowptr, m, c0);
        for (long long s0 = c0; s0 < c1; s0 += CS_BLOCK)
        {
            // a lane's 4 neighbouring entries, twice
            int4 v[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const long long j = s0 + h * 128 + lane * 4;
                if (vec && j + 4 <= c1)
                    v[h] = __ldg(reinterpret_cast<const int4 *>(col + j));
                else
                    v[h] = make_int4(j < c1 ? __ldg(col + j) : 0, j + 1 < c1 ? __ldg(col + j + 1) : 0,
                                     j + 2 < c1 ? __ldg(col + j + 2) : 0,
                                     j + 3 < c1 ? __ldg(col + j + 3) : 0);
            }
            int last = s0 > 0 ? __ldg(col + s0 - 1) : 0;
            cursor = mark_rows(bits, rowptr, m, cursor, s0, min(c1, s0 + CS_BLOCK));
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const long long j = s0 + h * 128 + lane * 4;
                unsigned st = bits[h * 4 + (lane >> 3)] >> ((lane & 7) * 4);
                if (j == 0)
                    st |= 1u;
                int p = __shfl_up_sync(FULL, v[h].w, 1);
                if (lane == 0)
                    p = last;
                last = __shfl_sync(FULL, v[h].w, 31);
                const int c[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
                const int k = (int)max(0ll, min(4ll, c1 - j)); // entries of the chunk
#pragma unroll
                for (int i = 0; i < 4; ++i)
                {
                    const bool in = i < k, start = (st >> i) & 1u;
                    col_bad |= in && (unsigned)c[i] >= (unsigned)n;
                    if (in && !start && c[i] <= p)
                    {
                        tile_dec |= (c[i] >> 4) < (p >> 4);
                        col_dec |= c[i] < p;
                        col_dup |= c[i] == p;
                    }
                    segs += in && (start || (unsigned)(c[i] ^ p) >= 16u);
                    p = c[i];
                }
            }
            __syncwarp(); // before the bitmap is cleared
        }
    }
    const unsigned fl = __reduce_or_sync(FULL, (tile_dec ? 1u : 0u) | (col_dec ? 2u : 0u) |
                                                   (col_dup ? 4u : 0u) | (col_bad ? 8u : 0u));
    if (lane == 0 && fl != 0u)
    {
        if (fl & 8u)
            set_error(err, DERR_CSR_COL);
        if ((fl & 9u) && unmade != nullptr)
            atomicOr(unmade, 1);
        for (int f = 0; f < 3; ++f)
            if ((fl >> f) & 1u)
                atomicOr(&flags[f], 1);
    }
    if (cta_cnt == nullptr)
        return;
    segs = warp_sum(segs);
    if (lane == 0)
    {
        warp_cnt[blockIdx.x * CS_WARPS + warp] = segs;
        atomicAdd(&s_total, segs);
    }
    __syncthreads();
    if (tid == 0)
        cta_cnt[blockIdx.x] = s_total;
}

// Row segments of a CSR whose rows have non-decreasing tile columns: every
// maximal run of a row's entries inside one tile column J becomes the segment
// (J << 16) | mask, mask bit (15 - c) for each column c of the run - the row's
// 16-bit row mask in tile J, as csr2tile writes it into mask[].  A run's mask
// is OR-ed over the lanes of its 32 entries by shuffles; what it has in the
// next 32 is carried along, and past the warp's chunk it is followed entry by
// entry.  word[i] = {segments that start in entries 32 i .. 32 i + 31, segments
// before them}, for segments_before.
// Nothing is written where unmade is set.
__global__ void __launch_bounds__(CS_THREADS, 4)
    k_csr_segments(int m, int nnz, const int *__restrict__ rowptr, const int *__restrict__ col,
                   int blocks, const int *__restrict__ cta_cnt, const int *__restrict__ warp_cnt,
                   uint2 *__restrict__ word, unsigned long long *__restrict__ seg,
                   const int *unmade)
{
    __shared__ uint32_t s_bits[CS_WARPS][CS_WORDS], s_starts[CS_WARPS][CS_WORDS];
    __shared__ int s_pre[CS_WARPS][CS_WORDS], s_base;
    const int stop = *(volatile const int *)unmade; // (looked at behind the first loads)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // segments of the CTAs and warps before
    if (tid == 0)
        s_base = 0;
    __syncthreads();
    int before = 0;
    for (int i = tid; i < (int)blockIdx.x; i += CS_THREADS)
        before += __ldg(cta_cnt + i);
    before = warp_sum(before);
    if (lane == 0 && before)
        atomicAdd(&s_base, before);
    const int wc = lane < warp ? __ldg(warp_cnt + blockIdx.x * CS_WARPS + lane) : 0;
    __syncthreads();
    if (stop != 0)
        return;
    int base = s_base + warp_sum(wc);
    const long long span = (long long)blocks * CS_BLOCK;
    const long long c0 = (blockIdx.x * (long long)CS_WARPS + warp) * span;
    const long long c1 = min((long long)nnz, c0 + span);
    if (c0 >= c1)
        return;
    uint32_t *bits = s_bits[warp], *starts = s_starts[warp];
    int *pre = s_pre[warp];
    int cursor = warp_lower_bound(rowptr, m, c0);
    // the run that is open at the end of the last 32 entries
    int open_at = -1, open_T = 0;
    unsigned open_mk = 0;
    for (long long s0 = c0; s0 < c1; s0 += CS_BLOCK)
    {
        int c[CS_WORDS];
#pragma unroll
        for (int i = 0; i < CS_WORDS; ++i)
            c[i] = s0 + i * 32 + lane < c1 ? __ldg(col + s0 + i * 32 + lane) : 0;
        int last = s0 > 0 ? __ldg(col + s0 - 1) : 0;
        cursor = mark_rows(bits, rowptr, m, cursor, s0, min(c1, s0 + CS_BLOCK));
        int n = 0; // segments of the block so far
#pragma unroll
        for (int i = 0; i < CS_WORDS; ++i)
        {
            const long long j = s0 + i * 32 + lane;
            int p = __shfl_up_sync(FULL, c[i], 1);
            if (lane == 0)
                p = last;
            last = __shfl_sync(FULL, c[i], 31);
            const bool in = j < c1;
            const bool start = in && (j == 0 || ((bits[i] >> lane) & 1u) || (c[i] >> 4) != (p >> 4));
            const unsigned st = __ballot_sync(FULL, start);
            if (lane == 0)
            {
                starts[i] = st;
                pre[i] = n;
            }
            unsigned mk = in ? 0x8000u >> (c[i] & 15) : 0u;
            // entries before the first start belong to the open run
            const int fs = st ? __ffs(st) - 1 : 32;
            open_mk |= __reduce_or_sync(FULL, lane < fs ? mk : 0u);
            if (st != 0u)
            {
                // OR over the lanes up to the next start
                const unsigned later = lane == 31 ? 0u : st >> (lane + 1);
                const int next = later ? lane + __ffs(later) : 32;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const unsigned v = __shfl_down_sync(FULL, mk, o);
                    if (lane + o < next)
                        mk |= v;
                }
                const int lst = 31 - __clz(st), at = base + n + __popc(st & ((1u << lane) - 1u));
                if (start && lane != lst)
                    seg[at] = ((unsigned long long)(c[i] >> 4) << 16) | mk;
                if (lane == 0 && open_at >= 0)
                    seg[open_at] = ((unsigned long long)open_T << 16) | open_mk;
                open_at = base + n + __popc(st) - 1;
                open_T = __shfl_sync(FULL, c[i] >> 4, lst);
                open_mk = __shfl_sync(FULL, mk, lst);
                n += __popc(st);
            }
        }
        __syncwarp();
        if (lane < CS_WORDS && s0 + lane * 32 < c1)
            word[(s0 >> 5) + lane] = make_uint2(starts[lane], (unsigned)(base + pre[lane]));
        base += n;
        __syncwarp(); // before the bitmaps are written again
    }
    if (open_at >= 0)
    {
        // the last run's entries past the chunk: up to the next row's start
        // (row `cursor`) or another tile column
        const long long stop = min((long long)nnz, cursor <= m ? (long long)__ldg(rowptr + cursor)
                                                               : (long long)nnz);
        for (long long t0 = c1;; t0 += 32)
        {
            const long long t = t0 + lane;
            const int ct = t < stop ? __ldg(col + t) : -1;
            const unsigned out = __ballot_sync(FULL, ct < 0 || (ct >> 4) != open_T);
            const int k = out ? __ffs(out) - 1 : 32;
            open_mk |= __reduce_or_sync(FULL, lane < k ? 0x8000u >> (ct & 15) : 0u);
            if (out)
                break;
        }
        if (lane == 0)
            seg[open_at] = ((unsigned long long)open_T << 16) | open_mk;
    }
    // rows that start past the last entry
    if (c1 == nnz && (nnz & 31) == 0 && lane == 0)
        word[nnz >> 5] = make_uint2(0u, (unsigned)base);
}

// Segments before row r's first entry (all of them for r = m).
__device__ __forceinline__ int segments_before(const int *__restrict__ rowptr,
                                               const uint2 *__restrict__ word, int r)
{
    const int d = __ldg(rowptr + r);
    const uint2 w = __ldg(word + (d >> 5));
    return (int)w.y + __popc(w.x & ((1u << (d & 31)) - 1u));
}

// seg_ptr where no tile index is made from the segments (k_seg_tiles writes it).
__global__ void k_seg_rows(int m, const int *__restrict__ rowptr, const uint2 *__restrict__ word,
                           int *__restrict__ seg_ptr, const int *unmade)
{
    const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (r <= m && *(volatile const int *)unmade == 0)
        seg_ptr[r] = segments_before(rowptr, word, (int)r);
}

// Tile index of every tile row from its rows' segments: the tile columns of
// its segments as a bitmap, a warp per tile row, windows of ST_BITS tile
// columns, or merged where its few segments span many windows.  Tile row I's list
// starts at its first segment, so its place needs no count of the tiles before it:
// tile_ptr[I] = seg_ptr[16 I], tile_end[I] one past its last tile.  seg_ptr[r] is
// the number of segments before row r's first entry.  out[0] += tiles, out[1] = the
// most segments of a row.
// One wave of ST_CTAS CTAs per SM (32 registers), not a CTA for every 4 tile
// rows: the 156,000 of a matrix of 10 million short rows queued for the two words
// of out.  That matrix 361 -> 198 us (10 and 12 CTAs per SM: 237), 96^3 stencil 51
// -> 39; 200,000 rows of 5 entries among 10 million columns 472 -> 39, by the merge.
constexpr int ST_WARPS = 4, ST_WORDS = 256, ST_BITS = ST_WORDS * 32, ST_CTAS = 16;
__global__ void __launch_bounds__(ST_WARPS * 32, ST_CTAS)
    k_seg_tiles(int m, int tilem, const int *__restrict__ rowptr, const uint2 *__restrict__ word,
                int *__restrict__ seg_ptr, const unsigned long long *__restrict__ seg,
                int *__restrict__ tile_ptr, int *__restrict__ tile_end,
                int *__restrict__ tile_col, int *out, const int *unmade)
{
    __shared__ uint32_t s_bits[ST_WARPS][ST_WORDS];
    __shared__ int s_count, s_max;
    const int stop = *(volatile const int *)unmade; // (looked at behind the first loads)
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t *bits = s_bits[warp];
    int count = 0, longest = 0;
    if (threadIdx.x == 0)
        s_count = s_max = 0;
    __syncthreads();
    // (tile rows and columns number at most 2^27)
    for (int I = blockIdx.x * ST_WARPS + warp; I < tilem; I += gridDim.x * ST_WARPS)
    {
        // lane r < 16: row r's segments
        const unsigned r = (unsigned)I * TD + lane; // (rows may number INT_MAX)
        const int d = lane <= TD ? __ldg(rowptr + min(r, (unsigned)m)) : 0;
        if (stop != 0)
            break;
        const uint2 wd = __ldg(word + (d >> 5));
        int p = (int)wd.y + __popc(wd.x & ((1u << (d & 31)) - 1u));
        int e = __shfl_down_sync(FULL, p, 1);
        if ((lane < TD || I == tilem - 1) && lane <= TD && r <= (unsigned)m)
            seg_ptr[r] = p;
        if (lane >= TD)
            p = e = 0;
        const int s0 = __shfl_sync(FULL, p, 0), s1 = __shfl_sync(FULL, e, TD - 1);
        int lo = INT_MAX, hi = -1;
        if (p < e)
        {
            lo = (int)(__ldg(seg + p) >> 16);
            hi = (int)(__ldg(seg + e - 1) >> 16);
        }
        lo = warp_min(lo);
        hi = warp_max(hi);
        const int most = (int)__reduce_max_sync(FULL, (unsigned)(e - p));
        int n = 0;
        // a window costs its words (32 units) and a read of 32 segments per unit,
        // the merge a step per segment (2 units: 4 left 20,000 rows of 600 entries
        // among 10 million columns at 10.1 ms of set-up, 2 and 1 take 8.0)
        const int windows = hi < 0 ? 0 : (hi - lo) / ST_BITS + 1;
        const bool merge =
            windows > 1 && (long long)windows * ((s1 - s0) / 32 + 32) > 2ll * (s1 - s0);
        if (merge)
        {
            // lane r walks row r's segments, one load ahead; the smallest
            // column of the 16 is the next tile
            int q = p;
            int cur = q < e ? (int)(__ldg(seg + q) >> 16) : INT_MAX;
            int next = q + 1 < e ? (int)(__ldg(seg + q + 1) >> 16) : INT_MAX;
            for (;;)
            {
                const int T = warp_min(cur);
                if (T == INT_MAX)
                    break;
                if (lane == 0)
                    tile_col[s0 + n] = T;
                ++n;
                if (cur == T)
                {
                    cur = next;
                    ++q;
                    next = q + 1 < e ? (int)(__ldg(seg + q + 1) >> 16) : INT_MAX;
                }
            }
        }
        for (int w = lo; w <= hi && !merge; w += ST_BITS)
        {
            const int nwords = (min(hi + 1 - w, ST_BITS) + 31) >> 5;
            for (int i = lane; i < nwords; i += 32)
                bits[i] = 0u;
            __syncwarp();
            // (four loads in flight: a hub's tile row has tens of thousands)
            for (unsigned q = s0 + lane; q < (unsigned)s1; q += 128)
            {
                unsigned long long v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    v[u] = q + 32 * u < (unsigned)s1 ? __ldg(seg + q + 32 * u) : ~0ull;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    const int d = (int)(v[u] >> 16) - w;
                    if ((unsigned)d < 32u * nwords)
                        atomicOr(&bits[d >> 5], 1u << (d & 31));
                }
            }
            __syncwarp();
            for (int q0 = 0; q0 < nwords; q0 += 32)
            {
                uint32_t set = q0 + lane < nwords ? bits[q0 + lane] : 0u;
                const int v = __popc(set), incl = warp_incl_scan(v);
                int at = s0 + n + incl - v;
                for (; set != 0u; set &= set - 1u)
                    tile_col[at++] = w + (q0 + lane) * 32 + __ffs(set) - 1;
                n += __shfl_sync(FULL, incl, 31);
            }
            __syncwarp();
        }
        if (lane == 0)
        {
            tile_ptr[I] = s0;
            tile_end[I] = s0 + n;
        }
        count += n;
        longest = max(longest, most);
    }
    if (lane == 0)
    {
        atomicAdd(&s_count, count);
        atomicMax(&s_max, longest);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (s_count > 0)
            atomicAdd(&out[0], s_count);
        if (s_max > *(volatile int *)&out[1])
            atomicMax(&out[1], s_max);
    }
}

// -------------------------------------------------------------- fast path
__global__ void __launch_bounds__(256) k_c2t_count(int m, int tilem, const int *__restrict__ rowptr,
                                                   const int *__restrict__ col, int *__restrict__ cnt,
                                                   const uint8_t *__restrict__ heavy)
{
    const int lane = threadIdx.x & 31, hl = lane & 15;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int I = gw * 2 + (lane >> 4);
    // heavy tile rows are counted by k_c2t_heavy_count
    const bool mine = I < tilem && !(heavy != nullptr && heavy[I]);
    int p = 0, e = 0;
    if (mine && I * TD + hl < m)
    {
        p = rowptr[I * TD + hl];
        e = rowptr[I * TD + hl + 1];
    }
    int cur = p < e ? (__ldg(col + p) >> 4) : INT_MAX;
    int count = 0;
    for (;;)
    {
        const int T = half_min(cur);
        const bool has = T != INT_MAX;
        if (!__any_sync(FULL, has))
            break;
        if (has)
        {
            ++count;
            while (p < e && (__ldg(col + p) >> 4) == T)
                ++p;
            cur = p < e ? (__ldg(col + p) >> 4) : INT_MAX;
        }
    }
    if (mine && hl == 0)
        cnt[I] = count;
}

__global__ void __launch_bounds__(256) k_c2t_fill(int m, int tilem, const int *__restrict__ rowptr,
                                                  const int *__restrict__ col,
                                                  const double *__restrict__ val,
                                                  const int *__restrict__ tile_ptr,
                                                  int *__restrict__ o_tcol, int *__restrict__ o_trow,
                                                  int *__restrict__ o_tnnz, uint8_t *__restrict__ o_ptr,
                                                  uint8_t *__restrict__ o_col,
                                                  double *__restrict__ o_val,
                                                  uint16_t *__restrict__ o_mask, int packed, int *err,
                                                  const uint8_t *__restrict__ heavy)
{
    const int lane = threadIdx.x & 31, hl = lane & 15;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int I = gw * 2 + (lane >> 4);
    // heavy tile rows are filled by k_c2t_heavy_fill
    const bool tr_ok = I < tilem && !(heavy != nullptr && heavy[I]);
    int p = 0, e = 0, base = 0, t = 0, tend = 0;
    if (tr_ok)
    {
        base = rowptr[min(I * TD, m)];
        t = tile_ptr[I];
        tend = tile_ptr[I + 1];
        if (I * TD + hl < m)
        {
            p = rowptr[I * TD + hl];
            e = rowptr[I * TD + hl + 1];
        }
    }
    int cur = p < e ? (__ldg(col + p) >> 4) : INT_MAX;
    for (;;)
    {
        const int T = half_min(cur);
        const bool has = T != INT_MAX;
        if (!__any_sync(FULL, has))
            break;
        int q = p;
        if (has)
            while (q < e && (__ldg(col + q) >> 4) == T)
                ++q;
        const int c = q - p;
        const int incl = half_incl_scan(c);
        const int excl = incl - c;
        const int total = __shfl_sync(FULL, incl, (lane & 16) | 15);
        if (has)
        {
            if (t >= tend)
            {
                set_error(err, DERR_C2T_OVERFLOW);
            }
            else
            {
                o_ptr[(size_t)t * TD + hl] = (uint8_t)excl;
                uint16_t mk = 0;
                int dst = base + excl;
                for (int j = p; j < q; ++j, ++dst)
                {
                    const int cc = __ldg(col + j) & 15;
                    mk |= (uint16_t)(0x8000u >> cc);
                    o_col[dst] = (uint8_t)(packed ? ((hl << 4) | cc) : cc);
                    o_val[dst] = __ldg(val + j);
                }
                o_mask[(size_t)t * TD + hl] = mk;
                if (hl == 0)
                {
                    o_tcol[t] = T;
                    o_trow[t] = I;
                    o_tnnz[t] = base;
                }
            }
            base += total;
            ++t;
            p = q;
            cur = p < e ? (__ldg(col + p) >> 4) : INT_MAX;
        }
    }
}

// ------------------------------------------------ fast path, heavy tile rows
// A tile row holding a row with thousands of entries (an R-MAT hub) spans
// thousands of tile columns; the half-warp above takes them one per step and
// becomes the tail of the launch.  Such tile rows get a CTA each: the tile
// columns of the 16 rows become a bitmap, a tile's index is the rank of its
// bit, and since each row's tile columns are non-decreasing, the entries of
// one (tile, row) are one run in the row (at most 16 entries unless columns
// repeat), found and written by the thread that holds its first entry.  Entry
// order inside a (tile, row) stays the CSR order, as on the half-warp path.
constexpr int HV_ENTRIES = 2048;            // tile rows with more entries take this path
constexpr int HV_WORDS = 4096;              // bitmap words: 131072 tile columns
constexpr int HV_THREADS = 256;
constexpr int HV_CHUNK = 2048;              // tiles written per pass

struct HeavySmem
{
    uint32_t bits[HV_WORDS];
    int pre[HV_WORDS + 1];      // set bits before each word
    uint8_t cnt[HV_CHUNK][TD];  // entries per (tile of the pass, row)
    int tbase[HV_CHUNK + 1];    // entries of the pass's tiles before each tile
    int rs[TD + 1], re[TD];     // rows' entry ranges in the pass
    int rpre[TD + 1];           // prefix of the ranges' lengths
    int jlo, count;
};

// First entry of [b, e) whose tile column is >= J (the row's tile columns are
// non-decreasing).
__device__ __forceinline__ int tile_lower_bound(const int *col, int b, int e, int J)
{
    while (b < e)
    {
        const int mid = (b + e) >> 1;
        if ((__ldg(col + mid) >> 4) < J)
            b = mid + 1;
        else
            e = mid;
    }
    return b;
}

// Marks heavy tile rows (flag and list); thread per tile row.
__global__ void k_c2t_heavy_mark(int m, int tilem, const int *__restrict__ rowptr,
                                 const int *__restrict__ col, uint8_t *__restrict__ heavy,
                                 int *__restrict__ list, int *__restrict__ count)
{
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= tilem)
        return;
    const int r0 = I * TD, r1 = min(r0 + TD, m);
    bool hv = rowptr[r1] - rowptr[r0] > HV_ENTRIES;
    if (hv)
    {
        int lo = INT_MAX, hi = -1;
        for (int r = r0; r < r1; ++r)
        {
            const int b = rowptr[r], e = rowptr[r + 1];
            if (b < e)
            {
                lo = min(lo, __ldg(col + b) >> 4);
                hi = max(hi, __ldg(col + e - 1) >> 4);
            }
        }
        hv = hi >= lo && hi - lo < HV_WORDS * 32;
    }
    heavy[I] = hv;
    if (hv)
        list[atomicAdd(count, 1)] = I;
}

// The heavy tile row's tile-column bitmap and the set bits before each word.
__device__ void heavy_bitmap(HeavySmem &S, int I, int m, const int *__restrict__ rowptr,
                             const int *__restrict__ col)
{
    const int tid = threadIdx.x;
    const int r0 = I * TD, r1 = min(r0 + TD, m);
    if (tid == 0)
        S.jlo = INT_MAX;
    for (int i = tid; i < HV_WORDS; i += HV_THREADS)
        S.bits[i] = 0u;
    __syncthreads();
    if (tid < r1 - r0)
    {
        const int b = rowptr[r0 + tid];
        if (b < rowptr[r0 + tid + 1])
            atomicMin(&S.jlo, __ldg(col + b) >> 4);
    }
    __syncthreads();
    const int jlo = S.jlo;
    const int s0 = rowptr[r0], s1 = rowptr[r1];
    for (int j = s0 + tid; j < s1; j += HV_THREADS)
    {
        const int d = (__ldg(col + j) >> 4) - jlo;
        if ((unsigned)d < (unsigned)(HV_WORDS * 32)) // checked by the mark kernel
            atomicOr(&S.bits[d >> 5], 1u << (d & 31));
    }
    __syncthreads();
    if (tid < 32)
    {
        int run = 0;
        for (int q0 = 0; q0 < HV_WORDS; q0 += 32)
        {
            const int v = __popc(S.bits[q0 + tid]);
            const int incl = warp_incl_scan(v);
            S.pre[q0 + tid] = run + incl - v;
            run += __shfl_sync(FULL, incl, 31);
        }
        if (tid == 0)
        {
            S.pre[HV_WORDS] = run;
            S.count = run;
        }
    }
    __syncthreads();
}

// Tile column of the k-th set bit.
__device__ __forceinline__ int heavy_select(const HeavySmem &S, int k)
{
    int lo = 0, hi = HV_WORDS - 1; // last word with pre <= k
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (S.pre[mid] <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    uint32_t w = S.bits[lo];
    for (int i = S.pre[lo]; i < k; ++i)
        w &= w - 1;
    return S.jlo + lo * 32 + __ffs(w) - 1;
}

__device__ __forceinline__ int heavy_rank(const HeavySmem &S, int J)
{
    const int d = J - S.jlo;
    return S.pre[d >> 5] + __popc(S.bits[d >> 5] & ((1u << (d & 31)) - 1u));
}

__global__ void __launch_bounds__(HV_THREADS)
    k_c2t_heavy_count(int m, const int *__restrict__ list, const int *__restrict__ count,
                      const int *__restrict__ rowptr, const int *__restrict__ col,
                      int *__restrict__ cnt)
{
    extern __shared__ __align__(16) unsigned char hv_dyn[];
    HeavySmem &S = *reinterpret_cast<HeavySmem *>(hv_dyn);
    const int n = *count;
    for (int li = blockIdx.x; li < n; li += gridDim.x)
    {
        const int I = list[li];
        heavy_bitmap(S, I, m, rowptr, col);
        if (threadIdx.x == 0)
            cnt[I] = S.count;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(HV_THREADS)
    k_c2t_heavy_fill(int m, const int *__restrict__ list, const int *__restrict__ count,
                     const int *__restrict__ rowptr, const int *__restrict__ col,
                     const double *__restrict__ val, const int *__restrict__ tile_ptr,
                     int *__restrict__ o_tcol, int *__restrict__ o_trow,
                     int *__restrict__ o_tnnz, uint8_t *__restrict__ o_ptr,
                     uint8_t *__restrict__ o_col, double *__restrict__ o_val,
                     uint16_t *__restrict__ o_mask, int packed, int *err)
{
    extern __shared__ __align__(16) unsigned char hv_dyn[];
    HeavySmem &S = *reinterpret_cast<HeavySmem *>(hv_dyn);
    const int tid = threadIdx.x;
    const int n = *count;
    for (int li = blockIdx.x; li < n; li += gridDim.x)
    {
        const int I = list[li];
        const int r0 = I * TD, nr = min(TD, m - r0);
        heavy_bitmap(S, I, m, rowptr, col);
        const int ntiles = S.count, t0 = tile_ptr[I];
        if (t0 + ntiles != tile_ptr[I + 1])
        {
            if (tid == 0)
                set_error(err, DERR_C2T_OVERFLOW);
            __syncthreads();
            continue;
        }
        int base = rowptr[r0]; // entries of the tile row before the pass
        for (int k0 = 0; k0 < ntiles; k0 += HV_CHUNK)
        {
            const int k1 = min(k0 + HV_CHUNK, ntiles), nk = k1 - k0;
            // the pass's entries: per row, the run of tile columns [Ja, Jb]
            if (tid < TD)
            {
                int b = 0, e = 0;
                if (tid < nr)
                {
                    const int Ja = heavy_select(S, k0), Jb = heavy_select(S, k1 - 1);
                    const int rb = rowptr[r0 + tid], rend = rowptr[r0 + tid + 1];
                    b = tile_lower_bound(col, rb, rend, Ja);
                    e = tile_lower_bound(col, b, rend, Jb + 1);
                }
                S.rs[tid] = b;
                S.re[tid] = e;
            }
            for (int i = tid; i < nk * TD; i += HV_THREADS)
                S.cnt[i >> 4][i & 15] = 0;
            __syncthreads();
            if (tid == 0)
            {
                int t = 0;
                for (int r = 0; r < TD; ++r)
                {
                    S.rpre[r] = t;
                    t += S.re[r] - S.rs[r];
                }
                S.rpre[TD] = t;
            }
            __syncthreads();
            const int total = S.rpre[TD];
            // pass 1: run lengths per (tile, row); a run starts where the
            // tile column changes inside the row
            for (int i = tid; i < total; i += HV_THREADS)
            {
                int r = 0;
                while (S.rpre[r + 1] <= i)
                    ++r;
                const int j = S.rs[r] + (i - S.rpre[r]);
                const int J = __ldg(col + j) >> 4;
                if (j == S.rs[r] || (__ldg(col + j - 1) >> 4) != J)
                {
                    int e = j + 1;
                    while (e < S.re[r] && (__ldg(col + e) >> 4) == J)
                        ++e;
                    if (e - j > 255) // repeated columns beyond a u8 row offset
                        set_error(err, DERR_C2T_OVERFLOW);
                    S.cnt[heavy_rank(S, J) - k0][r] = (uint8_t)min(e - j, 255);
                }
            }
            __syncthreads();
            // per tile: row offsets, size, column, tile row, empty masks
            for (int t = tid; t < nk; t += HV_THREADS)
            {
                int run = 0;
                const size_t g = (size_t)(t0 + k0 + t);
#pragma unroll
                for (int r = 0; r < TD; ++r)
                {
                    o_ptr[g * TD + r] = (uint8_t)run;
                    if (S.cnt[t][r] == 0)
                        o_mask[g * TD + r] = 0;
                    run += S.cnt[t][r];
                }
                S.tbase[t + 1] = run;
                o_tcol[g] = heavy_select(S, k0 + t);
                o_trow[g] = I;
            }
            __syncthreads();
            if (tid < 32)
            {
                int acc = 0;
                for (int q0 = 0; q0 < nk; q0 += 32)
                {
                    const int v = q0 + tid < nk ? S.tbase[q0 + tid + 1] : 0;
                    const int incl = warp_incl_scan(v);
                    if (q0 + tid < nk)
                        S.tbase[q0 + tid] = acc + incl - v;
                    acc += __shfl_sync(FULL, incl, 31);
                }
                if (tid == 0)
                    S.tbase[nk] = acc;
            }
            __syncthreads();
            for (int t = tid; t < nk; t += HV_THREADS)
                o_tnnz[t0 + k0 + t] = base + S.tbase[t];
            // pass 2: each run's first entry writes the run and its mask
            for (int i = tid; i < total; i += HV_THREADS)
            {
                int r = 0;
                while (S.rpre[r + 1] <= i)
                    ++r;
                const int j = S.rs[r] + (i - S.rpre[r]);
                const int J = __ldg(col + j) >> 4;
                if (j == S.rs[r] || (__ldg(col + j - 1) >> 4) != J)
                {
                    const int t = heavy_rank(S, J) - k0;
                    int off = 0;
                    for (int rr = 0; rr < r; ++rr)
                        off += S.cnt[t][rr];
                    int dst = base + S.tbase[t] + off;
                    const int len = S.cnt[t][r]; // the run, as counted in pass 1
                    uint16_t mk = 0;
                    for (int e = j; e < j + len; ++e, ++dst)
                    {
                        const int cc = __ldg(col + e) & 15;
                        mk |= (uint16_t)(0x8000u >> cc);
                        o_col[dst] = (uint8_t)(packed ? ((r << 4) | cc) : cc);
                        o_val[dst] = __ldg(val + e);
                    }
                    o_mask[(size_t)(t0 + k0 + t) * TD + r] = mk;
                }
            }
            base += S.tbase[nk];
            __syncthreads();
        }
    }
}

// ----------------------------------------------------------- generic path
__global__ void __launch_bounds__(256) k_c2t_count_generic(int m, int tilem,
                                                           const int *__restrict__ rowptr,
                                                           const int *__restrict__ col,
                                                           int *__restrict__ cnt)
{
    const int lane = threadIdx.x & 31;
    const int I = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (I >= tilem)
        return;
    const int s0 = rowptr[I * TD], s1 = rowptr[min(I * TD + TD, m)];
    int prev = -1, count = 0;
    for (;;)
    {
        int mn = INT_MAX;
        for (int j = s0 + lane; j < s1; j += 32)
        {
            int T = __ldg(col + j) >> 4;
            if (T > prev && T < mn)
                mn = T;
        }
        mn = warp_min(mn);
        if (mn == INT_MAX)
            break;
        ++count;
        prev = mn;
    }
    if (lane == 0)
        cnt[I] = count;
}

__global__ void __launch_bounds__(128) k_c2t_fill_generic(
    int m, int tilem, const int *__restrict__ rowptr, const int *__restrict__ col,
    const double *__restrict__ val, const int *__restrict__ tile_ptr, int *__restrict__ o_tcol,
    int *__restrict__ o_trow, int *__restrict__ o_tnnz, uint8_t *__restrict__ o_ptr,
    uint8_t *__restrict__ o_col, double *__restrict__ o_val, uint16_t *__restrict__ o_mask,
    int packed, int *err)
{
    __shared__ int s_rp[4][TD + 1];
    __shared__ int s_cnt[4][TD];
    __shared__ int s_cur[4][TD];
    __shared__ unsigned s_mask[4][TD];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int I = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (I >= tilem)
        return;
    const int r0 = I * TD, nrows = min(TD, m - r0);
    if (lane <= TD)
        s_rp[w][lane] = rowptr[r0 + min(lane, nrows)];
    __syncwarp();
    const int s0 = s_rp[w][0], s1 = s_rp[w][nrows];
    int prev = -1, t = tile_ptr[I];
    const int tend = tile_ptr[I + 1];
    int base = s0;
    const unsigned lt = (1u << lane) - 1u;
    for (;;)
    {
        int mn = INT_MAX;
        for (int j = s0 + lane; j < s1; j += 32)
        {
            int T = __ldg(col + j) >> 4;
            if (T > prev && T < mn)
                mn = T;
        }
        const int T = warp_min(mn);
        if (T == INT_MAX)
            break;
        prev = T;
        if (lane < TD)
        {
            s_cnt[w][lane] = 0;
            s_cur[w][lane] = 0;
            s_mask[w][lane] = 0;
        }
        __syncwarp();
        for (int j = s0 + lane; j < s1; j += 32)
        {
            if ((__ldg(col + j) >> 4) == T)
            {
                int r = 0;
                while (r + 1 < nrows && s_rp[w][r + 1] <= j)
                    ++r;
                atomicAdd(&s_cnt[w][r], 1);
            }
        }
        __syncwarp();
        int c = lane < TD ? s_cnt[w][lane] : 0;
        int incl = half_incl_scan(c);
        int excl = incl - c;
        int total = __shfl_sync(FULL, incl, 15);
        if (t >= tend)
        {
            set_error(err, DERR_C2T_OVERFLOW);
            return;
        }
        if (lane < TD)
        {
            o_ptr[(size_t)t * TD + lane] = (uint8_t)excl;
            s_cnt[w][lane] = excl;
        }
        __syncwarp();
        // place entries in CSR order, chunk by chunk
        for (int j0 = s0; j0 < s1; j0 += 32)
        {
            const int j = j0 + lane;
            bool in = false;
            int r = 0, cc = 0;
            if (j < s1)
            {
                const int cj = __ldg(col + j);
                if ((cj >> 4) == T)
                {
                    in = true;
                    cc = cj & 15;
                    while (r + 1 < nrows && s_rp[w][r + 1] <= j)
                        ++r;
                }
            }
            const int key = in ? r : (TD + lane);
            const unsigned peers = __match_any_sync(FULL, key);
            if (in)
            {
                const int rank = __popc(peers & lt);
                const int dst = base + s_cnt[w][r] + s_cur[w][r] + rank;
                o_col[dst] = (uint8_t)(packed ? ((r << 4) | cc) : cc);
                o_val[dst] = __ldg(val + j);
                atomicOr(&s_mask[w][r], 0x8000u >> cc);
            }
            __syncwarp();
            if (in && (peers & lt) == 0)
                s_cur[w][r] += __popc(peers);
            __syncwarp();
        }
        if (lane < TD)
            o_mask[(size_t)t * TD + lane] = (uint16_t)s_mask[w][lane];
        if (lane == 0)
        {
            o_tcol[t] = T;
            o_trow[t] = I;
            o_tnnz[t] = base;
        }
        base += total;
        ++t;
        __syncwarp();
    }
}

// Stable insertion sort of every (tile, row) segment by column byte: the
// in-tile order of csr2tile_col_major for rows whose columns are unsorted.
__global__ void k_sort_tile_rows(int numtile, const int *__restrict__ tnnz,
                                 const uint8_t *__restrict__ ptr, uint8_t *__restrict__ colb,
                                 double *__restrict__ v)
{
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= numtile * TD)
        return;
    int t = x >> 4, r = x & 15;
    int b = tnnz[t] + ptr[(size_t)t * TD + r];
    int e = r == TD - 1 ? tnnz[t + 1] : tnnz[t] + ptr[(size_t)t * TD + r + 1];
    for (int i = b + 1; i < e; ++i)
    {
        uint8_t kc = colb[i];
        double kv = v[i];
        int key = kc & 15;
        int j = i - 1;
        while (j >= b && (colb[j] & 15) > key)
        {
            colb[j + 1] = colb[j];
            v[j + 1] = v[j];
            --j;
        }
        colb[j + 1] = kc;
        v[j + 1] = kv;
    }
}

__global__ void k_set_int(int *p, int v) { *p = v; }

// ------------------------------------------------------ tile CSC / col-major
__global__ void k_iota(int *a, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        a[i] = i;
}

__global__ void k_lower_bound_ptr(const int *__restrict__ sorted_keys, int nkeys, int nbins,
                                  int *__restrict__ ptr)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nbins)
        return;
    ptr[b] = lower_bound(sorted_keys, 0, nkeys, b);
}

__global__ void k_gather_int(const int *__restrict__ src, const int *__restrict__ idx, int n,
                             int *__restrict__ dst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        dst[i] = src[idx[i]];
}

__global__ void k_tile_counts(const int *__restrict__ tnnz, const int *__restrict__ order, int n,
                              int *__restrict__ cnt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        int t = order[i];
        cnt[i] = tnnz[t + 1] - tnnz[t];
    }
}

// warp per destination tile: copy row offsets, mask and entries
__global__ void k_copy_tiles_colmajor(int n, const int *__restrict__ order,
                                      const int *__restrict__ src_tnnz,
                                      const uint8_t *__restrict__ src_ptr,
                                      const uint16_t *__restrict__ src_mask,
                                      const uint8_t *__restrict__ src_col,
                                      const double *__restrict__ src_val,
                                      const int *__restrict__ dst_tnnz, uint8_t *__restrict__ dst_ptr,
                                      uint16_t *__restrict__ dst_mask, uint8_t *__restrict__ dst_col,
                                      double *__restrict__ dst_val)
{
    const int lane = threadIdx.x & 31;
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= n)
        return;
    const int t = order[p];
    if (lane < TD)
    {
        dst_ptr[(size_t)p * TD + lane] = src_ptr[(size_t)t * TD + lane];
        dst_mask[(size_t)p * TD + lane] = src_mask[(size_t)t * TD + lane];
    }
    const int sb = src_tnnz[t], cnt = src_tnnz[t + 1] - sb, db = dst_tnnz[p];
    for (int i = lane; i < cnt; i += 32)
    {
        dst_col[db + i] = src_col[sb + i] & 15;
        dst_val[db + i] = src_val[sb + i];
    }
}

// ----------------------------------------------------------- CSR transpose
// A warp per 32 rows: a lane its own row up to 16 entries, the longer rows by
// the whole warp (a thread per row left an R-MAT hub row to one thread: 64 us
// at 2^16, now 7).  Nothing is written after an error (a row pointer not yet
// checked on the host).
__global__ void k_row_ids(int m, const int *__restrict__ rowptr, int *__restrict__ rows,
                          const int *err)
{
    if (*(volatile const int *)err != 0)
        return;
    const int lane = lane_id();
    const long long r0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * 32;
    if (r0 >= m)
        return;
    const int r = (int)min(r0 + lane, (long long)m - 1);
    const int b = rowptr[r], e = r0 + lane < m ? rowptr[r + 1] : b;
    const bool lng = e - b > 16;
    if (!lng)
        for (int j = b; j < e; ++j)
            rows[j] = r;
    for (unsigned ls = __ballot_sync(FULL, lng); ls != 0u; ls &= ls - 1u)
    {
        const int q = __ffs(ls) - 1;
        const int qb = __shfl_sync(FULL, b, q), qe = __shfl_sync(FULL, e, q);
        for (int j = qb + lane; j < qe; j += 32)
            rows[j] = (int)r0 + q;
    }
}

__global__ void k_gather_transpose(int nnz, const int *__restrict__ order,
                                   const int *__restrict__ rows, const double *__restrict__ val,
                                   int *__restrict__ t_col, double *__restrict__ t_val)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnz)
        return;
    int src = order[i];
    t_col[i] = rows[src];
    t_val[i] = val[src];
}

int bits_for(int maxval)
{
    int b = 1;
    while (b < 31 && (1 << b) <= maxval)
        ++b;
    return b;
}

int sort_pairs(Workspace &ws, const int *keys_in, int *keys_out, const int *vals_in, int *vals_out,
               int n, int max_key)
{
    if (n <= 0)
        return RTT_OK;
    size_t bytes = 0;
    const int end_bit = bits_for(max_key);
    RTT_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys_in, keys_out, vals_in, vals_out,
                                             n, 0, end_bit, ws.stream));
    RTT_CHECK(ws.scan_tmp.ensure(bytes, ws.stream));
    RTT_CUDA(cub::DeviceRadixSort::SortPairs(ws.scan_tmp.p, bytes, keys_in, keys_out, vals_in,
                                             vals_out, n, 0, end_bit, ws.stream));
    ws.launches += 3;
    return RTT_OK;
}

inline int grid_for(long long threads, int block) { return (int)((threads + block - 1) / block); }

// The warps' chunks of k_csr_scan and k_csr_segments: `blocks` times 256
// entries each.  One block for small matrices, so that they spread over the
// SMs; up to 8, where a chunk's own set-up (its first row, the segments before
// it) is spread over more entries, while every SM keeps 8 CTAs (64^3 stencil:
// the scan 18 us against 24 with one block; the symbolic step with a block per 400
// / 1200 / 4000 CTAs 489 / 497 / 506 us, of 96^3 1437 / 1437 / 1449); more only to
// stay within CS_CTAS_MAX.
struct CsChunks
{
    int blocks, ctas;
    explicit CsChunks(int nnz)
    {
        const int all = ceil_div(ceil_div(nnz, CS_BLOCK), CS_WARPS); // CTAs of one block a warp
        blocks = std::max(std::max(1, std::min(8, all / 1200)), ceil_div(all, CS_CTAS_MAX));
        ctas = ceil_div(all, blocks);
    }
    // CTAs of the scan: those of the entries, and enough for the row pointer
    int grid(int m) const
    {
        return std::max(1, std::max(ctas, std::min(1024, ceil_div(m, 4 * CS_THREADS))));
    }
};

} // namespace

int csr2tile_device(Workspace &ws, int m, int n, int nnz, const int *rowptr, const int *col,
                    const double *val, TileBufs &out, bool packed_col, bool sort_within_rows,
                    bool segments, bool payload, bool defer)
{
    if (m < 0 || n < 0 || nnz < 0)
        return fail(RTT_ERR_INVALID_ARGUMENT, "csr2tile: negative size");
    cudaStream_t s = ws.stream;
    out.m = m;
    out.n = n;
    out.nnz = nnz;
    out.has_segments = false;
    out.payload = true;
    out.tilem = ceil_div(m, TD);
    out.tilen = ceil_div(n, TD);
    const int tilem = out.tilem;

    RTT_CHECK(out.tile_ptr.ensure(sizeof(int) * (tilem + 1), s));
    RTT_CHECK(out.tmp0.ensure(sizeof(int) * (tilem + 1), s));
    // [0..2] flags of the rows, [3] heavy tile rows listed, [4] tiles, [5] the
    // most segments of a row
    RTT_CHECK(out.tmp1.ensure(sizeof(int) * 8, s));
    int *flags = out.tmp1.as<int>(), *unmade = ws.err.as<int>() + 1 + out.operand;
    RTT_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * 6, s));
    if (m == 0)
    {
        RTT_CUDA(cudaMemsetAsync(out.tile_ptr.p, 0, sizeof(int), s));
        out.numtile = 0;
        RTT_CHECK(out.tile_nnz.ensure(sizeof(int), s));
        RTT_CUDA(cudaMemsetAsync(out.tile_nnz.p, 0, sizeof(int), s));
        const size_t tiny = 16;
        RTT_CHECK(out.tile_col.ensure(tiny, s));
        RTT_CHECK(out.tile_row.ensure(tiny, s));
        RTT_CHECK(out.ptr.ensure(tiny, s));
        RTT_CHECK(out.mask.ensure(tiny, s));
        RTT_CHECK(out.col.ensure(tiny, s));
        RTT_CHECK(out.val.ensure(tiny, s));
        return RTT_OK;
    }
    const CsChunks ch(nnz);
    const bool want_segs = segments || !payload;
    if (want_segs)
    {
        RTT_CHECK(out.seg_cnt.ensure(sizeof(int) * ((size_t)ch.ctas * (CS_WARPS + 1) + 1), s));
        RTT_CHECK(out.seg_ptr.ensure(sizeof(int) * ((size_t)m + 1), s));
        RTT_CHECK(out.seg_word.ensure(sizeof(uint2) * ((size_t)nnz / 32 + 1), s));
        // at most one segment per entry: sized by nnz, no host read
        RTT_CHECK(out.seg.ensure(sizeof(unsigned long long) * ((size_t)nnz + 1), s));
    }
    if (!payload)
    {
        RTT_CHECK(out.tile_end.ensure(sizeof(int) * (size_t)tilem + 16, s));
        // a tile per segment at most: sized by nnz, no host read
        RTT_CHECK(out.tile_col.ensure(sizeof(int) * (size_t)nnz + 16, s));
    }
    // segments starting in each CTA's and each warp's entries
    int *cta_cnt = want_segs ? out.seg_cnt.as<int>() : nullptr;
    int *warp_cnt = want_segs ? cta_cnt + ch.ctas : nullptr;
    k_csr_scan<<<ch.grid(m), CS_THREADS, 0, s>>>(m, n, nnz, rowptr, col, ch.ctas, ch.blocks,
                                                 cta_cnt, warp_cnt, ws.err.as<int>(), flags,
                                                 want_segs ? unmade : nullptr);
    ws.launches++;
    // the segments and the tile index are made before the host sees the flags,
    // so that one synchronisation brings flags, errors and sizes
    if (want_segs)
    {
        if (nnz > 0)
        {
            k_csr_segments<<<ch.ctas, CS_THREADS, 0, s>>>(
                m, nnz, rowptr, col, ch.blocks, cta_cnt, warp_cnt, out.seg_word.as<uint2>(),
                out.seg.as<unsigned long long>(), unmade);
            ws.launches++;
        }
        else
            RTT_CUDA(cudaMemsetAsync(out.seg_word.p, 0, sizeof(uint2), s));
        if (payload)
        {
            k_seg_rows<<<grid_for((long long)m + 1, 256), 256, 0, s>>>(
                m, rowptr, out.seg_word.as<uint2>(), out.seg_ptr.as<int>(), unmade);
            ws.launches++;
        }
    }
    if (!payload)
    {
        const int sms = ws.sms;
        k_seg_tiles<<<std::min(ceil_div(tilem, ST_WARPS), ST_CTAS * sms), ST_WARPS * 32, 0, s>>>(
            m, tilem, rowptr, out.seg_word.as<uint2>(), out.seg_ptr.as<int>(),
            out.seg.as<unsigned long long>(),
            out.tile_ptr.as<int>(), out.tile_end.as<int>(), out.tile_col.as<int>(), flags + 4,
            unmade);
        ws.launches++;
    }
    if (defer && !payload)
    {
        // until csr2tile_settle
        const int none[CSR_WORDS] = {};
        csr2tile_settle(out, none);
        return RTT_OK;
    }
    Publish pub;
    pub.add(flags, ws.h_scalars + 2, CSR_WORDS);
    publish_error(ws, pub);
    RTT_CHECK(publish(ws, pub));
    RTT_CHECK(wait_published(ws, "csr2tile validate"));
    if (!payload && csr2tile_settle(out, ws.h_scalars + 2))
        return RTT_OK;
    const bool unsorted = ws.h_scalars[3] != 0;
    // rows that are unsorted may hide repeated columns too
    out.dup_cols = ws.h_scalars[4] != 0 || unsorted;
    out.generic = ws.h_scalars[2] != 0;
    out.has_segments = want_segs && !out.generic;
    out.max_row_segs = 0;
    if (want_segs && out.generic)
        RTT_CUDA(cudaMemsetAsync(unmade, 0, sizeof(int), s));
    return csr2tile_payload(ws, rowptr, col, val, out, packed_col, sort_within_rows && unsorted);
}

int csr2tile_payload(Workspace &ws, const int *rowptr, const int *col, const double *val,
                     TileBufs &out, bool packed_col, bool sort_rows)
{
    cudaStream_t s = ws.stream;
    const int m = out.m, nnz = out.nnz, tilem = out.tilem;
    const bool generic = out.generic;
    out.payload = true;
    int *cnt = out.tmp0.as<int>();
    // heavy tile rows (a CTA each) are listed on the device; their kernels
    // take the list length from device memory, so no host read is needed
    uint8_t *heavy = nullptr;
    int *hv_list = nullptr, *hv_count = out.tmp1.as<int>() + 3;
    int hv_grid = 0;
    const size_t hv_smem = sizeof(HeavySmem);
    if (!generic)
    {
        RTT_CHECK(out.tmp2.ensure((size_t)tilem + 16, s));
        RTT_CHECK(out.tmp3.ensure(sizeof(int) * (size_t)tilem + 16, s));
        heavy = out.tmp2.as<uint8_t>();
        hv_list = out.tmp3.as<int>();
        RTT_CUDA(cudaMemsetAsync(hv_count, 0, sizeof(int), s));
        k_c2t_heavy_mark<<<grid_for(tilem, 256), 256, 0, s>>>(m, tilem, rowptr, col, heavy,
                                                              hv_list, hv_count);
        ws.launches++;
        const int sms = ws.sms;
        hv_grid = std::min(tilem, 2 * sms);
        RTT_CUDA(cudaFuncSetAttribute(k_c2t_heavy_count, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)hv_smem));
        RTT_CUDA(cudaFuncSetAttribute(k_c2t_heavy_fill, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)hv_smem));
        k_c2t_heavy_count<<<hv_grid, HV_THREADS, hv_smem, s>>>(m, hv_list, hv_count, rowptr, col,
                                                               cnt);
        ws.launches++;
    }
    if (!generic)
        k_c2t_count<<<grid_for((long long)ceil_div(tilem, 2) * 32, 256), 256, 0, s>>>(m, tilem, rowptr,
                                                                                   col, cnt, heavy);
    else
        k_c2t_count_generic<<<grid_for((long long)tilem * 32, 256), 256, 0, s>>>(m, tilem, rowptr,
                                                                               col, cnt);
    ws.launches++;
    RTT_CHECK(scan_exclusive_int(ws, cnt, out.tile_ptr.as<int>(), tilem));
    int numtile = 0;
    RTT_CHECK(read_int(ws, out.tile_ptr.as<int>() + tilem, &numtile));
    out.numtile = numtile;

    RTT_CHECK(out.tile_col.ensure(sizeof(int) * (size_t)numtile, s));
    RTT_CHECK(out.tile_row.ensure(sizeof(int) * (size_t)numtile, s));
    RTT_CHECK(out.tile_nnz.ensure(sizeof(int) * ((size_t)numtile + 1), s));
    RTT_CHECK(out.ptr.ensure((size_t)numtile * TD, s));
    RTT_CHECK(out.mask.ensure(sizeof(uint16_t) * (size_t)numtile * TD, s));
    RTT_CHECK(out.col.ensure((size_t)nnz, s));
    RTT_CHECK(out.val.ensure(sizeof(double) * (size_t)nnz, s));

    if (!generic)
        k_c2t_fill<<<grid_for((long long)ceil_div(tilem, 2) * 32, 256), 256, 0, s>>>(
            m, tilem, rowptr, col, val, out.tile_ptr.as<int>(), out.tile_col.as<int>(),
            out.tile_row.as<int>(), out.tile_nnz.as<int>(), out.ptr.as<uint8_t>(),
            out.col.as<uint8_t>(), out.val.as<double>(), out.mask.as<uint16_t>(), packed_col ? 1 : 0,
            ws.err.as<int>(), heavy);
    else
        k_c2t_fill_generic<<<grid_for((long long)tilem * 32, 128), 128, 0, s>>>(
            m, tilem, rowptr, col, val, out.tile_ptr.as<int>(), out.tile_col.as<int>(),
            out.tile_row.as<int>(), out.tile_nnz.as<int>(), out.ptr.as<uint8_t>(),
            out.col.as<uint8_t>(), out.val.as<double>(), out.mask.as<uint16_t>(), packed_col ? 1 : 0,
            ws.err.as<int>());
    ws.launches++;
    if (!generic)
    {
        k_c2t_heavy_fill<<<hv_grid, HV_THREADS, hv_smem, s>>>(
            m, hv_list, hv_count, rowptr, col, val, out.tile_ptr.as<int>(), out.tile_col.as<int>(),
            out.tile_row.as<int>(), out.tile_nnz.as<int>(), out.ptr.as<uint8_t>(),
            out.col.as<uint8_t>(), out.val.as<double>(), out.mask.as<uint16_t>(),
            packed_col ? 1 : 0, ws.err.as<int>());
        ws.launches++;
    }
    k_set_int<<<1, 1, 0, s>>>(out.tile_nnz.as<int>() + numtile, nnz);
    ws.launches++;
    if (sort_rows && numtile > 0)
    {
        k_sort_tile_rows<<<grid_for((long long)numtile * TD, 256), 256, 0, s>>>(
            numtile, out.tile_nnz.as<int>(), out.ptr.as<uint8_t>(), out.col.as<uint8_t>(),
            out.val.as<double>());
        ws.launches++;
    }
    return RTT_OK;
}

const int *csr2tile_words(const TileBufs &t) { return t.tmp1.as<int>(); }

bool csr2tile_settle(TileBufs &t, const int *words)
{
    t.generic = words[0] != 0;
    // rows that are unsorted may hide repeated columns too
    t.dup_cols = words[2] != 0 || words[1] != 0;
    // the structure alone comes from the row segments, which need rows whose
    // tile columns never decrease; otherwise the whole tile payload is built
    t.has_segments = !t.generic;
    t.payload = t.generic;
    t.numtile = words[4];
    t.max_row_segs = words[5];
    return !t.generic;
}

int csr2tile_refill_device(Workspace &ws, const int *rowptr, const int *col, const double *val,
                           TileBufs &t, bool packed_col)
{
    cudaStream_t s = ws.stream;
    const int m = t.m, tilem = t.tilem;
    if (m == 0 || t.nnz == 0)
        return RTT_OK;
    // the fill kernels of the first build, with the new values: they rewrite
    // the structure arrays with the same bytes and the values in tile order
    if (!t.generic)
    {
        RTT_CHECK(t.tmp1.ensure(sizeof(int) * 8, s));
        RTT_CHECK(t.tmp2.ensure((size_t)tilem + 16, s));
        RTT_CHECK(t.tmp3.ensure(sizeof(int) * (size_t)tilem + 16, s));
        uint8_t *heavy = t.tmp2.as<uint8_t>();
        int *hv_list = t.tmp3.as<int>(), *hv_count = t.tmp1.as<int>() + 3;
        RTT_CUDA(cudaMemsetAsync(hv_count, 0, sizeof(int), s));
        k_c2t_heavy_mark<<<grid_for(tilem, 256), 256, 0, s>>>(m, tilem, rowptr, col, heavy,
                                                              hv_list, hv_count);
        k_c2t_fill<<<grid_for((long long)ceil_div(tilem, 2) * 32, 256), 256, 0, s>>>(
            m, tilem, rowptr, col, val, t.tile_ptr.as<int>(), t.tile_col.as<int>(),
            t.tile_row.as<int>(), t.tile_nnz.as<int>(), t.ptr.as<uint8_t>(), t.col.as<uint8_t>(),
            t.val.as<double>(), t.mask.as<uint16_t>(), packed_col ? 1 : 0, ws.err.as<int>(), heavy);
        const int sms = ws.sms;
        const size_t hv_smem = sizeof(HeavySmem);
        RTT_CUDA(cudaFuncSetAttribute(k_c2t_heavy_fill, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)hv_smem));
        k_c2t_heavy_fill<<<std::min(tilem, 2 * sms), HV_THREADS, hv_smem, s>>>(
            m, hv_list, hv_count, rowptr, col, val, t.tile_ptr.as<int>(), t.tile_col.as<int>(),
            t.tile_row.as<int>(), t.tile_nnz.as<int>(), t.ptr.as<uint8_t>(), t.col.as<uint8_t>(),
            t.val.as<double>(), t.mask.as<uint16_t>(), packed_col ? 1 : 0, ws.err.as<int>());
        ws.launches += 3;
    }
    else
    {
        k_c2t_fill_generic<<<grid_for((long long)tilem * 32, 128), 128, 0, s>>>(
            m, tilem, rowptr, col, val, t.tile_ptr.as<int>(), t.tile_col.as<int>(),
            t.tile_row.as<int>(), t.tile_nnz.as<int>(), t.ptr.as<uint8_t>(), t.col.as<uint8_t>(),
            t.val.as<double>(), t.mask.as<uint16_t>(), packed_col ? 1 : 0, ws.err.as<int>());
        ws.launches++;
    }
    RTT_CUDA(cudaGetLastError());
    return RTT_OK;
}

int validate_csr_device(Workspace &ws, int m, int n, int nnz, const int *rowptr, const int *col,
                        int *flags)
{
    RTT_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * 3, ws.stream));
    if (m > 0)
    {
        const CsChunks ch(nnz);
        k_csr_scan<<<ch.grid(m), CS_THREADS, 0, ws.stream>>>(
            m, n, nnz, rowptr, col, ch.ctas, ch.blocks, nullptr, nullptr, ws.err.as<int>(), flags,
            nullptr);
        ws.launches++;
    }
    Publish pub;
    pub.add(flags, ws.h_scalars + 4, 3);
    publish_error(ws, pub);
    RTT_CHECK(publish(ws, pub));
    return wait_published(ws, "csr validate");
}

int build_tile_csc(Workspace &ws, TileBufs &t)
{
    cudaStream_t s = ws.stream;
    const int nt = t.numtile;
    RTT_CHECK(t.csc_ptr.ensure(sizeof(int) * (t.tilen + 1), s));
    RTT_CHECK(t.csc_row.ensure(sizeof(int) * (size_t)(nt + 1), s));
    RTT_CHECK(t.csc_data.ensure(sizeof(int) * (size_t)(nt + 1), s));
    RTT_CHECK(t.tmp2.ensure(sizeof(int) * (size_t)(nt + 1), s));
    RTT_CHECK(t.tmp3.ensure(sizeof(int) * (size_t)(nt + 1), s));
    int *iota = t.tmp2.as<int>();
    int *sorted_keys = t.tmp3.as<int>();
    if (nt > 0)
    {
        k_iota<<<grid_for(nt, 256), 256, 0, s>>>(iota, nt);
        ws.launches++;
        RTT_CHECK(sort_pairs(ws, t.tile_col.as<int>(), sorted_keys, iota, t.csc_data.as<int>(), nt,
                             t.tilen));
        k_gather_int<<<grid_for(nt, 256), 256, 0, s>>>(t.tile_row.as<int>(), t.csc_data.as<int>(),
                                                       nt, t.csc_row.as<int>());
        ws.launches++;
    }
    k_lower_bound_ptr<<<grid_for(t.tilen + 1, 256), 256, 0, s>>>(sorted_keys, nt, t.tilen,
                                                                 t.csc_ptr.as<int>());
    ws.launches++;
    return RTT_OK;
}

int tiles_to_col_major(Workspace &ws, const TileBufs &rm, TileBufs &out)
{
    // rm must carry its CSC index (build_tile_csc)
    cudaStream_t s = ws.stream;
    const int nt = rm.numtile;
    out.m = rm.m;
    out.n = rm.n;
    out.nnz = rm.nnz;
    out.tilem = rm.tilem;
    out.tilen = rm.tilen;
    out.numtile = nt;
    RTT_CHECK(out.tile_nnz.ensure(sizeof(int) * ((size_t)nt + 1), s));
    RTT_CHECK(out.ptr.ensure((size_t)nt * TD + 16, s));
    RTT_CHECK(out.mask.ensure(sizeof(uint16_t) * (size_t)nt * TD + 16, s));
    RTT_CHECK(out.col.ensure((size_t)rm.nnz + 16, s));
    RTT_CHECK(out.val.ensure(sizeof(double) * (size_t)rm.nnz + 16, s));
    RTT_CHECK(out.tmp0.ensure(sizeof(int) * ((size_t)nt + 1), s));
    int *cnt = out.tmp0.as<int>();
    if (nt > 0)
    {
        k_tile_counts<<<grid_for(nt, 256), 256, 0, s>>>(rm.tile_nnz.as<int>(), rm.csc_data.as<int>(),
                                                         nt, cnt);
        ws.launches++;
    }
    RTT_CHECK(scan_exclusive_int(ws, cnt, out.tile_nnz.as<int>(), nt));
    if (nt > 0)
    {
        k_copy_tiles_colmajor<<<grid_for((long long)nt * 32, 256), 256, 0, s>>>(
            nt, rm.csc_data.as<int>(), rm.tile_nnz.as<int>(), rm.ptr.as<uint8_t>(),
            rm.mask.as<uint16_t>(), rm.col.as<uint8_t>(), rm.val.as<double>(),
            out.tile_nnz.as<int>(), out.ptr.as<uint8_t>(), out.mask.as<uint16_t>(),
            out.col.as<uint8_t>(), out.val.as<double>());
        ws.launches++;
    }
    return RTT_OK;
}

int csr_transpose_device(Workspace &ws, int m, int n, int nnz, const int *rowptr, const int *col,
                         const double *val, int *t_rowptr, int *t_col, double *t_val)
{
    cudaStream_t s = ws.stream;
    // grow-only scratch of the workspace: no cudaMalloc / cudaFree (which
    // would wait for every stream of the device) once it has grown
    const size_t bytes = sizeof(int) * (size_t)nnz + 16;
    for (DevBuf &b : ws.tmp)
        RTT_CHECK(b.ensure(bytes, s));
    int *rows = ws.tmp[0].as<int>(), *iota = ws.tmp[1].as<int>();
    int *keys = ws.tmp[2].as<int>(), *order = ws.tmp[3].as<int>();
    if (m > 0)
    {
        k_row_ids<<<grid_for(m, 256), 256, 0, s>>>(m, rowptr, rows, ws.err.as<int>());
        ws.launches++;
    }
    if (nnz > 0)
    {
        k_iota<<<grid_for(nnz, 256), 256, 0, s>>>(iota, nnz);
        ws.launches++;
        RTT_CHECK(sort_pairs(ws, col, keys, iota, order, nnz, n));
        k_gather_transpose<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, order, rows, val, t_col, t_val);
        ws.launches++;
    }
    k_lower_bound_ptr<<<grid_for(n + 1, 256), 256, 0, s>>>(keys, nnz, n, t_rowptr);
    ws.launches++;
    return RTT_OK;
}

} // namespace rtt
