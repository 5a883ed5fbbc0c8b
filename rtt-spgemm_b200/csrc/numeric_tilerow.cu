// numeric_tilerow.cu - numeric step of C tile rows that fit one window, C
// written as CSR: the stencil case of numeric_flat.cu's kernel.
//
// One CTA per C tile row, 8 warps x 2 scalar rows, warp-private Gustavson as
// there, with what that kernel needs for windows, tile output and repeated
// columns left out:
//   * the tile row's entries are one range of C's CSR, in the accumulator's
//     order, so the values are written out as they lie, each warp its own rows
//     without a CTA barrier, and the columns go to C straight from the masks
//     (once per entry) instead of beside every product;
//   * a product finds its entry by two loads and no branch: lanes without a
//     product repeat the row's last one and drop the sum; two B rows are
//     looked up together, then added in order;
//   * an A entry's list word holds its B row, row and value in 16 bytes.
// Every output is summed by one warp in the order of its row's A entries with
// fma: bitwise numeric_flat.cu's result.
//
// What bounds it: L1 and shared memory (93 % of L1 throughput; 16 shared
// wavefronts per B row of 27 products, 6 of them bank conflicts of the
// accumulator's read-modify-write, and 6 of loads), DRAM 10 %.  64^3 stencil
// 692 -> 575 us, 96^3 2.29 -> 1.95 ms against numeric_flat.cu's kernel (B200).
#include "rtt_internal.cuh"

#include <type_traits>

namespace rtt
{
namespace
{

constexpr int TR_WARPS = 8, TR_THREADS = TR_WARPS * 32;
// B rows looked up together, and CTAs per SM: 2 and 5 measured best on the 96^3
// stencil (whole product 3.42 ms; 2 and 6: 3.48, 4 and 5: 3.51, 4 and 4: 3.52).
constexpr int TR_UNROLL = 2, TR_CTAS = 5;
constexpr int TR_STRIDE = FLAT_SLOT_CAP + 1; // rows of cm in distinct banks
constexpr int TR_SPAN = 4096;               // tile columns of the slot table

// Place of tile column d in the slot table: its bank moves with the higher bits
// of d, since the lines and planes of a grid lie at strides that share banks.
__device__ __forceinline__ int slot_at(int d)
{
    return (d ^ ((d >> 5) & 0x7C)) & (TR_SPAN - 1);
}

struct TileRowSmem
{
    double acc[FLAT_ACC];
    int4 ent[TR_WARPS][32];      // B row's start; length | row << 16; a_ik
    uint32_t cm[TD * TR_STRIDE]; // [row][slot]: row mask << 16 | first entry
    int cJ[FLAT_SLOT_CAP];
    uint8_t slot8[TR_SPAN];      // tile column - first tile column -> slot
    int rowtot[TD];
};

__global__ void __launch_bounds__(TR_THREADS, TR_CTAS)
    k_numeric_tilerow(DevTiles A, DevTiles B, int tilem, long long nnzC,
                      const int *__restrict__ c_tile_ptr, const int *__restrict__ c_tile_col,
                      const uint16_t *__restrict__ c_mask, const int *__restrict__ csr_rowptr,
                      int *__restrict__ csr_col, double *__restrict__ csr_val,
                      long long *counters, int *err)
{
    extern __shared__ __align__(16) unsigned char tr_raw[];
    TileRowSmem &S = *reinterpret_cast<TileRowSmem *>(tr_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int I = blockIdx.x;
    const int cs0 = __ldg(c_tile_ptr + I), nW = __ldg(c_tile_ptr + I + 1) - cs0;
    if (nW == 0)
        return;
    const int nrows = min(TD, A.m - I * TD);
    const int dst = __ldg(csr_rowptr + I * TD);
    const int total = __ldg(csr_rowptr + I * TD + nrows) - dst;
    if (nW > FLAT_SLOT_CAP || total > FLAT_ACC || dst < 0 || (long long)dst + total > nnzC)
    {
        if (tid == 0)
            set_error(err, DERR_NUM_BOUNDS); // the caller's rows fit one window
        return;
    }
    // two rows' masks per 32-bit word (c_mask rows are 32-byte aligned per tile)
    const uint32_t *src = reinterpret_cast<const uint32_t *>(c_mask + (size_t)cs0 * TD);
    for (int i = tid; i < nW * (TD / 2); i += TR_THREADS)
    {
        const int s = i >> 3, r = (i & 7) * 2;
        const uint32_t v = __ldg(src + i);
        S.cm[r * TR_STRIDE + s] = v << 16;
        S.cm[(r + 1) * TR_STRIDE + s] = v & 0xFFFF0000u;
    }
    const int Jlo = __ldg(c_tile_col + cs0);
    const int Jspan = __ldg(c_tile_col + cs0 + nW - 1) - Jlo;
    const bool table = Jspan < TR_SPAN;
    for (int i = tid; i < nW; i += TR_THREADS)
    {
        const int J = __ldg(c_tile_col + cs0 + i);
        S.cJ[i] = J;
        // (a product's tile column is in the table: the others are not read)
        if (table)
            S.slot8[slot_at(J - Jlo)] = (uint8_t)i;
    }
    for (int i = tid; i < (total + 1) / 2; i += TR_THREADS)
        reinterpret_cast<double2 *>(S.acc)[i] = make_double2(0.0, 0.0);
    __syncthreads();
    {
        // first entry of (row r, slot s): the entries of rows < r plus those
        // of row r in slots < s.  Thread (r = tid / 16, part = tid % 16) owns
        // a run of slots; its entries' columns go to C.
        static_assert(TR_THREADS == TD * 16, "one half-warp per row");
        const int r = tid >> 4, part = tid & 15;
        const int per = (nW + 15) >> 4;
        const int s0 = min(part * per, nW), s1 = min(s0 + per, nW);
        uint32_t *cmr = S.cm + r * TR_STRIDE;
        int sum = 0;
        for (int s = s0; s < s1; ++s)
            sum += __popc(cmr[s]);
        const int incl = half_incl_scan(sum);
        if (part == 15)
            S.rowtot[r] = incl;
        __syncthreads();
        // entries of the rows before (a half-warp scan, every half its own)
        const int t = S.rowtot[part];
        const int tincl = half_incl_scan(t);
        int run = __shfl_sync(FULL, tincl - t, (lane & 16) | r) + incl - sum;
        for (int s = s0; s < s1; ++s)
        {
            const uint32_t w = cmr[s];
            cmr[s] = w | (uint32_t)run;
            run += __popc(w);
        }
    }
    __syncthreads();
    // C's columns, once per entry: neighbouring threads take neighbouring
    // tiles of a row, whose entries follow each other
    for (int i = tid; i < nW * TD; i += TR_THREADS)
    {
        const int r = i / nW, s = i - r * nW;
        const uint32_t w = S.cm[r * TR_STRIDE + s];
        int p = (int)(w & 0xFFFFu);
        const int c0 = S.cJ[s] * TD;
        for (uint32_t mk = w & 0xFFFF0000u; mk != 0u && p < total; ++p)
        {
            const int c = __clz(mk);
            mk &= ~(0x80000000u >> c);
            csr_col[(size_t)dst + p] = c0 + c;
        }
    }
    // ---- products: warp-private
    const int r0 = warp * 2;
    if (r0 >= nrows)
        return;
    const int *rp = A.csr_rowptr + (size_t)I * TD;
    const int e_a = __ldg(rp + r0), e_m = __ldg(rp + min(r0 + 1, nrows)),
              e_e = __ldg(rp + min(r0 + 2, nrows));
    int4 *ent = S.ent[warp];
    long long n_fma = 0;
    auto walk = [&](auto with_table) {
        constexpr bool TABLE = decltype(with_table)::value;
        const uint32_t *cm0 = S.cm + r0 * TR_STRIDE;
        // list items [0, n), in order
        auto items = [&](int n) {
            for (int j = 0; j < n; j += TR_UNROLL)
            {
                int4 g[TR_UNROLL];
                int c[TR_UNROLL], pos[TR_UNROLL];
                double b[TR_UNROLL];
                bool ok[TR_UNROLL];
#pragma unroll
                for (int u = 0; u < TR_UNROLL; ++u)
                {
                    g[u] = ent[(j + u) & 31];
                    const int len = g[u].y & 0xFFFF;
                    ok[u] = j + u < n && lane < len;
                    // (a lane without a product takes the last one's place:
                    // the same addresses, so no bank conflict of its own)
                    c[u] = 0;
                    b[u] = 0.0;
                    if (j + u < n && len > 0)
                    {
                        const int f = g[u].x + min(lane, len - 1);
                        c[u] = __ldg(B.csr_col + f);
                        b[u] = __ldg(B.csr_val + f);
                    }
                }
#pragma unroll
                for (int u = 0; u < TR_UNROLL; ++u)
                {
                    // (the masks on the indexes keep inconsistent operands
                    // inside this CTA's shared memory)
                    const int slot = TABLE ? (int)S.slot8[slot_at((c[u] >> 4) - Jlo)]
                                           : lower_bound(S.cJ, 0, nW, c[u] >> 4);
                    const uint32_t w = cm0[(g[u].y >= 0x10000 ? TR_STRIDE : 0) +
                                           (slot & (FLAT_SLOT_CAP - 1))];
                    pos[u] = (int)((w & 0xFFFFu) +
                                   __popc(__funnelshift_rc(w, 0u, 32 - (c[u] & 15)))) &
                             (FLAT_ACC - 1);
                }
#pragma unroll
                for (int u = 0; u < TR_UNROLL; ++u)
                {
                    const double sum =
                        fma(__hiloint2double(g[u].w, g[u].z), b[u], S.acc[pos[u]]);
                    if (ok[u])
                        S.acc[pos[u]] = sum;
                    __syncwarp();
                }
            }
        };
        for (int q0 = e_a; q0 < e_e; q0 += 32)
        {
            const int e = q0 + lane;
            int fs = 0, len = 0;
            double a = 0.0;
            if (e < e_e)
            {
                const int k = __ldg(A.csr_col + e);
                a = __ldg(A.csr_val + e);
                if ((unsigned)k < (unsigned)B.m)
                {
                    fs = min(max(__ldg(B.csr_rowptr + k), 0), B.nnz);
                    len = min(max(__ldg(B.csr_rowptr + k + 1), fs), B.nnz) - fs;
                }
                n_fma += len;
            }
            const int row = e < e_m ? 0 : 0x10000;
            if (!__any_sync(FULL, len > 32))
            {
                ent[lane] = make_int4(fs, len | row, __double2loint(a), __double2hiint(a));
                __syncwarp();
                items(min(32, e_e - q0));
                continue;
            }
            // B rows longer than a warp: an item per 32 of their entries
            const int nch = (len + 31) >> 5;
            const int cincl = warp_incl_scan(nch);
            const int ctotal = __shfl_sync(FULL, cincl, 31);
            for (int i0 = 0; i0 < ctotal; i0 += 32)
            {
                const int qi = i0 + lane;
                int own = 0;
#pragma unroll
                for (int h = 16; h > 0; h >>= 1)
                    if (__shfl_sync(FULL, cincl, own + h - 1) <= qi)
                        own += h;
                own = min(own, 31);
                const int k = qi - __shfl_sync(FULL, cincl - nch, own);
                const int ofs = __shfl_sync(FULL, fs, own), olen = __shfl_sync(FULL, len, own);
                const int orow = __shfl_sync(FULL, row, own);
                const double oa = __shfl_sync(FULL, a, own);
                __syncwarp(); // the previous items are done
                ent[lane] = make_int4(ofs + 32 * k, (qi < ctotal ? min(32, olen - 32 * k) : 0) | orow,
                                      __double2loint(oa), __double2hiint(oa));
                __syncwarp();
                items(min(32, ctotal - i0));
            }
        }
    };
    if (table)
        walk(std::true_type());
    else
        walk(std::false_type());
    // ---- values: the warp's rows lie together in the accumulator and in C
    const int b0 = __ldg(csr_rowptr + I * TD + r0) - dst;
    const int b1 = __ldg(csr_rowptr + I * TD + min(r0 + 2, nrows)) - dst;
    for (int p = max(b0, 0) + lane; p < min(b1, total); p += 32)
        csr_val[(size_t)dst + p] = S.acc[p];
    n_fma = warp_sum(n_fma);
    if (counters != nullptr && lane == 0 && n_fma)
        atomicAdd((unsigned long long *)&counters[1], (unsigned long long)n_fma);
}

} // namespace

int numeric_tilerow_device(Workspace &ws, const DevTiles &A, const DevTiles &B, SymbolicOut &S,
                           const NumericConfig &cfg)
{
    const size_t smem = sizeof(TileRowSmem);
    RTT_CUDA(cudaFuncSetAttribute(k_numeric_tilerow, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    k_numeric_tilerow<<<S.tilem, TR_THREADS, smem, ws.stream>>>(
        A, B, S.tilem, S.nnz, S.c_tile_ptr.as<int>(), S.c_tile_col.as<int>(),
        S.c_mask.as<uint16_t>(), cfg.csr_rowptr, cfg.csr_col, cfg.csr_val, cfg.counters,
        ws.err.as<int>());
    ws.launches++;
    return RTT_OK;
}

} // namespace rtt
