// Batched tiled SpGEMM: many independent products C_p = A_p * B_p of uneven
// size in ONE persistent, cooperatively launched kernel (and, for the SPA
// schedule, step 3's kernels after it), captured once in a CUDA graph and
// replayed by tsg_batch_run.
//
// The kernel runs its phases separated by a grid barrier; in each phase the
// work of all products is one flattened index space (product found by binary
// search over a prefix array), so small products do not leave the GPU idle:
//   1 step-1 counts: tile rows of products with many tile pairs a CTA each, the
//     others' a warp each                  2 per-product scan of them
//   3 item prefix over products (block 0)  4 step-1 emit, fused with step 2 for
//     narrow rows unless the row schedule runs its own
//   5 step 2 of the rest: units of wide rows, a CTA each (SPA), or a half-warp
//     per item                             6 per-product scan of tile nnz
//   7 step 3, a half-warp or warp per item; the SPA schedule leaves it to up to
//     six kernels: k_batch_wtab and k_batch_win (windows), k_batch_hyper and
//     k_batch_spa3 (the other sparse C tiles) and k_batch_dense3 in one or both of
//     its forms (dense C tiles), side by side on the context's streams
// An item is one C tile (tile and element schedules) or seg_tiles C tiles (row
// schedule); the per-item code is tsg_device.cuh's, identical to the one-product
// path.
//
// Memory: one arena per batch, sized at creation from per-product upper
// bounds computed on the device (C tiles <= matched tile pairs, C nonzeros <=
// scalar products), so a run needs no host round trip.  The grid barrier is
// bounded in time (%globaltimer): a wait longer than the batch's limit --
// BATCH_WAIT_FLOOR_NS plus BATCH_WAIT_NS_PER_PRODUCT per scalar product of
// the whole batch, or tsg_batch_set_wait_limit's -- sets TSG_ERR_TIMEOUT in
// the error word that tsg_batch_sync reports, and every block leaves.
#include <cooperative_groups.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "tsg_device.cuh"
#include "tsg_wide.cuh"
#include "tsg_window.cuh"

int tsg_count_c_tiles_async(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, unsigned long long *total);

struct BatchProd
{
    ProdView P;
    StepOneBits K; // step 1's bitmaps, kept in C's value range until step 3
    int *wide;     // per A tile row: 1 when step 2 runs apart (fused pass declined), 2 hypersparse
    WinPlan Q;     // step 3 by windows (win)
    int win;
    long long capT, capN;
    int tilemA;
    int hypT;   // C tiles of hypersparse rows
    int status; // 0 ok, 1 tile capacity, 2 value capacity
    int numC, nnzC;
};

struct tsg_batch
{
    tsg_context *ctx;
    int count;
    tsg_batch_params params;
    std::vector<BatchProd> host;    // descriptors (host copy)
    std::vector<long long> rowoff;  // prefix of tilemA over products
    BatchProd *d_prod;
    long long *d_rowoff;
    long long *d_itemoff;
    unsigned *d_bar; // [0] arrivals, [1] generation, [2] next tile block of the SPA step 3, [3] next
                     // wide unit of step 2, [4..5] the barrier's wait limit in ns (64-bit), [6] wide
                     // units, [7] parts of heavy rows, [8] next claim of the window step 3, [9] next
                     // unit of the hypersparse step 3
    int *d_err;
    int *d_bins;
    void *arena;
    size_t arena_bytes;
    int grid, block;
    size_t smem;
    int grid3, gridh; // persistent grids of k_batch_spa3 and k_batch_hyper (SPA schedule)
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    int graph_ok;
    std::vector<int> m, n, tilen; // per product C dimensions
    long long launches;
    unsigned long long wait_ns; // the grid barrier's wait limit
    unsigned bar_init[16];       // host image of d_bar at creation (zeros, the wait limit at [4])
    std::vector<long long> s1off;  // prefix of tilemA over the products whose step 1 takes a CTA per tile row, then the others'
    std::vector<long long> winoff; // window step 3: prefixes of rows of B, ctab entries, rows of A, claims
    long long *d_s1off, *d_winoff;
    int4 *d_wlist, *d_hlist; // wide units of step 2; heavy rows' parts of the window step 3
    int *win_tables;
    long long *d_denseoff;      // C tiles of the products with dense tiles, prefixes (rows form, columns form)
    int rows_form, cols_form;   // products of either form of the tile kernel
    int split;   // A entries of a unit of step 2's wide rows
    int wins;    // products that take the windows
    int gridw;   // persistent grid of k_batch_win
    int dense;                  // SPA schedule: values per C tile from which a product takes the tile kernel
};

#define BATCH_THREADS 128
#define BATCH_SPAN 3072 // tile columns of step 2's wide rows in a CTA's shared memory (two CTAs an SM)
// step 3 by windows: products with this many scalar products per (row, window)
// (win_worth says the rest; 4 products of 4,096 random rows, step 3 by
// k_batch_spa3 and by windows, with 8 products a (row, window) 0.066 and 0.086 ms,
// with 16 0.110 and 0.096), whose tables and lists together take up to this many
// words each and in all
#define BATCH_WIN_MIN 16
#define BATCH_WIN_WORDS (1LL << 23)
#define BATCH_WIN_TOTAL (1LL << 26)
// a barrier wait gives up after this floor plus a share of the batch's work
// (a B200 does well over 10 scalar products per ns, so the bound is loose)
#define BATCH_WAIT_FLOOR_NS 2000000000ULL
#define BATCH_WAIT_NS_PER_PRODUCT 10ULL

__device__ __forceinline__ unsigned long long batch_clock_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------
// bounded grid barrier (all blocks co-resident: cooperative launch)
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *err)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        volatile unsigned *vgen = bar + 1;
        const unsigned gen = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(bar, 1u) + 1u;
        if (arrived == gridDim.x)
        {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        }
        else
        {
            const unsigned long long limit = *(volatile unsigned long long *)(bar + 4);
            const unsigned long long t0 = batch_clock_ns();
            while (*vgen == gen)
            {
                if (*(volatile int *)err || batch_clock_ns() - t0 > limit)
                {
                    atomicCAS(err, 0, TSG_ERR_TIMEOUT);
                    break;
                }
                __nanosleep(100);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *(volatile int *)err == 0;
}

__device__ __forceinline__ int find_product(const long long *__restrict__ off, int count, long long x)
{
    int lo = 0, hi = count - 1; // largest p with off[p] <= x
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// The same for x at or after off[p] (a CTA's claims from a counter only grow):
// usually x is still in product p.
__device__ __forceinline__ int find_product_from(const long long *__restrict__ off, int count, long long x, int p)
{
    return off[p + 1] > x ? p : find_product(off, count, x);
}

// Block-wide exclusive scan of a[0..n) in place, a[n] = total (NT threads;
// s_tmp holds NT / 32 partial sums).
template <int NT>
__device__ long long block_scan_inplace(int *a, int n, long long *s_tmp)
{
    long long run = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < n; base += NT)
    {
        const int i = base + threadIdx.x;
        const long long v = i < n ? a[i] : 0;
        long long incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const long long o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
            if (lane >= d)
                incl += o;
        }
        if (lane == 31)
            s_tmp[warp] = incl;
        __syncthreads();
        long long woff = 0;
        for (int w = 0; w < warp; w++)
            woff += s_tmp[w];
        long long tot = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++)
            tot += s_tmp[w];
        if (i < n)
            a[i] = (int)(run + woff + incl - v);
        run += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        a[n] = (int)run;
    __syncthreads();
    return run;
}

// Block-wide sum of a[0..n) (NT threads).
template <int NT>
__device__ long long block_sum(const int *a, int n, long long *s_tmp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long v = 0;
    for (int i = threadIdx.x; i < n; i += NT)
        v += a[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        v += __shfl_xor_sync(TSG_FULL_MASK, v, d);
    if (lane == 0)
        s_tmp[warp] = v;
    __syncthreads();
    long long tot = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++)
        tot += s_tmp[w];
    __syncthreads();
    return tot;
}

// Block-wide exclusive scan of a[0..n) in place, offset by off (NT threads).
template <int NT>
__device__ void block_scan_offset(int *a, int n, long long off, long long *s_tmp)
{
    long long run = off;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < n; base += NT)
    {
        const int i = base + threadIdx.x;
        const long long v = i < n ? a[i] : 0;
        long long incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const long long o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
            if (lane >= d)
                incl += o;
        }
        if (lane == 31)
            s_tmp[warp] = incl;
        __syncthreads();
        long long woff = 0, tot = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++)
        {
            woff += w < warp ? s_tmp[w] : 0;
            tot += s_tmp[w];
        }
        if (i < n)
            a[i] = (int)(run + woff + incl - v);
        run += tot;
        __syncthreads();
    }
}

// Exclusive scan of v[0..n) in place (long long) by one block; returns the total.
template <int NT>
__device__ long long block_scan_ll(long long *v, int n, long long *s_tmp)
{
    long long run = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < n; base += NT)
    {
        const int i = base + threadIdx.x;
        const long long x = i < n ? v[i] : 0;
        long long incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const long long o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
            if (lane >= d)
                incl += o;
        }
        if (lane == 31)
            s_tmp[warp] = incl;
        __syncthreads();
        long long woff = 0, tot = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++)
        {
            woff += w < warp ? s_tmp[w] : 0;
            tot += s_tmp[w];
        }
        if (i < n)
            v[i] = run + woff + incl - x;
        run += tot;
        __syncthreads();
    }
    return run;
}

#define SCAN_CHUNK 4096 // C tiles per chunk of the tile-count scan

// GPU global timer (ns); block 0 stamps the end of each phase into
// stamp[1..6] and every block raises stamp[7] as it leaves.
__device__ __forceinline__ unsigned long long gtimer() { return batch_clock_ns(); }

#define BATCH_STAMP(k)                                                  \
    if (blockIdx.x == 0 && threadIdx.x == 0)                           \
        stamp[k] = gtimer();

template <int SCHED, int W, int CAP, int NT>
__global__ void __launch_bounds__(NT)
    k_batch(BatchProd *prods, int count, const long long *__restrict__ rowoff, const long long *__restrict__ s1off,
            int4 *wlist, int split, int per_pair, long long *denseoff, int dense, long long *itemoff, unsigned *bar, int *err, int *bins)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ long long s_tmp[NT / 32 + 1];
    __shared__ int s_row;
    __shared__ int s_bins[4];
    const int lane32 = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 15, hw = threadIdx.x >> 4;
    const unsigned hmask = TSG_HW_MASK(threadIdx.x);
    const long long nwarps = (long long)gridDim.x * (NT / 32);
    const long long nhw = (long long)gridDim.x * (NT / 16);
    const long long total_rows = rowoff[count];
    unsigned long long *stamp = reinterpret_cast<unsigned long long *>(itemoff + 2 * ((long long)count + 1));
    BATCH_STAMP(0)

    // phase 1: step-1 counts; the tile rows of products with many tile pairs
    // (prefix s1off) a CTA each, the others' (prefix after it) a warp each
    {
        S1cSmem<NT> &S1 = *reinterpret_cast<S1cSmem<NT> *>(s_raw);
        for (long long u = blockIdx.x; u < s1off[count]; u += gridDim.x)
        {
            const int p = find_product(s1off, count, u);
            const int i = (int)(u - s1off[p]);
            const int cnt = step1_row_cta<NT>(prods[p].P, i, S1, prods[p].K, nullptr);
            if (threadIdx.x == 0)
                prods[p].P.C_ptr[i] = cnt;
            __syncthreads();
        }
        const long long *woff = s1off + count + 1;
        unsigned *bm = reinterpret_cast<unsigned *>(s_raw) + warp * S1_WORDS;
        for (long long w = (long long)blockIdx.x * (NT / 32) + warp; w < woff[count]; w += nwarps)
        {
            const int p = find_product(woff, count, w);
            const ProdView &P = prods[p].P;
            const int i = (int)(w - woff[p]);
            const int cnt = step1_row<false>(P, i, bm, lane32, nullptr, prods[p].K);
            if (lane32 == 0)
                P.C_ptr[i] = cnt;
        }
    }
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(1)
    // phase 2: per-product scan of C tile counts
    for (int p = blockIdx.x; p < count; p += gridDim.x)
    {
        BatchProd &bp = prods[p];
        const long long tot = block_scan_inplace<NT>(bp.P.C_ptr, bp.tilemA, s_tmp);
        if (threadIdx.x == 0)
        {
            if (tot > bp.capT)
            {
                bp.status = 1;
                bp.numC = 0;
            }
            else
            {
                bp.status = 0;
                bp.numC = (int)tot;
            }
            bp.P.numC = bp.numC;
            bp.hypT = 0;
        }
    }
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(2)
    // phase 3: item prefix over products (block 0)
    if (blockIdx.x == 0)
    {
        if (threadIdx.x == 0)
        {
            long long run = 0;
            for (int p = 0; p < count; p++)
            {
                itemoff[p] = run;
                const long long nc = prods[p].numC;
                run += SCHED == 1 ? (nc + W - 1) / W : nc;
            }
            itemoff[count] = run;
            // SPA: blocks of SPA_BLK C tiles per product, prefix after itemoff
            long long *blkoff = itemoff + count + 1;
            run = 0;
            for (int p = 0; p < count; p++)
            {
                blkoff[p] = run;
                run += ((long long)prods[p].numC + SPA_BLK - 1) / SPA_BLK;
            }
            blkoff[count] = run;
            // tile-count scan chunks per product, prefix after the stamps
            long long *chunkoff = itemoff + 2 * ((long long)count + 1) + 8;
            run = 0;
            for (int p = 0; p < count; p++)
            {
                chunkoff[p] = run;
                run += ((long long)prods[p].numC + SCAN_CHUNK - 1) / SCAN_CHUNK;
            }
            chunkoff[count] = run;
            bar[2] = bar[3] = bar[6] = bar[7] = bar[8] = bar[9] = 0;
        }
        if (threadIdx.x < 4)
            bins[threadIdx.x] = 0;
    }
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(3)
    // phase 4: step-1 emit (fused with step 2 for narrow rows unless the
    // row schedule runs its own step 2)
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    __syncthreads();
    {
        unsigned *bm = reinterpret_cast<unsigned *>(s_raw) + warp * S1_WORDS;
        S12Smem *s12 = reinterpret_cast<S12Smem *>(s_raw) + warp;
        for (long long w = (long long)blockIdx.x * (NT / 32) + warp; w < total_rows; w += nwarps)
        {
            const int p = find_product(rowoff, count, w);
            if (prods[p].status)
                continue;
            const int i = (int)(w - rowoff[p]);
            if (SCHED == 1)
                step1_row<true>(prods[p].P, i, bm, lane32, nullptr);
            else
            {
                const int done = step12_row(prods[p].P, i, *s12, lane32, s_bins, SCHED == 3 ? per_pair : 0, prods[p].K);
                int kind = 0;
                if (!done)
                {
                    __syncwarp();
                    if (!step1_emit_kept(prods[p].P, i, lane32, prods[p].K))
                        step1_row<true>(prods[p].P, i, reinterpret_cast<unsigned *>(s12), lane32, nullptr);
                    __syncwarp(); // the row's C columns, emitted by all lanes
                    kind = SCHED == 3 ? wide_kind(prods[p].P, i, lane32) : 1;
                }
                if (lane32 == 0)
                {
                    prods[p].wide[i] = kind;
                    if (SCHED == 3 && kind)
                    {
                        const int parts = wide_parts(prods[p].P, i, split);
                        int4 *at = wlist + atomicAdd(&bar[6], (unsigned)parts);
                        for (int q = 0; q < parts; q++)
                            at[q] = make_int4(p, i, q | parts << 16, 0);
                        if (kind == 2)
                            atomicAdd(&prods[p].hypT, prods[p].P.C_ptr[i + 1] - prods[p].P.C_ptr[i]);
                    }
                }
                __syncwarp();
            }
        }
    }
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(4)
    // phase 5: step 2 (all tiles for the row schedule, tiles of wide rows otherwise)
    if (SCHED == 3)
    {
        // wide rows through B's row view; CTAs take units of the list
        WideSmem<NT> &S2 = *reinterpret_cast<WideSmem<NT> *>(s_raw);
        for (;;)
        {
            if (threadIdx.x == 0)
                s_row = (int)atomicAdd(&bar[3], 1u);
            __syncthreads();
            const int u = s_row;
            if (u >= (int)*(volatile unsigned *)&bar[6])
                break;
            const int4 w = __ldcg(wlist + u);
            step2_wide_row<NT, false>(prods[w.x].P, S2, BATCH_SPAN, w.y, w.z, s_bins);
        }
    }
    else
    {
        const long long total_items = itemoff[count];
        for (long long h = (long long)blockIdx.x * (NT / 16) + hw; h < total_items; h += nhw)
        {
            const int p = find_product(itemoff, count, h);
            const ProdView &P = prods[p].P;
            const long long item = h - itemoff[p];
            if (SCHED == 1)
                step2_rows_item<W>(P, item, hmask, lane, reinterpret_cast<S2RowsSmem<W> *>(s_raw)[hw], s_bins);
            else if (prods[p].wide[P.C_row[item]])
                step2_tile(P, (int)item, hmask, lane, s_bins);
        }
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(5)
    // phase 6: per-product exclusive scan of the tile counts, in chunks of
    // SCAN_CHUNK tiles spread over all blocks: chunk sums, a scan of each
    // product's chunk sums, then every chunk scanned with its offset
    {
        const long long *chunkoff = itemoff + 2 * ((long long)count + 1) + 8;
        long long *csum = const_cast<long long *>(chunkoff) + count + 1;
        const long long nch = chunkoff[count];
        for (long long c = blockIdx.x; c < nch; c += gridDim.x)
        {
            const int p = find_product(chunkoff, count, c);
            const BatchProd &bp = prods[p];
            const long long t0 = (c - chunkoff[p]) * SCAN_CHUNK;
            const int n = (int)min((long long)SCAN_CHUNK, (long long)bp.numC - t0);
            const long long tot = bp.status ? 0 : block_sum<NT>(bp.P.C_tnnz + t0, n, s_tmp);
            if (threadIdx.x == 0)
                csum[c] = tot;
        }
        if (!grid_barrier(bar, err))
            return;
        for (int p = blockIdx.x; p < count; p += gridDim.x)
        {
            BatchProd &bp = prods[p];
            const long long tot =
                block_scan_ll<NT>(csum + chunkoff[p], (int)(chunkoff[p + 1] - chunkoff[p]), s_tmp);
            if (threadIdx.x == 0 && !bp.status)
            {
                if (tot > bp.capN)
                {
                    bp.status = 2;
                    bp.nnzC = 0;
                }
                else
                    bp.nnzC = (int)tot;
                bp.P.C_tnnz[bp.numC] = (int)(tot > bp.capN ? 0 : tot);
            }
        }
        if (!grid_barrier(bar, err))
            return;
        for (long long c = blockIdx.x; c < nch; c += gridDim.x)
        {
            const int p = find_product(chunkoff, count, c);
            const BatchProd &bp = prods[p];
            if (bp.status)
                continue;
            const long long t0 = (c - chunkoff[p]) * SCAN_CHUNK;
            const int n = (int)min((long long)SCAN_CHUNK, (long long)bp.numC - t0);
            block_scan_offset<NT>(bp.P.C_tnnz + t0, n, csum[c], s_tmp);
        }
    }
    if (!grid_barrier(bar, err))
        return;
    BATCH_STAMP(6)
    // phase 7: step 3 (the SPA schedule's kernels follow this one, each at its own
    // occupancy; they get the prefix of the dense products' tiles)
    if (SCHED == 3)
    {
        // C tiles of the products that take the tile kernel by rows, prefix,
        // and by columns
        if (blockIdx.x == 0)
            for (int cols = 0; cols < 2; cols++)
            {
                long long *off = denseoff + cols * ((long long)count + 1);
                for (int p = threadIdx.x; p < count; p += NT)
                {
                    const BatchProd &bp = prods[p];
                    off[p] = bp.P.cols == cols && !bp.status && bp.numC > 0 && bp.nnzC >= (long long)dense * bp.numC
                                 ? bp.numC
                                 : 0;
                }
                __syncthreads();
                const long long all = block_scan_ll<NT>(off, count, s_tmp);
                if (threadIdx.x == 0)
                    off[count] = all;
            }
        return;
    }
    if (SCHED == 2)
    {
        int2 *pairs = reinterpret_cast<int2 *>(s_raw) + warp * S3E_PAIRS;
        const long long total_items = itemoff[count];
        for (long long w = (long long)blockIdx.x * (NT / 32) + warp; w < total_items; w += nwarps)
        {
            const int p = find_product(itemoff, count, w);
            if (prods[p].status)
                continue;
            step3_elems_tile(prods[p].P, (int)(w - itemoff[p]), pairs);
        }
    }
    else
    {
        double *tA = reinterpret_cast<double *>(s_raw) + hw * S3T_WORDS;
        bool clear = false; // tA is all zero, as step3_tile_rows takes and leaves it
        const long long total_items = itemoff[count];
        for (long long h = (long long)blockIdx.x * (NT / 16) + hw; h < total_items; h += nhw)
        {
            const int p = find_product(itemoff, count, h);
            if (prods[p].status)
                continue;
            const ProdView &P = prods[p].P;
            const long long item = h - itemoff[p];
            if (SCHED == 1)
                step3_rows_item<W, CAP>(P, item, hmask, lane, reinterpret_cast<S3RowsSmem<W, CAP> *>(s_raw)[hw]);
            else if (SCHED == 0 && P.cols)
            {
                step3_tile_cols(P, (int)item, hmask, lane, tA);
                clear = false;
            }
            else
            {
                if (!clear)
                    step3_tile_clear(tA, hmask, lane);
                step3_tile_rows(P, (int)item, hmask, lane, tA);
                clear = true;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
        atomicMax(&stamp[7], gtimer());
}

// Step 3 of the SPA schedule over a batch, after k_batch: products with
// sparse C tiles, CTAs taking blocks of SPA_BLK C tiles (all products) from a
// device counter.  Raises stamp[7] on exit.  Does nothing when k_batch left
// with an error (its later phases did not run).
__global__ void __launch_bounds__(SPA_THREADS, 3)
    k_batch_spa3(BatchProd *prods, int count, const long long *__restrict__ itemoff, unsigned *bar, const int *err,
                 int dense)
{
    if (*(volatile const int *)err)
        return;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_blk;
    SpaSmem &S = *reinterpret_cast<SpaSmem *>(s_raw);
    const long long *blkoff = itemoff + count + 1;
    unsigned nxt = 0; // thread 0: the next block, claimed one block ahead
    if (threadIdx.x == 0)
        nxt = atomicAdd(&bar[2], 1u);
    int p = 0;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_blk = (int)nxt;
            nxt = atomicAdd(&bar[2], 1u);
        }
        __syncthreads();
        const long long blk = s_blk;
        if (blk >= blkoff[count])
            break;
        p = find_product_from(blkoff, count, blk, p);
        if (prods[p].win || prods[p].status || prods[p].nnzC >= (long long)dense * prods[p].numC ||
            prods[p].hypT == prods[p].numC)
        {
            if (threadIdx.x == 0) // nothing of this product is left to take
                atomicMax(&bar[2], (unsigned)blkoff[p + 1]);
            continue;
        }
        const ProdView &P = prods[p].P;
        const long long tb = (blk - blkoff[p]) * SPA_BLK;
        if (threadIdx.x == 0)
            spa_skip_hyper(P, prods[p].wide, (int)tb, &bar[2], blkoff[p]);
        step3_spa_block<true>(P, S, (int)tb, (int)min((long long)P.numC, tb + SPA_BLK), prods[p].wide, nullptr, false);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(const_cast<long long *>(itemoff)) + 2 * ((long long)count + 1) +
                      7,
                  gtimer());
}

// ... the hypersparse rows of those products, a CTA each, from step 2's list
// (k_batch_spa3, behind it on its stream, raises the end stamp for both: a stamp of
// its own gave it a fifth more instructions, 16 products of 32,768 to 65,536 random
// rows of 8 entries 4.6 -> 5.2 ms) ...
__global__ void __launch_bounds__(SPA_THREADS, 3)
    k_batch_hyper(const BatchProd *prods, const int4 *__restrict__ wlist, unsigned *bar, const int *err, int dense)
{
    if (*(volatile const int *)err)
        return;
    extern __shared__ __align__(16) unsigned char s_raw[];
    HypSmem &S = *reinterpret_cast<HypSmem *>(s_raw);
    __shared__ int s_unit;
    const int units = (int)bar[6];
    unsigned nxt = 0; // thread 0: the next unit, claimed one ahead
    if (threadIdx.x == 0)
        nxt = atomicAdd(&bar[9], 1u);
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_unit = (int)nxt;
            nxt = atomicAdd(&bar[9], 1u);
        }
        __syncthreads();
        if (s_unit >= units)
            break;
        const int4 u = wlist[s_unit];
        const BatchProd &b = prods[u.x];
        if ((u.z & 0xFFFF) == 0 && b.wide[u.y] == 2 && !b.win && !b.status && b.nnzC < (long long)dense * b.numC)
            step3_hyper_row(b.P, S, u.y);
    }
}

// ... the tables of the products that take the windows (prefixes over the
// products of their rows of B, entries of ctab and rows of A), and their
// heavy rows' parts ...
__device__ __forceinline__ bool batch_win_on(const BatchProd &b, int dense)
{
    return b.win && !b.status && b.nnzC > 0 && b.nnzC < (long long)dense * b.numC;
}

__global__ void __launch_bounds__(256)
    k_batch_wtab(const BatchProd *prods, int count, const long long *__restrict__ winoff, int4 *hlist, unsigned *bar,
                 const int *err, int dense)
{
    if (*(volatile const int *)err)
        return;
    const long long *boff = winoff, *toff = boff + count + 1, *aoff = toff + count + 1;
    const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    for (long long w = gt >> 5; w < boff[count]; w += nt >> 5)
    {
        const BatchProd &b = prods[find_product(boff, count, w)];
        if (batch_win_on(b, dense))
            win_btab_row((int)(w - boff[&b - prods]), b.P.B_rptr, b.P.B_rcol, b.Q.blocks, b.Q.bits, b.Q.btab,
                         b.Q.windows, b.Q.wtab);
    }
    for (long long g = gt; g < toff[count]; g += nt)
    {
        const BatchProd &b = prods[find_product(toff, count, g)];
        if (batch_win_on(b, dense))
            win_ctab_entry(b.P, b.Q, g - toff[&b - prods]);
    }
    for (long long g = gt; g < aoff[count]; g += nt)
    {
        const int p = find_product(aoff, count, g);
        const BatchProd &b = prods[p];
        const int row = (int)(g - aoff[p]);
        if (batch_win_on(b, dense) && b.Q.A_rptr[row + 1] - b.Q.A_rptr[row] >= b.Q.heavy_min)
        {
            const int parts = (b.P.nB + WIN_PART - 1) / WIN_PART;
            int4 *at = hlist + atomicAdd(&bar[7], (unsigned)parts);
            for (int q = 0; q < parts; q++)
                at[q] = make_int4(p, row, q, 0);
        }
    }
}

// ... their numeric step ...
__global__ void __launch_bounds__(WIN_THREADS, WIN_CTAS)
    k_batch_win(const BatchProd *prods, int count, const long long *__restrict__ winoff, const int4 *__restrict__ hlist,
                const long long *itemoff, unsigned *bar, const int *err, int dense)
{
    if (*(volatile const int *)err)
        return;
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int lane = threadIdx.x & 31;
    WinTask &S = reinterpret_cast<WinTask *>(s_raw)[threadIdx.x >> 5];
    for (int q = lane; q < WIN_COLS; q += 32)
        S.acc[q] = 0.0;
    __syncwarp();
    const long long *coff = winoff + 3 * ((long long)count + 1);
    const unsigned hclaims = bar[7], claims = hclaims + (unsigned)coff[count];
    unsigned nxt = 0;
    int p = 0;
    if (lane == 0)
        nxt = atomicAdd(&bar[8], 1u);
    for (;;)
    {
        const unsigned c = __shfl_sync(TSG_FULL_MASK, nxt, 0);
        if (c >= claims)
            break;
        if (lane == 0)
            nxt = atomicAdd(&bar[8], 1u);
        if (c < hclaims)
        {
            const int4 h = hlist[c];
            win_claim_heavy(prods[h.x].P, prods[h.x].Q, S, h.y, h.z, lane);
            continue;
        }
        p = find_product_from(coff, count, c - hclaims, p);
        if (batch_win_on(prods[p], dense))
            win_claim_rows(prods[p].P, prods[p].Q, S, 0, (unsigned)(c - hclaims - coff[p]), lane);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(const_cast<long long *>(itemoff)) + 2 * ((long long)count + 1) +
                      7,
                  gtimer());
}

// ... and products with dense C tiles (>= the batch's threshold of values per
// tile on average): the tile kernel in the form of their A tiles (P.cols), a
// half-warp per C tile of theirs (denseoff: their tiles, prefix; walked among
// the tiles of all products, finding out cost four times the work).
#define DENSE3_THREADS 128
template <bool COLS>
__global__ void __launch_bounds__(DENSE3_THREADS, COLS ? 4 : 8)
    k_batch_dense3(BatchProd *prods, int count, const long long *__restrict__ denseoff, const long long *__restrict__ itemoff,
                   const int *err)
{
    if (*(volatile const int *)err)
        return;
    __shared__ __align__(16) double s_A[DENSE3_THREADS / 16][S3T_WORDS];
    const int lane = threadIdx.x & 15, hw = threadIdx.x >> 4;
    const unsigned hmask = TSG_HW_MASK(threadIdx.x);
    const long long total_items = denseoff[count];
    if (total_items == 0)
        return;
    if (!COLS)
        step3_tile_clear(s_A[hw], hmask, lane);
    const long long nhw = (long long)gridDim.x * (DENSE3_THREADS / 16);
    for (long long h = (long long)blockIdx.x * (DENSE3_THREADS / 16) + hw; h < total_items; h += nhw)
    {
        const int p = find_product(denseoff, count, h);
        if (COLS)
            step3_tile_cols(prods[p].P, (int)(h - denseoff[p]), hmask, lane, s_A[hw]);
        else
            step3_tile_rows(prods[p].P, (int)(h - denseoff[p]), hmask, lane, s_A[hw]);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(const_cast<long long *>(itemoff)) + 2 * ((long long)count + 1) +
                      7,
                  gtimer());
}

// ---------------------------------------------------------------------------
// upper bounds: matched tile pairs and scalar products per product
// ---------------------------------------------------------------------------
// half-warp per B tile row: element row lengths of B from the tile masks
__global__ void k_brow_len(int tilem, int m, const int *__restrict__ tile_ptr, const unsigned short *__restrict__ mask,
                           int *__restrict__ rowlen)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int tr = (int)(gid >> 4), lane = threadIdx.x & 15;
    if (tr >= tilem)
        return;
    int s = 0;
    for (int t = tile_ptr[tr]; t < tile_ptr[tr + 1]; t++)
        s += __popc((unsigned)mask[(long long)t * TSG_BS + lane]);
    if (tr * TSG_BS + lane < m)
        rowlen[tr * TSG_BS + lane] = s;
}

// half-warp per A tile: tile pairs and scalar products it generates
__global__ void k_bounds(int T, const int *__restrict__ A_col, const unsigned short *__restrict__ A_mask,
                         const int *__restrict__ B_ptr, const int *__restrict__ browlen, int mB,
                         unsigned long long *__restrict__ out)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = (int)(gid >> 4), lane = threadIdx.x & 15;
    unsigned long long prods = 0, pairs = 0;
    if (t < T)
    {
        const int k = A_col[t];
        unsigned ma = A_mask[(long long)t * TSG_BS + lane];
        while (ma)
        {
            const int bit = 31 - __clz(ma);
            const int row = k * TSG_BS + (15 - bit);
            if (row < mB)
                prods += (unsigned long long)browlen[row];
            ma ^= 1u << bit;
        }
        if (lane == 0)
            pairs = (unsigned long long)(B_ptr[k + 1] - B_ptr[k]);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
    {
        prods += __shfl_xor_sync(TSG_FULL_MASK, prods, d);
        pairs += __shfl_xor_sync(TSG_FULL_MASK, pairs, d);
    }
    if ((threadIdx.x & 31) == 0 && (prods || pairs))
    {
        atomicAdd(out, prods);
        atomicAdd(out + 1, pairs);
    }
}

extern "C" int tsg_product_bounds_many(tsg_context *ctx, int count, const tsg_tiled *A, const tsg_tiled *B,
                                       long long *products, long long *tile_pairs, long long *c_tiles)
{
    if (!ctx || count < 0 || (count && (!A || !B || !products || !tile_pairs)))
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    if (count == 0)
        return TSG_OK;
    int maxm = 0;
    for (int p = 0; p < count; p++)
        maxm = B[p].m > maxm ? B[p].m : maxm;
    int *rowlen;
    unsigned long long *d;
    TSG_TRY(tsg_alloc(ctx, &rowlen, (size_t)maxm + 1));
    TSG_TRY(tsg_alloc(ctx, &d, (size_t)count * 3));
    TSG_CUDA(cudaMemsetAsync(d, 0, (size_t)count * 3 * sizeof(unsigned long long), ctx->stream));
    int st = TSG_OK;
    for (int p = 0; p < count && st == TSG_OK; p++)
    {
        // k_brow_len writes every row of B below m: the buffer is reused in
        // stream order without clearing
        if (B[p].tilem > 0)
        {
            k_brow_len<<<tsg_blocks((long long)B[p].tilem * 16, 256), 256, 0, ctx->stream>>>(
                B[p].tilem, B[p].m, B[p].tile_ptr, B[p].mask, rowlen);
            TSG_LAUNCH_CHECK();
        }
        if (A[p].numtile > 0)
        {
            k_bounds<<<tsg_blocks((long long)A[p].numtile * 16, 256), 256, 0, ctx->stream>>>(
                A[p].numtile, A[p].tile_columnidx, A[p].mask, B[p].tile_ptr, rowlen, B[p].m, d + 3 * p);
            TSG_LAUNCH_CHECK();
        }
        if (c_tiles)
            st = tsg_count_c_tiles_async(ctx, &A[p], &B[p], d + 3 * p + 2);
    }
    if (st == TSG_OK)
    {
        std::vector<unsigned long long> h((size_t)count * 3);
        TSG_CUDA(cudaMemcpyAsync(h.data(), d, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 ctx->stream));
        TSG_CUDA(cudaStreamSynchronize(ctx->stream));
        for (int p = 0; p < count; p++)
        {
            products[p] = (long long)h[3 * p];
            tile_pairs[p] = (long long)h[3 * p + 1];
            if (c_tiles)
                c_tiles[p] = (long long)h[3 * p + 2];
        }
    }
    tsg_release(ctx, rowlen);
    tsg_release(ctx, d);
    return st;
}

extern "C" int tsg_product_bounds(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, long long *products,
                                  long long *tile_pairs)
{
    if (!ctx || !A || !B || !products || !tile_pairs)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    return tsg_product_bounds_many(ctx, 1, A, B, products, tile_pairs, nullptr);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef void (*batch_kernel_t)(BatchProd *, int, const long long *, const long long *, int4 *, int, int, long long *,
                               int, long long *, unsigned *, int *, int *);

// Kernel, dynamic shared memory and block size of a batch schedule.  cols:
// some product takes the columns form of the tile kernel, whose registers would
// halve the blocks of a batch that has none (SCHED 4).
static batch_kernel_t pick_kernel(const tsg_batch_params &p, bool cols, size_t *smem, int *threads)
{
    *threads = BATCH_THREADS;
    const size_t s1a = (size_t)(BATCH_THREADS / 32) * S1_WORDS * 4;
    const size_t s12 = (size_t)(BATCH_THREADS / 32) * sizeof(S12Smem);
    const size_t s1 = std::max(std::max(s1a, s12), sizeof(S1cSmem<BATCH_THREADS>));
    if (p.schedule == TSG_SCHED_SPA)
    {
        *threads = SPA_THREADS;
        const size_t t1a = (size_t)(SPA_THREADS / 32) * S1_WORDS * 4;
        const size_t t12 = (size_t)(SPA_THREADS / 32) * sizeof(S12Smem);
        *smem = std::max(std::max(t1a, t12), std::max(wide_smem<SPA_THREADS>(BATCH_SPAN), sizeof(S1cSmem<SPA_THREADS>)));
        return k_batch<3, 8, 256, SPA_THREADS>;
    }
    if (p.schedule == TSG_SCHED_ELEMS)
    {
        const size_t s3 = (size_t)(BATCH_THREADS / 32) * S3E_PAIRS * sizeof(int2);
        *smem = s1 > s3 ? s1 : s3;
        return k_batch<2, 8, 256, BATCH_THREADS>;
    }
    if (p.schedule == TSG_SCHED_TILES)
    {
        const size_t s3 = (size_t)(BATCH_THREADS / 16) * S3T_WORDS * 8;
        *smem = s1 > s3 ? s1 : s3;
        return cols ? k_batch<0, 8, 256, BATCH_THREADS> : k_batch<4, 8, 256, BATCH_THREADS>;
    }
#define TSG_PICK(w, c)                                                                          \
    if (p.seg_tiles == w && p.acc_cap == c)                                                     \
    {                                                                                           \
        size_t s2 = (size_t)(BATCH_THREADS / 16) * sizeof(S2RowsSmem<w>);                       \
        size_t s3 = (size_t)(BATCH_THREADS / 16) * sizeof(S3RowsSmem<w, c>);                    \
        size_t mx = s1 > s2 ? s1 : s2;                                                          \
        *smem = mx > s3 ? mx : s3;                                                              \
        return k_batch<1, w, c, BATCH_THREADS>;                                                 \
    }
    TSG_ROW_CONFIGS(TSG_PICK)
#undef TSG_PICK
    return nullptr;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static int record_run(tsg_batch *b, cudaStream_t st)
{
    size_t smem;
    int threads;
    batch_kernel_t kern = pick_kernel(b->params, b->cols_form > 0, &smem, &threads);
    TSG_CUDA(cudaMemsetAsync(b->d_err, 0, sizeof(int), st));
    TSG_CUDA(cudaMemsetAsync(b->d_bar, 0, sizeof(unsigned), st));
    // phase stamps (after the two item prefixes): [7] is a running maximum
    TSG_CUDA(cudaMemsetAsync(b->d_itemoff + 2 * ((size_t)b->count + 1), 0, 8 * sizeof(long long), st));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)b->grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = b->smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TSG_CUDA(cudaLaunchKernelEx(&cfg, kern, b->d_prod, b->count, (const long long *)b->d_rowoff,
                                (const long long *)b->d_s1off, b->d_wlist, b->split,
                                s12_per_pair(b->rowoff[b->count], b->ctx->num_sms), b->d_denseoff, b->dense,
                                b->d_itemoff,
                                b->d_bar, b->d_err, b->d_bins));
    if (b->params.schedule != TSG_SCHED_SPA)
        return TSG_OK;
    // step 3's kernels share no product: side by side, so that none waits for
    // another's last rows.  k_batch_hyper and k_batch_spa3, of the same products,
    // stay in order: a branch more costs every batch (64 tiny products, step 3 0.039
    // ms, 0.080 with a third).
    TSG_TRY(tsg_fork(b->ctx, st, TSG_SIDE_STREAMS));
    cudaStream_t *side = b->ctx->side;
    if (b->wins)
    {
        k_batch_wtab<<<b->ctx->num_sms * 8, 256, 0, st>>>(b->d_prod, b->count, b->d_winoff, b->d_hlist, b->d_bar, b->d_err,
                                                          b->dense);
        TSG_CUDA(cudaGetLastError());
        k_batch_win<<<b->gridw, WIN_THREADS, WIN_WARPS * sizeof(WinTask), st>>>(
            b->d_prod, b->count, b->d_winoff, b->d_hlist, b->d_itemoff, b->d_bar, b->d_err, b->dense);
        TSG_CUDA(cudaGetLastError());
    }
    k_batch_hyper<<<b->gridh, SPA_THREADS, sizeof(HypSmem), side[0]>>>(b->d_prod, b->d_wlist, b->d_bar, b->d_err, b->dense);
    TSG_CUDA(cudaGetLastError());
    k_batch_spa3<<<b->grid3, SPA_THREADS, sizeof(SpaSmem), side[0]>>>(b->d_prod, b->count, b->d_itemoff, b->d_bar, b->d_err,
                                                                    b->dense);
    TSG_CUDA(cudaGetLastError());
    // dense A tiles first, before the windows' CTAs hold the SMs' shared memory
    if (b->cols_form)
    {
        k_batch_dense3<true><<<b->ctx->num_sms * 4, DENSE3_THREADS, 0, side[1]>>>(
            b->d_prod, b->count, b->d_denseoff + b->count + 1, b->d_itemoff, b->d_err);
        TSG_CUDA(cudaGetLastError());
    }
    if (b->rows_form)
    {
        k_batch_dense3<false><<<b->ctx->num_sms * 8, DENSE3_THREADS, 0, side[1]>>>(b->d_prod, b->count, b->d_denseoff,
                                                                                 b->d_itemoff, b->d_err);
        TSG_CUDA(cudaGetLastError());
    }
    TSG_TRY(tsg_join(b->ctx, st, TSG_SIDE_STREAMS));
    return TSG_OK;
}

// A product's share of a batch, from its bounds: what batch_create lays out and
// tsg_batch_product_bytes predicts.
struct BatchShare
{
    long long capN;                        // values of C at most
    size_t arena;                          // C's arrays, tile rows' counts and kinds
    long long units, chunks;               // of step 2's wide rows; of the tile-count scan
    int win, windows, bits, blocks;        // step 3 by windows
    long long centries, claims, parts, words; // ctab's entries, claims, heavy rows' parts, words of all tables
    int heavy_min;
    bool wtab;
};

// win_words: table words that the batch has left
static BatchShare batch_share(const tsg_tiled *A, const tsg_tiled *B, int schedule, long long prods, long long capT,
                              int split, long long win_words)
{
    BatchShare S = {};
    S.capN = std::min(prods, 256 * capT);
    S.arena = align256(((size_t)A->tilem + 1) * 4) + align256((size_t)A->tilem * 4) + 2 * align256((size_t)capT * 4) +
              align256(((size_t)capT + 1) * 4) + align256((size_t)capT * 32) + align256((size_t)capT * 16) +
              align256((size_t)S.capN) + align256((size_t)S.capN * 8);
    S.units = (long long)wide_units(A->tilem, A->nnz, split);
    S.chunks = (capT + SCAN_CHUNK - 1) / SCAN_CHUNK;
    if (schedule != TSG_SCHED_SPA || !A->row_ptr || A->m < 1 || B->m < 1 || B->n < 1)
        return S;
    const long long windows = (B->n + WIN_COLS - 1LL) / WIN_COLS;
    if (prods < BATCH_WIN_MIN * windows * A->m)
        return S;
    S.heavy_min = win_heavy(A->nnz, A->m);
    S.centries = A->tilem * (windows + 1);
    S.claims = (long long)A->tilem * windows * WIN_PER;
    S.parts = std::min((long long)A->m, (long long)A->nnz / S.heavy_min) * ((B->n + WIN_PART - 1LL) / WIN_PART);
    // all that the windows take: btab (coarser blocks when it is large), wtab
    // unless it alone is too much, ctab and the list of heavy rows' parts
    const long long rest = S.centries + 4 * S.parts + 2;
    S.wtab = 2 * windows * B->m + rest <= BATCH_WIN_WORDS / 2;
    const long long fixed = rest + (S.wtab ? 2 * windows * B->m : 0);
    if (fixed >= BATCH_WIN_WORDS || !win_table(B->m, B->n, BATCH_WIN_WORDS - fixed, S.bits, S.blocks))
        return S;
    S.words = fixed + (S.blocks + 1LL) * B->m;
    S.windows = (int)windows;
    S.win = S.words <= win_words && win_worth(S.capN, (long long)((double)A->nnz * (double)B->nnz / B->m), A->nnz, capT,
                                              A->tilem, B->tilen, windows, S.words);
    return S;
}

// Bytes of a batch beside its arena and tables, and of a product in them (rounded up)
#define BATCH_FIXED_BYTES 2048
#define BATCH_PRODUCT_BYTES (sizeof(BatchProd) + 128)

static size_t batch_share_bytes(const BatchShare &S, long long tilem)
{
    return S.arena + BATCH_PRODUCT_BYTES + 8 * (size_t)S.chunks + sizeof(int4) * (size_t)S.units +
           (S.win ? 4 * (size_t)S.words : 0);
}

extern "C" int tsg_batch_product_bytes(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, int schedule,
                                       long long products, long long c_tiles, long long *bytes)
{
    if (!ctx || !A || !B || !bytes || products < 0 || c_tiles < 0)
        return tsg_set_error(TSG_ERR_INVALID, "bad arguments");
    // alone in its batch a product has the largest share: the whole of the
    // table words, rows in the most parts
    const int split = wide_split(A->nnz, ctx->num_sms);
    *bytes = BATCH_FIXED_BYTES +
             (long long)batch_share_bytes(batch_share(A, B, schedule, products, c_tiles, split, BATCH_WIN_TOTAL), A->tilem);
    return TSG_OK;
}

// products / c_tiles: the bounds of every product when the caller has them
// (tsg_product_bounds_many), else null and computed here
static int batch_create(tsg_context *ctx, int count, const tsg_tiled *A, const tsg_tiled *B,
                        const tsg_batch_params *params, const long long *products, const long long *c_tiles,
                        tsg_batch **out)
{
    if (!ctx || !out || count <= 0 || !A || !B)
        return tsg_set_error(TSG_ERR_INVALID, "bad batch arguments");
    *out = nullptr;
    tsg_batch_params prm;
    if (params)
        prm = *params;
    else
    {
        prm.schedule = TSG_SCHED_ROWS;
        prm.seg_tiles = 16;
        prm.acc_cap = 1024;
        prm.use_graph = 1;
        prm.dense_threshold = 0;
    }
    if (prm.dense_threshold < 0 || prm.dense_threshold > 257)
        return tsg_set_error(TSG_ERR_INVALID, "dense threshold %d outside [0, 257]", prm.dense_threshold);
    size_t smem;
    int threads;
    int cols_form = 0;
    for (int p = 0; p < count; p++)
        cols_form += step3_by_columns(&A[p]);
    batch_kernel_t kern = pick_kernel(prm, cols_form > 0, &smem, &threads);
    if (!kern)
        return tsg_set_error(TSG_ERR_INVALID, "unsupported batch schedule (%d, %d, %d)", prm.schedule, prm.seg_tiles,
                             prm.acc_cap);
    for (int p = 0; p < count; p++)
    {
        if (A[p].n != B[p].m || !B[p].csc_tile_ptr)
            return tsg_set_error(TSG_ERR_INVALID, "product %d: inner dimensions differ or B lacks its column view", p);
        if (prm.schedule == TSG_SCHED_ELEMS && !B[p].mask_t)
            return tsg_set_error(TSG_ERR_INVALID, "product %d: element schedule needs B's column masks", p);
        if (prm.schedule == TSG_SCHED_SPA && !B[p].row_ptr)
            return tsg_set_error(TSG_ERR_INVALID, "product %d: SPA schedule needs B's row view", p);
    }
    tsg_batch *b = new tsg_batch();
    b->ctx = ctx;
    b->count = count;
    b->params = prm;
    b->dense = prm.dense_threshold ? prm.dense_threshold : SPA_DENSE;
    b->host.resize(count);
    b->rowoff.resize(count + 1);
    b->m.resize(count);
    b->n.resize(count);
    b->tilen.resize(count);
    b->launches = 0;
    b->cols_form = cols_form;
    b->rows_form = count - cols_form;
    // bounds and arena layout
    size_t bytes = 0;
    std::vector<size_t> off(count);
    long long run = 0, chunk_cap = 0, total_prods = 0;
    // scalar products and the exact C tile count (step 1's count pass) of
    // every product, one synchronisation for the whole batch
    std::vector<long long> v_prods(count), v_pairs(count), v_tiles(count);
    if (products && c_tiles)
        for (int p = 0; p < count; p++)
        {
            if (products[p] < 0 || c_tiles[p] < 0)
            {
                delete b;
                return tsg_set_error(TSG_ERR_INVALID, "product %d: negative bound", p);
            }
            v_prods[p] = products[p];
            v_tiles[p] = c_tiles[p];
        }
    else
    {
        int st = tsg_product_bounds_many(ctx, count, A, B, v_prods.data(), v_pairs.data(), v_tiles.data());
        if (st != TSG_OK)
        {
            delete b;
            return st;
        }
    }
    b->s1off.assign(2 * ((size_t)count + 1), 0);
    b->winoff.assign(4 * ((size_t)count + 1), 0);
    std::vector<BatchShare> share(count);
    long long wunits = 0, hparts = 0, words = 0, entries = 0;
    for (int p = 0; p < count; p++)
        entries += A[p].nnz;
    b->split = wide_split(entries, ctx->num_sms);
    b->arena_bytes = BATCH_FIXED_BYTES;
    for (int p = 0; p < count; p++)
    {
        const long long prods = v_prods[p], capT = v_tiles[p];
        const bool cta = step1_by_cta(&A[p], &B[p]);
        b->s1off[p + 1] = b->s1off[p] + (cta ? A[p].tilem : 0);
        b->s1off[count + 2 + p] = b->s1off[count + 1 + p] + (cta ? 0 : A[p].tilem);
        total_prods += prods;
        if (std::min(prods, 256 * capT) > 2147483647LL || capT > 2147483647LL / 16)
        {
            delete b;
            return tsg_set_error(TSG_ERR_OVERFLOW, "product %d exceeds 32-bit offsets", p);
        }
        BatchShare &S = share[p] = batch_share(&A[p], &B[p], prm.schedule, prods, capT, b->split, BATCH_WIN_TOTAL - words);
        if (S.win && b->winoff[3 * ((size_t)count + 1) + p] + S.claims + hparts + S.parts >= 2147483647LL)
            S.win = 0;
        b->arena_bytes += batch_share_bytes(S, A[p].tilem);
        wunits += S.units;
        chunk_cap += S.chunks;
        BatchProd &h = b->host[p];
        memset(&h, 0, sizeof(h));
        h.capT = capT;
        h.capN = S.capN;
        h.tilemA = A[p].tilem;
        if (S.win)
        {
            h.win = 1;
            h.Q.windows = S.windows;
            h.Q.bits = S.bits;
            h.Q.blocks = S.blocks;
            h.Q.mA = A[p].m;
            h.Q.heavy_min = S.heavy_min;
            hparts += S.parts;
            words += S.words;
            b->wins++;
        }
        const long long add[4] = {B[p].m, S.centries, A[p].m, S.claims};
        for (int q = 0; q < 4; q++)
            b->winoff[q * ((size_t)count + 1) + p + 1] = b->winoff[q * ((size_t)count + 1) + p] + (h.win ? add[q] : 0);
        b->rowoff[p] = run;
        run += A[p].tilem;
        b->m[p] = A[p].m;
        b->n[p] = B[p].n;
        b->tilen[p] = B[p].tilen;
        off[p] = bytes;
        bytes += S.arena;
    }
    b->rowoff[count] = run;
    // the tables' words without the lists of heavy rows' parts
    const long long table_words = words - 4 * hparts;
    int st = TSG_OK;
    if ((st = tsg_alloc(ctx, (char **)&b->arena, bytes ? bytes : 256)) != TSG_OK)
    {
        delete b;
        return st;
    }
    if (prm.schedule == TSG_SCHED_SPA && (st = tsg_side_streams(ctx, TSG_SIDE_STREAMS)) != TSG_OK)
    {
        tsg_batch_destroy(b);
        return st;
    }
    if (b->wins && ((st = tsg_alloc(ctx, &b->win_tables, (size_t)table_words)) != TSG_OK ||
                    (st = tsg_alloc(ctx, &b->d_hlist, (size_t)hparts)) != TSG_OK ||
                    (st = tsg_alloc(ctx, &b->d_winoff, b->winoff.size())) != TSG_OK))
    {
        if (st != TSG_ERR_OOM)
        {
            tsg_batch_destroy(b);
            return st;
        }
        // no room for the tables, which the SPA kernel does without
        cudaGetLastError();
        tsg_release(ctx, b->win_tables);
        tsg_release(ctx, b->d_hlist);
        for (BatchProd &h : b->host)
            h.win = 0;
        b->wins = 0;
        b->arena_bytes -= 4 * (size_t)words;
    }
    if ((st = tsg_alloc(ctx, &b->d_denseoff, 2 * ((size_t)count + 1))) != TSG_OK ||
        (st = tsg_alloc(ctx, &b->d_s1off, b->s1off.size())) != TSG_OK ||
        (st = tsg_alloc(ctx, &b->d_wlist, (size_t)wunits)) != TSG_OK)
    {
        tsg_batch_destroy(b);
        return st;
    }
    long long table = 0;
    for (int p = 0; p < count; p++)
    {
        BatchProd &h = b->host[p];
        char *q = (char *)b->arena + off[p];
        auto take = [&](size_t nbytes) {
            char *r = q;
            q += align256(nbytes);
            return r;
        };
        ProdView &P = h.P;
        P.A_ptr = A[p].tile_ptr;
        P.A_col = A[p].tile_columnidx;
        P.A_tnnz = A[p].tile_nnz;
        P.A_Ptr = A[p].tile_csr_Ptr;
        P.A_Colb = A[p].tile_csr_Col;
        P.A_Val = A[p].tile_csr_Value;
        P.A_mask = A[p].mask;
        P.tilemA = A[p].tilem;
        P.B_ptr = B[p].tile_ptr;
        P.B_col = B[p].tile_columnidx;
        P.B_cptr = B[p].csc_tile_ptr;
        P.B_crow = B[p].csc_tile_rowidx;
        P.B_cpos = B[p].csc_tile_pos;
        P.B_tnnz = B[p].tile_nnz;
        P.B_Ptr = B[p].tile_csr_Ptr;
        P.B_Colb = B[p].tile_csr_Col;
        P.B_Val = B[p].tile_csr_Value;
        P.B_mask = B[p].mask;
        P.B_maskT = B[p].mask_t;
        P.B_rptr = B[p].row_ptr;
        P.B_rcol = B[p].row_col;
        P.B_rval = B[p].row_val;
        P.A_rptr = A[p].row_ptr;
        P.A_rcol = A[p].row_col;
        P.A_rval = A[p].row_val;
        P.mA = A[p].m;
        P.mB = B[p].m;
        P.nB = B[p].n;
        P.browB = B[p].m > 0 ? (int)(B[p].nnz / B[p].m) : 0;
        P.cols = step3_by_columns(&A[p]);
        P.tilenB = B[p].tilen;
        P.C_ptr = (int *)take(((size_t)A[p].tilem + 1) * 4);
        h.wide = (int *)take((size_t)A[p].tilem * 4);
        P.C_col = (int *)take((size_t)h.capT * 4);
        P.C_row = (int *)take((size_t)h.capT * 4);
        P.C_tnnz = (int *)take(((size_t)h.capT + 1) * 4);
        P.C_mask = (unsigned short *)take((size_t)h.capT * 32);
        P.C_Ptr = (unsigned char *)take((size_t)h.capT * 16);
        P.C_Colb = (unsigned char *)take((size_t)h.capN);
        P.C_Val = (double *)take((size_t)h.capN * 8);
        P.numC = 0;
        P.padded = 0;
        P.status = nullptr; // the batch's error word, set once it is allocated
        // step 1's bitmaps stay in the value range, which step 3 is the first to write
        const int stride = std::min((B[p].tilen + 31) / 32, S1_KEEP_WORDS);
        const size_t kept = ((size_t)A[p].tilem * stride * 4 + 15) & ~(size_t)15;
        if (prm.schedule != TSG_SCHED_ROWS && kept + (size_t)A[p].tilem * sizeof(int2) <= (size_t)h.capN * 8)
        {
            h.K.words = (unsigned *)P.C_Val;
            h.K.span = (int2 *)((char *)P.C_Val + kept);
            h.K.stride = stride;
        }
        if (h.win)
        {
            h.Q.A_rptr = P.A_rptr;
            h.Q.A_rcol = P.A_rcol;
            h.Q.A_rval = P.A_rval;
            table = (table + 1) & ~1LL; // wtab holds pairs
            h.Q.wtab = share[p].wtab ? (int2 *)(b->win_tables + table) : nullptr;
            h.Q.btab = b->win_tables + table + (share[p].wtab ? 2LL * h.Q.windows * P.mB : 0);
            h.Q.ctab = h.Q.btab + (h.Q.blocks + 1LL) * P.mB;
            table += share[p].words - 4 * share[p].parts;
        }
    }
    if ((st = tsg_alloc(ctx, &b->d_prod, (size_t)count)) != TSG_OK || (st = tsg_alloc(ctx, &b->d_rowoff, (size_t)count + 1)) ||
        (st = tsg_alloc(ctx, &b->d_itemoff, 3 * ((size_t)count + 1) + 8 + (size_t)chunk_cap)) || (st = tsg_alloc(ctx, &b->d_bar, 16)) ||
        (st = tsg_alloc(ctx, &b->d_err, 1)) || (st = tsg_alloc(ctx, &b->d_bins, 4)))
    {
        tsg_batch_destroy(b);
        return st;
    }
    cudaStream_t s = ctx->stream;
    // an in-kernel error (a numeric accumulator overflow) goes to the batch's error word
    for (BatchProd &h : b->host)
        h.P.status = b->d_err;
    // copies only (no memset kernels): creating a batch never waits for SMs
    // held by another stream's persistent kernel
    b->wait_ns = BATCH_WAIT_FLOOR_NS + BATCH_WAIT_NS_PER_PRODUCT * (unsigned long long)total_prods;
    memset(b->bar_init, 0, sizeof(b->bar_init));
    memcpy(&b->bar_init[4], &b->wait_ns, sizeof(unsigned long long));
    cudaMemcpyAsync(b->d_prod, b->host.data(), sizeof(BatchProd) * count, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(b->d_rowoff, b->rowoff.data(), sizeof(long long) * (count + 1), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(b->d_s1off, b->s1off.data(), sizeof(long long) * b->s1off.size(), cudaMemcpyHostToDevice, s);
    if (b->wins)
        cudaMemcpyAsync(b->d_winoff, b->winoff.data(), sizeof(long long) * b->winoff.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(b->d_bar, b->bar_init, sizeof(b->bar_init), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(b->d_err, &b->bar_init[0], sizeof(int), cudaMemcpyHostToDevice, s);
    // co-resident grid
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    {
        tsg_batch_destroy(b);
        return tsg_set_error(TSG_ERR_CUDA, "cannot reserve %zu bytes of shared memory", smem);
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (per_sm < 1)
    {
        tsg_batch_destroy(b);
        return tsg_set_error(TSG_ERR_CUDA, "batch kernel cannot be resident");
    }
    b->grid = per_sm * ctx->num_sms;
    b->grid3 = 0;
    if (prm.schedule == TSG_SCHED_SPA)
    {
        int per3 = 0, perh = 0;
        if (cudaFuncSetAttribute(k_batch_hyper, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HypSmem)) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perh, k_batch_hyper, SPA_THREADS, sizeof(HypSmem)) !=
                cudaSuccess ||
            perh < 1 ||
            cudaFuncSetAttribute(k_batch_spa3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SpaSmem)) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per3, k_batch_spa3, SPA_THREADS, sizeof(SpaSmem)) !=
                cudaSuccess ||
            per3 < 1)
        {
            tsg_batch_destroy(b);
            return tsg_set_error(TSG_ERR_CUDA, "batch numeric kernel cannot be resident");
        }
        b->grid3 = per3 * ctx->num_sms;
        b->gridh = perh * ctx->num_sms;
    }
    if (b->wins)
    {
        int perw = 0;
        const int wsmem = WIN_WARPS * (int)sizeof(WinTask);
        if (cudaFuncSetAttribute(k_batch_win, cudaFuncAttributeMaxDynamicSharedMemorySize, wsmem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perw, k_batch_win, WIN_THREADS, wsmem) != cudaSuccess || perw < 1)
        {
            tsg_batch_destroy(b);
            return tsg_set_error(TSG_ERR_CUDA, "batch window kernel cannot be resident");
        }
        b->gridw = perw * ctx->num_sms;
    }
    b->block = threads;
    b->smem = smem;
    b->graph_ok = 0;
    if (prm.use_graph)
    {
        cudaStream_t cs;
        if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) == cudaSuccess)
        {
            cudaStreamSynchronize(s);
            if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess)
            {
                int rs = record_run(b, cs);
                cudaGraph_t g = nullptr;
                cudaError_t e = cudaStreamEndCapture(cs, &g);
                if (rs == TSG_OK && e == cudaSuccess && g &&
                    cudaGraphInstantiate(&b->exec, g, 0) == cudaSuccess)
                {
                    b->graph = g;
                    b->graph_ok = 1;
                }
                else if (g)
                    cudaGraphDestroy(g);
            }
            cudaGetLastError(); // a failed capture falls back to direct launches
            cudaStreamDestroy(cs);
        }
    }
    TSG_CUDA(cudaStreamSynchronize(s));
    *out = b;
    return TSG_OK;
}

extern "C" int tsg_batch_create(tsg_context *ctx, int count, const tsg_tiled *A, const tsg_tiled *B,
                                const tsg_batch_params *params, tsg_batch **out)
{
    return batch_create(ctx, count, A, B, params, nullptr, nullptr, out);
}

extern "C" int tsg_batch_create_bounded(tsg_context *ctx, int count, const tsg_tiled *A, const tsg_tiled *B,
                                        const tsg_batch_params *params, const long long *products,
                                        const long long *c_tiles, tsg_batch **out)
{
    if (!products || !c_tiles)
        return tsg_set_error(TSG_ERR_INVALID, "null bounds");
    return batch_create(ctx, count, A, B, params, products, c_tiles, out);
}

extern "C" int tsg_batch_run(tsg_batch *b)
{
    if (!b)
        return tsg_set_error(TSG_ERR_INVALID, "null batch");
    tsg_context *ctx = b->ctx;
    if (b->graph_ok)
        TSG_CUDA(cudaGraphLaunch(b->exec, ctx->stream));
    else
        TSG_TRY(record_run(b, ctx->stream));
    ctx->launches++;
    b->launches++;
    return TSG_OK;
}

extern "C" int tsg_batch_sync(tsg_batch *b, long long *total_tiles, long long *total_nnz)
{
    if (!b)
        return tsg_set_error(TSG_ERR_INVALID, "null batch");
    tsg_context *ctx = b->ctx;
    int err = 0;
    TSG_CUDA(cudaMemcpyAsync(b->host.data(), b->d_prod, sizeof(BatchProd) * b->count, cudaMemcpyDeviceToHost,
                             ctx->stream));
    TSG_CUDA(cudaMemcpyAsync(&err, b->d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    TSG_CUDA(cudaStreamSynchronize(ctx->stream));
    if (err == TSG_ERR_OVERFLOW)
        return tsg_set_error(TSG_ERR_OVERFLOW, "a numeric accumulator of the batch overflowed");
    if (err)
        return tsg_set_error(TSG_ERR_TIMEOUT, "batch grid barrier gave up waiting (bound %.3f s)", b->wait_ns * 1e-9);
    long long tt = 0, tn = 0;
    for (int p = 0; p < b->count; p++)
    {
        if (b->host[p].status)
            return tsg_set_error(TSG_ERR_OVERFLOW, "product %d exceeded its bound (%d)", p, b->host[p].status);
        tt += b->host[p].numC;
        tn += b->host[p].nnzC;
    }
    if (total_tiles)
        *total_tiles = tt;
    if (total_nnz)
        *total_nnz = tn;
    return TSG_OK;
}

extern "C" int tsg_batch_set_wait_limit(tsg_batch *b, double seconds)
{
    if (!b || !(seconds >= 0.0) || seconds > 1e6)
        return tsg_set_error(TSG_ERR_INVALID, "bad batch wait limit");
    tsg_context *ctx = b->ctx;
    b->wait_ns = (unsigned long long)(seconds * 1e9);
    TSG_CUDA(cudaMemcpyAsync(b->d_bar + 4, &b->wait_ns, sizeof(unsigned long long), cudaMemcpyHostToDevice,
                             ctx->stream));
    TSG_CUDA(cudaStreamSynchronize(ctx->stream));
    return TSG_OK;
}

extern "C" int tsg_batch_product(tsg_batch *b, int p, tsg_tiled *C)
{
    if (!b || !C || p < 0 || p >= b->count)
        return tsg_set_error(TSG_ERR_INVALID, "bad batch product index");
    const BatchProd &h = b->host[p];
    memset(C, 0, sizeof(*C));
    C->m = b->m[p];
    C->n = b->n[p];
    C->tilem = h.tilemA;
    C->tilen = b->tilen[p];
    C->numtile = h.numC;
    C->nnz = h.nnzC;
    C->tile_ptr = h.P.C_ptr;
    C->tile_columnidx = h.P.C_col;
    C->tile_rowidx = h.P.C_row;
    C->tile_nnz = h.P.C_tnnz;
    C->mask = h.P.C_mask;
    C->tile_csr_Ptr = h.P.C_Ptr;
    C->tile_csr_Col = h.P.C_Colb;
    C->tile_csr_Value = h.P.C_Val;
    C->_alloc = (void *)b; // borrowed view into the batch arena
    return TSG_OK;
}

extern "C" int tsg_batch_phase_ms(tsg_batch *b, double *ms)
{
    if (!b || !ms)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    unsigned long long t[8];
    tsg_context *ctx = b->ctx;
    TSG_CUDA(cudaMemcpyAsync(t, b->d_itemoff + 2 * ((size_t)b->count + 1), sizeof(t), cudaMemcpyDeviceToHost,
                             ctx->stream));
    TSG_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int k = 0; k < 7; k++)
        ms[k] = t[k + 1] >= t[k] ? (double)(t[k + 1] - t[k]) * 1e-6 : 0.0;
    return TSG_OK;
}

extern "C" int tsg_batch_info(tsg_batch *b, int *graph, int *grid, size_t *arena_bytes, long long *launches)
{
    if (!b)
        return tsg_set_error(TSG_ERR_INVALID, "null batch");
    if (graph)
        *graph = b->graph_ok;
    if (grid)
        *grid = b->grid;
    if (arena_bytes)
        *arena_bytes = b->arena_bytes;
    if (launches)
        *launches = b->launches;
    return TSG_OK;
}

extern "C" int tsg_batch_destroy(tsg_batch *b)
{
    if (!b)
        return TSG_OK;
    tsg_context *ctx = b->ctx;
    cudaStreamSynchronize(ctx->stream);
    if (b->graph_ok)
    {
        cudaGraphExecDestroy(b->exec);
        cudaGraphDestroy(b->graph);
    }
    tsg_release(ctx, b->d_prod);
    tsg_release(ctx, b->d_rowoff);
    tsg_release(ctx, b->d_itemoff);
    tsg_release(ctx, b->d_bar);
    tsg_release(ctx, b->d_err);
    tsg_release(ctx, b->d_bins);
    tsg_release(ctx, b->d_s1off);
    tsg_release(ctx, b->d_denseoff);
    tsg_release(ctx, b->d_winoff);
    tsg_release(ctx, b->d_wlist);
    tsg_release(ctx, b->d_hlist);
    tsg_release(ctx, b->win_tables);
    char *a = (char *)b->arena;
    tsg_release(ctx, a);
    delete b;
    return TSG_OK;
}
