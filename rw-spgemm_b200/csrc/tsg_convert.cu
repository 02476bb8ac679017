// GPU format conversion: CSR -> 16x16 tiles, the column view of B, the
// column-major (reference B layout) gather, and tiles -> CSR.
//
// CSR -> tiles restates src/csr2tile.h:6-259 (row-major, packed (row<<4)|col
// bytes) and :261-478 (column-major B, plain bytes) of the reference, and
// tiles -> CSR restates src/tile2csr.h:8-137.  Rows must be sorted by
// strictly increasing column (checked by tsg_check_csr): the tile columns of
// one tile row are then the merge of 16 sorted lists, which a half-warp walks
// with one lane per row, so every tile row is converted in one pass with no
// scratch memory and the output comes out already sorted.
#include <limits.h>

#include <algorithm>

#include "tsg_internal.h"

#define HW_MASK(tid) (0xFFFFu << ((tid) & 16))

// Heavy tile rows are listed (heavy[0] of them) and done by a CTA each: the
// half-warp's merge takes one tile after another, a chain of loads as long as the
// tile row.  A CTA takes about 4 us for every HEAVY_SPAN tile columns that the row
// spans, but only three run on an SM at a time, where the half-warps of thousands
// of tile rows hide each other's loads: so a row is heavy from `entries` entries or
// `tiles` tiles on, if it holds `per_pass` entries for every HEAVY_SPAN columns, and
// all three grow with the rounds of CTAs that all rows would take.  Conversion on a
// B200, half-warps and CTAs:
//   8 random entries a row (128 tiles a tile row): 20,000 rows (64 entries a pass)
//     0.18 and 0.10 ms, 50,000 (32) 0.203 and 0.221, 100,000 (18) 0.22 and 0.57
//   40 entries a row over 1 M columns (10 a pass): 64 rows 0.64 and 0.27; 20 entries,
//     20,000 rows (5) 0.37 and 0.88
//   200,000 rows of 41 in 5 tiles 0.26 and 0.33, 50,000 of 61 in 5 0.144 and 0.127;
//     100,000 rows of 30 in 33 tiles 0.151 and 0.210, 1,000 rows of 1,000 in 63 0.69
//     and 0.13; R-MAT 16 of 8 edges a row 3.2 and 0.25
#define HEAVY_SPAN 1024
#define HEAVY_THREADS 256
struct HeavyRule
{
    int entries, tiles, per_pass;
};

static HeavyRule heavy_rule(const tsg_context *ctx, int tilem)
{
    const int rounds = std::max(1, tilem / (3 * ctx->num_sms));
    return HeavyRule{std::max(512, 48 * rounds), std::min(256, std::max(32, 8 * rounds)),
                     std::min(64, std::max(4, 3 * rounds))};
}

// entries a tile row of at least one needs to be heavy; lo: its first tile column,
// lane r of the half-warp holds row r's entries [p, e), or what is left of them
__device__ __forceinline__ int heavy_least(unsigned hmask, const HeavyRule &H, const int *__restrict__ col, int lo, int p,
                                           int e)
{
    const int hi = __reduce_max_sync(hmask, p < e ? col[e - 1] >> 4 : lo);
    return ((hi - lo) / HEAVY_SPAN + 1) * H.per_pass;
}

// ---------------------------------------------------------------------------
// Pass 1: number of non-empty tiles in each tile row (half-warp per row).
// ---------------------------------------------------------------------------
__global__ void k_tile_count(int m, int tilem, const int *__restrict__ rowptr,
                             const int *__restrict__ col, const int *__restrict__ err, HeavyRule H,
                             int *__restrict__ tile_cnt, int *__restrict__ heavy)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int tr = (int)(gid >> 4);
    const int lane = threadIdx.x & 15;
    const unsigned hmask = HW_MASK(threadIdx.x);
    if (tr >= tilem)
        return;
    const int r = tr * TSG_BS + lane;
    int p = 0, e = 0;
    if (r < m && *err == 0) // of malformed input no index is followed
    {
        p = rowptr[r];
        e = rowptr[r + 1];
    }
    const int entries = __reduce_add_sync(hmask, e - p);
    int cur = p < e ? (col[p] >> 4) : INT_MAX;
    const int first = __reduce_min_sync(hmask, cur);
    bool heavy_row = entries >= H.entries && entries >= heavy_least(hmask, H, col, first, p, e);
    int cnt = 0;
    while (!heavy_row)
    {
        const int jm = __reduce_min_sync(hmask, cur);
        if (jm == INT_MAX)
            break;
        if (++cnt == H.tiles + 1 && entries >= heavy_least(hmask, H, col, first, p, e))
        {
            heavy_row = true;
            break;
        }
        if (cur == jm)
        {
            do
            {
                ++p;
            } while (p < e && (col[p] >> 4) == jm);
            cur = p < e ? (col[p] >> 4) : INT_MAX;
        }
    }
    if (lane == 0)
    {
        tile_cnt[tr] = cnt; // of a heavy row k_tile_count_cta's
        if (heavy_row)
            heavy[1 + atomicAdd(&heavy[0], 1)] = tr;
    }
}

// ---------------------------------------------------------------------------
// Pass 2: tile columns, per-row offsets, masks and the in-tile entries.
// ---------------------------------------------------------------------------
__global__ void k_tile_fill(int m, int tilem, const int *__restrict__ rowptr,
                            const int *__restrict__ col, const double *__restrict__ val,
                            const int *__restrict__ tile_ptr, int packed, HeavyRule H,
                            int *__restrict__ tile_columnidx, int *__restrict__ tile_rowidx,
                            int *__restrict__ tile_nnz, unsigned char *__restrict__ tPtr,
                            unsigned char *__restrict__ tCol, double *__restrict__ tVal,
                            unsigned short *__restrict__ tMask)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int tr = (int)(gid >> 4);
    const int lane = threadIdx.x & 15;
    const unsigned hmask = HW_MASK(threadIdx.x);
    if (tr >= tilem)
        return;
    const int r = tr * TSG_BS + lane;
    int p = 0, e = 0;
    if (r < m)
    {
        p = rowptr[r];
        e = rowptr[r + 1];
    }
    const int entries = __reduce_add_sync(hmask, e - p);
    if ((tile_ptr[tr + 1] - tile_ptr[tr] > H.tiles || entries >= H.entries) &&
        entries >= heavy_least(hmask, H, col, __reduce_min_sync(hmask, p < e ? col[p] >> 4 : INT_MAX), p, e))
        return; // by k_tile_fill_cta
    // value offset of the tile row's first tile: the row's first CSR entry
    int run = __shfl_sync(hmask, p, 0, 16);
    int t = tile_ptr[tr];
    int cur = p < e ? (col[p] >> 4) : INT_MAX;
    while (true)
    {
        const int jm = __reduce_min_sync(hmask, cur);
        if (jm == INT_MAX)
            break;
        int c = 0;
        unsigned mk = 0;
        if (cur == jm)
        {
            int q = p;
            int cc;
            while (q < e && ((cc = col[q]) >> 4) == jm)
            {
                mk |= 0x8000u >> (cc & 15);
                q++;
            }
            c = q - p;
        }
        int incl = c;
#pragma unroll
        for (int d = 1; d < 16; d <<= 1)
        {
            int o = __shfl_up_sync(hmask, incl, d, 16);
            if (lane >= d)
                incl += o;
        }
        const int excl = incl - c;
        const int total = __shfl_sync(hmask, incl, 15, 16);
        tPtr[(long long)t * TSG_BS + lane] = (unsigned char)excl;
        tMask[(long long)t * TSG_BS + lane] = (unsigned short)mk;
        if (lane == 0)
        {
            tile_columnidx[t] = jm;
            tile_rowidx[t] = tr;
            tile_nnz[t] = run;
        }
        const int dst = run + excl;
        for (int i = 0; i < c; i++)
        {
            const int cc = col[p + i] & 15;
            tCol[dst + i] = (unsigned char)(packed ? ((lane << 4) | cc) : cc);
            tVal[dst + i] = val[p + i];
        }
        p += c;
        cur = p < e ? (col[p] >> 4) : INT_MAX;
        run += total;
        t++;
    }
    if (tr == tilem - 1 && lane == 0)
        tile_nnz[t] = run; // tile_nnz[numtile] = nnz
}

// exclusive prefix of v over the CTA's HEAVY_THREADS threads, and the total
__device__ __forceinline__ int heavy_scan(int v, int *s_sum, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
    {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d)
            incl += o;
    }
    if (lane == 31)
        s_sum[warp] = incl;
    __syncthreads();
    int off = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < HEAVY_THREADS / 32; w++)
    {
        off += w < warp ? s_sum[w] : 0;
        tot += s_sum[w];
    }
    __syncthreads();
    total = tot;
    return off + incl - v;
}

// first and last tile column of tile row tr (its 16 rows' ends; lanes 0..15)
__device__ __forceinline__ int2 heavy_span(int m, int tr, const int *__restrict__ rowptr, const int *__restrict__ col)
{
    const int r = tr * TSG_BS + (threadIdx.x & 15);
    int lo = INT_MAX, hi = -1;
    if (r < m && rowptr[r] < rowptr[r + 1])
    {
        lo = col[rowptr[r]] >> 4;
        hi = col[rowptr[r + 1] - 1] >> 4;
    }
    return make_int2(__reduce_min_sync(0xffffffffu, lo), __reduce_max_sync(0xffffffffu, hi));
}

// Pass 1 of the listed tile rows: a bitmap of tile columns, HEAVY_WORDS words
// at a time, every entry setting its bit unless it is set.
#define HEAVY_WORDS 2048
__global__ void __launch_bounds__(HEAVY_THREADS)
    k_tile_count_cta(int m, const int *__restrict__ rowptr, const int *__restrict__ col, const int *__restrict__ heavy,
                     int *__restrict__ tile_cnt)
{
    __shared__ unsigned bm[HEAVY_WORDS];
    __shared__ int s_cnt;
    for (int l = blockIdx.x; l < heavy[0]; l += gridDim.x)
    {
        const int tr = heavy[1 + l];
        const int e0 = rowptr[tr * TSG_BS], e1 = rowptr[min(m, tr * TSG_BS + TSG_BS)];
        const int2 span = heavy_span(m, tr, rowptr, col);
        if (threadIdx.x == 0)
            s_cnt = 0;
        for (int c0 = span.x; c0 <= span.y; c0 += HEAVY_WORDS * 32)
        {
            const int words = min(HEAVY_WORDS, ((span.y - c0) >> 5) + 1);
            for (int w = threadIdx.x; w < words; w += HEAVY_THREADS)
                bm[w] = 0u;
            __syncthreads();
            for (int e = e0 + threadIdx.x; e < e1; e += HEAVY_THREADS)
            {
                const int j = (col[e] >> 4) - c0;
                if (j < 0 || j >= words * 32)
                    continue;
                const unsigned bit = 1u << (j & 31);
                if (!(*(volatile unsigned *)&bm[j >> 5] & bit))
                    atomicOr(&bm[j >> 5], bit);
            }
            __syncthreads();
            int c = 0;
            for (int w = threadIdx.x; w < words; w += HEAVY_THREADS)
                c += __popc(bm[w]);
            c = __reduce_add_sync(0xffffffffu, c);
            if ((threadIdx.x & 31) == 0 && c)
                atomicAdd(&s_cnt, c);
            __syncthreads();
        }
        if (threadIdx.x == 0)
            tile_cnt[tr] = s_cnt;
        __syncthreads();
    }
}

// Pass 2 of the listed tile rows, HEAVY_SPAN tile columns at a time: the
// entries set their bits in the tiles' row masks; a thread per tile column
// numbers the tiles there are and writes their structure; the entries again
// find their place: the tile's first value, its row's offset, and the bits of
// the row's mask before their own.  A pass takes its part of every row, the rows
// being in order of columns, and begins at the first column that is left.
struct HeavyFill
{
    unsigned mask[HEAVY_SPAN][9];       // [tile column][two rows a word]; 9: a stride of its own bank
    unsigned char off[HEAVY_SPAN][TSG_BS + 4]; // row offsets in the tile
    int base[HEAVY_SPAN];               // the tile's first value
    int cur[TSG_BS], end[TSG_BS];       // what is left of the rows
    int seg[TSG_BS + 1];                // the pass's entries, row by row
    int sum[HEAVY_THREADS / 32];
};

__global__ void __launch_bounds__(HEAVY_THREADS)
    k_tile_fill_cta(int m, int tilem, const int *__restrict__ rowptr, const int *__restrict__ col,
                    const double *__restrict__ val, const int *__restrict__ tile_ptr, int packed,
                    const int *__restrict__ heavy, int *__restrict__ tile_columnidx, int *__restrict__ tile_rowidx,
                    int *__restrict__ tile_nnz, unsigned char *__restrict__ tPtr, unsigned char *__restrict__ tCol,
                    double *__restrict__ tVal, unsigned short *__restrict__ tMask)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    HeavyFill &S = *reinterpret_cast<HeavyFill *>(s_raw);
    const int tid = threadIdx.x;
    for (int l = blockIdx.x; l < heavy[0]; l += gridDim.x)
    {
        const int tr = heavy[1 + l];
        if (tid < TSG_BS)
        {
            S.cur[tid] = rowptr[min(m, tr * TSG_BS + tid)];
            S.end[tid] = rowptr[min(m, tr * TSG_BS + tid + 1)];
        }
        __syncthreads();
        // the pass's entry x: its row, and its place in the matrix
        auto entry = [&](int x, int &r) {
            r = 0;
#pragma unroll
            for (int h = 8; h > 0; h >>= 1)
                r += S.seg[r + h] <= x ? h : 0;
            return S.cur[r] + x - S.seg[r];
        };
        int t = tile_ptr[tr], v = S.cur[0]; // tiles and values before this pass
        for (;;)
        {
            // every warp for itself: the first column left, and the rows' ends in the pass
            const int row = tid & 15, p = S.cur[row], e = S.end[row];
            const int c0 = __reduce_min_sync(0xffffffffu, p < e ? col[p] >> 4 : INT_MAX);
            if (c0 == INT_MAX)
                break;
            const int c1 = __reduce_max_sync(0xffffffffu, p < e ? col[e - 1] >> 4 : -1);
            const int cols = min(HEAVY_SPAN, c1 - c0 + 1);
            int lo = c1 - c0 < HEAVY_SPAN ? e : p, hi = e; // the first entry past the pass
            while (lo < hi)
            {
                const int mid = (lo + hi) >> 1;
                if ((col[mid] >> 4) - c0 < cols)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            int incl = lo - p;
#pragma unroll
            for (int d = 1; d < TSG_BS; d <<= 1)
            {
                const int o = __shfl_up_sync(0xffffffffu, incl, d, 16);
                if ((tid & 15) >= d)
                    incl += o;
            }
            if (tid < TSG_BS)
                S.seg[tid + 1] = incl;
            if (tid == 0)
                S.seg[0] = 0;
            for (int q = tid; q < cols * 9; q += HEAVY_THREADS)
                (&S.mask[0][0])[q] = 0u;
            __syncthreads();
            const int n = S.seg[TSG_BS];
            for (int x = tid; x < n; x += HEAVY_THREADS)
            {
                int r;
                const int c = col[entry(x, r)], w = (c >> 4) - c0;
                atomicOr(&S.mask[w][r >> 1], 0x8000u >> (c & 15) << ((r & 1) * 16));
            }
            __syncthreads();
            for (int w0 = 0; w0 < cols; w0 += HEAVY_THREADS)
            {
                const int w = w0 + tid;
                unsigned mk[8], pk[4] = {0u, 0u, 0u, 0u};
                int n = 0;
                if (w < cols)
#pragma unroll
                    for (int h = 0; h < 8; h++)
                    {
                        mk[h] = S.mask[w][h];
                        pk[h >> 1] |= (unsigned)n << ((h & 1) * 16);
                        n += __popc(mk[h] & 0xFFFFu);
                        pk[h >> 1] |= (unsigned)n << ((h & 1) * 16 + 8);
                        n += __popc(mk[h] >> 16);
                    }
                int tiles, values;
                const int at = t + heavy_scan(n > 0 ? 1 : 0, S.sum, tiles);
                const int first = v + heavy_scan(n, S.sum, values);
                if (n > 0)
                {
                    S.base[w] = first;
                    unsigned *off = reinterpret_cast<unsigned *>(S.off[w]);
                    unsigned *tm = reinterpret_cast<unsigned *>(tMask + (long long)at * TSG_BS);
                    unsigned *tp = reinterpret_cast<unsigned *>(tPtr + (long long)at * TSG_BS);
#pragma unroll
                    for (int h = 0; h < 8; h++)
                        tm[h] = mk[h];
#pragma unroll
                    for (int h = 0; h < 4; h++)
                        tp[h] = off[h] = pk[h];
                    tile_columnidx[at] = c0 + w;
                    tile_rowidx[at] = tr;
                    tile_nnz[at] = first;
                }
                t += tiles;
                v += values;
            }
            __syncthreads();
            for (int x = tid; x < n; x += HEAVY_THREADS)
            {
                int r;
                const int e = entry(x, r), c = col[e], w = (c >> 4) - c0;
                const unsigned mr = (S.mask[w][r >> 1] >> ((r & 1) * 16)) & 0xFFFFu;
                const int at = S.base[w] + S.off[w][r] + __popc(mr >> (16 - (c & 15)));
                tCol[at] = (unsigned char)(packed ? ((r << 4) | (c & 15)) : (c & 15));
                tVal[at] = val[e];
            }
            __syncthreads();
            if (c1 - c0 < HEAVY_SPAN) // the rows' ends
                break;
            if (tid < TSG_BS)
                S.cur[tid] = lo;
            __syncthreads();
        }
        if (tr == tilem - 1 && tid == 0)
            tile_nnz[t] = v; // tile_nnz[numtile] = nnz
        __syncthreads();
    }
}

int tsg_tiled_alloc_arrays(tsg_context *ctx, tsg_tiled *t, int with_csc)
{
    const size_t T = (size_t)t->numtile;
    TSG_TRY(tsg_alloc(ctx, &t->tile_columnidx, T));
    TSG_TRY(tsg_alloc(ctx, &t->tile_rowidx, T));
    TSG_TRY(tsg_alloc(ctx, &t->tile_nnz, T + 1));
    TSG_TRY(tsg_alloc(ctx, &t->tile_csr_Ptr, T * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &t->mask, T * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &t->tile_csr_Col, (size_t)t->nnz));
    TSG_TRY(tsg_alloc(ctx, &t->tile_csr_Value, (size_t)t->nnz));
    if (with_csc)
    {
        TSG_TRY(tsg_alloc(ctx, &t->csc_tile_ptr, (size_t)t->tilen + 1));
        TSG_TRY(tsg_alloc(ctx, &t->csc_tile_rowidx, T));
        TSG_TRY(tsg_alloc(ctx, &t->csc_tile_pos, T));
    }
    return TSG_OK;
}

static int alloc_row_view(tsg_context *ctx, tsg_tiled *mat)
{
    TSG_TRY(tsg_alloc(ctx, &mat->row_ptr, (size_t)mat->m + 1));
    TSG_TRY(tsg_alloc(ctx, &mat->row_col, (size_t)mat->nnz));
    return tsg_alloc(ctx, &mat->row_val, (size_t)mat->nnz);
}

extern "C" int tsg_csr_to_tiled(tsg_context *ctx, int m, int n, int nnz, const int *d_rowptr,
                                const int *d_colidx, const double *d_val, int flags, tsg_tiled *out)
{
    if (!ctx || !out)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    memset(out, 0, sizeof(*out));
    const int *d_err;
    TSG_TRY(tsg_check_csr_start(ctx, m, n, nnz, d_rowptr, d_colidx, &d_err));
    out->m = m;
    out->n = n;
    out->nnz = nnz;
    out->tilem = (m + TSG_BS - 1) / TSG_BS;
    out->tilen = (n + TSG_BS - 1) / TSG_BS;
    out->col_packed = (flags & TSG_TILED_PACKED_COL) ? 1 : 0;
    const int tilem = out->tilem;
    TSG_TRY(tsg_alloc(ctx, &out->tile_ptr, (size_t)tilem + 1));
    long long T = 0;
    int *heavy = nullptr;
    const HeavyRule H = heavy_rule(ctx, tilem);
    const int most = std::min(tilem, nnz / std::min(H.entries, H.tiles + 1)); // tile rows that can be heavy
    TSG_TRY(tsg_alloc(ctx, &heavy, (size_t)most + 1));
    TSG_CUDA(cudaMemsetAsync(heavy, 0, sizeof(int), ctx->stream));
    if (tilem > 0)
    {
        k_tile_count<<<tsg_blocks((long long)tilem * 16, 256), 256, 0, ctx->stream>>>(
            m, tilem, d_rowptr, d_colidx, d_err, H, out->tile_ptr, heavy);
        TSG_LAUNCH_CHECK();
        if (most > 0)
        {
            k_tile_count_cta<<<std::min(most, ctx->num_sms * 4), HEAVY_THREADS, 0, ctx->stream>>>(m, d_rowptr, d_colidx,
                                                                                               heavy, out->tile_ptr);
            TSG_LAUNCH_CHECK();
        }
        TSG_CUDA(cudaMemcpyAsync(ctx->h_pinned + 3, heavy, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        TSG_TRY(tsg_scan_counts(ctx, out->tile_ptr, out->tile_ptr, tilem, &T));
        const int checked = tsg_check_csr_result(ctx, n);
        if (checked != TSG_OK)
        {
            tsg_release(ctx, heavy);
            tsg_release(ctx, out->tile_ptr);
            memset(out, 0, sizeof(*out));
            return checked;
        }
    }
    else
    {
        TSG_CUDA(cudaMemsetAsync(out->tile_ptr, 0, sizeof(int), ctx->stream));
    }
    out->numtile = (int)T;
    TSG_TRY(tsg_tiled_alloc_arrays(ctx, out, (flags & TSG_TILED_CSC_VIEW) ? 1 : 0));
    if (tilem > 0)
    {
        k_tile_fill<<<tsg_blocks((long long)tilem * 16, 256), 256, 0, ctx->stream>>>(
            m, tilem, d_rowptr, d_colidx, d_val, out->tile_ptr, out->col_packed, H, out->tile_columnidx,
            out->tile_rowidx, out->tile_nnz, out->tile_csr_Ptr, out->tile_csr_Col, out->tile_csr_Value,
            out->mask);
        TSG_LAUNCH_CHECK();
        const int rows = *(const int *)(ctx->h_pinned + 3);
        if (rows > 0)
        {
            const int smem = (int)sizeof(HeavyFill);
            TSG_CUDA(cudaFuncSetAttribute(k_tile_fill_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            k_tile_fill_cta<<<std::min(rows, ctx->num_sms * 3), HEAVY_THREADS, smem, ctx->stream>>>(
                m, tilem, d_rowptr, d_colidx, d_val, out->tile_ptr, out->col_packed, heavy, out->tile_columnidx,
                out->tile_rowidx, out->tile_nnz, out->tile_csr_Ptr, out->tile_csr_Col, out->tile_csr_Value, out->mask);
            TSG_LAUNCH_CHECK();
        }
    }
    else
    {
        TSG_CUDA(cudaMemsetAsync(out->tile_nnz, 0, sizeof(int), ctx->stream));
    }
    tsg_release(ctx, heavy);
    if (flags & TSG_TILED_CSC_VIEW)
    {
        // the row view is the input itself (of a matrix without rows nothing is read)
        TSG_TRY(alloc_row_view(ctx, out));
        if (m > 0)
            TSG_CUDA(cudaMemcpyAsync(out->row_ptr, d_rowptr, ((size_t)m + 1) * sizeof(int), cudaMemcpyDeviceToDevice,
                                     ctx->stream));
        else
            TSG_CUDA(cudaMemsetAsync(out->row_ptr, 0, sizeof(int), ctx->stream));
        if (nnz > 0)
        {
            TSG_CUDA(cudaMemcpyAsync(out->row_col, d_colidx, (size_t)nnz * sizeof(int), cudaMemcpyDeviceToDevice,
                                     ctx->stream));
            TSG_CUDA(cudaMemcpyAsync(out->row_val, d_val, (size_t)nnz * sizeof(double), cudaMemcpyDeviceToDevice,
                                     ctx->stream));
        }
        TSG_TRY(tsg_build_csc_view(ctx, out));
    }
    return TSG_OK;
}

// ---------------------------------------------------------------------------
// Column view: tiles by tile column, ascending by row inside a column:
// csc_tile_ptr / csc_tile_rowidx / csc_tile_pos.  Tiles are counted per column
// (with their transposed masks made in the same pass), dropped into their
// column in any order, and every column is put in order by itself: a warp
// ranks up to CSC_COL tiles by counting, a longer column (an R-MAT hub's) goes
// to a CTA that marks its rows in a bitmap, a tile's place being the number of
// marks before its own.  A radix sort of all tiles took two to three passes
// and as many launches again, whatever the size.  A 256^2 grid's
// matrix, conversion with column view: 0.16 -> 0.107 ms.  The sort stays where
// there are few, long columns, whose tiles wait for one another at the columns'
// counters and for the few CTAs that order them (column view alone, counted and
// sorted: 62,500 tile rows times 4 columns 0.346 and 0.130 ms, times 40 1.03 and
// 0.255, 18,750 times 800, 1,100 tiles a column, 0.232 and 0.154; 1,875 times 40,
// 1,300 a column, 0.064 and 0.067, times 10 0.047 and 0.060).
// ---------------------------------------------------------------------------
#define CSC_SORTED 1024       // mean tiles per tile column from which they are sorted,
#define CSC_SORTED_LEAST 24576 // if there are this many
#define CSC_COL 256
#define CSC_WARPS 8
#define CSC_WORDS 8192 // bitmap words of a pass: 262,144 tile rows
#define CSC_LONG_THREADS 512

// transposed masks (mask_t[t][c] has bit 15-r when mask[t][r] has bit 15-c)
// and, unless hist is null, the tiles of each column
__global__ void k_mask_transpose(int T, const unsigned short *__restrict__ mask, unsigned short *__restrict__ mask_t,
                                 const int *__restrict__ tile_col, int *__restrict__ hist)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = (int)(gid >> 4), c = threadIdx.x & 15;
    if (t >= T)
        return;
    const uint4 *mb = reinterpret_cast<const uint4 *>(mask + (long long)t * TSG_BS);
    const uint4 q0 = mb[0], q1 = mb[1];
    const unsigned w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    unsigned out = 0;
#pragma unroll
    for (int r = 0; r < 16; r++)
    {
        const unsigned row = (r & 1) ? (w[r >> 1] >> 16) : (w[r >> 1] & 0xFFFFu);
        out |= ((row >> (15 - c)) & 1u) << (15 - r);
    }
    mask_t[(long long)t * TSG_BS + c] = (unsigned short)out;
    if (hist && c == 0)
        atomicAdd(&hist[tile_col[t]], 1);
}

// tiles into their columns, in any order; count: zeros
__global__ void k_csc_scatter(int T, const int *__restrict__ tile_col, const int *__restrict__ ptr,
                              int *__restrict__ count, int *__restrict__ any)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < T)
        any[ptr[tile_col[t]] + atomicAdd(&count[tile_col[t]], 1)] = t;
}

// warp per column; columns of more than CSC_COL tiles to longs[1 ...],
// counted in longs[0]
__global__ void __launch_bounds__(CSC_WARPS * 32)
    k_csc_order(int tilen, const int *__restrict__ ptr, const int *__restrict__ any, const int *__restrict__ tile_row,
                int *__restrict__ pos, int *__restrict__ row, int *__restrict__ longs)
{
    __shared__ int s_t[CSC_WARPS][CSC_COL];
    int *ts = s_t[threadIdx.x >> 5];
    const int j = blockIdx.x * CSC_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= tilen)
        return;
    const int p0 = ptr[j], n = ptr[j + 1] - p0;
    if (n > CSC_COL)
    {
        if (lane == 0)
            longs[1 + atomicAdd(&longs[0], 1)] = j;
        return;
    }
    for (int q = lane; q < n; q += 32)
        ts[q] = any[p0 + q];
    __syncwarp();
    for (int q = lane; q < n; q += 32)
    {
        const int t = ts[q];
        int rank = 0;
        for (int o = 0; o < n; o++)
            rank += ts[o] < t ? 1 : 0; // row-major numbers: ascending by row
        pos[p0 + rank] = t;
        row[p0 + rank] = tile_row[t];
    }
}

__global__ void __launch_bounds__(CSC_LONG_THREADS)
    k_csc_order_long(int tilem, const int *__restrict__ ptr, const int *__restrict__ any,
                     const int *__restrict__ tile_row, int *__restrict__ pos, int *__restrict__ row,
                     const int *__restrict__ longs)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    unsigned *bits = reinterpret_cast<unsigned *>(s_raw);        // [CSC_WORDS]
    int *before = reinterpret_cast<int *>(s_raw) + CSC_WORDS;    // marks before each word
    __shared__ int s_sum[CSC_LONG_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int l = blockIdx.x; l < longs[0]; l += gridDim.x)
    {
        const int j = longs[1 + l], p0 = ptr[j], n = ptr[j + 1] - p0;
        int base = p0;
        for (int r0 = 0; r0 < tilem; r0 += CSC_WORDS * 32)
        {
            const int words = min(CSC_WORDS, (tilem - r0 + 31) >> 5);
            for (int w = tid; w < words; w += CSC_LONG_THREADS)
                bits[w] = 0u;
            __syncthreads();
            for (int q = tid; q < n; q += CSC_LONG_THREADS)
            {
                const int r = tile_row[any[p0 + q]] - r0;
                if (r >= 0 && r < words * 32)
                    atomicOr(&bits[r >> 5], 1u << (r & 31));
            }
            __syncthreads();
            int run = 0; // marks of the words before this round's
            for (int w0 = 0; w0 < words; w0 += CSC_LONG_THREADS)
            {
                const int w = w0 + tid;
                const int c = w < words ? __popc(bits[w]) : 0;
                int incl = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1)
                {
                    const int o = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d)
                        incl += o;
                }
                if (lane == 31)
                    s_sum[warp] = incl;
                __syncthreads();
                int off = 0, tot = 0;
                for (int q = 0; q < CSC_LONG_THREADS / 32; q++)
                {
                    off += q < warp ? s_sum[q] : 0;
                    tot += s_sum[q];
                }
                if (w < words)
                    before[w] = run + off + incl - c;
                run += tot;
                __syncthreads();
            }
            for (int q = tid; q < n; q += CSC_LONG_THREADS)
            {
                const int t = any[p0 + q], full = tile_row[t], r = full - r0;
                if (r >= 0 && r < words * 32)
                {
                    const int at = base + before[r >> 5] + __popc(bits[r >> 5] & ((1u << (r & 31)) - 1u));
                    pos[at] = t;
                    row[at] = full;
                }
            }
            base += run;
            __syncthreads();
        }
    }
}

__global__ void k_csc_keys(int T, const int *__restrict__ tile_col, unsigned int *__restrict__ keys,
                           int *__restrict__ vals)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < T)
    {
        keys[t] = (unsigned int)tile_col[t];
        vals[t] = t;
    }
}

// from the sorted keys: every column's first tile, and the tiles' rows
__global__ void k_csc_rows(int T, int tilen, const unsigned int *__restrict__ keys, const int *__restrict__ pos,
                           const int *__restrict__ tile_row, int *__restrict__ ptr, int *__restrict__ row)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= T)
        return;
    row[q] = tile_row[pos[q]];
    const int c = (int)keys[q];
    for (int j = q > 0 ? (int)keys[q - 1] + 1 : 0; j <= c; j++)
        ptr[j] = q;
    if (q == T - 1)
        for (int j = c + 1; j <= tilen; j++)
            ptr[j] = T;
}

static int csc_by_sort(tsg_context *ctx, tsg_tiled *mat)
{
    const int T = mat->numtile;
    unsigned int *keys;
    TSG_TRY(tsg_alloc(ctx, &keys, (size_t)T));
    k_csc_keys<<<tsg_blocks(T, 256), 256, 0, ctx->stream>>>(T, mat->tile_columnidx, keys, mat->csc_tile_pos);
    TSG_LAUNCH_CHECK();
    int bits = 1;
    while ((1LL << bits) < mat->tilen)
        bits++;
    TSG_TRY(tsg_sort_pairs_u32(ctx, keys, mat->csc_tile_pos, T, bits));
    k_csc_rows<<<tsg_blocks(T, 256), 256, 0, ctx->stream>>>(T, mat->tilen, keys, mat->csc_tile_pos, mat->tile_rowidx,
                                                           mat->csc_tile_ptr, mat->csc_tile_rowidx);
    TSG_LAUNCH_CHECK();
    tsg_release(ctx, keys);
    return TSG_OK;
}

int tsg_build_mask_t(tsg_context *ctx, tsg_tiled *mat, int *hist)
{
    const int T = mat->numtile;
    if (!mat->mask_t)
        TSG_TRY(tsg_alloc(ctx, &mat->mask_t, (size_t)T * TSG_BS));
    if (T > 0)
    {
        k_mask_transpose<<<tsg_blocks((long long)T * 16, 256), 256, 0, ctx->stream>>>(T, mat->mask, mat->mask_t,
                                                                                    mat->tile_columnidx, hist);
        TSG_LAUNCH_CHECK();
    }
    return TSG_OK;
}

// Row view (scalar CSR of the matrix), from its tiles.
int tsg_build_row_view(tsg_context *ctx, tsg_tiled *mat)
{
    if (!mat->row_ptr)
        TSG_TRY(alloc_row_view(ctx, mat));
    return tsg_tiled_to_csr(ctx, mat, mat->row_ptr, mat->row_col, mat->row_val);
}

int tsg_build_csc_view(tsg_context *ctx, tsg_tiled *mat)
{
    const int T = mat->numtile, tilen = mat->tilen, tilem = mat->tilem;
    cudaStream_t st = ctx->stream;
    if (!mat->csc_tile_ptr)
    {
        TSG_TRY(tsg_alloc(ctx, &mat->csc_tile_ptr, (size_t)tilen + 1));
        TSG_TRY(tsg_alloc(ctx, &mat->csc_tile_rowidx, (size_t)T));
        TSG_TRY(tsg_alloc(ctx, &mat->csc_tile_pos, (size_t)T));
    }
    TSG_CUDA(cudaMemsetAsync(mat->csc_tile_ptr, 0, ((size_t)tilen + 1) * sizeof(int), st));
    const bool sorted = T >= CSC_SORTED_LEAST && T >= (long long)CSC_SORTED * tilen;
    TSG_TRY(tsg_build_mask_t(ctx, mat, sorted ? nullptr : mat->csc_tile_ptr));
    if (!mat->row_ptr)
        TSG_TRY(tsg_build_row_view(ctx, mat));
    if (T == 0)
        return TSG_OK;
    if (sorted)
        return csc_by_sort(ctx, mat);
    TSG_TRY(tsg_scan_counts(ctx, mat->csc_tile_ptr, mat->csc_tile_ptr, tilen, nullptr));
    int *count, *any, *longs; // count: then longs, cleared together
    const int most = T / CSC_COL;
    TSG_TRY(tsg_alloc(ctx, &count, (size_t)tilen + 1 + most));
    TSG_TRY(tsg_alloc(ctx, &any, (size_t)T));
    longs = count + tilen;
    TSG_CUDA(cudaMemsetAsync(count, 0, ((size_t)tilen + 1) * sizeof(int), st));
    k_csc_scatter<<<tsg_blocks(T, 256), 256, 0, st>>>(T, mat->tile_columnidx, mat->csc_tile_ptr, count, any);
    TSG_LAUNCH_CHECK();
    k_csc_order<<<tsg_blocks(tilen, CSC_WARPS), CSC_WARPS * 32, 0, st>>>(tilen, mat->csc_tile_ptr, any, mat->tile_rowidx,
                                                                       mat->csc_tile_pos, mat->csc_tile_rowidx, longs);
    TSG_LAUNCH_CHECK();
    if (tilem > CSC_COL) // a column holds at most a tile of every row
    {
        const int smem = 2 * CSC_WORDS * (int)sizeof(int);
        TSG_CUDA(cudaFuncSetAttribute(k_csc_order_long, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        const int grid = most < ctx->num_sms * 3 ? most : ctx->num_sms * 3;
        if (grid > 0)
        {
            k_csc_order_long<<<grid, CSC_LONG_THREADS, smem, st>>>(tilem, mat->csc_tile_ptr, any, mat->tile_rowidx,
                                                                  mat->csc_tile_pos, mat->csc_tile_rowidx, longs);
            TSG_LAUNCH_CHECK();
        }
    }
    tsg_release(ctx, count);
    tsg_release(ctx, any);
    return TSG_OK;
}

// ---------------------------------------------------------------------------
// Column-major gather (the reference B layout): tile data reordered by the
// column view, Col bytes unpacked to plain columns.
// ---------------------------------------------------------------------------
__global__ void k_cm_counts(int T, const int *__restrict__ pos, const int *__restrict__ tnnz,
                            int *__restrict__ cnt)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < T; q += gridDim.x * blockDim.x)
    {
        int t = pos ? pos[q] : q;
        cnt[q] = tnnz[t + 1] - tnnz[t];
    }
}

// Half-warp per output tile q.
__global__ void k_cm_gather(int T, const int *__restrict__ pos, const int *__restrict__ tnnz_src,
                            const unsigned char *__restrict__ Ptr_src, const unsigned short *__restrict__ mask_src,
                            const unsigned char *__restrict__ Col_src, const double *__restrict__ Val_src,
                            const int *__restrict__ tnnz_dst, unsigned char *__restrict__ Ptr_dst,
                            unsigned short *__restrict__ mask_dst, unsigned char *__restrict__ Col_dst,
                            double *__restrict__ Val_dst)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = (int)(gid >> 4);
    const int lane = threadIdx.x & 15;
    if (q >= T)
        return;
    const int t = pos ? pos[q] : q;
    Ptr_dst[(long long)q * TSG_BS + lane] = Ptr_src[(long long)t * TSG_BS + lane];
    mask_dst[(long long)q * TSG_BS + lane] = mask_src[(long long)t * TSG_BS + lane];
    const int s = tnnz_src[t], n = tnnz_src[t + 1] - s, d = tnnz_dst[q];
    for (int i = lane; i < n; i += 16)
    {
        Col_dst[d + i] = Col_src[s + i] & 15;
        Val_dst[d + i] = Val_src[s + i];
    }
}

// ---------------------------------------------------------------------------
// Tiles -> CSR (src/tile2csr.h:8-137), one CTA per tile row.  Row r of a tile
// spans [Ptr[r], Ptr[r+1]); the last real row of the tile row ends at the
// tile nnz.  A tile row's values are one range in both layouts, so its 16 row
// offsets are the range's start plus a prefix of the 16 row lengths: no scan
// over the matrix is needed and both passes run in one launch.
//
// Bound: bytes (16 of row offsets, 4 + 4 of value offset and column per tile,
// 9 read and 12 written per value).  Pass 1 reads a tile's 16 row offsets as
// one 16-byte word per thread and adds the byte differences.  Pass 2 takes NT
// tiles at a time: their words go to shared memory, a ballot per row says
// which tiles hold entries of it, and the row's warp walks those tiles only,
// its entries flattened over the lanes: stores are consecutive, loads come
// from runs of a row in a tile, and tiles empty in a row (nearly all of them
// in a hypersparse product) cost one bit.
// Measured on a B200 (before: a half-warp per tile row, its lanes walking a
// row each, between a row-length pass and a scan): C of the 64^3 stencil,
// 31.0 M values in 84 tiles a tile row, 0.874 -> 0.196 ms (3.5 TB/s); of an
// R-MAT 16 graph, 164 M values in 3,075 tiles a row, 10.5 -> 1.47 ms; of
// 65,536 random rows, 4.2 M values in 4,011 tiles a row, 2.67 -> 0.36 ms.
// ---------------------------------------------------------------------------
enum
{
    T2C_BOTH, // rowptr, colidx and val
    T2C_ROWS, // rowptr alone
    T2C_FILL  // colidx and val; rowptr is there
};

__device__ __forceinline__ uint4 t2c_ptr16(const unsigned char *Ptr, int t, bool aligned)
{
    const unsigned char *p = Ptr + (long long)t * TSG_BS;
    if (aligned)
        return *reinterpret_cast<const uint4 *>(p);
    unsigned u[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
        u[q] = p[4 * q] | (p[4 * q + 1] << 8) | (p[4 * q + 2] << 16) | ((unsigned)p[4 * q + 3] << 24);
    return make_uint4(u[0], u[1], u[2], u[3]);
}

// the 16 row lengths of a tile of cnt values, a byte each; rows real rows
__device__ __forceinline__ void t2c_row_lens(uint4 w, int cnt, int rows, unsigned d[4])
{
    const unsigned p[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        const unsigned nxt = (p[q] >> 8) | (q < 3 ? p[q < 3 ? q + 1 : 3] << 24 : (unsigned)cnt << 24);
        d[q] = __vsub4(nxt, p[q]); // a full tile's 256 wraps to 0 and 0 - 240 to 16
    }
    if (rows < TSG_BS) // ragged last tile row
#pragma unroll
        for (int r = 0; r < TSG_BS; r++)
        {
            const int sh = (r & 3) * 8;
            if (r == rows - 1)
                d[r >> 2] = (d[r >> 2] & ~(0xFFu << sh)) | (((unsigned)cnt - ((p[r >> 2] >> sh) & 0xFFu)) & 0xFFu) << sh;
            else if (r >= rows)
                d[r >> 2] &= ~(0xFFu << sh);
        }
}

template <int NT>
struct T2cSmem
{
    uint4 ptr[NT];               // row offsets of the step's tiles
    int base[NT], col[NT];       // first value, first column
    unsigned short cnt[NT];      // values
    unsigned bits[TSG_BS][NT / 32]; // per row: tiles holding entries of it
    unsigned short list[TSG_BS][NT]; // those tiles, in order
    int len[TSG_BS], off[TSG_BS];    // row lengths; next output position of each row
};

// tile row tr, by the CTA (NT threads)
template <int NT, int MODE>
__device__ __forceinline__ void t2c_row(T2cSmem<NT> &S, int tr, int m, int tilem, const int *__restrict__ tile_ptr,
                                        const int *__restrict__ tile_col, const int *__restrict__ tnnz,
                                        const unsigned char *__restrict__ Ptr, const unsigned char *__restrict__ Col,
                                        const double *__restrict__ Val, int *__restrict__ rowptr, int *__restrict__ ccol,
                                        double *__restrict__ cval, int colmask)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = tr == tilem - 1 ? m - (tilem - 1) * TSG_BS : TSG_BS;
    const int t0 = tile_ptr[tr], t1 = tile_ptr[tr + 1];
    const bool aligned = ((uintptr_t)Ptr & 15) == 0;
    if (MODE != T2C_FILL)
    {
        if (tid < TSG_BS)
            S.len[tid] = 0;
        __syncthreads();
        // 16-bit sums of the byte lengths, emptied into S.len before they can
        // overflow (2048 tiles of at most 16)
        unsigned lo[4] = {0u, 0u, 0u, 0u}, hi[4] = {0u, 0u, 0u, 0u};
        int held = 0;
        auto drain = [&]() {
#pragma unroll
            for (int r = 0; r < TSG_BS; r++)
            {
                const unsigned v = ((r & 1 ? hi[r >> 2] : lo[r >> 2]) >> ((r & 2) * 8)) & 0xFFFFu;
                const unsigned sum = __reduce_add_sync(0xffffffffu, v);
                if (lane == r && sum)
                    atomicAdd(&S.len[r], (int)sum);
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                lo[q] = hi[q] = 0u;
        };
        for (int tb = t0; tb < t1; tb += NT)
        {
            const int t = tb + tid;
            if (t < t1)
            {
                unsigned d[4];
                t2c_row_lens(t2c_ptr16(Ptr, t, aligned), tnnz[t + 1] - tnnz[t], rows, d);
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    lo[q] += d[q] & 0x00FF00FFu;
                    hi[q] += (d[q] >> 8) & 0x00FF00FFu;
                }
            }
            if (++held == 2048)
            {
                drain();
                held = 0;
            }
        }
        if (t0 + warp * 32 < t1) // a warp that saw a tile
            drain();
        __syncthreads();
        if (tid < 32)
        {
            const int n = lane < TSG_BS ? S.len[lane] : 0;
            int incl = n;
#pragma unroll
            for (int d = 1; d < TSG_BS; d <<= 1)
            {
                const int o = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d)
                    incl += o;
            }
            const int at = tnnz[t0] + incl - n;
            if (lane < TSG_BS)
                S.off[lane] = at;
            if (lane < rows)
                rowptr[tr * TSG_BS + lane] = at;
            if (tr == tilem - 1 && lane == rows - 1)
                rowptr[m] = at + n;
        }
    }
    else if (tid < rows)
        S.off[tid] = rowptr[tr * TSG_BS + tid];
    if (MODE == T2C_ROWS)
        return;
    const unsigned char *pb = reinterpret_cast<const unsigned char *>(S.ptr);
    for (int tb = t0; tb < t1; tb += NT)
    {
        const int t = tb + tid;
        unsigned ne = 0; // rows the tile holds entries of
        if (t < t1)
        {
            const uint4 w = t2c_ptr16(Ptr, t, aligned);
            const int c0 = tnnz[t], cnt = tnnz[t + 1] - c0;
            unsigned d[4];
            t2c_row_lens(w, cnt, rows, d);
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                // 0xFF per non-zero byte -> 4 bits
                const unsigned f = __vcmpne4(d[q], 0u) & 0x08040201u;
                ne |= ((f | (f >> 8) | (f >> 16) | (f >> 24)) & 15u) << (4 * q);
            }
            S.ptr[tid] = w;
            S.base[tid] = c0;
            S.cnt[tid] = (unsigned short)cnt;
            S.col[tid] = tile_col[t] * TSG_BS;
        }
        unsigned mine = 0;
#pragma unroll
        for (int r = 0; r < TSG_BS; r++)
        {
            const unsigned b = __ballot_sync(0xffffffffu, (ne >> r) & 1u);
            if (lane == r)
                mine = b;
        }
        if (lane < TSG_BS)
            S.bits[lane][warp] = mine;
        __syncthreads();
        for (int r = warp; r < rows; r += NT / 32)
        {
            // the row's tiles of this step, listed
            unsigned word = lane < NT / 32 ? S.bits[r][lane] : 0u;
            const int c = __popc(word);
            int incl = c;
#pragma unroll
            for (int d = 1; d < NT / 32; d <<= 1)
            {
                const int o = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d)
                    incl += o;
            }
            const int listed = __shfl_sync(0xffffffffu, incl, NT / 32 - 1);
            for (int at = incl - c; word; word &= word - 1)
                S.list[r][at++] = (unsigned short)(lane * 32 + __ffs(word) - 1);
            __syncwarp();
            int off = S.off[r];
            for (int q0 = 0; q0 < listed; q0 += 32)
            {
                const int nv = min(32, listed - q0);
                int src = 0, cb = 0, len = 0;
                if (lane < nv)
                {
                    const int i = S.list[r][q0 + lane];
                    const int s = pb[i * TSG_BS + r];
                    len = (r == rows - 1 ? S.cnt[i] : pb[i * TSG_BS + r + 1]) - s;
                    src = S.base[i] + s;
                    cb = S.col[i];
                }
                int upto = len;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1)
                {
                    const int o = __shfl_up_sync(0xffffffffu, upto, d);
                    if (lane >= d)
                        upto += o;
                }
                const int n = __shfl_sync(0xffffffffu, upto, 31);
                if (n == nv) // one entry per tile
                {
                    if (lane < nv)
                    {
                        ccol[off + lane] = cb + (Col[src] & colmask);
                        cval[off + lane] = Val[src];
                    }
                }
                else
                {
                    const int pre = upto - len;
                    const int from = src - pre;
                    for (int j0 = 0; j0 < n; j0 += 32)
                    {
                        const int j = j0 + lane;
                        int l = 0; // the last listed tile starting at or before entry j
#pragma unroll
                        for (int sz = 16; sz > 0; sz >>= 1)
                        {
                            const int pc = __shfl_sync(0xffffffffu, pre, l + sz);
                            if (l + sz < nv && pc <= j)
                                l += sz;
                        }
                        const int fs = __shfl_sync(0xffffffffu, from, l);
                        const int fc = __shfl_sync(0xffffffffu, cb, l);
                        if (j < n)
                        {
                            ccol[off + j] = fc + (Col[fs + j] & colmask);
                            cval[off + j] = Val[fs + j];
                        }
                    }
                }
                off += n;
            }
            if (lane == 0)
                S.off[r] = off;
        }
        __syncthreads();
    }
}

template <int NT, int MODE>
__global__ void __launch_bounds__(NT, 2048 / NT)
    k_t2c(int m, int tr0, int tilem, const int *__restrict__ tile_ptr, const int *__restrict__ tile_col,
          const int *__restrict__ tnnz, const unsigned char *__restrict__ Ptr, const unsigned char *__restrict__ Col,
          const double *__restrict__ Val, int *__restrict__ rowptr, int *__restrict__ ccol, double *__restrict__ cval, int colmask)
{
    __shared__ T2cSmem<NT> S;
    t2c_row<NT, MODE>(S, tr0 + blockIdx.x, m, tilem, tile_ptr, tile_col, tnnz, Ptr, Col, Val, rowptr, ccol, cval, colmask);
}

// ... and a half-warp per tile row, lane = row, where a tile row holds few values:
// a CTA's barriers and its 16 rows' lists are more than their own work.  A tile
// row of more than T2C_LONG tiles among them is left to the CTA.
#define T2C_HALVES 16 // tile rows of a CTA
#define T2C_LONG 64
template <int MODE>
__global__ void __launch_bounds__(T2C_HALVES * 16)
    k_t2c_few(int m, int tr0, int tr1, int tilem, const int *__restrict__ tile_ptr, const int *__restrict__ tile_col,
              const int *__restrict__ tnnz, const unsigned char *__restrict__ Ptr, const unsigned char *__restrict__ Col,
              const double *__restrict__ Val, int *__restrict__ rowptr, int *__restrict__ ccol, double *__restrict__ cval,
              int colmask)
{
    __shared__ T2cSmem<T2C_HALVES * 16> S;
    const int lane = threadIdx.x & 15;
    const unsigned hmask = HW_MASK(threadIdx.x);
    const int first = tr0 + blockIdx.x * T2C_HALVES, tr = first + (threadIdx.x >> 4);
    const int t0 = tr < tr1 ? tile_ptr[tr] : 0, t1 = tr < tr1 ? tile_ptr[tr + 1] : 0;
    const bool mine = tr < tr1 && t1 - t0 <= T2C_LONG;
    if (mine)
    {
        const int rows = tr == tilem - 1 ? m - (tilem - 1) * TSG_BS : TSG_BS;
        auto start = [&](int t) { return (int)Ptr[(long long)t * TSG_BS + lane]; };
        auto end = [&](int t) {
            return lane == rows - 1 ? tnnz[t + 1] - tnnz[t] : (int)Ptr[(long long)t * TSG_BS + lane + 1];
        };
        int off = 0;
        if (MODE != T2C_FILL)
        {
            int n = 0;
            if (lane < rows)
                for (int t = t0; t < t1; t++)
                    n += end(t) - start(t);
            int incl = n;
#pragma unroll
            for (int d = 1; d < TSG_BS; d <<= 1)
            {
                const int o = __shfl_up_sync(hmask, incl, d, 16);
                if (lane >= d)
                    incl += o;
            }
            off = tnnz[t0] + incl - n;
            if (lane < rows)
                rowptr[tr * TSG_BS + lane] = off;
            if (tr == tilem - 1 && lane == rows - 1)
                rowptr[m] = off + n;
        }
        else if (lane < rows)
            off = rowptr[tr * TSG_BS + lane];
        if (MODE != T2C_ROWS && lane < rows)
            for (int t = t0; t < t1; t++)
            {
                const int base = tnnz[t], cb = tile_col[t] * TSG_BS, e = end(t);
                for (int q = start(t); q < e; q++, off++)
                {
                    ccol[off] = cb + (Col[base + q] & colmask);
                    cval[off] = Val[base + q];
                }
            }
    }
    if (!__syncthreads_or(tr < tr1 && !mine))
        return;
    for (int q = first; q < min(first + T2C_HALVES, tr1); q++)
        if (tile_ptr[q + 1] - tile_ptr[q] > T2C_LONG)
        {
            t2c_row<T2C_HALVES * 16, MODE>(S, q, m, tilem, tile_ptr, tile_col, tnnz, Ptr, Col, Val, rowptr, ccol, cval,
                                           colmask);
            __syncthreads();
        }
}

// Row pointers and / or entries of tile rows [tr0, tr1) of C; nothing is
// allocated.  512 threads for wide tile rows (R-MAT 16, 3,075 tiles a row:
// 1.47 ms, 1.80 with 256, 2.89 with 128; 8,192 rows of 366 tiles: 0.049, 0.052
// and 0.079 ms).  For narrow ones the step's barriers cost more than its width
// gives, so CTAs are small once there are enough of them to fill the GPU (64^3
// stencil, 16,384 rows of 84 tiles: 0.196 ms with 128, 0.224 with 256, 0.297
// with 512; 21^3, 579 rows of 36: 0.0215, 0.0177, 0.0176 ms).  Tile rows of few
// values are a half-warp's (half-warp and CTA: 31,250 tile rows of 48 values 0.017
// and 0.154 ms, 62,500 of 47 0.031 and 0.283, 12,500 of 188 0.037 and 0.079, 6,912 of
// 414 0.041 and 0.051, 3,125 of 496 0.033 and 0.025, of 976 0.060 and 0.032; few
// tile rows: 1,250 of 48 0.011 and 0.018, 625 of 96 0.020 and 0.014, 579 of 394
// 0.018 and 0.015).
#define T2C_WIDE 256       // mean tiles per tile row
#define T2C_FEW 64         // mean values per tile row up to which a tile row is a half-warp's,
#define T2C_FEW_OF_MANY 448 // also with T2C_MANY tile rows,
#define T2C_FEW_TILES 32   // in as many tiles at most (6,250 of 128 in 128: 0.106 and 0.067)
#define T2C_MANY 16        // tile rows per SM that fill it with 128-thread CTAs
template <int MODE>
static int t2c_launch(tsg_context *ctx, const tsg_tiled *C, int tr0, int tr1, int *rowptr, int *colidx, double *val,
                      int colmask = 0xFF)
{
    if (tr1 <= tr0)
        return TSG_OK;
    const unsigned grid = (unsigned)(tr1 - tr0);
    const bool many = tr1 - tr0 >= T2C_MANY * ctx->num_sms;
    if (C->nnz / C->tilem <= (many ? T2C_FEW_OF_MANY : T2C_FEW) && C->numtile / C->tilem <= T2C_FEW_TILES)
    {
        k_t2c_few<MODE><<<tsg_blocks(grid, T2C_HALVES), T2C_HALVES * 16, 0, ctx->stream>>>(
            C->m, tr0, tr1, C->tilem, C->tile_ptr, C->tile_columnidx, C->tile_nnz, C->tile_csr_Ptr, C->tile_csr_Col,
            C->tile_csr_Value, rowptr, colidx, val, colmask);
        TSG_LAUNCH_CHECK();
        return TSG_OK;
    }
    const int nt = C->numtile / C->tilem >= T2C_WIDE ? 512 : many ? 128 : 256;
#define T2C_GO(NT)                                                                                                  \
    k_t2c<NT, MODE><<<grid, NT, 0, ctx->stream>>>(C->m, tr0, C->tilem, C->tile_ptr, C->tile_columnidx, C->tile_nnz, \
                                                  C->tile_csr_Ptr, C->tile_csr_Col, C->tile_csr_Value, rowptr, colidx, val, colmask)
    if (nt == 512)
        T2C_GO(512);
    else if (nt == 256)
        T2C_GO(256);
    else
        T2C_GO(128);
#undef T2C_GO
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

int tsg_t2c_rows(tsg_context *ctx, const tsg_tiled *C, int *rowptr)
{
    return t2c_launch<T2C_ROWS>(ctx, C, 0, C->tilem, rowptr, nullptr, nullptr);
}

int tsg_t2c_fill(tsg_context *ctx, const tsg_tiled *C, int tr0, int tr1, int *rowptr, int *colidx, double *val)
{
    return t2c_launch<T2C_FILL>(ctx, C, tr0, tr1, rowptr, colidx, val);
}

// A matrix's row view; packed column bytes are told apart from the row
int tsg_t2c_view(tsg_context *ctx, const tsg_tiled *M, int *rowptr, int *colidx, double *val)
{
    return t2c_launch<T2C_BOTH>(ctx, M, 0, M->tilem, rowptr, colidx, val, 15);
}

extern "C" int tsg_tiled_to_csr(tsg_context *ctx, const tsg_tiled *C, int *d_rowptr, int *d_colidx,
                                double *d_val)
{
    if (!ctx || !C || !d_rowptr)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    if (C->m == 0)
    {
        TSG_CUDA(cudaMemsetAsync(d_rowptr, 0, sizeof(int), ctx->stream));
        return TSG_OK;
    }
    return t2c_launch<T2C_BOTH>(ctx, C, 0, C->tilem, d_rowptr, d_colidx, d_val);
}

// C's rows that tsg_tiled_to_csr_noalloc takes at most (its documented limit)
#define NOALLOC_MAX_ROWS (4096LL * 8192)

extern "C" int tsg_tiled_to_csr_noalloc(tsg_context *ctx, const tsg_tiled *C, int *d_rowptr, int *d_colidx,
                                        double *d_val)
{
    if (!ctx || !C || !d_rowptr)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    if (C->m < 0 || C->m > NOALLOC_MAX_ROWS)
        return tsg_set_error(TSG_ERR_INVALID,
                             "tsg_tiled_to_csr_noalloc: C has %d rows; without scratch memory at most %lld rows are "
                             "taken (use tsg_tiled_to_csr)",
                             C->m, NOALLOC_MAX_ROWS);
    if (C->nnz > 0 && (!d_colidx || !d_val))
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    return tsg_tiled_to_csr(ctx, C, d_rowptr, d_colidx, d_val);
}

// Column-major download helper used by tsg_tiled_download (tsg_api.cu).
int tsg_gather_colmajor(tsg_context *ctx, const tsg_tiled *src, int *tnnz_cm, unsigned char *Ptr_cm,
                        unsigned short *mask_cm, unsigned char *Col_cm, double *Val_cm)
{
    const int T = src->numtile;
    if (T == 0)
    {
        TSG_CUDA(cudaMemsetAsync(tnnz_cm, 0, sizeof(int), ctx->stream));
        return TSG_OK;
    }
    unsigned grid = tsg_blocks(T, 256);
    k_cm_counts<<<grid, 256, 0, ctx->stream>>>(T, src->csc_tile_pos, src->tile_nnz, tnnz_cm);
    TSG_LAUNCH_CHECK();
    TSG_TRY(tsg_scan_counts(ctx, tnnz_cm, tnnz_cm, T, nullptr));
    k_cm_gather<<<tsg_blocks((long long)T * 16, 256), 256, 0, ctx->stream>>>(
        T, src->csc_tile_pos, src->tile_nnz, src->tile_csr_Ptr, src->mask, src->tile_csr_Col,
        src->tile_csr_Value, tnnz_cm, Ptr_cm, mask_cm, Col_cm, Val_cm);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

// ---------------------------------------------------------------------------
// Column-major tile data (the reference's B layout) -> the library's layout:
// row-major tile data plus the column view (csc_tile_pos[q] = row-major
// index of column-major tile q).
// ---------------------------------------------------------------------------
// warp per tile column: row-major index of every tile of the column
__global__ void k_cm_rowpos(int tilen, const int *__restrict__ cptr, const int *__restrict__ crow,
                            const int *__restrict__ tile_ptr, const int *__restrict__ tile_col, int *__restrict__ pos)
{
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= tilen)
        return;
    const int j = (int)w;
    for (int q = cptr[j] + lane; q < cptr[j + 1]; q += 32)
    {
        const int R = crow[q];
        int lo = tile_ptr[R], n = tile_ptr[R + 1] - lo;
        while (n > 0)
        {
            const int h = n >> 1;
            if (tile_col[lo + h] < j)
            {
                lo += h + 1;
                n -= h + 1;
            }
            else
                n = h;
        }
        pos[q] = lo;
    }
}

__global__ void k_cm_rm_counts(int T, const int *__restrict__ pos, const int *__restrict__ tnnz_cm, int *__restrict__ cnt)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < T; q += gridDim.x * blockDim.x)
        cnt[pos[q]] = tnnz_cm[q + 1] - tnnz_cm[q];
}

// half-warp per column-major tile q, scattered to row-major slot pos[q]
__global__ void k_cm_rm_scatter(int T, const int *__restrict__ pos, const int *__restrict__ tnnz_cm,
                                const unsigned char *__restrict__ Ptr_cm, const unsigned short *__restrict__ mask_cm,
                                const unsigned char *__restrict__ Col_cm, const double *__restrict__ Val_cm,
                                const int *__restrict__ tnnz_rm, unsigned char *__restrict__ Ptr_rm,
                                unsigned short *__restrict__ mask_rm, unsigned char *__restrict__ Col_rm,
                                double *__restrict__ Val_rm)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = (int)(gid >> 4);
    const int lane = threadIdx.x & 15;
    if (q >= T)
        return;
    const int p = pos[q];
    Ptr_rm[(long long)p * TSG_BS + lane] = Ptr_cm[(long long)q * TSG_BS + lane];
    mask_rm[(long long)p * TSG_BS + lane] = mask_cm[(long long)q * TSG_BS + lane];
    const int s = tnnz_cm[q], n = tnnz_cm[q + 1] - s, d = tnnz_rm[p];
    for (int i = lane; i < n; i += 16)
    {
        Col_rm[d + i] = Col_cm[s + i];
        Val_rm[d + i] = Val_cm[s + i];
    }
}

__global__ void k_rowidx_from_ptr(int tilem, const int *__restrict__ tile_ptr, int *__restrict__ rowidx)
{
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= tilem)
        return;
    for (int t = tile_ptr[w] + lane; t < tile_ptr[w + 1]; t += 32)
        rowidx[t] = (int)w;
}

// mat holds column-major data (tile_nnz, Ptr, mask, Col, Value in csc order),
// row-major tile_ptr / tile_columnidx and csc_tile_ptr / csc_tile_rowidx.
int tsg_colmajor_data_to_rowmajor(tsg_context *ctx, tsg_tiled *mat)
{
    const int T = mat->numtile;
    cudaStream_t st = ctx->stream;
    TSG_TRY(tsg_alloc(ctx, &mat->csc_tile_pos, (size_t)T));
    int *tnnz, *rowidx;
    unsigned char *Ptr, *Col;
    unsigned short *mask;
    double *Val;
    TSG_TRY(tsg_alloc(ctx, &tnnz, (size_t)T + 1));
    TSG_TRY(tsg_alloc(ctx, &rowidx, (size_t)T));
    TSG_TRY(tsg_alloc(ctx, &Ptr, (size_t)T * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &mask, (size_t)T * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &Col, (size_t)mat->nnz));
    TSG_TRY(tsg_alloc(ctx, &Val, (size_t)mat->nnz));
    if (T > 0)
    {
        k_cm_rowpos<<<tsg_blocks((long long)mat->tilen * 32, 256), 256, 0, st>>>(
            mat->tilen, mat->csc_tile_ptr, mat->csc_tile_rowidx, mat->tile_ptr, mat->tile_columnidx, mat->csc_tile_pos);
        TSG_LAUNCH_CHECK();
        k_cm_rm_counts<<<tsg_blocks(T, 256), 256, 0, st>>>(T, mat->csc_tile_pos, mat->tile_nnz, tnnz);
        TSG_LAUNCH_CHECK();
        TSG_TRY(tsg_scan_counts(ctx, tnnz, tnnz, T, nullptr));
        k_cm_rm_scatter<<<tsg_blocks((long long)T * 16, 256), 256, 0, st>>>(
            T, mat->csc_tile_pos, mat->tile_nnz, mat->tile_csr_Ptr, mat->mask, mat->tile_csr_Col, mat->tile_csr_Value,
            tnnz, Ptr, mask, Col, Val);
        TSG_LAUNCH_CHECK();
        k_rowidx_from_ptr<<<tsg_blocks((long long)mat->tilem * 32, 256), 256, 0, st>>>(mat->tilem, mat->tile_ptr, rowidx);
        TSG_LAUNCH_CHECK();
    }
    else
        TSG_CUDA(cudaMemsetAsync(tnnz, 0, sizeof(int), st));
    tsg_release(ctx, mat->tile_nnz);
    tsg_release(ctx, mat->tile_rowidx);
    tsg_release(ctx, mat->tile_csr_Ptr);
    tsg_release(ctx, mat->mask);
    tsg_release(ctx, mat->tile_csr_Col);
    tsg_release(ctx, mat->tile_csr_Value);
    mat->tile_nnz = tnnz;
    mat->tile_rowidx = rowidx;
    mat->tile_csr_Ptr = Ptr;
    mat->mask = mask;
    mat->tile_csr_Col = Col;
    mat->tile_csr_Value = Val;
    TSG_TRY(tsg_build_mask_t(ctx, mat, nullptr));
    return tsg_build_row_view(ctx, mat);
}
