// Steps 1 and 2 for C tile rows with many tiles, a CTA per tile row.
//
// Restates the tile structure (step 1, src/tilespgemm-cuda.h:257-369) and the
// per-tile symbolic masks (step 2, :371-755) of the reference's tilespgemm()
// for tile rows whose work a warp cannot share out: R-MAT hub rows, random
// rows reaching most tile columns.
#pragma once

#include <stddef.h>

#include "tsg_device.cuh"

// ---------------------------------------------------------------------------
// Step 1, count pass.  The (A tile, B tile) pairs of the tile row are split
// evenly over the CTA's warps, each pair setting its tile column's bit in a
// shared-memory bitmap over the row's column window; most pairs of a wide row
// meet a bit already set, which a load tells cheaper than an atomic.  The
// bitmap words are kept (`words`, see StepOneBits) for the emit pass.
// ---------------------------------------------------------------------------
#define S1C_WORDS 2048
// A CTA per tile row from this many tile pairs per row (mean tiles per row of
// A times B's).  Step 1 by warps and by CTAs, random rows: 262,144 rows, 256 pairs
// 0.250 and 0.264 ms, 502 0.326 and 0.339, 1,024 0.423 and 0.417; 32,768 rows, 125
// 0.073 and 0.075, 502 0.071 and 0.058; 64^3 stencil (484) 0.384 and 0.411.
#define S1_CTA_PAIRS 512
// a row's words are kept up to this many (16,384 tile columns)
#define S1_KEEP_WORDS 512

static inline bool step1_by_cta(const tsg_tiled *A, const tsg_tiled *B)
{
    return A->tilem > 0 && B->tilem > 0 &&
           (long long)(A->numtile / A->tilem) * (B->numtile / B->tilem) >= S1_CTA_PAIRS;
}

template <int NT>
struct S1cSmem
{
    unsigned bm[S1C_WORDS];
    int b0[NT];      // per A tile of the chunk: its B tile row's first tile less its first pair ...
    int off[NT + 1]; // ... and its first pair
    int wsum[NT / 32];
    int lo, hi, cnt;
};

// exclusive prefix over the CTA's threads (NW warps) of v, and the total
template <int NW>
__device__ __forceinline__ int cta_excl_scan(int v, int *wsum, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
    {
        const int o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
        if (lane >= d)
            incl += o;
    }
    if (lane == 31)
        wsum[warp] = incl;
    __syncthreads();
    const int x = lane < NW ? wsum[lane] : 0;
    total = __reduce_add_sync(TSG_FULL_MASK, x);
    const int base = __reduce_add_sync(TSG_FULL_MASK, lane < warp ? x : 0);
    __syncthreads();
    return base + incl - v;
}

// the last of off[0..n) at or before x (off ascending, off[0] <= x)
__device__ __forceinline__ int last_at_or_before(const int *off, int n, int x)
{
    int lo = 0, hi = n - 1;
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

// C tiles of tile row i, counted by the CTA (NT threads); thread 0 gets the count
template <int NT>
__device__ __forceinline__ int step1_row_cta(const ProdView &P, int i, S1cSmem<NT> &S, const StepOneBits &K,
                                             unsigned long long *pairs)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a0 = P.A_ptr[i], a1 = P.A_ptr[i + 1];
    if (tid == 0)
    {
        S.lo = INT_MAX;
        S.hi = -1;
        S.cnt = 0;
    }
    __syncthreads();
    int lo = INT_MAX, hi = -1;
    unsigned long long np = 0;
    for (int pa = a0 + tid; pa < a1; pa += NT)
    {
        const int k = P.A_col[pa];
        const int b0 = P.B_ptr[k], b1 = P.B_ptr[k + 1];
        if (b1 > b0)
        {
            lo = min(lo, P.B_col[b0]);
            hi = max(hi, P.B_col[b1 - 1]);
            np += (unsigned long long)(b1 - b0);
        }
    }
    lo = __reduce_min_sync(TSG_FULL_MASK, lo);
    hi = __reduce_max_sync(TSG_FULL_MASK, hi);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        np += __shfl_xor_sync(TSG_FULL_MASK, np, d);
    if (lane == 0 && hi >= 0)
    {
        atomicMin(&S.lo, lo);
        atomicMax(&S.hi, hi);
        if (np && pairs)
            atomicAdd(pairs, np);
    }
    __syncthreads();
    lo = S.lo;
    hi = S.hi;
    if (hi < 0)
        return 0;
    if (tid == 0)
        step1_widest(K, lo, hi);
    const bool once = hi - (lo & ~31) < S1C_WORDS * 32;
    for (int c0 = lo & ~31; c0 <= hi; c0 += S1C_WORDS * 32)
    {
        const int c1 = min(hi + 1, c0 + S1C_WORDS * 32);
        const int nw = (c1 - c0 + 31) >> 5;
        for (int w = tid; w < nw; w += NT)
            S.bm[w] = 0u;
        for (int g = a0; g < a1; g += NT)
        {
            const int n = min(NT, a1 - g);
            int b0 = 0, len = 0;
            if (tid < n)
            {
                const int k = P.A_col[g + tid];
                b0 = P.B_ptr[k];
                len = P.B_ptr[k + 1] - b0;
            }
            int total;
            const int pre = cta_excl_scan<NT / 32>(len, S.wsum, total);
            S.b0[tid] = b0 - pre;
            S.off[tid] = pre;
            if (tid == n - 1)
                S.off[n] = total;
            __syncthreads();
            const int per = (total + (NT / 32) - 1) / (NT / 32);
            const int w1 = min(total, (warp + 1) * per);
            int item = warp * per + lane;
            if (item < w1)
            {
                int e = last_at_or_before(S.off, n, item);
                for (; item < w1; item += 32)
                {
                    while (S.off[e + 1] <= item)
                        e++;
                    const int j = P.B_col[S.b0[e] + item];
                    if (once || (j >= c0 && j < c1))
                    {
                        unsigned *word = &S.bm[(j - c0) >> 5];
                        const unsigned bit = 1u << ((j - c0) & 31);
                        if (!(*(volatile unsigned *)word & bit))
                            atomicOr(word, bit);
                    }
                }
            }
            __syncthreads();
        }
        int cnt = 0;
        const bool keep = K.words && once && nw <= K.stride;
        for (int w = tid; w < nw; w += NT)
        {
            const unsigned bits = S.bm[w];
            cnt += __popc(bits);
            if (keep)
                K.words[(long long)i * K.stride + w] = bits;
        }
        cnt = __reduce_add_sync(TSG_FULL_MASK, cnt);
        if (lane == 0 && cnt)
            atomicAdd(&S.cnt, cnt);
        if (K.words && tid == 0)
            K.span[i] = make_int2(c0, keep ? nw : 0);
        __syncthreads();
    }
    return S.cnt;
}

// ---------------------------------------------------------------------------
// Step 2 for wide tile rows, through B's row view.  The CTA holds the 16 row
// masks of WD tile columns at a time in shared memory, 32 bytes per tile
// column as C stores them (one pass for up to 98,304 columns of C): A's
// entries are staged a thread each, the B entries they reach split evenly
// over the warps, each setting its column's bit -- an OR, in any order --
// unless it is set already.  A thread per C tile then writes its masks, row
// offsets and count.  A tile row is walked once per WD tile columns, where
// segments of 1,024 tiles walked (and cut B's rows) four times as often at
// 65,536 columns; a hypersparse row is a special case only where its few tiles
// lie in more columns than that.
//
// Bound: instructions of the walk and, for hypersparse rows, the 52 bytes
// written per C tile.  On a B200, with the scan of the counts: R-MAT 16 (402 M
// products) 3.09 -> 1.51 ms, R-MAT 14 (53 M) 1.03 -> 0.295 ms, 65,536 random rows
// (16.4 M C tiles, 4.2 M products) 0.875 -> 0.480 ms.
// ---------------------------------------------------------------------------
#define WIDE_UNROLL 4
#define WIDE_SPARSE 4 // products a C tile up to which a row may take a slot per tile

template <int NT>
struct WideSmem
{
    int bs[NT];      // per staged A entry: its B row's first entry less its first item ...
    int off[NT + 1]; // ... and its first item
    int tile0[NT + 1];
    unsigned char row[NT];
    int wsum[NT / 32];
    int next, ptile;
    unsigned bits[1]; // [tile column][8 words], up to the launch's shared memory
};

template <int NT>
__host__ __device__ constexpr size_t wide_smem(int tiles)
{
    return offsetof(WideSmem<NT>, bits) + (size_t)tiles * 32;
}

// word of rows 2h, 2h + 1 of tile column w: swizzled so that one row's
// entries, and one thread per tile, both spread over the banks
__device__ __forceinline__ int wide_word(int w, int h)
{
    return w * 8 + (h ^ ((w >> 2) & 7));
}

// A wide row is one unit of work, or one for every `split` entries of A in it,
// each a part of its columns: the CTA that took an R-MAT hub row whole would
// finish last.  Every part stages all the row's entries, so rows are split
// only once they are half an SM's share of A (wide_split): R-MAT 14,
// step 2: 0.38 ms unsplit, 0.295 split; a band times random rows 0.062 unsplit,
// 0.103 split from 1,024 entries on.
// Units are listed as (row, part | parts << 16) in
// wide_units_of, wide[tilemA] of them; wide[tilemA + 1] counts the C tiles of
// hypersparse rows.
#define WIDE_PARTS 32

static inline int wide_split(long long nnzA, int num_sms)
{
    const long long share = nnzA / (2 * num_sms);
    return share < 1024 ? 1024 : (int)share;
}

static inline size_t wide_units(int tilem, int nnzA, int split)
{
    return (size_t)tilem + nnzA / split;
}

__device__ __forceinline__ int wide_parts(const ProdView &P, int i, int split)
{
    const int entries = P.A_tnnz[P.A_ptr[i + 1]] - P.A_tnnz[P.A_ptr[i]];
    return min(WIDE_PARTS, 1 + entries / split);
}

__device__ __forceinline__ const int2 *wide_units_of(const ProdView &P, const int *wide)
{
    return reinterpret_cast<const int2 *>(wide + ((P.tilemA + 3) & ~1));
}

__device__ __forceinline__ void wide_list(const ProdView &P, int i, int kind, int split, int *wide)
{
    const int parts = wide_parts(P, i, split);
    int2 *at = const_cast<int2 *>(wide_units_of(P, wide)) + atomicAdd(&wide[P.tilemA], parts);
    for (int q = 0; q < parts; q++)
        at[q] = make_int2(i, q | parts << 16);
    if (kind == 2)
        atomicAdd(&wide[P.tilemA + 1], P.C_ptr[i + 1] - P.C_ptr[i]);
}

// A unit by the CTA (NT threads); span: tile columns the launch's shared
// memory holds; ALL: no row's window is wider.
template <int NT, bool ALL>
__device__ __forceinline__ void step2_wide_row(const ProdView &P, WideSmem<NT> &S, int span, int I, int unit,
                                               int *s_bins)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rs = P.C_ptr[I];
    int rb = rs, re = P.C_ptr[I + 1];
    const int parts = unit >> 16, part = unit & 0xFFFF;
    const bool whole = parts == 1;
    if (!whole)
    {
        // the C tiles of this part of the row's columns: parts of about equal
        // counts of B's tiles (a skewed graph's first columns hold most of its
        // entries)
        const int first = P.C_col[rs], last = P.C_col[re - 1] + 1, n = re - rs;
        const int *bc = P.B_cptr + first;
        const long long all = bc[last - first] - bc[0];
        auto bound = [&](int q) {
            const int c = q == 0 ? 0 : q == parts ? last - first
                                                  : lower_bound_int(bc, last - first, bc[0] + (int)(all * q / parts));
            return rs + lower_bound_int(P.C_col + rs, n, first + c);
        };
        rb = bound(part);
        re = bound(part + 1);
    }
    const bool ptr16 = (reinterpret_cast<unsigned long long>(P.A_Ptr) & 15ULL) == 0;
    const int pa_beg = P.A_ptr[I], pa_end = P.A_ptr[I + 1];
    const int v_beg = P.A_tnnz[pa_beg], v_end = P.A_tnnz[pa_end];
    for (int t0 = rb; t0 < re;)
    {
        const int J0 = P.C_col[t0];
        // a row of few C tiles in more columns than a pass holds: a slot per tile,
        // found among their columns (300,000 rows of one entry, 16 tiles in four
        // passes: 2.46 ms, 0.82 with slots)
        const bool sparse = !ALL && P.C_col[re - 1] - J0 >= span && (re - t0) * 9LL <= span * 8LL &&
                            (v_end - v_beg) * (P.browB + 1LL) <= WIDE_SPARSE * (long long)(re - t0);
        int *cols = reinterpret_cast<int *>(S.bits) + (re - t0) * 8;
        const bool rest = sparse || P.C_col[re - 1] - J0 < span; // this pass reaches the row's end
        const int t1 = rest ? re : t0 + lower_bound_int(P.C_col + t0, re - t0, J0 + span);
        const int J1 = P.C_col[t1 - 1] + 1;
        const bool cut = !whole || !rest || t0 != rb;
        __syncthreads();
        if (sparse)
        {
            for (int q = tid; q < t1 - t0; q += NT)
                cols[q] = P.C_col[t0 + q];
            for (int q = tid; q < (t1 - t0) * 8; q += NT)
                S.bits[q] = 0u;
        }
        else
            for (int q = tid; q < (J1 - J0) * 8; q += NT)
                S.bits[q] = 0u;
        for (int c0 = v_beg; c0 < v_end; c0 += NT)
        {
            const int ne = min(NT, v_end - c0);
            if (tid == 0)
                S.ptile = a_tile_of(P, pa_beg, pa_end, c0);
            __syncthreads();
            const int p0 = S.ptile;
            const int ntl = min(ne, pa_end - p0); // tiles that can hold the chunk's entries
            for (int q = tid; q <= ntl; q += NT)
                S.tile0[q] = P.A_tnnz[p0 + q];
            __syncthreads();
            int b0 = 0, len = 0;
            if (tid < ne)
            {
                int row, k;
                a_entry(P, S.tile0, ntl, p0, ptr16, c0 + tid, row, k);
                b0 = P.B_rptr[k];
                int b1 = P.B_rptr[k + 1];
                if (cut)
                {
                    b0 += lower_bound_int(P.B_rcol + b0, b1 - b0, J0 * TSG_BS);
                    b1 = b0 + lower_bound_int(P.B_rcol + b0, b1 - b0, J1 * TSG_BS);
                }
                len = b1 - b0;
                S.row[tid] = (unsigned char)row;
            }
            int total;
            const int pre = cta_excl_scan<NT / 32>(len, S.wsum, total);
            S.bs[tid] = b0 - pre;
            S.off[tid] = pre;
            if (tid == ne - 1)
                S.off[ne] = total;
            __syncthreads();
            const int per = (total + NT / 32 - 1) / (NT / 32);
            const int w1 = min(total, (warp + 1) * per);
            int item = warp * per + lane;
            if (item < w1)
            {
                // four entries' loads in flight a lane: a hub row's CTA waits
                // on them alone
                int e = last_at_or_before(S.off, ne, item);
                int end = S.off[e + 1], from = S.bs[e], row = S.row[e];
                for (; item < w1; item += 32 * WIDE_UNROLL)
                {
                    int col[WIDE_UNROLL], rw[WIDE_UNROLL];
#pragma unroll
                    for (int u = 0; u < WIDE_UNROLL; u++)
                    {
                        const int it = item + 32 * u;
                        rw[u] = -1;
                        if (it < w1)
                        {
                            if (it >= end)
                            {
                                do
                                    end = S.off[++e + 1];
                                while (it >= end);
                                from = S.bs[e];
                                row = S.row[e];
                            }
                            rw[u] = row;
                            col[u] = P.B_rcol[from + it];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < WIDE_UNROLL; u++)
                        if (rw[u] >= 0)
                        {
                            const int w = sparse ? lower_bound_int(cols, t1 - t0, col[u] >> 4) : (col[u] >> 4) - J0;
                            unsigned *word = &S.bits[wide_word(w, rw[u] >> 1)];
                            const unsigned bit = 0x8000u >> (col[u] & 15) << ((rw[u] & 1) * 16);
                            if (!(*(volatile unsigned *)word & bit))
                                atomicOr(word, bit);
                        }
                }
            }
            __syncthreads();
        }
        __syncthreads();
        for (int tb = t0; tb < t1; tb += NT)
        {
            const int t = tb + tid;
            int run = 0;
            if (t < t1)
            {
                const int w = sparse ? t - t0 : P.C_col[t] - J0;
                unsigned m[8], pk[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int h = 0; h < 8; h++)
                {
                    m[h] = S.bits[wide_word(w, h)];
                    pk[h >> 1] |= (unsigned)run << ((h & 1) * 16);
                    run += __popc(m[h] & 0xFFFFu);
                    pk[h >> 1] |= (unsigned)run << ((h & 1) * 16 + 8);
                    run += __popc(m[h] >> 16);
                }
                uint4 *mk = reinterpret_cast<uint4 *>(P.C_mask + (long long)t * TSG_BS);
                mk[0] = make_uint4(m[0], m[1], m[2], m[3]);
                mk[1] = make_uint4(m[4], m[5], m[6], m[7]);
                *reinterpret_cast<uint4 *>(P.C_Ptr + (long long)t * TSG_BS) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                P.C_tnnz[t] = run;
            }
            const int bin = run > 0 ? nnz_bin(run) : -1;
#pragma unroll
            for (int b = 0; b < 4; b++)
            {
                const int in = __popc(__ballot_sync(TSG_FULL_MASK, bin == b));
                if (in && lane == 0)
                    atomicAdd(&s_bins[b], in);
            }
        }
        t0 = t1;
    }
    __syncthreads();
}
