// Numeric step (step 3) of the SPA schedule by column windows: a warp
// computes one C row's entries in one window of WIN_COLS columns.
//
// Restates the numeric step of the reference's tilespgemm()
// (src/tilespgemm-cuda.h:1505-2608) as a row Gustavson over the operands' row
// views, in the arithmetic order of the reference's CPU oracle
// (src/spgemm-cpu.h:330): every C entry is 0.0 + p1 + p2 + ... over k
// ascending, multiply and add rounded separately.
//
// For products of unstructured operands (R-MAT graphs, random rows, a band
// times random rows) the rows of one tile row differ by an order of magnitude
// in work, so a CTA that takes a tile row in segments waits at every barrier
// for its heaviest row.  Here nothing is shared between warps:
//  - a warp's accumulator is WIN_COLS doubles in shared memory, indexed by
//    column, so a product finds its slot by a subtraction;
//  - the part of B's row inside the window comes from a table of row pointers
//    at every window (or block of windows) boundary, made once per product,
//    instead of two binary searches per entry;
//  - the products of 32 A entries are flattened over the lanes in k order;
//    a batch's entries, or the lanes that meet the same column, add one after
//    another, batches follow one another behind warp barriers;
//  - the values leave through C's masks, which hold exactly the columns that
//    were written; what is read is cleared for the next task.
// Warps claim WIN_ROWS rows of a (tile row, window) at a time from a device
// counter, one claim ahead.
//
// Bound: instructions, about 200 per batch of 32 products (issue slots 60 %
// busy, shared memory 52 %); the latency of B's entries from L2 is hidden by
// as many warps as their accumulators fit.  On a B200, k_step3_spa<flat>
// before: R-MAT 16 (402 M products) 14.9 -> 5.5 ms, R-MAT 14 (53 M) 3.70 ->
// 0.72 ms, a band of 65 times 8,192 random rows (4.2 M) 0.169 -> 0.136 ms.
#pragma once

#include <algorithm>

#include "tsg_device.cuh"

#define WIN_COLS 1024 // (512: as many warps again, R-MAT 16 no faster)
#define WIN_PART_BITS 8
#define WIN_HEAVY 256 // fewest A entries that make a row heavy
#define WIN_HEAVY_SHARE 2048 // and the share of A's entries
#define WIN_HEAVY_MEANS 4    // and how many mean rows
#define WIN_ROWS 2 // rows per claim
#define WIN_CTAS 3
#define WIN_TILES (WIN_COLS / TSG_BS)
#define WIN_PART (1 << WIN_PART_BITS) // columns of a task of a heavy row
#define WIN_PARTS (WIN_COLS / WIN_PART)
#define WIN_WARPS 8
#define WIN_THREADS (WIN_WARPS * 32)
#define WIN_FEW 3 // values of a tile's row up to which a lane stores its tile's own
#define WIN_ROUNDS 6 // entries after the first that a batch adds entry by entry
// When a product takes the windows (win_worth).  A task costs its entries of A
// and its C tiles whatever the products in the window, the tables cost every row
// of B: C has to hold WIN_MIN_VALUES values (a batch, that knows no values:
// BATCH_WIN_MIN products) per (row, window) and WIN_MIN_TILES tiles per (tile
// row, window), and the tables may take WIN_TABLE_SHARE words per value of C, or
// WIN_TABLE_FREE.  What the windows are for is uneven work -- where C has WIN_SKEW
// times the products that A's entries and B's mean row give -- and A rows of few
// entries, WIN_VISIT_VALUES values of C for each and window: that is all there.
// Elsewhere C has to fill the windows, WIN_EVEN_TILES of 64 tiles or all there
// are -- k_step3_spa walks A's entries once for 256 tiles of C, however far apart
// -- and its tiles have to hold WIN_TILE_VALUES values on average -- below,
// k_step3_spa's hypersparse form keeps up -- or C one value for every entry of A
// and window.  Step 3, k_step3_spa<flat> and windows, B200:
//   uneven: R-MAT 13 2.2 and 0.40 ms, a 64th of R-MAT 16's rows 4.7 and 1.0
//   values a tile: 16,384 random rows of 11 (2) 0.125 and 0.244, 65,536 of 128
//     times 4 (2) 2.0 and 8.0, of 25 (2.4) 3.7 and 4.1, of 32 (4) 7.1 and 4.8;
//     4,096 rows of 256 times 65,536 of 16 (16) 2.6 and 1.3
//   words of table a value: rows of 60 times 100,000 x 40,000 of 12, 4,000 rows
//     (8) 0.53 and 0.35, 1,000 rows (33) 0.199 and 0.169, 256 rows (130) 0.078
//     and 0.124; 64 rows of 64 times 1 M x 16,384 (1,600) 0.067 and 0.25
//   tiles a window: batch of 24^3 grids (3) 0.35 and 0.51; a band of 129 times
//     random rows of 8, 65,536 rows (18) 3.2 and 7.5, 32,768 (31) 1.5 and 2.1, of 65
//     16,384 rows (36) 0.33 and 0.38, 8,192 (50) 0.169 and 0.136
//   values a visit: random rows of 8 times a band, 16,384 rows, 97 wide (6) 0.41
//     and 0.28, 17 (1) 0.19 and 0.20; 32,768, 33 (1) 0.43 and 0.63
#define WIN_MIN_VALUES 8
#define WIN_MIN_TILES 8
#define WIN_EVEN_TILES 38
#define WIN_VISIT_VALUES 2
#define WIN_SKEW 2
#define WIN_TILE_VALUES 3
#define WIN_TABLE_FREE (1LL << 21)
#define WIN_TABLE_SHARE 32
#define WIN_TABLE_WORDS (1LL << 26) // most words of the table of B's row pointers, and twice those of wtab

struct WinTask
{
    double acc[WIN_COLS]; // all zero between tasks
    double a[32];         // staged A entries of the group: value,
    int b[32];            // B index less the entry's first product,
    int end[32];          // and the product after its last; at the end of a task, per C tile of
    int pre[32];          // the row: its column and mask, its value offset and its first value
    unsigned char tag[TSG_TAGS];
};

// Rows of few C tiles (grid matrices, thin bands): a row's 25 products leave
// most of a CTA's 256 threads at its barriers, so a warp takes NAR_ROWS rows as
// above, a batch holding the products of several.  A slot for every tile (of
// NAR_ROWS rows, or fewer rows of more tiles) takes the place of the window,
// found through a table by tile column.  Only the table's entries at C tiles
// are set, and only those are read.
#define NAR_ROWS 4   // rows per claim
#define NAR_TILES 64 // (row, C tile) slots of the accumulator
#define NAR_SPAN 384 // tile columns of the table
// C tiles a tile row has on average, at most, in a product that takes this
// form.  k_step3_spa<flat> and this one on a B200: 10 tiles (64^2 grid) 0.044 and
// 0.024 ms, 12 (512^2) 0.364 and 0.137, 5 (65,536 rows, 3 entries) 0.114 and
// 0.039; 48 (32,768 rows of 17 times one entry a row) 0.074 and 0.088.
#define NAR_MEAN 32
struct NarTask : WinTask
{
    unsigned char map[NAR_SPAN]; // tile column less the first -> C tile
};
static_assert(NAR_TILES * TSG_BS == WIN_COLS, "slots of a task");

// Where the windows of a product lie.
struct WinPlan
{
    const int *A_rptr, *A_rcol; // A's row view
    const double *A_rval;
    int2 *wtab;         // [B row][windows]: the row's entries in the window (null: B too large, btab)
    int *btab;          // [B row][blocks + 1]: B's row pointer at every block of 1 << bits columns
    int *ctab;          // [tile row][windows + 1]: first C tile of every window
    int *heavy;         // heavy rows of A
    unsigned *claim, *nheavy; // counters: claims, heavy rows
    int blocks, bits, windows;
    int mA;
    int heavy_min;      // A entries that make a row heavy (win_heavy)
};

// A row is heavy when it would hold up the others: a task of 256 columns
// meets shorter parts of B's rows, so only then is it worth cutting.  R-MAT 14
// (228 K entries of A): 0.72 ms from 256 entries on, 0.81 from 512; R-MAT 16
// (955 K): 5.99 and 5.52 ms.  Rows of about the same length hold up none: 1,024
// rows of 256 entries times 65,536 of 16, 1.10 ms as heavy rows, 0.45 as others.
static inline int win_heavy(long long nnzA, long long rows)
{
    long long least = nnzA / WIN_HEAVY_SHARE;
    if (least < WIN_HEAVY)
        least = WIN_HEAVY;
    const long long mean = nnzA / (rows > 0 ? rows : 1);
    return (int)(least < WIN_HEAVY_MEANS * mean ? WIN_HEAVY_MEANS * mean : least);
}

// values: nnz(C), or a bound of it; products: the products of A's entries with
// B's mean row; tables: words of the tables
static inline bool win_worth(long long values, long long products, long long nnzA, long long tilesC, long long tile_rows,
                             long long tilen, long long windows, long long tables)
{
    const auto fills = [&](long long tiles) { return tilesC >= std::min(tiles * windows, tilen) * tile_rows; };
    if (!fills(WIN_MIN_TILES) || (tables > WIN_TABLE_FREE && tables > WIN_TABLE_SHARE * values))
        return false;
    const long long visits = nnzA * windows;
    return values >= WIN_SKEW * products || values >= WIN_VISIT_VALUES * visits ||
           (fills(WIN_EVEN_TILES) && (values >= WIN_TILE_VALUES * tilesC || values >= visits));
}

// B row w's entry offset at every block boundary, by a warp
__device__ __forceinline__ void win_btab_row(int w, const int *__restrict__ rptr, const int *__restrict__ rcol,
                                             int blocks, int bits, int *__restrict__ tab, int windows,
                                             int2 *__restrict__ wtab)
{
    const int lane = threadIdx.x & 31;
    const int e0 = rptr[w], e1 = rptr[w + 1];
    int *t = tab + (long long)w * (blocks + 1);
    // entry e opens the blocks after the previous entry's up to its own
    for (int e = e0 + lane; e <= e1; e += 32)
    {
        const int prev = e > e0 ? rcol[e - 1] >> bits : -1;
        const int cur = e < e1 ? rcol[e] >> bits : blocks;
        for (int b = prev + 1; b <= cur; b++)
            t[b] = e;
        if (wtab)
        {
            // ... and ends the window before it, which the entry before it was in
            int2 *u = wtab + (long long)w * windows;
            const int pw = e > e0 ? rcol[e - 1] / WIN_COLS : -1, cw = e < e1 ? rcol[e] / WIN_COLS : windows;
            if (pw >= 0 && cw > pw)
                u[pw].y = e;
            for (int b = pw + 1; b < cw; b++)
                u[b] = make_int2(e, e);
            if (cw > pw && cw < windows)
                u[cw].x = e;
        }
    }
}

// entry g of ctab, (tile row, window boundary): the first C tile at or after it
__device__ __forceinline__ void win_ctab_entry(const ProdView &P, const WinPlan &Q, long long g)
{
    const int I = (int)(g / (Q.windows + 1)), w = (int)(g % (Q.windows + 1));
    const int c0 = P.C_ptr[I], c1 = P.C_ptr[I + 1];
    Q.ctab[g] = c0 + lower_bound_int(P.C_col + c0, c1 - c0, w * WIN_TILES);
}

// The table's shape for m x n rows of B and at most `words` of table; false
// when even one block per row is too many.
static inline bool win_table(int mB, int nB, long long words, int &bits, int &blocks)
{
    for (bits = WIN_PART_BITS;; bits++)
    {
        blocks = ((nB - 1) >> bits) + 1;
        if ((blocks + 1LL) * mB <= words)
            return true;
        if (blocks == 1)
            return false;
    }
}

// an A entry's value and its part of B's row inside columns [c0, c1)
struct WinEntry
{
    double a;
    int b0, len;
};

// What a task covers: a part of a heavy row, a row's window, or whole rows
// with a slot per C tile (NarTask).
enum
{
    WIN_HEAVY_PART,
    WIN_WINDOW,
    WIN_WHOLE_ROWS
};

// entry x (none when x >= e1), column k of A
template <int FORM>
__device__ __forceinline__ WinEntry win_entry(const ProdView &P, const WinPlan &Q, int x, int e1, int k, int c0, int c1)
{
    WinEntry E = {0.0, 0, 0};
    if (FORM == WIN_WHOLE_ROWS)
    {
        if (x < e1)
        {
            E.a = Q.A_rval[x];
            E.b0 = P.B_rptr[k];
            E.len = P.B_rptr[k + 1] - E.b0;
        }
        return E;
    }
    if (x < e1 && FORM == WIN_WINDOW && Q.wtab)
    {
        const int2 t = Q.wtab[(long long)k * Q.windows + c0 / WIN_COLS];
        E.a = Q.A_rval[x];
        E.b0 = t.x;
        E.len = t.y - t.x;
    }
    else if (x < e1)
    {
        const int *t = Q.btab + (long long)k * (Q.blocks + 1);
        const int blk = c0 >> Q.bits;
        E.a = Q.A_rval[x];
        E.b0 = t[blk];
        E.len = t[min(max((c1 >> Q.bits), blk + 1), Q.blocks)] - E.b0;
        if (c1 - c0 < 1 << Q.bits && E.len > 0) // a block is wider than the window
        {
            const int lo = lower_bound_int(P.B_rcol + E.b0, E.len, c0);
            E.b0 += lo;
            E.len = lower_bound_int(P.B_rcol + E.b0, E.len - lo, c1);
        }
    }
    return E;
}

// column of the n-th entry (from 0) of a row mask, bit 15 - c for column c
__device__ __forceinline__ int win_nth_column(unsigned mask, int n)
{
    int c = 0;
#pragma unroll
    for (int half = 8; half > 0; half >>= 1)
    {
        // the mask's upper `half` of its lowest 2 * half bits
        const int t = __popc(mask >> half);
        const bool low = n >= t;
        n -= low ? t : 0;
        c += low ? half : 0;
        mask = low ? mask & ((1u << half) - 1u) : mask >> half;
    }
    return c;
}

// C row r of tile row I, columns [c0, c1); its A entries are [e0, e1) of the
// row view (E: this lane's of the first 32, loaded by the caller), its C tiles
// [t0, t1), at most 64.  All lanes of the warp call it.
// WIN_WHOLE_ROWS: nr rows from r on, whose entries begin at `ends` of lanes 0
// to nr - 1; c0 the first tile's column and c1 the tile columns to the last;
// nr * (t1 - t0) at most 64.
//
// Loads go ahead of their use, since a warp of short rows would wait on one
// chain of them after another: the entries' columns two groups of 32 ahead,
// their parts of B one group, B's entries two batches, the row's masks and
// value offsets from the start.
template <int FORM, class Task>
__device__ __forceinline__ void win_task(const ProdView &P, const WinPlan &Q, Task &S, int I, int r, int c0, int c1,
                                         int e0, int e1, WinEntry E, int t0, int t1, int lane, int nr = 1, int ends = 0)
{
    const unsigned upto = 0xffffffffu >> (31 - lane); // lanes up to this one
    unsigned mk[2];
    int at[2], base[2];
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const int t = t0 + 32 * h + lane;
        mk[h] = 0u;
        at[h] = base[h] = 0;
        if (FORM == WIN_WHOLE_ROWS)
        {
            const int q = 32 * h + lane, row = q / (t1 - t0);
            if (row < nr)
            {
                const long long w = (long long)(t - row * (t1 - t0)) * TSG_BS + r + row;
                base[h] = q * TSG_BS;
                mk[h] = P.C_mask[w];
                at[h] = P.C_tnnz[t - row * (t1 - t0)] + P.C_Ptr[w];
            }
        }
        else if (t < t1)
        {
            base[h] = P.C_col[t] * TSG_BS - c0;
            mk[h] = P.C_mask[(long long)t * TSG_BS + r];
            at[h] = P.C_tnnz[t] + P.C_Ptr[(long long)t * TSG_BS + r];
        }
    }
    bool any = false;
    int k = e0 + 32 + lane < e1 ? Q.A_rcol[e0 + 32 + lane] : 0;
    for (int g = e0; g < e1; g += 32)
    {
        const WinEntry nxt = win_entry<FORM>(P, Q, g + 32 + lane, e1, k, c0, c1);
        k = g + 64 + lane < e1 ? Q.A_rcol[g + 64 + lane] : 0;
        const int len = E.len;
        const unsigned full = __ballot_sync(TSG_FULL_MASK, len > 0);
        if (!full)
        {
            E = nxt;
            continue;
        }
        any = true;
        int incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const int o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
            if (lane >= d)
                incl += o;
        }
        const int total = __shfl_sync(TSG_FULL_MASK, incl, 31);
        const int pre = incl - len;
        if (len > 0)
        {
            const int at = __popc(full & upto) - 1;
            S.a[at] = E.a;
            S.b[at] = E.b0 - pre;
            S.end[at] = incl;
        }
        if constexpr (FORM == WIN_WHOLE_ROWS)
        {
            // the slots of the entry's row
            int row = 0;
#pragma unroll
            for (int q = 1; q < NAR_ROWS; q++)
                row += g + lane >= __shfl_sync(TSG_FULL_MASK, ends, q) && q < nr ? 1 : 0;
            if (len > 0)
                S.pre[__popc(full & upto) - 1] = row * (t1 - t0) * TSG_BS;
        }
        __syncwarp();
        // batches of 32 products, a batch's loads issued two batches before its
        // additions.  rel: the lane's entry, counted from the batch's
        // first, and the batch's last (<< 8)
        int cur = 0, until = S.end[0]; // the entry at the last loaded batch's end, and its end
        auto load = [&](int ib, int &rel, int &col, double &p) {
            rel = 0;
            col = -1;
            p = 0.0;
            if (ib >= total)
                return;
            const int item = ib + lane;
            int e = cur;
            if (ib + 32 > until && until < total)
            {
                // the lanes at which an entry's products begin, and the
                // entries begun before
                const bool mine = len > 0 && pre > ib && pre < ib + 32;
                const unsigned starts = __reduce_or_sync(TSG_FULL_MASK, mine ? 1u << (pre - ib) : 0u);
                const int before = __popc(__ballot_sync(TSG_FULL_MASK, len > 0 && pre <= ib)) - 1;
                rel = __popc(starts & upto) | __popc(starts) << 8;
                e = before + (rel & 0xFF);
                cur = before + __popc(starts);
                until = S.end[cur];
            }
            if (item < total)
            {
                const int bi = S.b[e] + item;
                if constexpr (FORM == WIN_WHOLE_ROWS)
                {
                    const int c = P.B_rcol[bi], w = (c >> 4) - c0;
                    if ((unsigned)w < (unsigned)c1)
                        col = S.map[w] * TSG_BS + (c & 15) + S.pre[e];
                }
                else
                    col = P.B_rcol[bi] - c0;
                p = __dmul_rn(S.a[e], P.B_rval[bi]);
            }
        };
        // products of one entry meet distinct columns; those of a few entries
        // are added entry by entry, others in lane order where columns meet
        auto add = [&](int rel, int col, double p) {
            int last = rel >> 8, rank = rel & 0xFF;
            if (last > WIN_ROUNDS)
                rank = same_key_rank(col, col >= 0, S.tag, lane, last);
            rank = col >= 0 ? rank : -1;
            double *acc = S.acc + max(col, 0);
            if (rank == 0)
                *acc = __dadd_rn(*acc, p);
            __syncwarp();
            for (int q = 1; q <= last; q++)
            {
                if (rank == q)
                    *acc = __dadd_rn(*acc, p);
                __syncwarp();
            }
        };
        int s0, s1, col0, col1;
        double p0, p1;
        load(0, s0, col0, p0);
        load(32, s1, col1, p1);
        for (int ib = 0; ib < total; ib += 64)
        {
            add(s0, col0, p0);
            load(ib + 64, s0, col0, p0);
            if (ib + 32 < total)
            {
                add(s1, col1, p1);
                load(ib + 96, s1, col1, p1);
            }
        }
        E = nxt;
    }
    if (!any)
        return;
    // the row's values out, 32 tiles at a time, flattened over the lanes:
    // consecutive lanes store consecutive values of a tile's row (a lane per
    // tile would touch a line per value, and read a bank 32 ways)
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const unsigned m = FORM == WIN_WHOLE_ROWS || (base[h] >= 0 && base[h] < c1 - c0) ? mk[h] : 0u; // a heavy row's part holds some of the tiles
        const int len = __popc(m);
        const unsigned full = __ballot_sync(TSG_FULL_MASK, len > 0);
        if (!full)
            continue;
        if (__reduce_max_sync(TSG_FULL_MASK, len) <= WIN_FEW)
        {
            double *acc = S.acc + base[h];
            int q = at[h];
            for (unsigned left = m; left;)
            {
                const int bit = 31 - __clz(left);
                left ^= 1u << bit;
                P.C_Val[q] = acc[15 - bit];
                acc[15 - bit] = 0.0;
                P.C_Colb[q++] = (unsigned char)(15 - bit);
            }
            continue;
        }
        int incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const int o = __shfl_up_sync(TSG_FULL_MASK, incl, d);
            if (lane >= d)
                incl += o;
        }
        const int total = __shfl_sync(TSG_FULL_MASK, incl, 31);
        const int pre = incl - len;
        if (len > 0)
        {
            const int e = __popc(full & upto) - 1;
            S.b[e] = base[h] << 16 | (int)m;
            S.end[e] = at[h] - pre;
            S.pre[e] = pre;
        }
        __syncwarp();
        for (int ib = 0; ib < total; ib += 32)
        {
            const bool mine = len > 0 && pre > ib && pre < ib + 32;
            const unsigned starts = __reduce_or_sync(TSG_FULL_MASK, mine ? 1u << (pre - ib) : 0u);
            const int e = __popc(__ballot_sync(TSG_FULL_MASK, len > 0 && pre <= ib)) - 1 + __popc(starts & upto);
            const int j = ib + lane;
            if (j < total)
            {
                const int w = S.b[e];
                const int c = win_nth_column((unsigned)w & 0xFFFFu, j - S.pre[e]);
                double *acc = S.acc + (w >> 16) + c;
                const int q = S.end[e] + j;
                P.C_Val[q] = *acc;
                *acc = 0.0;
                P.C_Colb[q] = (unsigned char)c;
            }
        }
        __syncwarp();
    }
}
static_assert(WIN_TILES <= 64, "C tiles of a window");

// columns [part * WIN_PART, ...) of heavy row `row`
__device__ __forceinline__ void win_claim_heavy(const ProdView &P, const WinPlan &Q, WinTask &S, int row, int part,
                                                int lane)
{
    const int *ct = Q.ctab + (long long)(row / TSG_BS) * (Q.windows + 1) + part / WIN_PARTS;
    const int e0 = Q.A_rptr[row], e1 = Q.A_rptr[row + 1], c0 = part * WIN_PART, c1 = c0 + WIN_PART;
    const int k = e0 + lane < e1 ? Q.A_rcol[e0 + lane] : 0;
    win_task<WIN_HEAVY_PART>(P, Q, S, row / TSG_BS, row % TSG_BS, c0, c1, e0, e1, win_entry<WIN_HEAVY_PART>(P, Q, e0 + lane, e1, k, c0, c1), ct[0],
             ct[1], lane);
}

// claim c of the tile rows from row0 on: WIN_ROWS rows of a (tile row, window)
#define WIN_PER (TSG_BS / WIN_ROWS) // claims of a (tile row, window)
__device__ __forceinline__ void win_claim_rows(const ProdView &P, const WinPlan &Q, WinTask &S, int row0, unsigned c,
                                               int lane)
{
    const int u = c / WIN_PER;
    const int I = row0 + u / Q.windows, w = u % Q.windows;
    const int r0 = (c % WIN_PER) * WIN_ROWS;
    const int *ct = Q.ctab + (long long)I * (Q.windows + 1) + w;
    const int t0 = ct[0], t1 = ct[1];
    if (t0 == t1)
        return;
    const int row = I * TSG_BS + r0;
    const int c0 = w * WIN_COLS, c1 = c0 + WIN_COLS;
    const int e = lane <= WIN_ROWS ? Q.A_rptr[min(row + lane, Q.mA)] : 0;
    // first entries of the rows: columns two rows ahead, parts of B one
    auto col = [&](int i) {
        const int x0 = __shfl_sync(TSG_FULL_MASK, e, i), x1 = __shfl_sync(TSG_FULL_MASK, e, i + 1);
        return i < WIN_ROWS && x0 + lane < x1 ? Q.A_rcol[x0 + lane] : 0;
    };
    int k1 = col(0);
    int k2 = col(1);
    int e0 = __shfl_sync(TSG_FULL_MASK, e, 0), e1 = __shfl_sync(TSG_FULL_MASK, e, 1);
    WinEntry E = win_entry<WIN_WINDOW>(P, Q, e0 + lane, e1, k1, c0, c1);
#pragma unroll 1
    for (int i = 0; i < WIN_ROWS; i++)
    {
        const int e2 = __shfl_sync(TSG_FULL_MASK, e, min(i + 2, WIN_ROWS));
        const WinEntry nxt = win_entry<WIN_WINDOW>(P, Q, e1 + lane, e2, k2, c0, c1);
        k2 = col(i + 2);
        if (e0 < e1 && e1 - e0 < Q.heavy_min)
            win_task<WIN_WINDOW>(P, Q, S, I, r0 + i, c0, c1, e0, e1, E, t0, t1, lane);
        e0 = e1;
        e1 = e2;
        E = nxt;
    }
}

// claim c of the tile rows from row0 on: NAR_ROWS rows of a tile row.  A wide
// row (kind: the row kinds of the fused step 1/2 pass, or null) is left.
#define NAR_PER (TSG_BS / NAR_ROWS)
__device__ __forceinline__ void nar_claim(const ProdView &P, const WinPlan &Q, NarTask &S, int row0, unsigned c,
                                          const int *__restrict__ kind, int *__restrict__ left, int lane)
{
    const int I = row0 + (int)(c / NAR_PER), r0 = (int)(c % NAR_PER) * NAR_ROWS;
    const int t0 = P.C_ptr[I], t1 = P.C_ptr[I + 1];
    const int ends = Q.A_rptr[min(I * TSG_BS + r0 + min(lane, NAR_ROWS), Q.mA)];
    if (t0 == t1)
        return;
    if (kind ? kind[I] != 0 : t1 - t0 > S12_MAXT)
    {
        if (r0 == 0 && lane == 0)
        {
            left[I] = 1;
            atomicAdd(&left[P.tilemA], 1);
        }
        return;
    }
    const int all0 = __shfl_sync(TSG_FULL_MASK, ends, 0), all1 = __shfl_sync(TSG_FULL_MASK, ends, NAR_ROWS);
    if (all0 == all1)
        return;
    // the first rows' entries and the C tiles at once
    int k = all0 + lane < all1 ? Q.A_rcol[all0 + lane] : 0;
    for (int ta = t0; ta < t1;)
    {
        const int J0 = P.C_col[ta];
        const int j0 = ta + lane < t1 ? P.C_col[ta + lane] - J0 : NAR_SPAN;
        const int j1 = ta + 32 + lane < t1 ? P.C_col[ta + 32 + lane] - J0 : NAR_SPAN;
        const bool in0 = j0 < NAR_SPAN, in1 = j1 < NAR_SPAN;
        const int nt = __popc(__ballot_sync(TSG_FULL_MASK, in0)) + __popc(__ballot_sync(TSG_FULL_MASK, in1));
        const int span = 1 + __reduce_max_sync(TSG_FULL_MASK, in1 ? j1 : in0 ? j0 : 0);
        if (in0)
            S.map[j0] = (unsigned char)lane;
        if (in1)
            S.map[j1] = (unsigned char)(lane + 32);
        __syncwarp();
        const int rows = nt <= NAR_TILES / 4 ? 4 : nt <= NAR_TILES / 2 ? 2 : 1;
#pragma unroll 1
        for (int r = 0; r < NAR_ROWS; r += rows)
        {
            const int e0 = __shfl_sync(TSG_FULL_MASK, ends, r), e1 = __shfl_sync(TSG_FULL_MASK, ends, r + rows);
            const int mine = __shfl_sync(TSG_FULL_MASK, ends, min(r + lane, NAR_ROWS));
            if (r > 0 || ta > t0)
                k = e0 + lane < e1 ? Q.A_rcol[e0 + lane] : 0;
            if (e0 < e1)
                win_task<WIN_WHOLE_ROWS>(P, Q, S, I, r0 + r, J0, span, e0, e1,
                                         win_entry<WIN_WHOLE_ROWS>(P, Q, e0 + lane, e1, k, 0, 0), ta, ta + nt, lane, rows,
                                         mine);
        }
        __syncwarp();
        ta += nt;
    }
}
