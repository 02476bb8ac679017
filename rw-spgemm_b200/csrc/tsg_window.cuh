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
//    lanes of one batch that meet the same column add one after another in
//    lane order, batches follow one another behind warp barriers;
//  - the values leave through C's masks, which hold exactly the columns that
//    were written; what is read is cleared for the next task.
// Warps claim WIN_ROWS rows of a (tile row, window) at a time from a device
// counter, one claim ahead.
//
// Bound: the latency of B's entries from L2 and the shared-memory
// read-modify-write, hidden by as many warps as their accumulators fit.
// On a B200, k_step3_spa<flat> before: R-MAT 16 (402 M products) 14.9 -> 5.8 ms,
// R-MAT 14 (53 M) 3.70 -> 1.10 ms, a band of 65 times 8,192 random rows (4.2 M)
// 0.169 -> 0.147 ms.
#pragma once

#include "tsg_device.cuh"

#ifndef WIN_COLS
#define WIN_COLS 1024
#endif
#ifndef WIN_PART_BITS
#define WIN_PART_BITS 8
#endif
#ifndef WIN_HEAVY
#define WIN_HEAVY 512 // A entries that make a row heavy
#endif
#ifndef WIN_ROWS
#define WIN_ROWS 4 // rows per claim
#endif
#ifndef WIN_CTAS
#define WIN_CTAS 3
#endif
#define WIN_TILES (WIN_COLS / TSG_BS)
#define WIN_PART (1 << WIN_PART_BITS) // columns of a task of a heavy row
#define WIN_PARTS (WIN_COLS / WIN_PART)
#define WIN_WARPS 8
#define WIN_THREADS (WIN_WARPS * 32)
// a product takes the windows when C holds at least this many values per (row, window)
#define WIN_MIN_VALUES 8
#define WIN_TABLE_WORDS (1LL << 26) // most words of the table of B's row pointers

struct WinTask
{
    double acc[WIN_COLS]; // all zero between tasks
    double a[32];         // staged A entries of the group: value,
    int b[32];            // B index less the entry's first product,
    int end[32];          // and the product after its last
};

// Where the windows of a product lie.
struct WinPlan
{
    const int *A_rptr, *A_rcol; // A's row view
    const double *A_rval;
    int *btab;          // [B row][blocks + 1]: B's row pointer at every block of 1 << bits columns
    int *ctab;          // [tile row][windows + 1]: first C tile of every window
    int *heavy;         // heavy rows of A
    unsigned *count;    // [0] claims, [1] heavy rows
    int blocks, bits, windows;
    int mA;
};

// an A entry's value and its part of B's row inside columns [c0, c1)
struct WinEntry
{
    double a;
    int b0, len;
};

__device__ __forceinline__ WinEntry win_entry(const ProdView &P, const WinPlan &Q, int x, int e1, int c0, int c1)
{
    WinEntry E = {0.0, 0, 0};
    if (x < e1)
    {
        const int *t = Q.btab + (long long)Q.A_rcol[x] * (Q.blocks + 1);
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

// C row r of tile row I, columns [c0, c1); its A entries are [e0, e1) of the
// row view, its C tiles [t0, t1).  All lanes of the warp call it.
__device__ __forceinline__ void win_task(const ProdView &P, const WinPlan &Q, WinTask &S, int I, int r, int c0, int c1,
                                         int e0, int e1, int t0, int t1, int lane)
{
    const unsigned upto = 0xffffffffu >> (31 - lane); // lanes up to this one
    bool any = false;
    WinEntry nxt = win_entry(P, Q, e0 + lane, e1, c0, c1);
    for (int g = e0; g < e1; g += 32)
    {
        const WinEntry E = nxt;
        if (g + 32 < e1)
            nxt = win_entry(P, Q, g + 32 + lane, e1, c0, c1);
        const int len = E.len;
        const unsigned full = __ballot_sync(TSG_FULL_MASK, len > 0);
        if (!full)
            continue;
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
        __syncwarp();
        // batches of 32 products, the next two batches' loads issued before
        // this pair's additions.  one: the batch holds one entry's products
        int cur = 0, until = S.end[0]; // the entry at the last loaded batch's end, and its end
        auto load = [&](int ib, bool &one, int &col, double &p) {
            one = true;
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
                e = before + __popc(starts & upto);
                one = starts == 0u;
                cur = before + __popc(starts);
                until = S.end[cur];
            }
            if (item < total)
            {
                const int bi = S.b[e] + item;
                col = P.B_rcol[bi] - c0;
                p = __dmul_rn(S.a[e], P.B_rval[bi]);
            }
        };
        auto add = [&](bool one, int col, double p) {
            if (one) // distinct columns
            {
                if (col >= 0)
                    S.acc[col] = __dadd_rn(S.acc[col], p);
            }
            else
            {
                const unsigned same = __match_any_sync(TSG_FULL_MASK, col);
                const int rank = col >= 0 ? __popc(same & upto) - 1 : 0;
                const int last = __reduce_max_sync(TSG_FULL_MASK, rank);
                for (int q = 0; q <= last; q++)
                {
                    if (q)
                        __syncwarp();
                    if (col >= 0 && rank == q)
                        S.acc[col] = __dadd_rn(S.acc[col], p);
                }
            }
            __syncwarp();
        };
        bool s0, s1;
        int col0, col1;
        double p0, p1;
        load(0, s0, col0, p0);
        load(32, s1, col1, p1);
        for (int ib = 0; ib < total; ib += 64)
        {
            bool n0, n1;
            int ncol0, ncol1;
            double np0, np1;
            load(ib + 64, n0, ncol0, np0);
            load(ib + 96, n1, ncol1, np1);
            add(s0, col0, p0);
            if (ib + 32 < total)
                add(s1, col1, p1);
            s0 = n0;
            s1 = n1;
            col0 = ncol0;
            col1 = ncol1;
            p0 = np0;
            p1 = np1;
        }
    }
    if (!any)
        return;
    for (int t = t0 + lane; t < t1; t += 32)
    {
        const int base = P.C_col[t] * TSG_BS - c0;
        const long long tt = (long long)t * TSG_BS + r;
        unsigned mk = P.C_mask[tt];
        if (!mk || base < 0 || base >= c1 - c0)
            continue;
        int q = P.C_tnnz[t] + P.C_Ptr[tt];
        double *acc = S.acc + base;
        do
        {
            const int bit = 31 - __clz(mk);
            mk ^= 1u << bit;
            P.C_Val[q] = acc[15 - bit];
            acc[15 - bit] = 0.0;
            P.C_Colb[q] = (unsigned char)(15 - bit);
            q++;
        } while (mk);
    }
    __syncwarp();
}
