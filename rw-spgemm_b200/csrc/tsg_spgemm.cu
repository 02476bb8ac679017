// Tiled SpGEMM C = A*B on 16x16 tiles, FP64, for sm_100a: one product.
//
// The per-item device code lives in tsg_device.cuh (shared with the batched
// persistent kernel of tsg_batch.cu); this file holds the one-product kernels
// and the host orchestration of tsg_spgemm:
//   step 1  count (warp per A tile row) -> scan -> emit sorted C tile columns
//   step 2  masks / row offsets / nnz per C tile -> scan of tile nnz
//   step 3  values and column bytes
// Steps 2 and 3 run in one of two work schedules with bit-identical results:
// the tile schedule (half-warp per C tile, A-row x B-column intersection, as
// the reference decomposes the work) or the row-segment schedule (half-warp
// per run of C tiles in one tile row, tile-level Gustavson, no intersection).
#include <limits.h>
#include <stddef.h>

#include <algorithm>

#include "tsg_device.cuh"
#include "tsg_staged.cuh"
#include "tsg_wide.cuh"
#include "tsg_window.cuh"

#define S1_WARPS 8
#define S1C_THREADS 256
// step 1's bitmaps are kept up to this many words in all
#define S1_KEEP_TOTAL (1LL << 24)
// tile columns of a CTA's shared memory in the wide-row step 2
#define WIDE_SPAN 6144

template <bool EMIT>
__global__ void __launch_bounds__(S1_WARPS * 32) k_step1(ProdView P, int *__restrict__ C_cnt,
                                                         unsigned long long *__restrict__ pairs, StepOneBits K)
{
    __shared__ unsigned int s_bm[S1_WARPS][S1_WORDS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * S1_WARPS + warp;
    if (i >= P.tilemA)
        return;
    const int cnt = step1_row<EMIT>(P, i, s_bm[warp], lane, pairs, K);
    if (!EMIT && lane == 0)
        C_cnt[i] = cnt;
}

// ... and a CTA per tile row (step1_row_cta)
__global__ void __launch_bounds__(S1C_THREADS) k_step1_cta(ProdView P, int *__restrict__ C_cnt,
                                                           unsigned long long *__restrict__ pairs, StepOneBits K)
{
    __shared__ S1cSmem<S1C_THREADS> S;
    const int cnt = step1_row_cta<S1C_THREADS>(P, blockIdx.x, S, K, pairs);
    if (threadIdx.x == 0)
        C_cnt[blockIdx.x] = cnt;
}

// step 1's count pass summed over the block into one device word
__global__ void __launch_bounds__(S1_WARPS * 32) k_step1_total(ProdView P, unsigned long long *__restrict__ total)
{
    __shared__ unsigned int s_bm[S1_WARPS][S1_WORDS];
    __shared__ int s_cnt[S1_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * S1_WARPS + warp;
    const int cnt = i < P.tilemA ? step1_row<false>(P, i, s_bm[warp], lane, nullptr) : 0;
    if (lane == 0)
        s_cnt[warp] = cnt;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long sum = 0;
        for (int w = 0; w < S1_WARPS; w++)
            sum += (unsigned long long)s_cnt[w];
        if (sum)
            atomicAdd(total, sum);
    }
}

// fused step-1 emit + step 2 (warp per A tile row).  Wide rows are emitted
// alone and left to the wide-row step 2: wide[i] says 1, or 2 when the row is
// hypersparse (0 otherwise), and wide[tilemA ...] lists their units (wide_list).
#define S12_WARPS 4
__global__ void __launch_bounds__(S12_WARPS * 32) k_step12(ProdView P, StepOneBits K, int split, int per_pair, int *__restrict__ wide,
                                                int *__restrict__ bins)
{
    __shared__ S12Smem sm[S12_WARPS];
    __shared__ int s_bins[4];
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * S12_WARPS + warp;
    if (i < P.tilemA)
    {
        const int done = step12_row(P, i, sm[warp], lane, s_bins, per_pair, K);
        int kind = 0;
        if (!done)
        {
            static_assert(sizeof(S12Smem) >= S1_WORDS * sizeof(unsigned), "bitmap scratch");
            __syncwarp();
            if (!step1_emit_kept(P, i, lane, K))
                step1_row<true>(P, i, reinterpret_cast<unsigned *>(&sm[warp]), lane, nullptr);
            __syncwarp(); // the row's C columns, emitted by all lanes
            kind = wide_kind(P, i, lane);
        }
        if (lane == 0)
        {
            wide[i] = kind;
            if (kind)
                wide_list(P, i, kind, split, wide);
        }
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
}

// step 2 (tile schedule) for the C tiles of rows k_step12 left to it
__global__ void __launch_bounds__(256) k_step2_wide(ProdView P, const int *__restrict__ wide, int *__restrict__ bins)
{
    __shared__ int s_bins[4];
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    __syncthreads();
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (t < P.numC && wide[P.C_row[t]])
        step2_tile(P, (int)t, TSG_HW_MASK(threadIdx.x), threadIdx.x & 15, s_bins);
    __syncthreads();
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
}

// step 2 of the wide rows k_step12 listed, through B's row view: CTAs take
// rows from a device counter
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_step2_cta(ProdView P, int span, const int *__restrict__ wide,
                                                  unsigned *__restrict__ ctr, int *__restrict__ bins)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    WideSmem<NT> &S = *reinterpret_cast<WideSmem<NT> *>(s_raw);
    __shared__ int s_bins[4];
    const int units = wide[P.tilemA];
    if (units == 0)
        return;
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    for (;;)
    {
        if (threadIdx.x == 0)
            S.next = (int)atomicAdd(ctr, 1u);
        __syncthreads();
        const int q = S.next;
        if (q >= units)
            break;
        const int2 u = wide_units_of(P, wide)[q];
        // with 512 threads the span is the widest row
        step2_wide_row<NT, NT == 512>(P, S, span, u.x, u.y, s_bins);
    }
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
}

__global__ void __launch_bounds__(256) k_step2(ProdView P, int *__restrict__ bins)
{
    __shared__ int s_bins[4];
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    __syncthreads();
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (t < P.numC)
        step2_tile(P, (int)t, TSG_HW_MASK(threadIdx.x), threadIdx.x & 15, s_bins);
    __syncthreads();
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
}

// fewest C tiles of a product that runs its hypersparse rows beside the others
#define HYP_APART (1 << 17)

#define S3_THREADS 128
#define S3_HW (S3_THREADS / 16)

__global__ void __launch_bounds__(S3_THREADS, 4) k_step3(ProdView P)
{
    __shared__ __align__(16) double s_A[S3_HW][S3T_WORDS];
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (t < P.numC)
        step3_tile_cols(P, (int)t, TSG_HW_MASK(threadIdx.x), threadIdx.x & 15, s_A[threadIdx.x >> 4]);
}

#define S3R_THREADS 256

__global__ void __launch_bounds__(S3R_THREADS) k_step3_tile_rows(ProdView P)
{
    __shared__ double s_acc[S3R_THREADS / 16][TSG_BS * S3R_STRIDE];
    const int lane = threadIdx.x & 15;
    const unsigned hmask = TSG_HW_MASK(threadIdx.x);
    double *acc = s_acc[threadIdx.x >> 4];
    step3_tile_clear(acc, hmask, lane);
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (t < P.numC)
        step3_tile_rows(P, (int)t, hmask, lane, acc);
}

__global__ void __launch_bounds__(256) k_step3_elems(ProdView P)
{
    __shared__ int2 s_pairs[8][S3E_PAIRS];
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t < P.numC)
        step3_elems_tile(P, (int)t, s_pairs[threadIdx.x >> 5]);
}

template <int W>
__global__ void __launch_bounds__(128) k_step2_rows(ProdView P, int *__restrict__ bins)
{
    __shared__ S2RowsSmem<W> sm[8];
    __shared__ int s_bins[4];
    if (threadIdx.x < 4)
        s_bins[threadIdx.x] = 0;
    __syncthreads();
    const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    step2_rows_item<W>(P, item, TSG_HW_MASK(threadIdx.x), threadIdx.x & 15, sm[threadIdx.x >> 4], s_bins);
    __syncthreads();
    if (threadIdx.x < 4 && s_bins[threadIdx.x])
        atomicAdd(&bins[threadIdx.x], s_bins[threadIdx.x]);
}

template <int W, int CAP>
__global__ void __launch_bounds__(128) k_step3_rows(ProdView P)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    S3RowsSmem<W, CAP> *sm = reinterpret_cast<S3RowsSmem<W, CAP> *>(s_raw);
    const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    step3_rows_item<W, CAP>(P, item, TSG_HW_MASK(threadIdx.x), threadIdx.x & 15, sm[threadIdx.x >> 4]);
}

// persistent: CTAs take blocks of C tiles from a device counter; kind (may
// be null) marks the hypersparse rows (2), each done whole.  RANGED: only
// the tile rows [row0, row1) are done -- the blocks holding their tiles, each
// clamped to those tiles (a separate instantiation keeps the whole-product
// form's registers).
template <bool FLAT, bool RANGED, int BLK>
__global__ void __launch_bounds__(SPA_THREADS, 3) k_step3_spa(ProdView P, const int *__restrict__ kind, int hyper,
                                                              int row0, int row1, unsigned *__restrict__ ctr)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    SpaSmem &S = *reinterpret_cast<SpaSmem *>(s_raw);
    __shared__ int s_blk;
    if (!hyper && kind[P.tilemA + 1] == P.numC) // every row was done by k_step3_hyper
        return;
    unsigned nxt = 0; // thread 0: the next block, claimed one block ahead
    if (threadIdx.x == 0)
        nxt = atomicAdd(ctr, 1u);
    const int t_beg = RANGED ? P.C_ptr[row0] : 0, t_end = RANGED ? P.C_ptr[row1] : P.numC;
    const long long blk0 = t_beg / BLK;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_blk = (int)nxt;
            nxt = atomicAdd(ctr, 1u);
        }
        __syncthreads();
        const long long tb = (blk0 + s_blk) * BLK;
        if (tb >= t_end)
            break;
        if (threadIdx.x == 0)
            spa_skip_hyper<BLK>(P, kind, (int)tb, ctr, -blk0);
        // the block, clamped to the tiles of rows [row0, row1)
        step3_spa_block<FLAT, BLK>(P, S, max((int)tb, t_beg), (int)min((long long)t_end, tb + BLK), kind, nullptr, hyper);
    }
}

// The hypersparse rows of tile rows [row0, row1), a CTA each, from step 2's
// list of wide rows.  Found through the blocks of C tiles they took longer to
// find than to compute: 65,536 rows of 64 products, 16 blocks to a tile row,
// 0.759 -> 0.391 ms.  Runs beside k_step3_spa, which takes the other rows: one
// after the other, each waited for the other's longest row (65,536 rows of
// uneven length times a band, step 3: 1.91 ms, 1.19 side by side; R-MAT 17 of 4
// edges a row 6.9 and 5.8; the two in one kernel spill, 65,536 random rows 0.38
// and 0.53).  k_step3_spa goes first, its rows being the longer ones.
__global__ void __launch_bounds__(SPA_THREADS, 3) k_step3_hyper(ProdView P, const int *__restrict__ wide, int row0,
                                                                int row1, unsigned *__restrict__ ctr)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    HypSmem &S = *reinterpret_cast<HypSmem *>(s_raw);
    __shared__ int s_unit;
    const int units = wide[P.tilemA];
    const int2 *list = wide_units_of(P, wide);
    unsigned nxt = 0; // thread 0: the next unit, claimed one ahead
    if (threadIdx.x == 0)
        nxt = atomicAdd(ctr, 1u);
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_unit = (int)nxt;
            nxt = atomicAdd(ctr, 1u);
        }
        __syncthreads();
        if (s_unit >= units)
            break;
        const int2 u = list[s_unit];
        if ((u.y & 0xFFFF) == 0 && u.x >= row0 && u.x < row1 && wide[u.x] == 2)
            step3_hyper_row(P, S, u.x);
    }
}

// The tile rows the staged numeric step left (left[I] != 0: its stage would
// not fit, or the row is hypersparse), by the SPA kernel; nothing unless it
// left some (left[tilemA]).
// FLAT: a product of short B rows.
template <bool RANGED, bool FLAT>
__global__ void __launch_bounds__(SPA_THREADS, 2) k_step3_rest(ProdView P, const int *__restrict__ kind,
                                                               const int *__restrict__ left, int row0, int row1,
                                                               unsigned *__restrict__ ctr)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    SpaSmem &S = *reinterpret_cast<SpaSmem *>(s_raw);
    __shared__ int s_blk;
    if (left[P.tilemA] == 0)
        return;
    unsigned nxt = 0;
    if (threadIdx.x == 0)
        nxt = atomicAdd(ctr, 1u);
    const int t_beg = RANGED ? P.C_ptr[row0] : 0, t_end = RANGED ? P.C_ptr[row1] : P.numC;
    const long long blk0 = t_beg / SPA_BLK;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            s_blk = (int)nxt;
            nxt = atomicAdd(ctr, 1u);
        }
        __syncthreads();
        const long long tb = (blk0 + s_blk) * SPA_BLK;
        if (tb >= t_end)
            break;
        if (threadIdx.x == 0)
            spa_skip_hyper(P, kind, (int)tb, ctr, -blk0);
        step3_spa_block<FLAT>(P, S, max((int)tb, t_beg), (int)min((long long)t_end, tb + SPA_BLK), kind, left);
    }
}

// The windows' tables of one product (a warp per row of B)
__global__ void __launch_bounds__(256) k_win_btab(int m, const int *__restrict__ rptr, const int *__restrict__ rcol,
                                                  int blocks, int bits, int *__restrict__ tab, int windows,
                                                  int2 *__restrict__ wtab)
{
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w < m)
        win_btab_row((int)w, rptr, rcol, blocks, bits, tab, windows, wtab);
}

// ctab, and the list of heavy rows
__global__ void __launch_bounds__(256) k_win_ctab(ProdView P, WinPlan Q)
{
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < Q.mA && Q.A_rptr[g + 1] - Q.A_rptr[g] >= Q.heavy_min)
        Q.heavy[atomicAdd(Q.nheavy, 1u)] = (int)g;
    if (g < (long long)P.tilemA * (Q.windows + 1))
        win_ctab_entry(P, Q, g);
}

// Step 3 by windows, tile rows [row0, row1); *Q.claim zeroed.  The claims are the heavy rows'
// (row, WIN_PART columns), then every other row's (tile row, window, WIN_ROWS
// rows).
__global__ void __launch_bounds__(WIN_THREADS, WIN_CTAS) k_step3_win(ProdView P, WinPlan Q, int row0, int row1)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int lane = threadIdx.x & 31;
    WinTask &S = reinterpret_cast<WinTask *>(s_raw)[threadIdx.x >> 5];
    for (int q = lane; q < WIN_COLS; q += 32)
        S.acc[q] = 0.0;
    __syncwarp();
    const unsigned parts = (unsigned)(P.nB + WIN_PART - 1) / WIN_PART;
    const unsigned hclaims = *Q.nheavy * parts;
    const unsigned claims = hclaims + (unsigned)(row1 - row0) * Q.windows * WIN_PER;
    unsigned nxt = 0;
    if (lane == 0)
        nxt = atomicAdd(Q.claim, 1u);
    for (;;)
    {
        const unsigned c = __shfl_sync(TSG_FULL_MASK, nxt, 0);
        if (c >= claims)
            break;
        if (lane == 0)
            nxt = atomicAdd(Q.claim, 1u);
        if (c >= hclaims)
            win_claim_rows(P, Q, S, row0, c - hclaims, lane);
        else
        {
            const int row = Q.heavy[c / parts], I = row / TSG_BS;
            if (I >= row0 && I < row1)
                win_claim_heavy(P, Q, S, row, (int)(c % parts), lane);
        }
    }
}

// Step 3 of narrow rows, tile rows [row0, row1); *Q.claim zeroed.
__global__ void __launch_bounds__(WIN_THREADS, WIN_CTAS)
    k_step3_nar(ProdView P, WinPlan Q, int row0, int row1, const int *__restrict__ kind, int *__restrict__ left)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int lane = threadIdx.x & 31;
    NarTask &S = reinterpret_cast<NarTask *>(s_raw)[threadIdx.x >> 5];
    for (int q = lane; q < WIN_COLS; q += 32)
        S.acc[q] = 0.0;
    __syncwarp();
    const unsigned claims = (unsigned)(row1 - row0) * NAR_PER;
    unsigned nxt = 0;
    if (lane == 0)
        nxt = atomicAdd(Q.claim, 1u);
    for (;;)
    {
        const unsigned c = __shfl_sync(TSG_FULL_MASK, nxt, 0);
        if (c >= claims)
            break;
        if (lane == 0)
            nxt = atomicAdd(Q.claim, 1u);
        nar_claim(P, Q, S, row0, c, kind, left, lane);
    }
}

// ---------------------------------------------------------------------------
// Host orchestration.
// ---------------------------------------------------------------------------
static int validate_operands(const tsg_tiled *A, const tsg_tiled *B)
{
    if (!A || !B)
        return tsg_set_error(TSG_ERR_INVALID, "null operand");
    if (A->n != B->m)
        return tsg_set_error(TSG_ERR_INVALID, "inner dimensions differ (A is %dx%d, B is %dx%d)", A->m,
                             A->n, B->m, B->n);
    if (!B->csc_tile_ptr || !B->csc_tile_rowidx)
        return tsg_set_error(TSG_ERR_INVALID, "B has no column view (build it with TSG_TILED_CSC_VIEW)");
    if (!A->tile_ptr || !B->tile_ptr)
        return tsg_set_error(TSG_ERR_INVALID, "operand without tile structure");
    return TSG_OK;
}

static float ev_ms(cudaEvent_t a, cudaEvent_t b)
{
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

static ProdView make_view(const tsg_tiled *A, const tsg_tiled *B, tsg_tiled *C)
{
    ProdView P;
    P.A_ptr = A->tile_ptr;
    P.A_col = A->tile_columnidx;
    P.A_tnnz = A->tile_nnz;
    P.A_Ptr = A->tile_csr_Ptr;
    P.A_Colb = A->tile_csr_Col;
    P.A_Val = A->tile_csr_Value;
    P.A_mask = A->mask;
    P.tilemA = A->tilem;
    P.B_ptr = B->tile_ptr;
    P.B_col = B->tile_columnidx;
    P.B_cptr = B->csc_tile_ptr;
    P.B_crow = B->csc_tile_rowidx;
    P.B_cpos = B->csc_tile_pos;
    P.B_tnnz = B->tile_nnz;
    P.B_Ptr = B->tile_csr_Ptr;
    P.B_Colb = B->tile_csr_Col;
    P.B_Val = B->tile_csr_Value;
    P.B_mask = B->mask;
    P.B_maskT = B->mask_t;
    P.B_rptr = B->row_ptr;
    P.B_rcol = B->row_col;
    P.B_rval = B->row_val;
    P.A_rptr = A->row_ptr;
    P.A_rcol = A->row_col;
    P.A_rval = A->row_val;
    P.mA = A->m;
    P.mB = B->m;
    P.nB = B->n;
    P.browB = B->m > 0 ? (int)(B->nnz / B->m) : 0;
    P.cols = step3_by_columns(A);
    P.tilenB = B->tilen;
    P.C_ptr = C->tile_ptr;
    P.C_col = C->tile_columnidx;
    P.C_row = C->tile_rowidx;
    P.C_tnnz = C->tile_nnz;
    P.C_mask = C->mask;
    P.C_Ptr = C->tile_csr_Ptr;
    P.C_Colb = C->tile_csr_Col;
    P.C_Val = C->tile_csr_Value;
    P.numC = C->numtile;
    // the staged numeric step copies ranges rounded out to 16-byte
    // boundaries: library allocations only (tsg_alloc's slack), 16-byte aligned
    const void *bases[] = {P.A_mask, P.A_Ptr, P.A_tnnz, P.A_col, P.A_Val, P.B_rcol, P.B_rval,
                           P.C_mask, P.C_Ptr, P.C_tnnz, P.C_col};
    bool aligned = true;
    for (const void *p : bases)
        aligned = aligned && ((uintptr_t)p & 15) == 0;
    P.padded = !A->_alloc && !B->_alloc && !C->_alloc && aligned;
    P.status = nullptr;
    return P;
}

template <int W, int CAP>
static int launch_step3_rows(tsg_context *ctx, const ProdView &P)
{
    const size_t smem = 8 * sizeof(S3RowsSmem<W, CAP>);
    TSG_CUDA(cudaFuncSetAttribute(k_step3_rows<W, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long items = ((long long)P.numC + W - 1) / W;
    k_step3_rows<W, CAP><<<tsg_blocks(items * 16, 128), 128, smem, ctx->stream>>>(P);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

template <int W>
static int launch_step2_rows(tsg_context *ctx, const ProdView &P, int *d_bins)
{
    const long long items = ((long long)P.numC + W - 1) / W;
    k_step2_rows<W><<<tsg_blocks(items * 16, 128), 128, 0, ctx->stream>>>(P, d_bins);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

static int launch_step2(tsg_context *ctx, const ProdView &P, int *d_bins)
{
    if (ctx->sched == TSG_SCHED_ROWS)
    {
        if (ctx->seg_tiles == 32)
            return launch_step2_rows<32>(ctx, P, d_bins);
        if (ctx->seg_tiles == 16)
            return launch_step2_rows<16>(ctx, P, d_bins);
        return launch_step2_rows<8>(ctx, P, d_bins);
    }
    k_step2<<<tsg_blocks((long long)P.numC * 16, 256), 256, 0, ctx->stream>>>(P, d_bins);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

// resident CTAs per SM of a kernel with smem bytes of dynamic shared memory,
// asked once per context
template <typename K>
static int resident_ctas(tsg_context *ctx, int slot, K kern, int threads, int smem, int *per_sm)
{
    if (!ctx->occ[slot])
    {
        int n = 0;
        TSG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        TSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem));
        if (n < 1)
            return tsg_set_error(TSG_ERR_CUDA, "a persistent kernel does not fit an SM");
        ctx->occ[slot] = n;
    }
    *per_sm = ctx->occ[slot];
    return TSG_OK;
}

// clears a step-3 kernel's counter for a range of tile rows after the first
// (the product's start cleared it before)
static int clear_counters(tsg_context *ctx, int row0, int first, int count)
{
    if (row0 > 0)
        TSG_CUDA(cudaMemsetAsync(&ctx->d_ctl->ctr[first], 0, count * sizeof(unsigned), ctx->stream));
    return TSG_OK;
}

// step 2 for the rows k_step12 listed, through B's row view.  span: at most
// WIDE_NARROW tile columns (512 threads) or WIDE_SPAN (1,024).  The kernel's
// shared-memory limit belongs to the function on the device, not to the launch:
// it is set to the largest size only, since a context on another host thread
// that set a smaller one between this one's set and launch would make the
// launch fail.
#define WIDE_NARROW 512
template <int NT>
static int launch_step2_cta(tsg_context *ctx, const ProdView &P, int span, size_t units, const int *d_wide, int *d_bins)
{
    int per_sm = 0;
    TSG_TRY(resident_ctas(ctx, NT == 512 ? TSG_OCC_WIDE : TSG_OCC_WIDE_WIDER, k_step2_cta<NT>, NT,
                          (int)wide_smem<NT>(NT == 512 ? WIDE_NARROW : WIDE_SPAN), &per_sm));
    // units, not tile rows: few rows of A may be many parts of rows (64 rows of
    // 1,000 entries times 1 M rows: 4.0 ms on 4 CTAs, 0.33 on 64)
    const int grid = (int)std::min(units, (size_t)ctx->num_sms * per_sm);
    k_step2_cta<NT><<<grid, NT, wide_smem<NT>(span), ctx->stream>>>(P, span, d_wide, &ctx->d_ctl->ctr[TSG_CTR_STEP2], d_bins);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

static int launch_step2_wide(tsg_context *ctx, const ProdView &P, int widest, size_t units, const int *d_wide,
                             int *d_bins)
{
    // the widest row of C, or as many columns as a CTA's shared memory holds;
    // narrow C leaves room for four CTAs of 512 threads on an SM (8,192 columns:
    // 0.073 ms, 0.083 with 1,024 threads; 16,384 columns of R-MAT 14: 0.45 and
    // 0.38)
    const int span = std::max(1, std::min(widest, WIDE_SPAN));
    return span <= WIDE_NARROW ? launch_step2_cta<512>(ctx, P, span, units, d_wide, d_bins)
                               : launch_step2_cta<1024>(ctx, P, span, units, d_wide, d_bins);
}

// What the window form of step 3 keeps for a product.
struct WinScratch
{
    WinPlan Q;
    int *rptr, *rcol; // A's row view, when A has none
    double *rval;
    bool ready;  // the tables are made
    bool failed; // no memory for them
};

// Whether wtab is made: B's rows times the windows
static bool win_has_wtab(const ProdView &P, const WinPlan &Q)
{
    return (long long)P.mB * Q.windows <= WIN_TABLE_WORDS / 2;
}

// Whether a product runs step 3 by windows, and their table's shape
static bool win_shape(const ProdView &P, long long nnzA, long long nnzB, long long nnzC, WinPlan &Q)
{
    if (!P.B_rptr || P.nB < 1 || P.mA < 1 || P.mB < 1)
        return false;
    const long long windows = (P.nB + WIN_COLS - 1LL) / WIN_COLS;
    // claims of every row as if it were heavy: 32-bit
    if (nnzC < WIN_MIN_VALUES * windows * P.mA || windows * WIN_PARTS * (P.mA + TSG_BS) > INT_MAX)
        return false;
    if (!win_table(P.mB, P.nB, WIN_TABLE_WORDS, Q.bits, Q.blocks))
        return false;
    Q.windows = (int)windows;
    Q.mA = P.mA;
    Q.heavy_min = win_heavy(nnzA, P.mA);
    const long long tables = (Q.blocks + 1LL + (win_has_wtab(P, Q) ? 2 * windows : 0)) * P.mB;
    return win_worth(nnzC, (long long)((double)nnzA * (double)nnzB / P.mB), nnzA, P.numC, P.tilemA,
                     P.tilenB, windows, tables);
}

static void win_release(tsg_context *ctx, WinScratch &W)
{
    tsg_release(ctx, W.Q.wtab);
    tsg_release(ctx, W.Q.btab);
    tsg_release(ctx, W.Q.ctab);
    tsg_release(ctx, W.rptr);
    tsg_release(ctx, W.rcol);
    tsg_release(ctx, W.rval);
    tsg_release(ctx, W.Q.heavy);
    W.ready = false;
}

// A's row view, made once per product when A has none
static int win_rows(tsg_context *ctx, const ProdView &P, const tsg_tiled *A, WinScratch &W)
{
    WinPlan &Q = W.Q;
    Q.claim = &ctx->d_ctl->ctr[TSG_CTR_STEP3];
    Q.nheavy = &ctx->d_ctl->ctr[TSG_CTR_HEAVY];
    Q.mA = P.mA;
    Q.A_rptr = P.A_rptr;
    Q.A_rcol = P.A_rcol;
    Q.A_rval = P.A_rval;
    if (P.A_rptr)
        return TSG_OK;
    if (!W.rptr)
    {
        TSG_TRY(tsg_alloc(ctx, &W.rptr, (size_t)A->m + 1));
        TSG_TRY(tsg_alloc(ctx, &W.rcol, (size_t)A->nnz));
        TSG_TRY(tsg_alloc(ctx, &W.rval, (size_t)A->nnz));
        TSG_TRY(tsg_t2c_view(ctx, A, W.rptr, W.rcol, W.rval));
    }
    Q.A_rptr = W.rptr;
    Q.A_rcol = W.rcol;
    Q.A_rval = W.rval;
    return TSG_OK;
}

// the tables of a product's windows, made once per product
static int win_prepare(tsg_context *ctx, const ProdView &P, const tsg_tiled *A, WinScratch &W)
{
    if (W.ready)
        return TSG_OK;
    cudaStream_t st = ctx->stream;
    WinPlan &Q = W.Q;
    TSG_TRY(tsg_alloc(ctx, &Q.btab, (size_t)P.mB * (Q.blocks + 1)));
    Q.wtab = nullptr;
    if (win_has_wtab(P, Q))
        TSG_TRY(tsg_alloc(ctx, &Q.wtab, (size_t)P.mB * Q.windows));
    TSG_TRY(tsg_alloc(ctx, &Q.ctab, (size_t)P.tilemA * (Q.windows + 1)));
    TSG_TRY(tsg_alloc(ctx, &Q.heavy, (size_t)P.mA));
    TSG_TRY(win_rows(ctx, P, A, W));
    k_win_btab<<<tsg_blocks((long long)P.mB * 32, 256), 256, 0, st>>>(P.mB, P.B_rptr, P.B_rcol, Q.blocks, Q.bits, Q.btab, Q.windows, Q.wtab);
    TSG_LAUNCH_CHECK();
    k_win_ctab<<<tsg_blocks(std::max((long long)P.mA, (long long)P.tilemA * (Q.windows + 1)), 256), 256, 0, st>>>(P, Q);
    TSG_LAUNCH_CHECK();
    W.ready = true;
    return TSG_OK;
}

// step 3 by windows for tile rows [row0, row1)
static int launch_step3_win(tsg_context *ctx, const ProdView &P, const tsg_tiled *A, WinScratch &W, int row0, int row1)
{
    TSG_TRY(win_prepare(ctx, P, A, W));
    const int smem = WIN_WARPS * (int)sizeof(WinTask);
    int per_sm = 0;
    TSG_TRY(resident_ctas(ctx, TSG_OCC_WIN, k_step3_win, WIN_THREADS, smem, &per_sm));
    TSG_TRY(clear_counters(ctx, row0, TSG_CTR_STEP3, 1));
    const long long claims = (long long)(row1 - row0) * W.Q.windows * (TSG_BS / WIN_ROWS);
    const long long grid = std::min((long long)ctx->num_sms * per_sm, (claims + WIN_WARPS - 1) / WIN_WARPS);
    k_step3_win<<<(unsigned)grid, WIN_THREADS, smem, ctx->stream>>>(P, W.Q, row0, row1);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

template <bool FLAT, bool RANGED, int BLK = SPA_BLK>
static int launch_step3_spa(tsg_context *ctx, const ProdView &P0, const int *d_kind, bool hyper_apart, int row0, int row1)
{
    ProdView P = P0;
    P.status = ctx->d_status;
    unsigned *ctr = ctx->d_ctl->ctr;
    const int smem = (int)sizeof(SpaSmem);
    int per_sm = 0;
    TSG_TRY(resident_ctas(ctx, TSG_OCC_SPA + (FLAT ? 1 : 0) + (RANGED ? 2 : 0) + (BLK == SPA_BLK ? 0 : 4),
                          k_step3_spa<FLAT, RANGED, BLK>, SPA_THREADS, smem, &per_sm));
    TSG_TRY(clear_counters(ctx, row0, TSG_CTR_STEP3, 2));
    if (hyper_apart)
        TSG_TRY(tsg_fork(ctx, ctx->stream, 1));
    k_step3_spa<FLAT, RANGED, BLK><<<ctx->num_sms * per_sm, SPA_THREADS, smem, ctx->stream>>>(
        P, d_kind, !hyper_apart, row0, row1, &ctr[TSG_CTR_STEP3]);
    TSG_LAUNCH_CHECK();
    if (!hyper_apart)
        return TSG_OK;
    int hper_sm = 0;
    TSG_TRY(resident_ctas(ctx, TSG_OCC_HYPER, k_step3_hyper, SPA_THREADS, (int)sizeof(HypSmem), &hper_sm));
    k_step3_hyper<<<ctx->num_sms * hper_sm, SPA_THREADS, sizeof(HypSmem), ctx->side[0]>>>(
        P, d_kind, RANGED ? row0 : 0, RANGED ? row1 : P.tilemA, &ctr[TSG_CTR_REST]);
    TSG_LAUNCH_CHECK();
    return tsg_join(ctx, ctx->stream, 1);
}

// the staged numeric step for tile rows [row0, row1), then the SPA kernel
// for the rows it left
template <bool RANGED>
static int launch_step3_stg(tsg_context *ctx, const ProdView &P0, const int *d_kind, int row0, int row1)
{
    ProdView P = P0;
    P.status = ctx->d_status;
    unsigned *ctr = ctx->d_ctl->ctr;
    int *left = nullptr;
    const int smem = (int)sizeof(StgSmem), rsmem = (int)sizeof(SpaSmem);
    int per_sm = 0, rest_per_sm = 0;
    TSG_TRY(resident_ctas(ctx, TSG_OCC_STG + (RANGED ? 1 : 0), k_step3_stg<RANGED>, STG_THREADS, smem, &per_sm));
    TSG_TRY(resident_ctas(ctx, TSG_OCC_REST + (RANGED ? 1 : 0), k_step3_rest<RANGED, false>, SPA_THREADS, rsmem, &rest_per_sm));
    TSG_TRY(clear_counters(ctx, row0, TSG_CTR_STEP3, 2));
    TSG_TRY(tsg_alloc(ctx, &left, (size_t)P.tilemA + 1));
    TSG_CUDA(cudaMemsetAsync(left, 0, ((size_t)P.tilemA + 1) * sizeof(int), ctx->stream));
    k_step3_stg<RANGED><<<ctx->num_sms * per_sm, STG_THREADS, smem, ctx->stream>>>(P, d_kind, row0, row1,
                                                                                 &ctr[TSG_CTR_STEP3], left, ctx->d_status);
    TSG_LAUNCH_CHECK();
    k_step3_rest<RANGED, false><<<ctx->num_sms * rest_per_sm, SPA_THREADS, rsmem, ctx->stream>>>(P, d_kind, left, row0, row1,
                                                                                       &ctr[TSG_CTR_REST]);
    TSG_LAUNCH_CHECK();
    tsg_release(ctx, left);
    return TSG_OK;
}

// step 3 of narrow rows for tile rows [row0, row1), then the SPA kernel for the
// rows it left
template <bool RANGED>
static int launch_step3_nar(tsg_context *ctx, const ProdView &P0, const tsg_tiled *A, WinScratch &W, const int *d_kind,
                            int row0, int row1)
{
    ProdView P = P0;
    P.status = ctx->d_status;
    TSG_TRY(win_rows(ctx, P, A, W));
    int *left = nullptr;
    const int smem = WIN_WARPS * (int)sizeof(NarTask), rsmem = (int)sizeof(SpaSmem);
    int per_sm = 0, rest_per_sm = 0;
    TSG_TRY(resident_ctas(ctx, TSG_OCC_NAR, k_step3_nar, WIN_THREADS, smem, &per_sm));
    TSG_TRY(resident_ctas(ctx, TSG_OCC_REST + (RANGED ? 1 : 0) + 2, k_step3_rest<RANGED, true>, SPA_THREADS, rsmem,
                          &rest_per_sm));
    TSG_TRY(clear_counters(ctx, row0, TSG_CTR_STEP3, 2));
    TSG_TRY(tsg_alloc(ctx, &left, (size_t)P.tilemA + 1));
    TSG_CUDA(cudaMemsetAsync(left, 0, ((size_t)P.tilemA + 1) * sizeof(int), ctx->stream));
    const long long claims = (long long)(row1 - row0) * NAR_PER;
    const long long grid = std::min((long long)ctx->num_sms * per_sm, (claims + WIN_WARPS - 1) / WIN_WARPS);
    k_step3_nar<<<(unsigned)grid, WIN_THREADS, smem, ctx->stream>>>(P, W.Q, row0, row1, d_kind, left);
    TSG_LAUNCH_CHECK();
    k_step3_rest<RANGED, true><<<ctx->num_sms * rest_per_sm, SPA_THREADS, rsmem, ctx->stream>>>(
        P, d_kind, left, row0, row1, &ctx->d_ctl->ctr[TSG_CTR_REST]);
    TSG_LAUNCH_CHECK();
    tsg_release(ctx, left);
    return TSG_OK;
}

// step 3 by the SPA kernel: the default schedule, except for products whose
// C tiles are dense on average (>= ctx->spa_dense values, SPA_DENSE unless
// set) and B without a row view (borrowed foreign buffers), which take the
// tile kernel
static bool step3_by_spa(const tsg_context *ctx, const ProdView &P, long long nnzC)
{
    return ctx->sched == TSG_SCHED_SPA && P.B_rptr && nnzC < (long long)ctx->spa_dense * P.numC;
}

// the SPA numeric step for tile rows [row0, row1)
static int launch_step3_spa_rows(tsg_context *ctx, const ProdView &P, const tsg_tiled *A, long long nnzB, long long nnzC,
                                 const int *d_kind, WinScratch &W, int row0, int row1)
{
    const bool flat = spa_wants_flat(P.browB, P.numC, nnzC, P.tilemA);
    const bool whole = row0 == 0 && row1 == P.tilemA;
    ctx->last_step3 = flat ? TSG_STEP3_FLAT : P.padded ? TSG_STEP3_STAGED : TSG_STEP3_SPA;
    if (flat && !W.failed && win_shape(P, A->nnz, nnzB, nnzC, W.Q))
    {
        const int kernel = ctx->last_step3;
        ctx->last_step3 = TSG_STEP3_WINDOWS;
        const int status = launch_step3_win(ctx, P, A, W, row0, row1);
        if (status != TSG_ERR_OOM || W.ready)
            return status;
        // no room for the tables, which the other kernels do without
        cudaGetLastError();
        win_release(ctx, W);
        W.failed = true;
        ctx->last_step3 = kernel;
    }
    if (flat && P.numC <= (long long)NAR_MEAN * P.tilemA)
    {
        ctx->last_step3 = TSG_STEP3_NARROW;
        return whole ? launch_step3_nar<false>(ctx, P, A, W, d_kind, row0, row1)
                     : launch_step3_nar<true>(ctx, P, A, W, d_kind, row0, row1);
    }
    if (flat && nnzC >= (long long)SPA_BLK_NARROW_VALUES * P.numC)
        return whole ? launch_step3_spa<true, false, SPA_BLK_NARROW>(ctx, P, d_kind, false, 0, 0)
                     : launch_step3_spa<true, true, SPA_BLK_NARROW>(ctx, P, d_kind, false, row0, row1);
    // mostly hypersparse rows (few values in many tiles): those by themselves,
    // unless the second stream costs more (4,096 random rows of 4, 65 K tiles:
    // 0.036 ms, 0.027 without)
    const bool hyper = d_kind && nnzC < (long long)HYP_RATIO * P.numC && P.numC > (long long)S12_MAXT * P.tilemA &&
                       P.numC >= HYP_APART;
    if (flat)
        return whole ? launch_step3_spa<true, false>(ctx, P, d_kind, hyper, 0, 0)
                     : launch_step3_spa<true, true>(ctx, P, d_kind, hyper, row0, row1);
    if (P.padded)
        return whole ? launch_step3_stg<false>(ctx, P, d_kind, 0, 0) : launch_step3_stg<true>(ctx, P, d_kind, row0, row1);
    // operands viewing a batch arena: not padded for the bulk copies' rounding
    return whole ? launch_step3_spa<false, false>(ctx, P, d_kind, false, 0, 0)
                 : launch_step3_spa<false, true>(ctx, P, d_kind, false, row0, row1);
}

// d_kind: the row kinds of the fused step 1/2 pass (0 narrow, 1 wide,
// 2 hypersparse), or null
static int launch_step3(tsg_context *ctx, const ProdView &P, const tsg_tiled *A, long long nnzB, long long nnzC,
                        const int *d_kind, WinScratch &W)
{
    if (step3_by_spa(ctx, P, nnzC))
        return launch_step3_spa_rows(ctx, P, A, nnzB, nnzC, d_kind, W, 0, P.tilemA);
    if (ctx->sched == TSG_SCHED_ROWS)
    {
        const int W = ctx->seg_tiles, cap = ctx->acc_cap;
        ctx->last_step3 = TSG_STEP3_ROWS;
#define TSG_DISPATCH3(w, c)                    \
    if (W == w && cap == c)                    \
        return launch_step3_rows<w, c>(ctx, P);
        TSG_ROW_CONFIGS(TSG_DISPATCH3)
#undef TSG_DISPATCH3
        return tsg_set_error(TSG_ERR_INVALID, "unsupported row schedule (%d, %d)", W, cap);
    }
    if (ctx->sched == TSG_SCHED_ELEMS)
    {
        if (!P.B_maskT)
            return tsg_set_error(TSG_ERR_INVALID, "element schedule needs B's column masks (mask_t)");
        ctx->last_step3 = TSG_STEP3_ELEMS;
        k_step3_elems<<<tsg_blocks((long long)P.numC * 32, 256), 256, 0, ctx->stream>>>(P);
        TSG_LAUNCH_CHECK();
        return TSG_OK;
    }
    ctx->last_step3 = P.cols ? TSG_STEP3_TILES : TSG_STEP3_TILE_ROWS;
    if (P.cols)
        k_step3<<<tsg_blocks((long long)P.numC * 16, S3_THREADS), S3_THREADS, 0, ctx->stream>>>(P);
    else
        k_step3_tile_rows<<<tsg_blocks((long long)P.numC * 16, S3R_THREADS), S3R_THREADS, 0, ctx->stream>>>(P);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}

// What steps 1-2 leave for step 3 and the statistics.
struct SpgemmRun
{
    int *d_wide; // row kinds of the fused pass, or null
    size_t units;     // units of the wide step 2 at most
    int widest;       // widest window of a C tile row, in tile columns
    StepOneBits bits; // step 1's bitmaps, until the emit pass has read them
    WinScratch win;
    long long numC, nnzC;
};

// Steps 1 and 2 of C = A*B: on return C's tile structure, masks, row offsets
// and tile value offsets are final, nnz(C) is known on the host and C's value
// arrays are allocated.  Records ev[0..2] when timing.
static int spgemm_structure(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, tsg_tiled *C, SpgemmRun &R)
{
    memset(&R, 0, sizeof(R));
    memset(C, 0, sizeof(*C));
    C->m = A->m;
    C->n = B->n;
    C->tilem = A->tilem;
    C->tilen = B->tilen;
    C->col_packed = 0;
    const int tilem = C->tilem;
    cudaStream_t st = ctx->stream;
    const int timing = ctx->timing;
    if (timing)
        TSG_CUDA(cudaEventRecord(ctx->ev[0], st));

    // step 1: structure
    unsigned long long *d_pairs = &ctx->d_ctl->pairs;
    int *d_bins = ctx->d_ctl->bins;
    TSG_CUDA(cudaMemsetAsync(ctx->d_ctl, 0, offsetof(TsgControl, status), st));
    TSG_TRY(tsg_alloc(ctx, &C->tile_ptr, (size_t)tilem + 1));
    long long numC = 0;
    if (tilem > 0)
    {
        ProdView P = make_view(A, B, C);
        const int stride = std::min((B->tilen + 31) / 32, S1_KEEP_WORDS);
        if ((long long)tilem * stride <= S1_KEEP_TOTAL)
        {
            R.bits.stride = stride;
            TSG_TRY(tsg_alloc(ctx, &R.bits.words, (size_t)tilem * stride));
            TSG_TRY(tsg_alloc(ctx, &R.bits.span, (size_t)tilem));
        }
        R.bits.widest = &ctx->d_ctl->widest;
        if (step1_by_cta(A, B))
            k_step1_cta<<<tilem, S1C_THREADS, 0, st>>>(P, C->tile_ptr, d_pairs, R.bits);
        else
            k_step1<false><<<tsg_blocks(tilem, S1_WARPS), S1_WARPS * 32, 0, st>>>(P, C->tile_ptr, d_pairs, R.bits);
        TSG_LAUNCH_CHECK();
        TSG_CUDA(cudaMemcpyAsync(ctx->h_pinned + 2, &ctx->d_ctl->widest, sizeof(int), cudaMemcpyDeviceToHost, st));
        TSG_TRY(tsg_scan_counts(ctx, C->tile_ptr, C->tile_ptr, tilem, &numC));
        R.widest = *(const int *)(ctx->h_pinned + 2);
    }
    else
        TSG_CUDA(cudaMemsetAsync(C->tile_ptr, 0, sizeof(int), st));
    C->numtile = (int)numC;
    R.numC = numC;
    TSG_TRY(tsg_alloc(ctx, &C->tile_columnidx, (size_t)numC));
    TSG_TRY(tsg_alloc(ctx, &C->tile_rowidx, (size_t)numC));
    TSG_TRY(tsg_alloc(ctx, &C->mask, (size_t)numC * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &C->tile_csr_Ptr, (size_t)numC * TSG_BS));
    TSG_TRY(tsg_alloc(ctx, &C->tile_nnz, (size_t)numC + 1));
    long long nnzC = 0;
    const bool fused = ctx->fuse12 && ctx->sched != TSG_SCHED_ROWS;
    if (numC > 0)
    {
        ProdView P = make_view(A, B, C);
        if (fused)
        {
            const int split = wide_split(A->nnz, ctx->num_sms);
            R.units = wide_units(tilem, A->nnz, split);
            TSG_TRY(tsg_alloc(ctx, &R.d_wide, (size_t)tilem + 3 + 2 * R.units));
            TSG_CUDA(cudaMemsetAsync(R.d_wide + tilem, 0, 2 * sizeof(int), st));
            k_step12<<<tsg_blocks(tilem, S12_WARPS), S12_WARPS * 32, 0, st>>>(
                P, R.bits, split, P.B_rptr ? s12_per_pair(tilem, ctx->num_sms) : 0, R.d_wide, d_bins);
            TSG_LAUNCH_CHECK();
        }
        else
        {
            k_step1<true><<<tsg_blocks(tilem, S1_WARPS), S1_WARPS * 32, 0, st>>>(P, nullptr, nullptr, StepOneBits{nullptr, nullptr, 0, nullptr});
            TSG_LAUNCH_CHECK();
        }
    }
    tsg_release(ctx, R.bits.words);
    tsg_release(ctx, R.bits.span);
    if (timing)
        TSG_CUDA(cudaEventRecord(ctx->ev[1], st));

    // step 2: symbolic (rows the fused kernel left, or all tiles)
    if (numC > 0)
    {
        ProdView P = make_view(A, B, C);
        if (fused && P.B_rptr)
            TSG_TRY(launch_step2_wide(ctx, P, R.widest, R.units, R.d_wide, d_bins));
        else if (fused)
        {
            k_step2_wide<<<tsg_blocks(numC * 16, 256), 256, 0, st>>>(P, R.d_wide, d_bins);
            TSG_LAUNCH_CHECK();
        }
        else
            TSG_TRY(launch_step2(ctx, P, d_bins));
        TSG_TRY(tsg_scan_counts(ctx, C->tile_nnz, C->tile_nnz, numC, &nnzC));
    }
    else
        TSG_CUDA(cudaMemsetAsync(C->tile_nnz, 0, sizeof(int), st));
    C->nnz = (int)nnzC;
    if (timing)
        TSG_CUDA(cudaEventRecord(ctx->ev[2], st));

    R.nnzC = nnzC;
    // C's value arrays
    TSG_TRY(tsg_alloc(ctx, &C->tile_csr_Col, (size_t)nnzC));
    TSG_TRY(tsg_alloc(ctx, &C->tile_csr_Value, (size_t)nnzC));
    return TSG_OK;
}

// Statistics of a product (tile pairs, bins, step times from ev[0..3]) and
// the release of the steps' scratch.
static int spgemm_finish(tsg_context *ctx, SpgemmRun &R, tsg_spgemm_info *info)
{
    cudaStream_t st = ctx->stream;
    tsg_release(ctx, R.d_wide);
    win_release(ctx, R.win);
    // the counters and the error word in one read-back
    TsgControl *h = (TsgControl *)ctx->h_pinned;
    TSG_CUDA(cudaMemcpyAsync(h, ctx->d_ctl, sizeof(TsgControl), cudaMemcpyDeviceToHost, st));
    TSG_CUDA(cudaStreamSynchronize(st));
    TSG_TRY(tsg_check_device_status(ctx, h->status));
    if (info)
    {
        memset(info, 0, sizeof(*info));
        info->numtile_C = R.numC;
        info->nnz_C = R.nnzC;
        info->tile_pairs = (long long)h->pairs;
        memcpy(info->bins, h->bins, sizeof(info->bins));
        info->step3_kernel = R.nnzC > 0 ? ctx->last_step3 : TSG_STEP3_NONE;
        if (ctx->timing)
        {
            info->ms_step1 = ev_ms(ctx->ev[0], ctx->ev[1]);
            info->ms_step2 = ev_ms(ctx->ev[1], ctx->ev[2]);
            info->ms_step3 = ev_ms(ctx->ev[2], ctx->ev[3]);
            info->ms_total = ev_ms(ctx->ev[0], ctx->ev[3]);
        }
    }
    return TSG_OK;
}

// the scratch of a product that failed
static void spgemm_drop(tsg_context *ctx, SpgemmRun &R)
{
    tsg_release(ctx, R.bits.words);
    tsg_release(ctx, R.bits.span);
    tsg_release(ctx, R.d_wide);
    win_release(ctx, R.win);
}

extern "C" int tsg_spgemm(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, tsg_tiled *C,
                          tsg_spgemm_info *info)
{
    if (!ctx || !C)
        return tsg_set_error(TSG_ERR_INVALID, "null argument");
    TSG_TRY(validate_operands(A, B));
    SpgemmRun R;
    int status = spgemm_structure(ctx, A, B, C, R);
    // step 3: numeric
    if (status == TSG_OK && R.nnzC > 0)
        status = launch_step3(ctx, make_view(A, B, C), A, B->nnz, R.nnzC, R.d_wide, R.win);
    if (status != TSG_OK)
    {
        spgemm_drop(ctx, R);
        return status;
    }
    if (ctx->timing)
        TSG_CUDA(cudaEventRecord(ctx->ev[3], ctx->stream));
    return spgemm_finish(ctx, R, info);
}

// C = A*B straight into host CSR buffers, the copy overlapping the numeric
// step.  After step 2 the row pointer of C is final: it is computed and
// copied first, so the host knows where every tile row's entries go.  Then
// the tile rows of C are taken in chunks of about equal nonzeros: a chunk's
// numeric step (the SPA kernel over its rows) and its CSR fill run on the
// context's stream while the previous chunks' column indices and values are
// copied out on the copy stream.  Products whose step 3 is not the SPA
// kernel run it whole first; their fill and copy are still chunked.
int tsg_spgemm_to_host(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, int *h_rowptr, int *h_colidx,
                       double *h_val, long long nnz_cap, int *nnzC_out, tsg_spgemm_info *info)
{
    TSG_TRY(validate_operands(A, B));
    tsg_tiled C;
    SpgemmRun R;
    int status = spgemm_structure(ctx, A, B, &C, R);
    int *d_rp = nullptr, *d_ci = nullptr;
    double *d_v = nullptr;
    cudaStream_t st = ctx->stream;
    const int m = C.m, tilem = C.tilem;
    if (status == TSG_OK)
    {
        *nnzC_out = R.nnzC > INT_MAX ? INT_MAX : (int)R.nnzC; // the scan rejects more than 32-bit offsets
        if (R.nnzC > nnz_cap)
            status = tsg_set_error(TSG_ERR_OVERFLOW, "C has %lld nonzeros; the output buffers hold %lld", R.nnzC,
                                   nnz_cap);
    }
    if (status == TSG_OK)
        status = tsg_alloc(ctx, &d_rp, (size_t)m + 1);
    if (status == TSG_OK)
        status = tsg_alloc(ctx, &d_ci, (size_t)R.nnzC);
    if (status == TSG_OK)
        status = tsg_alloc(ctx, &d_v, (size_t)R.nnzC);
    if (status == TSG_OK)
        status = ([&]() -> int {
            // row pointer, to the host first
            if (m > 0)
                TSG_TRY(tsg_t2c_rows(ctx, &C, d_rp));
            else
                TSG_CUDA(cudaMemsetAsync(d_rp, 0, sizeof(int), st));
            TSG_CUDA(cudaMemcpyAsync(h_rowptr, d_rp, ((size_t)m + 1) * sizeof(int), cudaMemcpyDeviceToHost, st));
            TSG_CUDA(cudaStreamSynchronize(st));
            if (R.nnzC == 0 || tilem == 0)
                return TSG_OK;
            TSG_TRY(tsg_copy_stream(ctx));
            const ProdView P = make_view(A, B, &C);
            const bool spa = step3_by_spa(ctx, P, R.nnzC);
            if (!spa)
                TSG_TRY(launch_step3(ctx, P, A, B->nnz, R.nnzC, R.d_wide, R.win));
            // chunks of about equal nonzeros (>= TSG_CHUNK_NNZ each, at most TSG_MAX_CHUNKS)
            const long long nch = std::max(1LL, std::min((long long)TSG_MAX_CHUNKS, R.nnzC / TSG_CHUNK_NNZ));
            int r0 = 0;
            for (long long c = 1; c <= nch; c++)
            {
                int r1 = tilem;
                if (c < nch)
                {
                    // first tile row whose entries start at or after c / nch of C's
                    const long long want = R.nnzC * c / nch;
                    int lo = r0 + 1, hi = tilem;
                    while (lo < hi)
                    {
                        const int mid = (lo + hi) >> 1;
                        if ((long long)h_rowptr[(long long)mid * TSG_BS] >= want)
                            hi = mid;
                        else
                            lo = mid + 1;
                    }
                    r1 = lo;
                }
                if (r1 <= r0)
                    continue;
                if (spa)
                    TSG_TRY(launch_step3_spa_rows(ctx, P, A, B->nnz, R.nnzC, R.d_wide, R.win, r0, r1));
                TSG_TRY(tsg_t2c_fill(ctx, &C, r0, r1, d_rp, d_ci, d_v));
                TSG_CUDA(cudaEventRecord(ctx->copy_ev, st));
                TSG_CUDA(cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_ev, 0));
                const long long e0 = h_rowptr[(long long)r0 * TSG_BS], e1 = h_rowptr[r1 * TSG_BS < m ? r1 * TSG_BS : m];
                if (e1 > e0)
                {
                    TSG_CUDA(cudaMemcpyAsync(h_colidx + e0, d_ci + e0, (size_t)(e1 - e0) * sizeof(int),
                                             cudaMemcpyDeviceToHost, ctx->copy_stream));
                    TSG_CUDA(cudaMemcpyAsync(h_val + e0, d_v + e0, (size_t)(e1 - e0) * sizeof(double),
                                             cudaMemcpyDeviceToHost, ctx->copy_stream));
                }
                r0 = r1;
            }
            return TSG_OK;
        })();
    // the copies end before the buffers are released on the context's stream
    if (ctx->copy_stream)
        cudaStreamSynchronize(ctx->copy_stream);
    if (status == TSG_OK && ctx->timing)
        status = cudaEventRecord(ctx->ev[3], st) == cudaSuccess ? TSG_OK
                                                                 : tsg_set_error(TSG_ERR_CUDA, "cudaEventRecord");
    tsg_release(ctx, d_rp);
    tsg_release(ctx, d_ci);
    tsg_release(ctx, d_v);
    if (status == TSG_OK)
        status = spgemm_finish(ctx, R, info);
    else
        spgemm_drop(ctx, R);
    tsg_tiled_free(ctx, &C);
    if (status == TSG_OK)
        TSG_CUDA(cudaStreamSynchronize(st));
    return status;
}

// Number of C tiles of A*B (step 1's count pass only) added to the device
// word *total, without synchronising; A and B need their row-major tile
// structure.
int tsg_count_c_tiles_async(tsg_context *ctx, const tsg_tiled *A, const tsg_tiled *B, unsigned long long *total)
{
    if (A->tilem == 0)
        return TSG_OK;
    tsg_tiled Cdummy;
    memset(&Cdummy, 0, sizeof(Cdummy));
    k_step1_total<<<tsg_blocks(A->tilem, S1_WARPS), S1_WARPS * 32, 0, ctx->stream>>>(make_view(A, B, &Cdummy), total);
    TSG_LAUNCH_CHECK();
    return TSG_OK;
}
