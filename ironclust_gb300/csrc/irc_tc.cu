// irc_tc.cu -- tensor-core (tcgen05) site kNN: BF16 distance filter, exact
// FP32 re-rank, FP64 at the k-th-neighbour boundary.
//
// A work item is up to four "slots", each a run of queries of one drift
// chunk (128, 64 or 32 rows), packed into the 128 TMEM lanes of one M=128
// tile; every slot owns a share of the TMEM accumulators and its own epilogue
// warps, and the slots' candidate tiles are issued round-robin so small
// chunks (a probe site has ~17 queries per chunk) share a CTA without waiting
// on each other.  The filter is persistent: one launch per packing class
// (one-, two- or four-slot items), one CTA per SM, each CTA taking items from
// the class's work queue (an atomic head over the items, ordered by cost,
// largest first) until it is empty.  Barrier phases, stage and accumulator
// counters run on across a CTA's items; the query tile is double-buffered,
// so the next item's tiles load and its first MMAs run while the epilogue
// still finishes the item before.
// The BF16 (kind::f16) or FP8-e4m3 (kind::f8f6f4) operand rows of
// irc_tc_host.cu -- 128 bytes each, so both use the same swizzled layout and
// one MMA per 32 bytes -- make every accumulator the approximate squared
// distance (FP8: a fixed positive multiple of it).
//
// A slot streams its chunk's 128-candidate tiles (a per-chunk tile table in
// the plan) in units: items of one or two slots use 256-wide units (two
// tiles, loaded by two TMA boxes into one stage, one N = 256 MMA per K slice,
// two 256-column accumulators) -- the issue cost of an MMA is the same at
// N = 256 as at 128, so this halves it per pair -- unless the plan asks for
// 128-wide units (irc_plan_tc_units), and four-slot items 128-wide units
// (four accumulators, one per slot).  Warp roles: warp 0 claims items and
// issues TMA loads (a ring of 4 wide or 6 narrow stages, four 32-row query
// boxes per item), warps 1 and 18 issue tcgen05.mma from one thread each, unit
// by unit in turn (warp 1 also owns TMEM), warps 2-17 are the epilogue: four
// per TMEM lane quarter, warp w of a quarter reading columns 32w .. 32w + 31
// of every 128-tile.  A warp releases an accumulator as soon as its values are
// in registers.  Each slot's units are streamed twice:
//   pass 1  every thread folds its columns into 32 per-column minima (the two
//           tiles of a wide unit with one three-input min); per query, the
//           r-th smallest of the 128 minima (r = 48 for BF16, 64 for FP8; a
//           bitwise search, rounded up by < 2^-11 relative, < 2^-7 for
//           slots of at most 16 tiles) is an upper bound
//           tau on the r-th nearest approximate distance (r distinct
//           candidates lie at or below it, against knn <= 32);
//   pass 2  the candidates at or below tau are appended to the query's list
//           in shared memory (~55-70 per query on random data, at most 192; an
//           overflowing query is finished by the exact fallback kernel).  In
//           the BF16 wide units the thresholds are folded into the MMA: each
//           query's -tau goes into three spare K columns of its operand row,
//           against 1s in the candidate rows, so the accumulators are
//           d2 - tau and a hit is a sign bit (one funnel shift per pair);
//           elsewhere every pair is compared with tau in the epilogue.
// The minima partition, and with it tau, is the same at both widths and in every
// layout (the lists of folded thresholds also hold what lies within 2^-10 above
// tau).  Measured on 400,000 spikes, D = 33 (1.2e10
// pairs, one launch): 3.65 ms with one MMA issuer, three stages and late
// releases, 3.02 ms as above; without any epilogue work the pipeline takes
// 1.81, and folding, marking and appending add 0.35, 0.48 and 0.46.
// Every listed candidate is then re-ranked
// with the reference FP32 arithmetic (exact), zero distances dropped, sorted
// by (distance, index) with a warp bitonic network; candidates within 16 ulps
// of the k-th distance are re-ordered by their FP64 distance.  The kernel is
// bound by its epilogue (TMEM loads, fold, compare, list appends), not by the
// tensor pipe.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <mutex>
#include <type_traits>
#include <vector>

#include "irc_common.cuh"
#include "irc_plan.cuh"
#include "irc_rerank.cuh"
#include "irc_sm100.cuh"
#include "irc_tc.cuh"

// Poll limit of the filter's pipeline waits (irc_set_wait_limit); the
// drains of a CTA's own copies and MMAs keep the full bound.
__constant__ uint32_t c_wait_polls = 1u << 22;

namespace {

using irc_tc::BM;
using irc_tc::Fmt;
using irc_tc::KP;
using irc_rr::emit;
using irc_rr::QROW4;
using irc_rr::TAU_LOW_BIT;
using irc_rr::WARP_KEYS;
constexpr int PARTS = 4;                          // epilogue warps per TMEM lane quarter
constexpr int PART = 32;                          // columns of a 128-tile per epilogue warp (one minimum each)
constexpr int BROW = 128 + 1;                     // minima row of a query (f32, 4 parts x 32) in the threshold step
constexpr int EPI_WARPS = 4 * PARTS;
constexpr int MMA_WARPS = 2;                      // MMA issuers: warp 1 and the last warp, alternate units
constexpr int THREADS = 32 * (1 + MMA_WARPS + EPI_WARPS);
constexpr uint32_t A_BYTES = BM * KP * 2;         // the query tile: 128 rows x 128 bytes
constexpr uint32_t HALF_BYTES = 128 * KP * 2;     // one 128-candidate tile
constexpr uint32_t TMEM_COLS = 512;               // all TMEM columns (one CTA per SM)
constexpr int LISTCAP = irc_tc::LIST_ROW;                      // candidate-list capacity per query (the four warps' hits pooled)
constexpr int MAX_SHORT_TILES = 512;              // tiles per chunk that a 16-bit list entry can name
// The threshold is the tau_rank-th smallest per-column minimum: tau_rank
// distinct candidates lie at or below it, a margin over knn (<= 32) for the
// rounding of the filter.  A list it cut must hold at least knn +
// crowd_margin positive distances (exact copies of the query, at distance 0,
// take places in it), else the query goes to the exact fallback.  BF16:
// measured against FP64, rank 48 keeps the kNN recall at 1.0 with the same
// rho / delta error as rank 64 on the 400k-spike drift site, a 1M-spike
// sample of the probe batch and the test sites, with 20% less re-rank work;
// rank 40 missed one neighbour on a 20k-spike site with exact duplicates (its
// BF16 distance error, ~2^-8 |a| / d relative, crossed the gap between the
// 30th and 40th neighbour), rank 44 did not.  FP8 (3 mantissa bits) keeps
// rank 64.
// F16 takes BF16's rank: its callers prove each query's list complete.
__host__ __device__ constexpr int tau_rank(Fmt f) { return f == Fmt::fp8 ? 64 : 48; }
__host__ __device__ constexpr int crowd_margin(Fmt f) { return f == Fmt::fp8 ? 16 : 8; }
static_assert(tau_rank(Fmt::bf16) >= irc_tc::KNN_MAX + crowd_margin(Fmt::bf16), "rank covers knn plus the margin");
static_assert(tau_rank(Fmt::fp8) >= irc_tc::KNN_MAX + crowd_margin(Fmt::fp8), "rank covers knn plus the margin");
static_assert(LISTCAP <= irc_tc::LIST_MAX, "the re-rank takes every list the filter hands over");

// Shapes of the filter for a unit width BN (MMA N): 256 for items of one or
// two slots (two 256-column accumulators; the MMA issue cost per instruction
// is the same at N = 256 as at 128, so the wider unit halves it per pair), 128
// for four-slot items (one accumulator per slot).
// A list entry is 16 bits -- place of the tile in the chunk's list (9 bits) and
// column (7) -- unless a chunk has more tiles than that (BIG: 32 bits, the
// candidate's row); the half-size lists make room for a fourth stage of a wide
// unit.  Stages matter because a load takes ~900 cycles from issue to arrival,
// and freeing a stage, waking the producer and issuing its loads ~700 more:
// three 32 KB stages held the pipeline at ~1,200 cycles a unit.
template <int BN, bool BIG>
struct Tile {
    static_assert(BN == 128 || BN == 256, "unit width");
    static constexpr int NBUF = TMEM_COLS / BN;   // accumulator buffers, split among the slots
    static constexpr int STAGES = BN == 256 ? (BIG ? 3 : 4) : (BIG ? 4 : 6);
    static constexpr uint32_t STAGE_BYTES = BN * KP * 2;
    using Entry = typename std::conditional<BIG, uint32_t, uint16_t>::type;
    static constexpr int LROW = LISTCAP + 4 / (int)sizeof(Entry);     // entries of a list row, an odd number of words
    // list rows of a lane quarter; its minima rows (threshold step) share the space
    static constexpr size_t MIN_BYTES = (size_t)BROW * 32 * 4, ROWS_BYTES = (size_t)LROW * 32 * sizeof(Entry);
    static constexpr size_t QUARTER_BYTES = ROWS_BYTES > MIN_BYTES ? ROWS_BYTES : MIN_BYTES;
    // two query tiles (the next item's loads while this one's MMAs run)
    static constexpr size_t SMEM_BYTES = 1024 /*align slack*/ + 2 * A_BYTES + (size_t)STAGE_BYTES * STAGES +
                                         4 * QUARTER_BYTES + BM * 4 /*tau*/ + BM * 4 /*counts*/ + 384 /*barriers*/;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static __device__ __forceinline__ const Entry *row(const unsigned char *lists, int quarter, int l)
    {
        return reinterpret_cast<const Entry *>(lists + quarter * QUARTER_BYTES) + l * LROW;
    }
};

// Work units of a slot per pass over its chunk's sequence of 128-candidate
// tiles (nts of them).  BN = 128: one tile per unit; BN = 256: tiles 2u and
// 2u + 1 in unit u, loaded by two TMA boxes into the halves of one 256-row
// stage (the second absent when the count is odd).  Either way epilogue warp
// w of a lane quarter reads columns 32w .. 32w + 31 of every 128-tile, and
// per-column minimum i of that warp covers column 32w + i of every tile, so
// the minima and the threshold do not depend on the width, nor on the work
// layout.
template <int BN>
__device__ __forceinline__ int units_per_pass(int nts)
{
    return BN == 256 ? (nts + 1) >> 1 : nts;
}

// A CTA's units of an item of U units a pass: PASS 0 all of them twice (unit k
// is unit k or k - U of the pass), else its part's, from u0.
template <int PASS>
__device__ __forceinline__ int span_of(int U, int idx, const irc_tc::SplitOut &sp, int &u0)
{
    u0 = 0;
    if (PASS == 0) return 2 * U;
    const int part = idx % sp.parts;
    u0 = U * part / sp.parts;
    return U * (part + 1) / sp.parts - u0;
}

template <int PASS>
__device__ __forceinline__ const irc_tc::TcItem &item_of(const irc_tc::TcItem *items, int idx, const irc_tc::SplitOut &sp)
{
    return items[PASS == 0 ? idx : idx / sp.parts];
}

// The MMA issuer of unit k (both passes counted) of slot s: alternate units of
// a one-slot item, whose accumulators alternate too, alternate slots else.  A
// slot's unit count over both passes is even, so an accumulator stays with
// its issuer from item to item.
template <int NS>
__device__ __forceinline__ int issuer_of(int k, int s)
{
    static_assert(MMA_WARPS == 2, "two issuers");
    return (NS == 1 ? k : s) & 1;
}

// A wait of the filter's pipeline (see sm100::mbar_wait), bounded by the
// poll limit set with irc_set_wait_limit.  One non-blocking test first: the
// producer's and the MMA threads' waits mostly find their phase complete, and
// a bare test costs a fraction of the bounded loop (147 cycles for a complete
// phase).  The loop then starts with try_wait (no more probes): a probing warp
// would take issue slots from the epilogue warps sharing its scheduler.  A
// limit below 64 polls makes every poll a non-blocking test, so such a limit
// gives up at the first phase that is not already complete (how the tests
// force the timeout path).
__device__ __forceinline__ bool pipe_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    if (sm100::mbar_test_wait(bar, parity)) return true;
    const uint32_t lim = c_wait_polls;
    return sm100::mbar_wait(bar, parity, abort_flag, lim, lim < 64u ? lim : 0u);
}

// The same by a whole warp: one answer for all lanes.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    return __all_sync(0xffffffffu, pipe_wait(bar, parity, abort_flag));
}

__device__ __forceinline__ double dist2_f64(const float *__restrict__ b, const float *__restrict__ a, int nd)
{
    double acc = 0.0;
    for (int c = 0; c < nd; ++c) {
        const double d = (double)__ldg(b + c) - (double)__ldg(a + c);
        acc = __dadd_rn(acc, __dmul_rn(d, d));
    }
    return acc;
}

// Exact re-rank of the cL candidates listed for query q (list[0 .. cL)),
// warp-cooperative; o = q - q_base.  Requires knn <= 32.  Candidate e is
// lane e % 32 of round e / 32, and every lane gathers its own rows.  nC is
// the row stride of F; nd <= nC the features that can be non-zero for this
// query and its candidates (the width of their site): the rest are zero in
// both rows and add exactly 0 to every distance, so they are skipped.
template <int PER>
__device__ __forceinline__ void rerank(const uint32_t *__restrict__ list, int cL, bool complete, int q,
                                       const float *__restrict__ F, const float4 *__restrict__ Fp, int Dp4,
                                       float4 *__restrict__ qs, int nC, int nd, int knn, size_t o,
                                       unsigned long long *ws, int lane, int margin, int *miKnn, float *d2Knn,
                                       float *vrKnn, float *rho, int *scratch)
{
    const float *a = F + (size_t)q * nC;
    unsigned long long kv[PER];
    irc_rr::list_keys<PER>(list, cL, Fp, Dp4, q, qs, nd, lane, kv);
    // A list cut by tau that holds fewer than knn + margin positive distances
    // (exact copies of the query, at distance 0 and excluded like the
    // reference's d > 0 test, crowded the threshold) may miss nearer
    // distinct candidates: such a query goes to the exact fallback.
    if (!complete) {
        unsigned nv = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) nv += kv[i] != ~0ull;
        if (__reduce_add_sync(0xffffffffu, nv) < (unsigned)(knn + margin)) {
            if (lane == 0) {
                const int k = atomicAdd(scratch + 0, 1);
                scratch[irc::kScratchLists + k] = q;
            }
            return;
        }
    }
    // ws[0 .. WARP_KEYS) <- the smallest keys, ascending; if more than
    // WARP_KEYS pass the selection's bound, the full sort runs
    unsigned tb;
    if (irc_rr::select_keys<PER>(kv, knn, ws, lane, tb) > WARP_KEYS) {
        irc_rr::warp_bitonic<unsigned long long, PER>(kv, lane);
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane * PER + i < WARP_KEYS) ws[lane * PER + i] = kv[i];
    }
    __syncwarp();
    // boundary band: keys within 16 ulps of the k-th distance, ordered by FP64
    const unsigned long long kk = ws[knn - 1];
    int lo = knn - 1, hi = knn;
    if (kk != ~0ull) {
        const float vk = __uint_as_float((unsigned)(kk >> 32));
        const float tol = vk * 0x1p-19f;
        unsigned mlo = 0xffffffffu, mhi = 0u;
#pragma unroll
        for (int i = 0; i < WARP_KEYS / 32; ++i) {
            const int e = lane + 32 * i;
            const unsigned long long k = ws[e];
            if (k != ~0ull && fabsf(__uint_as_float((unsigned)(k >> 32)) - vk) <= tol) {
                mlo = min(mlo, (unsigned)e);
                mhi = max(mhi, (unsigned)e + 1u);
            }
        }
        lo = (int)__reduce_min_sync(0xffffffffu, mlo);
        hi = (int)__reduce_max_sync(0xffffffffu, mhi);
    }
    const int nb = hi - lo;
    if (nb > 1 && nb <= 32) {
        // lanes j < nb hold band element lo + j; rank them by (FP64 distance, index)
        const unsigned long long kb = lane < nb ? ws[lo + lane] : ~0ull;
        const int ib = (int)(kb & 0xffffffffu);
        const double db = lane < nb ? dist2_f64(F + (size_t)ib * nC, a, nd) : 0.0;
        int rank = 0;
        for (int m = 0; m < nb; ++m) {
            const double dm = __shfl_sync(0xffffffffu, db, m);
            const int im = __shfl_sync(0xffffffffu, ib, m);
            rank += (dm < db || (dm == db && im < ib)) ? 1 : 0;
        }
        if (lane < nb && lo + rank < knn) emit(lo + rank, kb, q, knn, o, miKnn, d2Knn, vrKnn, rho);
        for (int e = lane; e < lo && e < knn; e += 32) emit(e, ws[e], q, knn, o, miKnn, d2Knn, vrKnn, rho);
    } else {
        for (int e = lane; e < knn; e += 32) emit(e, ws[e], q, knn, o, miKnn, d2Knn, vrKnn, rho);
    }
    __syncwarp();
}

__device__ __forceinline__ void slot_barrier(int slot, int nthreads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(nthreads) : "memory");
}

constexpr int TILE = 128;

__device__ __forceinline__ int chunk_tiles(const irc::PlanDev &p, int chunk)
{
    if (chunk < 0) return 0;
    int n = 0;
    for (int r = __ldg(p.roff + chunk); r < __ldg(p.roff + chunk + 1); ++r) n += (__ldg(p.rn + r) + TILE - 1) / TILE;
    return n;
}

// The accumulator goes back to the MMA issuer as soon as this warp's values
// are in registers: the rest of the unit's work then overlaps the next MMAs.
__device__ __forceinline__ void release_acc(uint64_t *empty, int lane)
{
    sm100::tc_fence_before();
    __syncwarp();
    if (lane == 0) sm100::mbar_arrive(empty);
}

// Pass 1 of one warp and 128-tile (BN = 128): fold its 32 columns (taddr:
// the first) into the per-column minima; lim = valid columns of the 32.
__device__ __forceinline__ void fold32(uint32_t taddr, int lim, uint64_t *empty, int lane, float (&bm)[PART])
{
    uint32_t x[16], y[16];
    sm100::tmem_ld16_nowait(taddr, x);
    sm100::tmem_ld16_nowait(taddr + 16, y);
    sm100::tmem_wait_ld(x, y);
    release_acc(empty, lane);
    if (lim >= 32) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            bm[i] = fminf(bm[i], __uint_as_float(x[i]));
            bm[16 + i] = fminf(bm[16 + i], __uint_as_float(y[i]));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i < lim) bm[i] = fminf(bm[i], __uint_as_float(x[i]));
            if (16 + i < lim) bm[16 + i] = fminf(bm[16 + i], __uint_as_float(y[i]));
        }
    }
}

// Pass 1 of one warp and 256-wide unit: its 32 columns of both 128-tiles
// (ta, tb: the first column of each; la, lb: valid columns) folded into the
// same minima with three-input mins.
__device__ __forceinline__ void fold2x32(uint32_t ta, int la, uint32_t tb, int lb, uint64_t *empty, int lane,
                                         float (&bm)[PART])
{
    const float inf = __int_as_float(0x7f800000);
#pragma unroll
    for (int r = 0; r < 2; ++r) {                 // minima 16r .. 16r + 15
        uint32_t x[16], y[16];
        sm100::tmem_ld16_nowait(ta + 16 * r, x);
        sm100::tmem_ld16_nowait(tb + 16 * r, y);
        sm100::tmem_wait_ld(x, y);
        if (r == 1) release_acc(empty, lane);
        if (la >= 32 && lb >= 32) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                bm[16 * r + i] = sm100::fmin3(bm[16 * r + i], __uint_as_float(x[i]), __uint_as_float(y[i]));
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                bm[16 * r + i] = sm100::fmin3(bm[16 * r + i], 16 * r + i < la ? __uint_as_float(x[i]) : inf,
                                              16 * r + i < lb ? __uint_as_float(y[i]) : inf);
        }
    }
}

__device__ __forceinline__ unsigned lim_mask(int lim)
{
    return lim >= 32 ? 0xffffffffu : lim <= 0 ? 0u : (1u << lim) - 1u;
}

// Pass 2 of one warp and 128-tile: the mask of its 32 columns at or below
// tau, limited to the lim valid columns.
__device__ __forceinline__ unsigned mark_regs(const uint32_t (&x)[16], const uint32_t (&y)[16], int lim, float tau)
{
    // four independent partial masks: short dependency chains
    unsigned a0 = 0u, a1 = 0u, a2 = 0u, a3 = 0u;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        if (__uint_as_float(x[i]) <= tau) a0 |= 1u << i;
        if (__uint_as_float(x[i + 1]) <= tau) a1 |= 1u << (i + 1);
        if (__uint_as_float(y[i]) <= tau) a2 |= 1u << (16 + i);
        if (__uint_as_float(y[i + 1]) <= tau) a3 |= 1u << (17 + i);
    }
    return ((a0 | a1) | (a2 | a3)) & lim_mask(lim);
}

// Bit c of the result = sign bit of v[c], one funnel shift per value in two
// independent chains.  (Half of the values through the carry of an add, on the
// other pipe, measured 1.6 times the rate alone and 1% slower here.)
__device__ __forceinline__ unsigned signs16(const uint32_t (&v)[16])
{
    unsigned c0 = 0u, c1 = 0u;                    // values 0-7, 8-15
#pragma unroll
    for (int i = 7; i >= 0; --i) {
        c0 = __funnelshift_l(v[i], c0, 1);
        c1 = __funnelshift_l(v[8 + i], c1, 1);
    }
    return c0 | (c1 << 8);
}

// Pass 2 of one warp and unit: the masks of its 32 columns of each tile (the
// second of a 256-wide unit) that are hits, limited to the valid columns.
// Every value is loaded before the accumulator is released; SIGNS: the
// threshold is folded into the MMA (accumulators d2 - tau), a hit is a sign bit.
template <int BN, bool SIGNS>
__device__ __forceinline__ void mark(uint32_t ta, int la, uint32_t tb, int lb, float tau, uint64_t *empty, int lane,
                                     unsigned &ma, unsigned &mb)
{
    uint32_t x[2][16], y[2][16];                  // columns 16r .. 16r + 15 of the two tiles
    sm100::tmem_ld16_nowait(ta, x[0]);
    sm100::tmem_ld16_nowait(ta + 16, x[1]);
    if constexpr (BN == 256) {
        sm100::tmem_ld16_nowait(tb, y[0]);
        sm100::tmem_ld16_nowait(tb + 16, y[1]);
    }
    sm100::tmem_wait_ld(x[0], x[1]);
    if constexpr (BN == 256) sm100::tmem_wait_ld(y[0], y[1]);
    release_acc(empty, lane);
    if constexpr (SIGNS) ma = (signs16(x[0]) | (signs16(x[1]) << 16)) & lim_mask(la);
    else ma = mark_regs(x[0], x[1], la, tau);
    if constexpr (BN == 256) {
        if constexpr (SIGNS) mb = (signs16(y[0]) | (signs16(y[1]) << 16)) & lim_mask(lb);
        else mb = mark_regs(y[0], y[1], lb, tau);
    }
}

// The pass-2 threshold of query row `row` into the query tile in shared
// memory: -tau' split into three BF16 (exactly) or F16 terms (to 2^-25
// absolute) at K positions tau_k ..
// tau_k + 2, against 1, 1, 1 in every candidate row, so the pass-2
// accumulators are d2 - tau'.  tau' = tau (1 + 2^-10), capped at 1e30 (F16:
// 60000; a cap that cuts is in the record of the proof, F16_TAU_MAX): the
// small margin keeps every candidate at or below tau negative whatever the
// rounding of the extra terms.  The tile is 128-byte swizzled: the 16-byte
// piece c of row r sits at piece c ^ (r % 8).
template <Fmt FMT>
__device__ __forceinline__ void put_tau(uint8_t *sA, int row, int tau_k, float tau)
{
    const float x = -fminf(tau * (1.0f + 0x1p-10f), FMT == Fmt::f16 ? 60000.0f : 1e30f);
    uint16_t v[3];
    float rem = x;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        if (FMT == Fmt::f16) {
            const __half h = __float2half_rn(rem);
            rem -= __half2float(h);
            v[t] = __half_as_ushort(h);
        } else {
            const __nv_bfloat16 h = __float2bfloat16_rn(rem);
            rem -= __bfloat162float(h);
            v[t] = __bfloat16_as_ushort(h);
        }
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int k = tau_k + t;
        *reinterpret_cast<uint16_t *>(sA + (size_t)row * 128 + (((k >> 3) ^ (row & 7)) << 4) + (k & 7) * 2) = v[t];
    }
}

// Append the hits of a unit's two 32-column masks (entries ca + bit, cb + bit)
// to the query's pooled list (its four epilogue warps share it): one
// shared-memory atomic reserves the room; entries past LISTCAP are dropped,
// and a count past it sends the query to the exact fallback.  (A share per
// warp with the count in a register measured the same.)
template <class E>
__device__ __forceinline__ void append_hits(E *lrow, int *cnt, unsigned ma, uint32_t ca, unsigned mb, uint32_t cb)
{
    if (!(ma | mb)) return;
    int e = atomicAdd(cnt, __popc(ma) + __popc(mb));
#pragma unroll 1
    while (ma | mb) {
        const bool first = ma != 0u;
        const unsigned m = first ? ma : mb;
        if (e < LISTCAP) lrow[e] = (E)((first ? ca : cb) + (uint32_t)(__ffs(m) - 1));
        ++e;
        if (first) ma &= ma - 1u;
        else mb &= mb - 1u;
    }
}

// Named barrier 1 + slot over the slot's epilogue warps that also returns the
// AND of v over them: every warp of the slot gets the same answer, so they
// leave the item loop together (a warp that left alone would leave the others
// waiting at the slot's next barrier).
__device__ __forceinline__ bool slot_barrier_and(int slot, int nthreads, bool v)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(1 + slot), "r"(nthreads)
        : "memory");
    return r != 0;
}

// The handoff of one item's lists to the re-rank kernel: this warp packs 8 of
// its quarter's queries (query L in lane L) into one bump allocation and
// records (offset, length) per query; a list past LISTCAP or a full list area
// sends the query to the exact fallback instead.
template <class T>
__device__ __forceinline__ void hand_off(const irc::PlanDev &p, const irc_tc::TcItem &it, int s, int quarter, int part,
                                         int qrow, int nq_s, const int2 *__restrict__ tl, const unsigned char *lists, const int *sCnt,
                                         const float *sTau, const irc_tc::ListOut &lo, int *scratch, int lane)
{
    constexpr int RL = 32 / PARTS;
    int cL = -1;                                  // -1: no query in this lane, -2: to the fallback
    if (lane < RL && qrow + part * RL + lane < nq_s) {
        const int t = sCnt[quarter * 32 + part * RL + lane];
        cL = t > LISTCAP ? -2 : t;
    }
    const unsigned len = cL > 0 ? (unsigned)cL : 0u;
    unsigned incl = len;
#pragma unroll
    for (int d = 1; d < RL; d <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    const unsigned total = __shfl_sync(0xffffffffu, incl, RL - 1);
    unsigned base = 0;
    if (lane == 0 && total) base = atomicAdd(lo.count, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    const bool fits = (unsigned long long)base + total <= (unsigned long long)lo.cap;
    if (lane < RL && cL != -1) {
        const int q = it.qs[s] + qrow + part * RL + lane;
        if (lo.cert)                              // the list's bound and its chunk, for the proof of completeness
            lo.cert[q - p.q_base] = make_int2(__float_as_int(fminf(sTau[quarter * 32 + part * RL + lane], irc_tc::F16_TAU_MAX)), it.chunk[s]);
        if (cL == -2 || !fits) {
            if (!lo.cert) {                       // (with the record above, its tile is searched again)
                const int k = atomicAdd(scratch + 0, 1);
                scratch[irc::kScratchLists + k] = q;
            }
        } else {
            // bit 30: the list holds every candidate of the chunk (nothing was cut by tau)
            const int complete = cL == __ldg(p.ncand + it.chunk[s]) ? (1 << 30) : 0;
            lo.qinfo[q - p.q_base] = make_int2((int)(base + incl - len), cL | complete);
        }
    }
    if (!fits) return;
#pragma unroll 1
    for (int L = 0; L < RL; ++L) {
        const int n = __shfl_sync(0xffffffffu, cL, L);
        const unsigned off = base + __shfl_sync(0xffffffffu, incl - len, L);
        if (n <= 0) continue;                     // warp-uniform
        const typename T::Entry *lr = T::row(lists, quarter, part * RL + L);
        for (int e = lane; e < n; e += 32) {
            const uint32_t v = lr[e];
            lo.lists[off + e] = sizeof(typename T::Entry) == 4 ? v : (uint32_t)__ldg(tl + (v >> 7)).x + (v & 127u);
        }
    }
}

// The same for a part of a split item: its entries go behind the other parts'
// in the query's list row; k_publish records the lists.
template <class T>
__device__ __forceinline__ void hand_off_part(const irc::PlanDev &p, const irc_tc::TcItem &it, int item, int piece, int quarter,
                                              int part, int qrow, int nq_s, const int2 *__restrict__ tl,
                                              const unsigned char *lists, const int *sCnt, const float *sTau,
                                              const irc_tc::ListOut &lo, int lane)
{
    constexpr int RL = 32 / PARTS;
    const int row = quarter * 32 + part * RL + lane;              // (lanes < RL: the warp's queries)
    int n = 0, base = 0;
    if (lane < RL && qrow + part * RL + lane < nq_s) {
        n = sCnt[row];
        if (n) base = atomicAdd(lo.split.cnt + item * BM + row, n);
        if (lo.cert && piece == 0) lo.cert[it.qs[0] + row - p.q_base] = make_int2(__float_as_int(fminf(sTau[row], irc_tc::F16_TAU_MAX)), it.chunk[0]);
        if (n > LISTCAP || base + n > LISTCAP) n = 0;             // (the count, past LISTCAP, tells)
    }
#pragma unroll 1
    for (int L = 0; L < RL; ++L) {
        const int m = __shfl_sync(0xffffffffu, n, L), b = __shfl_sync(0xffffffffu, base, L);
        const typename T::Entry *lr = T::row(lists, quarter, part * RL + L);
        uint32_t *out = lo.lists + lo.split.area + (size_t)(item * BM + quarter * 32 + part * RL + L) * LISTCAP + b;
        for (int e = lane; e < m; e += 32) {
            const uint32_t v = lr[e];
            out[e] = sizeof(typename T::Entry) == 4 ? v : (uint32_t)__ldg(tl + (v >> 7)).x + (v & 127u);
        }
    }
}

// Shared state of a persistent filter CTA: the item ring (the producer claims
// items from the launch's work queue and publishes their indices), the
// double-buffered query tile and the mbarriers of every stage.
struct Shared {
    uint8_t *sA;                                  // two query tiles, A_BYTES each
    uint8_t *sB;                                  // candidate stages
    unsigned char *lists;                         // list rows, QUARTER_BYTES a lane quarter
    float *sTau;                                  // [BM]
    int *sCnt;                                    // [BM] list counts
    uint64_t *full, *empty;                       // [MMA_WARPS][STAGES] a unit loaded (per issuer), [STAGES] stage consumed
    uint64_t *a_full, *a_empty;                   // [2] query tile loaded / its item's MMAs done
    uint64_t *acc_full, *acc_empty;               // [NBUF] accumulator written / read
    uint64_t *tau_ready;                          // [4] a slot's thresholds are in its query tile
    uint64_t *item_full, *item_empty;             // [2] item index published / read by every consumer
    uint64_t *mma_done;                           // [MMA_WARPS]
    int *item_idx;                                // [2]
    uint32_t *tmem_slot;
    volatile int *abort_flag;
};

// Epilogue of one warp: lane quarter `quarter` (the TMEM lanes it may read)
// and part `part` (columns 32 * part .. 32 * part + 31 of every 128-tile of
// its slot), over the items the CTA takes.  Each slot's epilogue warps
// synchronise only among themselves (named barrier 1 + slot).  Unit g of a
// slot (counted over all its items, both passes) goes to accumulator
// s * BPS + g % BPS, whose barriers are in phase g / BPS.
template <int BN, int NS, Fmt FMT, bool TAU, bool BIG, int PASS>
__device__ __forceinline__ void epilogue(const irc::PlanDev &p, const irc_tc::TcItem *__restrict__ items, int rank,
                                         uint32_t tmem, int tau_k, const Shared &sh, const irc_tc::ListOut &lo,
                                         int *scratch, int warp, int lane)
{
    using T = Tile<BN, BIG>;
    constexpr int QPS = 4 / NS;                   // lane quarters per slot
    constexpr int BPS = T::NBUF / NS;             // accumulator buffers per slot
    const int ew = warp - 2;                      // 0..15
    const int quarter = warp & 3;                 // TMEM lane quarter this warp may access
    const int part = ew >> 2;                     // its 32 columns of every 128-tile
    const int s = quarter / QPS;                  // slot of this lane quarter
    const int qrow = (quarter % QPS) * 32;        // first row of this quarter inside its slot
    const int slot_threads = 32 * PARTS * QPS;
    const int row = quarter * 32 + lane;
    const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + part * PART;
    // the minima rows of a quarter alias that quarter's own list rows
    float *qarea = reinterpret_cast<float *>(sh.lists + quarter * T::QUARTER_BYTES);
    typename T::Entry *lrow = const_cast<typename T::Entry *>(T::row(sh.lists, quarter, lane));
    unsigned g0 = 0;                              // this slot's units of the earlier items
    for (int seq = 0;; ++seq) {
        const int r = seq & 1;
        bool ok = pipe_wait(&sh.item_full[r], (seq >> 1) & 1, sh.abort_flag);
        if (!slot_barrier_and(s, slot_threads, ok)) break;
        const int idx = sh.item_idx[r];
        __syncwarp();
        if (lane == 0) sm100::mbar_arrive(&sh.item_empty[r]);
        if (idx < 0) break;                       // the queue is empty
        const irc_tc::TcItem it = item_of<PASS>(items, idx, lo.split);
        const int nq_s = it.chunk[s] >= 0 ? it.nq[s] : 0;
        const int nts = chunk_tiles(p, it.chunk[s]);
        const bool active = qrow < nq_s;          // warp-uniform: any valid query in this quarter
        const int U = units_per_pass<BN>(nts);
        int u0;
        const int K = span_of<PASS>(U, idx, lo.split, u0);
        const int K1 = PASS == 0 ? U : PASS == 1 ? K : 0;      // units of pass 1
        // the slot's tile list: unit u is tile u (BN = 128) or tiles 2u, 2u + 1
        // (BN = 256; the second is (0, 0) past the end of an odd count)
        const int2 *tl = nts ? p.tc_tiles + __ldg(p.tc_toff + it.chunk[s]) : p.tc_tiles;

        // Unit k of the two passes: (first row, columns) of its tile(s), loaded
        // one unit ahead of its use.
        auto load_unit = [&](int k) -> int4 {
            const int u = PASS ? u0 + k : k < U ? k : k - U;
            if constexpr (BN == 256) {
                return __ldg(reinterpret_cast<const int4 *>(tl) + u);
            } else {
                const int2 v = __ldg(tl + u);
                return make_int4(v.x, v.y, 0, 0);
            }
        };
        int4 cu = K ? load_unit(0) : make_int4(0, 0, 0, 0);
        // this warp's columns of the unit: first rows ra, rb and valid counts
        // na, nb of its 32 columns in each tile (none: <= 0)
        auto unit = [&](int k, int &ra, int &na, int &rb, int &nb) {
            const int4 nx = load_unit(k + 1 < K ? k + 1 : k);
            ra = cu.x;
            na = cu.y - part * PART;
            rb = cu.z;
            nb = cu.w - part * PART;
            cu = nx;
        };

        // pass 1: per-column minima of this warp's columns
        float bm[PART];
#pragma unroll
        for (int c = 0; c < PART; ++c) bm[c] = __int_as_float(0x7f800000);
        for (int k = 0; k < K1 && ok; ++k) {
            int ra, na, rb, nb;
            unit(k, ra, na, rb, nb);
            const unsigned g = g0 + (unsigned)k;
            const int b = s * BPS + (int)(g % BPS);
            if (!(ok = pipe_wait(&sh.acc_full[b], (g / BPS) & 1, sh.abort_flag))) break;
            sm100::tc_fence_after();
            uint64_t *empty = &sh.acc_empty[b];
            // (either tile may be the short one: the first when it ends a run)
            if (active && (na > 0 || nb > 0)) {
                if constexpr (BN == 256) fold2x32(tbase + b * BN, na, tbase + b * BN + 128, nb, empty, lane, bm);
                else fold32(tbase + b * BN, na, empty, lane, bm);
            } else {
                release_acc(empty, lane);
            }
        }
        // a part's minima meet the other parts' in global memory
        if constexpr (PASS != 0) {
            int *cm = lo.split.colmin + ((size_t)(idx / lo.split.parts) * 128 + part * PART) * BM + row;
#pragma unroll
            for (int c = 0; c < PART; ++c) {
                if (PASS == 1) {
                    if (active && bm[c] < FLT_MAX) atomicMin(cm + c * BM, __float_as_int(fmaxf(bm[c], 0.0f)));
                } else {
                    const int v = __ldg(cm + c * BM);
                    bm[c] = __int_as_float(v < 0x7f7f7f7f ? v : 0x7f800000);
                }
            }
        }
        // threshold: rank-th smallest of the 128 column minima of every query
        if constexpr (PASS != 1) {
            float *brow = qarea + lane * BROW + part * PART;
#pragma unroll
            for (int c = 0; c < PART; ++c) brow[c] = fmaxf(bm[c], 0.0f);
            if (part == 0) sh.sCnt[row] = 0;      // list counts of pass 2 (ordered by the barriers below)
            slot_barrier(s, slot_threads);
            // The warp's 8 rows at once (independent chains): a bitwise
            // search, from the top, of the largest t with fewer than rank
            // minima below it, i.e. of the rank-th smallest minimum, on the
            // non-negative float bit patterns.  It stops at bit lowb and
            // rounds up, so tau is an upper bound of the rank-th smallest
            // within 2^-(lowb - 1) relative of it (a few more candidates
            // listed, never fewer).  The search is a fixed cost per item,
            // the extra candidates a cost per tile: slots of at most 16
            // tiles stop 4 bits earlier (2^-7), longer ones search to 2^-11.
            constexpr int RL = 32 / PARTS;
            unsigned v4[RL][4], ans[RL];
#pragma unroll
            for (int L = 0; L < RL; ++L) {
                const float *bl = qarea + (part * RL + L) * BROW;
#pragma unroll
                for (int u = 0; u < 4; ++u) v4[L][u] = __float_as_uint(bl[u * 32 + lane]);
                ans[L] = 0u;
            }
            const int lowb = nts <= 16 ? TAU_LOW_BIT + 4 : TAU_LOW_BIT;   // uniform over the slot
            // bits above the highest one in which any two minima of the warp's
            // rows differ are common to every answer: start below them
            unsigned lo_v = 0xffffffffu, hi_v = 0u;
#pragma unroll
            for (int L = 0; L < RL; ++L)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    lo_v = min(lo_v, v4[L][u]);
                    hi_v = max(hi_v, v4[L][u]);
                }
            lo_v = __reduce_min_sync(0xffffffffu, lo_v);
            hi_v = __reduce_max_sync(0xffffffffu, hi_v);
            const int top = min(30, 31 - __clz((lo_v ^ hi_v) | 1u));
#pragma unroll
            for (int L = 0; L < RL; ++L) ans[L] = lo_v & ~((2u << top) - 1u);
#pragma unroll 1
            for (int b = top; b >= lowb; --b) {
#pragma unroll
                for (int L = 0; L < RL; ++L) {
                    const unsigned t = ans[L] | (1u << b);
                    const unsigned c = (unsigned)(v4[L][0] < t) + (unsigned)(v4[L][1] < t) +
                                       (unsigned)(v4[L][2] < t) + (unsigned)(v4[L][3] < t);
                    if (__reduce_add_sync(0xffffffffu, c) < (unsigned)rank) ans[L] = t;
                }
            }
            if (lane < RL) {
                unsigned a = ans[0];
#pragma unroll
                for (int L = 1; L < RL; ++L)
                    if (lane == L) a = ans[L];
                sh.sTau[quarter * 32 + part * RL + lane] =
                    __uint_as_float(min(a | ((1u << lowb) - 1u), 0x7f800000u));
            }
            slot_barrier(s, slot_threads);        // minima rows are read; the list rows may be written
        }
        const float tau = PASS == 1 ? 0.0f : sh.sTau[row];
        if (TAU && PASS != 1 && part == 0 && K > 0) {
            // the thresholds into the item's query tile; visible to the tensor
            // core (async proxy) before the MMA thread, released by tau_ready,
            // issues the slot's pass-2 MMAs (one phase per item with units).
            // Accumulators of pass 1 show that the tile has landed; where pass 1
            // was another launch, its load is waited for here: landing later, it
            // would put the rows' zeros over the thresholds.
            if (PASS == 2) ok = warp_wait(&sh.a_full[r], (seq >> 1) & 1, sh.abort_flag) && ok;
            put_tau<FMT>(sh.sA + (size_t)r * A_BYTES, row, tau_k, tau);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&sh.tau_ready[s]);
        }
        // pass 2: collect the candidates at or below tau
        for (int k = K1; k < K && ok; ++k) {
            int ra, na, rb, nb;
            unit(k, ra, na, rb, nb);
            const unsigned g = g0 + (unsigned)k;
            const int b = s * BPS + (int)(g % BPS);
            if (!(ok = pipe_wait(&sh.acc_full[b], (g / BPS) & 1, sh.abort_flag))) break;
            sm100::tc_fence_after();
            uint64_t *empty = &sh.acc_empty[b];
            if (active && (na > 0 || nb > 0)) {
                unsigned ma = 0u, mb = 0u;
                mark<BN, BN == 256 && TAU>(tbase + b * BN, na, tbase + b * BN + 128, nb, tau, empty, lane, ma, mb);
                // entries: rows, or (place of the tile in the list, column)
                const uint32_t ea = BIG ? (uint32_t)ra : (uint32_t)((PASS ? u0 + k : k - U) * (BN / 128)) << 7;
                const uint32_t eb = BIG ? (uint32_t)rb : ea + 128u;
                append_hits(lrow, sh.sCnt + row, ma, ea + part * PART, mb, eb + part * PART);
            } else {
                release_acc(empty, lane);
            }
        }
        slot_barrier(s, slot_threads);
        if (PASS == 2 && __all_sync(0xffffffffu, ok))
            hand_off_part<T>(p, it, idx / lo.split.parts, idx % lo.split.parts, quarter, part, qrow, nq_s, tl, sh.lists, sh.sCnt,
                             sh.sTau, lo, lane);
        if (PASS == 0 && __all_sync(0xffffffffu, ok)) hand_off<T>(p, it, s, quarter, part, qrow, nq_s, tl, sh.lists, sh.sCnt, sh.sTau, lo, scratch, lane);
        g0 += (unsigned)K;
        // every warp of the slot is done with this item's lists before the
        // next item's minima overwrite them; after a timed-out wait all stop
        if (!slot_barrier_and(s, slot_threads, ok && !*sh.abort_flag)) break;
    }
}

// TMA producer (one warp): claims items from the launch's work queue and
// publishes their indices (a two-entry ring), loads each item's four 32-row
// query boxes into the free query tile, then the slots' units round-robin,
// each slot's sequence twice (both passes).  A unit's 128-candidate tiles land
// in consecutive 128-row halves of its stage, lane h loading half h from its
// tile's first row, which it fetched a unit ahead (the table lookup is off the
// path between a free stage and its loads).  Stage and tile counters run on
// across items, so the ring never drains between them.
template <int BN, int NS, bool BIG, int PASS>
__device__ __forceinline__ void produce(const CUtensorMap &tmQ, const CUtensorMap &tmC, const irc::PlanDev &p,
                                        const irc_tc::TcItem *__restrict__ items, int n_items, unsigned *queue,
                                        const Shared &sh, const irc_tc::SplitOut &sp, int lane)
{
    using T = Tile<BN, BIG>;
    constexpr int QPS = 4 / NS;
    constexpr int NH = BN / 128;                  // 128-tiles of a unit
    if (lane == 0) {
        sm100::prefetch_tmap(&tmQ);
        sm100::prefetch_tmap(&tmC);
    }
    int n_a = 0, n_w[MMA_WARPS] = {};             // query tiles loaded, units loaded for each issuer
    int st = 0;                                   // stage of the next unit
    uint32_t ph = 1;                              // parity of the stage's last release
    bool ok = true;
    for (int seq = 0; ok; ++seq) {
        const int r = seq & 1;
        unsigned claim = 0;
        if (PASS) {                               // (one: its unit count may be odd, which would move the next item's
            claim = seq == 0 ? blockIdx.x : (unsigned)n_items;             // accumulators to the other issuer)
        } else {
            if (lane == 0) claim = atomicAdd(queue, 1u);
            claim = __shfl_sync(0xffffffffu, claim, 0);
        }
        const int idx = claim < (unsigned)n_items ? (int)claim : -1;
        if (!(ok = warp_wait(&sh.item_empty[r], ((seq >> 1) & 1) ^ 1, sh.abort_flag))) break;
        if (lane == 0) {
            sh.item_idx[r] = idx;
            sm100::mbar_arrive(&sh.item_full[r]); // release: the index is visible to the waiters
        }
        if (idx < 0) break;
        const irc_tc::TcItem it = item_of<PASS>(items, idx, sp);
        const int2 *tl[NS];
        int U[NS], nt[NS], row[NS];               // row: this lane's tile of the slot's next unit
        int K[NS], u0[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            nt[s] = chunk_tiles(p, it.chunk[s]);
            U[s] = units_per_pass<BN>(nt[s]);
            tl[s] = nt[s] ? p.tc_tiles + __ldg(p.tc_toff + it.chunk[s]) : p.tc_tiles;
            K[s] = span_of<PASS>(U[s], idx, sp, u0[s]);
            const int t = u0[s] * NH + lane;
            row[s] = lane < NH && t < nt[s] ? __ldg(tl[s] + t).x : 0;
        }
        // the query tile of item seq - 2 is free once that item's MMAs are done
        if (!(ok = warp_wait(&sh.a_empty[r], ((seq >> 1) & 1) ^ 1, sh.abort_flag))) break;
        uint8_t *sA = sh.sA + (size_t)r * A_BYTES;
        if (lane == 0) sm100::mbar_arrive_expect_tx(&sh.a_full[r], A_BYTES);
        __syncwarp();
        if (lane < 4) {
            int row0 = 0;                         // query box `lane` of the tile
#pragma unroll
            for (int s = 0; s < NS; ++s)
                if (lane / QPS == s && it.chunk[s] >= 0) row0 = it.qs[s] + (lane % QPS) * 32;
            sm100::tma_load_2d(&tmQ, &sh.a_full[r], sA + lane * (A_BYTES / 4), 0, row0);
        }
        ++n_a;
        for (int k = 0; ok; ++k) {
            bool any = false;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                if (ok && k < K[s]) {
                    any = true;
                    const int u = PASS ? u0[s] + k : k < U[s] ? k : k - U[s];
                    const int w = issuer_of<NS>(k, s);
                    if ((ok = warp_wait(&sh.empty[st], ph, sh.abort_flag))) {
                        const int nh = BN == 256 && 2 * u + 1 >= nt[s] ? 1 : NH;
                        uint64_t *full = sh.full + w * T::STAGES + (w == 0 ? n_w[0] : n_w[1]) % T::STAGES;
                        if (lane == 0) sm100::mbar_arrive_expect_tx(full, nh * HALF_BYTES);
                        __syncwarp();
                        if (lane < nh)
                            sm100::tma_load_2d(&tmC, full,
                                               sh.sB + (size_t)st * T::STAGE_BYTES + lane * HALF_BYTES, 0, row[s]);
                        const int un = u + 1 < U[s] ? u + 1 : 0, t = un * NH + lane;
                        if (lane < NH && t < nt[s]) row[s] = __ldg(tl[s] + t).x;
#pragma unroll
                        for (int v = 0; v < MMA_WARPS; ++v) n_w[v] += v == w;
                        if (++st == T::STAGES) {
                            st = 0;
                            ph ^= 1u;
                        }
                    }
                }
            }
            if (!any) break;
        }
    }
    // every issued load has landed before the CTA exits
#pragma unroll
    for (int w = 0; w < MMA_WARPS; ++w)
        for (int j = (n_w[w] > T::STAGES ? n_w[w] - T::STAGES : 0); j < n_w[w]; ++j)
            sm100::mbar_drain(&sh.full[w * T::STAGES + j % T::STAGES], (j / T::STAGES) & 1);
    for (int j = (n_a > 2 ? n_a - 2 : 0); j < n_a; ++j) sm100::mbar_drain(&sh.a_full[j & 1], (j >> 1) & 1);
}

// MMA issuers (one thread of each of MMA_WARPS warps), in the producer's order,
// each its own units (issuer_of).  One thread alone was the pipeline's
// bound: its waits, the issue of the MMAs (which blocks for about as long as
// they run) and the commits took ~1,450 cycles a unit in series, against ~300
// of MMA time; two threads overlap one's waits with the other's MMAs.  Unit g
// of slot s (counted over the CTA's items) goes to accumulator s*BPS + g % BPS
// and is issued once every epilogue warp of the slot released unit g - BPS of
// that buffer; a buffer, and with it every phase of its barriers, belongs to
// one issuer, and so do the load barriers (a waiter that did not see every
// phase could take an old phase's parity for the one it waits for).  With TAU
// an issuer's first pass-2 unit of a slot in an item also waits until the
// slot's epilogue wrote the thresholds into the query tile (tau_ready[s], one
// phase per item in which the slot has units).  After an item's last unit each
// issuer's commit lets its MMAs free the query tile.
template <int BN, int NS, Fmt FMT, bool TAU, bool BIG, int PASS>
__device__ __forceinline__ void issue(const irc::PlanDev &p, const irc_tc::TcItem *__restrict__ items, int nk,
                                      uint32_t tmem, const Shared &sh, const irc_tc::SplitOut &sp, int w)
{
    using T = Tile<BN, BIG>;
    constexpr int BPS = T::NBUF / NS;
    // bf16 x bf16 or f16 x f16 (kind::f16, K = 16) or e4m3 x e4m3 (kind::f8f6f4, K = 32)
    // -> f32; either way one MMA consumes 32 bytes of every 128-byte operand row
    constexpr uint32_t idesc = FMT == Fmt::bf16 ? sm100::idesc_make(BM, BN, 1, 1) : sm100::idesc_make(BM, BN, 0, 0);
    unsigned g0[NS], taus[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) g0[s] = taus[s] = 0;
    int st = 0;                                   // stage of the next unit
    int fw = 0;                                   // this issuer's next load barrier, and its parity
    uint32_t ph = 0;
    bool ok = true;
    for (int seq = 0; ok; ++seq) {
        const int r = seq & 1;
        if (!(ok = pipe_wait(&sh.item_full[r], (seq >> 1) & 1, sh.abort_flag))) break;
        const int idx = sh.item_idx[r];
        sm100::mbar_arrive(&sh.item_empty[r]);
        if (idx < 0) break;
        const irc_tc::TcItem it = item_of<PASS>(items, idx, sp);
        int U[NS], K[NS];
        bool tau_wait[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            U[s] = units_per_pass<BN>(chunk_tiles(p, it.chunk[s]));
            int u0;
            K[s] = span_of<PASS>(U[s], idx, sp, u0);
            tau_wait[s] = TAU && PASS != 1;
        }
        if (!(ok = pipe_wait(&sh.a_full[r], (seq >> 1) & 1, sh.abort_flag))) break;
        sm100::tc_fence_after();
        const uint64_t adesc = sm100::sdesc_sw128(sm100::smem_u32(sh.sA + (size_t)r * A_BYTES));
        for (int k = 0; ok; ++k) {
            bool any = false;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                if (ok && k < K[s]) {
                    any = true;
                    if (issuer_of<NS>(k, s) == w) {
                        const unsigned g = g0[s] + (unsigned)k, use = g / BPS;
                        const int b = s * BPS + (int)(g % BPS);
                        // (the load is usually there long before the accumulator is free)
                        ok = pipe_wait(&sh.full[w * T::STAGES + fw], ph, sh.abort_flag) &&
                             (use == 0 || pipe_wait(&sh.acc_empty[b], (use - 1) & 1, sh.abort_flag));
                        if (++fw == T::STAGES) {
                            fw = 0;
                            ph ^= 1u;
                        }
                        // the slot's thresholds are in the query tile before its pass 2 (after the
                        // accumulator's wait: the slot's epilogue is then in this item, so no
                        // earlier phase of tau_ready is open)
                        if (TAU && ok && (PASS == 2 || k >= U[s]) && tau_wait[s]) {
                            tau_wait[s] = false;
                            ok = pipe_wait(&sh.tau_ready[s], taus[s] & 1, sh.abort_flag);
                        }
                        if (ok) {
                            sm100::tc_fence_after();
                            const uint64_t bdesc =
                                sm100::sdesc_sw128(sm100::smem_u32(sh.sB + (size_t)st * T::STAGE_BYTES));
#pragma unroll
                            for (int kk = 0; kk < KP / 16; ++kk)
                                if (kk >= nk)
                                    break;                // the rest of every operand row is zero
                                else if (FMT == Fmt::fp8)
                                    sm100::mma_f8(tmem + b * BN, adesc + 2 * kk, bdesc + 2 * kk, idesc, kk > 0 ? 1u : 0u);
                                else
                                    sm100::mma_f16(tmem + b * BN, adesc + 2 * kk, bdesc + 2 * kk, idesc, kk > 0 ? 1u : 0u);
                            sm100::mma_commit(&sh.acc_full[b]);
                            sm100::mma_commit(&sh.empty[st]);
                        }
                    }
                    if (++st == T::STAGES) st = 0;
                }
            }
            if (!any) break;
        }
        if (!ok) break;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            g0[s] += (unsigned)K[s];
            taus[s] += K[s] > 0 ? 1u : 0u;
        }
        sm100::mma_commit(&sh.a_empty[r]);        // this item's MMAs done: its query tile may be replaced
    }
    // every MMA of this thread has completed before TMEM is released
    sm100::mma_commit(sh.mma_done + w);
    sm100::mbar_drain(sh.mma_done + w, 0);
}

// The filter over the work items of one packing class (NS slots per item:
// one or two at BN = 256, four at BN = 128), persistent: each CTA takes items
// from the class's work queue (queue: its head, items cost-ordered) until it
// is empty.  TAU: pass 2 reads the signs of d2 - tau (the thresholds written
// into the query tile at K position tau_k), else it compares d2 with tau in
// the epilogue.  PASS: 0 both passes; 1 or 2 one pass of a part of an item's
// units (irc_tc::SplitOut), one (item, part) per CTA.
template <Fmt FMT, int BN, bool TAU, int NS, bool BIG, int PASS = 0>
__global__ void __launch_bounds__(THREADS, 1)
k_knn_tc(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmC, irc::PlanDev p,
         const irc_tc::TcItem *__restrict__ items, int n_items, unsigned *queue, int nk, int tau_k, irc_tc::ListOut lo,
         int *__restrict__ scratch)
{
    using T = Tile<BN, BIG>;
    constexpr int QPS = 4 / NS;
    extern __shared__ unsigned char smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    Shared sh;
    sh.sA = base;
    sh.sB = base + 2 * A_BYTES;
    sh.lists = sh.sB + T::STAGES * T::STAGE_BYTES;
    sh.sTau = reinterpret_cast<float *>(sh.lists + 4 * T::QUARTER_BYTES);
    sh.sCnt = reinterpret_cast<int *>(sh.sTau + BM);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sh.sCnt + BM);
    sh.full = bars;
    sh.empty = sh.full + MMA_WARPS * T::STAGES;
    sh.a_full = sh.empty + T::STAGES;
    sh.a_empty = sh.a_full + 2;
    sh.acc_full = sh.a_empty + 2;
    sh.acc_empty = sh.acc_full + T::NBUF;
    sh.tau_ready = sh.acc_empty + T::NBUF;
    sh.item_full = sh.tau_ready + 4;
    sh.item_empty = sh.item_full + 2;
    sh.mma_done = sh.item_empty + 2;
    sh.item_idx = reinterpret_cast<int *>(sh.mma_done + MMA_WARPS);
    sh.tmem_slot = reinterpret_cast<uint32_t *>(sh.item_idx + 2);
    sh.abort_flag = reinterpret_cast<volatile int *>(sh.tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MMA_WARPS * T::STAGES; ++s) sm100::mbar_init(&sh.full[s], 1);
        for (int s = 0; s < T::STAGES; ++s) sm100::mbar_init(&sh.empty[s], 1);
        for (int r = 0; r < 2; ++r) {
            sm100::mbar_init(&sh.a_full[r], 1);
            sm100::mbar_init(&sh.a_empty[r], MMA_WARPS);
            sm100::mbar_init(&sh.item_full[r], 1);
            sm100::mbar_init(&sh.item_empty[r], MMA_WARPS + EPI_WARPS);   // the MMA threads and every epilogue warp
        }
        for (int b = 0; b < T::NBUF; ++b) {
            sm100::mbar_init(&sh.acc_full[b], 1);
            sm100::mbar_init(&sh.acc_empty[b], PARTS * QPS);       // the slot's epilogue warps
        }
        for (int w = 0; w < MMA_WARPS; ++w) sm100::mbar_init(sh.mma_done + w, 1);
        for (int s = 0; s < 4; ++s) sm100::mbar_init(&sh.tau_ready[s], QPS);   // the slot's quarters' writers
        *sh.abort_flag = 0;
        sm100::fence_mbar_init();
    }
    if (warp == 1) sm100::tmem_alloc(sh.tmem_slot, TMEM_COLS);
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t tmem = *sh.tmem_slot;
    after_previous();

    if (warp == 0) {
        produce<BN, NS, BIG, PASS>(tmQ, tmC, p, items, n_items, queue, sh, lo.split, lane);
        __syncwarp();
    } else if (warp == 1 || warp == 2 + EPI_WARPS) {
        if (lane == 0) issue<BN, NS, FMT, TAU, BIG, PASS>(p, items, nk, tmem, sh, lo.split, warp == 1 ? 0 : 1);
        __syncwarp();
    } else {
        epilogue<BN, NS, FMT, TAU, BIG, PASS>(p, items, tau_rank(FMT), tmem, tau_k, sh, lo, scratch, warp, lane);
    }
    sm100::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        sm100::tc_fence_after();
        sm100::tmem_dealloc(tmem, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *sh.abort_flag) atomicExch(scratch + irc::kScratchErr, 1);
}

// The split items' lists: (offset, length) of every query, as hand_off.
__global__ void __launch_bounds__(BM) k_publish(irc::PlanDev p, const irc_tc::TcItem *__restrict__ items,
                                                irc_tc::ListOut lo, int *__restrict__ scratch)
{
    after_previous(lo.split.cnt);
    if (blockIdx.x == 0 && threadIdx.x == 0) irc::count_stat(p, irc::kStatSplits, gridDim.x);
    const irc_tc::TcItem &it = items[blockIdx.x];
    const int row = threadIdx.x, slot = blockIdx.x * BM + row;
    if (row >= it.nq[0]) return;
    const int q = it.qs[0] + row, n = lo.split.cnt[slot];
    if (n > LISTCAP) {
        if (!lo.cert) scratch[irc::kScratchLists + atomicAdd(scratch + 0, 1)] = q;
        return;
    }
    const int complete = n == __ldg(p.ncand + it.chunk[0]) ? (1 << 30) : 0;
    lo.qinfo[q - p.q_base] = make_int2((int)(lo.split.area + (unsigned)slot * LISTCAP), n | complete);
}

// Exact re-rank kernel: one warp per query of the plan, in query order (the
// queries of a chunk share their candidate rows, which stay in L1/L2 for the
// block's warps); queries without a list (qinfo.x < 0) belong to the exact
// fallback or to no chunk.
constexpr int RR_WARPS = 8;
// Bound by L1's data pipe (a gathered 32-byte sector is about a pass through
// it) and the latency of the gathers: 5 blocks a SM with some registers spilled
// (56 bytes of stores, 220 of loads a thread) measure 633 us for 400,000 queries
// of 61 entries of 33 features and 797 for 3,600 chunks' 625,000, 4 without 665
// and 844.

__global__ void __launch_bounds__(32 * RR_WARPS, 5)
k_rerank(const int2 *__restrict__ qinfo, const uint32_t *__restrict__ lists, int n_out, int q_base,
         const float *__restrict__ F, const float4 *__restrict__ Fp, int nC, const uint8_t *__restrict__ row_dims,
         int knn, float *__restrict__ vrKnn, float *__restrict__ rho, int *__restrict__ miKnn,
         float *__restrict__ d2Knn, int margin, int *__restrict__ scratch)
{
    after_previous(qinfo, lists, Fp);
    __shared__ __align__(16) unsigned long long wkeys[RR_WARPS * WARP_KEYS];
    __shared__ float4 qrows[RR_WARPS * QROW4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int o = blockIdx.x * RR_WARPS + warp;
    if (o >= n_out) return;
    const int2 qi = __ldg(qinfo + o);
    if (qi.x < 0) return;
    const int Dp4 = irc_tc::fp_row4(nC);
    const uint32_t *lst = lists + (unsigned)qi.x;
    const int cL = qi.y & 0x3fffffff, q = q_base + o;
    const int nd = row_dims ? min(nC, (int)__ldg(row_dims + q)) : nC;
    const bool complete = (qi.y >> 30) & 1;
    unsigned long long *ws = wkeys + warp * WARP_KEYS;
    float4 *qs = qrows + warp * QROW4;
    if (cL <= 64)
        rerank<2>(lst, cL, complete, q, F, Fp, Dp4, qs, nC, nd, knn, (size_t)o, ws, lane, margin, miKnn, d2Knn, vrKnn, rho,
                  scratch);
    else if (cL <= 128)
        rerank<4>(lst, cL, complete, q, F, Fp, Dp4, qs, nC, nd, knn, (size_t)o, ws, lane, margin, miKnn, d2Knn, vrKnn, rho,
                  scratch);
    else
        rerank<8>(lst, cL, complete, q, F, Fp, Dp4, qs, nC, nd, knn, (size_t)o, ws, lane, margin, miKnn, d2Knn, vrKnn, rho,
                  scratch);
}

}  // namespace

namespace irc_tc {

// Kernel timing (irc_profile_begin / irc_profile_end): three events per
// tensor-core call -- before the filter, between filter and re-rank, after
// the re-rank -- in a table created by irc_profile_begin.
static std::mutex g_prof_mu;
static std::vector<cudaEvent_t> g_prof_ev;
static int g_prof_used = 0, g_prof_on = 0;

static cudaEvent_t *profile_slot()
{
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (!g_prof_on || 3 * (g_prof_used + 1) > (int)g_prof_ev.size()) return nullptr;
    return &g_prof_ev[3 * g_prof_used++];
}

template <Fmt FMT, int BN, bool TAU, int NS>
static int launch_filter(const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, const irc_tc::TcItem *items,
                         int n_items, unsigned *queue, int nk, int tau_k, const ListOut &lo, int *scratch, cudaStream_t s)
{
    if (n_items <= 0) return IRC_OK;
    const bool big = pl->tc_max_tiles > MAX_SHORT_TILES;
    auto kern = big ? k_knn_tc<FMT, BN, TAU, NS, true> : k_knn_tc<FMT, BN, TAU, NS, false>;
    const int smem = (int)(big ? Tile<BN, true>::SMEM_BYTES : Tile<BN, false>::SMEM_BYTES);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(tensor core): launch attributes");
    // persistent: one CTA per SM (shared memory and TMEM allow one), each
    // taking items from the queue until it is empty
    const int grid = n_items < pl->sms ? n_items : pl->sms;
    launch_next(kern, grid, THREADS, smem, s, mq, mc, pl->dev, items, n_items, queue, nk, tau_k, lo, scratch);
    IRC_CHECK_LAUNCH("irc_site_knn(tensor core)");
    return IRC_OK;
}

// The items of lo.split: pass 1, pass 2, their lists published.
template <Fmt FMT>
static int launch_split(const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, const irc_tc::TcItem *items, int nk,
                        int tau_k, const ListOut &lo, int *scratch, cudaStream_t s)
{
    const bool big = pl->tc_max_tiles > MAX_SHORT_TILES;
    auto pass1 = big ? k_knn_tc<FMT, 256, true, 1, true, 1> : k_knn_tc<FMT, 256, true, 1, false, 1>;
    auto pass2 = big ? k_knn_tc<FMT, 256, true, 1, true, 2> : k_knn_tc<FMT, 256, true, 1, false, 2>;
    const int smem = (int)(big ? Tile<256, true>::SMEM_BYTES : Tile<256, false>::SMEM_BYTES);
    const SplitOut &sp = lo.split;
    cudaError_t e = cudaFuncSetAttribute(pass1, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(pass2, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(tensor core): split items");
    const int n = sp.items * sp.parts;
    launch_next(pass1, n, THREADS, smem, s, mq, mc, pl->dev, items, n, nullptr, nk, tau_k, lo, scratch);
    launch_next(pass2, n, THREADS, smem, s, mq, mc, pl->dev, items, n, nullptr, nk, tau_k, lo, scratch);
    launch_next(k_publish, sp.items, BM, 0, s, pl->dev, items, lo, scratch);
    IRC_CHECK_LAUNCH("irc_site_knn(tensor core) split items");
    return IRC_OK;
}

// The last one-slot items that leave SMs idle: n mod 152 of them take one more
// turn, as long as the longest of them (1.42 us a unit, D = 24).  Cut into parts that
// fill the machine they take two launches of a part's units and 57 us of their
// own (memory cleared, prologues, the threshold search after pass 1, lists
// published); 22 more than the launch they replace where they are all there
// is.  us a call, whole -> split: 20,000 spikes in one chunk (157 items of 79
// units) 302 -> 248, 21,000 273 -> 219, 60,001 in 30 chunks 675 -> 602,
// 100,003 in 50 1,007 -> 959; not kept where it loses: 3,000 (24 of 12 units)
// 71 -> 79, 8,000 (63 of 32, two parts) 100.5 -> 101.5.
static SplitOut split_of(const irc_plan *pl, int nC, Fmt fmt)
{
    SplitOut sp{};
    const int rest = pl->n_tc_one % pl->sms, units = (pl->tc_rest_tiles + 1) / 2;
    if (fmt == Fmt::fp8 || nC + 9 > KP || pl->tc_wide_bn == 128 || rest == 0) return sp;
    const int parts = std::min(pl->sms / rest, units / 4), saved = units - units / std::max(parts, 1);
    if (parts < 2 || saved < (pl->n_tc_one > pl->sms ? 34 : 20)) return sp;
    sp.items = rest;
    sp.parts = parts;
    return sp;
}

static size_t item_bytes(int items) { return (size_t)items * BM * (128 + 1 + LIST_ROW) * 4; }

size_t split_bytes(const irc_plan *pl, int nC, Fmt fmt) { return item_bytes(split_of(pl, nC, fmt).items); }

// (parts >= 2: at most half as many items as SMs; below 24 units nothing is saved)
size_t split_reserve(const irc_plan *pl)
{
    return (pl->tc_max_tiles + 1) / 2 < 24 ? 0 : item_bytes(pl->sms / 2);
}

void split_area(const irc_plan *pl, int nC, Fmt fmt, void *mem, ListOut *lo)
{
    SplitOut sp = split_of(pl, nC, fmt);
    if (!sp.items) return;
    sp.colmin = (int *)mem;
    sp.cnt = sp.colmin + (size_t)sp.items * BM * 128;
    uint32_t *rows = (uint32_t *)(sp.cnt + (size_t)sp.items * BM);
    const size_t at = (size_t)(rows - lo->lists);
    if (at + (size_t)sp.items * BM * LIST_ROW > (size_t)0x7fffff00) return;       // (offsets are int32)
    sp.area = (unsigned)at;
    lo->split = sp;
}

cudaError_t clear_lists(const ListOut &lo, int n_out, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(lo.qinfo, 0xff, (size_t)n_out * sizeof(int2), s);   // (-1, -1): no list
    if (e == cudaSuccess) e = cudaMemsetAsync(lo.count, 0, 4 * sizeof(unsigned), s);     // count, queue heads
    const SplitOut &sp = lo.split;
    if (e == cudaSuccess && sp.items) e = cudaMemsetAsync(sp.colmin, 0x7f, (size_t)sp.items * BM * 128 * 4, s);
    if (e == cudaSuccess && sp.items) e = cudaMemsetAsync(sp.cnt, 0, (size_t)sp.items * BM * 4, s);
    return e;
}

// The filter of every packing class of the plan on stream s.
int launch_filters(Fmt fmt, const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, int nC, const ListOut &lo,
                   int *scratch, cudaStream_t s)
{
    // BF16, F16: the pass-2 thresholds go into K positions nC + 6 .. nC + 8 of
    // the query rows when they fit (else, and for FP8, pass 2 compares in the
    // epilogue).  MMAs per unit: only the 32-byte K slices that hold data
    // (nC features, 6 BF16 / F16 or 12 FP8 norm entries, the threshold terms).
    const bool fp8 = fmt == Fmt::fp8;
    const int tau_k = (!fp8 && nC + 9 <= KP) ? nC + 6 : -1;
    const int used = fp8 ? nC + 12 : 2 * (nC + (tau_k >= 0 ? 9 : 6));
    const int nk = (used + 31) / 32;
    // one persistent launch per packing class: one-slot and two-slot items on
    // 256-candidate units (or 128, irc_plan_tc_units), then four-slot items
    // on 128.  The threshold goes into the MMA only on 256-wide units; the
    // narrower ones compare in the epilogue.  Four-slot items (small chunks)
    // keep the compare: their CTAs are short, and waiting for the thresholds
    // before the pass-2 MMAs would put the threshold step on their critical
    // path.  Every form lists all candidates at or below tau; with folded
    // thresholds a list also holds what lies within 2^-10 above it.
    const int n1 = pl->n_tc_one, n2 = pl->n_tc_wide - pl->n_tc_one, n4 = pl->n_tc_items - pl->n_tc_wide;
    const irc_tc::TcItem *it1 = pl->tc_items, *it2 = it1 + n1, *it4 = it2 + n2;
    const bool narrow = pl->tc_wide_bn == 128;
    auto run = [&](auto fmt_c, auto tau_c) {
        constexpr Fmt F = decltype(fmt_c)::value;
        constexpr bool T = decltype(tau_c)::value;
        const int rest = T && !narrow ? lo.split.items : 0;
        int r = narrow ? launch_filter<F, 128, false, 1>(mq, mc, pl, it1, n1, lo.count + 1, nk, tau_k, lo, scratch, s)
                       : launch_filter<F, 256, T, 1>(mq, mc, pl, it1, n1 - rest, lo.count + 1, nk, tau_k, lo, scratch, s);
        if constexpr (T)
            if (r == IRC_OK && rest)
                r = launch_split<F>(mq, mc, pl, it1 + n1 - rest, nk, tau_k, lo, scratch, s);
        if (r != IRC_OK) return r;
        r = narrow ? launch_filter<F, 128, false, 2>(mq, mc, pl, it2, n2, lo.count + 2, nk, tau_k, lo, scratch, s)
                   : launch_filter<F, 256, T, 2>(mq, mc, pl, it2, n2, lo.count + 2, nk, tau_k, lo, scratch, s);
        if (r != IRC_OK) return r;
        return launch_filter<F, 128, false, 4>(mq, mc, pl, it4, n4, lo.count + 3, nk, tau_k, lo, scratch, s);
    };
    using yes = std::true_type;
    using no = std::false_type;
    if (fp8) return run(std::integral_constant<Fmt, Fmt::fp8>{}, no{});
    if (fmt == Fmt::f16)
        return tau_k >= 0 ? run(std::integral_constant<Fmt, Fmt::f16>{}, yes{})
                          : run(std::integral_constant<Fmt, Fmt::f16>{}, no{});
    return tau_k >= 0 ? run(std::integral_constant<Fmt, Fmt::bf16>{}, yes{})
                      : run(std::integral_constant<Fmt, Fmt::bf16>{}, no{});
}

int launch_knn_tc(Fmt fmt, const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, const float *F,
                  const float4 *Fp, int nC, int knn, float *vrKnn, float *rho, int32_t *miKnn, float *d2Knn,
                  const ListOut &lo, cudaStream_t s)
{
    const int n_out = pl->dev.n_out;
    cudaEvent_t *ev = profile_slot();
    if (ev) cudaEventRecord(ev[0], s);
    const int rc = launch_filters(fmt, mq, mc, pl, nC, lo, pl->scratch, s);
    if (rc != IRC_OK) return rc;
    if (ev) cudaEventRecord(ev[1], s);
    launch_next(k_rerank, (n_out + RR_WARPS - 1) / RR_WARPS, 32 * RR_WARPS, 0, s, 
        lo.qinfo, lo.lists, n_out, pl->dev.q_base, F, Fp, nC, pl->row_dims, knn, vrKnn, rho, miKnn, d2Knn,
        crowd_margin(fmt), pl->scratch);
    IRC_CHECK_LAUNCH("irc_site_knn(tensor core) re-rank");
    if (ev) cudaEventRecord(ev[2], s);
    return IRC_OK;
}

}  // namespace irc_tc

extern "C" {

int irc_set_wait_limit(int polls)
{
    const uint32_t v = polls > 0 ? (uint32_t)polls : (1u << 22);
    cudaError_t e = cudaMemcpyToSymbol(c_wait_polls, &v, sizeof(v));
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_set_wait_limit");
    return IRC_OK;
}

int irc_profile_begin(int max_calls)
{
    using namespace irc_tc;
    if (max_calls <= 0 || max_calls > 65536) {
        irc_host::set_error("irc_profile_begin: max_calls must be in 1..65536");
        return IRC_E_INVAL;
    }
    std::lock_guard<std::mutex> lk(g_prof_mu);
    for (cudaEvent_t e : g_prof_ev) cudaEventDestroy(e);
    g_prof_ev.clear();
    for (int i = 0; i < 3 * max_calls; ++i) {
        cudaEvent_t e;
        cudaError_t r = cudaEventCreate(&e);
        if (r != cudaSuccess) {
            for (cudaEvent_t x : g_prof_ev) cudaEventDestroy(x);
            g_prof_ev.clear();
            return irc_host::cuda_status(r, "irc_profile_begin");
        }
        g_prof_ev.push_back(e);
    }
    g_prof_used = 0;
    g_prof_on = 1;
    return IRC_OK;
}

int irc_profile_end(float *filter_ms, float *rerank_ms, int *calls)
{
    using namespace irc_tc;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    float a = 0.0f, b = 0.0f;
    for (int i = 0; i < g_prof_used; ++i) {
        float x = 0.0f, y = 0.0f;
        cudaError_t r = cudaEventSynchronize(g_prof_ev[3 * i + 2]);
        if (r == cudaSuccess) r = cudaEventElapsedTime(&x, g_prof_ev[3 * i], g_prof_ev[3 * i + 1]);
        if (r == cudaSuccess) r = cudaEventElapsedTime(&y, g_prof_ev[3 * i + 1], g_prof_ev[3 * i + 2]);
        if (r != cudaSuccess) {
            g_prof_on = 0;
            return irc_host::cuda_status(r, "irc_profile_end");
        }
        a += x;
        b += y;
    }
    if (filter_ms) *filter_ms = a;
    if (rerank_ms) *rerank_ms = b;
    if (calls) *calls = g_prof_used;
    for (cudaEvent_t e : g_prof_ev) cudaEventDestroy(e);
    g_prof_ev.clear();
    g_prof_used = 0;
    g_prof_on = 0;
    return IRC_OK;
}

}  // extern "C"
