// irc_cert.cu -- the plain forms (EXACT kNN, REF kNN, REF delta) through the
// tensor-core filter, with a proof per query.
//
// The plain forms are defined over every candidate of a query: their FP32
// distances in the reference arithmetic, ordered by (distance, row) (EXACT)
// or put through the reference's bins (REF).  Only a few dozen candidates can
// reach the result, so computing every distance in FP32 (2 x 2 x D operations
// a pair; 22 ms for 3.0e9 pairs of 33 features) is work the result does not
// need.  Here the filter (irc_tc.cu) lists each query's nearest candidates by
// half-precision operands on the tensor cores, the list's distances are
// computed in FP32 exactly as the plain kernels compute them, and the result
// is taken from the list if the list provably holds every candidate that
// could matter.  Otherwise the query's window is read again in FP32 (k_second),
// and what even that cannot decide goes, with its 16-query tile, through the
// plain kernel, so the outputs are the plain form's bit for bit in every case.
//
// The proof.  Scaled by the power of two s, a row is x = s (a - ref) and its
// operand x^ = half(x): |x^ - x| <= u |x| + e0 (u = 2^-11 for the rounding,
// enlarged to cover the FP32 subtraction; e0 the subnormals of 64 features).
// A candidate outside the list has a computed value v > tau, or no operand: a
// row that is not finite is never a result of these forms, one longer than
// kNorm is met below.  With an operand,
//     |v - |x^ - y^|^2| <= c (|x|^2 + |y|^2 + tau) + e1
// (FP32 norms of <= 64 terms, their three half-precision pieces, and <= 64
// products accumulated in FP32 by at most five MMAs: 2^-16 covers them with
// truncating additions; c = 2^-15 doubles it).  Suppose such a candidate had
// a plain FP32 distance d2 <= D.  Its real distance is then at most
// delta = sqrt(D) (1 + 1e-5) (FP32: <= 70 roundings of 2^-24), its norm at
// most |x| + s delta, so its operands' distance is at most
//     h = s delta + u (2 |x| + s delta) + 2 e0
// and v <= h^2 + c (|x|^2 + (|x| + s delta)^2 + tau) + e1.  If the right-hand
// side is below tau and |x| + s delta at most kNorm (the candidate then has an
// operand), no such candidate exists.  |x| comes from the operand preparation
// (an upper bound).  What weakens the proof: queries far from the centre
// (rounding grows with |x|: units 30 times their noise apart leave a few
// percent of the queries open, 60 times most) and a scale that many far rows
// have pulled down.  A few far rows change neither (k_centre_robust), because a
// candidate's norm is bounded through the triangle inequality.
//
// Measured: EXACT kNN + delta of 100,003 spikes (D = 33, 50 chunks, 3.0e9
// pairs) 22.1 -> 1.08 ms; REF kNN + delta of 60,001 spikes and 12,001 copies
// (D = 24, 30 chunks, 2.2e9 pairs) 29.2 -> 1.48 ms.  kNN alone of 100,000 spikes
// (D = 33, 50 chunks) by how far apart the units lie in their noise, plain ->
// proven, ms, EXACT | REF: 10 apart 22.3 -> 1.02 | 17.4 -> 1.14, 30 apart -> 2.6 |
// 2.9, 60 apart -> 9.2 | 9.7 (nearly every query looked at twice), 100 apart ->
// 9.7 | 9.8.  The contraction's error, on rows of this layout against FP64, is at
// most 2^-20.7 of the sum that c multiplies.
#include <algorithm>
#include <mutex>

#include "irc_cert.cuh"
#include "irc_common.cuh"
#include "irc_plan.cuh"
#include "irc_rerank.cuh"
#include "irc_rows.cuh"
#include "irc_tc.cuh"

namespace {

using irc_rr::QROW4;
using irc_rr::WARP_KEYS;
using irc_tc::Fmt;

constexpr int kWarps = 8;                 // queries per block of the list kernels
constexpr int kTile = 16;                 // queries per tile of the plain kernels
constexpr int kRefKeys = 52;              // REF: list entries used (of 64 places; left-over bins take the others)

// Counter words of a call's working memory (zeroed before it).
constexpr int W_ERR = irc::kScratchErr;   // a wait of the filter gave up
constexpr int W_TILES = 4;                // tiles left to the plain kernel
constexpr int W_TICKET = 6;               // block ticket of the centring
constexpr int W_GROUPS = 7;               // groups of the second look
constexpr int W_UNITS = 8;                // its units taken
constexpr size_t kHdrBytes = 256;

constexpr float kNorm = 240.0f;           // rows up to here have operands: kNorm^2 < F16_NORM2, with the rounding's room
static_assert(kNorm * kNorm * 1.002f < irc_tc::F16_NORM2, "rows within kNorm have operands");

// Could a candidate outside a list with threshold tau have an FP32 distance
// <= D?  False only if it cannot (the proof above).
__device__ __forceinline__ bool may_miss(float D, float tau, float s, float x)
{
    constexpr float u = 0x1p-11f * 1.02f, e0 = 3e-7f, c = 0x1p-15f, e1 = 1e-6f;
    const float sd = s * __fsqrt_rn(D) * (1.0f + 1e-5f);
    const float h = sd + u * (2.0f * x + sd) + 2.0f * e0;
    const float y = x + sd;
    const float rhs = (h * h + c * (x * x + y * y + tau) + e1) * (1.0f + 1e-5f);
    return !(rhs < tau) || !(y <= kNorm);
}

// The reference's bin of row idx for the queries of a chunk: bin t scans run
// t % nBB from t / nBB in steps of nT / nBB, so a row at offset j of run b is
// in bin (j % step) nBB + b; the bins left over when nBB does not divide nT
// start one step later, so a row with j % step == 0, j >= step is in one of
// them too (*extra, or -1).
__device__ __forceinline__ int bin_of(const irc::PlanDev &p, int r0, int nBB, int nT, int idx, int *extra)
{
    int lo = 0, hi = nBB;                     // the run with the largest start <= idx (starts ascend)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(p.rsr + r0 + mid) <= idx) lo = mid; else hi = mid;
    }
    const int j = idx - __ldg(p.rsr + r0 + lo), step = nT / nBB, m = j % step;
    const int t2 = step * nBB + lo;
    *extra = m == 0 && j >= step && t2 < nT ? t2 : -1;
    return m * nBB + lo;
}

struct Call {
    irc::PlanDev p;
    const int2 *qinfo, *cert;
    const uint32_t *lists;
    const float4 *Fp;
    int nC;
    const uint8_t *row_dims;
    const float *scale, *qnorm;
    int *words, *tile_flag, *tile_queue;
};

// Query q of chunk goes to the plain kernel (chunk < 0: no record of it was
// handed over, so it is in no chunk, or a wait gave up and every tile is
// searched again).
__device__ __forceinline__ void leave(const Call &c, int chunk, int q, int lane)
{
    if (lane != 0 || chunk < 0) return;
    const int t = __ldg(c.p.tile_off[irc::tile_slot(kTile)] + chunk) + (q - __ldg(c.p.q0 + chunk)) / kTile;
    if (atomicExch(c.tile_flag + t, 1) == 0) c.tile_queue[atomicAdd(c.words + W_TILES, 1)] = t;
}

// One query's list to its EXACT or REF result; false when it is not proven.  The
// list holds every candidate with an FP32 distance up to lim (infinity: every
// one), or it is a filter's list with threshold tau (kFiltered), or just some
// candidates (kSome: never proven).  bound: when not proven, an upper bound of
// the distances that the result needs (infinity: unknown).
constexpr float kFiltered = -1.0f, kSome = -2.0f;

template <int PER, bool REF, bool FRESH = false>
__device__ __forceinline__ bool from_list(const Call &c, const uint32_t *list, int cL, float lim, float tau, int chunk,
                                          int o, int knn, int nT, float4 *qs, unsigned long long *ws, unsigned *bits,
                                          int lane, float *vrKnn, float *rho, int *miKnn, float *d2Knn, float &bound)
{
    const float inf = __int_as_float(0x7f800000);
    const int q = c.p.q_base + o;
    const int nd = c.row_dims ? min(c.nC, (int)__ldg(c.row_dims + q)) : c.nC;
    unsigned long long kv[PER];
    irc_rr::list_keys<PER, FRESH>(list, cL, c.Fp, irc_tc::fp_row4(c.nC), q, qs, nd, lane, kv);
    unsigned tb;
    int n = irc_rr::select_keys<PER>(kv, REF ? kRefKeys : knn, ws, lane, tb);
    const float x = __ldg(c.qnorm + o), s = __ldg(c.scale);
    if (n > WARP_KEYS) {                      // many nearly equal distances
        if (!FRESH) {                         // the second look, up to this bound of the k-th
            bound = x <= kNorm ? __uint_as_float(tb) : inf;      // (without an operand: a list of any rows)
            return false;
        }
        irc_rr::warp_bitonic<unsigned long long, PER>(kv, lane);
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane * PER + i < WARP_KEYS) ws[lane * PER + i] = kv[i];
        __syncwarp();
        n = WARP_KEYS;
    }
    if (!REF) {
        if (n < knn && lim != inf) return false;
        if (n >= knn) {
            const float D = __uint_as_float((unsigned)(ws[knn - 1] >> 32));
            if (lim < 0.0f && (lim == kSome || !(s > 0.0f) || may_miss(D, tau, s, x))) {
                if (lim == kSome || x <= kNorm) bound = D;
                return false;
            }
        }
        if (lane < knn) irc_rr::emit(lane, ws[lane], q, knn, (size_t)o, miKnn, d2Knn, vrKnn, rho);
        return true;
    }
    if (n > kRefKeys) {
        tb = (unsigned)(ws[kRefKeys] >> 32);
        n = kRefKeys;
    }
    // REF: the first candidate of every bin in (d2, row) order is the bin's
    // minimum; the bins' values sqrt(d2) in (value, bin) order are MATLAB's
    // stable sort.  A key per bin: value bits | bin (10) | place in ws (6).
    const int r0 = __ldg(c.p.roffr + chunk), nBB = __ldg(c.p.roffr + chunk + 1) - r0;
    bits[lane] = 0u;                              // the bins seen, one bit each (nT <= 1024)
    __syncwarp();
    unsigned long long k2[2] = {~0ull, ~0ull};
    int nk = 0;                                   // bins found
    unsigned long long ex[2] = {~0ull, ~0ull};    // keys of the left-over bins
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        if (b * 32 >= n) break;
        const int e = b * 32 + lane;
        const bool have = e < n;
        int t = -1, t2 = -1;
        unsigned long long key = 0;
        if (have) {
            const unsigned long long w = ws[e];
            t = bin_of(c.p, r0, nBB, nT, (int)(w & 0xffffffffu), &t2);
            key = ((unsigned long long)__float_as_uint(irc::ref_sqrt_abs(__uint_as_float((unsigned)(w >> 32)))) << 32) |
                  (unsigned)e;
        }
        const unsigned same = __match_any_sync(0xffffffffu, have ? t : -1 - lane);
        const bool first = have && (same & ((1u << lane) - 1u)) == 0u && !((bits[t >> 5] >> (t & 31)) & 1u);
        __syncwarp();
        if (first) {
            atomicOr(bits + (t >> 5), 1u << (t & 31));
            k2[b] = key | ((unsigned long long)t << 16);
        }
        nk += __popc(__ballot_sync(0xffffffffu, first));
        if (__any_sync(0xffffffffu, t2 >= 0)) {
            const unsigned s2 = __match_any_sync(0xffffffffu, t2 >= 0 ? t2 : -1 - lane);
            const bool f2 = t2 >= 0 && (s2 & ((1u << lane) - 1u)) == 0u && !((bits[t2 >> 5] >> (t2 & 31)) & 1u);
            __syncwarp();
            if (f2) {
                atomicOr(bits + (t2 >> 5), 1u << (t2 & 31));
                ex[b] = key | ((unsigned long long)t2 << 16);
            }
            nk += __popc(__ballot_sync(0xffffffffu, f2));
        }
        __syncwarp();
    }
    // (bins without a candidate come last: the sentinel's root, the query's own number)
    if (nk < knn && (lim != inf || tb < 0x7f800000u)) return false;
    // the left-over bins' keys take free places (at most 64 keys are sorted)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        const unsigned mx = __ballot_sync(0xffffffffu, ex[b] != ~0ull);
        if (!mx) continue;
        const unsigned f0 = __ballot_sync(0xffffffffu, k2[0] == ~0ull), f1 = __ballot_sync(0xffffffffu, k2[1] == ~0ull);
        if (__popc(mx) > __popc(f0) + __popc(f1)) return false;
        // free place number i: the i-th set bit of f0, then of f1
        const unsigned lt = (1u << lane) - 1u;
        const int p0 = __popc(f0 & lt), p1 = __popc(f0) + __popc(f1 & lt);
        unsigned rest = mx;
        for (int i = 0; rest; ++i, rest &= rest - 1u) {
            const unsigned long long kx = __shfl_sync(0xffffffffu, ex[b], __ffs(rest) - 1);
            if (((f0 >> lane) & 1u) && p0 == i) k2[0] = kx;
            if (((f1 >> lane) & 1u) && p1 == i) k2[1] = kx;
        }
    }
    irc_rr::warp_bitonic<unsigned long long, 2>(k2, lane);        // element 2 lane + i
    const float none = irc::ref_sqrt_abs(IRC_SINGLE_INF_F);
    const int last = min(knn, nk) - 1;
    const unsigned long long kth = __shfl_sync(0xffffffffu, (last & 1) ? k2[1] : k2[0], max(last, 0) >> 1);
    float v = last >= 0 ? __uint_as_float((unsigned)(kth >> 32)) : 0.0f;
    if (!(v < none)) return false;                               // (a tie with the empty bins)
    const float need = __fmul_rn(v, v) * (1.0f + 1e-6f);         // every distance whose root may be v lies below
    if (nk >= knn) {
        // every candidate left out must have a larger square root than the knn-th
        // value: the listed ones not used (d2 >= tb) and the unlisted ones
        const bool used = tb >= 0x7f800000u || __fsqrt_rn(__uint_as_float(tb)) > v;
        const bool all = lim < 0.0f ? lim != kSome && s > 0.0f && !may_miss(need, tau, s, x) : __fsqrt_rn(lim) > v;
        if (!used || !all) {
            if (lim == kSome || x <= kNorm) bound = need;
            return false;
        }
    } else {
        v = none;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int e = 2 * lane + i;
        if (e < knn) __stcs(miKnn + (size_t)e + (size_t)knn * o, e < nk ? (int)(ws[k2[i] & 63u] & 0xffffffffu) + 1 : q + 1);
    }
    if (lane == 0) {
        __stcs(vrKnn + o, v);
        if (rho) __stcs(rho + o, __fdiv_rn(1.0f, v));
    }
    return true;
}

// The second look.  A query whose list does not prove its result goes on a list
// of its chunk, with the distance that its list's best rows bound the result by
// (kind 0, from the front of the chunk's segment of slot) or without one (kind 1,
// from its end: lists that overflowed, rows without an operand).  64 of them
// make a group, and a block reads a group's window, or a part of it, once for
// all of them (k_second).
constexpr int kGroup = 64, kCollect = 128;    // queries a group; rows collected for a query

struct Second {
    int2 *slot;                               // (query, bits of its bound)
    int *cnt;                                 // rows collected
    int2 *groups;                             // (chunk | kind << 30, first place in its list)
    int *counts, *done;                       // of a chunk's kinds; parts of a group that have ended
    uint32_t *rows;                           // [kCollect] of a slot
};

// Place i of a chunk's list.
__device__ __forceinline__ int slot_at(const irc::PlanDev &p, int chunk, int kind, int i)
{
    const int at = __ldg(p.qseg + chunk);
    return kind ? at + __ldg(p.nq + chunk) - 1 - i : at + i;
}

__device__ __forceinline__ void look_again(const Call &c, const Second &z, int chunk, int q, float bound, int lane)
{
    if (lane != 0 || chunk < 0) return;       // (as in leave)
    const int kind = !(bound < __int_as_float(0x7f800000));
    const int i = atomicAdd(z.counts + 2 * chunk + kind, 1), at = slot_at(c.p, chunk, kind, i);
    z.slot[at] = make_int2(q, __float_as_int(bound));
    z.cnt[at] = 0;
    if (i % kGroup == 0) {
        const int g = atomicAdd(c.words + W_GROUPS, 1);
        z.groups[g] = make_int2(chunk | kind << 30, i);
        z.done[g] = 0;
    }
}

template <bool REF>
__global__ void __launch_bounds__(32 * kWarps, 5)
k_cert_knn(Call c, Second z, int knn, int nT, float *__restrict__ vrKnn, float *__restrict__ rho, int *__restrict__ miKnn,
           float *__restrict__ d2Knn)
{
    after_previous(c.qinfo, c.cert, c.lists, c.Fp, c.scale, c.qnorm);
    __shared__ __align__(16) unsigned long long wkeys[kWarps * WARP_KEYS];
    __shared__ float4 qrows[kWarps * QROW4];
    __shared__ unsigned wbits[REF ? kWarps * 32 : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int o = blockIdx.x * kWarps + warp;
    if (o >= c.p.n_out) return;
    const int2 qi = __ldg(c.qinfo + o), ce = __ldg(c.cert + o);
    float bound = __int_as_float(0x7f800000);
    bool ok = false;
    if (qi.x >= 0) {
        const uint32_t *l = c.lists + (unsigned)qi.x;
        const int cL = qi.y & 0x3fffffff;
        const float lim = (qi.y >> 30) & 1 ? bound : kFiltered;   // (a list of every candidate)
        const float tau = __int_as_float(ce.x);
        unsigned long long *ws = wkeys + warp * WARP_KEYS;
        float4 *qs = qrows + warp * QROW4;
        unsigned *bits = wbits + (REF ? warp * 32 : 0);
        if (cL <= 64) ok = from_list<2, REF>(c, l, cL, lim, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn, bound);
        else if (cL <= 128) ok = from_list<4, REF>(c, l, cL, lim, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn, bound);
        else ok = from_list<8, REF>(c, l, cL, lim, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn, bound);
    }
    if (!ok) look_again(c, z, ce.y, c.p.q_base + o, bound, lane);
}


// The second look at the groups' queries: the candidates of a window up to each
// query's distance, in FP32 as the plain kernels compute it, then the result
// from these few dozen rows.  Queries without a bound get one from a first pass:
// the rank-th smallest of 128 stripe minima, as the plain EXACT kernel finds
// its own.  With more than kCollect rows up to a bound that half precision left
// too wide, the collected ones give a closer one, and the block that ends the
// group reads the window for it (then, if need be, as without a bound).  Rows are
// staged and shared as in k_search_drift, but no minimum is kept, so the scan
// runs at the rate of the distances.  Windows of known bounds are cut into
// parts, the units taken from a counter; the block that ends a group last makes
// its queries' results.  What is left then (mass ties) goes to the plain kernel.
//
// Before it, an open query sent its 16-query tile there, two passes over the
// window on one SM: a single one cost 3,000 spikes as much as all of them in the
// plain kernel, and every query of a site with far apart units 20% more than no
// search at all.  With all of 100,000 spikes open (3.0e9 pairs of 33 features) it
// takes some 8 ms: 12 of the FP32 pipe's 38 T terms a second, as k_search_drift.
constexpr int kSecondWarps = 8;
constexpr int kSecondBlocks = 8;              // blocks of 64 rows in shared memory, in use or on their way
constexpr int kSecondPart = 256;              // fewest rows of a part

size_t second_smem(int nC)
{
    const size_t stages = (size_t)kSecondBlocks * 64 * irc::row_pitch(nC), minima = (size_t)kGroup * 128;
    return ((size_t)nC * kGroup + (stages > minima ? stages : minima)) * sizeof(float);
}

// A unit's queries (rows q, places slot, m <= NG QB of them; t: collect up to, lim:
// the bound) over positions [lo, hi) of their chunk's window.  NG warps share a
// block of rows, QB queries each; the warps' NS sets take blocks in turn.  With
// few queries QB is 4 and the arithmetic no longer covers the latency of a copy:
// NB blocks of a set are in flight.
template <int QB, int NG>
__device__ __forceinline__ void look(const Call &c, const Second &z, const float *__restrict__ F, int chunk, int m, int lo, int hi,
                                     bool two_pass, unsigned rank, float *sm, float *sT, float *sLim, const int *sQ,
                                     const int *sSlot, int *sRow)
{
    constexpr int NS = kSecondWarps / NG, NB = kSecondBlocks / NS, kStripes = 64 * NS;
    static_assert(QB * NG * kStripes <= kGroup * 128, "room for the minima");
    const float inf = __int_as_float(0x7f800000), below = __int_as_float(__float_as_int(IRC_SINGLE_INF_F) - 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = warp % NG, sub = warp / NG;
    const int nC = c.nC, P = irc::row_pitch(nC);
    const float *sA = sm + g * nC * QB;
    float *area = sm + nC * kGroup;                           // stages, then minima
    float *buf = area + sub * (NB * 64 * P);
    int *rows = sRow + sub * (NB * 64) + lane;                // the rows of the set's blocks
    const irc::RowCopy<NG> rc(nC, lane, g);
    for (int i = threadIdx.x; i < nC * QB * NG; i += 32 * kSecondWarps) {
        const int k = i / nC, f = i - k * nC;
        sm[((k / QB) * nC + f) * QB + k % QB] = -__ldg(F + (size_t)sQ[min(k, m - 1)] * nC + f);
    }
    __syncthreads();
    const int n = min(QB, m - g * QB);                        // this warp's queries (n <= 0: none)
    const int r0 = __ldg(c.p.roff + chunk), r1 = __ldg(c.p.roff + chunk + 1);
    const int steps = (hi - lo - sub * 64 + NS * 64 - 1) / (NS * 64);
    // body(rows, distances) for this set's blocks of 64 rows of [lo, hi)
    auto scan = [&](auto body) {
        int pos[2], run[2], base[2], rs[2], rn[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            pos[h] = lo + sub * 64 + h * 32 + lane;
            run[h] = r0;
            base[h] = 0;
            rs[h] = __ldg(c.p.rs + r0);
            rn[h] = __ldg(c.p.rn + r0);
        }
        auto stage = [&](int s) {                             // the next block
            int row[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                while (pos[h] >= base[h] + rn[h] && run[h] + 1 < r1) {
                    base[h] += rn[h];
                    ++run[h];
                    rs[h] = __ldg(c.p.rs + run[h]);
                    rn[h] = __ldg(c.p.rn + run[h]);
                }
                row[h] = pos[h] < hi ? rs[h] + pos[h] - base[h] : -1;
                pos[h] += NS * 64;
                if (g == 0) rows[s * 64 + h * 32] = row[h];
            }
            __syncwarp();
            rc.issue(buf + s * 64 * P, P, F, nC, row);
            irc::copies_commit();
        };
#pragma unroll
        for (int s = 0; s < NB - 1; ++s) stage(s);
        for (int k = 0; k < steps; ++k) {
            const int s = k % NB;
            stage((k + NB - 1) % NB);
            irc::copies_wait<NB - 1>();
            irc::rows_sync<NG>(sub);
            if (n > 0) {
                const int at[2] = {rows[s * 64], rows[s * 64 + 32]};
                float d[2][QB];
                irc::pair_dist<QB>(buf + (s * 64 + lane) * P, buf + (s * 64 + 32 + lane) * P, nC, sA, d[0], d[1]);
                body(at, d);
            }
            irc::rows_sync<NG>(sub);
        }
        irc::copies_wait<0>();
        __syncthreads();
    };
    if (two_pass) {
        float mn[2][QB];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < QB; ++q) mn[h][q] = inf;
        scan([&](const int (&at)[2], const float (&d)[2][QB]) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < QB; ++q)
                    if (at[h] >= 0 && d[h][q] > 0.0f && d[h][q] < mn[h][q]) mn[h][q] = d[h][q];
        });
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < QB; ++q) area[(g * QB + q) * kStripes + sub * 64 + h * 32 + lane] = mn[h][q];
        __syncthreads();
        for (int q = warp; q < m; q += kSecondWarps) {
            unsigned v[kStripes / 32], ans = 0;
#pragma unroll
            for (int i = 0; i < kStripes / 32; ++i) v[i] = __float_as_uint(area[q * kStripes + i * 32 + lane]);
#pragma unroll 1
            for (int b = 30; b >= 0; --b) {
                const unsigned t = ans | (1u << b);
                unsigned k = 0;
#pragma unroll
                for (int i = 0; i < kStripes / 32; ++i) k += v[i] < t;
                if (__reduce_add_sync(0xffffffffu, k) < rank) ans = t;
            }
            const float t = __uint_as_float(ans);
            if (lane == 0) {
                sT[q] = fminf(t, below);
                sLim[q] = t < below ? t : inf;
            }
        }
        __syncthreads();
    }
    const unsigned mine = n > 0 ? (1u << n) - 1u : 0u;
    scan([&](const int (&at)[2], const float (&d)[2][QB]) {
        unsigned hit[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < QB / 4; ++j) {
            const float4 t4 = reinterpret_cast<const float4 *>(sT + g * QB)[j];
            const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    hit[h] |= (unsigned)(d[h][4 * j + e] <= t[e] && d[h][4 * j + e] > 0.0f) << (4 * j + e);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            for (unsigned w = at[h] >= 0 ? hit[h] & mine : 0u; w; w &= w - 1u) {
                const int slot = sSlot[g * QB + __ffs(w) - 1], e = atomicAdd(z.cnt + slot, 1);
                if (e < kCollect) z.rows[(size_t)slot * kCollect + e] = (uint32_t)at[h];
            }
    });
    __threadfence();
    __syncthreads();
}

template <bool REF>
__global__ void __launch_bounds__(32 * kSecondWarps, 2)
k_second(Call c, Second z, const float *__restrict__ F, int knn, int nT, float *__restrict__ vrKnn, float *__restrict__ rho,
         int *__restrict__ miKnn, float *__restrict__ d2Knn)
{
    after_previous(z.slot, z.groups, z.counts, c.words, c.scale, c.qnorm, c.Fp);
    extern __shared__ __align__(16) float second_sm[];
    __shared__ __align__(16) float sT[kGroup];                // rows up to here are collected
    __shared__ float sLim[kGroup];                            // the bound (infinity: every row is)
    __shared__ float sNew[kGroup];
    __shared__ int sQ[kGroup], sSlot[kGroup], sAgain[kGroup], sRow[kSecondBlocks * 64], sNext[2], sLast, sM;
    const int G = c.words[W_GROUPS];
    if (G == 0 || c.words[W_ERR]) return;                     // (a wait gave up: every tile is searched anyway)
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float *area = second_sm + c.nC * kGroup;
    unsigned long long *ws = reinterpret_cast<unsigned long long *>(area) + warp * WARP_KEYS;
    float4 *qs = reinterpret_cast<float4 *>(area + kSecondWarps * WARP_KEYS * 2) + warp * QROW4;
    unsigned *bits = reinterpret_cast<unsigned *>(area + kSecondWarps * (WARP_KEYS * 2 + QROW4 * 4)) + warp * 32;
    const unsigned rank = REF ? knn + knn / 2 + 8 : knn;      // (of 128 stripes and more; a few share a bin)
    const int parts = min(16, (4 * (int)gridDim.x - 1) / G + 1);
    for (int u = blockIdx.x, turn = 0; u < G * parts; u = sNext[turn & 1], ++turn) {
        if (t == 0) sNext[turn & 1] = (int)gridDim.x + atomicAdd(c.words + W_UNITS, 1);
        const int part = u / G, gi = u - part * G;
        const int2 gr = z.groups[gi];
        const int chunk = gr.x & 0x3fffffff, kind = gr.x >> 30;
        int m = min(kGroup, z.counts[2 * chunk + kind] - gr.y);
        const int ntot = __ldg(c.p.ncand + chunk), per = kind ? ntot : max(kSecondPart, (ntot + parts - 1) / parts);
        int lo = part * per, hi = min(ntot, lo + per);
        if (lo < hi) {
            if (t < kGroup) {
                const int slot = slot_at(c.p, chunk, kind, gr.y + min(t, m - 1));
                const int2 e = z.slot[slot];
                const float b = __int_as_float(e.y);
                sQ[t] = e.x;
                sSlot[t] = slot;
                sT[t] = fminf(b, __int_as_float(__float_as_int(IRC_SINGLE_INF_F) - 1));
                sLim[t] = b;
            }
            for (int round = kind ? 2 : 0, first = round;; ++round) {
                const bool two_pass = round == 2;
                __syncthreads();
                if (m <= 8) look<4, 2>(c, z, F, chunk, m, lo, hi, two_pass, rank, second_sm, sT, sLim, sQ, sSlot, sRow);
                else if (m <= 16) look<4, 4>(c, z, F, chunk, m, lo, hi, two_pass, rank, second_sm, sT, sLim, sQ, sSlot, sRow);
                else look<16, 4>(c, z, F, chunk, m, lo, hi, two_pass, rank, second_sm, sT, sLim, sQ, sSlot, sRow);
                if (t == 0) {
                    sLast = round > first || atomicAdd(z.done + gi, 1) == (ntot + per - 1) / per - 1;
                    sM = 0;
                }
                __syncthreads();
                if (!sLast) break;
                __threadfence();
                for (int q = warp; q < m; q += kSecondWarps) {
                    const int cnt = __ldcg(z.cnt + sSlot[q]), o = sQ[q] - c.p.q_base;
                    const uint32_t *l = z.rows + (size_t)sSlot[q] * kCollect;
                    const float lim = cnt <= kCollect ? sLim[q] : kSome;
                    float b = sT[q];
                    bool ok;
                    if (cnt <= 64)
                        ok = from_list<2, REF, true>(c, l, cnt, lim, 0.0f, chunk, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn, b);
                    else
                        ok = from_list<4, REF, true>(c, l, min(cnt, kCollect), lim, 0.0f, chunk, o, knn, nT, qs, ws, bits, lane, vrKnn, rho,
                                                     miKnn, d2Knn, b);
                    if (!ok && two_pass) leave(c, chunk, sQ[q], lane);
                    if (!ok && !two_pass && lane == 0) {
                        const int i = atomicAdd(&sM, 1);
                        sAgain[i] = q;
                        sNew[i] = b;
                        z.cnt[sSlot[q]] = 0;
                    }
                    __syncwarp();
                }
                if (t == 0 && round == first) irc::count_stat(c.p, irc::kStatSecond, m);
                __syncthreads();
                if (two_pass || sM == 0) break;
                m = sM;                                       // (at most as many: places move to the front)
                const int i = min(t, m - 1), from = t < kGroup ? sAgain[i] : 0, q = sQ[from], slot = sSlot[from];
                __threadfence();
                __syncthreads();
                if (t < kGroup) {
                    sQ[t] = q;
                    sSlot[t] = slot;
                    sT[t] = sLim[t] = sNew[i];
                }
                lo = 0;
                hi = ntot;
            }
        }
        __syncthreads();
    }
}

// REF delta of one query per warp: among its listed candidates with a higher
// rho (the reference's mask), the smallest sqrt(d2), then the lowest bin, then
// in the bin the smallest (d2, row).  Queries whose list holds none, or not
// provably the nearest, are listed for the drift-window search.
__global__ void __launch_bounds__(32 * kWarps, 4)
k_cert_delta(Call c, const float *__restrict__ R, int nT, float *__restrict__ delta, int *__restrict__ nneigh,
             int *__restrict__ counts, int *__restrict__ list_out)
{
    after_previous(c.qinfo, c.cert, c.lists, c.Fp, c.scale, c.qnorm);
    __shared__ float4 qrows[kWarps * QROW4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int o = blockIdx.x * kWarps + warp;
    if (o >= c.p.n_out) return;
    const int2 qi = __ldg(c.qinfo + o), ce = __ldg(c.cert + o);
    const int q = c.p.q_base + o;
    bool ok = false;
    if (qi.x >= 0) {
        const uint32_t *list = c.lists + (unsigned)qi.x;
        const int cL = qi.y & 0x3fffffff, Dp4 = irc_tc::fp_row4(c.nC);
        const int nd = c.row_dims ? min(c.nC, (int)__ldg(c.row_dims + q)) : c.nC;
        const float rq = __ldg(R + q);
        float4 *qs = qrows + warp * QROW4;
        if (lane < Dp4) qs[lane] = __ldg(c.Fp + (size_t)q * Dp4 + lane);
        __syncwarp();
        const int r0 = __ldg(c.p.roffr + ce.y), nBB = __ldg(c.p.roffr + ce.y + 1) - r0;
        unsigned bv = 0xffffffffu;                // this lane's best: value bits, bin, (d2, row)
        int bt = INT32_MAX;
        unsigned long long bk = ~0ull;
        for (int e = lane; e < cL; e += 32) {
            const int idx = (int)__ldg(list + e);
            if (__ldg(R + idx) <= rq) continue;
            const int row[1] = {idx};
            float acc[1];
            irc_rr::row_dists<1>(c.Fp, Dp4, row, qs, nd, acc);
            const float d2 = acc[0];
            if (!(d2 > 0.0f) || !(d2 < IRC_SINGLE_INF_F)) continue;
            const unsigned v = __float_as_uint(irc::ref_sqrt_abs(d2));
            if (v > bv) continue;
            int ex;
            const int t = bin_of(c.p, r0, nBB, nT, idx, &ex);      // (a left-over bin never comes before its row's own)
            const unsigned long long k = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)idx;
            if (v < bv || t < bt || (t == bt && k < bk)) { bv = v; bt = t; bk = k; }
        }
        __syncwarp();
        const unsigned v = __reduce_min_sync(0xffffffffu, bv);
        const int t = __reduce_min_sync(0xffffffffu, bv == v ? bt : INT32_MAX);
        const unsigned long long k = irc::warp_min_u64(bv == v && bt == t ? bk : ~0ull);
        if (v != 0xffffffffu && __ldg(c.scale) > 0.0f) {
            const float vf = __uint_as_float(v);
            ok = ((qi.y >> 30) & 1) ||
                 !may_miss(__fmul_rn(vf, vf) * (1.0f + 1e-6f), __int_as_float(ce.x), __ldg(c.scale), __ldg(c.qnorm + o));
            if (ok && lane == 0) {
                delta[o] = __fmul_rn(vf, rq);
                nneigh[o] = (int)(k & 0xffffffffu) + 1;
            }
        }
    }
    // (without a record the query is in no chunk, or a wait gave up and every query is searched again)
    if (lane == 0 && !ok && ce.y >= 0)
        list_out[__ldg(c.p.qseg + ce.y) + atomicAdd(counts + ce.y, 1)] = q;
}

// Working memory of the proven searches: a block of the library's pool per call
// (a call of another stream or thread gets other memory, so concurrent calls on
// one plan stay independent, as the plain kernels' are).
//
// A captured call takes a block of its own, which the plan keeps (a graph is
// of no use without its plan), so that the graph holds no allocations: one
// that does can be instantiated only once at a time and be no child graph.
// Beyond kMaxCaptured captured calls of a plan, the plain kernels are captured.
constexpr int kMaxCaptured = sizeof(irc_plan::captured) / sizeof(void *);
std::mutex g_captured_mu;

void *captured_block(irc_plan *pl, size_t bytes)
{
    std::lock_guard<std::mutex> lk(g_captured_mu);
    if (pl->n_captured == kMaxCaptured) return nullptr;
    irc_host::Uncaptured mode;
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return pl->captured[pl->n_captured++] = p;
}

// Stream-ordered working memory of one call, returned in stream order.
struct Work {
    cudaStream_t s;
    void *base = nullptr;
    bool kept = false;
    Work(irc_plan *pl, size_t bytes, cudaStream_t st) : s(st)
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) cudaGetLastError();
        if (cs != cudaStreamCaptureStatusNone) {
            kept = true;
            base = captured_block(pl, bytes);
            return;
        }
        if (irc_search_alloc(&base, bytes, pl->device, s) != cudaSuccess) {
            cudaGetLastError();                   // not served: the plain kernels need no memory
            base = nullptr;
        }
    }
    ~Work()
    {
        if (base && !kept) cudaFreeAsync(base, s);
    }
};

size_t up(size_t n) { return (n + 255) & ~(size_t)255; }

// Where the filter pays.  The plain kernels' time grows with the pairs times
// the features and with the 16-query tiles; the search has a dozen launches to
// make first, and queries without a proof, few or all of them by the data, are
// looked at twice.  Microseconds, plain -> proven (every query looked at twice),
// EXACT | REF | REF delta:
//     2,048 spikes, one chunk, D = 24 (1.0e8)    70 -> 63 (117) |  83 -> 66 (133) |  26 -> 77 (95)
//     2,048, D = 45 (1.9e8, 4.2e6 pairs)         98 -> 72 (333) |  99 -> 76 (395) |  42 -> 93 (118)
//     2,450, D = 24 (1.4e8, 154 tiles)          115 -> 78 (133) | 167 -> 86 (154) |  52 -> 80 (97)
//     2,900, D = 24 (2.0e8, 8.4e6 pairs)        130 -> 70 (136) | 176 -> 76 (157) |  62 -> 83 (105)
//     3,000, D = 33 (3.0e8)                     146 -> 79 (159) | 196 -> 85 (181) |  84 -> 91 (117)
//     4,000, D = 9 (1.4e8)                       91 -> 79 (140) | 157 -> 86 (166) |  42 -> 88 (139)
//     5,000, D = 24 (6.0e8)                     266 -> 98 (213) | 309 -> 108 (237) | 144 -> 98 (177)
//     4,000, 200 chunks (2.9e7, 400 tiles)       83 -> 74 (104) | 171 -> 83 (122) |  32 -> 88 (93)
//     10,000, 400 chunks (9.0e7, 800 tiles)     142 -> 74 (140) | 378 -> 89 (167) |  57 -> 93 (96)
//     20,000, 1,200 chunks (1.2e8, 2,400 tiles) 265 -> 96 (159) | 715 -> 123 (207) | 108 -> 113 (118)
// The lines lie where the column in parentheses is at most some percent above
// the plain kernel's.  Tiles alone count only where a window is likely to hold
// knn candidates.
enum class Form { exact, ref, ref_delta };

bool serves(const irc_plan *pl, int nC, Form f)
{
    if (!pl->runs_ascend || !pl->disjoint || nC + 6 > irc_tc::KP) return false;
    if ((size_t)pl->dev.n_out * kCollect > irc_tc::list_cap(pl->dev.n_out)) return false;      // (offsets are int32)
    const bool many = f == Form::ref_delta ? pl->pairs * nC >= 800000000 : pl->pairs * nC >= 200000000 && pl->pairs >= 6000000;
    const int tiles = f == Form::exact ? 500 : f == Form::ref ? 150 : 4000;
    return many || (pl->ntiles[irc::tile_slot(kTile)] >= tiles && pl->pairs >= 64LL * pl->dev.n_out);
}

// Lists of every query on stream s: words | more (zeroed) ... | cert | lists | operands.
struct Lists {
    Call c;
    irc_tc::Operands op;
    char *more;
};

size_t lists_bytes(irc_plan *pl, int nC, size_t more)
{
    return kHdrBytes + up(more) + up((size_t)pl->dev.n_out * sizeof(int2)) + up(irc_tc::list_area_bytes(pl->dev.n_out)) +
           irc_tc::ops_bytes(pl, nC, Fmt::f16) + irc_tc::split_bytes(pl, nC, Fmt::f16);
}

int make_lists(irc_plan *pl, const float *F, int nC, char *base, size_t more, size_t zero, Lists *L, cudaStream_t s)
{
    int *words = (int *)base;
    L->more = base + kHdrBytes;
    int2 *cert = (int2 *)(L->more + up(more));
    char *la = (char *)cert + up((size_t)pl->dev.n_out * sizeof(int2));
    char *ops = la + up(irc_tc::list_area_bytes(pl->dev.n_out));
    irc_tc::ListOut lo = irc_tc::list_area(la, pl->dev.n_out);
    irc_tc::split_area(pl, nC, Fmt::f16, ops + irc_tc::ops_bytes(pl, nC, Fmt::f16), &lo);
    lo.cert = cert;
    cudaError_t e = cudaMemsetAsync(base, 0, kHdrBytes + zero, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(cert, 0xff, (size_t)pl->dev.n_out * sizeof(int2), s);
    if (e == cudaSuccess) e = irc_tc::clear_lists(lo, pl->dev.n_out, s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn: memset");
    int rc = irc_tc::make_operands(Fmt::f16, pl, F, nC, ops, nullptr, (unsigned *)words + W_TICKET, &L->op, s);
    if (rc != IRC_OK) return rc;
    rc = irc_tc::launch_filters(Fmt::f16, L->op.mq, L->op.mc, pl, nC, lo, words, s);
    L->c = Call{pl->dev, lo.qinfo, cert, lo.lists, L->op.fp, nC, pl->row_dims, L->op.scale, L->op.qnorm, words, nullptr, nullptr};
    return rc;
}

}  // namespace

void irc_cert_release(irc_plan *pl)
{
    for (int i = 0; i < pl->n_captured; ++i) cudaFree(pl->captured[i]);
}

int irc_cert_site_knn(irc_plan *pl, const float *F, int nC, int knn, int nThreads, int mode, float *vrKnn, float *rho,
                      int32_t *miKnn, float *d2Knn, cudaStream_t s)
{
    if (!serves(pl, nC, mode == IRC_MODE_EXACT ? Form::exact : Form::ref) || knn > irc_tc::KNN_MAX) return IRC_CERT_PASS;
    const int tiles = pl->ntiles[irc::tile_slot(kTile)];
    const size_t n = (size_t)pl->dev.n_out, chunks = (size_t)pl->dev.nChunks, groups = n / kGroup + 2 * chunks;
    // zeroed: tile flags, counts of the second look's lists
    const size_t flags = up((size_t)tiles * 4), counts = up(8 * chunks), queue = up((size_t)tiles * 4);
    const size_t more = flags + counts + queue + up(8 * n) + up(4 * n) + up(8 * groups) + up(4 * groups);
    Work w(pl, lists_bytes(pl, nC, more), s);
    if (!w.base) return IRC_CERT_PASS;
    Lists L;
    int rc = make_lists(pl, F, nC, (char *)w.base, more, flags + counts, &L, s);
    if (rc != IRC_OK) return rc;
    L.c.tile_flag = (int *)L.more;
    L.c.tile_queue = (int *)(L.more + flags + counts);
    char *b = L.more + flags + counts + queue;
    Second z;
    z.counts = (int *)(L.more + flags);
    z.slot = (int2 *)b;
    z.cnt = (int *)(b += up(8 * n));
    z.groups = (int2 *)(b += up(4 * n));
    z.done = (int *)(b + up(8 * groups));
    static_assert(kCollect <= irc_tc::LIST_AVG, "the collected rows lie over the lists, which are no longer read");
    z.rows = const_cast<uint32_t *>(L.c.lists);
    const unsigned grid = (unsigned)((n + kWarps - 1) / kWarps);
    const bool exact = mode == IRC_MODE_EXACT;
    auto first = exact ? k_cert_knn<false> : k_cert_knn<true>;
    auto second = exact ? k_second<false> : k_second<true>;
    float *d2 = exact ? d2Knn : nullptr;
    launch_next(first, grid, 32 * kWarps, 0, s, L.c, z, knn, nThreads, vrKnn, rho, miKnn, d2);
    IRC_CHECK_LAUNCH("irc_site_knn lists");
    const size_t smem = second_smem(nC);
    cudaError_t e = cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn: smem attribute");
    launch_next(second, 2 * pl->sms, 32 * kSecondWarps, smem, s, L.c, z, F, knn, nThreads, vrKnn, rho, miKnn, d2);
    IRC_CHECK_LAUNCH("irc_site_knn second look");
    const irc::TileQueue tq{L.c.tile_queue, L.c.words + W_TILES, L.c.words + W_ERR, tiles};
    if (exact)
        return irc_exact_tiles(pl, F, nC, knn, vrKnn, rho, miKnn, d2Knn, tq, s);
    return irc_ref_tiles(pl, F, nC, knn, nThreads, vrKnn, rho, miKnn, tq, s);
}

int irc_cert_site_delta_ref(irc_plan *pl, const float *F, int nC, const float *R, int nThreads, float *delta,
                            int32_t *nneigh, cudaStream_t s)
{
    // (a bin's step number has 20 bits in the drift-window search's keys: a
    // run of at most 2^20 rows always fits)
    if (!serves(pl, nC, Form::ref_delta) || pl->max_rn > (1 << 20)) return IRC_CERT_PASS;
    const size_t more = delta_bytes(pl->dev.n_out, pl->dev.n_qry, pl->dev.nChunks);
    Work w(pl, lists_bytes(pl, nC, more), s);
    if (!w.base) return IRC_CERT_PASS;
    Lists L;
    // (the counters lie at the front of the scratch)
    int rc = make_lists(pl, F, nC, (char *)w.base, more, 4 * (4 + (size_t)pl->dev.nChunks), &L, s);
    if (rc != IRC_OK) return rc;
    const irc_delta_scratch sc = irc_delta_carve(pl, L.more, L.c.words + W_ERR);
    launch_next(k_cert_delta, (pl->dev.n_out + kWarps - 1) / kWarps, 32 * kWarps, 0, s, L.c, R, nThreads, delta, nneigh, sc.counts,
                                                                             sc.list);
    IRC_CHECK_LAUNCH("irc_site_delta lists");
    return irc_delta_window(pl, F, nC, R, nThreads, sc, delta, nneigh, s);
}
