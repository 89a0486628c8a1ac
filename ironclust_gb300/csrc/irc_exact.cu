// irc_exact.cu -- EXACT-mode site kNN and the kNN-list delta.  (Plans large
// enough are served by the proven search of irc_cert.cu; the kernel here then
// finishes the tiles it leaves open.)
//
// EXACT kNN: the true k nearest candidates (squared distance > 0, the irc2
// GPU convention) under the reference FP32 arithmetic, ordered by the key
// (d2 bits, index).  Two passes per query tile:
//   1. every thread keeps the minimum over a disjoint stripe of the linked
//      candidates (256 stripes); the k-th smallest stripe minimum tau bounds
//      the k-th neighbour distance from above (k distinct candidates lie at
//      or below it);
//   2. the stripes are rescanned and candidates with d2 <= tau are appended
//      to a per-query shared-memory list, which one warp sorts with a
//      bitonic network; the first k are the answer.
// A query whose list overflows (mass ties) is finished by a bounded
// fallback: k ordered scans, each taking the smallest key above the last.
//
// kNN-list delta: with the exact kNN list of every spike and rho for all of
// them, the nearest higher-rho spike is the first list entry whose rho
// exceeds the query's, whenever the list holds one (any closer higher-rho
// spike would rank earlier in the list).  Queries without one -- local
// density peaks -- go to a drift-window scan over all linked candidates.
#include <climits>
#include <cstdio>
#include <mutex>

#include "irc_cert.cuh"
#include "irc_common.cuh"
#include "irc_plan.cuh"
#include "irc_rows.cuh"
#include "irc_scan.cuh"

namespace {

constexpr int kThreads = 256;     // = number of stripes
constexpr int kQB = 16;           // queries per CTA
constexpr int kCap = 256;         // list capacity per query
constexpr float kInfSentinel = IRC_SINGLE_INF_F;
constexpr int kQueueBlocks = 152 * 4;   // grid of the queue-draining kernels (8 warps per block)

__device__ __forceinline__ unsigned long long dkey(float d2, int idx)
{
    return ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)idx;
}

// Distance of candidate iB to QB staged queries (reference arithmetic).
template <int QB>
__device__ __forceinline__ void dist_qb(const float *__restrict__ fb, int nC, const float *sA,
                                        float (&acc)[QB])
{
#pragma unroll
    for (int q = 0; q < QB; ++q) acc[q] = 0.0f;
    for (int c = 0; c < nC; ++c) {
        const float bv = __ldg(fb + c);
        const float4 *a4 = reinterpret_cast<const float4 *>(sA + c * QB);
#pragma unroll
        for (int j = 0; j < QB / 4; ++j) {
            const float4 a = a4[j];
            acc[4 * j + 0] = irc::dterm(acc[4 * j + 0], bv, a.x);
            acc[4 * j + 1] = irc::dterm(acc[4 * j + 1], bv, a.y);
            acc[4 * j + 2] = irc::dterm(acc[4 * j + 2], bv, a.z);
            acc[4 * j + 3] = irc::dterm(acc[4 * j + 3], bv, a.w);
        }
    }
}

// Walk this thread's stripe (list positions p = t, t+256, ...) of the
// concatenated runs r0..r1-1, calling f(candidate index).
template <class Fn>
__device__ __forceinline__ void walk_stripe(const irc::PlanDev &p, int r0, int r1, int t, Fn f)
{
    int pos = 0;                                   // list position of the run start
    for (int r = r0; r < r1; ++r) {
        const int rs = __ldg(p.rs + r), rn = __ldg(p.rn + r);
        int first = (t - pos) % kThreads;
        if (first < 0) first += kThreads;
        for (int i = first; i < rn; i += kThreads) f(rs + i);
        pos += rn;
    }
}

// Warp-wide ascending bitonic sort of kCap 64-bit keys in shared memory.
__device__ __forceinline__ void warp_sort_keys(unsigned long long *keys, int lane)
{
    constexpr int PER = kCap / 32;
    unsigned long long v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = keys[lane * PER + i];   // element id = lane*PER + i
    // bitonic over element ids e in [0, kCap)
#pragma unroll
    for (int size = 2; size <= kCap; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= PER) {
                const int lstride = stride / PER;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = lane * PER + i;
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[i], lstride);
                    const bool up = ((e & size) == 0);
                    const bool lower = ((e & stride) == 0);
                    const bool keep_min = (lower == up);
                    v[i] = keep_min ? (o < v[i] ? o : v[i]) : (o > v[i] ? o : v[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const int e = lane * PER + i;
                        const bool up = ((e & size) == 0);
                        const unsigned long long a = v[i], b = v[j];
                        const bool swap = up ? (a > b) : (a < b);
                        v[i] = swap ? b : a;
                        v[j] = swap ? a : b;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) keys[lane * PER + i] = v[i];
}

// One 16-query tile.
__device__ __forceinline__ void
exact_tile(const irc::PlanDev &p, int tile, const float *__restrict__ F, int nC, int knn, float *__restrict__ vrKnn,
           float *__restrict__ rho, int *__restrict__ miKnn, float *__restrict__ d2Knn, int *__restrict__ ovf_count,
           int *__restrict__ ovf_list)
{
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ float sTau[kQB];
    __shared__ int sCnt[kQB];
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sList = reinterpret_cast<unsigned long long *>(dyn);   // [kQB][kCap]
    float *sMin = reinterpret_cast<float *>(sList + kQB * kCap);              // [kQB][kThreads]
    int chunk, qs, n;
    irc::tile_lookup<kQB>(p, tile, chunk, qs, n);
    const int r0 = __ldg(p.roff + chunk), r1 = __ldg(p.roff + chunk + 1);
    irc::stage_queries<kQB>(F, nC, qs, n, sA);
    if (threadIdx.x < kQB) sCnt[threadIdx.x] = 0;
    __syncthreads();
    const int t = threadIdx.x;
    // pass 1: stripe minima
    float mn[kQB];
#pragma unroll
    for (int q = 0; q < kQB; ++q) mn[q] = __int_as_float(0x7f800000);
    walk_stripe(p, r0, r1, t, [&](int iB) {
        float acc[kQB];
        dist_qb<kQB>(F + (size_t)iB * nC, nC, sA, acc);
#pragma unroll
        for (int q = 0; q < kQB; ++q)
            if (acc[q] > 0.0f && acc[q] < mn[q]) mn[q] = acc[q];
    });
#pragma unroll
    for (int q = 0; q < kQB; ++q) sMin[q * kThreads + t] = mn[q];
    __syncthreads();
    // tau = k-th smallest stripe minimum (by value); +inf if fewer than k finite
    const int lane = t & 31, warp = t >> 5, nw = kThreads / 32;
    for (int q = warp; q < kQB; q += nw) {
        float *m = sMin + q * kThreads;
        float kth = __int_as_float(0x7f800000);
        for (int k = 0; k < knn; ++k) {
            unsigned long long best = ~0ull;
            for (int s = lane; s < kThreads; s += 32) {
                const unsigned long long key = dkey(m[s], s);
                best = key < best ? key : best;
            }
            best = irc::warp_min_u64(best);
            const int s = (int)(best & 0xffffffffu);
            kth = __uint_as_float((unsigned)(best >> 32));
            __syncwarp();
            if (lane == 0) m[s] = __int_as_float(0x7fffffff);      // NaN bits: sorts last
            __syncwarp();
            if (!(kth < __int_as_float(0x7f800000))) break;
        }
        if (lane == 0) sTau[q] = kth;
    }
    __syncthreads();
    // pass 2: collect d2 <= tau
    walk_stripe(p, r0, r1, t, [&](int iB) {
        float acc[kQB];
        dist_qb<kQB>(F + (size_t)iB * nC, nC, sA, acc);
#pragma unroll
        for (int q = 0; q < kQB; ++q)
            if (acc[q] > 0.0f && acc[q] <= sTau[q]) {
                const int slot = atomicAdd(&sCnt[q], 1);
                if (slot < kCap) sList[q * kCap + slot] = dkey(acc[q], iB);
            }
    });
    __syncthreads();
    for (int q = warp; q < n; q += nw) {
        const int cnt = sCnt[q];
        const size_t o = (size_t)(qs + q - p.q_base);
        if (cnt > kCap) {                          // overflow: finished by the fallback kernel
            if (lane == 0) { int i = atomicAdd(ovf_count, 1); ovf_list[i] = qs + q; }
            continue;
        }
        unsigned long long *L = sList + q * kCap;
        for (int i = cnt + lane; i < kCap; i += 32) L[i] = ~0ull;
        __syncwarp();
        warp_sort_keys(L, lane);
        __syncwarp();
        for (int k = lane; k < knn; k += 32) {
            const unsigned long long key = L[k];
            const bool ok = k < cnt;
            const float d2 = ok ? __uint_as_float((unsigned)(key >> 32)) : kInfSentinel;
            const int idx = ok ? (int)(key & 0xffffffffu) : qs + q;
            miKnn[(size_t)k + (size_t)knn * o] = idx + 1;
            if (d2Knn) d2Knn[(size_t)k + (size_t)knn * o] = d2;
            if (k == knn - 1) {
                const float v = irc::ref_sqrt_abs(d2);
                vrKnn[o] = v;
                if (rho) rho[o] = __fdiv_rn(1.0f, v);
            }
        }
        __syncwarp();
    }
}

// A tile per block.
__global__ void __launch_bounds__(kThreads)
k_site_knn_exact(irc::PlanDev p, const float *__restrict__ F, int nC, int knn, float *__restrict__ vrKnn,
                 float *__restrict__ rho, int *__restrict__ miKnn, float *__restrict__ d2Knn, int *__restrict__ ovf_count,
                 int *__restrict__ ovf_list)
{
    exact_tile(p, blockIdx.x, F, nC, knn, vrKnn, rho, miKnn, d2Knn, ovf_count, ovf_list);
}

// One query by k ordered scans of all linked candidates, each a block-wide
// minimum of the keys above the previous one.  Serves the rare queries whose
// candidate list overflowed (mass ties, or an unlucky spread of the tensor-core
// filter's list parts).
__device__ __forceinline__ void ordered_scans(const irc::PlanDev &p, const float *__restrict__ F, int nC, int knn, int q,
                                              float *__restrict__ vrKnn, float *__restrict__ rho, int *__restrict__ miKnn,
                                              float *__restrict__ d2Knn)
{
    __shared__ unsigned long long red[kThreads / 32];
    __shared__ unsigned long long sBest;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int lo = 0, hi = p.nChunks;                // the query's chunk, where the chunks ascend
    while (hi - lo > 1) { int mid = (lo + hi) >> 1; if (__ldg(p.q0 + mid) <= q) lo = mid; else hi = mid; }
    if (q < __ldg(p.q0 + lo) || q >= __ldg(p.q0 + lo) + __ldg(p.nq + lo)) {      // else the first that holds it
        __shared__ int sChunk;
        if (threadIdx.x == 0) sChunk = INT_MAX;
        __syncthreads();
        for (int c = threadIdx.x; c < p.nChunks; c += kThreads)
            if (q >= __ldg(p.q0 + c) && q < __ldg(p.q0 + c) + __ldg(p.nq + c)) atomicMin(&sChunk, c);
        __syncthreads();
        lo = min(sChunk, p.nChunks - 1);
        __syncthreads();
    }
    const int r0 = __ldg(p.roff + lo), r1 = __ldg(p.roff + lo + 1);
    const float *a = F + (size_t)q * nC;
    const size_t o = (size_t)(q - p.q_base);
    unsigned long long prev = 0;
    bool have_prev = false;
    for (int k = 0; k < knn; ++k) {
        unsigned long long best = ~0ull;
        walk_stripe(p, r0, r1, threadIdx.x, [&](int iB) {
            const float *b = F + (size_t)iB * nC;
            float acc = 0.0f;
            for (int c = 0; c < nC; ++c) acc = irc::dterm(acc, __ldg(b + c), __ldg(a + c));
            if (!(acc > 0.0f) || !(acc < kInfSentinel)) return;
            const unsigned long long key = dkey(acc, iB);
            if ((!have_prev || key > prev) && key < best) best = key;
        });
        best = irc::warp_min_u64(best);
        if (lane == 0) red[warp] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long b = red[0];
            for (int i = 1; i < kThreads / 32; ++i) b = red[i] < b ? red[i] : b;
            sBest = b;
            const bool ok = b != ~0ull;
            const float d2 = ok ? __uint_as_float((unsigned)(b >> 32)) : kInfSentinel;
            const int idx = ok ? (int)(b & 0xffffffffu) : q;
            miKnn[(size_t)k + (size_t)knn * o] = idx + 1;
            if (d2Knn) d2Knn[(size_t)k + (size_t)knn * o] = d2;
            if (k == knn - 1) {
                const float v = irc::ref_sqrt_abs(d2);
                vrKnn[o] = v;
                if (rho) rho[o] = __fdiv_rn(1.0f, v);
            }
        }
        __syncthreads();
        best = sBest;
        if (best != ~0ull) { prev = best; have_prev = true; }
    }
}

// The tiles of a queue.  (A kernel of its own: with the loop around it the tile
// spills, 4% on a site of 1,500 spikes.)  A tile's overflowed queries follow it.
__global__ void __launch_bounds__(kThreads)
k_site_knn_exact_queue(irc::PlanDev p, const float *__restrict__ F, int nC, int knn, float *__restrict__ vrKnn,
                       float *__restrict__ rho, int *__restrict__ miKnn, float *__restrict__ d2Knn, irc::TileQueue tq)
{
    after_previous(tq.list, tq.count, tq.all);
    __shared__ int sOvf[kQB], sOvfN;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        irc::count_stat(p, irc::kStatSearches, 1);
        irc::count_stat(p, irc::kStatTiles, tq.size());
    }
    for (int w = blockIdx.x, n_tiles = tq.size(); w < n_tiles; w += gridDim.x) {
        if (threadIdx.x == 0) sOvfN = 0;                     // (the tile has barriers before it counts)
        exact_tile(p, tq.tile(w), F, nC, knn, vrKnn, rho, miKnn, d2Knn, &sOvfN, sOvf);
        __syncthreads();
        const int n = sOvfN;
        for (int i = 0; i < n; ++i) ordered_scans(p, F, nC, knn, sOvf[i], vrKnn, rho, miKnn, d2Knn);
        if (threadIdx.x == 0) irc::count_stat(p, irc::kStatScans, n);
        __syncthreads();
    }
}

// The queued queries, one per block.
__global__ void __launch_bounds__(kThreads)
k_exact_overflow(irc::PlanDev p, const float *__restrict__ F, int nC, int knn,
                 const int *__restrict__ ovf_count, const int *__restrict__ ovf_list,
                 float *__restrict__ vrKnn, float *__restrict__ rho,
                 int *__restrict__ miKnn, float *__restrict__ d2Knn)
{
    after_previous(ovf_count, ovf_list);
    const int n = *ovf_count;
    if (blockIdx.x == 0 && threadIdx.x == 0) irc::count_stat(p, irc::kStatScans, n);
    for (int w = blockIdx.x; w < n; w += gridDim.x) ordered_scans(p, F, nC, knn, ovf_list[w], vrKnn, rho, miKnn, d2Knn);
}

// delta from the kNN list, a thread per query, a warp per 32-query tile of a
// chunk; queries without a higher-rho list entry go to the chunk's segment of
// fb_list, in any order.  Entries are read four at a time (their rho gathers in
// flight together): the first or second decides for most queries, and one at a
// time the two dependent loads of each made a 3,000-query site take 10 us.
constexpr int kListTile = 32, kListWarps = 4;

__global__ void __launch_bounds__(32 * kListWarps)
k_delta_list(irc::PlanDev p, int ntiles, const float *__restrict__ R, int knn, const int *__restrict__ miKnn,
             const float *__restrict__ d2Knn, float *__restrict__ delta, int *__restrict__ nneigh,
             int *__restrict__ counts, int *__restrict__ fb_list)
{
    after_previous();
    const int lane = threadIdx.x & 31, tile = blockIdx.x * kListWarps + (threadIdx.x >> 5);
    if (tile >= ntiles) return;
    int chunk, qs, n;
    irc::tile_lookup<kListTile>(p, tile, chunk, qs, n);
    int miss = 0;
    if (lane < n) {
        const int q = qs + lane, o = q - p.q_base;
        const float rq = __ldg(R + q);
        const int *mi = miKnn + (size_t)knn * o;
        const float *dk = d2Knn + (size_t)knn * o;
        miss = 1;
        bool more = true;
        for (int k = 0; k < knn && more; k += 4) {
            int j[4];                                        // -1: no entry
            float d2[4], rj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                j[u] = k + u < knn ? __ldg(mi + k + u) - 1 : -1;
                d2[u] = k + u < knn ? __ldg(dk + k + u) : kInfSentinel;
            }
            // (a list may be padded with any index, and rows of a search that gave up were never written)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!(d2[u] < kInfSentinel) || (unsigned)j[u] >= (unsigned)p.nF) j[u] = -1;
                rj[u] = j[u] >= 0 ? __ldg(R + j[u]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!more) continue;
                if (j[u] < 0) more = false;                          // list exhausted
                else if (!(rj[u] <= rq)) {                           // reference mask: rb <= ra is excluded
                    delta[o] = __fmul_rn(irc::ref_sqrt_abs(d2[u]), rq);
                    nneigh[o] = j[u] + 1;
                    miss = 0;
                    more = false;
                }
            }
        }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, miss);
    if (!bal) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(counts + chunk, __popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (miss) fb_list[__ldg(p.qseg + chunk) + base + __popc(bal & ((1u << lane) - 1u))] = qs + lane;
}

constexpr int kParts = 8;        // most parts of one candidate window (part < 2^3: 3 bits at bit 28)
constexpr int kMinPart = 2048;   // fewest candidates of a part
constexpr int kMinDense = 512;   // the same where 16 queries share it (968 queries of 6,000 spikes: 203 -> 171 us)
constexpr int kWide = 512;       // candidates of a window that whole blocks search, in parts
constexpr int kWideParts = 16;   // most parts (of kMinPart candidates and more)
// A part costs a block some 5 us before its first round, so many queries are
// searched in few parts: as many as make four units a block, taken from a
// counter (their work differs by the rows of higher rho).  us, window search and
// the rest of delta, 16 parts each -> so: 3,200 queries of a random rho among 100,000
// spikes 705 -> 293; 491 of a 400,000-spike site 228 -> 206 (two units 247, eight 226).
constexpr int kWideTurns = 4;
constexpr int kDense = 64;       // fewest queries of a chunk that are searched 16 at a time

// Distributes the queries without a listed neighbour, a warp per chunk.  There
// are few of them (0.1% of a drift site's queries, 1% of a probe's: density
// peaks), and few candidates have a higher rho than one of them (2%): they are
// searched one by one -- wide windows by blocks, a part each (sparse[0 ..
// words[1]); words[3] counts the units taken), the others by a warp (words[2] of
// them, from sparse's end).  (A
// part, because a spike alone among noise has a low rho: nearly every candidate
// of its window exceeds it.)  A chunk with at least kDense of
// them and one in eight (a rho of another kind, a search that proved little)
// has its windows read once for 16 queries: (16-query tile, part) units,
// {chunk | part << 28, (first << 5) | count}.  all (may be null): a word that,
// if set, sends every query there.
__global__ void k_delta_items(irc::PlanDev p, const int *__restrict__ all, const int *__restrict__ counts,
                              int *__restrict__ fb_list, int *__restrict__ words, int2 *__restrict__ sparse,
                              int2 *__restrict__ items, unsigned long long *__restrict__ keys)
{
    after_previous(all, counts);
    const int chunk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (chunk >= p.nChunks) return;
    const int q0 = __ldg(p.q0 + chunk), nq = __ldg(p.nq + chunk);
    int *list = fb_list + __ldg(p.qseg + chunk);
    int m = __ldg(counts + chunk);
    if (all && __ldg(all)) {
        m = nq;
        for (int i = lane; i < m; i += 32) list[i] = q0 + i;
        __syncwarp();
    }
    if (all && lane == 0) {
        irc::count_stat(p, irc::kStatDeltas, chunk == 0);
        irc::count_stat(p, irc::kStatWindows, m);
    }
    if (m == 0) return;
    const int ncand = __ldg(p.ncand + chunk);
    int base = 0;
    if (m >= kDense && m * 8 >= nq) {
        const int ntile = (m + kQB - 1) / kQB, np = min(kParts, max(1, ncand / kMinDense)), nunit = ntile * np;
        if (lane == 0) base = atomicAdd(words, nunit);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int j = lane; j < nunit; j += 32) {
            const int t = j / np, part = j - t * np;
            items[base + j] = make_int2(chunk | (part << 28), ((t * kQB) << 5) | min(kQB, m - t * kQB));
        }
        for (int i = lane; i < m; i += 32) keys[list[i] - p.q_base] = ~0ull;
    } else {
        const bool wide = ncand > kWide;
        if (lane == 0) base = atomicAdd(words + (wide ? 1 : 2), m);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int i = lane; i < m; i += 32)
            sparse[wide ? base + i : p.n_qry - 1 - (base + i)] = make_int2(list[i], chunk);
        if (wide)
            for (int i = lane; i < m; i += 32) keys[list[i] - p.q_base] = ~0ull;
    }
}

// The reference's tie rule of the delta search (REF): the smallest
// sqrt(d2), then the lowest bin, then inside the bin the smallest d2 and the
// first row.  One 64-bit key orders them: sqrt bits (31, positive) | bin (10)
// | d2 among the at most 5 FP32 values that share a square root (3: its offset
// from the rounded square) | step inside the bin (20; row = run start + bin /
// runs + step * stride).
__device__ __forceinline__ unsigned long long ref_key(float d2, int bin, int step)
{
    const float v = irc::ref_sqrt_abs(d2);
    const unsigned dd = __float_as_uint(d2) - __float_as_uint(__fmul_rn(v, v)) + 4u;
    return ((unsigned long long)__float_as_uint(v) << 33) | ((unsigned long long)bin << 23) |
           ((unsigned long long)(dd & 7u) << 20) | (unsigned)step;
}

// delta and nneigh of query qq of a chunk from the best key of its window (~0:
// no candidate, i.e. sqrt(SINGLE_INF) .* rho and the query itself, as
// search_delta_drift_).
template <bool REF>
__device__ __forceinline__ void put_delta(const irc::PlanDev &p, const float *__restrict__ R, int chunk, int qq,
                                          unsigned long long b, int nT, float *__restrict__ delta, int *__restrict__ nneigh)
{
    const bool ok = b != ~0ull;
    float v;
    int row = qq;
    if (REF) {
        v = ok ? __uint_as_float((unsigned)(b >> 33)) : irc::ref_sqrt_abs(kInfSentinel);
        if (ok) {
            const int r0 = __ldg(p.roffr + chunk), nBB = __ldg(p.roffr + chunk + 1) - r0;
            const int bin = (int)(b >> 23) & 1023;
            row = __ldg(p.rsr + r0 + bin % nBB) + bin / nBB + (int)(b & 0xfffffu) * (nT / nBB);
        }
    } else {
        v = irc::ref_sqrt_abs(ok ? __uint_as_float((unsigned)(b >> 32)) : kInfSentinel);
        if (ok) row = (int)(b & 0xffffffffu);
    }
    const size_t o = (size_t)(qq - p.q_base);
    delta[o] = __fmul_rn(v, __ldg(R + qq));
    nneigh[o] = row + 1;
}

// One query's best key over positions [lo, hi) of its chunk's window, by `nw`
// warps of which this is the w-th: the warp reads rho of 256 candidates at a
// time, queues the rows that exceed the query's, and evaluates 32 queued rows
// at once, copied to shared memory (a lane reading its row from global memory
// touches 32 cache lines a feature: 240 us for a window of 28,500 such rows).
// qrow: the warp's copy of the query's features; queue: 288 words; buf: 32 rows.
template <bool REF>
__device__ __forceinline__ unsigned long long scan_query(const irc::PlanDev &p, const float *__restrict__ F,
                                                         const float *__restrict__ R, int nC, int nd, int chunk, int q,
                                                         int nT, int lo, int hi, int w, int nw, float *qrow, int *queue,
                                                         float *buf, int lane)
{
    constexpr int NL = 8;                                    // rho loads in flight
    const float rq = __ldg(R + q);
    const int P = irc::row_pitch(nC);
    __syncwarp();
    for (int c = lane; c < nd; c += 32) qrow[c] = __ldg(F + (size_t)q * nC + c);
    __syncwarp();
    unsigned long long best = ~0ull;
    const int rr0 = __ldg(p.roffr + chunk), nBB = __ldg(p.roffr + chunk + 1) - rr0, step = REF ? nT / nBB : 1;
    const irc::RowCopy<2> rc(nC, lane, 0);                   // rows 0 .. 31
    int cnt = 0;
    auto round = [&](int first, int m) {
        __syncwarp();
        const int iB = lane < m ? queue[first + lane] : -1;
        const int rows[2] = {iB, -1};
        rc.issue(buf, P, F, nC, rows);
        irc::copies_commit();
        irc::copies_wait<0>();
        __syncwarp();
        if (lane < m) {
            const float *fb = buf + lane * P;
            float acc = 0.0f;
#pragma unroll 4
            for (int c = 0; c < nd; ++c) acc = irc::dterm(acc, fb[c], qrow[c]);
            if (acc > 0.0f && acc < kInfSentinel) {
                unsigned long long key = dkey(acc, iB);
                if (REF) {
                    int a = 0, b = nBB;                      // the row's run (their starts ascend)
                    while (b - a > 1) {
                        const int mid = (a + b) >> 1;
                        if (__ldg(p.rsr + rr0 + mid) <= iB) a = mid; else b = mid;
                    }
                    const int j = iB - __ldg(p.rsr + rr0 + a);
                    key = ref_key(acc, (j % step) * nBB + a, j / step);
                }
                best = key < best ? key : best;
            }
        }
        __syncwarp();
    };
    int pos = 0;                                             // position of run r's first candidate
    for (int r = __ldg(p.roff + chunk); r < __ldg(p.roff + chunk + 1) && pos < hi; ++r) {
        const int rs = __ldg(p.rs + r), rn = __ldg(p.rn + r);
        const int a = max(lo - pos, 0), b = min(hi - pos, rn);
        for (int i0 = a + w * 32 * NL; i0 < b; i0 += nw * 32 * NL) {
            float rb[NL];
#pragma unroll
            for (int u = 0; u < NL; ++u) {
                const int i = i0 + 32 * u + lane;
                rb[u] = i < b ? __ldg(R + rs + i) : rq;
            }
#pragma unroll
            for (int u = 0; u < NL; ++u) {
                const bool hit = !(rb[u] <= rq) && i0 + 32 * u + lane < b;        // the search_delta_drift mask
                const unsigned bal = __ballot_sync(0xffffffffu, hit);
                if (hit) queue[cnt + __popc(bal & ((1u << lane) - 1u))] = rs + i0 + 32 * u + lane;
                cnt += __popc(bal);
            }
            while (cnt >= 32) round(cnt -= 32, 32);          // the last 32 queued
        }
        pos += rn;
    }
    if (cnt) round(0, cnt);
    return irc::warp_min_u64(best);
}

// The drift-window search of the queries that k_delta_items distributed.  The
// 16-query units: a unit loads every candidate of its part once for the 16
// queries, keeps per query the candidates whose rho exceeds the query's, and
// folds its best key into the query's key with a 64-bit atomicMin -- the
// minimum of the same keys in any order, so the split changes no result.
// Before the queries were searched one by one, 16 of a chunk (2.6 on average)
// shared a pass over all its candidates: 390 us for the 491 queries of a
// 400,000-spike site.
template <bool REF>
__global__ void __launch_bounds__(kThreads)
k_delta_window(irc::PlanDev p, const float *__restrict__ F, const float *__restrict__ R, int nC,
               const uint8_t *__restrict__ row_dims, int *words, const int2 *__restrict__ sparse,
               const int2 *__restrict__ items, const int *__restrict__ fb_list, unsigned long long *__restrict__ keys,
               int nT, float *__restrict__ delta, int *__restrict__ nneigh)
{
    after_previous(words, sparse, items, fb_list);
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ float sRA[kQB];
    __shared__ int sQ[kQB];
    __shared__ unsigned long long redt[kQB][kThreads / 32];
    __shared__ int queues[kThreads / 32][288];
    extern __shared__ __align__(16) float rows_sm[];         // 32 rows per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kThreads / 32;
    const int total = words[0], n_wide = words[1], n_narrow = words[2];
    float *qrow = sA + warp * IRC_NC_MAX;                    // (kQB >= the warps of a block)
    float *buf = rows_sm + warp * 32 * irc::row_pitch(nC);
    const int parts = n_wide ? min(kWideParts, (kWideTurns * (int)gridDim.x - 1) / n_wide + 1) : 0;
    __shared__ int sNext[2];                                 // (in turns: read after the barrier, written before the next)
    for (int u = blockIdx.x, turn = 0; u < n_wide * parts; u = sNext[turn & 1], ++turn) {
        if (threadIdx.x == 0) sNext[turn & 1] = (int)gridDim.x + atomicAdd(words + 3, 1);
        const int part = u / n_wide;
        const int2 e = sparse[u - part * n_wide];
        const int ntot = __ldg(p.ncand + e.y), per = max(kMinPart, (ntot + parts - 1) / parts);
        if (part * per < ntot) {
            const int nd = row_dims ? min(nC, (int)__ldg(row_dims + e.x)) : nC;
            const unsigned long long b = scan_query<REF>(p, F, R, nC, nd, e.y, e.x, nT, part * per, min(ntot, part * per + per),
                                                         warp, nw, qrow, queues[warp], buf, lane);
            if (lane == 0 && b != ~0ull) atomicMin(keys + (e.x - p.q_base), b);
        }
        __syncthreads();
    }
    for (int w = blockIdx.x * nw + warp; w < n_narrow; w += gridDim.x * nw) {
        const int2 e = sparse[p.n_qry - 1 - w];
        const int nd = row_dims ? min(nC, (int)__ldg(row_dims + e.x)) : nC;
        const unsigned long long b = scan_query<REF>(p, F, R, nC, nd, e.y, e.x, nT, 0, INT_MAX, 0, 1, qrow, queues[warp],
                                                     buf, lane);
        if (lane == 0) put_delta<REF>(p, R, e.y, e.x, b, nT, delta, nneigh);
    }
    __syncthreads();
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        const int2 item = items[u];
        const int chunk = item.x & 0x0fffffff, part = item.x >> 28, first = item.y >> 5, n = item.y & 31;
        const int ntot = __ldg(p.ncand + chunk);
        const int np = min(kParts, max(1, ntot / kMinDense));
        // REF: the runs as the reference passes them (its bins depend on them)
        const int32_t *prs = REF ? p.rsr : p.rs, *prn = REF ? p.rnr : p.rn;
        const int r0 = __ldg((REF ? p.roffr : p.roff) + chunk), r1 = __ldg((REF ? p.roffr : p.roff) + chunk + 1);
        const int nBB = r1 - r0, nT0 = REF ? nT / nBB : 1;
        const int seg = __ldg(p.qseg + chunk);
        // features that can be non-zero for this chunk's queries and candidates
        // (their site's width, irc_plan_set_site_dims): the rest add exactly 0
        const int nd = row_dims ? min(nC, (int)__ldg(row_dims + __ldg(p.q0 + chunk))) : nC;
        if (threadIdx.x < kQB) {
            const int q = fb_list[seg + first + min((int)threadIdx.x, n - 1)];
            sQ[threadIdx.x] = q;
            sRA[threadIdx.x] = __ldg(R + q);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nd * kQB; i += kThreads) {
            const int c = i / kQB, q = i - c * kQB;
            sA[i] = __ldg(F + (size_t)sQ[q] * nC + c);
        }
        __syncthreads();
        unsigned long long best[kQB];
#pragma unroll
        for (int q = 0; q < kQB; ++q) best[q] = ~0ull;
        float thr[kQB];                                      // REF: distances above it cannot be the minimum
#pragma unroll
        for (int q = 0; q < kQB; ++q) thr[q] = kInfSentinel;
        const int per = (ntot + np - 1) / np, lo = part * per, hi = min(ntot, lo + per);
        int pos = 0;                                         // position of run r's first candidate
        for (int r = r0; r < r1 && pos < hi; ++r) {
            const int rs = __ldg(prs + r), rn = __ldg(prn + r);
            const int a = max(lo - pos, 0), b = min(hi - pos, rn);
            for (int i = a + (int)threadIdx.x; i < b; i += kThreads) {
                const int iB = rs + i;
                const float rb = __ldg(R + iB);
                unsigned live = 0;
#pragma unroll
                for (int q = 0; q < kQB; ++q)
                    if (!(rb <= sRA[q])) live |= 1u << q;
                if (!live) continue;
                float acc[kQB];
                dist_qb<kQB>(F + (size_t)iB * nC, nd, sA, acc);
#pragma unroll
                for (int q = 0; q < kQB; ++q)
                    if (((live >> q) & 1u) && acc[q] > 0.0f && acc[q] < kInfSentinel) {
                        if (REF) {
                            if (acc[q] <= thr[q]) {
                                const unsigned long long key = ref_key(acc[q], (i % nT0) * nBB + (r - r0), i / nT0);
                                best[q] = key < best[q] ? key : best[q];
                                thr[q] = fminf(thr[q], acc[q] * (1.0f + 0x1p-20f));   // every d2 sharing its root
                            }
                        } else {
                            const unsigned long long key = dkey(acc[q], iB);
                            best[q] = key < best[q] ? key : best[q];
                        }
                    }
            }
            pos += rn;
        }
#pragma unroll
        for (int q = 0; q < kQB; ++q) {
            const unsigned long long b = irc::warp_min_u64(best[q]);
            if (lane == 0) redt[q][warp] = b;
        }
        __syncthreads();
        if (threadIdx.x < n) {
            unsigned long long b = redt[threadIdx.x][0];
            for (int w = 1; w < kThreads / 32; ++w) b = redt[threadIdx.x][w] < b ? redt[threadIdx.x][w] : b;
            if (b != ~0ull) atomicMin(keys + (sQ[threadIdx.x] - p.q_base), b);
        }
        __syncthreads();
    }
}

// delta and nneigh of the queries with keys: the wide windows' and the
// 16-query units'.
template <bool REF>
__global__ void k_delta_finish(irc::PlanDev p, const float *__restrict__ R, const int *__restrict__ words,
                               const int2 *__restrict__ sparse, const int2 *__restrict__ items, const int *__restrict__ fb_list,
                               const unsigned long long *__restrict__ keys, float *__restrict__ delta,
                               int *__restrict__ nneigh, int nT)
{
    after_previous(words, sparse, items, fb_list, keys);
    const int total = words[0] * kQB, n_wide = words[1];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_wide; t += gridDim.x * blockDim.x) {
        const int2 e = sparse[t];
        put_delta<REF>(p, R, e.y, e.x, keys[e.x - p.q_base], nT, delta, nneigh);
    }
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int2 item = items[t / kQB];
        const int j = t - (t / kQB) * kQB;
        const int chunk = item.x & 0x0fffffff, first = item.y >> 5, n = item.y & 31;
        if ((item.x >> 28) != 0 || j >= n) continue;        // each tile once (its part 0)
        const int qq = fb_list[__ldg(p.qseg + chunk) + first + j];
        put_delta<REF>(p, R, chunk, qq, keys[qq - p.q_base], nT, delta, nneigh);
    }
}

}  // namespace

constexpr size_t kExactSmem = (size_t)kQB * kCap * 8 + (size_t)kQB * kThreads * 4;
constexpr int kExactBlocks = 3;          // resident on an SM (registers)

static int exact_overflow(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho, int32_t *miKnn,
                          float *d2Knn, int *cnt, int *ovf_list, cudaStream_t s)
{
    // the overflow list is usually empty; size the grid for the worst case
    launch_next(k_exact_overflow, kQueueBlocks, 256, 0, s, pl->dev, F, nC, knn, cnt, ovf_list, vrKnn, rho, miKnn, d2Knn);
    IRC_CHECK_LAUNCH("irc_site_knn(EXACT) overflow");
    return IRC_OK;
}

// The EXACT kernel over the tiles of tq.  As many blocks as run at once: a second
// wave would find its share of the tiles still waiting (100,003 spikes, every
// tile: 26.0 ms with four blocks an SM asked for, 22.3 a tile per block).
int irc_exact_tiles(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho, int32_t *miKnn,
                    float *d2Knn, const irc::TileQueue &tq, cudaStream_t s)
{
    cudaError_t e = cudaFuncSetAttribute(k_site_knn_exact_queue, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExactSmem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(EXACT): smem attribute");
    const int tiles = pl->ntiles[irc::tile_slot(kQB)], most = pl->sms * kExactBlocks;
    launch_next(k_site_knn_exact_queue, tiles < most ? tiles : most, kThreads, kExactSmem, s, pl->dev, F, nC, knn, vrKnn, rho,
                miKnn, d2Knn, tq);
    IRC_CHECK_LAUNCH("irc_site_knn(EXACT)");
    return IRC_OK;
}

int irc_site_knn_exact(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho,
                       int32_t *miKnn, float *d2Knn, cudaStream_t s)
{
    if (knn > kCap / 2) { irc_host::set_error("irc_site_knn(EXACT): knn %d > %d", knn, kCap / 2); return IRC_E_INVAL; }
    int *cnt = pl->scratch, *queue = pl->scratch + irc::kScratchLists;
    cudaError_t e = cudaMemsetAsync(cnt, 0, 2 * sizeof(int), s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(EXACT): memset");
    e = cudaFuncSetAttribute(k_site_knn_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExactSmem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(EXACT): smem attribute");
    k_site_knn_exact<<<pl->ntiles[irc::tile_slot(kQB)], kThreads, kExactSmem, s>>>(pl->dev, F, nC, knn, vrKnn, rho, miKnn, d2Knn,
                                                                                   cnt, queue);
    IRC_CHECK_LAUNCH("irc_site_knn(EXACT)");
    return exact_overflow(pl, F, nC, knn, vrKnn, rho, miKnn, d2Knn, cnt, queue, s);
}

int irc_site_delta_list(irc_plan *pl, const float *F, int nC, const float *R, int knn,
                        const int32_t *miKnn, const float *d2Knn, float *delta, int32_t *nneigh,
                        cudaStream_t s)
{
    const irc_delta_scratch sc = irc_delta_carve(pl, pl->delta_mem, nullptr);
    cudaError_t e = irc_delta_clear(pl, sc, s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_delta: memset");
    const int tiles = pl->ntiles[irc::tile_slot(kListTile)];
    launch_next(k_delta_list, (tiles + kListWarps - 1) / kListWarps, 32 * kListWarps, 0, s, 
        pl->dev, tiles, R, knn, miKnn, d2Knn, delta, nneigh, sc.counts, sc.list);
    IRC_CHECK_LAUNCH("irc_site_delta list");
    return irc_delta_window(pl, F, nC, R, 0, sc, delta, nneigh, s);
}

// Scratch of the drift-window search in mem (delta_bytes(...)).
irc_delta_scratch irc_delta_carve(const irc_plan *pl, void *mem, const int *all)
{
    const size_t n = (size_t)pl->dev.n_qry;
    char *b = (char *)mem;
    irc_delta_scratch sc;
    sc.all = all;
    sc.words = (int *)b;
    sc.counts = sc.words + 4;
    b += delta_part(4 * (4 + (size_t)pl->dev.nChunks));
    sc.list = (int *)b;
    b += delta_part(4 * n);
    sc.sparse = (int2 *)b;
    b += delta_part(8 * n);
    sc.keys = (unsigned long long *)b;
    b += delta_part(8 * (size_t)pl->dev.n_out);
    sc.items = (int2 *)b;
    return sc;
}

cudaError_t irc_delta_clear(const irc_plan *pl, const irc_delta_scratch &sc, cudaStream_t s)
{
    return cudaMemsetAsync(sc.words, 0, 4 * (4 + (size_t)pl->dev.nChunks), s);
}

// The drift-window search of the queries in sc.list (sc.counts of every
// chunk): ties by (d2, row), or by the reference's rule over nT bins (nT > 0).
int irc_delta_window(irc_plan *pl, const float *F, int nC, const float *R, int nT, const irc_delta_scratch &sc,
                     float *delta, int32_t *nneigh, cudaStream_t s)
{
    launch_next(k_delta_items, (pl->dev.nChunks + 7) / 8, 256, 0, s, pl->dev, sc.all, sc.counts, sc.list, sc.words, sc.sparse,
                                                            sc.items, sc.keys);
    IRC_CHECK_LAUNCH("irc_site_delta items");
    auto window = nT > 0 ? k_delta_window<true> : k_delta_window<false>;
    auto finish = nT > 0 ? k_delta_finish<true> : k_delta_finish<false>;
    const size_t smem = (size_t)(kThreads / 32) * 32 * irc::row_pitch(nC) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(window, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_delta: smem attribute");
    launch_next(window, kQueueBlocks, kThreads, smem, s, pl->dev, F, R, nC, pl->row_dims, sc.words, sc.sparse, sc.items, sc.list,
                                             sc.keys, nT, delta, nneigh);
    IRC_CHECK_LAUNCH("irc_site_delta window");
    launch_next(finish, kQueueBlocks / 4, kThreads, 0, s, pl->dev, R, sc.words, sc.sparse, sc.items, sc.list, sc.keys, delta, nneigh, nT);
    IRC_CHECK_LAUNCH("irc_site_delta finish");
    return IRC_OK;
}

// Finish the queries the tensor-core kernel queued (list overflow) with the
// exact ordered-scan kernel; the queue lies in the plan's scratch.
int irc_exact_overflow_drain(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho,
                             int32_t *miKnn, float *d2Knn, cudaStream_t s)
{
    return exact_overflow(pl, F, nC, knn, vrKnn, rho, miKnn, d2Knn, pl->scratch, pl->scratch + irc::kScratchLists, s);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the EXACT site kNN (irc_site_knn_exact_noalloc).
//
// For callers that cannot call cudaMalloc: everything the kernels need
// besides the caller's inputs and outputs -- the device copy of the plan,
// the tile table, the overflow queue and its counter -- lives in the fixed
// array below, which every GPU that loads the library holds until the
// process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocWords = (size_t)2 << 20;     // 8 MiB of int32 words
static __device__ __align__(256) int32_t g_noalloc_scratch[kNoAllocWords];

// Device address of g_noalloc_scratch per device, looked up once per device
// with that device current (a host-side reference to the array is only a
// stand-in, not a device address).  The address belongs to the device's
// primary context: cudaDeviceReset destroys that context and the array with
// it, so a process that resets a device must not call the entry point on that
// device afterwards (the cached address would be stale).
constexpr int kMaxDevices = 64;
int32_t *g_noalloc_ptr[kMaxDevices];
std::mutex g_noalloc_mu;

int noalloc_scratch(int32_t **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn_exact_noalloc: cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) {
        irc_host::set_error("irc_site_knn_exact_noalloc: device %d out of range", dev);
        return IRC_E_INVAL;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn_exact_noalloc: cudaGetSymbolAddress");
        g_noalloc_ptr[dev] = (int32_t *)p;
    }
    *out = g_noalloc_ptr[dev];
    return IRC_OK;
}

// Word offsets of everything the entry point keeps in the fixed array, in
// order: the plan scratch words (queue counters), the overflow queue (2 n_out,
// or all chunks' queries where a query is in several),
// q0 [nChunks], nq [nChunks], roff [nChunks+1], rs [nRuns], rn [nRuns] and
// the 16-query tile table [nChunks+1].  The size check and the pointers both
// come from here, so they cannot disagree.
struct NoAllocLayout {
    size_t q0, nq, roff, rs, rn, tile, total;
};

NoAllocLayout noalloc_layout(long long n_out, long long n_qry, long long nChunks, long long nRuns)
{
    NoAllocLayout L;
    L.q0 = (size_t)irc::kScratchLists + (size_t)(n_qry > 2 * n_out ? n_qry : 2 * n_out);
    L.nq = L.q0 + (size_t)nChunks;
    L.roff = L.nq + (size_t)nChunks;
    L.rs = L.roff + (size_t)nChunks + 1;
    L.rn = L.rs + (size_t)nRuns;
    L.tile = L.rn + (size_t)nRuns;
    L.total = L.tile + (size_t)nChunks + 1;
    return L;
}

// tile_off[i] = sum_{j<i} ceil(nq[j] / QB), one block, chunked scan.
__global__ void k_noalloc_tiles(const int32_t *__restrict__ nq, int nChunks, int qb, int32_t *__restrict__ tile_off)
{
    __shared__ int32_t part[1024];
    const int t = threadIdx.x, nt = blockDim.x;
    const int per = (nChunks + nt - 1) / nt;
    const int lo = min(t * per, nChunks), hi = min(lo + per, nChunks);
    int32_t s = 0;
    for (int i = lo; i < hi; ++i) s += (nq[i] + qb - 1) / qb;
    part[t] = s;
    __syncthreads();
    if (t == 0) {
        int32_t acc = 0;
        for (int i = 0; i < nt; ++i) { const int32_t v = part[i]; part[i] = acc; acc += v; }
    }
    __syncthreads();
    int32_t acc = part[t];
    for (int i = lo; i < hi; ++i) { tile_off[i] = acc; acc += (nq[i] + qb - 1) / qb; }
    if (hi == nChunks && lo < hi) tile_off[nChunks] = acc;
    if (nChunks == 0 && t == 0) tile_off[0] = 0;
}

}  // namespace

extern "C" int irc_site_knn_exact_noalloc(const float *F, int nC, const int32_t *q0, const int32_t *nq,
                                          const int32_t *roff, const int32_t *rs, const int32_t *rn, int nChunks,
                                          int q_base, int n_out, int nF, int knn, float *vrKnn, float *rho,
                                          int32_t *miKnn, float *d2Knn, void *stream)
{
    const char *me = "irc_site_knn_exact_noalloc";
    if (!F || !vrKnn || !miKnn) {
        irc_host::set_error("%s: null pointer", me);
        return IRC_E_INVAL;
    }
    if (nC > IRC_NC_MAX) { irc_host::set_error("%s: nC=%d > %d", me, nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || knn <= 0 || knn > kCap / 2) { irc_host::set_error("%s: bad nC=%d / knn=%d", me, nC, knn); return IRC_E_INVAL; }
    // the same checks as irc_plan_create (64-bit bounds)
    int rc = irc_host::check_plan(me, q0, nq, roff, rs, rn, nChunks, q_base, n_out, nF, nullptr, nullptr);
    if (rc != IRC_OK) return rc;
    const int nRuns = roff[nChunks];
    long long n_qry = 0;
    for (int i = 0; i < nChunks; ++i) n_qry += nq[i];
    const NoAllocLayout L = noalloc_layout(n_out, n_qry, nChunks, nRuns);
    if (L.total > kNoAllocWords) {
        irc_host::set_error("%s: plan needs %zu scratch words (4 + 2*n_out + 4*chunks + 2 + 2*runs), "
                            "the fixed array holds %zu", me, L.total, kNoAllocWords);
        return IRC_E_INVAL;
    }
    long long tiles = 0;
    for (int i = 0; i < nChunks; ++i) tiles += (nq[i] + kQB - 1) / kQB;
    int32_t *base = nullptr;
    rc = noalloc_scratch(&base);
    if (rc != IRC_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    int32_t *d_q0 = base + L.q0, *d_nq = base + L.nq, *d_roff = base + L.roff;
    int32_t *d_rs = base + L.rs, *d_rn = base + L.rn, *d_tile = base + L.tile;
    cudaError_t e = cudaMemsetAsync(base, 0, irc::kScratchLists * sizeof(int32_t), s);    // counters start at zero
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_q0, q0, 4 * (size_t)nChunks, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_nq, nq, 4 * (size_t)nChunks, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_roff, roff, 4 * ((size_t)nChunks + 1), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_rs, rs, 4 * (size_t)nRuns, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_rn, rn, 4 * (size_t)nRuns, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn_exact_noalloc: upload");
    k_noalloc_tiles<<<1, 1024, 0, s>>>(d_nq, nChunks, kQB, d_tile);
    IRC_CHECK_LAUNCH("irc_site_knn_exact_noalloc tiles");
    irc::PlanDev p;
    p.q0 = d_q0; p.nq = d_nq; p.roff = d_roff; p.rs = d_rs; p.rn = d_rn;
    p.roffr = d_roff; p.rsr = d_rs; p.rnr = d_rn;         // the EXACT kernels take any run split
    for (int k = 0; k < irc::kNumTileSizes; ++k) p.tile_off[k] = d_tile;     // only the 16-query table is read
    p.ncand = p.qseg = nullptr;                           // read only by the delta kernels
    p.tc_toff = nullptr;                                  // read only by the tensor-core filter
    p.tc_tiles = nullptr;
    p.stat = nullptr;
    p.n_qry = (int)(n_qry < INT32_MAX ? n_qry : INT32_MAX);
    p.nChunks = nChunks; p.q_base = q_base; p.n_out = n_out; p.nF = nF; p.nRuns = nRuns;
    e = cudaFuncSetAttribute(k_site_knn_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExactSmem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn_exact_noalloc: smem attribute");
    int32_t *cnt = base, *queue = base + irc::kScratchLists;
    k_site_knn_exact<<<(unsigned)tiles, kThreads, kExactSmem, s>>>(p, F, nC, knn, vrKnn, rho, miKnn, d2Knn, cnt, queue);
    IRC_CHECK_LAUNCH("irc_site_knn_exact_noalloc");
    launch_next(k_exact_overflow, kQueueBlocks, 256, 0, s, p, F, nC, knn, cnt, queue, vrKnn, rho, miKnn, d2Knn);
    IRC_CHECK_LAUNCH("irc_site_knn_exact_noalloc overflow");
    return IRC_OK;
}
