// irc_dropin.cu -- the five drop-in kernels (one call == one MATLAB feval).
//
// Each kernel reproduces the output arrays of the reference kernel it
// replaces bit for bit, but is organised for sm_103a: many queries per CTA
// (fewer re-reads of the candidate features from L2), candidate rows staged by
// asynchronous copies and shared between queries (irc_rows.cuh), bins or
// candidate strides walked by independent threads, and warp- and cluster-level
// arg-min reductions in place of the reference's single-thread loops.
#include <algorithm>
#include <climits>
#include <cooperative_groups.h>
#include <type_traits>

#include "irc_common.cuh"
#include "irc_rerank.cuh"
#include "irc_rows.cuh"
#include "irc_scan.cuh"

namespace {

constexpr int kQB = 16;         // queries per thread (search kernels) or CTA

// Shared memory of a scan CTA of nw warps: 16 ng query rows, and per block of
// 64 candidate rows (nw / ng of them) two stages, which also hold the minima
// of all blocks but the first when they are put together.
constexpr int kScanThreads = 128, kScanWarps = kScanThreads / 32;
__host__ __device__ inline size_t scan_smem(int nC, int ng, int nw = kScanWarps)
{
    const size_t ns = nw / ng, stages = ns * 2 * 64 * irc::row_pitch(nC), mins = (ns - 1) * ng * kQB * 64;
    return ((size_t)nC * kQB * ng + (stages > mins ? stages : mins)) * sizeof(float);
}

// search_min_drift / search_delta_drift: D, I [nT x nA].  A CTA of NW warps
// takes 16 NG queries and 64 of the nT bins (thread t of the reference's block
// scans run t % nBB from t / nBB in steps of nT / nBB), a thread two bins and
// 16 queries; the NW / NG sets of NG warps take the bins' steps in turn, and
// their minima are put together (the smallest, then the first row, as a bin's
// own scan leaves it).  A thread's minima stay in registers over the bins'
// candidates, whose rows are staged a step ahead (irc_rows.cuh); a minimum's
// row number changes rarely and lives in shared memory (in registers it costs
// a fourth CTA per SM).  2,000 queries x 30,000 candidates x 33 features: the
// FP32 pipe's rate allows 100 us; 400 us with a lane's features read from
// global memory and one CTA for all bins, 230 as below (the distances alone
// 180, the copies 45).
template <bool DELTA, int NG, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
k_search_drift(float *__restrict__ D, int *__restrict__ I, const float *__restrict__ F,
               const float *__restrict__ R, const int *__restrict__ IBB,
               const int *__restrict__ NBB, int nC, int nBB, int iA0, int nA, int nT)
{
    constexpr int NS = NW / NG, NT = 32 * NW;
    extern __shared__ __align__(16) float scan_sm[];
    __shared__ __align__(16) float sRA[kQB * NG];
    const int lane = threadIdx.x & 31, g = (threadIdx.x >> 5) % NG, sub = (threadIdx.x >> 5) / NG;
    const int P = irc::row_pitch(nC);
    const float *sA = scan_sm + g * nC * kQB;
    float *buf = scan_sm + nC * kQB * NG + sub * (2 * 64 * P);     // [2][64][P]
    // row numbers: this thread's of query q, bin h at mi[(q * 2 + h) * NT]
    int *mi = reinterpret_cast<int *>(scan_sm + scan_smem(nC, NG, NW) / sizeof(float)) + threadIdx.x;
    const int c0 = blockIdx.x * kQB * NG;            // first query of this CTA (chunk-relative)
    irc::stage_negated<kQB, NG>(F, nC, iA0 + c0, min(kQB * NG, nA - c0), scan_sm);
    if (DELTA && threadIdx.x < kQB * NG) sRA[threadIdx.x] = __ldg(R + iA0 + min(c0 + (int)threadIdx.x, nA - 1));
    __syncthreads();
    const int a0 = c0 + g * kQB, n = min(kQB, nA - a0);            // this warp's queries (n <= 0: none)
    const int nT0 = nT / nBB;                        // a step; this set of warps takes every NS-th
    const irc::RowCopy<NG> rc(nC, lane, g);
    int t[2], row[2], end[2];
    float mn[2][kQB];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        // bins run by run (consecutive lanes then scan consecutive rows), the left-over ones last
        const int k = blockIdx.y * 64 + h * 32 + lane;
        const int b = k < nT0 * nBB ? k / nT0 : k - nT0 * nBB, off = k < nT0 * nBB ? k - b * nT0 : nT0;
        t[h] = off * nBB + b;
        row[h] = end[h] = 0;
        if (k >= nT) t[h] = nT;
        else {
            const int ib0 = __ldg(IBB + b);
            row[h] = ib0 + off + sub * nT0;
            end[h] = ib0 + __ldg(NBB + b);
        }
#pragma unroll
        for (int q = 0; q < kQB; ++q) mn[h][q] = IRC_SINGLE_INF_F;
    }
    auto stage = [&](int s) {
        const int r[2] = {row[0] < end[0] ? row[0] : -1, row[1] < end[1] ? row[1] : -1};
        rc.issue(buf + s * 64 * P, P, F, nC, r);
        irc::copies_commit();
    };
    stage(0);
    // (the warps that share a block hold the same rows and take the same steps)
    for (int s = 0; __any_sync(0xffffffffu, row[0] < end[0] || row[1] < end[1]); s ^= 1) {
        const int at[2] = {row[0], row[1]};
        row[0] += NS * nT0;
        row[1] += NS * nT0;
        stage(s ^ 1);
        unsigned live[2] = {at[0] < end[0] ? 0xffffu : 0u, at[1] < end[1] ? 0xffffu : 0u};   // queries a row may serve
        if (DELTA) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (live[h]) live[h] = irc::higher_rho<kQB>(__ldg(R + at[h]), sRA + g * kQB);
        }
        irc::copies_wait<1>();
        irc::rows_sync<NG>(sub);
        float d[2][kQB];
        irc::pair_dist<kQB>(buf + (s * 64 + lane) * P, buf + (s * 64 + 32 + lane) * P, nC, sA, d[0], d[1]);
        irc::rows_sync<NG>(sub);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < kQB; ++q) {
                const bool less = ((live[h] >> q) & 1u) & (unsigned)(d[h][q] < mn[h][q]) & (unsigned)(d[h][q] > 0.0f);
                if (less) mi[(q * 2 + h) * NT] = at[h];
                mn[h][q] = less ? d[h][q] : mn[h][q];
            }
    }
    irc::copies_wait<0>();
    if (NS > 1) {
        float *bm = scan_sm + nC * kQB * NG + (threadIdx.x & (32 * NG - 1));     // [NS - 1][kQB][2][32 NG]
        __syncthreads();
        if (sub > 0) {
#pragma unroll
            for (int q = 0; q < kQB; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) bm[(((sub - 1) * kQB + q) * 2 + h) * 32 * NG] = mn[h][q];
        }
        __syncthreads();
        if (sub > 0) return;
#pragma unroll
        for (int v = 1; v < NS; ++v)
#pragma unroll
            for (int q = 0; q < kQB; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float x = bm[(((v - 1) * kQB + q) * 2 + h) * 32 * NG];
                    int *own = mi + (q * 2 + h) * NT;
                    if (x < IRC_SINGLE_INF_F && (x < mn[h][q] || (x == mn[h][q] && own[v * 32 * NG] < *own))) {
                        mn[h][q] = x;
                        *own = own[v * 32 * NG];
                    }
                }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (t[h] < nT) {
#pragma unroll
            for (int q = 0; q < kQB; ++q)
                if (q < n) {
                    const size_t o = (size_t)t[h] + (size_t)nT * (a0 + q);
                    D[o] = irc::ref_sqrt_abs(mn[h][q]);
                    I[o] = (mn[h][q] < IRC_SINGLE_INF_F ? mi[(q * 2 + h) * NT] : iA0 + a0 + q) + 1;
                }
        }
}

// The same for short scans: 16 queries a CTA, a bin a thread, rows read where
// they are.  A bin of a few rows is over before the kernel above has staged
// them.
constexpr int kDirectThreads = 256;

template <bool DELTA>
__global__ void __launch_bounds__(kDirectThreads)
k_search_direct(float *__restrict__ D, int *__restrict__ I, const float *__restrict__ F,
                const float *__restrict__ R, const int *__restrict__ IBB,
                const int *__restrict__ NBB, int nC, int nBB, int iA0, int nA, int nT)
{
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ float sRA[kQB];
    const int a0 = blockIdx.x * kQB;                 // first query of this CTA (chunk-relative)
    const int n = min(kQB, nA - a0);
    irc::stage_queries<kQB>(F, nC, iA0 + a0, n, sA);
    if (DELTA && threadIdx.x < kQB) sRA[threadIdx.x] = __ldg(R + iA0 + a0 + min((int)threadIdx.x, n - 1));
    __syncthreads();
    const int nT0 = nT / nBB;
    for (int t = threadIdx.x; t < nT; t += blockDim.x) {
        const int b = t % nBB;
        const int ib0 = __ldg(IBB + b), nb0 = __ldg(NBB + b);
        float mn[kQB];
        int mi[kQB];
#pragma unroll
        for (int q = 0; q < kQB; ++q) { mn[q] = IRC_SINGLE_INF_F; mi[q] = iA0 + a0 + min(q, n - 1); }
        irc::scan_bin<kQB, DELTA>(F, R, nC, ib0 + t / nBB, ib0 + nb0, nT0, sA, sRA, mn, mi);
#pragma unroll
        for (int q = 0; q < kQB; ++q)
            if (q < n) {
                const size_t o = (size_t)t + (size_t)nT * (a0 + q);
                D[o] = irc::ref_sqrt_abs(mn[q]);
                I[o] = mi[q] + 1;
            }
    }
}

// Which of the two: by the row features that a thread of k_search_direct reads
// (bins a thread x rows a bin, if the window is all of F, x nC), among windows of
// some thousand rows at most, or queries for two turns of the chip.  Several runs
// cost the kernel above more (its blocks of 64 bins straddle them).  us, direct |
// staged, D = 12 (kNN with 1,024 bins, delta with 512): 300 x 300 one run 8.6 | 9.1,
// 7.3 | 9.0; 1,000 x 1,000 in 15 runs 11.1 | 15.9, 10.5 | 13.8, one run 10.7 | 10.1,
// 10.6 | 12.4; 50 x 1,000 11.0 | 8.7, 10.4 | 11.9; 5,000 x 5,000 in 15 runs 55 | 59, 77 | 62.
template <bool DELTA>
inline bool direct_search(int nF, int nC, int nBB, int nA, int nT)
{
    if (nF <= 0) return false;
    const long long w = (long long)((nT + kDirectThreads - 1) / kDirectThreads) * ((nF - 1) / nT + 1) * nC;
    if (nBB > 1 && nA >= 2 * 152 * kQB && w <= (DELTA ? 120 : 240)) return true;
    return DELTA ? nF <= 2048 && w <= (nBB > 1 ? 100 : 72) : nF <= 1024 && nA > 64 && w <= (nBB > 1 ? 180 : 48);
}

template <bool DELTA>
int launch_search(float *D, int32_t *I, const float *F, const float *R, const int32_t *IBB, const int32_t *NBB, int nF,
                  int nC, int nBB, int iA0, int nA, int nT, cudaStream_t s, const char *who)
{
    if (direct_search<DELTA>(nF, nC, nBB, nA, nT)) {
        k_search_direct<DELTA><<<(nA + kQB - 1) / kQB, kDirectThreads, 0, s>>>(D, I, F, R, IBB, NBB, nC, nBB, iA0, nA, nT);
        IRC_CHECK_LAUNCH(who);
        return IRC_OK;
    }
    // 64 queries share the staged rows when there are so many; 8 warps a CTA when 4 would leave the
    // SMs fewer than three CTAs (kNN, 1,024 bins: 512 CTAs of 4; delta, 512 bins: 256 of 8)
    const int cols = (nT + 63) / 64, ng = nA > 32 ? 4 : nA > 16 ? 2 : 1;
    const bool big = scan_smem(nC, ng, 8) + (size_t)kQB * 64 * 8 * sizeof(int) > 232448 - 1024;     // (wide rows, few queries)
    const int nw = big || (nA + kQB * ng - 1) / (kQB * ng) * cols >= 3 * 152 ? 4 : 8;
    auto kern = nw == 4 ? (ng == 4 ? k_search_drift<DELTA, 4, 4> : ng == 2 ? k_search_drift<DELTA, 2, 4> : k_search_drift<DELTA, 1, 4>)
                        : (ng == 4 ? k_search_drift<DELTA, 4, 8> : ng == 2 ? k_search_drift<DELTA, 2, 8> : k_search_drift<DELTA, 1, 8>);
    const size_t smem = scan_smem(nC, ng, nw) + (size_t)kQB * 64 * nw * sizeof(int);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, who);
    const dim3 grid((nA + kQB * ng - 1) / (kQB * ng), cols);
    kern<<<grid, 32 * nw, smem, s>>>(D, I, F, R, IBB, NBB, nC, nBB, iA0, nA, nT);
    IRC_CHECK_LAUNCH(who);
    return IRC_OK;
}

// The binned minimum + selection sort of cuda_knn_index, cuda_knn,
// cuda_knn_full and cuda_knn_ib: per-bin minimum over iiB = t, t+nT, ...
// (self kept; IND maps iiB through IB, 1-based, and records the mapped
// column), then the reference's in-kernel selection sort with swaps, one warp
// per query (each step = first position of the minimum over [iK, nT)).  The
// swaps only matter between equal values: when the knn smallest bins and the
// next have different values, a threshold search and a sort of the ~knn bins
// below it give the same order in about a third of the instructions; ties take
// the steps as they stand.  (A bin's value is never NaN: only distances below
// the sentinel replace it.)  A cluster of CTAs takes 32 queries, a CTA 64 of
// the bins per turn (scanned as in k_search_drift), so that 1,500 queries make
// 380 CTAs; after the scan each warp collects a query's bins from the cluster's shared memories.  KALL
// writes every sorted distance [knn x nA], else the knn-th [nA]; I is
// optional.  IB entries outside 1..nF are skipped and counted in *bad.
// The steps of a bin are dealt to two sets of warps, each with its own table
// (a warp issues an instruction every ~4 cycles here: 192 CTAs of 4 warps took
// 134 us for 1,507 queries x 15,000 candidates x 30 features).
constexpr int kBinNG = 2, kBinBlocks = 1, kBinSets = 2, kBinWarps = kBinNG * kBinBlocks * kBinSets;
constexpr int kBinQ = kQB * kBinNG, kBinTurn = 64 * kBinBlocks;

// shared memory: the scan's, whose stages then hold a row of all nT bins per
// warp, and the CTA's bin tables [kBinSets][turns][kBinQ][kBinTurn] of (value, row)
__host__ __device__ inline size_t bins_scan_smem(int nC, int nT)
{
    const size_t a = scan_smem(nC, kBinNG, kBinWarps), b = 8 * (size_t)kBinWarps * nT;
    return a > b ? a : b;
}
size_t bins_smem(int nC, int nT, int turns)
{
    return bins_scan_smem(nC, nT) + 8 * (size_t)kBinSets * turns * kBinQ * kBinTurn;
}

template <bool IND, bool KALL>
__global__ void __launch_bounds__(32 * kBinWarps, 4)
k_knn_bins(float *__restrict__ K, int *__restrict__ I, const float *__restrict__ B,
           const float *__restrict__ A, const int *__restrict__ IB, int nF, int *__restrict__ bad, int nB, int nA,
           int nC, int knn, int nT, int turns)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) float scan_sm[];
    __shared__ unsigned long long wkeys[kBinWarps][irc_rr::WARP_KEYS];
    auto cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), nr = (int)cluster.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = warp % kBinNG, sub = warp / kBinNG;
    const int block = sub % kBinBlocks, set = sub / kBinBlocks;
    const int P = irc::row_pitch(nC);
    const float *sA = scan_sm + g * nC * kQB;
    float *buf = scan_sm + nC * kBinQ + sub * (2 * 64 * P);
    float2 *table = reinterpret_cast<float2 *>(scan_sm + bins_scan_smem(nC, nT) / sizeof(float));
    float *rowd = scan_sm + warp * 2 * nT;
    const int tsize = turns * kBinQ * kBinTurn;
    const int a0 = blockIdx.x * kBinQ, n = min(kBinQ, nA - a0);
    irc::stage_negated<kQB, kBinNG>(A, nC, a0, n, scan_sm);
    __syncthreads();
    const irc::RowCopy<kBinNG> rc(nC, lane, g);
    for (int u = 0; u < turns; ++u) {
        // this warp's bins of the turn: the cluster takes nr * kBinTurn at a time
        const int tb = (u * nr + rank) * kBinTurn + block * 64;
        int t[2], at[2], row[2];                             // bins, list positions and rows of the next step
        float mn[2][kQB];
        float2 *own = table + set * tsize + (u * kBinQ + g * kQB) * kBinTurn + block * 64 + lane;     // bin h of query q at own[q * kBinTurn + 32 h]
        auto look = [&](int h) {                             // the row at list position at[h], or -1
            row[h] = -1;
            if (t[h] >= nT || at[h] >= nB) return;
            int iB = at[h];
            if (IND) {
                iB = __ldg(IB + at[h]) - 1;
                if (iB < 0 || iB >= nF) {
                    if (blockIdx.x == 0 && g == 0) atomicAdd(bad, 1);
                    return;
                }
            }
            row[h] = iB;
        };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            t[h] = tb + h * 32 + lane;
            at[h] = t[h] + set * nT;
#pragma unroll
            for (int q = 0; q < kQB; ++q) {
                mn[h][q] = IRC_SINGLE_INF_F;
                own[q * kBinTurn + 32 * h].y = __int_as_float(-1);   // list position of the minimum
            }
        }
        auto stage = [&](int s) {
            look(0);
            look(1);
            rc.issue(buf + s * 64 * P, P, B, nC, row);
            irc::copies_commit();
        };
        stage(0);
        const int steps = (nB - tb - set * nT + kBinSets * nT - 1) / (kBinSets * nT);     // of the block's first bin, the most of any
        for (int k = 0, s = 0; k < steps; ++k, s ^= 1) {
            const int cur[2] = {row[0], row[1]}, pos[2] = {at[0], at[1]};
            at[0] += kBinSets * nT;
            at[1] += kBinSets * nT;
            stage(s ^ 1);
            irc::copies_wait<1>();
            irc::rows_sync<kBinNG>(sub);
            float d[2][kQB];
            irc::pair_dist<kQB>(buf + (s * 64 + lane) * P, buf + (s * 64 + 32 + lane) * P, nC, sA, d[0], d[1]);
            irc::rows_sync<kBinNG>(sub);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (cur[h] >= 0) {
#pragma unroll
                    for (int q = 0; q < kQB; ++q)
{
                            const bool less = d[h][q] < mn[h][q];
                            if (less) own[q * kBinTurn + 32 * h].y = __int_as_float(pos[h]);
                            mn[h][q] = less ? d[h][q] : mn[h][q];
                        }
                }
        }
        irc::copies_wait<0>();
        irc::rows_sync<kBinNG>(sub);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < kQB; ++q) own[q * kBinTurn + 32 * h].x = mn[h][q];
    }
    cluster.sync();
    // 1-based B column of a list position (1 for a bin without candidates)
    auto column = [&](int at) { return at < 0 ? 1 : IND ? __ldg(IB + at) : at + 1; };
    for (int q = rank * kBinWarps + warp; q < n; q += nr * kBinWarps) {
        float *d = rowd;
        int *ix = reinterpret_cast<int *>(rowd + nT);
        for (int t = lane; t < nT; t += 32) {
            const int o = t / kBinTurn, u = o / nr;
            const float2 *p = cluster.map_shared_rank(table + (u * kBinQ + q) * kBinTurn + (t - o * kBinTurn), o - u * nr);
            // the sets' minima: the smaller, of equal ones the earlier step's
            const float2 v = p[0], w = p[tsize];
            const bool second = w.x < v.x || (w.x == v.x && w.x < IRC_SINGLE_INF_F && __float_as_int(w.y) < __float_as_int(v.y));
            d[t] = second ? w.x : v.x;
            ix[t] = __float_as_int(second ? w.y : v.y);
        }
        __syncwarp();
        const int qa = a0 + q;
        // the knn smallest by selection; false where ties want the reference's steps
        auto select = [&](auto per) {
            constexpr int PER = decltype(per)::value;
            unsigned long long kv[PER], *ws = wkeys[warp];
#pragma unroll
            for (int i = 0; i < PER; ++i) kv[i] = i * 32 + lane < nT ? irc::sort_key(d[i * 32 + lane], i * 32 + lane) : ~0ull;
            unsigned tbits;
            const int m = irc_rr::select_keys<PER>(kv, knn, ws, lane, tbits);
            if (m < knn || m > irc_rr::WARP_KEYS) return false;
            bool tie = false;
            for (int e = lane; e < knn; e += 32) tie |= e + 1 < m && (ws[e] >> 32) == (ws[e + 1] >> 32);
            if (__any_sync(0xffffffffu, tie)) return false;
            for (int e = lane; e < knn; e += 32) {
                const float v = irc::ref_sqrt_abs(__uint_as_float((unsigned)(ws[e] >> 32)));
                if (KALL) K[e + (size_t)knn * qa] = v;
                else if (e == knn - 1) K[qa] = v;
                if (I) I[e + (size_t)knn * qa] = column(ix[(int)(ws[e] & 0xffffffffu)]);
            }
            __syncwarp();
            return true;
        };
        // (2,000 queries x 2,000 candidates, 1,024 bins: 103 us with the steps, 60 so)
        if (nT <= 512 ? select(std::integral_constant<int, 16>{}) : select(std::integral_constant<int, 32>{})) continue;
        for (int iK = 0; iK < knn; ++iK) {
            unsigned long long best = ~0ull;
            for (int p = iK + lane; p < nT; p += 32) {
                const unsigned long long k = irc::sort_key(d[p], p);
                best = k < best ? k : best;
            }
            best = irc::warp_min_u64(best);
            if (lane == 0) {
                const int p = (int)(best & 0xffffffffu);
                const float tf = d[p]; d[p] = d[iK]; d[iK] = tf;
                const int ti = ix[p]; ix[p] = ix[iK]; ix[iK] = ti;
            }
            __syncwarp();
        }
        if (KALL) {
            for (int iK = lane; iK < knn; iK += 32) K[iK + (size_t)knn * qa] = irc::ref_sqrt_abs(d[iK]);
        } else if (lane == 0) {
            K[qa] = irc::ref_sqrt_abs(d[knn - 1]);
        }
        if (I)
            for (int iK = lane; iK < knn; iK += 32) I[iK + (size_t)knn * qa] = column(ix[iK]);
        __syncwarp();
    }
    cluster.sync();                                          // the CTA's table is read
}

// cuda_delta_knn: thread t keeps the minimum over iB = t, t+128, ... with
// R_B > R_A (strict), then the lowest slot holding the overall minimum wins,
// i.e. the smallest (d2, iB % 128, iB); when no slot found a candidate the
// index falls back to the query (A-space).  A cluster of CTAs shares the
// candidates of kQB queries (a strided slice each, so that a few hundred
// queries fill the chip), every thread two candidates a step, staged as in
// k_search_drift; CTA 0 takes the least of the cluster's keys.
template <int NG, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
k_delta_knn(float *__restrict__ D, unsigned *__restrict__ N, const float *__restrict__ B,
            const float *__restrict__ A, const float *__restrict__ RB, const float *__restrict__ RA,
            int nB, int nA, int nC)
{
    namespace cg = cooperative_groups;
    constexpr int NS = NW / NG, NT = 32 * NW;
    extern __shared__ __align__(16) float scan_sm[];
    __shared__ __align__(16) float sRA[kQB * NG];
    __shared__ unsigned long long sKey[kQB * NG];
    const int lane = threadIdx.x & 31, g = (threadIdx.x >> 5) % NG, sub = (threadIdx.x >> 5) / NG;
    const int P = irc::row_pitch(nC);
    const float *sA = scan_sm + g * nC * kQB;
    float *buf = scan_sm + nC * kQB * NG + sub * (2 * 64 * P);
    int *mi = reinterpret_cast<int *>(scan_sm + scan_smem(nC, NG, NW) / sizeof(float)) + threadIdx.x;   // as in k_search_drift
    const int a0 = blockIdx.x * kQB * NG;
    const int n = min(kQB * NG, nA - a0);
    irc::stage_negated<kQB, NG>(A, nC, a0, n, scan_sm);
    if (threadIdx.x < kQB * NG) {
        sRA[threadIdx.x] = __ldg(RA + a0 + min((int)threadIdx.x, n - 1));
        sKey[threadIdx.x] = ~0ull;
    }
    __syncthreads();
    float low = __int_as_float(0x7f800000);                  // no query takes a candidate with rho <= low
    for (int q = 0; q < kQB * NG; ++q) low = fminf(low, sRA[q]);
    const irc::RowCopy<NG> rc(nC, lane, g);
    // blocks of 64 candidates, dealt over the cluster's CTAs and their sub-blocks in turn
    const int step = gridDim.y * NS * 64, first = (blockIdx.y * NS + sub) * 64;
    int at[2] = {first + lane, first + 32 + lane}, row[2];
    float rb[2];
    float mn[2][kQB];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < kQB; ++q) mn[h][q] = IRC_SINGLE_INF_F;
    auto stage = [&](int s) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            row[h] = at[h] < nB ? at[h] : -1;
            rb[h] = at[h] < nB ? __ldg(RB + at[h]) : low;
        }
        if (__any_sync(0xffffffffu, rb[0] > low || rb[1] > low)) rc.issue(buf + s * 64 * P, P, B, nC, row);
        irc::copies_commit();
    };
    stage(0);
    for (int k = first, s = 0; k < nB; k += step, s ^= 1) {
        const int cur[2] = {row[0], row[1]};
        const unsigned live[2] = {row[0] < 0 ? 0u : irc::strictly_higher_rho<kQB>(rb[0], sRA + g * kQB),
                                  row[1] < 0 ? 0u : irc::strictly_higher_rho<kQB>(rb[1], sRA + g * kQB)};
        at[0] += step;
        at[1] += step;
        stage(s ^ 1);
        irc::copies_wait<1>();
        irc::rows_sync<NG>(sub);
        float d[2][kQB];
        irc::pair_dist<kQB>(buf + (s * 64 + lane) * P, buf + (s * 64 + 32 + lane) * P, nC, sA, d[0], d[1]);
        irc::rows_sync<NG>(sub);
        // equal distances are settled by the key's order (iB % 128 first), not by who came first
        bool equal = false;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < kQB; ++q) {
                const bool on = (live[h] >> q) & 1u, less = on & (d[h][q] < mn[h][q]);
                equal |= on & (d[h][q] == mn[h][q]);
                if (less) mi[(q * 2 + h) * NT] = cur[h];
                mn[h][q] = less ? d[h][q] : mn[h][q];
            }
        if (equal) {                                         // (a distance just taken over compares equal to itself: no change)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < kQB; ++q) {
                    int *own = mi + (q * 2 + h) * NT;
                    if (((live[h] >> q) & 1u) && d[h][q] == mn[h][q] && d[h][q] < IRC_SINGLE_INF_F &&
                        (cur[h] & 127) < (*own & 127))
                        *own = cur[h];
                }
        }
    }
    irc::copies_wait<0>();
#pragma unroll
    for (int q = 0; q < kQB; ++q) {
        unsigned long long k = ~0ull;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (mn[h][q] < IRC_SINGLE_INF_F) {
                const int j = mi[(q * 2 + h) * NT];
                const unsigned long long e = ((unsigned long long)__float_as_uint(mn[h][q]) << 32) |
                                             ((unsigned)(j & 127) << 25) | (unsigned)(j >> 7);
                k = e < k ? e : k;
            }
        k = irc::warp_min_u64(k);
        if (lane == 0 && k != ~0ull) atomicMin(sKey + g * kQB + q, k);
    }
    auto cluster = cg::this_cluster();
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x < n) {
        unsigned long long k = ~0ull;
        for (unsigned r = 0; r < cluster.num_blocks(); ++r) {
            const unsigned long long e = *cluster.map_shared_rank(sKey + threadIdx.x, r);
            k = e < k ? e : k;
        }
        const bool found = k != ~0ull;
        const unsigned lo = (unsigned)k;
        const int qa = a0 + threadIdx.x;
        D[qa] = irc::ref_sqrt_abs(found ? __uint_as_float((unsigned)(k >> 32)) : IRC_SINGLE_INF_F);
        N[qa] = (found ? ((lo & 0x1ffffffu) << 7 | lo >> 25) : (unsigned)qa) + 1u;
    }
    cluster.sync();                                          // the other CTAs' keys are read
}

// The same without staging: 16 queries a CTA of the reference's 128 threads, rows
// read where they are.
__global__ void __launch_bounds__(128)
k_delta_direct(float *__restrict__ D, unsigned *__restrict__ N, const float *__restrict__ B,
               const float *__restrict__ A, const float *__restrict__ RB, const float *__restrict__ RA,
               int nB, int nA, int nC)
{
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ __align__(16) float sRA[kQB];
    __shared__ unsigned long long sKey[kQB][4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int a0 = blockIdx.x * kQB;
    const int n = min(kQB, nA - a0);
    irc::stage_queries<kQB>(A, nC, a0, n, sA);
    if (t < kQB) sRA[t] = __ldg(RA + a0 + min(t, n - 1));
    __syncthreads();
    float mn[kQB];
    int mi[kQB];
#pragma unroll
    for (int q = 0; q < kQB; ++q) { mn[q] = IRC_SINGLE_INF_F; mi[q] = 0; }
    for (int iB = t; iB < nB; iB += 128) {
        const unsigned live = irc::strictly_higher_rho<kQB>(__ldg(RB + iB), sRA);
        if (!live) continue;
        const float *fb = B + (size_t)iB * nC;
        float acc[kQB];
#pragma unroll
        for (int q = 0; q < kQB; ++q) acc[q] = 0.0f;
        for (int c = 0; c < nC; ++c) {
            const float bv = __ldg(fb + c);
            const float4 *a4 = reinterpret_cast<const float4 *>(sA + c * kQB);
#pragma unroll
            for (int j = 0; j < kQB / 4; ++j) {
                const float4 a = a4[j];
                acc[4 * j + 0] = irc::dterm(acc[4 * j + 0], bv, a.x);
                acc[4 * j + 1] = irc::dterm(acc[4 * j + 1], bv, a.y);
                acc[4 * j + 2] = irc::dterm(acc[4 * j + 2], bv, a.z);
                acc[4 * j + 3] = irc::dterm(acc[4 * j + 3], bv, a.w);
            }
        }
#pragma unroll
        for (int q = 0; q < kQB; ++q)
            if (((live >> q) & 1u) && acc[q] < mn[q]) { mn[q] = acc[q]; mi[q] = iB; }
    }
#pragma unroll
    for (int q = 0; q < kQB; ++q) {
        // (a thread's rows share iB % 128, its first strict minimum is the first)
        unsigned long long k = ~0ull;
        if (mn[q] < IRC_SINGLE_INF_F)
            k = ((unsigned long long)__float_as_uint(mn[q]) << 32) | ((unsigned)t << 25) | (unsigned)(mi[q] >> 7);
        k = irc::warp_min_u64(k);
        if (lane == 0) sKey[q][warp] = k;
    }
    __syncthreads();
    if (t < n) {
        unsigned long long k = sKey[t][0];
        for (int w = 1; w < 4; ++w) k = sKey[t][w] < k ? sKey[t][w] : k;
        const bool found = k != ~0ull;
        const unsigned lo = (unsigned)k;
        D[a0 + t] = irc::ref_sqrt_abs(found ? __uint_as_float((unsigned)(k >> 32)) : IRC_SINGLE_INF_F);
        N[a0 + t] = (found ? ((lo & 0x1ffffffu) << 7 | lo >> 25) : (unsigned)(a0 + t)) + 1u;
    }
}

// jrc3_cuda_rho_drift (DELTA false): the fraction of site-matched candidates
// within dc2.  jrc3_cuda_delta_drift (DELTA): the nearest site-matched
// candidate with strictly higher rho; the reference's thread t keeps its first
// strict minimum over j = t, t + 128, ... and the lowest thread holding the
// overall minimum wins, i.e. the smallest (d2, j % 128, j); none -> the query.
//
// A candidate j matches a query when its primary site (features f1) or else
// its secondary site (f2) is the query's, a few percent of the pairs on a
// probe.  Testing a match per lane and computing the distance there walks the
// whole feature loop for one lane's sake (1.52 + 1.07 ms for 2,003 queries x
// 20,011 candidates of 18 features on 64 sites).  Here a warp looks up which
// of the CTA's 16 queries a site belongs to (a table of query masks by site;
// sites outside it are compared one by one) and queues the matching pairs;
// every 32 of them become one full-warp round of distances, a pair per lane.
// Counts and the minimum of 64-bit keys do not depend on the order.
constexpr int kDriftThreads = 512, kDriftWarps = kDriftThreads / 32;
constexpr int kSiteTable = 2048;

template <int V>
struct FVec;
template <> struct FVec<1> { using T = float; };
template <> struct FVec<2> { using T = float2; };
template <> struct FVec<4> { using T = float4; };

template <bool DELTA, int V>
__global__ void __launch_bounds__(kDriftThreads)
k_drift_window(float *__restrict__ out, unsigned *__restrict__ nneigh, const int *__restrict__ site12,
               const float *__restrict__ f1, const float *__restrict__ f2, const float *__restrict__ rho, int n1,
               int n12, int nC, float dc2)
{
    using Vec = typename FVec<V>::T;
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ int sSite[kQB], sRho[kQB], sComp[kQB];
    __shared__ float sR[kQB];
    __shared__ unsigned long long sKey[kQB];
    __shared__ unsigned qj[kDriftWarps][64];      // a warp's queued pairs: candidate | f2 << 31
    __shared__ uint8_t qq[kDriftWarps][64];       // and query
    __shared__ unsigned sMask[kSiteTable];        // queries of each site
    __shared__ int sOut;                          // some query's site is outside the table
    const int a0 = blockIdx.x * kQB;
    const int n = min(kQB, n1 - a0);
    irc::stage_queries<kQB>(f1, nC, a0, n, sA);
    if (threadIdx.x < kQB) {
        sSite[threadIdx.x] = threadIdx.x < n ? __ldg(site12 + a0 + threadIdx.x) : 0;
        sRho[threadIdx.x] = 0;
        sComp[threadIdx.x] = 0;
        sKey[threadIdx.x] = ~0ull;
        if (DELTA) sR[threadIdx.x] = __ldg(rho + a0 + min((int)threadIdx.x, n - 1));
    }
    for (int i = threadIdx.x; i < kSiteTable; i += kDriftThreads) sMask[i] = 0u;
    if (threadIdx.x == 0) sOut = 0;
    __syncthreads();
    if (threadIdx.x < n) {
        const unsigned site = (unsigned)sSite[threadIdx.x];
        if (site < kSiteTable) atomicOr(sMask + site, 1u << threadIdx.x);
        else sOut = 1;
    }
    __syncthreads();
    const bool table = !sOut;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned *wj = qj[warp];
    uint8_t *wq = qq[warp];
    // one queued pair per lane (the first `m` of the queue)
    auto round = [&](int m) {
        __syncwarp();
        if (lane < m) {
            const unsigned e = wj[lane];
            const int q = wq[lane], j = (int)(e & 0x7fffffffu);
            const Vec *src = reinterpret_cast<const Vec *>(((e >> 31) ? f2 : f1) + (size_t)j * nC);
            float acc = 0.0f;
#pragma unroll 4
            for (int c = 0; c < nC; c += V) {
                const Vec b = __ldg(src + c / V);
                const float *bv = reinterpret_cast<const float *>(&b);
#pragma unroll
                for (int u = 0; u < V; ++u) acc = irc::dterm(acc, sA[(c + u) * kQB + q], bv[u]);
            }
            if (DELTA) {
                if (acc < IRC_SINGLE_INF_F) {
                    const unsigned long long key = ((unsigned long long)__float_as_uint(acc) << 32) |
                                                   ((unsigned)(j & 127) << 25) | (unsigned)(j >> 7);
                    if (key < *(volatile unsigned long long *)(sKey + q)) atomicMin(sKey + q, key);
                }
            } else {
                atomicAdd(sComp + q, 1);
                if (acc <= dc2) atomicAdd(sRho + q, 1);
            }
        }
        __syncwarp();
    };
    int cnt = 0;                                  // queued pairs (warp-uniform)
    for (int j0 = warp * 32; j0 < n12; j0 += kDriftThreads) {
        const int j = j0 + lane;
        const bool in = j < n12;
        const int s1 = in ? __ldg(site12 + j) : 0, s2 = in ? __ldg(site12 + j + n12) : 0;
        const float rj = DELTA && in ? __ldg(rho + j) : 0.0f;
        unsigned m1 = 0, m2 = 0;                  // queries matched by the primary, else the secondary site
        if (table) {
            if (in && (unsigned)s1 < kSiteTable) m1 = sMask[s1];
            if (in && (unsigned)s2 < kSiteTable) m2 = sMask[s2] & ~m1;
        } else if (in) {
            for (int q = 0; q < n; ++q) {
                if (s1 == sSite[q]) m1 |= 1u << q;
                else if (s2 == sSite[q]) m2 |= 1u << q;
            }
        }
        unsigned m = m1 | m2;
        for (unsigned bal; (bal = __ballot_sync(0xffffffffu, m != 0u)) != 0u;) {
            const int q = m ? __ffs(m) - 1 : 0;
            bool hit = m != 0u;
            m &= m - 1u;
            if (DELTA) {
                hit = hit && !(rj <= sR[q]);
                bal = __ballot_sync(0xffffffffu, hit);
            }
            if (hit) {
                const int at = cnt + __popc(bal & ((1u << lane) - 1u));
                wj[at] = (unsigned)j | ((m1 >> q) & 1u ? 0u : 0x80000000u);
                wq[at] = (uint8_t)q;
            }
            cnt += __popc(bal);
            if (cnt >= 32) {
                round(32);
                // the rest moves to the front
                cnt -= 32;
                unsigned e = 0;
                uint8_t k = 0;
                if (lane < cnt) { e = wj[32 + lane]; k = wq[32 + lane]; }
                __syncwarp();
                if (lane < cnt) { wj[lane] = e; wq[lane] = k; }
                __syncwarp();
            }
        }
    }
    if (cnt) round(cnt);
    __syncthreads();
    if (threadIdx.x >= n) return;
    const int q = threadIdx.x;
    if (!DELTA) {
        out[a0 + q] = (float)((double)sRho[q] / (double)sComp[q]);
        return;
    }
    const unsigned long long k = sKey[q];
    const bool found = k != ~0ull;
    const float dmin = found ? __uint_as_float((unsigned)(k >> 32)) : IRC_SINGLE_INF_F;
    const unsigned lo = (unsigned)k;
    out[a0 + q] = __fsqrt_rn(__fdiv_rn(fabsf(dmin), dc2));
    nneigh[a0 + q] = (found ? ((lo & 0x1ffffffu) << 7 | lo >> 25) : (unsigned)(a0 + q)) + 1u;
}

// The widest feature loads that the rows of both matrices allow.
template <bool DELTA>
void launch_drift_window(float *out, unsigned *nneigh, const int *site12, const float *f1, const float *f2,
                         const float *rho, int n1, int n12, int nC, float dc2, cudaStream_t s)
{
    const uintptr_t al = (uintptr_t)f1 | (uintptr_t)f2 | ((uintptr_t)nC * 4);
    auto k = al % 16 == 0 ? k_drift_window<DELTA, 4> : al % 8 == 0 ? k_drift_window<DELTA, 2> : k_drift_window<DELTA, 1>;
    k<<<(n1 + kQB - 1) / kQB, kDriftThreads, 0, s>>>(out, nneigh, site12, f1, f2, rho, n1, n12, nC, dc2);
}

// jrc3_cuda_rho (irc_cuda_rho.cu): query i1 < n1 counts the candidates j < n12
// within the time window |ord[i1] - ord[j]| <= dn_max (itself included) and
// those at d2 <= dc2 (fdc = 1: d2 < dc2 * |query|^2, fused-accumulated in
// feature order, then one multiply).  Integer counts, so the result does not
// depend on the scan order; rho = count / compared, divided in double.
__global__ void __launch_bounds__(128)
k_rho_st(float *__restrict__ rho, const float *__restrict__ F, const int *__restrict__ ord, int n1, int n12,
         int nC, int dn_max, int fdc, float dc2)
{
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ int sOrd[kQB], sRho[kQB], sComp[kQB];
    __shared__ float sCut[kQB];
    const int a0 = blockIdx.x * kQB;
    const int n = min(kQB, n1 - a0);
    irc::stage_queries<kQB>(F, nC, a0, n, sA);
    if (threadIdx.x < kQB) {
        sOrd[threadIdx.x] = threadIdx.x < n ? __ldg(ord + a0 + threadIdx.x) : 0;
        sRho[threadIdx.x] = 0;
        sComp[threadIdx.x] = 0;
    }
    __syncthreads();
    if (threadIdx.x < kQB) {
        float cut = dc2;
        if (fdc == 1) {
            float v = 0.0f;
            for (int c = 0; c < nC; ++c) v = __fmaf_rn(sA[c * kQB + threadIdx.x], sA[c * kQB + threadIdx.x], v);
            cut = __fmul_rn(v, dc2);
        }
        sCut[threadIdx.x] = cut;
    }
    __syncthreads();
    int nr[kQB], nc[kQB];
#pragma unroll
    for (int q = 0; q < kQB; ++q) { nr[q] = 0; nc[q] = 0; }
    for (int j = threadIdx.x; j < n12; j += blockDim.x) {
        const int oj = __ldg(ord + j);
        const float *src = F + (size_t)j * nC;
#pragma unroll
        for (int q = 0; q < kQB; ++q) {
            if (q >= n || abs(sOrd[q] - oj) > dn_max) continue;
            float acc = 0.0f;
            for (int c = 0; c < nC; ++c) acc = irc::dterm(acc, __ldg(src + c), sA[c * kQB + q]);
            nr[q] += fdc == 0 ? (acc <= sCut[q]) : (acc < sCut[q]);
            nc[q] += 1;
        }
    }
#pragma unroll
    for (int q = 0; q < kQB; ++q) {
        int r = nr[q], c = nc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_xor_sync(0xffffffffu, r, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if ((threadIdx.x & 31) == 0 && c) { atomicAdd(&sRho[q], r); atomicAdd(&sComp[q], c); }
    }
    __syncthreads();
    if (threadIdx.x < n)
        rho[a0 + threadIdx.x] = (float)((double)sRho[threadIdx.x] / (double)sComp[threadIdx.x]);
}

// jrc3_cuda_delta (irc_cuda_delta.cu): nearest candidate within the time
// window ranked before the query in rho order (rr[j] < rr[i1]).  One thread
// per bin (blockDim = the reference's nThreads): thread t keeps its first
// strict minimum over j = t, t+nT, ...; the lowest thread holding the
// overall minimum wins; none below SINGLE_INF -> the query itself.
// delta = sqrt(d2 / dc2) (fdc = 1: / (dc2 * |query|^2)).
__global__ void __launch_bounds__(128)
k_delta_st(float *__restrict__ delta, unsigned *__restrict__ nneigh, const float *__restrict__ F,
           const int *__restrict__ ord, const int *__restrict__ rr, int n1, int n12, int nC, int dn_max, int fdc,
           float dc2)
{
    __shared__ __align__(16) float sA[IRC_NC_MAX * kQB];
    __shared__ int sOrd[kQB], sRR[kQB];
    __shared__ float sCut[kQB];
    __shared__ unsigned long long sKey[kQB][128 / 32];
    __shared__ unsigned sIdx[kQB][128 / 32];
    const int a0 = blockIdx.x * kQB;
    const int n = min(kQB, n1 - a0);
    irc::stage_queries<kQB>(F, nC, a0, n, sA);
    if (threadIdx.x < kQB) {
        sOrd[threadIdx.x] = threadIdx.x < n ? __ldg(ord + a0 + threadIdx.x) : 0;
        sRR[threadIdx.x] = threadIdx.x < n ? __ldg(rr + a0 + threadIdx.x) : INT_MIN;
    }
    __syncthreads();
    if (threadIdx.x < kQB) {
        float cut = dc2;
        if (fdc == 1) {
            float v = 0.0f;
            for (int c = 0; c < nC; ++c) v = __fmaf_rn(sA[c * kQB + threadIdx.x], sA[c * kQB + threadIdx.x], v);
            cut = __fmul_rn(v, dc2);
        }
        sCut[threadIdx.x] = cut;
    }
    __syncthreads();
    float mn[kQB];
    unsigned mi[kQB];
#pragma unroll
    for (int q = 0; q < kQB; ++q) { mn[q] = IRC_SINGLE_INF_F; mi[q] = 0u; }
    for (int j = threadIdx.x; j < n12; j += blockDim.x) {
        const int oj = __ldg(ord + j), rj = __ldg(rr + j);
        const float *src = F + (size_t)j * nC;
#pragma unroll
        for (int q = 0; q < kQB; ++q) {
            if (!(rj < sRR[q]) || abs(sOrd[q] - oj) > dn_max) continue;
            float acc = 0.0f;
            for (int c = 0; c < nC; ++c) acc = irc::dterm(acc, __ldg(src + c), sA[c * kQB + q]);
            if (acc < mn[q]) { mn[q] = acc; mi[q] = (unsigned)j; }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < kQB; ++q) {
        unsigned long long k = irc::sort_key(mn[q], threadIdx.x);
        unsigned idx = mi[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(0xffffffffu, k, o);
            const unsigned oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ok < k) { k = ok; idx = oi; }
        }
        if (lane == 0) { sKey[q][warp] = k; sIdx[q][warp] = idx; }
    }
    __syncthreads();
    if (threadIdx.x < n) {
        const int q = threadIdx.x;
        unsigned long long k = sKey[q][0];
        unsigned idx = sIdx[q][0];
        for (int w = 1; w < nw; ++w)
            if (sKey[q][w] < k) { k = sKey[q][w]; idx = sIdx[q][w]; }
        const float v = __uint_as_float((unsigned)(k >> 32));
        const bool found = v < IRC_SINGLE_INF_F;
        const float dmin = found ? v : IRC_SINGLE_INF_F;
        delta[a0 + q] = __fsqrt_rn(__fdiv_rn(dmin, sCut[q]));
        nneigh[a0 + q] = (found ? idx : (unsigned)(a0 + q)) + 1u;
    }
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

// Launch with the CTAs of a column (grid.y = cluster) as one cluster.
template <class... P, class... Q>
cudaError_t launch_cluster(void (*kern)(P...), dim3 grid, int cluster, int threads, size_t smem, cudaStream_t s, Q... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1;
    attr.val.clusterDim.y = cluster;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace

// Exact top-k fill of the search_min_drift output (IRC_MODE_EXACT), in irc_site.cu.
int irc_exact_chunk_fill(float *D, int32_t *I, const float *F, const int32_t *IBB,
                         const int32_t *NBB, int nC, int nBB, int iA0, int nA, int nT, int knn,
                         int nF, cudaStream_t s);

extern "C" {

int irc_search_min_drift(float *D, int32_t *I, const float *F, const int32_t *IBB,
                         const int32_t *NBB, const int32_t *vnConst, int nThreads, int mode,
                         int knn, void *stream)
{
    if (!D || !I || !F || !IBB || !NBB || !vnConst) {
        irc_host::set_error("irc_search_min_drift: null pointer");
        return IRC_E_INVAL;
    }
    const int nC = vnConst[0], nBB = vnConst[2], iA0 = vnConst[3], nA = vnConst[4];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_search_min_drift: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || nA <= 0 || iA0 < 0 || nBB <= 0 || nThreads <= 0 || nThreads > 1024 || nBB > nThreads) {
        irc_host::set_error("irc_search_min_drift: bad sizes nC=%d nBB=%d iA0=%d nA=%d nThreads=%d",
                            nC, nBB, iA0, nA, nThreads);
        return IRC_E_INVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (mode == IRC_MODE_EXACT) {
        if (knn <= 0 || knn > nThreads) { irc_host::set_error("irc_search_min_drift: bad knn %d", knn); return IRC_E_INVAL; }
        return irc_exact_chunk_fill(D, I, F, IBB, NBB, nC, nBB, iA0, nA, nThreads, knn, vnConst[1], s);
    }
    if (mode != IRC_MODE_REF) { irc_host::set_error("irc_search_min_drift: unsupported mode %d", mode); return IRC_E_UNSUPPORTED; }
    return launch_search<false>(D, I, F, nullptr, IBB, NBB, vnConst[1], nC, nBB, iA0, nA, nThreads, s, "irc_search_min_drift");
}

int irc_search_delta_drift(float *D, int32_t *I, const float *F, const float *R,
                           const int32_t *IBB, const int32_t *NBB, const int32_t *vnConst,
                           int nThreads, void *stream)
{
    if (!D || !I || !F || !R || !IBB || !NBB || !vnConst) {
        irc_host::set_error("irc_search_delta_drift: null pointer");
        return IRC_E_INVAL;
    }
    const int nC = vnConst[0], nBB = vnConst[2], iA0 = vnConst[3], nA = vnConst[4];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_search_delta_drift: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || nA <= 0 || iA0 < 0 || nBB <= 0 || nThreads <= 0 || nThreads > 1024 || nBB > nThreads) {
        irc_host::set_error("irc_search_delta_drift: bad sizes");
        return IRC_E_INVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    return launch_search<true>(D, I, F, R, IBB, NBB, vnConst[1], nC, nBB, iA0, nA, nThreads, s, "irc_search_delta_drift");
}

}  // extern "C"

namespace {

// Shared host side of the four binned-kNN drop-ins.  IB entries outside
// 1..nF are counted on the device and reported after a stream sync.
template <bool IND, bool KALL>
int launch_knn_bins(const char *name, float *K, int32_t *I, const float *B, const float *A, const int32_t *IB,
                    int nF, const int32_t *vnConst, int nThreads, void *stream)
{
    if (!K || !B || !A || !vnConst || (IND && !IB)) { irc_host::set_error("%s: null pointer", name); return IRC_E_INVAL; }
    const int nB = vnConst[0], nA = vnConst[1], nC = vnConst[2], knn = vnConst[3];
    if (nC > IRC_NC_MAX) { irc_host::set_error("%s: nC=%d > %d", name, nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || nA <= 0 || nB <= 0 || knn <= 0 || nThreads <= 0 || nThreads > 1024 || knn > nThreads ||
        (IND && nF <= 0)) {
        irc_host::set_error("%s: bad sizes nB=%d nA=%d nC=%d knn=%d nThreads=%d", name, nB, nA, nC, knn, nThreads);
        return IRC_E_INVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    // CTAs per cluster: a turn each where 8 suffice (512 bins)
    int nr = 1;
    while (nr < 8 && nr * kBinTurn < nThreads) nr *= 2;
    const int turns = cdiv(nThreads, nr * kBinTurn);
    const size_t smem = bins_smem(nC, nThreads, turns);
    auto kern = k_knn_bins<IND, KALL>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, name);
    int *bad = nullptr;
    if (IND) {
        e = irc_scratch_alloc((void **)&bad, sizeof(int), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(int), s);
        if (e != cudaSuccess) return irc_host::cuda_status(e, name);
    }
    e = launch_cluster(kern, dim3(cdiv(nA, kBinQ), nr), nr, 32 * kBinWarps, smem, s, K, I, B, A, IB, nF, bad, nB, nA, nC, knn, nThreads, turns);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        if (bad) cudaFreeAsync(bad, s);
        return irc_host::cuda_status(e, name);
    }
    if (IND) {
        int hbad = 0;
        e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaFreeAsync(bad, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return irc_host::cuda_status(e, name);
        if (hbad) {
            irc_host::set_error("%s: %d IB entries outside 1..%d (skipped)", name, hbad, nF);
            return IRC_E_INVAL;
        }
    }
    return IRC_OK;
}

}  // namespace

extern "C" {

int irc_cuda_knn_index(float *K, int32_t *I, const float *B, const float *A,
                       const int32_t *vnConst, int nThreads, void *stream)
{
    if (!I) { irc_host::set_error("irc_cuda_knn_index: null pointer"); return IRC_E_INVAL; }
    return launch_knn_bins<false, false>("irc_cuda_knn_index", K, I, B, A, nullptr, 0, vnConst, nThreads, stream);
}

int irc_cuda_knn(float *K, const float *B, const float *A, const int32_t *vnConst, int nThreads, void *stream)
{
    return launch_knn_bins<false, false>("irc_cuda_knn", K, nullptr, B, A, nullptr, 0, vnConst, nThreads, stream);
}

int irc_cuda_knn_full(float *K, int32_t *I, const float *B, const float *A, const int32_t *vnConst, int nThreads,
                      void *stream)
{
    if (!I) { irc_host::set_error("irc_cuda_knn_full: null pointer"); return IRC_E_INVAL; }
    return launch_knn_bins<false, true>("irc_cuda_knn_full", K, I, B, A, nullptr, 0, vnConst, nThreads, stream);
}

int irc_cuda_knn_ib(float *K, int32_t *I, const float *B, const float *A, const int32_t *IB, int nF,
                    const int32_t *vnConst, int nThreads, void *stream)
{
    if (!I) { irc_host::set_error("irc_cuda_knn_ib: null pointer"); return IRC_E_INVAL; }
    return launch_knn_bins<true, false>("irc_cuda_knn_ib", K, I, B, A, IB, nF, vnConst, nThreads, stream);
}

int irc_cuda_rho(float *vrRho1, const float *mrFet12, const int32_t *viiSpk12_ord, const int32_t *vnConst,
                 float dc2, void *stream)
{
    if (!vrRho1 || !mrFet12 || !viiSpk12_ord || !vnConst) { irc_host::set_error("irc_cuda_rho: null pointer"); return IRC_E_INVAL; }
    const int n1 = vnConst[0], n12 = vnConst[1], nC = vnConst[2], dn_max = vnConst[3], fdc = vnConst[4];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_cuda_rho: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || n1 <= 0 || n12 < n1 || dn_max < 0 || (fdc != 0 && fdc != 1)) {
        irc_host::set_error("irc_cuda_rho: bad sizes n1=%d n12=%d nC=%d dn_max=%d fDc_spk=%d", n1, n12, nC, dn_max, fdc);
        return IRC_E_INVAL;
    }
    k_rho_st<<<cdiv(n1, kQB), 128, 0, (cudaStream_t)stream>>>(vrRho1, mrFet12, viiSpk12_ord, n1, n12, nC, dn_max,
                                                              fdc, dc2);
    IRC_CHECK_LAUNCH("irc_cuda_rho");
    return IRC_OK;
}

int irc_cuda_delta(float *vrDelta1, uint32_t *viNneigh1, const float *mrFet12, const int32_t *viiSpk12_ord,
                   const int32_t *viiRho12_ord, const int32_t *vnConst, float dc2, int nThreads, void *stream)
{
    if (!vrDelta1 || !viNneigh1 || !mrFet12 || !viiSpk12_ord || !viiRho12_ord || !vnConst) {
        irc_host::set_error("irc_cuda_delta: null pointer");
        return IRC_E_INVAL;
    }
    const int n1 = vnConst[0], n12 = vnConst[1], nC = vnConst[2], dn_max = vnConst[3], fdc = vnConst[4];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_cuda_delta: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || n1 <= 0 || n12 < n1 || dn_max < 0 || (fdc != 0 && fdc != 1) || nThreads < 32 ||
        nThreads > 128 || nThreads % 32) {
        irc_host::set_error("irc_cuda_delta: bad sizes n1=%d n12=%d nC=%d dn_max=%d fDc_spk=%d nThreads=%d "
                            "(nThreads: a multiple of 32 up to 128, the reference's NTHREADS)",
                            n1, n12, nC, dn_max, fdc, nThreads);
        return IRC_E_INVAL;
    }
    k_delta_st<<<cdiv(n1, kQB), nThreads, 0, (cudaStream_t)stream>>>(vrDelta1, viNneigh1, mrFet12, viiSpk12_ord,
                                                                     viiRho12_ord, n1, n12, nC, dn_max, fdc, dc2);
    IRC_CHECK_LAUNCH("irc_cuda_delta");
    return IRC_OK;
}

int irc_cuda_delta_knn(float *D, uint32_t *N, const float *B, const float *A, const float *R_B,
                       const float *R_A, const int32_t *vnConst, int nThreads, void *stream)
{
    if (!D || !N || !B || !A || !R_B || !R_A || !vnConst) { irc_host::set_error("irc_cuda_delta_knn: null pointer"); return IRC_E_INVAL; }
    const int nB = vnConst[0], nA = vnConst[1], nC = vnConst[2];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_cuda_delta_knn: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || nA <= 0 || nB < 0 || nThreads != 128) {
        irc_host::set_error("irc_cuda_delta_knn: bad sizes (nThreads must be 128, the reference block size)");
        return IRC_E_INVAL;
    }
    // short scans are over before the kernel below has staged them; with few features and queries for
    // two turns of the chip its minima cost more than the distances (us, direct | staged: 300 x 300 of
    // 24 features 8.8 | 15.9, 1,000 x 1,000 17.2 | 20.6, 300 x 2,000 of 9 19 | 15; 5,000 x 5,000 of 6 41 | 52)
    if (nB <= 1024 || (nC <= 9 && nA >= 2 * 152 * kQB)) {
        k_delta_direct<<<cdiv(nA, kQB), 128, 0, (cudaStream_t)stream>>>(D, N, B, A, R_B, R_A, nB, nA, nC);
        IRC_CHECK_LAUNCH("irc_cuda_delta_knn");
        return IRC_OK;
    }
    const int ng = nA > 32 ? 4 : nA > 16 ? 2 : 1;
    auto bytes = [&](int nw) { return scan_smem(nC, ng, nw) + (size_t)kQB * 64 * nw * sizeof(int); };
    const int nw = bytes(8) <= 232448 - 1024 ? 8 : 4, block = 64 * nw / ng;
    const size_t smem = bytes(nw);
    auto kern = nw == 8 ? (ng == 4 ? k_delta_knn<4, 8> : ng == 2 ? k_delta_knn<2, 8> : k_delta_knn<1, 8>)
                        : (ng == 4 ? k_delta_knn<4, 4> : ng == 2 ? k_delta_knn<2, 4> : k_delta_knn<1, 4>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_cuda_delta_knn");
    // up to 8 CTAs share a query tile's candidates, as many as keep the fullest SM busy for the shortest
    // time: two CTAs run together, one alone takes two thirds of their time, each costs some two steps
    // besides its own.  154 tiles put two whole tiles on some SMs, or nine eighths (9,800 queries of
    // 20,000 candidates: 1,006 us whole, 597 so; 1,507 of 15,000, 24 tiles: 8 CTAs 10 us faster than 4)
    const int tiles = cdiv(nA, kQB * ng);
    int split = 1;
    long long best = LLONG_MAX;
    for (int k = 1; k <= 8 && (k == 1 || nB >= k * 2 * block); k *= 2) {
        const long long c = cdiv((long long)tiles * k, 152), t = (c / 2 * 3 + c % 2 * 2) * (cdiv(nB, (long long)k * block) + 2);
        if (t < best) { best = t; split = k; }
    }
    e = launch_cluster(kern, dim3(tiles, split), split, 32 * nw, smem, (cudaStream_t)stream, D, N, B, A, R_B, R_A, nB, nA, nC);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_cuda_delta_knn");
    IRC_CHECK_LAUNCH("irc_cuda_delta_knn");
    return IRC_OK;
}

int irc_rho_drift(float *vrRho1, const int32_t *miSite12, const float *mrFet1, const float *mrFet2,
                  const int32_t *vnConst, float dc2, void *stream)
{
    if (!vrRho1 || !miSite12 || !mrFet1 || !mrFet2 || !vnConst) { irc_host::set_error("irc_rho_drift: null pointer"); return IRC_E_INVAL; }
    const int n1 = vnConst[0], n12 = vnConst[1], nC = vnConst[2];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_rho_drift: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || n1 <= 0 || n12 < n1) { irc_host::set_error("irc_rho_drift: bad sizes n1=%d n12=%d nC=%d", n1, n12, nC); return IRC_E_INVAL; }
    launch_drift_window<false>(vrRho1, nullptr, miSite12, mrFet1, mrFet2, nullptr, n1, n12, nC, dc2, (cudaStream_t)stream);
    IRC_CHECK_LAUNCH("irc_rho_drift");
    return IRC_OK;
}

int irc_delta_drift(float *vrDelta1, uint32_t *viNneigh1, const int32_t *miSite12, const float *mrFet1,
                    const float *mrFet2, const float *vrRho1, const int32_t *vnConst, float dc2, void *stream)
{
    if (!vrDelta1 || !viNneigh1 || !miSite12 || !mrFet1 || !mrFet2 || !vrRho1 || !vnConst) {
        irc_host::set_error("irc_delta_drift: null pointer");
        return IRC_E_INVAL;
    }
    const int n1 = vnConst[0], n12 = vnConst[1], nC = vnConst[2];
    if (nC > IRC_NC_MAX) { irc_host::set_error("irc_delta_drift: nC=%d > %d", nC, IRC_NC_MAX); return IRC_E_NC; }
    if (nC <= 0 || n1 <= 0 || n12 < n1) { irc_host::set_error("irc_delta_drift: bad sizes n1=%d n12=%d nC=%d", n1, n12, nC); return IRC_E_INVAL; }
    launch_drift_window<true>(vrDelta1, viNneigh1, miSite12, mrFet1, mrFet2, vrRho1, n1, n12, nC, dc2, (cudaStream_t)stream);
    IRC_CHECK_LAUNCH("irc_delta_drift");
    return IRC_OK;
}

}  // extern "C"
