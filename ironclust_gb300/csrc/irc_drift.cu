// irc_drift.cu -- the drift linkage of calc_drift_ (matlab/irc2.m:6373-6465)
// on the device: which drift chunks a chunk's spikes are compared with.
//
//   limits     viLim = [0, ceil((1:n)/n * nSpk)] (equal spike counts)
//   edges      quantile_vr_ (matlab/irc2.m:6481-6490) of the amplitudes
//              (nQuantile + 1 edges) and of the positions (nSites + 1 edges):
//              the values of a fixed subsample (subsample_vr_, a function of
//              the spike count alone) at the ranks round(m * q) of MATLAB's
//              ascending sort, selected by four histogram levels of an
//              order-preserving 32-bit key
//   counts     histcounts2 of (amplitude, position) per chunk into
//              [nQuantile x nSites] bins (bins [e_k, e_k+1), the last closed;
//              values outside the edges dropped), a chunk per block
//   linkage    per chunk j, the nTime_batch nearest chunks by the Euclidean
//              distance between count columns, ties by chunk index (MATLAB's
//              stable sort), over all chunks when n <= nTime_max_drift, else
//              over the band calc_drift_ masks (|i - j| <= nTime_max_drift/4
//              widened at both ends) -- for every column that mask is one
//              contiguous interval of rows.  Counts are integers, so the
//              squared distances are exact int64 and the order is the order
//              of the true distances.
//
// Six launches and nothing read from host memory.  A call on 1,000,000 spikes
// (64 sites, 400 chunks) took 900 us when the subsample's positions were made
// on the host and copied, two radix sorts of 100,000 keys found the edges and a
// thread read a chunk's counts column by column in the linkage (142 us).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "ircgb300.h"
#include "irc_common.cuh"

namespace {

constexpr int TPB = 256;
constexpr int kMaxEdges = 1025;

__device__ __forceinline__ uint32_t asc_key(float f)
{
    if (isnan(f)) return 0xffffffffu;                 // NaN last
    uint32_t u = __float_as_uint(f);
    if (f == 0.0f) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float asc_float(uint32_t o)
{
    if (o == 0xffffffffu) return __uint_as_float(0x7fc00000u);
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// subsample_vr_ (matlab/irc2.m:1557-1573) of the positions 0 .. N-1: every
// skip-th one, m0 of them, less the nRemove at round(linspace(1, m0, nRemove)).
struct Subsample {
    int64_t skip;
    int m0, nRemove, m;
    double step;                                      // linspace's
};

Subsample subsample(int64_t N, int64_t nMax)
{
    Subsample u{1, 0, 0, 0, 0.0};
    if (N > nMax) u.skip = std::max<int64_t>(1, N / nMax);
    u.m0 = (int)((N + u.skip - 1) / u.skip);
    u.nRemove = N > nMax && u.m0 > nMax ? u.m0 - (int)nMax : 0;
    u.m = u.m0 - u.nRemove;                           // (step >= 1: the removed ones are all different)
    if (u.nRemove > 1) u.step = ((double)u.m0 - 1.0) / (double)(u.nRemove - 1);
    return u;
}

// 0-based place of the k-th removed position; without contraction, as MATLAB.
__device__ __forceinline__ int removed(const Subsample &u, int k)
{
    const double x = k == u.nRemove - 1 ? (double)u.m0 : __dadd_rn(__dmul_rn((double)k, u.step), 1.0);
    const double r = floor(__dadd_rn(x, 0.5));
    return (int)fmin(fmax(r, 1.0), (double)u.m0) - 1;
}

__device__ __forceinline__ int64_t sample_position(const Subsample &u, int i)
{
    int lo = 0, hi = u.nRemove;                       // removed places up to the i-th that stays
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (removed(u, mid) - mid <= i) lo = mid + 1; else hi = mid;
    }
    return (int64_t)(i + lo) * u.skip;
}

// The edges of one value: quantile_vr_ for the fractions (0:nq)/nq.  A rank
// has a slot, the keys that share its digits so far (ranks with the same ones
// share it), and its rank among them.
struct Select {
    const float *v;
    uint32_t *keys;                                   // [m]
    uint16_t *slot;                                   // [m] a key's slot (kNone: none)
    int *hist;                                        // [nq+1][256], zero between levels
    uint16_t *next;                                   // [nq+1][256] slot of the next level
    uint32_t *prefix;                                 // [nq+1] digits so far
    int *rank, *rslot;                                // [nq+1]
    int *words;                                       // [0] slots, [1] ticket; zero at the start
    float *edges;                                     // [nq+1]
    int nq;
};
constexpr uint16_t kNone = 0xffff;
constexpr int kSharedSlots = 40, kSelectBlocks = 48, kSelectThreads = 512;

// One level (8 bits) of both selections (blockIdx.y).  Latency-bound: the
// blocks share the keys, the one that ends last ranks.  Blocks count in shared
// memory while the slots fit; more slots than that have little contention.
template <int LEVEL>
__global__ void __launch_bounds__(kSelectThreads) k_select(Select s0, Select s1, Subsample u)
{
    __shared__ int sh[kSharedSlots * 256];
    __shared__ int chosen[kMaxEdges];                 // slot * 256 + digit of every rank
    __shared__ bool last;
    const Select &s = blockIdx.y ? s1 : s0;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, ns = LEVEL == 0 ? 1 : __ldcg(s.words);
    const bool shared = ns <= kSharedSlots;
    if (shared)
        for (int k = t; k < ns * 256; k += kSelectThreads) sh[k] = 0;
    __syncthreads();
    for (int i = blockIdx.x * kSelectThreads + t; i < u.m; i += gridDim.x * kSelectThreads) {
        uint32_t key;
        int sl = 0;
        if constexpr (LEVEL == 0) {
            key = asc_key(__ldg(s.v + sample_position(u, i)));
            s.keys[i] = key;
        } else {
            key = s.keys[i];
            if (LEVEL > 1) sl = s.slot[i];
            if (sl == kNone) continue;
            sl = s.next[sl * 256 + ((key >> (32 - 8 * LEVEL)) & 255u)];
            s.slot[i] = (uint16_t)sl;
            if (sl == kNone) continue;
        }
        atomicAdd((shared ? sh : s.hist) + sl * 256 + ((key >> (24 - 8 * LEVEL)) & 255u), 1);
    }
    __syncthreads();
    if (shared)
        for (int k = t; k < ns * 256; k += kSelectThreads)
            if (sh[k]) atomicAdd(s.hist + k, sh[k]);
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicInc(reinterpret_cast<unsigned *>(s.words + 1), gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = warp; k <= s.nq; k += kSelectThreads / 32) {
        int r, sl = 0;
        uint32_t pre = 0;
        if constexpr (LEVEL == 0) {                   // round(m * q), clamped to 1 .. m
            const double q = (double)k / (double)s.nq;
            const double x = floor(__dadd_rn(__dmul_rn((double)u.m, q), 0.5));
            r = (int)fmax(fmin(x, (double)u.m), 1.0) - 1;
        } else {
            r = __ldcg(s.rank + k);
            sl = __ldcg(s.rslot + k);
            pre = __ldcg(s.prefix + k);
        }
        const int4 *h = reinterpret_cast<const int4 *>(s.hist + sl * 256) + 2 * lane;
        const int4 a = __ldcg(h), b = __ldcg(h + 1);
        const int c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        int sum = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) sum += c[e];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += w;
        }
        int at = incl - sum, digit = -1;
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (digit < 0) {
                if (r < at + c[e]) digit = 8 * lane + e;
                else at += c[e];
            }
        // (the first lane whose keys reach past rank r)
        const int who = __ffs(__ballot_sync(0xffffffffu, r < incl)) - 1;
        digit = __shfl_sync(0xffffffffu, digit, who);
        at = __shfl_sync(0xffffffffu, at, who);
        if (lane == 0) {
            chosen[k] = sl * 256 + digit;
            pre = pre << 8 | (uint32_t)digit;
            if (LEVEL == 3) s.edges[k] = asc_float(pre);
            s.prefix[k] = pre;
            s.rank[k] = r - at;
        }
    }
    __syncthreads();
    if constexpr (LEVEL < 3) {
        for (int k = t; k < ns * 256; k += kSelectThreads) {
            s.hist[k] = 0;
            s.next[k] = kNone;
        }
        __syncthreads();
        if (warp == 0) {                                  // ranks ascend: the ones that share a slot are neighbours
            int n = 0;
            for (int k0 = 0; k0 <= s.nq; k0 += 32) {
                const int k = k0 + lane;
                const bool in = k <= s.nq, first = in && (k == 0 || chosen[k] != chosen[k - 1]);
                const unsigned bal = __ballot_sync(0xffffffffu, first);
                const int id = n + __popc(bal & (0xffffffffu >> (31 - lane))) - 1;
                if (in) s.rslot[k] = id;
                if (first) s.next[chosen[k]] = (uint16_t)id;
                n += __popc(bal);
            }
            if (lane == 0) s.words[0] = n;
        }
    }
}

// histcounts2 bin of x for edges e[0..nb]: -1 when outside
__device__ __forceinline__ int hbin(float x, const float *e, int nb)
{
    if (!(x >= e[0]) || !(x <= e[nb])) return -1;
    if (x == e[nb]) return nb - 1;
    int lo = 0, hi = nb;                              // largest k with e[k] <= x
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (e[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// viLim: the chunk limits [0, ceil((1:n)/n * nSpk)]
__device__ __forceinline__ int64_t chunk_limit(int k, int n, int64_t nSpk)
{
    return k == 0 ? 0 : (int64_t)ceil(__dmul_rn((double)k / (double)n, (double)nSpk));
}

constexpr int kSharedBins = 8192, kPartRows = 8192;

// counts of chunk blockIdx.x (part blockIdx.y of its spikes): in shared memory
// and stored once (added, where a chunk has several parts), or -- more bins than
// fit -- added one by one to counts that are zero.
__global__ void __launch_bounds__(TPB) k_hist2(const float *__restrict__ amp, const float *__restrict__ pos, int64_t nSpk,
                                               int64_t *__restrict__ lim, int n, const float *__restrict__ ampE, int nA,
                                               const float *__restrict__ posE, int nP, int *__restrict__ counts)
{
    __shared__ float sA[kMaxEdges], sP[kMaxEdges];
    extern __shared__ int sc[];
    const int c = blockIdx.x, nBins = nA * nP;
    const bool shared = nBins <= kSharedBins;
    const int64_t l0 = chunk_limit(c, n, nSpk), l1 = chunk_limit(c + 1, n, nSpk);
    if (threadIdx.x == 0 && blockIdx.y == 0) {
        lim[c] = l0;
        if (c == n - 1) lim[n] = l1;
    }
    for (int k = threadIdx.x; k <= nA; k += TPB) sA[k] = ampE[k];
    for (int k = threadIdx.x; k <= nP; k += TPB) sP[k] = posE[k];
    if (shared)
        for (int k = threadIdx.x; k < nBins; k += TPB) sc[k] = 0;
    __syncthreads();
    int *out = counts + (size_t)c * nBins;
    int *h = shared ? sc : out;
#pragma unroll 4
    for (int64_t s = l0 + blockIdx.y * (int64_t)TPB + threadIdx.x; s < l1; s += (int64_t)gridDim.y * TPB) {
        const int ia = hbin(__ldg(amp + s), sA, nA), ip = hbin(__ldg(pos + s), sP, nP);
        if (ia >= 0 && ip >= 0) atomicAdd(h + ia + nA * ip, 1);
    }
    if (!shared) return;
    __syncthreads();
    for (int k = threadIdx.x; k < nBins; k += TPB) {
        if (gridDim.y == 1) out[k] = sc[k];
        else if (sc[k]) atomicAdd(out + k, sc[k]);
    }
}

// One CTA per chunk j: the nb nearest rows of [lo, hi] by (squared distance,
// row).  A warp per candidate row reads its counts in order, V at a time; a
// row's place is the number of rows before it.
constexpr int LINK_TPB = 512;

template <int V>
__global__ void __launch_bounds__(LINK_TPB) k_link(const int *__restrict__ counts, int nBins, int n, int nb, int quarter,
                                                   int masked, int32_t *__restrict__ members)
{
    constexpr int MAXC = 1024;
    __shared__ long long sD[MAXC];
    const int j = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int lo = 0, hi = n - 1;
    if (masked) {
        if (j < quarter) { lo = 0; hi = min(n - 1, 2 * quarter); }
        else if (j >= n - quarter) { lo = max(0, n - 2 * quarter - 1); hi = n - 1; }
        else { lo = j - quarter; hi = j + quarter; }
    }
    const int m = hi - lo + 1;                        // <= MAXC (checked on the host)
    const int *cj = counts + (size_t)j * nBins;
    for (int t = warp; t < m; t += LINK_TPB / 32) {
        const int *ci = counts + (size_t)(lo + t) * nBins;
        long long d = 0;
#pragma unroll 5
        for (int b = lane * V; b < nBins; b += 32 * V) {
            int x[V];
            if constexpr (V == 4) {
                const int4 p = __ldg(reinterpret_cast<const int4 *>(ci + b)), q = __ldg(reinterpret_cast<const int4 *>(cj + b));
                x[0] = p.x - q.x; x[1] = p.y - q.y; x[2] = p.z - q.z; x[3] = p.w - q.w;
            } else {
                x[0] = __ldg(ci + b) - __ldg(cj + b);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) d += (long long)x[v] * x[v];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0) sD[t] = d;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < m; t += LINK_TPB) {
        const long long d = sD[t];
        int place = 0;
#pragma unroll 8
        for (int k = 0; k < m; ++k) place += sD[k] < d || (sD[k] == d && k < t);
        if (place < nb) members[place + (size_t)nb * j] = lo + t;
    }
}

struct Scratch {
    cudaStream_t s;
    void *base = nullptr;
    ~Scratch()
    {
        if (base) cudaFreeAsync(base, s);
    }
};

size_t up(size_t n) { return (n + 255) & ~(size_t)255; }

}  // namespace

extern "C" int irc_calc_drift(int32_t *miDrift, int64_t *viLim, int *nDrift_out, const float *vrAmp,
                              const float *vrPos, int64_t nSpk, int nSites, int nTime_drift, int nTime_batch,
                              int nTime_max_drift, int nQuantile, void *stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!miDrift || !viLim || !nDrift_out || !vrAmp || !vrPos || nSpk < 1 || nSites < 1 || nQuantile < 1 ||
        nSites > 1024 || nQuantile > 1024 || nTime_max_drift < 4 || nTime_max_drift % 4) {
        irc_host::set_error("irc_calc_drift: need non-null arrays, nSpk >= 1, 1 <= nSites, nQuantile <= 1024, "
                            "nTime_max_drift a positive multiple of 4");
        return IRC_E_INVAL;
    }
    // the single-chunk branch (matlab/irc2.m:6386-6389)
    if (nTime_batch <= 0 || nTime_drift <= 0 || nTime_batch >= nTime_drift) {
        const int64_t lim[2] = {0, nSpk};
        std::vector<int32_t> mem((size_t)(nTime_batch > 0 ? nTime_batch : 1), 0);
        cudaError_t e = cudaMemcpyAsync(viLim, lim, sizeof(lim), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(miDrift, mem.data(), sizeof(int32_t) * mem.size(), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_calc_drift");
        *nDrift_out = 1;
        return IRC_OK;
    }
    const int n = nTime_drift;
    const bool masked = n > nTime_max_drift;
    const int quarter = nTime_max_drift / 4;
    const int span = masked ? 2 * quarter + 1 : n;
    if (span > 1024 || nTime_batch > span) {
        irc_host::set_error("irc_calc_drift: %d candidate chunks per chunk (limit 1024, and >= nTime_batch = %d)",
                            span, nTime_batch);
        return IRC_E_INVAL;
    }
    const Subsample u = subsample(nSpk, 100000);
    const int nBins = nQuantile * nSites, nq[2] = {nQuantile, nSites};
    const int64_t chunk_max = nSpk / n + 2;
    const int parts = (int)std::min<int64_t>(64, (chunk_max + kPartRows - 1) / kPartRows);

    // scratch, one allocation: words and histograms (zeroed) | counts | the rest
    Select sel[2];
    float *edges[2];
    int *counts = nullptr;
    size_t zero = 0;
    auto carve = [&](char *b) {
        size_t at = 0;
        auto take = [&](size_t bytes) { char *q = b + at; at += up(bytes); return q; };
        for (int k = 0; k < 2; ++k) {
            sel[k].nq = nq[k];
            sel[k].words = (int *)take(8);
            sel[k].hist = (int *)take(1024 * ((size_t)nq[k] + 1));
        }
        if (parts > 1 || nBins > kSharedBins) { counts = (int *)take(sizeof(int) * (size_t)nBins * n); zero = at; }
        else { zero = at; counts = (int *)take(sizeof(int) * (size_t)nBins * n); }
        for (int k = 0; k < 2; ++k) {
            const size_t ne = (size_t)nq[k] + 1;
            sel[k].keys = (uint32_t *)take(4 * (size_t)u.m);
            sel[k].slot = (uint16_t *)take(2 * (size_t)u.m);
            sel[k].next = (uint16_t *)take(512 * ne);
            sel[k].prefix = (uint32_t *)take(4 * ne);
            sel[k].rank = (int *)take(4 * ne);
            sel[k].rslot = (int *)take(4 * ne);
            sel[k].edges = edges[k] = (float *)take(4 * ne);
        }
        return at;
    };
    Scratch sc{s};
    cudaError_t e = irc_scratch_alloc(&sc.base, carve(nullptr), s);
    if (e != cudaSuccess) { sc.base = nullptr; return irc_host::cuda_status(e, "irc_calc_drift: scratch"); }
    carve((char *)sc.base);
    sel[0].v = vrAmp;
    sel[1].v = vrPos;
    e = cudaMemsetAsync(sc.base, 0, zero, s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_calc_drift: scratch");
    const dim3 grid((unsigned)std::min(kSelectBlocks, (u.m + kSelectThreads - 1) / kSelectThreads), 2);
    k_select<0><<<grid, kSelectThreads, 0, s>>>(sel[0], sel[1], u);
    k_select<1><<<grid, kSelectThreads, 0, s>>>(sel[0], sel[1], u);
    k_select<2><<<grid, kSelectThreads, 0, s>>>(sel[0], sel[1], u);
    k_select<3><<<grid, kSelectThreads, 0, s>>>(sel[0], sel[1], u);
    k_hist2<<<dim3((unsigned)n, (unsigned)parts), TPB, nBins <= kSharedBins ? sizeof(int) * nBins : 0, s>>>(
        vrAmp, vrPos, nSpk, viLim, n, edges[0], nQuantile, edges[1], nSites, counts);
    (nBins % 4 ? k_link<1> : k_link<4>)<<<n, LINK_TPB, 0, s>>>(counts, nBins, n, nTime_batch, quarter, masked ? 1 : 0, miDrift);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_calc_drift");
    *nDrift_out = n;
    return IRC_OK;
}
