// irc_rerank.cuh -- the exact FP32 re-rank of a query's candidate list, one warp
// per query: distances of the listed candidates, selection of the smallest,
// their sort.  Used by the tensor-core forms (irc_tc.cu) and by the proven
// lists of the plain forms (irc_cert.cu).
#pragma once
#include "irc_common.cuh"
#include "irc_tc.cuh"

namespace irc_rr {

constexpr int WARP_KEYS = 64;                     // sorted re-rank keys kept per warp
constexpr int QROW4 = 16;                         // float4 of a staged query row (nC <= 64)
constexpr int TAU_LOW_BIT = 12;                   // threshold searches stop at this bit (2^-11 relative)

// Ascending bitonic sort of 32*PER keys held PER per lane (element e = lane*PER + i).
template <class T, int PER>
__device__ __forceinline__ void warp_bitonic(T (&v)[PER], int lane)
{
    constexpr int N = 32 * PER;
#pragma unroll
    for (int size = 2; size <= N; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= PER) {
                const int ls = stride / PER;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = lane * PER + i;
                    const T o = __shfl_xor_sync(0xffffffffu, v[i], ls);
                    const bool up = (e & size) == 0, lower = (e & stride) == 0;
                    v[i] = (lower == up) ? (o < v[i] ? o : v[i]) : (o > v[i] ? o : v[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const int e = lane * PER + i;
                        const bool up = (e & size) == 0;
                        const T a = v[i], b = v[j];
                        const bool sw = up ? (a > b) : (a < b);
                        v[i] = sw ? b : a;
                        v[j] = sw ? a : b;
                    }
                }
            }
        }
    }
}

// 256-bit read-only load of 8 floats (32-byte aligned).
__device__ __forceinline__ void ld_nc_v8(const float *p, float (&v)[8])
{
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// Entry e of query q's sorted list (key ~0: the reference's "no candidate").
__device__ __forceinline__ void emit(int e, unsigned long long key, int q, int knn, size_t o, int *miKnn,
                                     float *d2Knn, float *vrKnn, float *rho)
{
    const bool have = key != ~0ull;
    const float d2 = have ? __uint_as_float((unsigned)(key >> 32)) : IRC_SINGLE_INF_F;
    const int idx = have ? (int)(key & 0xffffffffu) : q;
    // streaming stores: the outputs are not read again by this kernel and
    // should not push the gathered feature rows out of L2
    __stcs(miKnn + (size_t)e + (size_t)knn * o, idx + 1);
    if (d2Knn) __stcs(d2Knn + (size_t)e + (size_t)knn * o, d2);
    if (e == knn - 1) {
        const float vk = irc::ref_sqrt_abs(d2);
        __stcs(vrKnn + o, vk);
        if (rho) __stcs(rho + o, __fdiv_rn(1.0f, vk));
    }
}

// FP32 squared distances of NR rows to the staged query row, reference
// arithmetic, the first nd features.  (Two rows at a time share the query's
// shared-memory reads and keep twice the gathers in flight.)
template <int NR>
__device__ __forceinline__ void row_dists(const float4 *__restrict__ Fp, int Dp4, const int (&idx)[NR], const float4 *qs,
                                          int nd, float (&acc)[NR])
{
    const float *bs[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        bs[r] = reinterpret_cast<const float *>(Fp + (size_t)idx[r] * Dp4);
        acc[r] = 0.0f;
    }
    const int full = nd >> 3, tail = nd & 7;       // whole groups of 8 features, then the rest
#pragma unroll 2
    for (int c8 = 0; c8 < full; ++c8) {
        float bv[NR][8];
#pragma unroll
        for (int r = 0; r < NR; ++r) ld_nc_v8(bs[r] + 8 * c8, bv[r]);
        const float4 a0 = qs[2 * c8], a1 = qs[2 * c8 + 1];
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int r = 0; r < NR; ++r) acc[r] = irc::dterm(acc[r], bv[r][u], av[u]);
    }
    if (tail) {
        float bv[NR][8];
#pragma unroll
        for (int r = 0; r < NR; ++r) ld_nc_v8(bs[r] + 8 * full, bv[r]);
        const float4 a0 = qs[2 * full], a1 = qs[2 * full + 1];
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < tail) {
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r] = irc::dterm(acc[r], bv[r][u], av[u]);
            }
    }
}

// Exact FP32 squared distances of the cL listed candidates of query q
// (cL <= 32 PER) with the reference arithmetic (d = b - a, fused accumulate in
// feature order) as sort keys (distance bits, row); ~0 for no candidate, a
// distance of 0 or one that is not below the reference's sentinel.  Candidate
// e is lane e % 32 of round e / 32, and every lane gathers its own rows; Fp:
// rows padded to Dp4 float4 (whole 32-byte sectors); nd: the features that can
// be non-zero for this query and its candidates (the width of their site): the
// rest are zero in both rows and add exactly 0 to every distance, so they are
// skipped.  qs: the warp's staging row.  FRESH: other blocks of this kernel wrote
// the list.
template <int PER, bool FRESH = false>
__device__ __forceinline__ void list_keys(const uint32_t *__restrict__ list, int cL, const float4 *__restrict__ Fp,
                                          int Dp4, int q, float4 *__restrict__ qs, int nd, int lane,
                                          unsigned long long (&kv)[PER])
{
    // the query row, staged once per warp (broadcast reads below)
    if (lane < Dp4) qs[lane] = __ldg(Fp + (size_t)q * Dp4 + lane);
    const int nbatch = (cL + 31) / 32;                // <= PER (checked by the caller)
#pragma unroll
    for (int i = 0; i < PER; ++i) kv[i] = ~0ull;
    __syncwarp();
#pragma unroll
    for (int bi = 0; bi < PER; bi += 2) {
        if (bi >= nbatch) break;
        int idx[2];                                   // (past the end: the query itself, at distance 0)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int e = (bi + r) * 32 + lane;
            idx[r] = e >= cL ? q : FRESH ? (int)__ldcg(list + e) : (int)__ldg(list + e);
        }
        float acc[2];
        row_dists<2>(Fp, Dp4, idx, qs, nd, acc);
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (acc[r] > 0.0f && acc[r] < IRC_SINGLE_INF_F)
                kv[bi + r] = ((unsigned long long)__float_as_uint(acc[r]) << 32) | (unsigned)idx[r];
    }
}

// Ascending bitonic sort of 64 32-bit keys, element 2 lane + i in v[i]; a
// comparison is one shuffle and one minimum or maximum.
__device__ __forceinline__ void warp_bitonic64(unsigned (&v)[2], int lane)
{
#pragma unroll
    for (int size = 2; size <= 64; size <<= 1) {
        const bool up = (2 * lane & size) == 0;
#pragma unroll
        for (int stride = size >> 1; stride > 1; stride >>= 1) {
            const bool keep_min = ((2 * lane & stride) == 0) == up;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned o = __shfl_xor_sync(0xffffffffu, v[i], stride >> 1);
                v[i] = keep_min ? min(v[i], o) : max(v[i], o);
            }
        }
        const unsigned a = min(v[0], v[1]), b = max(v[0], v[1]);
        v[0] = up ? a : b;
        v[1] = up ? b : a;
    }
}

// ws[0 .. 64) <- the keys of lists of at most 64 entries, all of them, ascending
// and ~0 behind them; false (ws untouched) if the short keys cannot order
// them.  A short key is the distance bits above the smallest one's (26 bits: d2
// within a factor of 256, whatever the scale) and the entry (6 bits), so equal
// distances are not ordered by it.  Sorting 64 short keys costs less than
// finding the knn-th distance, compacting and sorting half as many 64-bit keys
// (re-rank of 3,600 chunks' 625,000 queries 884 us so, 1,060 instructions a
// query).
__device__ __forceinline__ bool sort_short(const unsigned long long (&kv)[2], unsigned lo, unsigned hi,
                                           unsigned long long *ws, int lane)
{
    if (lo > hi || hi - lo >= (1u << 26) - 1u) return false;       // (uniform)
    unsigned v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
        v[i] = kv[i] == ~0ull ? ~0u : ((unsigned)(kv[i] >> 32) - lo) << 6 | (unsigned)(i * 32 + lane);
    warp_bitonic64(v, lane);
    const unsigned next = __shfl_down_sync(0xffffffffu, v[0], 1);
    const bool tie = (v[0] >> 6 == v[1] >> 6 && v[1] != ~0u) || (lane < 31 && v[1] >> 6 == next >> 6 && next != ~0u);
    if (__any_sync(0xffffffffu, tie)) return false;
    unsigned long long out[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const unsigned i0 = __shfl_sync(0xffffffffu, (unsigned)kv[0], v[i] & 31u);
        const unsigned i1 = __shfl_sync(0xffffffffu, (unsigned)kv[1], v[i] & 31u);
        out[i] = v[i] == ~0u ? ~0ull : (unsigned long long)(lo + (v[i] >> 6)) << 32 | ((v[i] & 32u) ? i1 : i0);
    }
    __syncwarp();
    *reinterpret_cast<ulonglong2 *>(ws + 2 * lane) = make_ulonglong2(out[0], out[1]);
    __syncwarp();
    return true;
}

// ws[0 .. n) <- the keys with distance bits <= tb, ascending, the rest of ws
// ~0; returns n.  tb bounds the k-th smallest distance from above: a bitwise
// search (stopped at TAU_LOW_BIT, rounded up), plus 2^-16 relative, so that
// the FP64 band of the tensor-core forms lies inside it; +inf when there are
// fewer than k keys.  The keys are a prefix of the full sort.  When more than
// WARP_KEYS pass, ws is not usable.  Lists of at most 64 entries are sorted
// whole where sort_short can.
template <int PER>
__device__ __forceinline__ int select_keys(const unsigned long long (&kv)[PER], int k, unsigned long long *ws, int lane,
                                           unsigned &tb)
{
    static_assert(PER >= 2, "lists of at least two rounds");
    // the bits above the highest one in which the keys' distances differ
    // are common to all of them, hence the answer's: start below them
    unsigned lo = 0xffffffffu, hi = 0u;
#pragma unroll
    for (int i = 0; i < PER; ++i)
        if (kv[i] != ~0ull) {
            lo = min(lo, (unsigned)(kv[i] >> 32));
            hi = max(hi, (unsigned)(kv[i] >> 32));
        }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if constexpr (PER == 2) {
        if (sort_short(kv, lo, hi, ws, lane)) {
            tb = 0x7f800000u;
            return __popc(__ballot_sync(0xffffffffu, kv[0] != ~0ull)) + __popc(__ballot_sync(0xffffffffu, kv[1] != ~0ull));
        }
    }
    unsigned ans = 0;
    int top = 30;
    if (lo <= hi) {                               // some key: distances are below 2^31 as bit patterns
        const unsigned x = lo ^ hi;
        top = x ? 31 - __clz(x) : TAU_LOW_BIT;
        ans = top < 31 ? lo & ~((2u << top) - 1u) : 0u;
        top = min(top, 30);
    }
#pragma unroll 1
    for (int b = top; b >= TAU_LOW_BIT; --b) {
        const unsigned t = ans | (1u << b);
        unsigned c = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) c += (unsigned)((unsigned)(kv[i] >> 32) < t);
        if (__reduce_add_sync(0xffffffffu, c) < (unsigned)k) ans = t;
    }
    const unsigned ub = ans | ((1u << TAU_LOW_BIT) - 1u);
    tb = ub >= 0x7f800000u ? 0x7f800000u : __float_as_uint(__uint_as_float(ub) * (1.0f + 0x1p-16f));
    int n = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const bool pr = (unsigned)(kv[i] >> 32) <= tb;          // never an empty slot (~0)
        const unsigned bal = __ballot_sync(0xffffffffu, pr);
        const int pos = n + __popc(bal & ((1u << lane) - 1u));
        if (pr && pos < WARP_KEYS) ws[pos] = kv[i];
        n += __popc(bal);
    }
    __syncwarp();
    if (n <= 32) {                                // ~k keys, one per lane
        unsigned long long v1[1] = {lane < n ? ws[lane] : ~0ull};
        __syncwarp();
        warp_bitonic<unsigned long long, 1>(v1, lane);
        ws[lane] = v1[0];
        ws[32 + lane] = ~0ull;
    } else if (n <= WARP_KEYS) {
        unsigned long long v2[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) v2[i] = lane * 2 + i < n ? ws[lane * 2 + i] : ~0ull;
        __syncwarp();
        warp_bitonic<unsigned long long, 2>(v2, lane);
#pragma unroll
        for (int i = 0; i < 2; ++i) ws[lane * 2 + i] = v2[i];
    }
    __syncwarp();
    return n;
}

}  // namespace irc_rr
