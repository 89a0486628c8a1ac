// irc_rows.cuh -- plain FP32 distances of a tile: candidate rows staged per
// warp, two candidates and QB queries per thread.
//
// One lane per candidate reading its own row of F from global memory costs a
// load of 32 different cache lines for every feature, and the L1 spends more
// time on it than the FP32 pipe on the 2 QB operations it feeds (5 to 7 times
// off that pipe's rate).  Here 64 rows (any rows: each is nC consecutive floats) are copied into
// shared memory with coalesced asynchronous copies, a step ahead of their use,
// at an odd row pitch so that a lane reading its own row has no bank
// conflicts, and NG warps share them, each for its own QB queries (unshared,
// the copies took more issue slots than they fed arithmetic: 350 us against
// the FP32 pipe's 106 for 2,000 queries x 30,000 candidates x 33 features).
// Each thread works on two rows: a broadcast of four query features feeds
// eight pairs (a 16-byte broadcast takes two cycles of the SM's shared memory,
// so one row per thread would be bound by it).  The operations are packed two
// queries at a time (add / fma .f32x2, each half rounded as the scalar
// operation): the same FP32 pipe time in half the issue slots.  Queries are
// staged negated, b + (-a) being b - a.
#pragma once
#include "irc_common.cuh"

namespace irc {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float x, float y)
{
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &x, float &y)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
// b + a and a * b + c per half, each rounded as the scalar operation: d = b +
// (-a), acc + d * d is the reference's distance term (irc::dterm)
__device__ __forceinline__ f32x2 add2(f32x2 b, f32x2 a)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(b), "l"(a));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__host__ __device__ inline int row_pitch(int nC) { return nC | 1; }

// Copies of a block of 64 rows by NG warps (this one the g-th): every warp
// holds the row numbers (-1: no row), lane l those of rows l and 32 + l.
template <int NG>
struct RowCopy {
    static constexpr int ROWS = 64 / NG;          // rows this warp copies
    int r0, c0, dr, dc, g;
    __device__ __forceinline__ RowCopy(int nC, int lane, int group) : g(group)
    {
        r0 = lane / nC;
        c0 = lane - r0 * nC;
        dr = 32 / nC;
        dc = 32 - dr * nC;
    }
    // dst[r * pitch + c] <- F[row r][c]
    __device__ __forceinline__ void issue(float *dst, int pitch, const float *__restrict__ F, int nC,
                                          const int (&row)[2]) const
    {
        const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
#pragma unroll
        for (int h = 0; h < 2; ++h) {             // rows 32h .. 32h + 31
            constexpr int N = ROWS < 32 ? ROWS : 32;
            if (ROWS < 64 && (g * ROWS) / 32 != h) continue;
            const int first = (g * ROWS) & 31;    // its first row of the half
            int r = r0, c = c0;
            const int lane = threadIdx.x & 31, b0 = __shfl_sync(0xffffffffu, row[h], 0);
            if (b0 >= 0 && __all_sync(0xffffffffu, row[h] == b0 + lane)) {       // 32 consecutive rows: one block of F
                const float *src = F + (size_t)(b0 + first) * nC;
                const uint32_t o = d + 4u * (uint32_t)((32 * h + first) * pitch);
                const bool flat = pitch == nC;
#pragma unroll 4
                for (int e = lane; e < N * nC; e += 32) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(o + 4u * (uint32_t)(flat ? e : e + r)),
                                 "l"(src + e)
                                 : "memory");
                    if (!flat) {
                        c += dc;
                        r += dr;
                        if (c >= nC) { c -= nC; ++r; }
                    }
                }
                continue;
            }
#pragma unroll 4
            for (int i = 0; i < (N * nC + 31) / 32; ++i) {
                const int s = __shfl_sync(0xffffffffu, row[h], first + (r < N ? r : 0));
                if (r < N && s >= 0)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                     d + 4u * (uint32_t)((32 * h + first + r) * pitch + c)),
                                 "l"(F + (size_t)s * nC + c)
                                 : "memory");
                c += dc;
                r += dr;
                if (c >= nC) { c -= nC; ++r; }
            }
        }
    }
};

// Barrier of the NG warps that share block `sub`'s rows.
template <int NG>
__device__ __forceinline__ void rows_sync(int sub)
{
    if (NG == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(32 * NG) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// NG groups of QB query rows of A (first row a0, n valid; the rest repeat the
// last), negated: group g's feature c of query q at sA[(g * nC + c) * QB + q].
template <int QB, int NG>
__device__ __forceinline__ void stage_negated(const float *__restrict__ A, int nC, int a0, int n, float *sA)
{
    for (int i = threadIdx.x; i < nC * QB * NG; i += blockDim.x) {
        const int k = i / nC, c = i - k * nC, g = k / QB, q = k - g * QB;
        sA[(g * nC + c) * QB + q] = -__ldg(A + (size_t)(a0 + min(k, n - 1)) * nC + c);
    }
}

// Squared distances of two staged rows (p0, p1) to the QB staged queries.
template <int QB>
__device__ __forceinline__ void pair_dist(const float *p0, const float *p1, int nC, const float *sA, float (&d0)[QB],
                                          float (&d1)[QB])
{
    static_assert(QB % 4 == 0, "float4 broadcasts");
    f32x2 a0[QB / 2], a1[QB / 2];
#pragma unroll
    for (int i = 0; i < QB / 2; ++i) a0[i] = a1[i] = 0ull;
#pragma unroll 4
    for (int c = 0; c < nC; ++c) {
        const float x = p0[c], y = p1[c];
        const f32x2 bx = pack2(x, x), by = pack2(y, y);
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(sA + c * QB);
        f32x2 dx[QB / 2], dy[QB / 2];             // differences first: the dependent halves lie apart
#pragma unroll
        for (int j = 0; j < QB / 4; ++j) {
            const ulonglong2 a = q[j];
            dx[2 * j] = add2(bx, a.x);
            dx[2 * j + 1] = add2(bx, a.y);
            dy[2 * j] = add2(by, a.x);
            dy[2 * j + 1] = add2(by, a.y);
        }
#pragma unroll
        for (int i = 0; i < QB / 2; ++i) {
            a0[i] = fma2(dx[i], dx[i], a0[i]);
            a1[i] = fma2(dy[i], dy[i], a1[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < QB / 2; ++i) {
        unpack2(a0[i], d0[2 * i], d0[2 * i + 1]);
        unpack2(a1[i], d1[2 * i], d1[2 * i + 1]);
    }
}

// Which of QB queries (rho ra[q], 16-byte aligned) a candidate of rho rb may
// serve: not rb <= ra (the search kernels' mask), or rb > ra.
template <int QB>
__device__ __forceinline__ unsigned higher_rho(float rb, const float *ra)
{
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < QB; ++q) m |= (unsigned)!(rb <= ra[q]) << q;
    return m;
}
template <int QB>
__device__ __forceinline__ unsigned strictly_higher_rho(float rb, const float *ra)
{
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < QB; ++q) m |= (unsigned)(rb > ra[q]) << q;
    return m;
}

}  // namespace irc
