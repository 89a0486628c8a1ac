// irc_tc_host.cu -- operand preparation and launch of the tensor-core kNN.
//
// Operand rows.  Every spike is stored twice in BF16, padded to K = 64 (one
// 128-byte swizzle row):
//     query row     [ -2*a_1 .. -2*a_D,  na_h, na_m, na_l,  1, 1, 1,  0, 0, 0,  0 ... ]
//     candidate row [    b_1 ..    b_D,     1,    1,    1, nb_h, nb_m, nb_l, 1, 1, 1, 0 ... ]
// where a, b are the BF16-rounded features and na = |a|^2 (FP32, from the
// rounded values) split exactly into three BF16 terms, so one K = 64
// contraction yields |a|^2 + |b|^2 - 2 a.b = |a - b|^2 of the rounded
// features, accumulated in FP32.  The filter's second pass writes a query's
// threshold, -tau split into three BF16 terms, into the three zeros of its
// row in shared memory (irc_tc.cu): its accumulators are then d2 - tau.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "irc_common.cuh"
#include "irc_plan.cuh"
#include "irc_tc.cuh"

namespace {

using irc_tc::Fmt;

// Centring of the tensor-core operands.  Distances do not change when every
// feature vector is shifted by the same reference point, but the rounding
// error of the BF16 / FP8 contraction grows with the operands' magnitude, and
// drift can carry features far from the origin.  The operand rows are built
// from F - ref with ref = the column means of a strided sample of at most
// 64K of the plan's query rows (fixed summation order, so the rows are the
// same on every call); the exact re-rank keeps reading the unshifted
// features.
//
// One launch: every block sums its rows (a thread per (row, column), so that a
// block reads whole consecutive rows), and the block that ends last adds the
// partial sums -- with all of its threads: one thread per column adding 256
// partials in a kernel of its own took 25 us of every call, the sums before it
// 4 to 12.  Latency-bound: 9 us for 3,000 rows, 24 for 65,536 rows out of 400,000.
constexpr int kMeanBlocks = 152, kMeanThreads = 512;

__global__ void __launch_bounds__(kMeanThreads)
k_centre(const float *__restrict__ F, int nC, int stride, int nS, float *__restrict__ part, unsigned *__restrict__ ticket,
         float *__restrict__ ref)
{
    after_previous();
    __shared__ double red[kMeanThreads];
    __shared__ bool last;
    const int t = threadIdx.x, lanes = kMeanThreads / nC, rl = t / nC, c = t - rl * nC;
    const int per = (nS + gridDim.x - 1) / gridDim.x;
    const int k0 = blockIdx.x * per, k1 = min(nS, k0 + per);
    float acc = 0.0f;
    if (rl < lanes) {
#pragma unroll 8
        for (int k = k0 + rl; k < k1; k += lanes) acc += __ldg(F + (size_t)k * stride * nC + c);
    }
    float *redf = reinterpret_cast<float *>(red);
    redf[t] = acc;
    __syncthreads();
    if (t < nC) {
        float sum = 0.0f;
#pragma unroll 4
        for (int r = 0; r < lanes; ++r) sum += redf[r * nC + t];
        part[(size_t)blockIdx.x * 64 + t] = sum;
        __threadfence();
    }
    __syncthreads();
    if (t == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double sum = 0.0;
    if (rl < lanes) {
#pragma unroll 4
        for (int b = rl; b < gridDim.x; b += lanes) sum += (double)__ldcg(part + (size_t)b * 64 + c);
    }
    red[t] = sum;
    __syncthreads();
    if (t < nC) {
        for (int r = 1; r < lanes; ++r) sum += red[r * nC + t];
        ref[t] = nS > 0 ? (float)(sum / (double)nS) : 0.0f;
    }
}

// Bits of x in ascending order of x.
__device__ __forceinline__ unsigned ordered(float x)
{
    const unsigned u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Centre and scale of the F16 operands, of which each query's proof needs that
// most rows are well inside the half-precision range.  A few spikes far out
// (artefacts), or not finite, must not move either: with the mean and the
// largest magnitude, five rows of 10,000 at 1,000 times the others left every
// query without a proof.  Every block takes the column means of its rows and
// their largest distance from its first row; ref is the median of 32 blocks' means
// per column, and *scale the power of two that brings the upper quartile over the
// blocks of (that distance + the mean's distance from ref) to at most 8.  Rows
// that are then too long for F16 get no operand (k_prep), which the proof takes
// into account.  Values that are not finite are left out.  *scale 0 (nothing is
// proven): the squared distances leave FP32's range.  part, the magnitudes in
// column 63 (nC <= 58); ticket: zero, and zero again at the end.
__global__ void __launch_bounds__(kMeanThreads)
k_centre_robust(const float *__restrict__ F, int nC, int stride, int nS, float *__restrict__ part,
                unsigned *__restrict__ ticket, float *__restrict__ ref, float *__restrict__ scale)
{
    after_previous();
    __shared__ float means[kMeanBlocks][65];                 // (a warp reads a column)
    __shared__ float red[kMeanThreads], mags[kMeanThreads / 32], sref[64];
    __shared__ int cnt[kMeanThreads];
    __shared__ bool last;
    const float none = __int_as_float(0x7fc00000);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int lanes = kMeanThreads / nC, rl = t / nC, c = t - rl * nC;
    const int per = (nS + gridDim.x - 1) / gridDim.x;
    const int k0 = blockIdx.x * per, k1 = min(nS, k0 + per);
    float acc = 0.0f, mx = 0.0f, first = 0.0f;               // sums from the first row: no offset to lose digits to
    int n = 0;
    if (rl < lanes && k0 < k1) {
        first = __ldg(F + (size_t)k0 * stride * nC + c);
        if (!isfinite(first)) first = 0.0f;
#pragma unroll 8
        for (int k = k0 + rl; k < k1; k += lanes) {
            const float v = __ldg(F + (size_t)k * stride * nC + c);
            const bool in = isfinite(v);
            const float d = in ? v - first : 0.0f;
            acc += d;
            mx = fmaxf(mx, fabsf(d));
            n += in;
        }
    }
    red[t] = acc;
    cnt[t] = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) mags[warp] = mx;
    __syncthreads();
    if (t < nC) {
        for (int r = 1; r < lanes; ++r) {
            acc += red[r * nC + t];
            n += cnt[r * nC + t];
        }
        part[(size_t)blockIdx.x * 64 + t] = n ? first + acc / (float)n : none;
    } else if (t == 63) {
        for (int w = 0; w < kMeanThreads / 32; ++w) mx = fmaxf(mx, mags[w]);
        part[(size_t)blockIdx.x * 64 + 63] = k0 < k1 ? mx : none;
    }
    if (t < 64) __threadfence();
    __syncthreads();
    if (t == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    static_assert(kMeanBlocks * 64 % kMeanThreads == 0, "whole turns");
#pragma unroll
    for (int k = 0; k < kMeanBlocks * 64 / kMeanThreads; ++k) {
        const int i = k * kMeanThreads + t;
        means[i >> 6][i & 63] = __ldcg(part + i);
    }
    __syncthreads();
    // median of 32 blocks' means per column, a warp per column, by rank
#pragma unroll 1
    for (int k = warp; k < nC; k += kMeanThreads / 32) {
        const float v = means[lane * kMeanBlocks / 32][k];
        const unsigned key = isfinite(v) ? ordered(v) : ~0u;
        unsigned rank = 0;
#pragma unroll
        for (int o = 0; o < 32; ++o) {
            const unsigned other = __shfl_sync(0xffffffffu, key, o);
            rank += other < key || (other == key && o < lane);
        }
        const unsigned m = __popc(__ballot_sync(0xffffffffu, key != ~0u));
        if (key != ~0u && rank == m / 2) sref[k] = v;
        if (m == 0 && lane == 0) sref[k] = 0.0f;
    }
    __syncthreads();
    if (t < nC) ref[t] = sref[t];
    float size = none;
    if (t < kMeanBlocks) {
        size = means[t][63];
        float d = 0.0f;
        for (int k = 0; k < nC; ++k) d = fmaxf(d, fabsf(means[t][k] - sref[k]));
        size += d;
    }
    red[t] = size;
    if (t == 0) mags[0] = 0.0f;
    __syncthreads();
    if (t < kMeanBlocks) {
        int rank = 0, m = 0;
#pragma unroll 8
        for (int b = 0; b < kMeanBlocks; ++b) {
            const float o = red[b];
            m += o == o;
            rank += o < size || (o == size && b < t);
        }
        if (size == size && rank == (3 * m + 3) / 4 - 1) mags[0] = size;
    }
    __syncthreads();
    if (t == 0) {
        const float b = mags[0];
        *scale = !(b > 0.0f) ? 1.0f : !(b < 0x1p62f) ? 0.0f : ldexpf(1.0f, min(30, 2 - ilogbf(b)));
    }
}

// |F| maximum (bits of a non-negative float, so integer max == float max).
__global__ void k_absmax(const float *__restrict__ F, size_t n, int nC, const float *__restrict__ ref,
                         unsigned *__restrict__ out)
{
    after_previous(ref);
    unsigned m = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(fabsf(__ldg(F + i) - __ldg(ref + i % nC))));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__device__ __forceinline__ unsigned char to_e4m3(float x)
{
    return (unsigned char)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}

__device__ __forceinline__ float from_e4m3(unsigned char v)
{
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)v, __NV_E4M3);
    return __half2float(__half(h));
}

// FP8 rows of 128 e4m3 values (K = 128, 128 bytes).  With x = e4m3(s*a),
// y = e4m3(s*b) and s = 32 / max|F| (so |x| <= 32 and -2x is exact):
//     query row     [ -2x_1 .. -2x_D, nx_0 .. nx_5, 2^e_0 .. 2^e_5, 0 ... ]
//     candidate row [    y_1 ..  y_D, 2^e_0 .. 2^e_5, ny_0 .. ny_5, 0 ... ]
// where |x|^2 = sum_t nx_t * 2^e_t (e = 8, 4, 0, -4, -8, -9: each e4m3 piece
// takes the next 4 bits of the remainder), so the contraction is
// s^2 |a - b|^2 of the rounded features -- a positive multiple, which the
// filter only compares.
constexpr int kFp8Pieces = 6;
__device__ __forceinline__ int piece_exp(int t) { return t < 5 ? 8 - 4 * t : -9; }

// Operand preparation, one warp per 32 consecutive rows of a row interval.
// The rows (contiguous in F) are read coalesced into shared memory with an
// odd row stride (nC | 1 words), so lane r working on row r has no bank
// conflicts; every lane builds its row's query and candidate operand rows
// (BF16: above the file; FP8: above) and stages them in shared memory in
// 16-byte pieces XOR-swizzled by row; the warp then writes its 32 rows of
// every output -- the re-rank's FP32 rows padded to Dp4 float4 too -- with
// contiguous stores.  Bound by the memory it writes once the instructions are
// few and a warp's rows are all in flight at once: 52 us for 400,000 rows of
// 33 features (220 MB).  With element counters by division, four loads in flight
// and every operand element through the general form it took 79.
constexpr int kPrepWarps = 4;

size_t prep_smem(int nC)
{
    return (size_t)kPrepWarps * (2 * 32 * 128 + 32 * (size_t)(nC | 1) * 4) + 64 * 4;
}

// The 16-bit operand value of x: its bits, and the value they stand for.
template <Fmt FMT>
__device__ __forceinline__ unsigned short op16(float x)
{
    return FMT == Fmt::f16 ? __half_as_ushort(__float2half_rn(x)) : __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

template <Fmt FMT>
__device__ __forceinline__ float val16(unsigned short v)
{
    return FMT == Fmt::f16 ? __half2float(__ushort_as_half(v)) : __bfloat162float(__ushort_as_bfloat16(v));
}

__device__ __forceinline__ void copy_word(float *shared, const float *global)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(shared)), "l"(global)
                 : "memory");
}

// 16-bit element `at` of a row that is otherwise written in 16-byte pieces.
__device__ __forceinline__ void st_shared_u16(uint4 *row, int at, unsigned short v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(row) + 2u * at), "h"(v) : "memory");
}

// qnorm (f16): an upper bound of every query's scaled norm |s (a - ref)|: the
// rounded row's norm, plus the rounding (2^-11 relative, 2^-25 absolute per
// feature), with room.  A row longer than irc_tc::F16_NORM2 allows, or not
// finite, gets an operand without features: as a candidate at distance inf.
template <Fmt FMT>
__global__ void __launch_bounds__(32 * kPrepWarps)
k_prep(const float *__restrict__ F, int lo, int n, int nC, const float *__restrict__ ref,
       const unsigned *__restrict__ amax, uint4 *__restrict__ Fq, uint4 *__restrict__ Fc, float *__restrict__ Fp,
       int Dp4, int q_lo, int q_hi, const float *__restrict__ scale, float *__restrict__ qnorm)
{
    after_previous(ref, amax, scale);
    extern __shared__ __align__(16) unsigned char prep_sm[];
    const int nCs = nC | 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint4 *sq = reinterpret_cast<uint4 *>(prep_sm) + (size_t)warp * 2 * 32 * 8;     // [32 rows][8], swizzled
    uint4 *sc = sq + 32 * 8;
    float *sref = reinterpret_cast<float *>(prep_sm + (size_t)kPrepWarps * 2 * 32 * 128);
    float *w = sref + 64 + (size_t)warp * 32 * nCs;
    for (int k = threadIdx.x; k < nC; k += blockDim.x) sref[k] = __ldg(ref + k);
    __syncthreads();
    const long long r0 = (long long)lo + ((long long)blockIdx.x * kPrepWarps + warp) * 32;
    if (r0 >= (long long)lo + n) return;
    const int nr = (int)min(32LL, (long long)lo + n - r0);
    const float *src = F + (size_t)r0 * nC;
    // (4-byte copies: the rows start on any word; all of them in flight at once)
    for (int c = lane; c < nC; c += 32) {
#pragma unroll 8
        for (int r = 0; r < nr; ++r) copy_word(w + r * nCs + c, src + r * nC + c);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const int W = 4 * Dp4;
    float *dst = Fp + (size_t)r0 * W;
    for (int c = lane; c < W; c += 32) {
#pragma unroll 8
        for (int r = 0; r < nr; ++r) dst[r * W + c] = c < nC ? w[r * nCs + c] : 0.0f;
    }
    if (lane < nr) {
        const float *a = w + lane * nCs;
        uint4 *oq = sq + lane * 8, *oc = sc + lane * 8;
        const int sw = lane & 7;
        if (FMT != Fmt::fp8) {
            const float s16 = FMT == Fmt::f16 ? *scale : 1.0f;         // a power of two: exact
            float na = 0.0f;
#pragma unroll 1
            for (int j = 0; j < irc_tc::KP / 8; ++j) {
                __align__(16) unsigned short wq[8], wc[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = j * 8 + e;
                    wq[e] = wc[e] = 0;
                    if (k < nC) {
                        wc[e] = op16<FMT>((a[k] - sref[k]) * s16);
                        const float f = val16<FMT>(wc[e]);
                        na = __fmaf_rn(f, f, na);
                        wq[e] = op16<FMT>(-2.0f * f);
                    }
                }
                oq[j ^ sw] = *reinterpret_cast<uint4 *>(wq);
                oc[j ^ sw] = *reinterpret_cast<uint4 *>(wc);
            }
            const bool out = FMT == Fmt::f16 && !(na <= irc_tc::F16_NORM2);
            if (out) {
                for (int j = 0; j < irc_tc::KP / 8; ++j) oq[j] = oc[j] = make_uint4(0u, 0u, 0u, 0u);
            }
            // the 9 elements behind the features (nC + 9 may pass the row's
            // end, where only the zeros of the query row are missing)
            const unsigned short h = op16<FMT>(na);
            const float rem1 = na - val16<FMT>(h);
            const unsigned short m = op16<FMT>(rem1);
            const unsigned short l = op16<FMT>(rem1 - val16<FMT>(m));
            const unsigned short one = op16<FMT>(1.0f);
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const int k = nC + i;
                if (k >= irc_tc::KP) break;
                const int at = ((k >> 3) ^ sw) * 8 + (k & 7);
                const unsigned short n3 = i % 3 == 0 ? h : i % 3 == 1 ? m : l;
                if (i < 6) st_shared_u16(oq, at, i >= 3 ? one : out ? 0 : n3);
                st_shared_u16(oc, at, i < 3 || i >= 6 ? one : !out ? n3 : i == 3 ? op16<FMT>(__int_as_float(0x7f800000)) : 0);
            }
            const long long row = r0 + lane;
            if (FMT == Fmt::f16 && row >= q_lo && row < q_hi)
                qnorm[row - q_lo] = __fsqrt_ru(na) * (1.0f + 0x1p-9f) + 1e-6f;
        } else {
            const float am = __uint_as_float(*amax);
            const float scl = am > 0.0f ? 32.0f / am : 1.0f;
            float nx = 0.0f;
            for (int k = 0; k < nC; ++k) {
                const float x = from_e4m3(to_e4m3(scl * (a[k] - sref[k])));
                nx = __fmaf_rn(x, x, nx);
            }
            unsigned char pc[kFp8Pieces], pf[kFp8Pieces];
            float rem = nx;
#pragma unroll
            for (int t = 0; t < kFp8Pieces; ++t) {
                const float f = ldexpf(1.0f, piece_exp(t));
                pc[t] = to_e4m3(rem / f);
                pf[t] = to_e4m3(f);
                rem -= from_e4m3(pc[t]) * f;
            }
#pragma unroll 1
            for (int j = 0; j < 128 / 16; ++j) {
                __align__(16) unsigned char wq[16], wc[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int k = j * 16 + e;
                    unsigned char vq = 0, vc = 0;
                    if (k < nC) {
                        const unsigned char y = to_e4m3(scl * (a[k] - sref[k]));
                        vc = y;
                        vq = to_e4m3(-2.0f * from_e4m3(y));
                    } else if (k < nC + kFp8Pieces) {
                        vq = pc[k - nC];
                        vc = pf[k - nC];
                    } else if (k < nC + 2 * kFp8Pieces) {
                        vq = pf[k - nC - kFp8Pieces];
                        vc = pc[k - nC - kFp8Pieces];
                    }
                    wq[e] = vq;
                    wc[e] = vc;
                }
                oq[j ^ sw] = *reinterpret_cast<uint4 *>(wq);
                oc[j ^ sw] = *reinterpret_cast<uint4 *>(wc);
            }
        }
    }
    __syncwarp();
    // query rows (the plan's own queries, q_lo .. q_hi-1) are only read as query operands
    uint4 *gq = Fq + (size_t)r0 * 8, *gc = Fc + (size_t)r0 * 8;
    for (int t = lane; t < nr * 8; t += 32) {
        const int r = t >> 3, j = t & 7;
        if (r0 + r >= q_lo && r0 + r < q_hi) gq[t] = sq[r * 8 + (j ^ (r & 7))];
        gc[t] = sc[r * 8 + (j ^ (r & 7))];
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// Tensor map over [rows x 128 bytes] operand rows (64 BF16 or F16, or 128 e4m3 values),
// box_rows-row boxes, 128-byte swizzle.
int make_map(CUtensorMap *m, void *base, int rows, int box_rows, Fmt fmt)
{
    const bool fp8 = fmt == Fmt::fp8;
    EncodeTiledFn enc = encode_fn();
    if (!enc) { irc_host::set_error("cuTensorMapEncodeTiled unavailable"); return IRC_E_CUDA; }
    const int inner = fp8 ? 128 : irc_tc::KP;
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)128};
    cuuint32_t box[2] = {(cuuint32_t)inner, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                            : fmt == Fmt::f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                     2, base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { irc_host::set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return IRC_E_CUDA; }
    return IRC_OK;
}

}  // namespace

// The plan's tensor-core working memory (irc_site.cu) and the exact
// fallback for queries whose candidate list overflowed (irc_exact.cu).
int irc_plan_tc_buffer(irc_plan *pl, size_t need, void **buf);
int irc_exact_overflow_drain(irc_plan *pl, const float *F, int nC, int knn, float *vrKnn, float *rho,
                             int32_t *miKnn, float *d2Knn, cudaStream_t s);

namespace irc_tc {

constexpr size_t kPartBytes = sizeof(float) * kMeanBlocks * 64;

static size_t fp_bytes(const irc_plan *pl, int nC)
{
    return ((size_t)pl->dev.nF * (size_t)fp_row4(nC) * 16 + 255) & ~(size_t)255;
}

// query rows | candidate rows | padded FP32 rows | column sums | centre (256
// bytes) | f16: scale (256 bytes), query norms
size_t ops_bytes(const irc_plan *pl, int nC, Fmt fmt)
{
    const size_t q = fmt == Fmt::f16 ? 256 + (((size_t)pl->dev.n_out * 4 + 255) & ~(size_t)255) : 0;
    return 2 * (size_t)pl->dev.nF * 128 + fp_bytes(pl, nC) + kPartBytes + 256 + q;
}

int make_operands(Fmt fmt, irc_plan *pl, const float *F, int nC, void *buf, unsigned *amax, unsigned *ticket,
                  Operands *out, cudaStream_t s)
{
    const bool fp8 = fmt == Fmt::fp8, f16 = fmt == Fmt::f16;
    const int nF = pl->dev.nF, Dp4 = fp_row4(nC);
    const size_t one = (size_t)nF * 128;
    char *b = (char *)buf;
    void *fq = b, *fc = b + one, *fp = b + 2 * one;
    float *part = (float *)(b + 2 * one + fp_bytes(pl, nC));
    float *ref = (float *)((char *)part + kPartBytes);
    float *scale = ref + 64, *qnorm = ref + 128;
    const int nQ = pl->dev.n_out;                                     // the query rows q_base ..
    const int stride = nQ > 65536 ? (nQ + 65535) / 65536 : 1;
    const int nS = (nQ + stride - 1) / stride;                        // sampled: q_base + k * stride
    const float *Fq0 = F + (size_t)pl->dev.q_base * nC;
    if (f16) {
        launch_next(k_centre_robust, kMeanBlocks, kMeanThreads, 0, s, Fq0, nC, stride, nS, part, ticket, ref, scale);
    } else {
        launch_next(k_centre, kMeanBlocks, kMeanThreads, 0, s, Fq0, nC, stride, nS, part, ticket, ref);
        for (int v = 0; fp8 && v < pl->n_row_iv; ++v) {
            const int lo = pl->row_iv[2 * v], n = pl->row_iv[2 * v + 1] - lo;
            launch_next(k_absmax, 152 * 4, 256, 0, s, F + (size_t)lo * nC, (size_t)n * nC, nC, ref, amax);
        }
    }
    IRC_CHECK_LAUNCH("irc_site_knn(tensor core) centre");
    // operand rows for the rows the plan reads (its row intervals)
    const size_t psm = prep_smem(nC);
    auto prep = fp8 ? k_prep<Fmt::fp8> : f16 ? k_prep<Fmt::f16> : k_prep<Fmt::bf16>;
    cudaError_t e = cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psm);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(tensor core): prep smem attribute");
    for (int v = 0; v < pl->n_row_iv; ++v) {
        const int lo = pl->row_iv[2 * v], n = pl->row_iv[2 * v + 1] - lo;
        const int rows_per_block = 32 * kPrepWarps;
        launch_next(prep, (n + rows_per_block - 1) / rows_per_block, 32 * kPrepWarps, psm, s, 
            F, lo, n, nC, ref, amax, (uint4 *)fq, (uint4 *)fc, (float *)fp, Dp4, pl->dev.q_base,
            pl->dev.q_base + pl->dev.n_out, scale, qnorm);
    }
    IRC_CHECK_LAUNCH("irc_site_knn(tensor core) prep");
    int rc = make_map(&out->mq, fq, nF, 32, fmt);                     // 32 query rows per lane quarter
    if (rc == IRC_OK) rc = make_map(&out->mc, fc, nF, 128, fmt);      // 128-row candidate tiles
    out->fp = (const float4 *)fp;
    out->scale = scale;
    out->qnorm = qnorm;
    return rc;
}

}  // namespace irc_tc

int irc_site_knn_tc(irc_plan *pl, const float *F, int nC, int knn, int mode, float *vrKnn, float *rho,
                    int32_t *miKnn, float *d2Knn, cudaStream_t s)
{
    const bool fp8 = mode == IRC_MODE_FP8;
    const Fmt fmt = fp8 ? Fmt::fp8 : Fmt::bf16;
    if (nC + (fp8 ? 2 * kFp8Pieces : 6) > (fp8 ? 128 : irc_tc::KP)) {
        irc_host::set_error("irc_site_knn(tensor core): nC=%d too large", nC);
        return IRC_E_NC;
    }
    if (knn > irc_tc::KNN_MAX) { irc_host::set_error("irc_site_knn(BF16): knn %d > %d", knn, irc_tc::KNN_MAX); return IRC_E_INVAL; }
    void *buf;
    const size_t ops = irc_tc::ops_bytes(pl, nC, fmt);
    const size_t need = ops + irc_tc::list_area_bytes(pl->dev.n_out);
    size_t reserve = irc_tc::split_reserve(pl);
    if (pl->tc_external && pl->tc_bytes < need + reserve) reserve = 0;      // the caller's memory is enough without
    int rc = irc_plan_tc_buffer(pl, need + reserve, &buf);
    if (rc != IRC_OK) return rc;
    irc_tc::ListOut lo = irc_tc::list_area((char *)buf + ops, pl->dev.n_out);
    if (reserve) irc_tc::split_area(pl, nC, fmt, (char *)buf + need, &lo);
    cudaError_t e = cudaMemsetAsync(pl->scratch, 0, 2 * sizeof(int), s);   // overflow-queue count, largest magnitude
    if (e == cudaSuccess) e = irc_tc::clear_lists(lo, pl->dev.n_out, s);
    if (e != cudaSuccess) return irc_host::cuda_status(e, "irc_site_knn(BF16): memset");
    irc_tc::Operands op;
    unsigned *words = reinterpret_cast<unsigned *>(pl->scratch);
    rc = irc_tc::make_operands(fmt, pl, F, nC, buf, words + 1, words + irc::kScratchTicket, &op, s);
    if (rc != IRC_OK) return rc;
    rc = irc_tc::launch_knn_tc(fmt, op.mq, op.mc, pl, F, op.fp, nC, knn, vrKnn, rho, miKnn, d2Knn, lo, s);
    if (rc != IRC_OK) return rc;
    return irc_exact_overflow_drain(pl, F, nC, knn, vrKnn, rho, miKnn, d2Knn, s);
}
