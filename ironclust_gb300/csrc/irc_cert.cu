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
// could matter.  Otherwise the query's 16-query tile goes through the plain
// kernel, so the outputs are the plain form's bit for bit in every case.
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
// pairs) 22.2 -> 1.09 ms; REF kNN + delta of 60,001 spikes and 12,001 copies
// (D = 24, 30 chunks, 2.2e9 pairs) 29.2 -> 1.46 ms (a site with one
// query without a proof: 0.2 to 0.3 more, a 16-query tile on one SM).  The contraction's error,
// on rows of this layout against FP64, is at most 2^-20.7 of the sum that c
// multiplies.
#include <algorithm>
#include <mutex>

#include "irc_cert.cuh"
#include "irc_common.cuh"
#include "irc_plan.cuh"
#include "irc_rerank.cuh"
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
constexpr int W_OVF = 5;                  // its overflow queue
constexpr int W_TICKET = 6;               // block ticket of the centring
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

// One query's list to its EXACT or REF result; false when it is not proven.
template <int PER, bool REF>
__device__ __forceinline__ bool from_list(const Call &c, const uint32_t *list, int cL, bool complete, float tau, int chunk,
                                          int o, int knn, int nT, float4 *qs, unsigned long long *ws, unsigned *bits,
                                          int lane, float *vrKnn, float *rho, int *miKnn, float *d2Knn)
{
    const int q = c.p.q_base + o;
    const int nd = c.row_dims ? min(c.nC, (int)__ldg(c.row_dims + q)) : c.nC;
    unsigned long long kv[PER];
    irc_rr::list_keys<PER>(list, cL, c.Fp, irc_tc::fp_row4(c.nC), q, qs, nd, lane, kv);
    unsigned tb;
    int n = irc_rr::select_keys<PER>(kv, REF ? kRefKeys : knn, ws, lane, tb);
    const float x = __ldg(c.qnorm + o), s = __ldg(c.scale);
    if (n < knn || n > WARP_KEYS || !(s > 0.0f)) return false;
    if (!REF) {
        const float D = __uint_as_float((unsigned)(ws[knn - 1] >> 32));
        if (!complete && may_miss(D, tau, s, x)) return false;
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
    if (nk < knn) return false;
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
    const unsigned long long kth = __shfl_sync(0xffffffffu, ((knn - 1) & 1) ? k2[1] : k2[0], (knn - 1) >> 1);
    const float v = __uint_as_float((unsigned)(kth >> 32));
    // every candidate left out must have a larger square root than the knn-th
    // value: the listed ones not used (d2 >= tb) and the unlisted ones
    if (tb < 0x7f800000u && !(__fsqrt_rn(__uint_as_float(tb)) > v)) return false;
    if (!complete && may_miss(__fmul_rn(v, v) * (1.0f + 1e-6f), tau, s, x)) return false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int e = 2 * lane + i;
        if (e < knn) __stcs(miKnn + (size_t)e + (size_t)knn * o, (int)(ws[k2[i] & 63u] & 0xffffffffu) + 1);
    }
    if (lane == 0) {
        __stcs(vrKnn + o, v);
        if (rho) __stcs(rho + o, __fdiv_rn(1.0f, v));
    }
    return true;
}

template <bool REF>
__global__ void __launch_bounds__(32 * kWarps, 5)
k_cert_knn(Call c, int knn, int nT, float *__restrict__ vrKnn, float *__restrict__ rho, int *__restrict__ miKnn,
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
    bool ok = false;
    if (qi.x >= 0) {
        const uint32_t *l = c.lists + (unsigned)qi.x;
        const int cL = qi.y & 0x3fffffff;
        const bool complete = (qi.y >> 30) & 1;
        const float tau = __int_as_float(ce.x);
        unsigned long long *ws = wkeys + warp * WARP_KEYS;
        float4 *qs = qrows + warp * QROW4;
        unsigned *bits = wbits + (REF ? warp * 32 : 0);
        if (cL <= 64) ok = from_list<2, REF>(c, l, cL, complete, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn);
        else if (cL <= 128) ok = from_list<4, REF>(c, l, cL, complete, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn);
        else ok = from_list<8, REF>(c, l, cL, complete, tau, ce.y, o, knn, nT, qs, ws, bits, lane, vrKnn, rho, miKnn, d2Knn);
    }
    if (!ok) leave(c, ce.y, c.p.q_base + o, lane);
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

// Working memory of the proven searches: one pool per device, shared by the
// plans, its blocks handed out in stream order (a call of another stream or
// thread gets other memory, so concurrent calls on one plan stay independent,
// as the plain kernels' are).  It keeps at most 1/32 of the device's memory
// between calls and gives everything back when the last plan that used it is
// destroyed.
//
// A captured call takes a block of its own, which the plan keeps (a graph is
// of no use without its plan), so that the graph holds no allocations: one
// that does can be instantiated only once at a time and be no child graph.
// Beyond kMaxCaptured captured calls of a plan, the plain kernels are captured.
constexpr int kMaxDevices = 64;
constexpr int kMaxCaptured = sizeof(irc_plan::captured) / sizeof(void *);
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices];
int g_pool_plans[kMaxDevices];

cudaMemPool_t pool_of(irc_plan *pl)
{
    const int dev = pl->device;
    if (dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        irc_host::Uncaptured mode;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        size_t fr = 0, total = 0;
        cudaMemGetInfo(&fr, &total);
        unsigned long long keep = total / 32;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        g_pool[dev] = pool;
    }
    if (!pl->uses_pool) {
        pl->uses_pool = 1;
        ++g_pool_plans[dev];
    }
    return g_pool[dev];
}

void *captured_block(irc_plan *pl, size_t bytes)
{
    std::lock_guard<std::mutex> lk(g_pool_mu);
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
        cudaMemPool_t pool = pool_of(pl);
        if (!pool || cudaMallocFromPoolAsync(&base, bytes, pool, s) != cudaSuccess) {
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
// make first.  Microseconds, plain -> proven (EXACT | REF | REF delta):
//     1,000 spikes, one chunk, D = 24 (1.0e6 pairs)    55 -> 74  |  75 -> 73  |  17 -> 86
//     2,048, D = 9 (4.2e6)                             54 -> 76  |  74 -> 77  |  17 -> 87
//     2,048, D = 24                                    78 -> 79  |  82 -> 79  |  25 -> 99
//     2,048, D = 45                                   118 -> 88  |  98 -> 85  |  40 -> 108
//     4,000, D = 9 (1.6e7)                             94 -> 89  | 156 -> 92  |  41 -> 97
//     5,000, D = 24 (2.5e7)                           264 -> 99  | 309 -> 104 | 143 -> 118
//     4,000, 200 chunks (1.2e6, 400 tiles)             86 -> 89  | 172 -> 89  |  31 -> 101
//     10,000, 400 chunks (3.8e6, 800 tiles)           144 -> 90  | 383 -> 98  |  55 -> 105
//     20,000, 1,200 chunks (5.0e6, 2,400 tiles)       266 -> 109 | 725 -> 123 | 107 -> 125
// Tiles alone count only where a window is likely to hold knn candidates.
enum class Form { exact, ref, ref_delta };

bool serves(const irc_plan *pl, int nC, Form f)
{
    if (!pl->runs_ascend || !pl->disjoint || nC + 6 > irc_tc::KP) return false;
    const long long work = f == Form::exact ? 100000000 : f == Form::ref ? 20000000 : 500000000;
    const int tiles = f == Form::exact ? 500 : f == Form::ref ? 150 : 4000;
    return pl->pairs * nC >= work ||
           (pl->ntiles[irc::tile_slot(kTile)] >= tiles && pl->pairs >= 64LL * pl->dev.n_out);
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
    if (!pl->uses_pool) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (--g_pool_plans[pl->device] == 0 && g_pool[pl->device]) cudaMemPoolTrimTo(g_pool[pl->device], 0);
}

int irc_cert_site_knn(irc_plan *pl, const float *F, int nC, int knn, int nThreads, int mode, float *vrKnn, float *rho,
                      int32_t *miKnn, float *d2Knn, cudaStream_t s)
{
    if (!serves(pl, nC, mode == IRC_MODE_EXACT ? Form::exact : Form::ref) || knn > irc_tc::KNN_MAX) return IRC_CERT_PASS;
    const int tiles = pl->ntiles[irc::tile_slot(kTile)];
    const size_t flags = up((size_t)tiles * 4), queue = up((size_t)tiles * 4);
    const size_t ovf = mode == IRC_MODE_EXACT ? up((size_t)pl->dev.n_out * 4) : 0, more = flags + queue + ovf;
    Work w(pl, lists_bytes(pl, nC, more), s);
    if (!w.base) return IRC_CERT_PASS;
    Lists L;
    int rc = make_lists(pl, F, nC, (char *)w.base, more, flags, &L, s);
    if (rc != IRC_OK) return rc;
    L.c.tile_flag = (int *)L.more;
    L.c.tile_queue = (int *)(L.more + flags);
    const unsigned grid = (unsigned)((pl->dev.n_out + kWarps - 1) / kWarps);
    if (mode == IRC_MODE_EXACT)
        launch_next(k_cert_knn<false>, grid, 32 * kWarps, 0, s, L.c, knn, 1, vrKnn, rho, miKnn, d2Knn);
    else
        launch_next(k_cert_knn<true>, grid, 32 * kWarps, 0, s, L.c, knn, nThreads, vrKnn, rho, miKnn, nullptr);
    IRC_CHECK_LAUNCH("irc_site_knn lists");
    const irc::TileQueue tq{L.c.tile_queue, L.c.words + W_TILES, L.c.words + W_ERR, tiles};
    if (mode == IRC_MODE_EXACT)
        return irc_exact_tiles(pl, F, nC, knn, vrKnn, rho, miKnn, d2Knn, tq, L.c.words + W_OVF,
                               (int *)(L.more + flags + queue), s);
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
