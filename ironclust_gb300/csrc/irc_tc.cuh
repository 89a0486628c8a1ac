// irc_tc.cuh -- shared constants of the tensor-core kNN (internal).
#pragma once
#include <cuda.h>

#include "irc_plan.cuh"

namespace irc_tc {

constexpr int BM = 128;          // queries per CTA (TMEM lanes)
constexpr int KP = 64;           // padded feature dimension (bf16 elements, one 128-byte row)
constexpr int KNN_MAX = 32;      // largest knn served (candidate lists hold >= 64 for the re-rank)
constexpr int LIST_MAX = 256;    // longest candidate list re-ranked (else: the exact fallback)
constexpr int LIST_AVG = 128;    // list area per plan: LIST_AVG entries per query
using TcItem = irc::TcItem;

// Operand formats of the filter (128-byte rows in all of them).  f16: the
// BF16 row layout in half precision, the features scaled by a power of two to
// about 8 in magnitude at most; 8 times BF16's resolution at the same MMA cost, so
// that a query's candidate list can be proven complete (irc_cert.cu).
enum class Fmt : int { bf16 = 0, fp8 = 1, f16 = 2 };

// f16: the longest scaled row (squared) whose norm the operand rows can hold
// (half precision ends at 65,504).
constexpr float F16_NORM2 = 60000.0f;
// f16: distances up to here are listed whenever the threshold says so (the
// threshold in the operand rows ends at 60,000).
constexpr float F16_TAU_MAX = 59900.0f;

// The re-rank's FP32 copy of a feature row, zero-padded to a multiple of 8
// floats (32 bytes) so that it is read with whole-sector 256-bit loads:
// width in float4.
inline __host__ __device__ int fp_row4(int nC) { return 2 * ((nC + 7) / 8); }

// Items that do not fill a turn of the machine, split over their candidates:
// `items` of them (the last one-slot ones) in `parts` pieces each, one piece per
// CTA, one launch per pass.  colmin: the per-column minima of every item,
// [items][128 columns][128 queries] (bits); cnt: list lengths, [items][128];
// area: where the items' list rows (LIST_ROW entries a query) begin in lists.
constexpr int LIST_ROW = 192;
struct SplitOut {
    int items, parts;
    int *colmin, *cnt;
    unsigned area;
};

// Candidate lists handed from the filter kernel to the re-rank kernel:
// qinfo[o] = (offset into lists, length) of query q_base + o, or (-1, -1);
// lists packed by a bump allocator (count) of cap entries.
struct ListOut {
    int2 *qinfo;
    uint32_t *lists;
    unsigned *count;             // count[0]: list entries used; count[1..3]: work-queue heads of the
    unsigned cap;                // filter's one-, two- and four-slot launches
    int2 *cert;                  // per query (threshold bits, chunk), or null when nobody asks
    SplitOut split;
};

// Entries of the list area of a plan with n_out queries (offsets are int32).
inline size_t list_cap(long long n_out)
{
    const size_t c = (size_t)n_out * LIST_AVG, m = (size_t)0x7fffff00;
    return c < m ? c : m;
}

// Bytes of the list area of a plan with n_out queries (qinfo, the count and
// the filter's three work-queue counters in one 256-byte block, lists).
inline size_t list_area_bytes(long long n_out)
{
    return (((size_t)n_out * 8 + 255) & ~(size_t)255) + 256 + list_cap(n_out) * 4;
}

inline ListOut list_area(void *base, long long n_out)
{
    ListOut lo;
    char *b = (char *)base;
    lo.qinfo = (int2 *)b;
    b += ((size_t)n_out * 8 + 255) & ~(size_t)255;
    lo.count = (unsigned *)b;
    lo.lists = (uint32_t *)(b + 256);
    lo.cap = (unsigned)list_cap(n_out);
    lo.cert = nullptr;
    lo.split = SplitOut{};
    return lo;
}

// Memory of the split items (0: none), the most that any layout, width or form
// of the plan takes (a buffer that the plan keeps has room for it: it is not
// allocated again, and captured graphs that use it stay valid), and its place
// in lo: behind lo.lists, in the same allocation.
size_t split_bytes(const irc_plan *pl, int nC, Fmt fmt);
size_t split_reserve(const irc_plan *pl);
void split_area(const irc_plan *pl, int nC, Fmt fmt, void *mem, ListOut *lo);

// The filter (one persistent launch per packing class: items of one or two
// slots on 256-candidate units, four-slot items on 128-candidate units; mc is
// the candidate-row map with 128-row boxes) and the re-rank, on stream s.
int launch_knn_tc(Fmt fmt, const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, const float *F,
                  const float4 *Fp, int nC, int knn, float *vrKnn, float *rho, int32_t *miKnn, float *d2Knn,
                  const ListOut &lo, cudaStream_t s);

// What the filter expects cleared (before the operands are made: nothing then
// stands between the kernels).
cudaError_t clear_lists(const ListOut &lo, int n_out, cudaStream_t s);

// The filter alone; scratch: the counter words of its overflow queue and error
// word (irc_plan.cuh), the queue after them (unused when lo.cert is set).
int launch_filters(Fmt fmt, const CUtensorMap &mq, const CUtensorMap &mc, irc_plan *pl, int nC, const ListOut &lo,
                   int *scratch, cudaStream_t s);

// Operand rows of the plan's rows of F and the tensor maps over them
// (irc_tc_host.cu); buf: ops_bytes(...) of device memory.
struct Operands {
    CUtensorMap mq, mc;
    const float4 *fp;            // padded FP32 rows of the re-rank
    const float *scale;          // f16: the power of two the features were scaled by
    const float *qnorm;          // f16: upper bound of every query's scaled norm, [n_out]
};
size_t ops_bytes(const irc_plan *pl, int nC, Fmt fmt);
// amax (fp8): the largest magnitude, zero before; ticket: zero.
int make_operands(Fmt fmt, irc_plan *pl, const float *F, int nC, void *buf, unsigned *amax, unsigned *ticket,
                  Operands *out, cudaStream_t s);

}  // namespace irc_tc
