// irc_pool.cu -- stream-ordered scratch of the calls: small scratch (cluster
// assignment, drift linkage, drop-in checks, conversions) and the working memory
// of the proven searches.
//
// One pool of each kind per device, its blocks handed out in stream order, so
// calls on any stream or thread are independent.  Between calls a pool keeps at
// most 64 MB, or 1/32 of the device's memory for the searches, and gives it back
// when the device's last plan is destroyed.  The device's default pool gives
// everything back at the next synchronisation: a drift linkage of 1,000,000
// spikes spent 290 of 470 us mapping its 3 MB again.
#include <mutex>

#include "irc_common.cuh"
#include "irc_plan.cuh"

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKeep = 64ull << 20;
enum { kSmall, kSearch, kKinds };
std::mutex g_mu;
cudaMemPool_t g_pool[kKinds][kMaxDevices];
int g_plans[kMaxDevices];

// The pool, made on its first use; null if it cannot be.
cudaMemPool_t pool_of(int kind, int dev)
{
    if (dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    cudaMemPool_t &pool = g_pool[kind][dev];
    if (!pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        irc_host::Uncaptured mode;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            pool = nullptr;
            return nullptr;
        }
        unsigned long long keep = kKeep;
        if (kind == kSearch) {
            size_t fr = 0, total = 0;
            if (cudaMemGetInfo(&fr, &total) == cudaSuccess) keep = total / 32;
            else cudaGetLastError();
        }
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    return pool;
}

}  // namespace

cudaError_t irc_scratch_alloc(void **p, size_t bytes, cudaStream_t s)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = pool_of(kSmall, dev);
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

cudaError_t irc_search_alloc(void **p, size_t bytes, int dev, cudaStream_t s)
{
    cudaMemPool_t pool = pool_of(kSearch, dev);
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaErrorMemoryAllocation;
}

void irc_scratch_plan(int dev, int change)
{
    if (dev < 0 || dev >= kMaxDevices) return;
    std::lock_guard<std::mutex> lk(g_mu);
    g_plans[dev] += change;
    if (change < 0 && g_plans[dev] == 0)
        for (int k = 0; k < kKinds; ++k)
            if (g_pool[k][dev]) cudaMemPoolTrimTo(g_pool[k][dev], 0);
}
