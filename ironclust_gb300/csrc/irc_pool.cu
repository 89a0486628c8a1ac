// irc_pool.cu -- scratch of the calls that have no plan to keep it (cluster
// assignment, drift linkage, drop-in checks, conversions).
//
// One pool per device, its blocks handed out in stream order, so calls on any
// stream or thread are independent.  It keeps at most kKeep bytes between
// calls and gives them back when the device's last plan is destroyed.  The
// device's default pool gives everything back at the next synchronisation: a
// drift linkage of 1,000,000 spikes spent 290 of 470 us mapping its 3 MB again.
#include <mutex>

#include "irc_common.cuh"
#include "irc_plan.cuh"

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKeep = 64ull << 20;
std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices];
int g_plans[kMaxDevices];

}  // namespace

cudaError_t irc_scratch_alloc(void **p, size_t bytes, cudaStream_t s)
{
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < kMaxDevices) {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_pool[dev]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            irc_host::Uncaptured mode;
            if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
                unsigned long long keep = kKeep;
                cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
                g_pool[dev] = pool;
            } else {
                cudaGetLastError();
            }
        }
        pool = g_pool[dev];
    }
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

void irc_scratch_plan(int dev, int change)
{
    if (dev < 0 || dev >= kMaxDevices) return;
    std::lock_guard<std::mutex> lk(g_mu);
    g_plans[dev] += change;
    if (change < 0 && g_plans[dev] == 0 && g_pool[dev]) cudaMemPoolTrimTo(g_pool[dev], 0);
}
