// Launch set-up shared by the kernels' host sides.
#include <map>
#include <mutex>
#include <tuple>

#include "plk_internal.h"

namespace plk {

// Asked once per device, context and kernel: a plan is made for every
// evaluation, and the attribute calls cost a microsecond each.
size_t smem_limit(const void* fn) {
    static std::mutex mu;
    static std::map<std::tuple<int, unsigned long long, const void*>, size_t> limits;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    size_t& limit = limits[std::make_tuple(dev, current_ctx_id(), fn)];
    if (limit > 0) return limit;
    int optin = 0;
    cudaFuncAttributes fa{};
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, fn) != cudaSuccess || (size_t)optin <= fa.sharedSizeBytes) {
        cudaGetLastError();
        return 0;
    }
    limit = (size_t)optin - fa.sharedSizeBytes;
    return limit;
}

}  // namespace plk
