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

// A thread that lowered the attribute for a smaller launch between another
// thread's setting and launch made that launch fail, so it only ever rises.
cudaError_t allow_smem(const void* fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::tuple<int, unsigned long long, const void*>, size_t> allowed;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const auto at = allowed.try_emplace(std::make_tuple(dev, current_ctx_id(), fn), 0);
    size_t& now = at.first->second;
    if (at.second) {
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess) now = (size_t)fa.maxDynamicSharedSizeBytes;
        else cudaGetLastError();
    }
    if (bytes <= now) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) now = bytes;
    else cudaGetLastError();
    return e;
}

}  // namespace plk
