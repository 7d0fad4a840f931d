// down_any_kernel (plk_prune_any.cuh), float, 13 to 24 states.
#include "plk_prune_any.cuh"

namespace plk {

cudaError_t launch_down32_hi(const PreorderArgs& a, int S, int H, const dev::AnyLaunch& p, int blocks, cudaStream_t st) {
    switch (S) {
        PLK_ANY_HI(float)
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace plk
