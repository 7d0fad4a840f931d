// down_any_kernel (plk_prune_any.cuh), float, 2 to 12 states.
#include "plk_prune_any.cuh"

namespace plk {

cudaError_t launch_down32_lo(const PreorderArgs& a, int S, int H, const dev::AnyLaunch& p, int blocks, cudaStream_t st) {
    switch (S) {
        PLK_ANY_LO(float)
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace plk
