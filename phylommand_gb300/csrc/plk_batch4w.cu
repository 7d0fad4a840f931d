// batch_prune4w_kernel: the batch's post-order pass with streamed tables.
//
// The staged forms (plk_batch.cu) hold a CTA at a barrier and a cp.async loop
// for every op of its tree.  Here the warps of a CTA walk the op list of their
// work unit (one item's 128 x SPT sites) alone, as prune4w_kernel does
// (plk_prune4w.cuh): the item's tables come through the CTA's shared-memory ring
// in the order of the ops, tip codes through per-warp rings, spilled vectors lie
// in tensor memory.  What bounds it is the issue of the walk and the latency of
// its shared-memory loads, so a unit's four warps form a CTA of their own and
// as many CTAs share an SM as its registers allow (four at 2 sites x 2 pairs a
// thread): another unit's warps fill the gaps at a unit's start and end.  A ring
// has three slots, so that four CTAs' rings, op lists and stack entries fit.
// Measured, 48 items of 8-256 taxa and 200-50,000 sites, C = 4: 850 -> 392 us (two CTAs an SM: 532, three: 428; one site a thread, five: 540).
//
// Per-site values are the bits of the staged forms (same arithmetic, same order).
#include <algorithm>

#include "plk_batch.h"
#include "plk_prune4w.cuh"

namespace plk {
using namespace dev;
using namespace dev4w;

namespace {

constexpr int kSlots = 3;
constexpr int kUnitWarps = 4;  // of a CTA: a unit is 32 x 4 x SPT sites
constexpr size_t kMaxOpBytes = 16 * 1024;  // op lists up to this size lie in shared memory

// CTAs an SM's registers hold, without spills worth the name.
__host__ __device__ constexpr int ctas_per_sm(int KP, int SPT) {
    return SPT == 1 ? (KP >= 3 ? 4 : 5) : (KP >= 3 ? 2 : 4);
}

template <int KP, int SPT>
__global__ void __launch_bounds__(32 * kUnitWarps, ctas_per_sm(KP, SPT)) batch_prune4w_kernel(BatchDev b, BatchStreamShape sh) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_unit;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t smem0 = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    RingTables<KP, kSlots> tab;
    ring_init(tab, smem0, smem0 + kRingCtlBytes, tid == 0);
    tab.warps = kUnitWarps;
    tab.withhold = 0;
    tab.stream = b.stream;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_tmem))),
                     "r"(sh.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tstack = s_tmem + ((uint32_t)(32 * warp) << 16);
    const uint32_t over =
        smem0 + (uint32_t)(sh.over_at + warp * max(b.max_depth - sh.levels, 0) * KP * 8 * SPT * 128 + lane * 4);
    Op* const s_ops = reinterpret_cast<Op*>(sm + sh.ops_at);
    bool dead = false;  // a stage did not arrive (a bounded wait ran out)
    for (;;) {
        __syncthreads();  // every slot is free, the last unit's ops are no longer read
        if (tid == 0) s_unit = atomicAdd(b.counter, 1);
        __syncthreads();
        const int u = s_unit;
        if (u >= b.n_units) break;
        if (dead) {  // no unit keeps an earlier evaluation's sum
            if (tid == 0) b.unit_sums[2 * u] = b.unit_sums[2 * u + 1] = (double)__int_as_float(0x7fc00000);
            continue;
        }
        const int2 unit = b.units[u];
        const BatchItemDev it = b.items[unit.x];
        const Op* ops = b.sops + it.ops_off;
        tab.stages = b.stages + it.stage_off;
        tab.n_stages = it.n_stages;
        if (tid == 0) tab.start();
        if (sh.ops_in_smem) {
            const int4* g = reinterpret_cast<const int4*>(ops);
            for (int i = tid; i < it.n_ops * 2; i += 32 * kUnitWarps) reinterpret_cast<int4*>(s_ops)[i] = __ldg(g + i);
            ops = s_ops;
            __syncthreads();
        }
        tab.ops = ops;
        SiteSum32 sum;
        const int first = (unit.y * kUnitWarps + warp) * 32 * SPT;  // the warp's first site
        if (first < it.n_sites) {
            f2 acc[SPT][KP][4];
            int scale_e[SPT];
            CodeRing<SPT, 1> codes;
            codes.sm = smem0 + (uint32_t)(sh.codes_at + warp * CodeRing<SPT, 1>::kBytes);
            codes.codes = b.codes + it.codes_off;
            codes.first = first;
            codes.stride = it.site_stride;
            walk4w<KP, SPT, 1>(tab, it.n_ops, codes, tstack, sh.levels, over, 0, acc, scale_e);
            if (tab.ok)
                root4w<KP, SPT, 1>(acc, scale_e, first + lane * SPT, it.n_sites, true, b.model + it.model_off + 36,
                                   b.model + it.model_off + 40 + b.C, b.C, nullptr, sum);
        } else {
            tab.skip();
        }
        if (!tab.ok) site_sum_add(sum, __int_as_float(0x7fc00000), 0);  // a stage did not arrive
        double ts, tc;
        block_sum_site32(sum, ts, tc);
        if (tid == 0) {
            b.unit_sums[2 * u] = ts;
            b.unit_sums[2 * u + 1] = tc;
        }
        dead = __syncthreads_or(!tab.ok) != 0;
    }
    tmem_wait_st();  // every warp is done with its stack: free the TMEM
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s_tmem), "r"(sh.tmem_cols)
                     : "memory");
    }
}

typedef void (*StreamKernel)(BatchDev, BatchStreamShape);

StreamKernel stream_kernel(int C, int spt) {
    switch ((C + 1) / 2 * 10 + spt) {
        case 11: return batch_prune4w_kernel<1, 1>;
        case 12: return batch_prune4w_kernel<1, 2>;
        case 21: return batch_prune4w_kernel<2, 1>;
        case 22: return batch_prune4w_kernel<2, 2>;
        case 31: return batch_prune4w_kernel<3, 1>;
        case 32: return batch_prune4w_kernel<3, 2>;
        case 41: return batch_prune4w_kernel<4, 1>;
        case 42: return batch_prune4w_kernel<4, 2>;
        default: return nullptr;
    }
}

}  // namespace

// The shared and tensor memory of a CTA when per_sm of them share an SM; smem =
// 0 where that many do not fit.  The tensor memory is split evenly, in powers of
// two; stack entries above a CTA's share lie in shared memory.
BatchStreamShape batch_stream_shape(int C, int spt, int max_ops, int max_depth, int per_sm) {
    BatchStreamShape s{};
    const StreamKernel kern = stream_kernel(C, spt);
    if (!kern || per_sm < 1) return s;
    const int KP = (C + 1) / 2, entry = KP * 8 * spt, depth = std::max(max_depth, 1);
    int share = 512;
    while (share * per_sm > 512) share /= 2;
    s.tmem_cols = 32;
    while (s.tmem_cols < std::min(depth * entry, share)) s.tmem_cols *= 2;
    s.levels = std::min(depth, s.tmem_cols / entry);
    if (s.levels < 1 || s.tmem_cols > share) return s;
    const size_t op_bytes = (size_t)max_ops * sizeof(Op);
    s.ops_in_smem = op_bytes <= kMaxOpBytes;
    size_t at = kRingCtlBytes + (size_t)kSlots * kStageUnits * KP * 128;
    s.ops_at = (int)at;
    if (s.ops_in_smem) at += op_bytes;
    s.codes_at = (int)at;
    at += (size_t)kUnitWarps * 4 * 2 * 32 * spt;
    s.over_at = (int)at;
    at += (size_t)kUnitWarps * (depth - s.levels) * entry * 128;
    // counted here: the occupancy calculator gives every kernel that allocates
    // tensor memory one CTA per SM
    int dev = 0, sm_bytes = 0, reserved = 0;
    cudaFuncAttributes fa{};
    if (at > 227 * 1024 || cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&fa, kern) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess ||
        allow_smem(reinterpret_cast<const void*>(kern), at) != cudaSuccess) {
        cudaGetLastError();
        return s;
    }
    const int regs = (fa.numRegs + 7) / 8 * 8 * 32 * kUnitWarps;
    if (per_sm > 65536 / regs || (size_t)per_sm * (at + fa.sharedSizeBytes + reserved + 127) > (size_t)sm_bytes) return s;
    s.smem = at;
    return s;
}

cudaError_t launch_batch_prune4w(const BatchDev& b, const BatchStreamShape& sh, int spt, int grid, cudaStream_t st) {
    const StreamKernel kern = stream_kernel(b.C, spt);
    if (!kern || !b.stream || sh.smem == 0) return cudaErrorInvalidValue;
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), sh.smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, 32 * kUnitWarps, sh.smem, st>>>(b, sh);
    return cudaGetLastError();
}

}  // namespace plk
