// prune4w: the 4-state FP32 post-order pass (src/simpleML.cpp:127-197) with
// every warp on its own sites, SPT sites per thread, and nothing staged.
//
// The staged forms (prune4s, prune4p) copy each op's P(t) rows and tip
// tables into shared memory and hold the CTA at a barrier per op; on the
// 128-taxon x 100,000-site benchmark that staging, the barrier and the
// generic op decoding cost more instructions than the arithmetic itself.
// Here a warp walks the op list alone, over 32 x SPT sites:
//  * a thread carries SPT adjacent sites (SPT lane + s of the warp's tile),
//    so every P(t) row it loads feeds the products of SPT sites, the SPT
//    sites' independent products hide the latency of the next loads, and one
//    load of SPT bytes brings a child's tip codes for all of them;
//  * TS = 1 (trees whose tables fit): the CTA first brings the paired tables
//    and the op list into shared memory with bulk copies (cp.async.bulk on
//    one mbarrier, a bounded wait) and reads them there;
//  * TS = 2 (any tree): the tables stream through a shared-memory ring in the
//    order of the ops that read them, one bulk copy a stage of several ops,
//    read by all warps of the CTA (RingTables, plk_prune4w.cuh).  Before it
//    such trees had the staged forms, a barrier and a cp.async loop per op:
//    501 taxa x 299,999 sites, C = 4, 1,507 -> 857 us;
//  * spilled vectors sit in tensor memory (tcgen05.st / tcgen05.ld, one
//    instruction per category pair and op), not in shared memory;
//  * the tip codes come three ops ahead into a per-warp ring in shared memory;
//  * every branch on the op's shape is uniform across the warp, and no CTA
//    barrier stands between ops; one CTA per SM, its warp count chosen per
//    launch so that every warp has a tile;
//  * the rescale test first takes the maximum of one category pair; only when
//    a lane of the warp falls below the threshold does the warp take the full
//    maximum (the same decision and factors);
//  * a streamed alignment's codes land while the pass runs: a warp waits
//    (bounded) for its tile's chunk flag before its walk, with TS = 2 the CTA's
//    warps together before a round of tiles;
//  * the launch overlaps the P(t) kernel before it (programmatic stream
//    serialization; griddepcontrol.wait before any read of its tables).
// The arithmetic is run_tile4p's (plk_prune4p.cuh) in the same order -- every
// product, rescale and root sum on fma.rn.f32x2 / mul.rn.f32x2 lanes -- so the
// per-site results are the bits of prune4s and prune4p; the sites' sum is the
// FP32 record epilogue of every FP32 form (block_sum_site32f).
#include "plk_prune4w.cuh"

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

namespace plk {
using namespace dev;
using namespace dev4w;

int device_sm_count() {
    static std::atomic<int> n{0};
    int v = n.load();
    if (v > 0) return v;
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0) c = 1;
    n.store(c);
    return c;
}

namespace {

constexpr int kWMinWarps = 4;
constexpr int kWMaxWarps = 24;
constexpr uint32_t kWChunk = 16384;  // bytes per bulk copy of the TS = 1 prologue

// One CTA per SM (the launch keeps the occupancy at one), blockDim.x / 32
// warps, each walking warp tiles of 32 SPT sites g, g + T, ... with g = warp
// x gridDim.x + blockIdx.x and T the grid's warps, so that the tiles of a
// last, partial round fall on every SM alike.  tmem_cols: the CTA's TMEM
// allocation (a power of two >= 32 holding every warp's stack).
// TS = 1: the CTA first copies the tree's paired P(t) and tip tables into
// shared memory and reads them there (trees whose tables fit); Pp, Tp are those
// tables.  TS = 2: the tables stream through a ring, once a round of tiles; Pp
// is the stream.
// TPS = 2: the two lanes 2i, 2i + 1 share sites, each holding half of the
// category pairs (they exchange their maxima for the rescale, and the even
// lane adds up the root in category order, so the bits are those of TPS = 1);
// a warp tile is 16 x SPT sites.
template <int KP, int SPT, int TS, int TPS>
__global__ void __maxnreg__(prune4w_maxnreg(KP, SPT, TPS, TS)) prune4w_kernel(PruneArgs a, const float* __restrict__ Pp,
                                                                          const float* __restrict__ Tp, int tmem_cols, int levels, int code_at,
                                                                          int over_at, int ops_smem) {
    // the kernel before this one in the stream (P(t), which writes the
    // tables) has completed and its writes are visible
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    constexpr int NC = 8 * SPT;     // TMEM columns of one category pair of a slot
    constexpr int KPT = KP / TPS;   // category pairs per thread
    constexpr int WS = 32 / TPS;    // sites per warp and site index s
    __shared__ uint32_t s_tmem;
    const int nthr = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = TPS == 2 ? (lane & 1) : 0;
    const int q0 = half * KPT;      // this thread's first pair
    const int n_wtiles = (a.n_sites + WS * SPT - 1) / (WS * SPT);
    const int total_warps = (nthr >> 5) * gridDim.x;
    extern __shared__ __align__(16) unsigned char wtab[];
    __shared__ __align__(8) uint64_t s_bar;
    const uint32_t smem0 = static_cast<uint32_t>(__cvta_generic_to_shared(wtab));
    typename std::conditional<TS == 1, SmemTables<KP>, RingTables<KP>>::type tab;
    if constexpr (TS == 1) {
        // [P(t) of every node][tip tables of every tip][ops] by bulk copies
        // (cp.async.bulk, 16-byte aligned, sizes multiples of 16) that one
        // thread issues in chunks, completing on one mbarrier; the TMEM
        // allocation below overlaps them
        const uint32_t pb = (uint32_t)a.n_nodes * KP * 128, tb = (uint32_t)a.n_tips * KP * 512;
        const uint32_t ob = (uint32_t)a.n_ops * (uint32_t)sizeof(Op);
        const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(&s_bar));
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(pb + tb + ob)
                         : "memory");
            if (!a.withhold_first_stage) {
                const unsigned char* src[3] = {reinterpret_cast<const unsigned char*>(Pp),
                                               reinterpret_cast<const unsigned char*>(Tp),
                                               reinterpret_cast<const unsigned char*>(a.ops)};
                const uint32_t len[3] = {pb, tb, ob};
                uint32_t dst = smem0;
                for (int k = 0; k < 3; ++k) {
                    for (uint32_t off = 0; off < len[k]; off += kWChunk) {
                        const uint32_t n = min(kWChunk, len[k] - off);
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                                dst + off),
                            "l"(src[k] + off), "r"(n), "r"(bar)
                            : "memory");
                    }
                    dst += len[k];
                }
            }
        }
        tab.P = smem0;
        tab.T = smem0 + pb;
        tab.ops = smem0 + pb + tb;
    } else {
        // [control][ring][ops, where they fit]
        ring_init(tab, smem0, smem0 + kRingCtlBytes, tid == 0);
        tab.ops = a.sops;
        if (ops_smem) {
            int4* d = reinterpret_cast<int4*>(wtab + kRingCtlBytes + kRingSlots * RingTables<KP>::kSlotBytes);
            for (int i = tid; i < a.n_ops * 2; i += nthr) d[i] = __ldg(reinterpret_cast<const int4*>(a.sops) + i);
            tab.ops = reinterpret_cast<const Op*>(d);
        }
        tab.stages = a.stages;
        tab.stream = Pp;
        tab.n_stages = a.n_stages;
        tab.warps = nthr >> 5;
        tab.withhold = a.withhold_first_stage;
    }
    const int n_ops = a.n_ops;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_tmem))),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // TS = 1: the tables have landed (a bounded wait; one that runs out
    // leaves this warp's sums NaN, so the evaluation reports a non-finite
    // value, after a second bounded wait for copies still in flight)
    bool tables_ok = true;
    if constexpr (TS == 1) {
        const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(&s_bar));
        tables_ok = __all_sync(0xffffffffu, mbar_try_wait_bounded(bar, 0));
        if (!tables_ok && !a.withhold_first_stage) mbar_try_wait_bounded(bar, 0);
    }
    // this warp's stack: its lanes, its column range
    const uint32_t tstack =
        s_tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * levels * KPT * NC);
    const uint32_t over = smem0 + (uint32_t)(over_at + warp * max(a.max_depth - levels, 0) * KPT * NC * 128 + lane * 4);
    SiteSum32 sum;
    const int stride = a.site_stride;
    if (!tables_ok) site_sum_add(sum, __int_as_float(0x7fc00000), 0);
    const int rounds = (n_wtiles + total_warps - 1) / total_warps;
    for (int round = 0; tables_ok && round < rounds; ++round) {
        const int wtile = warp * gridDim.x + blockIdx.x + round * total_warps;
        bool sites = wtile < n_wtiles;
        if (TS == 1 && !sites) break;
        if (sites && a.arrive) {  // a streamed alignment: this tile's chunk of codes first (the test hook withholds it)
            const int want = a.withhold_arrival ? (a.arrive_gen ^ 0x40000000) : a.arrive_gen;
            if (!wait_arrival(a.arrive + (wtile * WS * SPT) / a.chunk_sites, want)) {
                site_sum_add(sum, __int_as_float(0x7fc00000), 0);  // NaN: the evaluation reports a numeric error
                sites = false;
            }
        }
        if constexpr (TS == 2) {
            // every slot is free again, and every warp has its tile's codes (a warp
            // that still waited for them would hold up the ring, whose waits have
            // a bound of their own): the tree's first stages
            if (round > 0 || a.arrive) __syncthreads();
            if (tid == 0) tab.start();
        }
        if (!sites) {
            if constexpr (TS == 2) tab.skip();
            continue;
        }
        const int base = wtile * WS * SPT + (TPS == 2 ? lane >> 1 : lane) * SPT;  // site s: base + s
        f2 acc[SPT][KPT][4];
        int scale_e[SPT];
        std::conditional_t<TS == 2, CodeRing<SPT, TPS>, CodeRegs<SPT>> codes;
        if constexpr (TS == 2) {
            codes.sm = smem0 + (uint32_t)(code_at + warp * CodeRing<SPT, TPS>::kBytes);
            codes.codes = a.codes, codes.first = wtile * WS * SPT;
        } else {
            codes.colp = a.codes + min(base, stride - SPT);
        }
        codes.stride = stride;
        walk4w<KP, SPT, TPS>(tab, n_ops, codes, tstack, levels, over, q0, acc, scale_e);
        if constexpr (TS == 2) {
            if (!__all_sync(0xffffffffu, tab.ok)) {  // a stage did not arrive
                site_sum_add(sum, __int_as_float(0x7fc00000), 0);
                continue;
            }
        }
        root4w<KP, SPT, TPS>(acc, scale_e, base, a.n_sites, half == 0, a.root_w, a.cat_w, a.C, a.site_lnl, sum);
    }
    // every warp is done with its stack (its stores complete): free the TMEM
    tmem_wait_st();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s_tmem), "r"(tmem_cols)
                     : "memory");
    }
    const SiteSum32 bsum = block_sum_site32f(sum);
    if (tid == 0) store_site_record(a.block_sum, blockIdx.x, bsum);
    if (a.grid_done) finish_grid_sum32(a.block_sum, a.grid_done, a.lnl_out);
}

template <int KP, int SPT, int TS, int TPS = 1>
const void* prune4w_fn() {
    return reinterpret_cast<const void*>(prune4w_kernel<KP, SPT, TS, TPS>);
}

const void* prune4w_fn_of(int KP, int SPT, int TS, int TPS = 1) {
    if (TPS == 2) return KP == 2 ? prune4w_fn<2, 2, 1, 2>() : prune4w_fn<4, 2, 1, 2>();
    if (TS == 1) {
        switch (KP * 10 + SPT) {
            case 11: return prune4w_fn<1, 1, 1>();
            case 12: return prune4w_fn<1, 2, 1>();
            case 14: return prune4w_fn<1, 4, 1>();
            case 21: return prune4w_fn<2, 1, 1>();
            case 22: return prune4w_fn<2, 2, 1>();
            case 24: return prune4w_fn<2, 4, 1>();
            case 41: return prune4w_fn<4, 1, 1>();
            default: return prune4w_fn<4, 2, 1>();
        }
    }
    switch (KP * 10 + SPT) {
        case 11: return prune4w_fn<1, 1, 2>();
        case 12: return prune4w_fn<1, 2, 2>();
        case 14: return prune4w_fn<1, 4, 2>();
        case 21: return prune4w_fn<2, 1, 2>();
        case 22: return prune4w_fn<2, 2, 2>();
        case 24: return prune4w_fn<2, 4, 2>();
        case 31: return prune4w_fn<3, 1, 2>();
        case 32: return prune4w_fn<3, 2, 2>();
        case 41: return prune4w_fn<4, 1, 2>();
        default: return prune4w_fn<4, 2, 2>();
    }
}

// shared memory of the TS = 1 form: the tree's paired tables
size_t prune4w_table_bytes(const PruneArgs& a) {
    return (size_t)a.n_nodes * (a.C / 2) * 128 + (size_t)a.n_tips * (a.C / 2) * 512 + (size_t)a.n_ops * sizeof(Op);
}
constexpr size_t kWMaxTable = kMaxSmem - 8 * 1024;
// a warp's code ring
int prune4w_code_bytes(int ts, int spt, int tps) { return ts == 2 ? 4 * 2 * (32 / tps * spt) : 0; }
// TS = 2: ops in shared memory up to this size
constexpr size_t kWMaxOps = 96 * 1024;

// TMEM columns a CTA of `warps` warps needs for stacks of `levels` slots: the
// warps sharing a lane quarter stack their column ranges; a power of two of
// at least 32 (0: more than the 512 an SM has)
int prune4w_tmem_cols(int KP, int SPT, int warps, int levels, int TPS = 1) {
    const int need = ((warps + 3) / 4) * (levels > 0 ? levels : 1) * (KP / TPS) * 8 * SPT;
    int cols = 32;
    while (cols < need) cols *= 2;
    return cols <= 512 ? cols : 0;
}

// The stack slots a warp has in the TMEM (all `depth` where they fit), and the
// bytes of shared memory for a warp's others.  The streamed form alone has
// shared memory left for those: its CTA may then have the warps that its
// registers allow (501 taxa, a stack of 5, 2 sites x 2 pairs a thread: 16
// instead of 12, 1021 -> 857 us over 299,999 sites).
int prune4w_levels(int KP, int SPT, int TS, int warps, int depth, int TPS) {
    depth = depth > 0 ? depth : 1;
    const int fit = 512 / (((warps + 3) / 4) * (KP / TPS) * 8 * SPT);
    return fit >= depth ? depth : (TS == 2 ? fit : 0);
}
size_t prune4w_over_bytes(int KP, int SPT, int levels, int depth, int TPS) {
    return depth > levels ? (size_t)(depth - levels) * (KP / TPS) * 8 * SPT * 128 : 0;
}

// resident CTAs per SM with `warps` warps and `smem` bytes (occupancy
// calculator, cached per device, context and kernel: the launch runs every
// evaluation)
int prune4w_ctas_per_sm(int KP, int SPT, int TS, int warps, size_t smem, int TPS = 1) {
    const void* fn = prune4w_fn_of(KP, SPT, TS, TPS);
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long ctx = current_ctx_id();  // a device reset starts the caches over
    static std::mutex mu;
    static std::map<std::tuple<int, unsigned long long, const void*, int, size_t>, int> occ;
    if (allow_smem(fn, smem) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(dev, ctx, fn, warps, smem);
    const auto it = occ.find(key);
    if (it != occ.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, warps * 32, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    occ[key] = n;
    return n;
}

// warps per CTA: enough that every SM's CTA has a tile per warp where the
// tiles allow, at most what keeps the stacks within the TMEM and the
// registers (and, for TS = 1, the tables) within one CTA per SM (0: no size
// works)
int prune4w_warps(int KP, int SPT, int TS, int TPS, size_t smem, int depth, int tiles, int sms) {
    int hi = 0;
    const size_t limit = smem_limit(prune4w_fn_of(KP, SPT, TS, TPS));
    for (int w = kWMaxWarps; w >= kWMinWarps; --w) {
        const int levels = prune4w_levels(KP, SPT, TS, w, depth, TPS);
        const size_t warp_bytes = prune4w_code_bytes(TS, SPT, TPS) + prune4w_over_bytes(KP, SPT, levels, depth, TPS);
        if (levels > 0 && smem + w * warp_bytes <= limit &&
            prune4w_ctas_per_sm(KP, SPT, TS, w, smem + w * warp_bytes, TPS) >= 1) {
            hi = w;
            break;
        }
    }
    if (hi == 0) return 0;
    const int want = (tiles + sms - 1) / sms;
    // TS = 2 walks its rounds in step: the warps that divide the tiles into the
    // fewest rounds evenly
    if (TS == 2 && want > hi) {
        const int rounds = (want + hi - 1) / hi;
        return std::max(kWMinWarps, (want + rounds - 1) / rounds);
    }
    return std::max(kWMinWarps, std::min(hi, want));
}

}  // namespace

bool prune4w_fits(const PruneArgs& a, int spt, int ts, int tps) {
    if (spt != 1 && spt != 2 && spt != 4) return false;
    if (ts == 2) {  // any number of categories, an odd last one paired with itself
        const int KP = (a.C + 1) / 2;
        return tps == 1 && a.C >= 1 && a.C <= 8 && !(spt == 4 && KP > 2) && a.n_stages > 0 &&
               prune4w_tmem_cols(KP, spt, kWMinWarps, a.max_depth) > 0;
    }
    if (a.C != 2 && a.C != 4 && a.C != 8) return false;
    if (tps == 2 && (a.C == 2 || spt != 2)) return false;  // instantiated: two sites
    if (tps == 2)
        return prune4w_table_bytes(a) <= kWMaxTable && prune4w_tmem_cols(a.C / 2, spt, kWMinWarps, a.max_depth, 2) > 0;
    if (spt == 4 && a.C == 8) return false;  // four sites of 8 categories exceed the registers
    if (prune4w_table_bytes(a) > kWMaxTable) return false;
    return prune4w_tmem_cols(a.C / 2, spt, kWMinWarps, a.max_depth) > 0;
}

cudaError_t launch_prune4w(const PruneArgs& a, int spt, int ts, int tps, int* n_blocks, cudaStream_t st) {
    if (!prune4w_fits(a, spt, ts, tps) || (ts == 1 ? a.scratch == nullptr : a.stream == nullptr)) return cudaErrorInvalidValue;
    const int KP = (a.C + 1) / 2;
    float *Pp, *Tp = nullptr;
    if (ts == 1) {
        prune4p_scratch_parts(a.scratch, a.n_nodes, a.C, &Pp, &Tp);
        if (!a.paired_ready) {
            cudaError_t e = launch_relayout4p(a, Pp, Tp, st);
            if (e != cudaSuccess) return e;
        }
    } else {
        Pp = a.stream;
        if (!a.stream_ready) {
            cudaError_t e = launch_relayout_stream(a, st);
            if (e != cudaSuccess) return e;
        }
    }
    const size_t op_bytes = (size_t)a.n_ops * sizeof(Op);
    const int ops_smem = ts == 2 && op_bytes <= kWMaxOps;
    const size_t tables = ts == 1 ? (prune4w_table_bytes(a) + 15) / 16 * 16
                                  : kRingCtlBytes + (size_t)kRingSlots * kStageUnits * KP * 128 + (ops_smem ? op_bytes : 0);
    const int ws = 32 / tps * spt;  // sites per warp tile
    const int tiles = (a.n_sites + ws - 1) / ws;
    const int sms = device_sm_count();
    const int warps = prune4w_warps(KP, spt, ts, tps, tables, a.max_depth, tiles, sms);
    if (warps == 0) return cudaErrorInvalidConfiguration;
    const int levels = prune4w_levels(KP, spt, ts, warps, a.max_depth, tps);
    const int tmem_cols = prune4w_tmem_cols(KP, spt, warps, levels, tps);
    const int blocks = std::max(1, std::min(sms, (tiles + warps - 1) / warps));
    *n_blocks = blocks;
    // launched with programmatic stream serialization: the CTAs may be
    // scheduled while the P(t) kernel before them finishes (it lets its
    // dependents launch at its start); the kernel waits for it
    // (griddepcontrol.wait) before reading anything it wrote
    // (after a relayout of this call's own the kernel before is not P(t), and
    // completes first all the same)
    const void* fn = prune4w_fn_of(KP, spt, ts, tps);
    PruneArgs args_a = a;
    const float* args_p = Pp;
    const float* args_t = Tp;
    // beside the tables: the warps' code rings, the stacks' slots above the TMEM
    const size_t codes_at = tables, over_at = tables + (size_t)warps * prune4w_code_bytes(ts, spt, tps);
    const size_t smem = over_at + (size_t)warps * prune4w_over_bytes(KP, spt, levels, a.max_depth, tps);
    int args_cols = tmem_cols, args_levels = levels, args_codes = (int)codes_at, args_over = (int)over_at, args_ops = ops_smem;
    if (prune4w_ctas_per_sm(KP, spt, ts, warps, smem, tps) < 1) return cudaErrorInvalidConfiguration;
    void* args[] = {&args_a, &args_p, &args_t, &args_cols, &args_levels, &args_codes, &args_over, &args_ops};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace plk
