// Parts of the warp-independent 4-state FP32 post-order pass (plk_prune4w.cu)
// shared by the single-tree and the batch kernel: the tables' places, the spill
// stack in tensor memory, the walk over the op list and the root.
#pragma once

#include "plk_prune4p.cuh"

namespace plk {
namespace dev4w {
using namespace dev;

// FP32 lane pairs as float2, multiplied on the packed FP32x2 path
// (fma.rn.f32x2 / mul.rn.f32x2 through __ffma2_rn / __fmul2_rn)
typedef float2 f2;
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 pk2(float lo, float hi) { return make_float2(lo, hi); }
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) {
    lo = v.x;
    hi = v.y;
}
// three-input maximum (PTX ISA 8.8+, sm_100+): the same value as two fmaxf
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ void lds_v2(uint32_t addr, f2& a, f2& b) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(a.x), "=f"(a.y), "=f"(b.x), "=f"(b.y) : "r"(addr));
}
__device__ __forceinline__ int4 lds_int4(uint32_t addr) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ int2 lds_int2(uint32_t addr) {
    int2 v;
    asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// Where the paired tables and the ops are read.
//   p_pair(e, q, r): one category pair of a P(t) block, rows j = 0..3, each the
//     pairs of states i = 0..3;
//   tip(e, q, code, out): pair q of the tip table row of a code
//     ([pair][half][code][state in the half][2]);
//   op(o): the op's e0, e1 and s0, s1, push, flag; enter(flag) before its
//     tables are read.
// SmemTables: the whole tree's tables in shared memory (32-bit addresses), e a
// node.  RingTables: the tables of the coming ops in a shared-memory ring, e an
// offset into the op's stage.
template <int KP>
struct SmemTables {
    static constexpr bool kOver = false;  // stack entries above the TMEM's in shared memory
    uint32_t P, T, ops;  // shared-memory addresses
    __device__ __forceinline__ void p_pair(int node, int q, f2 (&r)[4][4]) const {
        const uint32_t b = P + (uint32_t)node * (KP * 128) + q * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            lds_v2(b + j * 32, r[j][0], r[j][1]);
            lds_v2(b + j * 32 + 16, r[j][2], r[j][3]);
        }
    }
    __device__ __forceinline__ void tip(int t, int q, int code, f2 (&out)[4]) const {
        const uint32_t b = T + (uint32_t)t * (KP * 512) + q * 512 + (uint32_t)code * 16;
        lds_v2(b, out[0], out[1]);
        lds_v2(b + 256, out[2], out[3]);
    }
    __device__ __forceinline__ void op(int o, int4& ea, int4& sb) const {
        ea = lds_int4(ops + (uint32_t)o * 32);
        sb = lds_int4(ops + (uint32_t)o * 32 + 16);
    }
    __device__ __forceinline__ int2 sources(int o) const { return lds_int2(ops + (uint32_t)o * 32 + 16); }
    __device__ __forceinline__ void enter(int) {}
    __device__ __forceinline__ void finish() {}
};

// The ring: a tree's P(t) blocks and tip tables lie in memory in the order of
// the ops that read them (stream_program), cut into stages of whole ops; a
// stage is one bulk copy into a slot, completing on the slot's mbarrier.  All
// warps of a group read it; the last one to leave a slot issues the copy that
// fills it next, so nothing waits for a free slot and no thread is set aside to
// produce.  A wait for a stage is bounded: one that runs out stops further
// copies and leaves ok false, and the caller makes its sites NaN.
constexpr int kRingSlots = 4;      // at most, and where one group has the SM
constexpr int kRingCtlBytes = 64;  // per group: 4 mbarriers, 4 counters, the abort flag

template <int KP, int SLOTS = kRingSlots>
struct RingTables {
    static_assert(SLOTS <= kRingSlots, "the control words hold four slots");
    static constexpr bool kOver = true;  // stack entries above the TMEM's in shared memory
    static constexpr uint32_t kSlotBytes = kStageUnits * KP * 128;
    uint32_t ring, ctl;   // shared-memory addresses of the slots and of the control words
    const Op* ops;        // the stream program (generic: in shared memory where it fits)
    const int2* stages;   // (first unit, units)
    const float* stream;
    int n_stages, warps, withhold;
    int g;                // the stage being read, -1 before the first
    uint32_t base;        // its slot's address
    uint32_t phases;      // parity of every slot's next fill, kept from tree to tree
    bool ok;              // of this lane; a caller that branches on it votes first
    int drain;            // stages that may be in flight after a wait ran out

    __device__ __forceinline__ void issue(int gg) const {  // one thread
        const int2 st = __ldg(stages + gg);
        const uint32_t slot = (uint32_t)gg % SLOTS, bar = ctl + 8 * slot, bytes = (uint32_t)st.y * (KP * 128);
        if (withhold) return;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                ring + slot * kSlotBytes),
            "l"(stream + (size_t)st.x * (KP * 32)), "r"(bytes), "r"(bar)
            : "memory");
    }
    __device__ __forceinline__ void start() const {  // one thread, all slots free
        int stop;
        asm volatile("ld.shared.s32 %0, [%1];\n" : "=r"(stop) : "r"(ctl + 48) : "memory");
        for (int i = 0; !stop && i < SLOTS && i < n_stages; ++i) issue(i);
    }
    __device__ __forceinline__ void release() const {
        const uint32_t cnt = ctl + 32 + 4 * ((uint32_t)g % SLOTS);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
            int old, stop;
            asm volatile("fence.acq_rel.cta;\natom.shared.add.s32 %0, [%1], 1;\n" : "=r"(old) : "r"(cnt) : "memory");
            if (old == warps - 1) {  // every warp has left the slot
                asm volatile("st.shared.s32 [%0], 0;\nfence.acq_rel.cta;\n" ::"r"(cnt) : "memory");
                asm volatile("ld.shared.s32 %0, [%1];\n" : "=r"(stop) : "r"(ctl + 48) : "memory");
                if (!stop && g + SLOTS < n_stages) issue(g + SLOTS);
            }
        }
    }
    __device__ __forceinline__ void enter(int first_of_stage) {
        if (!first_of_stage) return;
        if (g >= 0) release();
        ++g;
        const uint32_t slot = (uint32_t)g % SLOTS, bar = ctl + 8 * slot, par = (phases >> slot) & 1u;
        if (ok && !mbar_try_wait_bounded(bar, par)) {
            ok = false;
            drain = withhold ? 0 : SLOTS;
            asm volatile("st.shared.s32 [%0], 1;\n" ::"r"(ctl + 48) : "memory");
        }
        if (!ok && drain > 0) {  // copies still in flight, this one and those issued ahead
            --drain;
            mbar_try_wait_bounded(bar, par);
        }
        phases ^= 1u << slot;
        base = ring + slot * kSlotBytes;
    }
    __device__ __forceinline__ void finish() {
        if (g >= 0) release();
        g = -1;
    }
    // a warp without sites keeps step with the others
    __device__ __forceinline__ void skip() {
        for (int i = 0; i < n_stages; ++i) enter(1);
        finish();
    }
    __device__ __forceinline__ void p_pair(int e, int q, f2 (&r)[4][4]) const {
        const uint32_t b = base + (uint32_t)e * (KP * 128) + q * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            lds_v2(b + j * 32, r[j][0], r[j][1]);
            lds_v2(b + j * 32 + 16, r[j][2], r[j][3]);
        }
    }
    __device__ __forceinline__ void tip(int e, int q, int code, f2 (&out)[4]) const {
        const uint32_t b = base + (uint32_t)e * (KP * 128) + q * 512 + (uint32_t)code * 16;
        lds_v2(b, out[0], out[1]);
        lds_v2(b + 256, out[2], out[3]);
    }
    __device__ __forceinline__ void op(int o, int4& ea, int4& sb) const {
        ea = *reinterpret_cast<const int4*>(ops + o);
        sb = *(reinterpret_cast<const int4*>(ops + o) + 1);
    }
    __device__ __forceinline__ int2 sources(int o) const { return *reinterpret_cast<const int2*>(&ops[o].s0); }
};

// A group's control words at ctl, its slots at ring; one thread initialises
// them, a barrier of the group follows before their use.
template <int KP, int SLOTS>
__device__ __forceinline__ void ring_init(RingTables<KP, SLOTS>& tab, uint32_t ctl, uint32_t ring, bool leader) {
    if (leader) {
        for (int i = 0; i < kRingSlots; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\nst.shared.s32 [%1], 0;\n" ::"r"(ctl + 8 * i),
                         "r"(ctl + 32 + 4 * i)
                         : "memory");
        asm volatile("st.shared.s32 [%0], 0;\nfence.mbarrier_init.release.cluster;\n" ::"r"(ctl + 48) : "memory");
    }
    tab.ctl = ctl;
    tab.ring = ring;
    tab.g = -1;
    tab.base = ring;
    tab.phases = 0;
    tab.ok = true;
    tab.drain = 0;
}

// out[i] = sum_j r[j][i] x[j], j ascending, the first term a product (the
// order of mv4p)
__device__ __forceinline__ void mv_pair(const f2 (&r)[4][4], const f2 (&x)[4], f2 (&out)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f2 acc = mul2(x[0], r[0][i]);
        acc = fma2(x[1], r[1][i], acc);
        acc = fma2(x[2], r[2][i], acc);
        acc = fma2(x[3], r[3][i], acc);
        out[i] = acc;
    }
}

// ---- the spill stack in tensor memory ------------------------------------
// A spilled slot holds, for every category pair q and every site s of the
// thread, the 4 pairs = 8 32-bit values: 8 x SPT TMEM columns per pair,
// [q][s][8].  Warp w owns TMEM lanes 32 (w % 4) .. + 31 (the lanes a warp may
// access) and, among the warps sharing those lanes, the column range
// (w / 4) x depth x KP x SPT x 8.  N = 8 SPT columns move in one instruction.
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[N]) {
    static_assert(N == 8 || N == 16 || N == 32, "8, 16 or 32 columns");
    if constexpr (N == 8) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr),
                     "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                     : "memory");
    } else if constexpr (N == 16) {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::
                "r"(taddr),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
            "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
            : "memory");
    } else {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
            "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
            "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
            "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
            "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
            : "memory");
    }
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]) {
    static_assert(N == 8 || N == 16 || N == 32, "8, 16 or 32 columns");
    if constexpr (N == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr)
                     : "memory");
    } else if constexpr (N == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr)
            : "memory");
    } else {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
            "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
              "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
              "=r"(r[30]), "=r"(r[31])
            : "r"(taddr)
            : "memory");
    }
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// The arrival of a streamed tile's codes: arrive[c] reaching gen (written by a
// copy after the chunk's copy on the alignment's copy stream).  Every lane
// reads the flag with acquire semantics, so its code loads that follow see
// the chunk.  Bounded: false, for the whole warp, where a lane waited kArriveLimitNs.
constexpr unsigned long long kArriveLimitNs = 2000000000ull;  // 2 s: far above any chunk's copy time
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool lane_arrival(const int* flag, int gen) {
    if (ld_acquire_gpu(flag) == gen) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        __nanosleep(256);
        if (ld_acquire_gpu(flag) == gen) return true;
        if (global_ns() - t0 > kArriveLimitNs) return false;
    }
}
__device__ __forceinline__ bool wait_arrival(const int* flag, int gen) {
    return __all_sync(0xffffffffu, lane_arrival(flag, gen));
}

// this thread's tip codes (SPT adjacent sites, one load of SPT bytes),
// loaded without allocating in L1 (which holds the tables).  Plain (coherent)
// loads, not the read-only path: a streamed alignment's codes land while the
// pass runs (a warp reads its tile's codes only after their arrival flag).
template <int SPT>
__device__ __forceinline__ int ldg_codes_na(const uint8_t* p) {
    if constexpr (SPT == 1) {
        unsigned short v;
        asm volatile("ld.global.L1::no_allocate.u8 %0, [%1];\n" : "=h"(v) : "l"(p));
        return (int)v;
    } else if constexpr (SPT == 2) {
        unsigned short v;
        asm volatile("ld.global.L1::no_allocate.u16 %0, [%1];\n" : "=h"(v) : "l"(p));
        return (int)v;
    } else {
        int v;
        asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];\n" : "=r"(v) : "l"(p));
        return v;
    }
}

// A warp's tip codes: those of the coming ops' tip children, its tile's sites,
// come by cp.async into a ring of four op slots in shared memory, three ops
// ahead.  Held in registers they were waited for when a register moved on to
// the next op: an L2 or DRAM latency an op where the codes do not stay in L2
// (501 taxa x 299,999 sites: 1185 us a pass, with the ring 1021; the
// long-scoreboard stall 3.2 an instruction, with it 1.2).  (A streamed alignment's codes land while the pass runs: a warp
// starts its copies only after their arrival flag.)
template <int SPT, int TPS>
struct CodeRing {
    static constexpr int kTile = 32 / TPS * SPT;  // bytes of a child
    static constexpr int kBytes = 4 * 2 * kTile;  // of a warp
    uint32_t sm;            // the warp's ring
    const uint8_t* codes;   // the alignment's rows
    int stride, first;      // bytes of a row, the tile's first site

    __device__ __forceinline__ void fetch(int o, int2 src) const {
        const int lane = threadIdx.x & 31, c = lane / (kTile / 16), q = lane % (kTile / 16);
        const int tip = c == 0 ? src.x : src.y;
        if (c < 2 && tip >= 0) {
            // a chunk past the row's end: the row's last one (sites past n_sites)
            const uint8_t* from = codes + (size_t)tip * stride + min(first + 16 * q, stride - 16);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm + (o & 3) * 2 * kTile + c * kTile + 16 * q),
                         "l"(from)
                         : "memory");
        }
    }
    // the codes of a child of op o at this thread's SPT adjacent sites
    __device__ __forceinline__ int get(int o, int c) const {
        const uint32_t at = sm + (o & 3) * 2 * kTile + c * kTile + (TPS == 2 ? (threadIdx.x & 31) >> 1 : (threadIdx.x & 31)) * SPT;
        int v;
        if constexpr (SPT == 1) asm volatile("ld.shared.u8 %0, [%1];\n" : "=r"(v) : "r"(at) : "memory");
        else if constexpr (SPT == 2) asm volatile("ld.shared.u16 %0, [%1];\n" : "=r"(v) : "r"(at) : "memory");
        else asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(at) : "memory");
        return v;
    }
    // Codes of ops 0, 1, 2 on their way; then, for o = 0, 1, ..., those of op o.
    template <class Tab>
    __device__ __forceinline__ void start(const Tab& tab, int n_ops) {
        __syncwarp();  // an earlier tile's codes are read
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            if (o < n_ops) fetch(o, tab.sources(o));
            cp_async_commit();
        }
    }
    template <class Tab>
    __device__ __forceinline__ void step(const Tab& tab, int n_ops, int o, int& c0, int& c1) {
        cp_async_wait<2>();
        __syncwarp();  // op o's codes are in every lane's view, op o - 1's slot is free
        if (o + 3 < n_ops) fetch(o + 3, tab.sources(o + 3));
        cp_async_commit();
        c0 = get(o, 0), c1 = get(o, 1);
    }
    __device__ __forceinline__ void next() {}
    __device__ __forceinline__ void finish() { cp_async_wait<0>(); }
};

// The same held in registers, two ops ahead.
template <int SPT>
struct CodeRegs {
    const uint8_t* colp;  // the alignment's rows at this thread's sites
    int stride;
    int a0, a1, b0, b1;   // codes of the ops o, o + 1
    int m0, m1;           // and o + 2, on their way

    template <class Tab>
    __device__ __forceinline__ void load(const Tab& tab, int n_ops, int o, int& c0, int& c1) const {
        c0 = c1 = 0;
        if (o >= n_ops) return;
        const int2 sv = tab.sources(o);
        if (sv.x >= 0) c0 = ldg_codes_na<SPT>(colp + (size_t)sv.x * stride);
        if (sv.y >= 0) c1 = ldg_codes_na<SPT>(colp + (size_t)sv.y * stride);
    }
    template <class Tab>
    __device__ __forceinline__ void start(const Tab& tab, int n_ops) {
        load(tab, n_ops, 0, a0, a1);
        load(tab, n_ops, 1, b0, b1);
    }
    template <class Tab>
    __device__ __forceinline__ void step(const Tab& tab, int n_ops, int o, int& c0, int& c1) {
        load(tab, n_ops, o + 2, m0, m1);
        c0 = a0, c1 = a1;
    }
    __device__ __forceinline__ void next() {
        a0 = b0, a1 = b1;
        b0 = m0, b1 = m1;
    }
    __device__ __forceinline__ void finish() {}
};

// An entry's words in shared memory, [word][lane]: a warp's own, each lane reads
// what it wrote.  at: the entry's first word of this lane.
template <int N>
__device__ __forceinline__ void over_st(uint32_t at, const uint32_t (&w)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(at + 128 * k), "r"(w[k]) : "memory");
}
template <int N>
__device__ __forceinline__ void over_ld(uint32_t at, uint32_t (&w)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w[k]) : "r"(at + 128 * k) : "memory");
}

// The register budget of a thread: one CTA of 32 x warps threads per SM.  The
// streamed form (TS = 2) takes the fewest registers without spills, for warps
// (2 sites x 2 pairs: 16 of them instead of 12); the tree of TS = 1 rarely
// leaves more than 12 warps a tile, and 168 registers keep its loads ahead
// (128 taxa x 100,000 sites: 76 us, at 128 registers 79).
__host__ __device__ constexpr int prune4w_maxnreg(int KP, int SPT, int TPS, int TS) {
    return TPS == 2 ? (KP == 4 ? 168 : 124)
                    : (SPT == 1 ? (KP >= 3 ? 128 : 96)
                                : (SPT == 2 ? (KP >= 3 ? 232 : (KP == 2 && TS == 1 ? 168 : 128)) : (KP == 1 ? 192 : 255)));
}

// Walks the op list over the warp's sites: acc the root's vectors, scale_e the
// sites' exponents.  q0: this thread's first category pair.
//
// tmem_levels: the stack's entries that the warp's TMEM columns hold; the
// entries above them, which a tree needs seldom (its pushes are the fewer the
// higher the entry), lie in shared memory at over ([entry][word][lane]), so that
// the TMEM does not bound the warps of a CTA.
template <int KP, int SPT, int TPS, class Tab, class Codes>
__device__ __forceinline__ void walk4w(Tab& tab, int n_ops, Codes codes, uint32_t tstack, int tmem_levels, uint32_t over, int q0,
                                       f2 (&acc)[SPT][KP / TPS][4], int (&scale_e)[SPT]) {
    constexpr int NC = 8 * SPT;    // TMEM columns of one category pair of a slot
    constexpr int KPT = KP / TPS;  // category pairs per thread
    const f2 one2 = pk2(1.0f, 1.0f);
#pragma unroll
    for (int s = 0; s < SPT; ++s) {
        scale_e[s] = 0;
#pragma unroll
        for (int q = 0; q < KPT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[s][q][i] = one2;
    }
    int sp = 0;
    codes.start(tab, n_ops);
    for (int o = 0; o < n_ops; ++o) {
        int c0, c1;
        codes.step(tab, n_ops, o, c0, c1);
        // the op (32 bytes, 32-byte aligned): node, rank, e0, e1 | s0, s1, push, pad
        int4 oa, ob;
        tab.op(o, oa, ob);
        const int e0 = oa.z, e1 = oa.w, s0 = ob.x, s1 = ob.y, push = ob.z;
        tab.enter(ob.w);
        // the three shapes the op program has (build_program) with their
        // branches taken once per op; anything else (one child) below
        if (s0 >= 0 && s1 >= 0) {  // two tips
#pragma unroll
            for (int q = 0; q < KPT; ++q)
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    f2 d0[4], d1[4];
                    tab.tip(e1, q0 + q, (c1 >> (8 * s)) & (kCodes - 1), d1);
                    tab.tip(e0, q0 + q, (c0 >> (8 * s)) & (kCodes - 1), d0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[i]);
                }
        } else if (s0 == kSrcAcc && s1 >= 0) {  // the running vector and a tip
#pragma unroll
            for (int q = 0; q < KPT; ++q) {
                f2 r[4][4];
                tab.p_pair(e0, q0 + q, r);
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    f2 d0[4], d1[4];
                    tab.tip(e1, q0 + q, (c1 >> (8 * s)) & (kCodes - 1), d1);
                    mv_pair(r, acc[s][q], d0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[i]);
                }
            }
        } else if (s0 == kSrcPop && s1 == kSrcAcc) {  // the popped vector and the running one
            --sp;
            // the popped slot's loads go out first (after the stores of
            // earlier pushes), the running vector's messages cover them
            tmem_wait_st();
            uint32_t w[KPT][NC];
            if (!Tab::kOver || sp < tmem_levels) {
#pragma unroll
                for (int q = 0; q < KPT; ++q) tmem_ld<NC>(tstack + (uint32_t)((sp * KPT + q) * NC), w[q]);
            } else {
#pragma unroll
                for (int q = 0; q < KPT; ++q) over_ld<NC>(over + (uint32_t)(((sp - tmem_levels) * KPT + q) * NC * 128), w[q]);
            }
            f2 d1[SPT][KPT][4];
#pragma unroll
            for (int q = 0; q < KPT; ++q) {
                f2 r[4][4];
                tab.p_pair(e1, q0 + q, r);
#pragma unroll
                for (int s = 0; s < SPT; ++s) mv_pair(r, acc[s][q], d1[s][q]);
            }
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < KPT; ++q)
#pragma unroll
                for (int k = 0; k < NC; ++k) asm volatile("" : "+r"(w[q][k]));  // no use ahead of the wait
#pragma unroll
            for (int q = 0; q < KPT; ++q) {
                f2 r[4][4];
                tab.p_pair(e0, q0 + q, r);
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    f2 x[4], d0[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        x[i] = pk2(__uint_as_float(w[q][8 * s + 2 * i]), __uint_as_float(w[q][8 * s + 2 * i + 1]));
                    mv_pair(r, x, d0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[s][q][i]);
                }
            }
        } else {
            if (s0 == kSrcPop) --sp;
#pragma unroll
            for (int q = 0; q < KPT; ++q) {
                const int qg = q0 + q;  // the pair in the tables
                // the second child's messages first: they read the running
                // vector, which the products then overwrite
                f2 d1[SPT][4];
                if (s1 >= 0) {
#pragma unroll
                    for (int s = 0; s < SPT; ++s) tab.tip(e1, qg, (c1 >> (8 * s)) & (kCodes - 1), d1[s]);
                } else if (s1 == kSrcAcc) {
                    f2 r[4][4];
                    tab.p_pair(e1, qg, r);
#pragma unroll
                    for (int s = 0; s < SPT; ++s) mv_pair(r, acc[s][q], d1[s]);
                } else {
#pragma unroll
                    for (int s = 0; s < SPT; ++s)
#pragma unroll
                        for (int i = 0; i < 4; ++i) d1[s][i] = one2;
                }
                if (s0 >= 0) {
#pragma unroll
                    for (int s = 0; s < SPT; ++s) {
                        f2 d0[4];
                        tab.tip(e0, qg, (c0 >> (8 * s)) & (kCodes - 1), d0);
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[s][i]);
                    }
                } else {
                    f2 r[4][4];
                    tab.p_pair(e0, qg, r);
                    if (s0 == kSrcPop) {
                        uint32_t w[NC];
                        if (!Tab::kOver || sp < tmem_levels) {
                            tmem_wait_st();
                            tmem_ld<NC>(tstack + (uint32_t)((sp * KPT + q) * NC), w);
                            tmem_wait_ld();
                        } else {
                            over_ld<NC>(over + (uint32_t)(((sp - tmem_levels) * KPT + q) * NC * 128), w);
                        }
#pragma unroll
                        for (int s = 0; s < SPT; ++s) {
                            f2 x[4], d0[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                x[i] = pk2(__uint_as_float(w[8 * s + 2 * i]), __uint_as_float(w[8 * s + 2 * i + 1]));
                            mv_pair(r, x, d0);
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[s][i]);
                        }
                    } else {
#pragma unroll
                        for (int s = 0; s < SPT; ++s) {
                            f2 d0[4];
                            mv_pair(r, acc[s][q], d0);
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(d0[i], d1[s][i]);
                        }
                    }
                }
            }
        }
        // a quick exact test first (TPS = 1, two or more pairs): when the
        // maximum of the first pair's eight values reaches the threshold
        // so does the node maximum, and no rescale follows; only when
        // some lane of the warp falls short does the warp take the full
        // maximum below, with the decision and factors it always had
        bool full_test = true;
        if constexpr (TPS == 1 && KPT >= 2) {
            bool near = false;
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                const f2* a0 = acc[s][0];
                const float pm = fmax3(fmax3(a0[0].x, a0[0].y, a0[1].x), fmax3(a0[1].y, a0[2].x, a0[2].y),
                                       fmaxf(a0[3].x, a0[3].y));
                near |= !(pm >= scale_threshold<float>());
            }
            full_test = __any_sync(0xffffffffu, near);
        }
        if (full_test) {
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                // the node maximum (three-input max: the same value as the
                // fmaxf chain of run_tile4p; TPS = 2: with the partner's)
                float v[KPT * 8];
#pragma unroll
                for (int q = 0; q < KPT; ++q)
#pragma unroll
                    for (int i = 0; i < 4; ++i) unpack2(acc[s][q][i], v[q * 8 + 2 * i], v[q * 8 + 2 * i + 1]);
                float mx;
                if constexpr (KPT == 1) {
                    mx = fmax3(fmax3(v[0], v[1], v[2]), fmax3(v[3], v[4], v[5]), fmaxf(v[6], v[7]));
                } else if constexpr (KPT == 2) {
                    const float m0x = fmax3(v[0], v[1], v[2]), m1x = fmax3(v[3], v[4], v[5]);
                    const float m2x = fmax3(v[6], v[7], v[8]), m3x = fmax3(v[9], v[10], v[11]);
                    const float m4x = fmax3(v[12], v[13], v[14]);
                    mx = fmax3(fmax3(m0x, m1x, m2x), fmax3(m3x, m4x, v[15]), 0.0f);
                } else if constexpr (KPT == 3) {
                    float m[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) m[k] = fmax3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
                    mx = fmax3(fmax3(m[0], m[1], m[2]), fmax3(m[3], m[4], m[5]), fmax3(m[6], m[7], 0.0f));
                } else {
                    float m[11];
#pragma unroll
                    for (int k = 0; k < 10; ++k) m[k] = fmax3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
                    m[10] = fmaxf(v[30], v[31]);
                    const float g0 = fmax3(m[0], m[1], m[2]), g1 = fmax3(m[3], m[4], m[5]);
                    const float g2 = fmax3(m[6], m[7], m[8]), g3 = fmaxf(m[9], m[10]);
                    mx = fmax3(fmax3(g0, g1, g2), g3, 0.0f);
                }
                if constexpr (TPS == 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                if (mx < scale_threshold<float>() && mx > 0.0f) {
                    int e;
                    float g1, g2;
                    pow2_factors(mx, &e, &g1, &g2);
                    const f2 h1 = pk2(g1, g1), h2 = pk2(g2, g2);
#pragma unroll
                    for (int q = 0; q < KPT; ++q)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[s][q][i] = mul2(mul2(acc[s][q][i], h1), h2);
                    scale_e[s] += e;
                }
            }
        }
        if (push) {
            // the slot's columns, all pairs (KPT x NC), leave in as few
            // instructions as fit; the wait for them stands before the
            // next pop's loads
            uint32_t w[KPT * NC];
#pragma unroll
            for (int q = 0; q < KPT; ++q)
#pragma unroll
                for (int s = 0; s < SPT; ++s)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float lo, hi;
                        unpack2(acc[s][q][i], lo, hi);
                        w[q * NC + 8 * s + 2 * i] = __float_as_uint(lo);
                        w[q * NC + 8 * s + 2 * i + 1] = __float_as_uint(hi);
                    }
            const uint32_t ta = tstack + (uint32_t)(sp * KPT * NC);
            if (Tab::kOver && sp >= tmem_levels) {
                over_st<KPT * NC>(over + (uint32_t)((sp - tmem_levels) * KPT * NC * 128), w);
            } else if constexpr (KPT * NC == 8 || KPT * NC == 16 || KPT * NC == 32) {
                tmem_st<KPT * NC>(ta, w);
            } else {
#pragma unroll
                for (int q = 0; q < KPT; ++q) {
                    uint32_t wq[NC];
#pragma unroll
                    for (int k = 0; k < NC; ++k) wq[k] = w[q * NC + k];
                    tmem_st<NC>(ta + (uint32_t)(q * NC), wq);
                }
            }
            ++sp;
        }
        codes.next();
    }
    codes.finish();
    tab.finish();
}

// The root of the sites base + s, their log-likelihoods (to site_lnl where it
// is not null) added to sum; first: this thread adds the site up (TPS = 2: the
// even lane).
template <int KP, int SPT, int TPS>
__device__ __forceinline__ void root4w(const f2 (&acc)[SPT][KP / TPS][4], const int (&scale_e)[SPT], int base, int n_sites,
                                       bool first, const double* root_w, const double* cat_w, int C, double* site_lnl,
                                       SiteSum32& sum) {
    constexpr int KPT = KP / TPS;
    // root: L = sum_k w_k sum_s v_k[s] root_w[s] in FP32, categories in
    // order (run_tile4p), log L = lm + ee ln 2
    float rw[4], cw[2 * KP];
#pragma unroll
    for (int i = 0; i < 4; ++i) rw[i] = (float)root_w[i];
#pragma unroll
    for (int k = 0; k < 2 * KP; ++k) cw[k] = k < C ? (float)cat_w[k] : 0.0f;
#pragma unroll
    for (int s = 0; s < SPT; ++s) {
        float lk[2 * KP];  // this thread's categories first (the even lane's are 0 .. 2 KPT - 1)
#pragma unroll
        for (int q = 0; q < KPT; ++q) {
            float vv[2][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) unpack2(acc[s][q][i], vv[0][i], vv[1][i]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float x = vv[h][0] * rw[0];
#pragma unroll
                for (int i = 1; i < 4; ++i) x = fmaf(vv[h][i], rw[i], x);
                lk[2 * q + h] = x;
            }
        }
        if constexpr (TPS == 2) {
#pragma unroll
            for (int k = 0; k < 2 * KPT; ++k) lk[2 * KPT + k] = __shfl_xor_sync(0xffffffffu, lk[k], 1);
        }
        float lsum = 0.0f;
#pragma unroll
        for (int k = 0; k < 2 * KP; ++k) lsum = fmaf(cw[k], lk[k], lsum);
        const int site = base + s;
        if (site < n_sites && first) {
            float lm;
            int ee;
            site_log32(lsum, scale_e[s], lm, ee);
            if (site_lnl) site_lnl[site] = site_lnl64(lm, ee);
            site_sum_add(sum, lm, ee);
        }
    }
}

}  // namespace dev4w
}  // namespace plk
