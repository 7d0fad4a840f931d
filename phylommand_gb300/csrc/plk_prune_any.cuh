// prune_any: the post-order pass (src/simpleML.cpp:127-197) for any state
// count of 2..24 and up to 16 categories, FP64 in the reference's operation
// order or FP32 with FMA chains, and for 4 states in FP64 where the sites are
// too few to fill the chip one thread each.
//
// A site's vectors are spread over C x H neighbouring lanes of one warp: lane
// (k, h) holds rows h R .. h R + R - 1 of category k (R = ceil(S / H), both
// compile-time, so they sit in registers), W = 32 / (C H) sites to a warp.
//  * What bounds it: in FP64 the FP64 pipe (a warp instruction occupies it for
//    16 cycles of its SM), in FP32 at the usual site counts the latency of one
//    op after another.  Both want the sites over all SMs and the work of a site
//    over several lanes; a plan (any_plan) picks H and the warps per CTA from
//    the counts.  One thread a site in 128-thread CTAs, as prune_generic_kernel
//    runs, left 1,501 sites of 20 states on 12 of 152 SMs, its vectors in local
//    and strided global memory: 6,540 us for 40 taxa, C = 4, FP64.
//  * Everything an op reads is in shared memory: the op list and the CTA's tip
//    codes from the start, and either all P(t) and tip tables too (kRes, when
//    they fit: no barrier between ops), or the two children's tables of an op
//    in a ring filled two ops ahead by cp.async (one ahead where three slots
//    do not fit).  Reading ops, codes and tables from global memory a few ops
//    ahead into registers cost 400 instructions and 3,800 cycles an op (each
//    rotation of a prefetched register waits for its load).
//  * A lane that needs the whole vector reads it from its warp's exchange rows
//    in shared memory (H = 1 and S <= 8: from its own registers).
//  * The rescale decision is the node maximum over all states and categories
//    against the threshold, as in every other form: a ballot settles it unless
//    some site of the warp has no lane at or above the threshold.
// Operation order per value is prune_generic_kernel's, so are the bits.
// Measured, pass alone, before (prune_generic_kernel / prune4_kernel) and here:
// 20 states FP64 C = 4, 40 x 1,501: 6,540 -> 451 us; 5 states FP32 C = 4,
// 77 x 5,000: 681 -> 37 us; 4 states FP64 C = 1, 103 x 694: 212 -> 65 us.
#pragma once

#include <type_traits>

#include "plk_device.cuh"
#include "plk_internal.h"

namespace plk {
namespace dev {

struct AnyLaunch {
    int warps;       // per CTA
    int slots;       // stage ring slots, 2 or 3; 0: all tables resident
    int child_elems; // T elements between the two children of a slot
    int depth;       // spill-stack slots
    int stage_tips;  // tip tables go through the ring (else tip rows come from global memory)
    // node states (plk_node_states)
    void* msg;       // T [internal node][site][C][S]: messages to the parents, or null
    double* nodes;   // [rank][site][S]: normalised conditional vectors, or null
};

template <typename T, int S, int H>
struct AnyShape {
    static constexpr int R = (S + H - 1) / H;
    static constexpr bool kFp64 = std::is_same<T, double>::value;
    // elements per shared-memory load of a P row or of the exchanged vector
    static constexpr int V = kFp64 ? (S % 2 == 0 ? 2 : 1) : (S % 4 == 0 ? 4 : (S % 2 == 0 ? 2 : 1));
    // row stride of the exchange rows: an odd number of loads, no bank conflicts
    static constexpr int SX = (S / V) % 2 == 1 ? S : S + V;
    static constexpr bool kRegX = H == 1 && S <= 8;
    static constexpr int kRows = 32 / H;  // exchange rows of a warp (sites x categories)
    static constexpr int kExch = kRegX ? 0 : 2 * kRows * SX;  // exchange elements of a warp
};

// Shared memory of a launch: tables (the ring [slots][2][child], or all P(t)
// then all tip tables) | [warps] exchange rows | what the pass itself needs |
// [warps] pairs of vectors and sums of the node output (node_out) | ops or node
// table | tip codes [tip][sites of the CTA].
inline size_t any_node_bytes(int S, int C, int H, bool fp64) {  // of a warp
    return (size_t)(32 / H) * S * (fp64 ? 16 : 8) + (size_t)(32 / (C * H)) * (S + 2) * 8;
}
inline size_t any_base_smem(int S, int H, bool fp64, const AnyLaunch& p, int C, int n_nodes, int n_tips, int n_codes) {
    const int V = fp64 ? (S % 2 == 0 ? 2 : 1) : (S % 4 == 0 ? 4 : (S % 2 == 0 ? 2 : 1));
    const int SX = (S / V) % 2 == 1 ? S : S + V;
    const size_t exch = H == 1 && S <= 8 ? 0 : 2 * (size_t)(32 / H) * SX, tsz = fp64 ? 8 : 4;
    const size_t tables = p.slots ? (size_t)p.slots * 2 * p.child_elems
                                  : ((size_t)n_nodes * C * S * S + 3) / 4 * 4 + (size_t)n_tips * C * n_codes * S;
    return (tsz * tables + 15) / 16 * 16 + tsz * p.warps * exch + (size_t)n_tips * p.warps * (32 / (C * H));
}
// the post-order pass: its spill stack [depth][warps][R][32] and op list
inline size_t any_smem(int S, int H, bool fp64, const AnyLaunch& p, const PruneArgs& a) {
    const int R = (S + H - 1) / H;
    return any_base_smem(S, H, fp64, p, a.C, a.n_nodes, a.n_tips, a.n_codes) +
           (size_t)(fp64 ? 8 : 4) * p.depth * p.warps * R * 32 + (size_t)a.n_ops * sizeof(Op) +
           (p.nodes ? (p.warps * any_node_bytes(S, a.C, H, fp64) + 15) / 16 * 16 : 0);
}
// the pre-order pass: its node table, int4 a node
inline size_t any_down_smem(int S, int H, bool fp64, const AnyLaunch& p, const PreorderArgs& a) {
    return any_base_smem(S, H, fp64, p, a.C, a.n_nodes, a.n_tips, a.n_codes) + (size_t)a.n_int * 16 +
           (p.warps * any_node_bytes(S, a.C, H, fp64) + 15) / 16 * 16;
}

template <int BYTES>
__device__ __forceinline__ void cp_async_n(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}

// bytes (a multiple of 4) by all threads of the CTA in copies of unit bytes,
// the widest of 16, 8 and 4 that divides it: table offsets are multiples of
// the table's bytes from an aligned base
__device__ __forceinline__ int copy_unit(int bytes) { return bytes % 16 == 0 ? 16 : (bytes % 8 == 0 ? 8 : 4); }
__device__ __forceinline__ void stage_bytes(char* dst, const char* src, int bytes, int unit) {
    for (int i = threadIdx.x * unit; i < bytes; i += blockDim.x * unit) {
        if (unit == 16) cp_async16(dst + i, src + i);
        else if (unit == 8) cp_async_n<8>(dst + i, src + i);
        else cp_async_n<4>(dst + i, src + i);
    }
}

template <typename T, int V>
struct alignas(V * sizeof(T)) VecN {
    T v[V];
};

// one step of a row's sum: the first term a product, then in order
template <typename T, bool EXACT>
__device__ __forceinline__ T row_step(T acc, T x, T p, bool first) {
    if (first) return EXACT ? mul_rn(x, p) : x * p;
    return EXACT ? add_rn(acc, mul_rn(x, p)) : fma(x, p, acc);
}

// the category weights in shared memory, FP64 and as two FP32 parts
struct NodeWeights {
    double w[kMaxCats];
    float2 w2[kMaxCats];
    __device__ __forceinline__ void load(const double* cat_w, int C) {
        if ((int)threadIdx.x < C) {
            const double v = cat_w[threadIdx.x];
            w[threadIdx.x] = v;
            w2[threadIdx.x] = make_float2((float)v, (float)(v - (double)(float)v));
        }
    }
};

// One node's normalised output for the warp's sites: p_s proportional to
// sum_k w_k O[k][s] c[k][s] (O = 1 for the conditional vectors).  Every lane
// hands its rows in (its category's, h R ..) and takes (site, state) pairs out,
// so that a pair's sum over the categories runs in one lane and the doubles go
// out in order.  In FP64 the sum, the total and the division are FP64, the
// operations of the reference's order.  In FP32 they would put ten FP64
// instructions a value on a pipe that takes 16 cycles for each (the larger part
// of the pass); there the sums over the categories are carried as two FP32 parts
// (products and sums with their exact rounding errors, Dekker 1971 / Knuth's
// TwoSum), 2^-47 relative, under vectors that are good to 2^-22.  The total is kept
// in three parts and the quotient rounded at 2^-50, so that a site's outputs sum
// to one within 1.3e-15; a quotient in two rough parts left them up to 3e-13 from
// it.  Conditionals and marginals with their copy, rough and now: 4 states, 100 x
// 10,000, C = 4, 379 and 490 -> 365 and 492 us (FP64 for total and quotient: 501
// and 605); 20 states, 40 x 2,000, 192 and 257 -> 216 and 280.
// Static shared memory of the kernels, which counts towards a CTA's limit: the
// site sum's words and the last CTA's flag (post-order), the category weights
// (node states).
constexpr size_t kSumStatic = 32 * 2 * 8 + 32 * 4 + 16, kWeightStatic = sizeof(NodeWeights);

template <typename T, int S, int H>
struct NodeOut {
    T* oc;         // [site * C + k][S][2]
    double* sums;  // [site][S], then [site][2]
    const double* w;  // category weights, and as two FP32 parts
    const float2* w2;

    __device__ __forceinline__ void put(int row, int s, T o, T c) const {
        oc[(row * S + s) * 2] = o;
        oc[(row * S + s) * 2 + 1] = c;
    }
    // (hi, lo) + x + y with hi's rounding error kept in lo
    static __device__ __forceinline__ void add2(float& hi, float& lo, float x, float y) {
        float t, e;
        two_sum_f(hi, x, t, e);
        hi = t;
        lo = __fadd_rn(lo, __fadd_rn(e, y));
    }
    // all lanes of the warp; out = this node's doubles, site0 the warp's first site
    __device__ __forceinline__ void write(int C, int W, int site0, int n_sites, double* out) const {
        const int lane = threadIdx.x & 31;
        __syncwarp();
        if constexpr (std::is_same<T, double>::value) {
            double* tot = sums + W * S;
            for (int i = lane; i < W * S; i += 32) {
                double m = 0.0;
                for (int k = 0; k < C; ++k) {
                    const T* v = oc + ((i / S * C + k) * S + i % S) * 2;
                    m = fma(w[k] * v[0], v[1], m);
                }
                sums[i] = m;
            }
            __syncwarp();
            if (lane < W) {
                double t = 0.0;
                for (int s = 0; s < S; ++s) t += sums[lane * S + s];
                tot[lane] = t;
            }
            __syncwarp();
            for (int i = lane; i < W * S; i += 32)
                if (site0 + i / S < n_sites) out[(size_t)site0 * S + i] = sums[i] / tot[i / S];
        } else {
            float2* sum2 = reinterpret_cast<float2*>(sums);
            float2* tot = sum2 + W * S;
            for (int i = lane; i < W * S; i += 32) {
                float hi = 0.0f, lo = 0.0f;
                for (int k = 0; k < C; ++k) {
                    const float2 v = *reinterpret_cast<const float2*>(oc + ((i / S * C + k) * S + i % S) * 2);
                    const float wh = w2[k].x, wl = w2[k].y;
                    // 2^40 on both keeps products of small entries off the subnormals
                    const float o = v.x * 1099511627776.0f, c = v.y * 1099511627776.0f;
                    const float p = __fmul_rn(o, c), pe = fmaf(o, c, -p);
                    const float q = __fmul_rn(p, wh);
                    const float qe = __fadd_rn(fmaf(p, wh, -q), fmaf(p, wl, __fmul_rn(pe, wh)));
                    add2(hi, lo, q, qe);
                }
                sum2[i] = make_float2(hi, lo);
            }
            __syncwarp();
            if (lane < W) {
                Sum3 t;
                for (int s = 0; s < S; ++s) t.add(sum2[lane * S + s].x, sum2[lane * S + s].y, 0.0f);
                tot[2 * lane] = make_float2(t.h, t.l);
                tot[2 * lane + 1] = make_float2(t.ll, __frcp_rn(t.h));
            }
            __syncwarp();
            for (int i = lane; i < W * S; i += 32) {
                // long division: q1, rounded as a division would be, leaves a
                // remainder that is exact, q2 and q3 one in two parts; then the
                // quotient's two parts, the first one rounded
                const float2 m = sum2[i], t = tot[2 * (i / S)], u = tot[2 * (i / S) + 1];
                const float q0 = __fmul_rn(m.x, u.y), q1 = fmaf(fmaf(-q0, t.x, m.x), u.y, q0), c = __fmul_rn(q1, t.y);
                float r, e1, e2;
                two_sum_f(fmaf(-q1, t.x, m.x), m.y, r, e1);
                two_sum_f(r, -c, r, e2);
                const float low = __fadd_rn(__fadd_rn(e1, e2), fmaf(-q1, u.x, -fmaf(q1, t.y, -c)));
                const float q2 = __fmul_rn(r, u.y);
                const float q3 = __fmul_rn(__fadd_rn(fmaf(-q2, t.x, r), fmaf(-q2, t.y, low)), u.y);
                const float p1 = __fadd_rn(q1, q2), p2 = __fadd_rn(__fsub_rn(q2, __fsub_rn(p1, q1)), q3);
                if (site0 + i / S < n_sites) out[(size_t)site0 * S + i] = (double)p1 + (double)p2;
            }
        }
        __syncwarp();  // the next node's values may be put
    }
};

template <typename T, int S, int H, bool kRes, bool kNodes>
__global__ void __launch_bounds__(256) prune_any_kernel(PruneArgs a, AnyLaunch pl) {
    using Sh = AnyShape<T, S, H>;
    constexpr int R = Sh::R, V = Sh::V, SX = Sh::SX;
    constexpr bool EXACT = Sh::kFp64;
    constexpr bool kEven = R * H == S;  // every lane's rows are below S
    extern __shared__ __align__(16) unsigned char any_smem_raw[];
    const int C = a.C, G = C * H, W = 32 / G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // lanes past the last whole site repeat the first one's work and store nothing
    const int l = lane < W * G ? lane : lane - W * G;
    const int site_l = l / G, rem = l % G, k = rem / H, h = rem % H;
    const int tile = pl.warps * W, col = warp * W + site_l;  // the CTA's sites, this lane's among them
    const int site = blockIdx.x * tile + col;
    const bool valid = lane < W * G && site < a.n_sites;
    const int n_ops = a.n_ops;
    const int p_elems = C * S * S, t_elems = C * a.n_codes * S;  // of one node's P(t), one tip's table
    T* const tables = reinterpret_cast<T*>(any_smem_raw);
    // resident tables: P(t) of every node, then (16-byte aligned) every tip's
    const int tips_at = kRes ? (a.n_nodes * p_elems + 3) & ~3 : 0;
    const size_t table_elems = kRes ? (size_t)tips_at + (size_t)a.n_tips * t_elems
                                    : (size_t)pl.slots * 2 * pl.child_elems;
    T* const work = reinterpret_cast<T*>(any_smem_raw + (table_elems * sizeof(T) + 15) / 16 * 16);
    T* const xch = work + warp * Sh::kExch;
    T* const stack0 = work + pl.warps * Sh::kExch;
    T* stack = stack0 + warp * R * 32 + lane;
    const int stack_slot = pl.warps * R * 32;
    unsigned char* after = reinterpret_cast<unsigned char*>(stack0 + pl.depth * stack_slot);
    NodeOut<T, S, H> node{nullptr, nullptr, nullptr, nullptr};
    if (kNodes && pl.nodes) {  // doubles first, then the pairs of T
        __shared__ NodeWeights s_w;
        s_w.load(a.cat_w, C);
        node.w = s_w.w;
        node.w2 = s_w.w2;
        const int per = (32 / H) * S * 2 * (int)sizeof(T) + W * (S + 2) * 8;
        node.sums = reinterpret_cast<double*>(after + warp * per);
        node.oc = reinterpret_cast<T*>(after + warp * per + W * (S + 2) * 8);
        after += (pl.warps * per + 15) / 16 * 16;
    }
    Op* const s_ops = reinterpret_cast<Op*>(after);
    uint8_t* const s_codes = reinterpret_cast<uint8_t*>(s_ops + n_ops);
    T* const my_row = xch + (site_l * C + k) * SX;  // this site and category's exchange row
    T* const my_row2 = my_row + (Sh::kRegX ? 0 : Sh::kRows * SX);
    const T* P = static_cast<const T*>(a.P);
    const T* tipT = static_cast<const T*>(a.tipT);
    const int code_mask = S <= 4 ? (1 << S) - 1 : 255;  // a streamed alignment's codes are the caller's bytes
    const int p_unit = copy_unit(p_elems * (int)sizeof(T)), t_unit = copy_unit(t_elems * (int)sizeof(T));
    const unsigned site_mask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << (site_l * G);

    // ---- the op list, the tip codes and, with kRes, the tables
    for (int i = threadIdx.x; i < n_ops * (int)(sizeof(Op) / 16); i += blockDim.x)
        cp_async16(reinterpret_cast<char*>(s_ops) + 16 * i, reinterpret_cast<const char*>(a.ops) + 16 * i);
    if constexpr (kRes) {
        // whole tables (16-byte copies, a tail of words)
        auto all = [&](T* dst, const T* src, int elems) {
            char* d = reinterpret_cast<char*>(dst);
            const char* g = reinterpret_cast<const char*>(src);
            const int bytes = elems * (int)sizeof(T), whole = bytes / 16 * 16;
#pragma unroll 8
            for (int i = threadIdx.x * 16; i < whole; i += blockDim.x * 16) cp_async16(d + i, g + i);
            stage_bytes(d + whole, g + whole, bytes - whole, 4);
        };
        all(tables, P, a.n_nodes * p_elems);
        all(tables + tips_at, tipT, a.n_tips * t_elems);
    }
    cp_async_commit();
    {
        const int rows = blockDim.x / tile, s = threadIdx.x % tile;  // tile <= 32 warps = blockDim.x
        const uint8_t* src = a.codes + min(blockIdx.x * tile + s, a.n_sites - 1);
        int t = threadIdx.x / tile;
        if (t < rows)
#pragma unroll 4
            for (; t < a.n_tips; t += rows) s_codes[t * tile + s] = src[(size_t)t * a.site_stride] & code_mask;
    }
    cp_async_wait<0>();
    __syncthreads();
    // the tables of op o's children into ring slot `slot`
    auto stage = [&](int o, int slot) {
        const int4 ea = *reinterpret_cast<const int4*>(s_ops + o);
        const int4 sb = *(reinterpret_cast<const int4*>(s_ops + o) + 1);
        char* d0 = reinterpret_cast<char*>(tables + slot * 2 * pl.child_elems);
        char* d1 = d0 + pl.child_elems * sizeof(T);
        if (sb.x < 0)
            stage_bytes(d0, reinterpret_cast<const char*>(P + (size_t)ea.z * p_elems), p_elems * (int)sizeof(T), p_unit);
        else if (pl.stage_tips)
            stage_bytes(d0, reinterpret_cast<const char*>(tipT + (size_t)sb.x * t_elems), t_elems * (int)sizeof(T), t_unit);
        if (sb.y == kSrcAcc)
            stage_bytes(d1, reinterpret_cast<const char*>(P + (size_t)ea.w * p_elems), p_elems * (int)sizeof(T), p_unit);
        else if (sb.y >= 0 && pl.stage_tips)
            stage_bytes(d1, reinterpret_cast<const char*>(tipT + (size_t)sb.y * t_elems), t_elems * (int)sizeof(T), t_unit);
    };

    T acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = T(1);
    int scale_e = 0, sp = 0;
    int slot_now = 0, slot_next = pl.slots == 3 ? 2 : 1;  // ring slots of op o and of the op staged beside it
    if constexpr (!kRes) {
        stage(0, 0);
        cp_async_commit();
        if (pl.slots == 3) {
            if (n_ops > 1) stage(1, 1);
            cp_async_commit();
        }
    }
    int4 na = *reinterpret_cast<const int4*>(s_ops), nb = *(reinterpret_cast<const int4*>(s_ops) + 1);
    for (int o = 0; o < n_ops; ++o) {
        const int4 oa = na, ob = nb;
        if constexpr (!kRes) {
            if (pl.slots == 3) cp_async_wait<1>();
            else cp_async_wait<0>();
            __syncthreads();  // op o's tables are in; every warp is done with the slot filled next
            if (o + pl.slots - 1 < n_ops) stage(o + pl.slots - 1, slot_next);
            cp_async_commit();
        }
        if (o + 1 < n_ops) {
            na = *reinterpret_cast<const int4*>(s_ops + o + 1);
            nb = *(reinterpret_cast<const int4*>(s_ops + o + 1) + 1);
        }
        const int s0 = ob.x, s1 = ob.y;
        // the children's tables, and a tip child's row of its code
        const T *b0, *b1;
        if constexpr (kRes) {
            b0 = tables + (s0 >= 0 ? tips_at + s0 * t_elems : oa.z * p_elems);
            b1 = tables + (s1 >= 0 ? tips_at + s1 * t_elems : oa.w * p_elems);
        } else {
            b0 = tables + slot_now * 2 * pl.child_elems;
            b1 = b0 + pl.child_elems;
            slot_now = slot_now + 1 == pl.slots ? 0 : slot_now + 1;
            slot_next = slot_next + 1 == pl.slots ? 0 : slot_next + 1;
        }
        auto tip_rows = [&](int tip, const T* b, T (&t)[R]) {
            const int row = (k * a.n_codes + s_codes[tip * tile + col]) * S;
            if (kRes || pl.stage_tips) {
#pragma unroll
                for (int r = 0; r < R; ++r) t[r] = b[row + (kEven ? h * R + r : min(h * R + r, S - 1))];
            } else {
                const T* src = tipT + (size_t)tip * t_elems + row;
#pragma unroll
                for (int r = 0; r < R; ++r) t[r] = __ldg(src + (kEven ? h * R + r : min(h * R + r, S - 1)));
            }
        };
        T d0[R], d1[R], x0[R];
        if (s0 == kSrcPop) {
            --sp;
#pragma unroll
            for (int r = 0; r < R; ++r) x0[r] = stack[sp * stack_slot + r * 32];
        } else if (s0 == kSrcAcc) {
#pragma unroll
            for (int r = 0; r < R; ++r) x0[r] = acc[r];
        }
        if constexpr (!Sh::kRegX) {
            if (s0 < 0 || s1 == kSrcAcc) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) {
                        if (s0 < 0) my_row[h * R + r] = x0[r];
                        if (s1 == kSrcAcc) my_row2[h * R + r] = acc[r];
                    }
                __syncwarp();
            }
        }
        // out[r] = sum_j x[j] P[row r][j], j ascending
        auto product = [&](const T* Pc, const T (&xr)[R], const T* xs, T (&out)[R]) {
            const T* Pk = Pc + k * S * S;
            if constexpr (Sh::kRegX) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const VecN<T, V>* row = reinterpret_cast<const VecN<T, V>*>(Pk + r * S);
#pragma unroll
                    for (int j = 0; j < S / V; ++j) {
                        const VecN<T, V> p = row[j];
#pragma unroll
                        for (int q = 0; q < V; ++q)
                            out[r] = row_step<T, EXACT>(out[r], xr[j * V + q], p.v[q], j == 0 && q == 0);
                    }
                }
            } else {
                const VecN<T, V>* xv = reinterpret_cast<const VecN<T, V>*>(xs);
                const T* Ph = Pk + h * R * S;
                auto chunk = [&](int j, bool first) {
                    const VecN<T, V> x = xv[j];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const T* row = kEven ? Ph + r * S : Pk + min(h * R + r, S - 1) * S;
                        const VecN<T, V> p = reinterpret_cast<const VecN<T, V>*>(row)[j];
#pragma unroll
                        for (int q = 0; q < V; ++q) out[r] = row_step<T, EXACT>(out[r], x.v[q], p.v[q], first && q == 0);
                    }
                };
                chunk(0, true);
#pragma unroll 3
                for (int j = 1; j < S / V; ++j) chunk(j, false);
            }
        };
        // ---- child vectors
        if (s0 >= 0) tip_rows(s0, b0, d0);
        else product(b0, x0, my_row, d0);
        if (s1 >= 0) tip_rows(s1, b1, d1);
        else if (s1 == kSrcAcc) product(b1, acc, my_row2, d1);
        if (kNodes && pl.msg && valid) {  // the internal children's messages, for the pre-order pass
            T* const m = static_cast<T*>(pl.msg);
            if (s0 < 0) {
                T* dst = m + (((size_t)(oa.z - a.n_tips) * a.n_sites + site) * C + k) * S + h * R;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) dst[r] = d0[r];
            }
            if (s1 == kSrcAcc) {
                T* dst = m + (((size_t)(oa.w - a.n_tips) * a.n_sites + site) * C + k) * S + h * R;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) dst[r] = d1[r];
            }
        }
        T mx = T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            acc[r] = s1 == kSrcNone ? d0[r] : (EXACT ? mul_rn(d0[r], d1[r]) : d0[r] * d1[r]);
            // for the node states by magnitude: where rounding noise of P(0) is all a
            // vector has, its larger entries may be negative, and scaled by the
            // largest positive one they would overflow in the output
            mx = fmax(mx, kNodes ? fabs(acc[r]) : acc[r]);
        }
        // ---- per-site power-of-two scaling (exact)
        const unsigned high = __ballot_sync(0xffffffffu, mx >= scale_threshold<T>());
        if (__any_sync(0xffffffffu, (high & site_mask) == 0u)) {
            T node = mx;
            for (int q = 0; q < G; ++q) node = fmax(node, __shfl_sync(0xffffffffu, mx, site_l * G + q));
            if (node < scale_threshold<T>() && node > T(0)) {
                int e;
                T f1, f2;
                pow2_factors(node, &e, &f1, &f2);
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = (acc[r] * f1) * f2;
                scale_e += e;
            }
        }
        if (kNodes && pl.nodes) {
            if (lane < W * G)
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) node.put(site_l * C + k, h * R + r, T(1), acc[r]);
            node.write(C, W, blockIdx.x * tile + warp * W, a.n_sites, pl.nodes + (size_t)oa.y * a.n_sites * S);
        }
        if (ob.z) {
#pragma unroll
            for (int r = 0; r < R; ++r) stack[sp * stack_slot + r * 32] = acc[r];
            ++sp;
        }
        if constexpr (kRes && !Sh::kRegX) __syncwarp();  // the exchange rows are read before the next op writes them
    }
    cp_async_wait<0>();
    // ---- root: sum_k w_k sum_s L[s] root_w[s], states then categories in order
    __syncwarp();
    if constexpr (!Sh::kRegX) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (kEven || h * R + r < S) my_row[h * R + r] = acc[r];
        __syncwarp();
    }
    // 4 states in FP32 with up to 8 categories: the root in FP32, as every
    // 4-state FP32 form has it (site_log32)
    constexpr bool kRoot32 = S == 4 && !EXACT;
    double lk = 0.0;
    float lk32 = 0.0f;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        double v;
        if constexpr (Sh::kRegX) v = (double)acc[s];
        else v = (double)my_row[s];
        if constexpr (EXACT) lk = s == 0 ? __dmul_rn(v, a.root_w[0]) : __dadd_rn(lk, __dmul_rn(v, a.root_w[s]));
        else lk = s == 0 ? v * a.root_w[0] : fma(v, a.root_w[s], lk);
        if constexpr (kRoot32)
            lk32 = s == 0 ? (float)v * (float)a.root_w[0] : fmaf((float)v, (float)a.root_w[s], lk32);
    }
    SiteSum64 sum;
    double lsum = 0.0;
    float lsum32 = 0.0f;
    for (int q = 0; q < C; ++q) {
        if constexpr (kRoot32) {
            if (C <= 8) {
                const float x = __shfl_sync(0xffffffffu, lk32, site_l * G + q * H);
                lsum32 = fmaf((float)a.cat_w[q], x, lsum32);
                continue;
            }
        }
        const double x = __shfl_sync(0xffffffffu, lk, site_l * G + q * H);
        if constexpr (EXACT)
            lsum = q == 0 ? __dmul_rn(a.cat_w[0], x) : __dadd_rn(lsum, __dmul_rn(a.cat_w[q], x));
        else lsum = fma(a.cat_w[q], x, lsum);
    }
    if (valid && rem == 0) {
        double lnl;
        if (kRoot32 && C <= 8) {
            float lm;
            int ee;
            site_log32(lsum32, scale_e, lm, ee);
            lnl = site_lnl64(lm, ee);
        } else {
            lnl = log(lsum) + (double)scale_e * 0.69314718055994530942;
        }
        a.site_lnl[site] = lnl;
        site_sum64_add(sum, lnl);
    }
    const SiteSum64 bsum = block_sum_site64(sum);
    if (threadIdx.x == 0) store_site_record64(a.block_sum, blockIdx.x, bsum);
    if (a.grid_done) finish_grid_sum64(a.block_sum, a.grid_done, a.lnl_out);
}

// The pre-order pass and the normalised marginals (absent in the reference).
// At node u, from the root down: cond(u) is the product of its children's
// messages (prune_any left them in pl.msg), the output the normalised sum over
// the categories of Out(u) x cond(u), and every internal child v gets
//   Out(v)[b] = sum_i Out(u)[i] D_w[i] P_v[i][b],  i ascending, w its sibling,
// rescaled like a conditional vector.  The child visited next (rank r - 1) finds
// its vector in registers; another one's takes the place of its message, which
// no one reads again.  Lanes, tables and codes as in prune_any_kernel; the next
// node's messages are loaded while this one is worked on.  One thread a site
// with vectors in local memory took 1,161 us for 100 x 10,000 (C = 4, FP32) and
// recomputed D_w; this takes 200 us (and the pass before it 94 instead of 168).
template <typename T, int S, int H, bool kRes>
__global__ void __launch_bounds__(256) down_any_kernel(PreorderArgs a, AnyLaunch pl) {
    using Sh = AnyShape<T, S, H>;
    constexpr int R = Sh::R, SX = Sh::SX;
    constexpr bool kEven = R * H == S;
    constexpr bool kPre = R * (int)sizeof(T) <= 48;  // the next node's messages wait in registers
    extern __shared__ __align__(16) unsigned char any_smem_raw[];
    const int C = a.C, G = C * H, W = 32 / G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = lane < W * G ? lane : lane - W * G;
    const int site_l = l / G, rem = l % G, k = rem / H, h = rem % H;
    const int tile = pl.warps * W, col = warp * W + site_l;
    const int site = blockIdx.x * tile + col;
    const bool valid = lane < W * G && site < a.n_sites;
    const int n_int = a.n_int, n_tips = a.n_tips;
    const int p_elems = C * S * S, t_elems = C * a.n_codes * S;
    T* const tables = reinterpret_cast<T*>(any_smem_raw);
    const int tips_at = kRes ? (a.n_nodes * p_elems + 3) & ~3 : 0;
    const size_t table_elems = kRes ? (size_t)tips_at + (size_t)n_tips * t_elems : (size_t)pl.slots * 2 * pl.child_elems;
    T* const work = reinterpret_cast<T*>(any_smem_raw + (table_elems * sizeof(T) + 15) / 16 * 16);
    T* const xch = work + warp * Sh::kExch;
    unsigned char* after = reinterpret_cast<unsigned char*>(work + pl.warps * Sh::kExch);
    const int per = (32 / H) * S * 2 * (int)sizeof(T) + W * (S + 2) * 8;
    __shared__ NodeWeights s_w;
    s_w.load(a.cat_w, C);
    const NodeOut<T, S, H> node{reinterpret_cast<T*>(after + warp * per + W * (S + 2) * 8),
                                reinterpret_cast<double*>(after + warp * per), s_w.w, s_w.w2};
    int4* const s_kids = reinterpret_cast<int4*>(after + (pl.warps * per + 15) / 16 * 16);  // left, right, id
    uint8_t* const s_codes = reinterpret_cast<uint8_t*>(s_kids + n_int);
    T* const my_row = xch + (site_l * C + k) * SX;
    const T* P = static_cast<const T*>(a.P);
    const T* tipT = static_cast<const T*>(a.tipT);
    T* const msg = static_cast<T*>(pl.msg) + ((size_t)min(site, a.n_sites - 1) * C + k) * S;
    const size_t node_elems = (size_t)a.n_sites * C * S;
    const int code_mask = S <= 4 ? (1 << S) - 1 : 255;
    const int p_unit = copy_unit(p_elems * (int)sizeof(T)), t_unit = copy_unit(t_elems * (int)sizeof(T));
    const unsigned site_mask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << (site_l * G);

    for (int r = threadIdx.x; r < n_int; r += blockDim.x) {
        const int u = a.order[r];
        s_kids[r] = make_int4(a.left[u], a.right[u], u, 0);
    }
    if constexpr (kRes) {
        auto all = [&](T* dst, const T* src, int elems) {
            char* d = reinterpret_cast<char*>(dst);
            const char* g = reinterpret_cast<const char*>(src);
            const int bytes = elems * (int)sizeof(T), whole = bytes / 16 * 16;
#pragma unroll 8
            for (int i = threadIdx.x * 16; i < whole; i += blockDim.x * 16) cp_async16(d + i, g + i);
            stage_bytes(d + whole, g + whole, bytes - whole, 4);
        };
        all(tables, P, a.n_nodes * p_elems);
        all(tables + tips_at, tipT, n_tips * t_elems);
    }
    cp_async_commit();
    {
        const int rows = blockDim.x / tile, s = threadIdx.x % tile;
        const uint8_t* src = a.codes + min(blockIdx.x * tile + s, a.n_sites - 1);
        int t = threadIdx.x / tile;
        if (t < rows)
#pragma unroll 4
            for (; t < n_tips; t += rows) s_codes[t * tile + s] = src[(size_t)t * a.site_stride] & code_mask;
    }
    cp_async_wait<0>();
    __syncthreads();
    auto stage = [&](int r, int slot) {  // both children's tables of the node of rank r
        const int4 kd = s_kids[r];
        for (int c = 0; c < 2; ++c) {
            const int v = c ? kd.y : kd.x;
            char* d = reinterpret_cast<char*>(tables + (slot * 2 + c) * pl.child_elems);
            if (v >= n_tips)
                stage_bytes(d, reinterpret_cast<const char*>(P + (size_t)v * p_elems), p_elems * (int)sizeof(T), p_unit);
            else if (v >= 0 && pl.stage_tips)
                stage_bytes(d, reinterpret_cast<const char*>(tipT + (size_t)v * t_elems), t_elems * (int)sizeof(T), t_unit);
        }
    };
    auto row_of = [&](int r) { return kEven ? h * R + r : min(h * R + r, S - 1); };
    auto load_msg = [&](int v, T (&d)[R]) {
        const T* src = msg + (size_t)(v - n_tips) * node_elems;
#pragma unroll
        for (int r = 0; r < R; ++r) d[r] = src[row_of(r)];
    };
    // x's rescale, as in prune_any_kernel's node passes
    auto rescale = [&](T (&x)[R]) {
        T mx = T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) mx = fmax(mx, fabs(x[r]));
        const unsigned high = __ballot_sync(0xffffffffu, mx >= scale_threshold<T>());
        if (__any_sync(0xffffffffu, (high & site_mask) == 0u)) {
            T top = mx;
            for (int q = 0; q < G; ++q) top = fmax(top, __shfl_sync(0xffffffffu, mx, site_l * G + q));
            if (top < scale_threshold<T>() && top > T(0)) {
                int e;
                T f1, f2;
                pow2_factors(top, &e, &f1, &f2);
#pragma unroll
                for (int r = 0; r < R; ++r) x[r] = (x[r] * f1) * f2;
            }
        }
    };
    int slot_now = 0, slot_next = pl.slots == 3 ? 2 : 1;
    if constexpr (!kRes) {
        stage(n_int - 1, 0);
        cp_async_commit();
        if (pl.slots == 3) {
            if (n_int > 1) stage(n_int - 2, 1);
            cp_async_commit();
        }
    }
    T ou[R], co[R];
    bool carried = true;
    {
        // FP32: the root weights by the power of two that brings the largest
        // into [0.5, 1) (it cancels), so that node_out's scaled products fit
        T f = T(1);
        if constexpr (!Sh::kFp64) {
            float top = 0.0f;
            for (int s = 0; s < S; ++s) top = fmaxf(top, fabsf((float)a.root_w[s]));
            if (top > 0.0f && top <= 3.0e38f) f = ldexpf(1.0f, -max(-126, min(126, ilogbf(top) + 1)));
        }
#pragma unroll
        for (int r = 0; r < R; ++r) co[r] = (T)a.root_w[row_of(r)] * f;
    }
    T pl_[R], pr_[R];  // the messages of the next node's internal children
    if constexpr (kPre) {
        const int4 kd = s_kids[n_int - 1];
        if (kd.x >= n_tips) load_msg(kd.x, pl_);
        if (kd.y >= n_tips) load_msg(kd.y, pr_);
    }
    for (int rk = n_int - 1; rk >= 0; --rk) {
        const int4 kd = s_kids[rk];
        if constexpr (!kRes) {
            if (pl.slots == 3) cp_async_wait<1>();
            else cp_async_wait<0>();
            __syncthreads();
            if (rk - (pl.slots - 1) >= 0) stage(rk - (pl.slots - 1), slot_next);
            cp_async_commit();
        }
        const T *b0, *b1;
        if constexpr (kRes) {
            b0 = tables + (kd.x < n_tips ? tips_at + max(kd.x, 0) * t_elems : kd.x * p_elems);
            b1 = tables + (kd.y < n_tips ? tips_at + max(kd.y, 0) * t_elems : kd.y * p_elems);
        } else {
            b0 = tables + slot_now * 2 * pl.child_elems;
            b1 = b0 + pl.child_elems;
            slot_now = slot_now + 1 == pl.slots ? 0 : slot_now + 1;
            slot_next = slot_next + 1 == pl.slots ? 0 : slot_next + 1;
        }
        if (carried) {
#pragma unroll
            for (int r = 0; r < R; ++r) ou[r] = co[r];
        } else {
            load_msg(kd.z, ou);
        }
        carried = false;
        // ---- the children's messages
        T dl[R], dr[R];
        auto child = [&](int v, const T* b, const T (&pre)[R], T (&d)[R]) {
            if (v >= n_tips) {
                if constexpr (kPre) {
#pragma unroll
                    for (int r = 0; r < R; ++r) d[r] = pre[r];
                } else {
                    load_msg(v, d);
                }
            } else if (v >= 0) {
                const int row = (k * a.n_codes + s_codes[v * tile + col]) * S;
                if (kRes || pl.stage_tips) {
#pragma unroll
                    for (int r = 0; r < R; ++r) d[r] = b[row + row_of(r)];
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) d[r] = __ldg(tipT + (size_t)v * t_elems + row + row_of(r));
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) d[r] = T(1);
            }
        };
        child(kd.x, b0, pl_, dl);
        child(kd.y, b1, pr_, dr);
        const int next_id = rk > 0 ? s_kids[rk - 1].z : -1;
        if constexpr (kPre) {
            if (rk > 0) {
                const int4 kn = s_kids[rk - 1];
                if (kn.x >= n_tips) load_msg(kn.x, pl_);
                if (kn.y >= n_tips) load_msg(kn.y, pr_);
            }
        }
        // ---- this node's output
        {
            T c[R];
#pragma unroll
            for (int r = 0; r < R; ++r) c[r] = dl[r] * dr[r];
            rescale(c);
            if (lane < W * G)
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) node.put(site_l * C + k, h * R + r, ou[r], c[r]);
            node.write(C, W, blockIdx.x * tile + warp * W, a.n_sites, a.out + (size_t)rk * a.n_sites * S);
        }
        // ---- the internal children's outside vectors
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            const int v = c ? kd.y : kd.x;
            if (v < n_tips) continue;
            T t[R], ov[R];
#pragma unroll
            for (int r = 0; r < R; ++r) t[r] = ou[r] * (c ? dl[r] : dr[r]);
            const T* Pk = (c ? b1 : b0) + k * S * S;
            if constexpr (Sh::kRegX) {
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    T acc = T(0);
#pragma unroll
                    for (int i = 0; i < S; ++i) acc = fma(t[i], Pk[i * S + b], acc);
                    ov[b] = acc;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) my_row[h * R + r] = t[r];
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; ++r) ov[r] = T(0);
#pragma unroll 4
                for (int i = 0; i < S; ++i) {
                    const T x = my_row[i];
#pragma unroll
                    for (int r = 0; r < R; ++r) ov[r] = fma(x, Pk[i * S + row_of(r)], ov[r]);
                }
                __syncwarp();  // the exchange row is read before it is written again
            }
            rescale(ov);
            if (v == next_id) {
#pragma unroll
                for (int r = 0; r < R; ++r) co[r] = ov[r];
                carried = true;
            } else if (valid) {
                T* dst = msg + (size_t)(v - n_tips) * node_elems + h * R;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (kEven || h * R + r < S) dst[r] = ov[r];
            }
        }
    }
    cp_async_wait<0>();
}

template <typename T, int S, int H, bool kRes, bool kNodes>
cudaError_t launch_any_t(const PruneArgs& a, const AnyLaunch& p, int blocks, cudaStream_t st) {
    auto kern = prune_any_kernel<T, S, H, kRes, kNodes>;
    const size_t smem = any_smem(S, H, std::is_same<T, double>::value, p, a);
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, p.warps * 32, smem, st>>>(a, p);
    return cudaGetLastError();
}
template <typename T, int S, int H>
cudaError_t launch_any_h(const PruneArgs& a, const AnyLaunch& p, int blocks, cudaStream_t st) {
    // the tables of more than 8 states fit whole in shared memory only for a
    // handful of nodes: the ring alone there
    const bool nodes = p.msg || p.nodes;
    if constexpr (S <= 8) {
        if (p.slots == 0)
            return nodes ? launch_any_t<T, S, H, true, true>(a, p, blocks, st)
                         : launch_any_t<T, S, H, true, false>(a, p, blocks, st);
    }
    return nodes ? launch_any_t<T, S, H, false, true>(a, p, blocks, st)
                 : launch_any_t<T, S, H, false, false>(a, p, blocks, st);
}

template <typename T, int S, int H, bool kRes>
cudaError_t launch_down_any_t(const PreorderArgs& a, const AnyLaunch& p, int blocks, cudaStream_t st) {
    auto kern = down_any_kernel<T, S, H, kRes>;
    const size_t smem = any_down_smem(S, H, std::is_same<T, double>::value, p, a);
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, p.warps * 32, smem, st>>>(a, p);
    return cudaGetLastError();
}
template <typename T, int S, int H>
cudaError_t launch_any_h(const PreorderArgs& a, const AnyLaunch& p, int blocks, cudaStream_t st) {
    if constexpr (S <= 8) {
        if (p.slots == 0) return launch_down_any_t<T, S, H, true>(a, p, blocks, st);
    }
    return launch_down_any_t<T, S, H, false>(a, p, blocks, st);
}

// H is 1, 2 or 4 up to 8 states, 2 or 4 above (any_plan chooses no other);
// Args: PruneArgs (post-order) or PreorderArgs
template <typename T, int S, class Args>
cudaError_t launch_any_s(const Args& a, int H, const AnyLaunch& p, int blocks, cudaStream_t st) {
    if constexpr (S <= 8) {
        if (H == 1) return launch_any_h<T, S, 1>(a, p, blocks, st);
    }
    if (H == 2) return launch_any_h<T, S, 2>(a, p, blocks, st);
    if constexpr (S >= 4) {
        if (H == 4) return launch_any_h<T, S, 4>(a, p, blocks, st);
    }
    return cudaErrorInvalidConfiguration;
}

}  // namespace dev

// the state counts of each translation unit (S = 2..12 and 13..24)
#define PLK_ANY_DECLARE(name, Args) \
    cudaError_t name(const Args& a, int S, int H, const dev::AnyLaunch& p, int blocks, cudaStream_t st);
PLK_ANY_DECLARE(launch_any32_lo, PruneArgs)
PLK_ANY_DECLARE(launch_any32_hi, PruneArgs)
PLK_ANY_DECLARE(launch_any64_lo, PruneArgs)
PLK_ANY_DECLARE(launch_any64_hi, PruneArgs)
PLK_ANY_DECLARE(launch_down32_lo, PreorderArgs)
PLK_ANY_DECLARE(launch_down32_hi, PreorderArgs)
PLK_ANY_DECLARE(launch_down64_lo, PreorderArgs)
PLK_ANY_DECLARE(launch_down64_hi, PreorderArgs)

#define PLK_ANY_CASE(T, S) \
    case S: return dev::launch_any_s<T, S>(a, H, p, blocks, st);
#define PLK_ANY_LO(T)                                                                                           \
    PLK_ANY_CASE(T, 2) PLK_ANY_CASE(T, 3) PLK_ANY_CASE(T, 4) PLK_ANY_CASE(T, 5) PLK_ANY_CASE(T, 6)                \
    PLK_ANY_CASE(T, 7) PLK_ANY_CASE(T, 8) PLK_ANY_CASE(T, 9) PLK_ANY_CASE(T, 10) PLK_ANY_CASE(T, 11)              \
    PLK_ANY_CASE(T, 12)
#define PLK_ANY_HI(T)                                                                                           \
    PLK_ANY_CASE(T, 13) PLK_ANY_CASE(T, 14) PLK_ANY_CASE(T, 15) PLK_ANY_CASE(T, 16) PLK_ANY_CASE(T, 17)           \
    PLK_ANY_CASE(T, 18) PLK_ANY_CASE(T, 19) PLK_ANY_CASE(T, 20) PLK_ANY_CASE(T, 21) PLK_ANY_CASE(T, 22)           \
    PLK_ANY_CASE(T, 23) PLK_ANY_CASE(T, 24)

}  // namespace plk
