// NNI-neighbour scoring and branch-length derivatives of a batch.
//
// NNI: the likelihood of every tree one nearest neighbour interchange away
// from each batch tree (the rearrangements treebender --nni writes out,
// src/tree.cpp:2482-2548, which treeator then re-parses and scores from
// scratch, src/treeator.cpp:705-990), with branch lengths kept on their edges.
//
// One kernel, two passes over a tree per warp and its sites:
//  up    post-order: at every internal non-root node its message to the parent,
//        D = P(t) x conditional vector, goes to the warp's scratch slice with
//        its power-of-two exponent;
//  down  pre-order: the outside vector Out(v) = P_v^T (Out(u) x D_sibling) of
//        every internal child v of u (Out(root) = frequencies), and on the way
//        what the mode asks for, from vectors that are in registers then:
//    kNni   the two interchanges across the edge (u, v): with a, b the children
//           of v and c its sibling, L = sum_k w_k sum_s Out_u[s] D_z[s]
//           (P_v (D_x x D_y))[s] for (x, y, z) = (a, c, b) and (c, b, a); across
//           the root edge (v, c) the pairs of v's and c's children;
//    kBlen  the derivatives of the edges above u's children.
// What bounds it: shared-memory loads of P(t) rows and, in DRAM and L2, the
// scratch vectors.  An earlier form ran the moves as a third pass from scratch:
// 12 vector transfers per node and site, against 4 here (D once out and twice
// in; Out stays in registers for the child visited next and goes to scratch
// for the other one only where both are internal).  P_v is loaded once for the
// outside vector and both interchanges.
// A site's category pairs lie on neighbouring lanes (KP = ceil(C / 2) lanes a
// site, 32 / KP sites a warp; an odd last category is paired with itself, with
// weight 0), so a lane's vector is 8 registers of packed FP32 pairs; every
// warp walks its tree alone.  An item's tables sit in shared memory: P(t) of
// every node, whose columns are also the tip messages of the single-state
// codes, and one more row per tip for the all-states code (other ambiguity
// codes come from the full table in global memory).  Items whose tables do
// not fit read everything through L1.
// 12 warps of 168 registers an SM: with 16 of 128 the outside vector, the
// messages and P_v spilled (8.3 against 6.1 ms on the batch below).
// Measured, items of 8-256 taxa and 200-50,000 sites, C = 4, before and here:
// NNI of 48 items 17.4 -> 5.9 ms, derivatives of 24 items 7.0 -> 3.2 ms.
//
// All arithmetic on partials is FP32 in the order of run_tile / mv4: a site's
// log-likelihood is logf of the mantissa of L plus its power-of-two exponent
// times ln 2; the sites of a warp are summed with FP32 TwoSum and integer
// exponents into one record per move, and a last kernel folds an item's
// records in site order.
#include <algorithm>

#include "plk_batch.h"
#include "plk_device.cuh"
#include "plk_prune4s.cuh"

namespace plk {
using namespace dev;

namespace {

typedef float2 f2;  // one state of a category pair
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }

struct Vec {  // a vector of one category pair: 4 states
    f2 v[4];
};

__device__ __forceinline__ Vec mulv(const Vec& a, const Vec& b) {
    Vec r;
#pragma unroll
    for (int i = 0; i < 4; ++i) r.v[i] = mul2(a.v[i], b.v[i]);
    return r;
}
// three-input maximum (PTX ISA 8.8+, sm_100+): the same value as two fmaxf
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float maxv(const Vec& a) {
    return fmax3(fmax3(a.v[0].x, a.v[0].y, a.v[1].x), fmax3(a.v[1].y, a.v[2].x, a.v[2].y), fmaxf(a.v[3].x, a.v[3].y));
}

// P(t) of one node and category pair: p[j][i] = P[i][j] of both categories
struct Mat {
    f2 p[4][4];
};
// out[i] = sum_j P[i][j] x[j], j ascending, the first term a product (mv4)
__device__ __forceinline__ Vec times(const Mat& m, const Vec& x) {
    Vec o;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f2 a = mul2(x.v[0], m.p[0][i]);
        a = fma2(x.v[1], m.p[1][i], a);
        a = fma2(x.v[2], m.p[2][i], a);
        o.v[i] = fma2(x.v[3], m.p[3][i], a);
    }
    return o;
}
// out[b] = sum_a x[a] P[a][b], a ascending
__device__ __forceinline__ Vec times_t(const Mat& m, const Vec& x) {
    Vec o;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        f2 a = mul2(x.v[0], m.p[b][0]);
        a = fma2(x.v[1], m.p[b][1], a);
        a = fma2(x.v[2], m.p[b][2], a);
        o.v[b] = fma2(x.v[3], m.p[b][3], a);
    }
    return o;
}

constexpr int kNni = 0, kBlen = 1;
constexpr int kDownRegs = 168;
constexpr int kSlots = 8;  // moves or edges whose site values are buffered between two sums

// floats of one (node, pair) of the P(t) layout and of one (tip, pair) of the
// tip layout: [j][i][2] and [code][i][2]
constexpr int kPBlock = 32, kTipBlock = kCodes * 8;

struct Shape {  // of a launch
    int warps;      // per CTA
    int table_P;    // bytes of P(t) in shared memory for the largest item
    int table_all;  // bytes of the all-states rows
    int ops, kids;  // bytes of the op list and of the node table
    int codes;      // bytes of the tip codes, two sites a byte
    int smem;
};

// Shared memory: P(t) [node][pair][j][i][2] | all-states rows [tip][pair][i][2]
// | ops | node table int4 (left, right, first move, -) | codes | eigenvectors
// (kBlen) | per warp: site values [slot][site] (kNni: L, exponent; kBlen: L,
// L', L''), the slots' outputs.
template <int KP, bool kSmem>
Shape down_shape(int mode, int warps, int max_nodes, int max_tips, int n_int) {
    constexpr int W = 32 / KP;
    Shape s{};
    s.warps = warps;
    if (kSmem) {
        s.table_P = max_nodes * KP * kPBlock * 4;
        s.table_all = max_tips * KP * 32;
        s.ops = n_int * (int)sizeof(Op);
        s.kids = n_int * 16;
        s.codes = (max_tips * ((warps * W + 1) / 2) + 15) / 16 * 16;
    }
    const int per_warp = kSlots * (W + 1) * (mode == kNni ? 8 : 12) + kSlots * 4;
    s.smem = s.table_P + s.table_all + s.ops + s.kids + s.codes + 128 + (warps * per_warp + 15) / 16 * 16;
    return s;
}

__device__ __forceinline__ Vec vec_of(const float4& x, const float4& y) {
    Vec r;
    r.v[0] = make_float2(x.x, x.y);
    r.v[1] = make_float2(x.z, x.w);
    r.v[2] = make_float2(y.x, y.y);
    r.v[3] = make_float2(y.z, y.w);
    return r;
}

#define PLK_INLINE __attribute__((always_inline))

template <int KP, bool kSmem, int MODE>
__global__ void __maxnreg__(kDownRegs) batch_down_kernel(BatchDev b, BlenDev bd, Shape sh, int unit0, int unit1) {
    constexpr int W = 32 / KP, NV = MODE == kNni ? 2 : 3;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_unit;
    __shared__ BatchItemDev s_it;
    unsigned char* sp = sm;
    float* const s_P = reinterpret_cast<float*>(sp);
    sp += sh.table_P;
    float* const s_all = reinterpret_cast<float*>(sp);
    sp += sh.table_all;
    Op* const s_ops = reinterpret_cast<Op*>(sp);
    sp += sh.ops;
    int4* const s_kids = reinterpret_cast<int4*>(sp);
    sp += sh.kids;
    uint8_t* const s_codes = sp;
    sp += sh.codes;
    float* const s_eig = reinterpret_cast<float*>(sp);
    sp += 128;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int l = lane < W * KP ? lane : lane - W * KP;  // KP = 3: two lanes repeat the first site
    const int sl = l / KP, q = l % KP;
    const int tile = sh.warps * W, half_tile = (tile + 1) / 2, col = warp * W + sl;
    float* const vals = reinterpret_cast<float*>(sp) + warp * (kSlots * (W + 1) * NV + kSlots);
    int* const slot_out = reinterpret_cast<int*>(vals + kSlots * (W + 1) * NV);
    // this warp's scratch slice: messages, then outside vectors, [node rank][lane];
    // their exponents [node rank][site]
    const size_t gw = (size_t)blockIdx.x * sh.warps + warp;
    float4* const scr = b.scr + gw * b.scratch_int * 128 + 2 * lane;
    int* const scr_e = b.scr_e + gw * b.scratch_int * 2 * W + sl;
    const int out_at = b.scratch_int;  // the outside vectors' first rank
    const float thr = scale_threshold<float>();
    int loaded = -1;  // the item whose tables are in shared memory
    for (;;) {
        __syncthreads();  // the last unit's codes and tables are no longer read
        if (tid == 0) {
            s_unit = unit0 + atomicAdd(b.counter, 1);
            if (s_unit < unit1) s_it = b.items[b.units[s_unit].x];
        }
        __syncthreads();
        const int u_idx = s_unit;
        if (u_idx >= unit1) break;
        const int2 unit = b.units[u_idx];
        const int n_tips = s_it.n_tips, n_int = s_it.n_int, n_ops = s_it.n_ops;
        const int base = unit.y * tile;
        if (loaded != unit.x) {
            loaded = unit.x;
            if constexpr (kSmem) {
                const float* gP = b.Pn + (size_t)s_it.node_off * KP * kPBlock;
                const float* gT = b.tipn + (size_t)s_it.tip_off * KP * kTipBlock + (kCodes - 1) * 8;
                // 16-byte halves of a row are swapped for odd pairs, so that two
                // pairs' lanes read different banks
                for (int i = tid; i < (n_tips + n_int) * KP * 8; i += blockDim.x)
                    cp_async16(s_P + 4 * (i ^ ((i / 8) % KP & 1)), gP + 4 * i);
                for (int i = tid; i < n_tips * KP * 2; i += blockDim.x)
                    cp_async16(s_all + 4 * (i ^ ((i / 2) % KP & 1)), gT + (size_t)(i / 2) * kTipBlock + 4 * (i & 1));
                const int4* gops = reinterpret_cast<const int4*>(b.ops + s_it.ops_off);
                for (int i = tid; i < n_ops * 2; i += blockDim.x) cp_async16(reinterpret_cast<int4*>(s_ops) + i, gops + i);
                const int4* gkids = b.kids + (s_it.node_off - s_it.tip_off);
                for (int i = tid; i < n_int; i += blockDim.x) cp_async16(s_kids + i, gkids + i);
            }
            if (MODE == kBlen && tid < 32) s_eig[tid] = (float)b.model[s_it.model_off + 4 + tid];
        }
        cp_async_commit();
        if constexpr (kSmem) {
            // two sites' codes a byte; a warp a tip row at a time
            for (int t = warp; t < n_tips; t += sh.warps) {
                const uint8_t* row = b.codes + s_it.codes_off + (size_t)t * s_it.site_stride;
                for (int i = lane; i < half_tile; i += 32) {
                    const int c = base + 2 * i, last = s_it.site_stride - 1;
                    const int c0 = row[min(c, last)] & 15, c1 = row[min(c + 1, last)] & 15;
                    s_codes[t * half_tile + i] = (uint8_t)(c0 | (c1 << 4));
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        if (base + warp * W >= s_it.n_sites) continue;  // no sites for this warp (warp-uniform)
        const bool valid = base + col < s_it.n_sites;

        auto kids = [&](int rank) PLK_INLINE {
            if constexpr (kSmem) return s_kids[rank];
            else return __ldg(b.kids + (s_it.node_off - s_it.tip_off) + rank);
        };
        auto matrix = [&](int node) PLK_INLINE {
            Mat m;
            if constexpr (kSmem) {
                const float* p0 = s_P + (node * KP + q) * kPBlock + 4 * (q & 1);
                const float* p1 = s_P + (node * KP + q) * kPBlock + 4 * (1 ^ (q & 1));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const Vec v = vec_of(*reinterpret_cast<const float4*>(p0 + 8 * j),
                                         *reinterpret_cast<const float4*>(p1 + 8 * j));
#pragma unroll
                    for (int i = 0; i < 4; ++i) m.p[j][i] = v.v[i];
                }
            } else {
                const float4* p = reinterpret_cast<const float4*>(b.Pn + ((size_t)(s_it.node_off + node) * KP + q) * kPBlock);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const Vec v = vec_of(__ldg(p + 2 * j), __ldg(p + 2 * j + 1));
#pragma unroll
                    for (int i = 0; i < 4; ++i) m.p[j][i] = v.v[i];
                }
            }
            return m;
        };
        auto tip_code = [&](int tip) PLK_INLINE {
            if constexpr (kSmem) return (s_codes[tip * half_tile + (col >> 1)] >> (4 * (col & 1))) & 15;
            else
                return (int)b.codes[s_it.codes_off + (size_t)tip * s_it.site_stride +
                                    min(base + col, s_it.site_stride - 1)] & 15;
        };
        auto tip_row = [&](int tip, int code) PLK_INLINE {
            if constexpr (kSmem) {
                // a code of one state: that column of P(t) (code 0 only past the last site)
                const bool single = (code & (code - 1)) == 0;
                if (single || code == kCodes - 1) {
                    const float* r = single ? s_P + (tip * KP + q) * kPBlock + (31 - __clz(code | 1)) * 8
                                            : s_all + (tip * KP + q) * 8;
                    return vec_of(*reinterpret_cast<const float4*>(r + 4 * (q & 1)),
                                  *reinterpret_cast<const float4*>(r + 4 * (1 ^ (q & 1))));
                }
            }
            const float4* g =
                reinterpret_cast<const float4*>(b.tipn + ((size_t)(s_it.tip_off + tip) * KP + q) * kTipBlock + code * 8);
            return vec_of(__ldg(g), __ldg(g + 1));
        };
        auto load_vec = [&](int rank) PLK_INLINE {
            const float4* s = scr + (size_t)rank * 64;
            return vec_of(s[0], s[1]);
        };
        auto store_vec = [&](int rank, const Vec& r) PLK_INLINE {
            float4* s = scr + (size_t)rank * 64;
            s[0] = make_float4(r.v[0].x, r.v[0].y, r.v[1].x, r.v[1].y);
            s[1] = make_float4(r.v[2].x, r.v[2].y, r.v[3].x, r.v[3].y);
        };
        // message of a node to its parent and its exponent
        auto message = [&](int node, int& e) PLK_INLINE {
            if (node < n_tips) {
                e = 0;
                return tip_row(node, tip_code(node));
            }
            e = scr_e[(size_t)(node - n_tips) * W];
            return load_vec(node - n_tips);
        };
        // rescales x where its maximum over the site's pairs lies below the
        // threshold; the exponent taken out (0 where nothing was done).  When
        // every lane's own maximum reaches it, so does every site's.
        auto rescale = [&](Vec& x) PLK_INLINE {
            const float own = maxv(x);
            int e = 0;
            if (__any_sync(0xffffffffu, !(own >= thr))) {
                float mx = fmaxf(own, 0.0f);
#pragma unroll
                for (int d = 1; d < KP; ++d) mx = fmaxf(mx, __shfl_sync(0xffffffffu, own, sl * KP + (q + d) % KP));
                if (mx < thr && mx > 0.0f) {
                    float g1, g2;
                    pow2_factors(mx, &e, &g1, &g2);
                    const f2 h1 = make_float2(g1, g1), h2 = make_float2(g2, g2);
#pragma unroll
                    for (int i = 0; i < 4; ++i) x.v[i] = mul2(mul2(x.v[i], h1), h2);
                }
            }
            return e;
        };

        // ---- up
        {
            Vec run;  // the last node's message
            int run_e = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) run.v[i] = make_float2(1.0f, 1.0f);
            for (int o = 0; o + 1 < n_ops; ++o) {  // the last op is the root
                int4 oa, ob;
                if constexpr (kSmem) {
                    oa = *reinterpret_cast<const int4*>(s_ops + o);
                    ob = *(reinterpret_cast<const int4*>(s_ops + o) + 1);
                } else {
                    const int4* g = reinterpret_cast<const int4*>(b.ops + s_it.ops_off + o);
                    oa = __ldg(g);
                    ob = __ldg(g + 1);
                }
                Vec x = run;
                int e = run_e;
                if (ob.x != kSrcAcc) x = message(ob.x >= 0 ? ob.x : oa.z, e);
                if (ob.y >= 0) {
                    x = mulv(x, tip_row(ob.y, tip_code(ob.y)));
                } else if (ob.y == kSrcAcc) {
                    x = mulv(x, run);
                    e += run_e;
                }
                e += rescale(x);
                run = times(matrix(oa.x), x);
                run_e = e;
                store_vec(oa.y, run);
                if (q == 0) scr_e[(size_t)oa.y * W] = e;
            }
        }
        __syncwarp();  // a site's exponents were stored by its first lane

        // ---- down
        const double* const mdl = b.model + s_it.model_off;
        auto root_weights = [&]() PLK_INLINE {
            Vec r;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float w = (float)mdl[36 + i];
                r.v[i] = make_float2(w, w);
            }
            return r;
        };
        float wk[2 * KP];
#pragma unroll
        for (int k = 0; k < 2 * KP; ++k) wk[k] = k < b.C ? (float)mdl[40 + b.C + k] : 0.0f;
        const bool odd_cats = (b.C & 1) != 0;
        int slot = 0;
        [[maybe_unused]] f2 rho[4];  // kBlen: the pair's rates
        if constexpr (MODE == kBlen) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
                rho[m] = make_float2((float)(mdl[m] * mdl[40 + 2 * q]),
                                     (float)(mdl[m] * mdl[40 + min(2 * q + 1, b.C - 1)]));
        }
        // The buffered values of up to kSlots moves or edges: four lanes a slot
        // take a quarter of the sites each, then one record a slot.
        auto flush = [&]() PLK_INLINE {
            __syncwarp();
            const int s = lane >> 2, part = lane & 3;
            float h1 = 0.0f, l1 = 0.0f, h2 = 0.0f, l2 = 0.0f;
            int esum = 0;
            for (int c = part; c < W; c += 4) {
                if constexpr (MODE == kNni) {
                    const float2 v = reinterpret_cast<const float2*>(vals)[s * (W + 1) + c];
                    const int bits = __float_as_int(v.x);
                    // zero, a negative one (rounding noise of P(0)), infinity and NaN keep
                    // logf's own result (-inf, NaN, inf, NaN), as in site_log32
                    const float lm = v.x > 0.0f && v.x <= 3.40282347e38f
                                         ? logf(__int_as_float((bits & 0x007fffff) | 0x3f800000))
                                         : logf(v.x);
                    float ns, er;
                    two_sum_f(h1, lm, ns, er);
                    h1 = ns;
                    l1 = __fadd_rn(l1, er);
                    esum += __float_as_int(v.y) + ((bits >> 23) & 255) - 127;
                } else {
                    const float* v = vals + (s * (W + 1) + c) * 3;
                    const float g = __fdiv_rn(v[1], v[0]);
                    const float d = __fsub_rn(__fdiv_rn(v[2], v[0]), __fmul_rn(g, g));
                    float ns, er;
                    two_sum_f(h1, g, ns, er);
                    h1 = ns;
                    l1 = __fadd_rn(l1, er);
                    two_sum_f(h2, d, ns, er);
                    h2 = ns;
                    l2 = __fadd_rn(l2, er);
                }
            }
#pragma unroll
            for (int off = 1; off <= 2; off <<= 1) {
                float oh = __shfl_xor_sync(0xffffffffu, h1, off), ol = __shfl_xor_sync(0xffffffffu, l1, off);
                float ns, er;
                two_sum_f(h1, oh, ns, er);
                h1 = ns;
                l1 = __fadd_rn(l1, __fadd_rn(ol, er));
                if constexpr (MODE == kNni) {
                    esum += __shfl_xor_sync(0xffffffffu, esum, off);
                } else {
                    oh = __shfl_xor_sync(0xffffffffu, h2, off);
                    ol = __shfl_xor_sync(0xffffffffu, l2, off);
                    two_sum_f(h2, oh, ns, er);
                    h2 = ns;
                    l2 = __fadd_rn(l2, __fadd_rn(ol, er));
                }
            }
            if (part == 0 && s < slot) {
                const int n_out = MODE == kNni ? s_it.n_moves : 2 * n_int;
                float4* rec = b.records + b.rec_off[unit.x] + (size_t)(base / W + warp) * n_out;
                if constexpr (MODE == kNni) rec[slot_out[s]] = make_float4(h1, l1, __int_as_float(esum), 0.0f);
                else rec[slot_out[s]] = make_float4(h1, l1, h2, l2);
            }
            __syncwarp();
            slot = 0;
        };
        // sum over the categories in order of w_k x_k, valid in a site's first lane
        auto mix = [&](f2 x) PLK_INLINE {
            float s = fmaf(wk[0], x.x, 0.0f);
            if (KP > 1 || !odd_cats) s = fmaf(wk[1], x.y, s);
#pragma unroll
            for (int d = 1; d < KP; ++d) {
                const int src = sl * KP + min(q + d, KP - 1);
                const float y0 = __shfl_sync(0xffffffffu, x.x, src), y1 = __shfl_sync(0xffffffffu, x.y, src);
                s = fmaf(wk[2 * d], y0, s);
                if (d < KP - 1 || !odd_cats) s = fmaf(wk[2 * d + 1], y1, s);
            }
            return s;
        };
        // likelihood of an interchange: lsum 2^etot into the buffer
        auto score = [&](const Vec& o, const Vec& a, const Vec& z, int etot, int move) PLK_INLINE {
            auto cats = [&](float scale) PLK_INLINE {
                const f2 sc = make_float2(scale, scale);
                f2 lk = mul2(mul2(o.v[0], sc), mul2(a.v[0], z.v[0]));
#pragma unroll
                for (int i = 1; i < 4; ++i) lk = fma2(mul2(o.v[i], sc), mul2(a.v[i], z.v[i]), lk);
                return lk;
            };
            f2 lk = mul2(o.v[0], mul2(a.v[0], z.v[0]));
#pragma unroll
            for (int i = 1; i < 4; ++i) lk = fma2(o.v[i], mul2(a.v[i], z.v[i]), lk);
            float lsum = mix(lk);
            // below the normal range (or zero): again with 2^64 on the weights
            const bool low = q == 0 && !(lsum >= 1.17549435e-38f);
            if (__any_sync(0xffffffffu, low)) {
                const float l2 = mix(cats(1.8446744073709552e19f));
                if (low) {
                    lsum = l2;
                    etot -= 64;
                }
            }
            if (q == 0 && lane < W * KP)
                reinterpret_cast<float2*>(vals)[slot * (W + 1) + sl] =
                    valid ? make_float2(lsum, __int_as_float(etot)) : make_float2(1.0f, 0.0f);
            if (lane == 0) slot_out[slot] = move;
            ++slot;
        };
        // The outside vector and the children's messages of the next node down
        // (rank r - 1 is the child visited last where that is internal): both
        // were in registers when its parent was visited.
        Vec co = root_weights(), cl, cr;
        int co_e = 0, cl_e = 0, cr_e = 0;
        bool have = false;
        for (int r = n_int - 1; r >= 0; --r) {
            const int4 kd = kids(r);
            Vec ou = co, ml = cl, mr = cr;
            int eu = co_e, el = cl_e, er = cr_e;
            if (!have) {
                if (r != n_int - 1) {
                    ou = load_vec(out_at + r);
                    eu = scr_e[(size_t)(out_at + r) * W];
                }
                if (kd.x >= 0) ml = message(kd.x, el);
                if (kd.y >= 0) mr = message(kd.y, er);
            }
            have = false;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int v = c == 0 ? kd.x : kd.y, w = c == 0 ? kd.y : kd.x;
                if (v < 0 || (MODE == kNni && v < n_tips)) continue;
                const int rv = v - n_tips;
                int4 kv = make_int4(-1, -1, -1, -1);
                if (v >= n_tips) {  // messages of v's children
                    kv = kids(rv);
                    if (kv.x >= 0) cl = message(kv.x, cl_e);
                    if (kv.y >= 0) cr = message(kv.y, cr_e);
                }
                Vec t = ou;  // what the sibling's side sends to the edge above v
                int et = eu;
                if (w >= 0) {
                    t = mulv(t, c == 0 ? mr : ml);
                    et += c == 0 ? er : el;
                }
                if constexpr (MODE == kBlen) {
                    // L(t) = sum_k w_k sum_m (L^T A)_m (R c)_m exp(rho_km t)
                    const float4* ex = reinterpret_cast<const float4*>(bd.ex + ((size_t)(s_it.node_off + v) * KP + q) * 8);
                    const Vec exm = vec_of(__ldg(ex), __ldg(ex + 1));
                    Vec cv;
                    if (v < n_tips) {
                        const int code = tip_code(v);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float x = (float)((code >> i) & 1);
                            cv.v[i] = make_float2(x, x);
                        }
                    } else {
                        cv = kv.x >= 0 ? cl : cr;
                        if (kv.x >= 0 && kv.y >= 0) cv = mulv(cv, cr);
                    }
                    f2 s0 = make_float2(0.f, 0.f), s1 = s0, s2 = s0;
                    Vec ax;  // L^T A, i ascending
#pragma unroll
                    for (int m = 0; m < 4; ++m) ax.v[m] = s0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 L4 = *reinterpret_cast<const float4*>(s_eig + 4 * i);
                        const float Lm[4] = {L4.x, L4.y, L4.z, L4.w};
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            ax.v[m].x = fmaf(t.v[i].x, Lm[m], ax.v[m].x);
                            ax.v[m].y = fmaf(t.v[i].y, Lm[m], ax.v[m].y);
                        }
                    }
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const float4 R4 = *reinterpret_cast<const float4*>(s_eig + 16 + 4 * m);
                        f2 y = make_float2(0.f, 0.f);
                        const float Ri[4] = {R4.x, R4.y, R4.z, R4.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            y.x = fmaf(Ri[i], cv.v[i].x, y.x);
                            y.y = fmaf(Ri[i], cv.v[i].y, y.y);
                        }
                        const f2 term = mul2(mul2(ax.v[m], y), exm.v[m]);
                        s0 = __fadd2_rn(s0, term);
                        s1 = fma2(rho[m], term, s1);
                        s2 = fma2(mul2(rho[m], rho[m]), term, s2);
                    }
                    const float l0 = mix(s0), l1 = mix(s1), l2 = mix(s2);
                    if (q == 0 && lane < W * KP) {
                        float* dst = vals + (slot * (W + 1) + sl) * 3;
                        dst[0] = valid ? l0 : 1.0f;
                        dst[1] = valid ? l1 : 0.0f;
                        dst[2] = valid ? l2 : 0.0f;
                    }
                    if (lane == 0) slot_out[slot] = 2 * r + c;
                    if (++slot == kSlots) flush();
                    if (v < n_tips) continue;
                }
                const Mat m = matrix(v);
                Vec ov = times_t(m, t);
                const int eo = et + rescale(ov);
                if constexpr (MODE == kNni) {
                    if (kv.z >= 0 && r != n_int - 1) {  // the sibling's message is ml or mr
                        const int e_all = et + cl_e + cr_e;
                        Vec t1 = mulv(cl, c == 0 ? mr : ml);
                        int e1 = rescale(t1);
                        score(ou, times(m, t1), cr, e_all + e1, kv.z);
                        t1 = mulv(cr, c == 0 ? mr : ml);
                        e1 = rescale(t1);
                        score(ou, times(m, t1), cl, e_all + e1, kv.z + 1);
                        if (slot == kSlots) flush();
                    }
                }
                if (rv == r - 1) {  // visited next: its children's messages stay in cl, cr
                    co = ov;
                    co_e = eo;
                    have = true;
                } else {
                    store_vec(out_at + rv, ov);
                    if (q == 0) scr_e[(size_t)(out_at + rv) * W] = eo;
                }
            }
            __syncwarp();  // stored exponents are read by the site's other lanes
        }
        // the interchanges across the root edge (v left, w right, both internal)
        if constexpr (MODE == kNni) {
            const int4 kd = kids(n_int - 1);
            const int4 kv = kd.x >= n_tips ? kids(kd.x - n_tips) : make_int4(-1, -1, -1, -1);
            if (kv.z >= 0) {
                const int4 kw = kids(kd.y - n_tips);
#pragma unroll 1
                for (int which = 0; which < 2; ++which) {  // (a, d)(b, e), then (a, e)(d, b)
                    int ex, ey, ep, eq;
                    Vec t1 = message(kv.x, ex);
                    t1 = mulv(t1, message(which ? kw.y : kw.x, ey));
                    const int e1 = rescale(t1);
                    Vec t4 = message(which ? kw.x : kv.y, ep);
                    t4 = mulv(t4, message(which ? kv.y : kw.y, eq));
                    score(root_weights(), times(matrix(kd.x), t1), times(matrix(kd.y), t4), ex + ey + e1 + ep + eq,
                          kv.z + which);
                }
            }
        }
        if (slot > 0) flush();
    }
}

constexpr int kFoldWarps = 32;
// One CTA per (item, 32 outputs): its warps fold the records of the item's
// warp tiles, each every 32nd tile in order, a lane per output; then the
// warps' sums in order.  Latency bound (a 50,000-site item has 3,125 tiles):
// 32 warps with four loads in flight took the fold of the 24-item derivative
// batch from 83 us (eight warps) to 30 us; with the third part of the
// derivatives' sums it issues for 48 us.
template <int MODE>
__global__ void __launch_bounds__(32 * kFoldWarps) batch_down_reduce_kernel(BatchDev b, BlenDev bd, int W) {
    const int2 blk = b.reduce_blocks[blockIdx.x];
    const BatchItemDev it = b.items[blk.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_out = MODE == kNni ? it.n_moves : 2 * it.n_int, m = blk.y + lane;
    const int tiles = (it.n_sites + W - 1) / W;
    const float4* rec = b.records + b.rec_off[blk.x] + m;
    if constexpr (MODE == kBlen) {
        __shared__ Sum3 part[2][kFoldWarps][32];
        Sum3 d1, d2;
        if (m < n_out) {
#pragma unroll 4
            for (int t = warp; t < tiles; t += kFoldWarps) {
                const float4 v = rec[(size_t)t * n_out];
                d1.add(v.x, v.y, 0.0f);
                d2.add(v.z, v.w, 0.0f);
            }
        }
        part[0][warp][lane] = d1;
        part[1][warp][lane] = d2;
        __syncthreads();
        if (warp != 0 || m >= n_out) return;
        for (int w = 1; w < kFoldWarps; ++w) {
            const Sum3 a = part[0][w][lane], c = part[1][w][lane];
            d1.add(a.h, a.l, a.ll);
            d2.add(c.h, c.l, c.ll);
        }
        const int g = bd.item_edge_off[blk.x] + m;
        bd.edge_out[2 * g] = d1.value();
        bd.edge_out[2 * g + 1] = d2.value();
    } else {
        __shared__ float2 part[kFoldWarps][32];
        __shared__ long long part_e[kFoldWarps][32];
        float h = 0.0f, l = 0.0f;
        long long e = 0;
        auto add = [&](float oh, float ol) {
            float ns, er;
            two_sum_f(h, oh, ns, er);
            h = ns;
            l = __fadd_rn(l, __fadd_rn(ol, er));
        };
        if (m < n_out) {
#pragma unroll 4
            for (int t = warp; t < tiles; t += kFoldWarps) {
                const float4 v = rec[(size_t)t * n_out];
                add(v.x, v.y);
                e += __float_as_int(v.z);
            }
        }
        part[warp][lane] = make_float2(h, l);
        part_e[warp][lane] = e;
        __syncthreads();
        if (warp != 0 || m >= n_out) return;
        for (int w = 1; w < kFoldWarps; ++w) {
            add(part[w][lane].x, part[w][lane].y);
            e += part_e[w][lane];
        }
        // an infinite sum is what it is (its low part is not a number)
        b.nni_out[it.move_out_off + m] = isinf(h) ? (double)h : fma((double)e, 0.69314718055994530942, (double)h + (double)l);
    }
}

// P(t) = L diag(exp(lambda r t)) R of every (node, category) of every item
// (FP64, stored as FP32) and the tip tables in the layouts above, an odd last
// category also in the place of its missing partner; for kBlen also
// exp(rho t) [node][pair][m][2] and the items' FP32 eigenvectors.  One FP64
// sum per code and state: a code's sum over its allowed states, ascending, is
// that of the code without its highest state plus one term.
__global__ void __launch_bounds__(128) batch_down_tables_kernel(BatchDev b, BlenDev bd) {
    const int C = b.C, KP = (C + 1) / 2;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)b.n_nodes_total * C) return;
    const int g = (int)(gid / C), k = (int)(gid % C);
    const int2 nm = b.node_item[g];
    const BatchItemDev it = b.items[nm.x];
    const double* mdl = b.model + it.model_off;
    const double t = b.t_eff[g] * mdl[40 + k];
    double ex[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) ex[m] = exp(mdl[m] * t);
    const int last = (k == C - 1 && (C & 1)) ? 2 : 1;  // places this category fills
    float* dP = b.Pn + ((size_t)g * KP + k / 2) * kPBlock + (k & 1);
    float* dT = nm.y < it.n_tips ? b.tipn + ((size_t)(it.tip_off + nm.y) * KP + k / 2) * kTipBlock + (k & 1) : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double row[4], sum[kCodes];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double acc = 0.0;
#pragma unroll
            for (int m = 0; m < 4; ++m) acc = fma(mdl[4 + i * 4 + m] * ex[m], mdl[20 + m * 4 + j], acc);
            row[j] = acc;
            for (int q = 0; q < last; ++q) dP[j * 8 + i * 2 + q] = (float)acc;
        }
        if (!dT) continue;
        sum[0] = 0.0;
#pragma unroll
        for (int code = 1; code < kCodes; ++code) {
            const int top = code >= 8 ? 3 : (code >= 4 ? 2 : (code >= 2 ? 1 : 0));
            sum[code] = code == (1 << top) ? row[top] : sum[code ^ (1 << top)] + row[top];
        }
#pragma unroll
        for (int code = 0; code < kCodes; ++code)
            for (int q = 0; q < last; ++q) dT[code * 8 + i * 2 + q] = (float)sum[code];
    }
    if (bd.ex) {
        const float t32 = (float)b.t_eff[g];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            for (int q = 0; q < last; ++q)
                bd.ex[((size_t)g * KP + k / 2) * 8 + m * 2 + (k & 1) + q] = expf((float)(mdl[m] * mdl[40 + k]) * t32);
    }
}

template <int KP, bool kSmem, int MODE>
cudaError_t launch_t(const BatchDev& b, const BlenDev& bd, const Shape& sh, int unit0, int unit1, int grid,
                     cudaStream_t st) {
    auto kern = batch_down_kernel<KP, kSmem, MODE>;
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), sh.smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, sh.warps * 32, sh.smem, st>>>(b, bd, sh, unit0, unit1);
    return cudaGetLastError();
}

template <int KP, bool kSmem, int MODE>
int occupancy_t(const Shape& sh) {
    auto kern = batch_down_kernel<KP, kSmem, MODE>;
    int n = 0;
    if (allow_smem(reinterpret_cast<const void*>(kern), sh.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, sh.warps * 32, sh.smem) != cudaSuccess) {
        cudaGetLastError();  // a size that does not fit is no error of the next launch
        return 0;
    }
    return n;
}

// calls f<KP, kSmem, MODE>() for a launch
template <class F>
auto dispatch(int C, bool in_smem, bool blen, F f) {
    const int KP = (C + 1) / 2;
#define PLK_DOWN(K)                                                                                     \
    if (KP == K) {                                                                                      \
        if (in_smem) return blen ? f.template operator()<K, true, kBlen>()                                   \
                                 : f.template operator()<K, true, kNni>();                                    \
        return blen ? f.template operator()<K, false, kBlen>() : f.template operator()<K, false, kNni>();  \
    }
    PLK_DOWN(1) PLK_DOWN(2) PLK_DOWN(3)
#undef PLK_DOWN
    if (in_smem) return blen ? f.template operator()<4, true, kBlen>() : f.template operator()<4, true, kNni>();
    return blen ? f.template operator()<4, false, kBlen>() : f.template operator()<4, false, kNni>();
}

struct ShapeOf {
    int mode, warps, nodes, tips, ints;
    template <int KP, bool kSmem, int MODE>
    Shape operator()() const { return down_shape<KP, kSmem>(mode, warps, nodes, tips, ints); }
};
struct LimitOf {
    template <int KP, bool kSmem, int MODE>
    size_t operator()() const { return smem_limit(reinterpret_cast<const void*>(batch_down_kernel<KP, kSmem, MODE>)); }
};
struct OccOf {
    Shape sh;
    template <int KP, bool kSmem, int MODE>
    int operator()() const { return occupancy_t<KP, kSmem, MODE>(sh); }
};
struct LaunchOf {
    const BatchDev& b;
    const BlenDev& bd;
    Shape sh;
    int unit0, unit1, grid;
    cudaStream_t st;
    template <int KP, bool kSmem, int MODE>
    cudaError_t operator()() const { return launch_t<KP, kSmem, MODE>(b, bd, sh, unit0, unit1, grid, st); }
};

}  // namespace

int down_sites_per_warp(int C) { return 32 / ((C + 1) / 2); }

int down_smem_bytes(int C, bool blen, bool in_smem, const DownSize& z) {
    return dispatch(C, in_smem, blen, ShapeOf{blen ? kBlen : kNni, z.warps, z.nodes, z.tips, z.ints}).smem;
}

size_t down_smem_limit(int C, bool blen, bool in_smem) { return dispatch(C, in_smem, blen, LimitOf{}); }

int down_occupancy(int C, bool blen, bool in_smem, const DownSize& z) {
    const Shape sh = dispatch(C, in_smem, blen, ShapeOf{blen ? kBlen : kNni, z.warps, z.nodes, z.tips, z.ints});
    return dispatch(C, in_smem, blen, OccOf{sh});
}

cudaError_t launch_down_tables(const BatchDev& b, const BlenDev& bd, cudaStream_t st) {
    const long long n = (long long)b.n_nodes_total * b.C;
    const unsigned blocks = (unsigned)((n + 127) / 128);
    if (blocks == 0) return cudaSuccess;
    batch_down_tables_kernel<<<blocks, 128, 0, st>>>(b, bd);
    return cudaGetLastError();
}

cudaError_t launch_down(const BatchDev& b, const BlenDev& bd, bool blen, bool in_smem, const DownSize& z, int unit0,
                        int unit1, int grid, cudaStream_t st) {
    const Shape sh = dispatch(b.C, in_smem, blen, ShapeOf{blen ? kBlen : kNni, z.warps, z.nodes, z.tips, z.ints});
    return dispatch(b.C, in_smem, blen, LaunchOf{b, bd, sh, unit0, unit1, grid, st});
}

cudaError_t launch_down_reduce(const BatchDev& b, const BlenDev& bd, bool blen, int blocks, cudaStream_t st) {
    if (blocks == 0) return cudaSuccess;
    const int W = down_sites_per_warp(b.C);
    if (blen) batch_down_reduce_kernel<kBlen><<<blocks, 32 * kFoldWarps, 0, st>>>(b, bd, W);
    else batch_down_reduce_kernel<kNni><<<blocks, 32 * kFoldWarps, 0, st>>>(b, bd, W);
    return cudaGetLastError();
}

}  // namespace plk
