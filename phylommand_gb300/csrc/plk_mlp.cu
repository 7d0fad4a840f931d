// The warm-start network: a fully connected ReLU MLP trained and run with
// hand-written kernels (absent in the reference, whose optimiser always starts
// from fixed values, src/treeator.cpp:612-615).
//
//  rows_kernel       (networks up to 256 wide) the whole forward pass, the loss
//                    and the chain of activation gradients of a row block in one
//                    cluster of four CTAs, activations staying on chip.
//  update_kernel     weight and bias gradients of a tile over the whole batch,
//                    and on them, still in registers, the Adam step.
// Wider networks run layer by layer:
//  gemm_tc_kernel    C[M x N] = sum_k A(m, k) B(n, k) with BF16 operands read
//                    through arbitrary strides (so one kernel serves X W^T,
//                    dZ W and dZ^T A), FP32 accumulation in tensor memory
//                    (tcgen05.mma kind::f16), fused epilogue: + bias, ReLU,
//                    ReLU mask of the backward pass, FP32 and/or BF16 stores.
//  loss_kernel       mean squared error over the real outputs and its
//                    gradient (BF16) for the backward GEMMs.
//  colsum_kernel     bias gradients.
//  adam_kernel       Adam (Kingma & Ba 2015) on the FP32 master weights, then
//                    the BF16 copies the GEMMs read.
// Weights are BF16 in every GEMM (the network's storage precision), master
// weights and optimiser moments FP32.  Feature dimensions are padded to 16
// and the batch to 64 with zeros.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_bf16.h>

#include "plk_internal.h"

namespace plk {

namespace {

inline int pad16(int x) { return (x + 15) & ~15; }
inline int pad64(int x) { return (x + 63) & ~63; }

struct GemmArgs {
    const __nv_bfloat16* A;
    long long sa_m, sa_k;
    const __nv_bfloat16* B;
    long long sb_n, sb_k;
    int M, N, K;
    const float* bias;           // [N] or null
    const __nv_bfloat16* mask;   // ReLU mask source (mask(m, n) > 0 keeps), or null
    long long smask_m;           // row stride of mask
    int relu;
    float* Cf;                   // fp32 out or null
    __nv_bfloat16* Cb;           // bf16 out or null
    long long ldc;
};

// loss = mean over rows < n_rows and columns < n_out of (y - t)^2;
// dY = 2 (y - t) / (n_rows n_out) as BF16, zero in the padding
__global__ void loss_kernel(const float* y, int ldy, const float* t, int n_rows, int rows_pad, int n_out, int cols_pad,
                            __nv_bfloat16* dy, float* loss) {
    __shared__ float red[256];
    float s = 0.f;
    const float scale = 2.f / ((float)n_rows * n_out);
    for (int i = threadIdx.x; i < rows_pad * cols_pad; i += blockDim.x) {
        const int r = i / cols_pad, c = i % cols_pad;
        float g = 0.f;
        if (r < n_rows && c < n_out) {
            const float d = y[r * ldy + c] - t[r * n_out + c];
            s += d * d;
            g = scale * d;
        }
        dy[r * cols_pad + c] = __float2bfloat16(g);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / ((float)n_rows * n_out);
}

__global__ void colsum_kernel(const __nv_bfloat16* d, int rows, int cols, int ld, float* out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    float s = 0.f;
    for (int r = 0; r < rows; ++r) s += __bfloat162float(d[r * ld + c]);
    out[c] = s;
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, int n, float lr, float b1, float b2, float eps,
                            float c1, float c2, __nv_bfloat16* pb, int rows, int cols, int ldb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    m[i] = b1 * m[i] + (1.f - b1) * gi;
    v[i] = b2 * v[i] + (1.f - b2) * gi * gi;
    p[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
    if (pb) {
        const int r = i / cols, c = i % cols;
        if (r < rows) pb[r * ldb + c] = __float2bfloat16(p[i]);
    }
}

__global__ void to_bf16_padded(const float* x, int rows, int cols, __nv_bfloat16* out, int rows_pad, int cols_pad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows_pad * cols_pad) return;
    const int r = i / cols_pad, c = i % cols_pad;
    out[i] = __float2bfloat16((r < rows && c < cols) ? x[r * cols + c] : 0.f);
}

// ---------------------------------------------------------------------------
// The same GEMM on Blackwell's fifth-generation tensor cores: a CTA computes a
// 128 x 64 tile of C with tcgen05.mma.kind::f16 (BF16 operands, FP32
// accumulator in TMEM), K in chunks of 64 staged in shared memory in the
// K-major canonical layout without swizzle (8-row x 16-byte core matrices:
// 16 bytes = 8 BF16 along K; A: 128 rows, 2 KB between K-adjacent core
// matrices; B: 32 rows, 512 bytes), four MMAs of K = 16 per chunk issued by one
// thread and completed through an mbarrier (a bounded wait: one that runs
// out turns the tile's outputs NaN, so the loss shows it).  The operands are
// gathered through the same arbitrary strides as gemm_bf16_kernel (rows and
// K beyond the matrix read as zero); the epilogue reads each thread's TMEM
// lane (its row) and applies the same bias / ReLU / mask.
// ---------------------------------------------------------------------------
constexpr int kGM = 128, kGN = 32, kGK = 64;  // N = 32: more CTAs for the network's small GEMMs
constexpr uint32_t kGIdesc = (1u << 4)            // D: F32
                             | (1u << 7)          // A: BF16
                             | (1u << 10)         // B: BF16
                             | ((kGN >> 3) << 17)  // N
                             | ((kGM >> 4) << 24); // M
constexpr int kGWaitLimit = 1 << 20;

__device__ __forceinline__ uint64_t g_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__global__ void __launch_bounds__(128, 1) gemm_tc_kernel(GemmArgs g) {
    __shared__ __align__(128) __nv_bfloat16 As[kGM * kGK];  // [K group 8][row 128][8]
    __shared__ __align__(128) __nv_bfloat16 Bs[kGN * kGK];  // [K group 8][row 32][8]
    __shared__ __align__(8) uint64_t s_mbar;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * kGM, n0 = blockIdx.x * kGN;
    const uint32_t mbar = static_cast<uint32_t>(__cvta_generic_to_shared(&s_mbar));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_tmem))),
                     "r"(kGN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_fail = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t a_base = static_cast<uint32_t>(__cvta_generic_to_shared(As));
    const uint32_t b_base = static_cast<uint32_t>(__cvta_generic_to_shared(Bs));
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    uint32_t phase = 0;
    for (int k0 = 0; k0 < g.K; k0 += kGK) {
        // element (row r, column c) of a chunk at [c / 8][r][c % 8]
        for (int i = tid; i < kGM * kGK; i += 128) {
            const int r = i / kGK, c = i % kGK, m = m0 + r, k = k0 + c;
            As[((c >> 3) * kGM + r) * 8 + (c & 7)] = (m < g.M && k < g.K) ? g.A[m * g.sa_m + k * g.sa_k] : zero;
        }
        for (int i = tid; i < kGN * kGK; i += 128) {
            const int r = i / kGK, c = i % kGK, n = n0 + r, k = k0 + c;
            Bs[((c >> 3) * kGN + r) * 8 + (c & 7)] = (n < g.N && k < g.K) ? g.B[n * g.sb_n + k * g.sb_k] : zero;
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the rows -> the tensor cores
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int ks = 0; ks < kGK / 16; ++ks) {
                const uint64_t ad = g_smem_desc(a_base + ks * 2 * (kGM * 16), kGM * 16, 128);
                const uint64_t bd = g_smem_desc(b_base + ks * 2 * (kGN * 16), kGN * 16, 128);
                const uint32_t accum = (k0 > 0 || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(kGIdesc), "r"(accum));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                         : "memory");
        }
        // the chunk's MMAs done: the accumulator is current and the staged
        // operands may be overwritten (bounded wait)
        bool done = false;
        for (int it = 0; it < kGWaitLimit && !done; ++it) {
            uint32_t ok;
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                "selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(ok)
                : "r"(mbar), "r"(phase)
                : "memory");
            done = ok != 0;
        }
        if (!done) s_fail = 1;
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (s_fail) {
            // the MMAs whose completion was not seen get one more bounded
            // wait before the CTA gives up their TMEM and operands
            for (int it = 0; it < kGWaitLimit; ++it) {
                uint32_t ok;
                asm volatile(
                    "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                    "selp.u32 %0, 1, 0, p;\n}\n"
                    : "=r"(ok)
                    : "r"(mbar), "r"(phase ^ 1u)
                    : "memory");
                if (ok) break;
            }
            break;
        }
    }
    // epilogue: this thread's row m0 + 32 warp + lane is its TMEM lane
    uint32_t r[kGN];
    const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
#pragma unroll
    for (int c = 0; c < kGN / 16; ++c)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
            : "=r"(r[16 * c + 0]), "=r"(r[16 * c + 1]), "=r"(r[16 * c + 2]), "=r"(r[16 * c + 3]),
              "=r"(r[16 * c + 4]), "=r"(r[16 * c + 5]), "=r"(r[16 * c + 6]), "=r"(r[16 * c + 7]),
              "=r"(r[16 * c + 8]), "=r"(r[16 * c + 9]), "=r"(r[16 * c + 10]), "=r"(r[16 * c + 11]),
              "=r"(r[16 * c + 12]), "=r"(r[16 * c + 13]), "=r"(r[16 * c + 14]), "=r"(r[16 * c + 15])
            : "r"(taddr + 16 * c)
            : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    const int m = m0 + 32 * warp + lane;
    const bool fail = s_fail != 0;
    if (m < g.M) {
#pragma unroll
        for (int c = 0; c < kGN; ++c) {
            const int n = n0 + c;
            if (n >= g.N) break;
            float v = fail ? __int_as_float(0x7fc00000) : __uint_as_float(r[c]);
            if (g.bias) v += g.bias[n];
            if (g.relu) v = fmaxf(v, 0.f);
            if (g.mask && !(__bfloat162float(g.mask[m * g.smask_m + n]) > 0.f)) v = 0.f;
            if (g.Cf) g.Cf[m * g.ldc + n] = v;
            if (g.Cb) g.Cb[m * g.ldc + n] = __float2bfloat16(v);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kGN) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Networks whose layers are at most 256 wide: two kernels a training step.
//
// Layer by layer, a step of 43-256-256-256-7 on 256 rows was 25 kernels and 11 clears, the
// GEMMs 30 us each (operands gathered two bytes at a time, K in four waits, 16
// CTAs): 525 us.  Rows do not depend on one another until the weight
// gradients, so rows_kernel takes 128 rows through every layer, forward and
// back, in one cluster of four CTAs.  It is a chain of products with nothing to
// run beside it, so what counts is the latency of a link: each CTA computes a
// quarter of a layer's columns (its weights a contiguous slice of an image
// that update_kernel keeps in the operand's layout, brought in by one bulk
// copy a layer ahead), one thread issues the MMAs, and the epilogue writes the
// BF16 results as a slice of the next layer's A operand (K-major core matrices,
// no swizzle), which one bulk copy each takes to the other CTAs' shared memory
// and their barriers.  One CTA a row block did the same in 56 us a pass, four
// with every thread storing to every CTA and a cluster barrier a layer in 34,
// this in 29.  update_kernel then has a CTA per 128 x 32 tile of every
// weight matrix, the batch as K; its operands are transposed on the way by
// ldmatrix.trans / stmatrix.  A step, with the host's part, 525 -> 65 us.
// Every wait on an mbarrier is bounded.  One that runs out in rows_kernel raises
// `fail`, on which update_kernel leaves the weights as they were, and the host's
// word; one that runs out in update_kernel raises the host's other word (that
// tile's weights stay as they were, other tiles' do not).  The host reads both
// after the pass and reports PLK_ERR_TIMEOUT.
// ---------------------------------------------------------------------------
constexpr int kNetWide = 256;   // widest layer (padded to 16)
constexpr int kNetLayers = 8;   // weight layers
constexpr int kNetThreads = 256;
constexpr int kNetCtas = 4;     // of a row block's cluster
constexpr uint32_t kNetToken = 16;  // bytes a CTA without columns sends
constexpr int kUpN = 32, kUpK = 256;  // update tile: inputs, batch rows per pass

struct NetLayer {
    int in, out, pin, pout;           // real and padded widths
    const __nv_bfloat16* wf;          // image of W (N = out, K = in), see net_image_at
    const __nv_bfloat16* wt;          // image of W^T (N = in, K = out)
    const float* bias;
    __nv_bfloat16 *act, *dz;          // layer input [rows][pin], output gradient [rows][pout]
    size_t w_off, b_off;              // into the flat parameters
    int tiles_n, tile0;               // update_kernel: input tiles, first CTA of the layer
};

struct NetArgs {
    int L, batch, backward, adam;
    NetLayer layer[kNetLayers];
    const float *x, *t;               // [batch][n_in], [batch][n_out]
    float* y;                         // [batch][n_out]
    float* loss_part;                 // [CTAs]
    float* loss;
    int* fail;                        // rows_kernel gave up
    volatile int* gave_up;            // the same for the host [rows_kernel, update_kernel]
    int withhold;                     // test of the failure path (plk_mlp_test_withhold)
    float *p, *g, *m, *v;
    float lr, b1, b2, eps, c1, c2;
};

// Columns a CTA of the cluster takes of N, and where element (n, k) of a
// weight image sits: [CTA][K / 8][columns][8].
__host__ __device__ constexpr int net_share(int N) { return (N / 16 + kNetCtas - 1) / kNetCtas * 16; }
__host__ __device__ constexpr size_t net_image_elems(int N, int K) { return (size_t)kNetCtas * net_share(N) * K; }
__device__ __forceinline__ size_t net_image_at(int n, int k, int N, int K) {
    const int w = net_share(N);
    return ((size_t)(n / w * (K / 8) + (k >> 3)) * w + n % w) * 8 + (k & 7);
}

constexpr int kNetWaitLimit = 1 << 18;  // about a second
__device__ __forceinline__ bool net_wait(uint32_t mbar, uint32_t parity) {
    for (int it = 0; it < kNetWaitLimit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// the MMAs of a K-deep product, A [K / 8][128][8] and B [K / 8][N][8], committed to mbar
__device__ __forceinline__ void net_mma(uint32_t tmem, uint32_t a, uint32_t b, int N, int K, bool first, uint32_t mbar,
                                        bool commit = true) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((kGM >> 4) << 24);
    // one thread issues them: a step of K is an addition to each descriptor's
    // address (16-byte units; the operands lie below 256 KB, so nothing carries)
    uint64_t ad = g_smem_desc(a, kGM * 16, 128), bd = g_smem_desc(b, N * 16, 128);
    uint32_t accum = first ? 0u : 1u;
#pragma unroll 4
    for (int ks = 0; ks < K / 16; ++ks) {
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(accum));
        ad += 2 * kGM;
        bd += 2 * N;
        accum = 1u;
    }
    if (commit)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void net_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void net_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    net_ld16_issue(taddr, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        asm volatile("" : "+r"(r[i]));  // no use ahead of the wait
        v[i] = __uint_as_float(r[i]);
    }
}

__device__ __forceinline__ uint4 net_pack8(const float* v) {
    uint4 o;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    o.x = w[0]; o.y = w[1]; o.z = w[2]; o.w = w[3];
    return o;
}

// TMEM and the mbarriers of a CTA (all threads call it)
constexpr int kNetBars = 5;
__device__ __forceinline__ uint32_t net_begin(uint32_t* s_tmem, uint64_t* s_bar, int cols) {
    const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(s_bar));
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(s_tmem))),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kNetBars; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    return *s_tmem;
}
__device__ __forceinline__ void net_end(uint32_t tmem, int cols) {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(cols) : "memory");
    }
}

constexpr int kRowsA = kGM * kNetWide * 2;                          // one A operand
constexpr int kRowsW = net_share(kNetWide) * kNetWide * 2;          // one weight slice
constexpr int kRowsSmem = 2 * kRowsA + 2 * kRowsW;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__global__ void __cluster_dims__(kNetCtas, 1, 1) __launch_bounds__(kNetThreads, 1)
    rows_kernel(const __grid_constant__ NetArgs n) {
    extern __shared__ __align__(128) unsigned char net_sm[];
    // MMAs done, weights landed (two buffers), the other CTAs' slices of A landed (two)
    __shared__ __align__(8) uint64_t s_bar[kNetBars];
    __shared__ uint32_t s_tmem;
    __shared__ float s_red[kNetThreads];
    __shared__ __align__(16) float s_bias[kNetLayers][net_share(kNetWide)];
    __shared__ __align__(16) unsigned char s_token[kNetToken];  // its contents mean nothing
    __shared__ uint32_t s_pos[kNetLayers][kNetThreads];  // ReLU: the positive ones of a thread's 32 columns
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % kNetCtas, row0 = blockIdx.x / kNetCtas * kGM;
    const uint32_t a_sm = static_cast<uint32_t>(__cvta_generic_to_shared(net_sm)), w_sm = a_sm + 2 * kRowsA;
    const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(s_bar));
    const uint32_t tmem = net_begin(&s_tmem, s_bar, net_share(kNetWide));
    const int L = n.L, steps = n.backward ? 2 * L - 1 : L;
    // step st: layer l forward (st < L) or back (layers L - 1 .. 1)
    auto layer_of = [&](int st) { return st < L ? st : 2 * L - 1 - st; };
    // thread 0: this CTA's slice of step st's weights, in 32 KB copies
    auto load_w = [&](int st) {
        if (n.withhold == 1 && blockIdx.x == kNetCtas - 1 && st == steps - 1) return;
        const NetLayer& ly = n.layer[layer_of(st)];
        const int N = st < L ? ly.pout : ly.pin, K = st < L ? ly.pin : ly.pout;
        const uint32_t bytes = (uint32_t)(net_share(N) * K * 2), to = w_sm + (st & 1) * kRowsW, b = bar + 8 + 8 * (st & 1);
        const char* src = reinterpret_cast<const char*>(st < L ? ly.wf : ly.wt) + (size_t)rank * bytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(b), "r"(bytes) : "memory");
        for (uint32_t off = 0; off < bytes; off += 32768) {
            const uint32_t c = min(32768u, bytes - off);
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(to + off),
                "l"(src + off), "r"(c), "r"(b)
                : "memory");
        }
    };
    if (tid == 0) load_w(0);
    const int r = 32 * (warp & 3) + lane, row = row0 + r;
    // the biases of this CTA's columns, and the targets of this thread's first
    // sixteen outputs: their latency passes beside the inputs'
    float bv[kNetLayers];
#pragma unroll
    for (int l = 0; l < kNetLayers; ++l) {
        const int share = l < L ? net_share(n.layer[l].pout) : 0, c = rank * share + tid;
        bv[l] = l < L && tid < share && c < n.layer[l].out ? n.layer[l].bias[c] : 0.0f;
    }
    float tv[16];
    if (n.backward) {
        const int out = n.layer[L - 1].out, c0 = rank * net_share(n.layer[L - 1].pout) + 16 * (warp >> 2);
#pragma unroll
        for (int j = 0; j < 16; ++j) tv[j] = row < n.batch && c0 + j < out ? n.t[(size_t)row * out + c0 + j] : 0.0f;
    }
    // the rows' inputs as BF16: A operand and, for the weight gradients, the first layer's input
    {
        const NetLayer& l0 = n.layer[0];
        const int chunks = l0.pin / 8, total = kGM * chunks;
        for (int base = tid; base < total; base += 4 * kNetThreads) {
            float v[4][8];  // four chunks' loads in flight: they come over the host link
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = base + u * kNetThreads, rr = i / chunks, c = i % chunks;
                const bool in = i < total && row0 + rr < n.batch;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    v[u][j] = in && 8 * c + j < l0.in ? n.x[(size_t)(row0 + rr) * l0.in + 8 * c + j] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = base + u * kNetThreads, rr = i / chunks, c = i % chunks;
                if (i >= total) break;
                const uint4 o = net_pack8(v[u]);
                *reinterpret_cast<uint4*>(net_sm + ((size_t)c * kGM + rr) * 16) = o;
                if (n.backward && rank == 0 && row0 + rr < n.batch)
                    *reinterpret_cast<uint4*>(l0.act + (size_t)(row0 + rr) * l0.pin + 8 * c) = o;
            }
        }
    }
#pragma unroll
    for (int l = 0; l < kNetLayers; ++l)
        if (tid < net_share(kNetWide)) s_bias[l][tid] = bv[l];
    asm volatile("fence.proxy.async;\n" ::: "memory");  // the A rows -> the tensor cores
    cluster_barrier();  // every CTA of the cluster runs before anything is written into it
    const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    float sq = 0.0f;
    uint32_t mma_phase = 0;
    // failed: a wait ran out; the CTA then multiplies and loads no more but keeps
    // step, as the others wait for its slices.  loaded: this step's weights were asked for.
    bool failed = false, loaded = true;
    for (int st = 0; st < steps; ++st) {
        const bool fwd = st < L, last = st == L - 1;
        const int l = layer_of(st);
        const NetLayer& ly = n.layer[l];
        const int N = fwd ? ly.pout : ly.pin, K = fwd ? ly.pin : ly.pout, share = net_share(N), n0 = rank * share;
        if (loaded && !net_wait(bar + 8 + 8 * (st & 1), (st >> 1) & 1)) {
            net_wait(bar + 8 + 8 * (st & 1), (st >> 1) & 1);  // a last bounded wait for the copy in flight
            failed = true;
        }
        if (st > 0 && !net_wait(bar + 24 + 8 * (st & 1), ((st - 1) >> 1) & 1)) {
            net_wait(bar + 24 + 8 * (st & 1), ((st - 1) >> 1) & 1);
            failed = true;
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        failed = __syncthreads_or(failed) != 0;
        loaded = !failed;
        const bool go = !failed && n0 < N;  // a CTA past the last columns only keeps step
        if (go && tid == 0) {
            asm volatile("fence.proxy.async;\n" ::: "memory");
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            net_mma(tmem, a_sm + (st & 1) * kRowsA, w_sm + (st & 1) * kRowsW, share, K, true, bar);
        }
        // the other buffer's products were waited for in the step before
        if (tid == 32 && st + 1 < steps && loaded) load_w(st + 1);
        bool done = false;
        if (go) {
            done = net_wait(bar, mma_phase) || net_wait(bar, mma_phase);
            if (!done) failed = true;
            mma_phase ^= 1u;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // this thread's row: its half of the CTA's columns
        const bool all_done = __all_sync(0xffffffffu, done);
        uint32_t acc[2][16];
        if (all_done) {
            net_ld16_issue(trow + 16 * (warp >> 2), acc[0]);
            net_ld16_issue(trow + 16 * (warp >> 2) + 32, acc[1]);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int cl = 16 * (warp >> 2) + 32 * q, c0 = n0 + cl;  // in the CTA's columns, in the layer's
            if (cl >= share || c0 >= N || !all_done) continue;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                asm volatile("" : "+r"(acc[q][j]));  // no use ahead of the wait
                v[j] = __uint_as_float(acc[q][j]);
            }
            if (fwd) {
                uint32_t pos = 0;
#pragma unroll
                for (int j = 0; j < 16; j += 4) {  // past the width the products and the biases are zero
                    const float4 b4 = *reinterpret_cast<const float4*>(&s_bias[l][cl + j]);
                    v[j] += b4.x;
                    v[j + 1] += b4.y;
                    v[j + 2] += b4.z;
                    v[j + 3] += b4.w;
                }
                if (!last)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f);
                if (!last && n.backward) {
                    // what the gradient lets through: the output as it is stored
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (__bfloat162float(__float2bfloat16(v[j])) > 0.0f) pos |= 1u << j;
                    s_pos[l][tid] = q == 0 ? pos : (s_pos[l][tid] | (pos << 16));
                }
            } else {
                const uint32_t pos = s_pos[l - 1][tid] >> (16 * q);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (!((pos >> j) & 1u)) v[j] = 0.0f;
            }
            if (last) {
                const float scale = 2.f / ((float)n.batch * ly.out);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float gr = 0.0f;
                    if (row < n.batch && c0 + j < ly.out) {
                        if (n.y) n.y[(size_t)row * ly.out + c0 + j] = v[j];
                        if (n.backward) {
                            const float d = v[j] - (q == 0 ? tv[j] : n.t[(size_t)row * ly.out + c0 + j]);
                            sq += d * d;
                            gr = scale * d;
                        }
                    }
                    v[j] = gr;
                }
            }
            const uint4 o0 = net_pack8(v), o1 = net_pack8(v + 8);
            if (st + 1 < steps) {
                // this CTA's slice of the next step's A operand
                unsigned char* at = net_sm + ((st + 1) & 1) * kRowsA + ((c0 / 8) * kGM + r) * 16;
                *reinterpret_cast<uint4*>(at) = o0;
                *reinterpret_cast<uint4*>(at + kGM * 16) = o1;
            }
            if (n.backward && row < n.batch) {
                // a layer's output is the next one's input; its gradient that of the layer below
                __nv_bfloat16* dst = last ? ly.dz : (fwd ? n.layer[l + 1].act : n.layer[l - 1].dz);
                uint4* g = reinterpret_cast<uint4*>(dst + (size_t)row * N + c0);
                g[0] = o0;
                g[1] = o1;
            }
        }
        // the slice to the other CTAs, or a token from one without columns; theirs
        // arrive on this one's barrier.  So a CTA reaches this point only when
        // every other one has been here in the step before: their products that
        // read the buffer are done, and their barrier, which serves every other
        // step, is in this step's phase.  (Remote arrivals instead of tokens cost
        // 5 % of a training step: three more cluster operations a layer.)
        asm volatile("fence.proxy.async;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (tid == 0 && st + 1 < steps) {
            const int own = max(0, min(share, N - n0)), idle = kNetCtas - (N + share - 1) / share;  // CTAs without columns
            const uint32_t b = bar + 24 + 8 * ((st + 1) & 1), bytes = own > 0 ? (uint32_t)own * kGM * 2 : kNetToken;
            const uint32_t at = own > 0 ? a_sm + ((st + 1) & 1) * kRowsA + (uint32_t)(n0 / 8 * kGM) * 16
                                        : static_cast<uint32_t>(__cvta_generic_to_shared(s_token));
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(b),
                         "r"((uint32_t)(N - own) * kGM * 2 + (idle - (own > 0 ? 0 : 1)) * kNetToken)
                         : "memory");
            for (int d = 1; d < kNetCtas; ++d) {
                const int cta = (rank + d) % kNetCtas;
                uint32_t to, tb;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(to) : "r"(at), "r"(cta));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(tb) : "r"(b), "r"(cta));
                asm volatile(
                    "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(to),
                    "r"(at), "r"(bytes), "r"(tb)
                    : "memory");
            }
        }
    }
    cluster_barrier();  // every copy from and into this CTA's shared memory has landed
    if (__syncthreads_or(failed) && tid == 0) *n.fail = n.gave_up[0] = 1;
    if (n.backward) {
        s_red[tid] = sq;
        __syncthreads();
        for (int off = kNetThreads / 2; off > 0; off >>= 1) {
            if (tid < off) s_red[tid] += s_red[tid + off];
            __syncthreads();
        }
        if (tid == 0) n.loss_part[blockIdx.x] = s_red[0];
    }
    net_end(tmem, net_share(kNetWide));
}

// Shared memory of update_kernel: the row-major tiles (rows padded by 16 bytes
// against bank conflicts), then the operands [K / 8][rows][8].
constexpr int kUpPitchA = kGM * 2 + 16, kUpPitchB = kUpN * 2 + 16;
constexpr int kUpStageA = kUpK * kUpPitchA, kUpStageB = kUpK * kUpPitchB;
constexpr int kUpOpA = kUpK * kGM * 2, kUpOpB = kUpK * kUpN * 2;
constexpr int kUpSmem = kUpOpA + kUpOpB + kUpStageA + kUpStageB;

// 8 x 8 blocks of src (row-major [k][columns], `pitch` bytes a row) into dst
// ([k / 8][columns][8]): four blocks of neighbouring columns an instruction
__device__ __forceinline__ void net_transpose(uint32_t src, int pitch, uint32_t dst, int cols, int k) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quads = cols / 32, n = k / 8 * quads;
    for (int i = warp; i < n; i += kNetThreads / 32) {
        const int kg = i / quads, col = (i % quads) * 32 + (lane >> 3) * 8, r = lane & 7;
        const uint32_t s = src + (uint32_t)((8 * kg + r) * pitch + col * 2);
        const uint32_t d = dst + (uint32_t)((kg * cols + col + r) * 16);
        uint32_t x[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
                     : "r"(s)
                     : "memory");
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(d), "r"(x[0]), "r"(x[1]),
                     "r"(x[2]), "r"(x[3])
                     : "memory");
    }
}

// rows [k0, k0 + kUpK) of src ([rows][width]), columns [c0, c0 + cols), zero past the batch and the width
template <int COLS>
__device__ __forceinline__ void net_stage(unsigned char* dst, int pitch, const __nv_bfloat16* src, int width, int c0,
                                          int k0, int batch) {
    constexpr int chunks = COLS / 8;
    const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
#pragma unroll
    for (int i0 = 0; i0 < kUpK * chunks; i0 += kNetThreads) {
        const int r = (i0 + threadIdx.x) / chunks, c = threadIdx.x % chunks;
        const bool in = k0 + r < batch && c0 + 8 * c < width;
        const __nv_bfloat16* from = in ? src + (size_t)(k0 + r) * width + c0 + 8 * c : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to + r * pitch + 16 * c), "l"(from),
                     "r"(in ? 16 : 0)
                     : "memory");
    }
}

// one Adam update of a parameter from its gradient, every rounding spelt out
// (those adam_kernel's expressions compile to): training amplifies a last bit
__device__ __forceinline__ void net_adam(const NetArgs& n, float gi, float& p, float& m, float& v) {
    m = fmaf(__fsub_rn(1.f, n.b1), gi, __fmul_rn(n.b1, m));
    v = fmaf(__fmul_rn(__fsub_rn(1.f, n.b2), gi), gi, __fmul_rn(n.b2, v));
    p -= n.lr * (m / n.c1) / (sqrtf(v / n.c2) + n.eps);
}

__global__ void __launch_bounds__(kNetThreads, 1) update_kernel(const __grid_constant__ NetArgs n, int row_ctas) {
    extern __shared__ __align__(128) unsigned char net_sm[];
    __shared__ __align__(8) uint64_t s_bar[kNetBars];
    __shared__ uint32_t s_tmem;
    if (*n.fail) return;  // a row block gave up (nothing in this launch writes the flag): no update
    int l = 0;
    while (l + 1 < n.L && (int)blockIdx.x >= n.layer[l + 1].tile0) ++l;
    const NetLayer& ly = n.layer[l];
    const int t = blockIdx.x - ly.tile0, m0 = t / ly.tiles_n * kGM, n0 = t % ly.tiles_n * kUpN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *stA = net_sm + kUpOpA + kUpOpB, *stB = stA + kUpStageA;
    const uint32_t a_sm = static_cast<uint32_t>(__cvta_generic_to_shared(net_sm));
    const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(s_bar));
    const uint32_t tmem = net_begin(&s_tmem, s_bar, kUpN);
    float bias = 0.0f;  // thread o < 128 of the tiles with n0 = 0: the bias gradient of output m0 + o
    bool ok = true;
    uint32_t phase = 0;
    for (int k0 = 0; k0 < n.batch; k0 += kUpK, phase ^= 1u) {
        net_stage<kGM>(stA, kUpPitchA, ly.dz, ly.pout, m0, k0, n.batch);
        net_stage<kUpN>(stB, kUpPitchB, ly.act, ly.pin, n0, k0, n.batch);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        const int K = (min(kUpK, n.batch - k0) + 15) / 16 * 16;
        net_transpose(a_sm + kUpOpA + kUpOpB, kUpPitchA, a_sm, kGM, K);
        net_transpose(a_sm + kUpOpA + kUpOpB + kUpStageA, kUpPitchB, a_sm + kUpOpA, kUpN, K);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            net_mma(tmem, a_sm, a_sm + kUpOpA, kUpN, K, k0 == 0, bar, n.withhold != 2 || blockIdx.x + 1 < gridDim.x);
        }
        if (n0 == 0 && tid < kGM)
#pragma unroll 16
            for (int r = 0; r < K; ++r)
                bias += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(stA + (size_t)r * kUpPitchA + 2 * tid));
        const bool done = net_wait(bar, phase) || net_wait(bar, phase);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        ok = __syncthreads_and(done) != 0;
        if (!ok) break;
    }
    // the tile's gradient through shared memory, so that the parameters and
    // moments go by whole rows of 32 (a thread a row of sixteen touched 32 rows
    // an instruction: 12 of the kernel's 21 us)
    float* const s_g = reinterpret_cast<float*>(stA);                                   // [128][33]
    __nv_bfloat16* const s_h = reinterpret_cast<__nv_bfloat16*>(stB);                   // [128][40]
    {
        float v[16];
        net_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 16 * (warp >> 2), v);
#pragma unroll
        for (int j = 0; j < 16; ++j) s_g[(32 * (warp & 3) + lane) * 33 + 16 * (warp >> 2) + j] = v[j];
    }
    __syncthreads();
    if (ok) {
        constexpr int kRows = kGM / (kNetThreads / 32);  // rows of a warp
        const int c = n0 + lane;
        const size_t at = ly.w_off + (size_t)(m0 + warp) * ly.in + c, step = (size_t)(kNetThreads / 32) * ly.in;
        if (n.adam) {
            float p[kRows], m[kRows], v[kRows];
            bool in[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                in[i] = c < ly.in && m0 + warp + 8 * i < ly.out;
                p[i] = m[i] = v[i] = 0.0f;
                if (in[i]) {
                    p[i] = n.p[at + i * step];
                    m[i] = n.m[at + i * step];
                    v[i] = n.v[at + i * step];
                }
            }
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                if (in[i]) {
                    net_adam(n, s_g[(warp + 8 * i) * 33 + lane], p[i], m[i], v[i]);
                    n.p[at + i * step] = p[i];
                    n.m[at + i * step] = m[i];
                    n.v[at + i * step] = v[i];
                }
                s_h[(warp + 8 * i) * 40 + lane] = __float2bfloat16(p[i]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < kRows; ++i)
                if (c < ly.in && m0 + warp + 8 * i < ly.out) n.g[at + i * step] = s_g[(warp + 8 * i) * 33 + lane];
        }
    }
    __syncthreads();
    if (ok && n.adam) {
        // the images, eight weights at a time (shares and tiles are multiples of eight)
        __nv_bfloat16* wf = const_cast<__nv_bfloat16*>(ly.wf);
        __nv_bfloat16* wt = const_cast<__nv_bfloat16*>(ly.wt);
        for (int i = tid; i < kGM * (kUpN / 8); i += kNetThreads) {
            const int o = i % kGM, c8 = i / kGM * 8;
            if (m0 + o < ly.pout && n0 + c8 < ly.pin)
                *reinterpret_cast<uint4*>(wf + net_image_at(m0 + o, n0 + c8, ly.pout, ly.pin)) =
                    *reinterpret_cast<const uint4*>(s_h + o * 40 + c8);
            const int c = i % kUpN, o8 = i / kUpN * 8;
            if (m0 + o8 < ly.pout && n0 + c < ly.pin) {
                __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) h[j] = s_h[(o8 + j) * 40 + c];
                *reinterpret_cast<uint4*>(wt + net_image_at(n0 + c, m0 + o8, ly.pin, ly.pout)) =
                    *reinterpret_cast<const uint4*>(h);
            }
        }
    }
    if (ok && n0 == 0 && tid < kGM && m0 + tid < ly.out) {
        const size_t i = ly.b_off + m0 + tid;
        if (n.adam) {
            float p = n.p[i], m = n.m[i], vv = n.v[i];
            net_adam(n, bias, p, m, vv);
            n.p[i] = p;
            n.m[i] = m;
            n.v[i] = vv;
        } else {
            n.g[i] = bias;
        }
    }
    if (tid == 0 && !ok) n.gave_up[1] = 1;
    if (blockIdx.x == 0 && tid == 0) {
        float s = 0.0f;
        for (int i = 0; i < row_ctas; ++i) s += n.loss_part[i];
        const NetLayer& top = n.layer[n.L - 1];
        *n.loss = s / ((float)n.batch * top.out);
    }
    net_end(tmem, kUpN);
}

// both images of one layer's weights from the FP32 parameters, zero in the padding
__global__ void pack_images_kernel(const float* w, int in, int out, int pin, int pout, __nv_bfloat16* wf,
                                   __nv_bfloat16* wt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pin * pout) return;
    const int o = i / pin, c = i % pin;
    const __nv_bfloat16 h = __float2bfloat16(o < out && c < in ? w[(size_t)o * in + c] : 0.0f);
    wf[net_image_at(o, c, pout, pin)] = h;
    wt[net_image_at(c, o, pin, pout)] = h;
}

cudaError_t gemm(const GemmArgs& g, cudaStream_t st) {
    dim3 grid((g.N + kGN - 1) / kGN, (g.M + kGM - 1) / kGM);
    gemm_tc_kernel<<<grid, 128, 0, st>>>(g);
    return cudaGetLastError();
}

}  // namespace
}  // namespace plk

using namespace plk;

struct plk_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    std::vector<int> dims;      // real sizes: n_in, hidden..., n_out
    std::vector<int> pdims;     // padded to 16
    std::vector<size_t> w_off, b_off;  // offsets of each layer's W [out x in] and b [out] in the flat vector
    size_t n_params = 0;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // FP32 master, gradient, Adam moments
    std::vector<__nv_bfloat16*> wb;   // BF16 weight copies [pout x pin]
    int batch_cap = 0;
    std::vector<__nv_bfloat16*> act;  // BF16 activations [batch_pad x pdims[l]]
    std::vector<float*> pre;          // FP32 layer outputs [batch_pad x pdims[l]]
    __nv_bfloat16 *dz = nullptr, *dz2 = nullptr;
    float *xin = nullptr, *tin = nullptr, *loss = nullptr;
    long long step = 0;
    // networks up to kNetWide wide (rows_kernel, update_kernel): the weight
    // images, the layers' inputs and gradients [cap rows], row blocks' losses,
    // and a pinned block the kernels read the rows from and write the loss to
    bool narrow = false;
    std::vector<__nv_bfloat16*> wf, wt, n_act, n_dz;
    int n_cap = 0;
    float *loss_part = nullptr, *y_dev = nullptr;
    int* fail = nullptr;
    char *host = nullptr, *host_dev = nullptr;
    size_t host_bytes = 0;
    int withhold = 0;  // armed by plk_mlp_test_withhold for the next pass
    ~plk_mlp() {
        for (auto* v : {&wf, &wt, &n_act, &n_dz})
            for (auto* q : *v) cudaFree(q);
        cudaFree(loss_part); cudaFree(y_dev); cudaFree(fail);
        if (host) cudaFreeHost(host);
        cudaFree(p); cudaFree(g); cudaFree(m); cudaFree(v);
        for (auto* q : wb) cudaFree(q);
        for (auto* q : act) cudaFree(q);
        for (auto* q : pre) cudaFree(q);
        cudaFree(dz); cudaFree(dz2); cudaFree(xin); cudaFree(tin); cudaFree(loss);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

plk_status mfail(plk_mlp* m, plk_status s, const std::string& msg) {
    if (m) m->err = msg;
    else report_error(s, msg);
    return s;
}

#define PLK_MCUDA(m, expr, what)                                                                        \
    do {                                                                                                \
        cudaError_t _e = (expr);                                                                        \
        if (_e != cudaSuccess) {                                                                        \
            cudaGetLastError(); /* reported here, not by the next launch */                             \
            return mfail(m, _e == cudaErrorMemoryAllocation ? PLK_ERR_ALLOC : PLK_ERR_CUDA,              \
                         std::string(what) + ": " + cudaGetErrorString(_e));                            \
        }                                                                                               \
    } while (0)

int n_layers(const plk_mlp* m) { return (int)m->dims.size() - 1; }

plk_status ensure_batch(plk_mlp* m, int batch) {
    const int bp = pad64(batch);
    if (bp <= m->batch_cap) return PLK_OK;
    for (auto* q : m->act) cudaFree(q);
    for (auto* q : m->pre) cudaFree(q);
    m->act.assign(m->dims.size(), nullptr);
    m->pre.assign(m->dims.size(), nullptr);
    cudaFree(m->dz); cudaFree(m->dz2); cudaFree(m->xin); cudaFree(m->tin);
    int widest = 0;
    for (size_t l = 0; l < m->dims.size(); ++l) {
        widest = std::max(widest, m->pdims[l]);
        PLK_MCUDA(m, cudaMalloc(&m->act[l], (size_t)bp * m->pdims[l] * sizeof(__nv_bfloat16)), "allocate activations");
        PLK_MCUDA(m, cudaMalloc(&m->pre[l], (size_t)bp * m->pdims[l] * sizeof(float)), "allocate activations");
    }
    PLK_MCUDA(m, cudaMalloc(&m->dz, (size_t)bp * widest * sizeof(__nv_bfloat16)), "allocate gradients");
    PLK_MCUDA(m, cudaMalloc(&m->dz2, (size_t)bp * widest * sizeof(__nv_bfloat16)), "allocate gradients");
    PLK_MCUDA(m, cudaMalloc(&m->xin, (size_t)bp * m->dims.front() * sizeof(float)), "allocate inputs");
    PLK_MCUDA(m, cudaMalloc(&m->tin, (size_t)bp * m->dims.back() * sizeof(float)), "allocate targets");
    m->batch_cap = bp;
    return PLK_OK;
}

// ---- networks up to kNetWide wide --------------------------------------------
// Rows larger than this are copied to the device instead of read in place from the
// pinned block: forward of 205 inputs, in place and copied, 109 KB 39 and 45 us, 320 KB
// 43 and 43 (32 inputs), 876 KB 87 and 50, 3.4 MB 289 and 75.
constexpr size_t kHostRows = 320 << 10;

plk_status net_images(plk_mlp* m) {
    PLK_MCUDA(m, cudaStreamSynchronize(nullptr), "upload weights");  // copied on the default stream
    for (int l = 0; l < n_layers(m); ++l) {
        const int n = m->pdims[l] * m->pdims[l + 1];
        pack_images_kernel<<<(n + 255) / 256, 256, 0, m->stream>>>(m->p + m->w_off[l], m->dims[l], m->dims[l + 1],
                                                                  m->pdims[l], m->pdims[l + 1], m->wf[l], m->wt[l]);
    }
    PLK_MCUDA(m, cudaGetLastError(), "weight images");
    PLK_MCUDA(m, cudaStreamSynchronize(m->stream), "weight images");
    return PLK_OK;
}

// Room for `batch` rows, and the pinned block: [loss, the kernels' gave-up
// words][x][t], read and written by the kernels in place.
plk_status net_ensure(plk_mlp* m, int batch, bool train) {
    const int rows = (batch + kGM - 1) / kGM * kGM;
    const size_t xb = (size_t)batch * m->dims.front() * sizeof(float), tb = (size_t)batch * m->dims.back() * sizeof(float);
    const size_t want = 256 + (xb + tb <= kHostRows ? (xb + 255) / 256 * 256 + tb : 0);
    if (want > m->host_bytes) {
        if (m->host) cudaFreeHost(m->host);
        m->host = nullptr;
        m->host_bytes = 0;
        PLK_MCUDA(m, cudaHostAlloc(&m->host, want, cudaHostAllocMapped), "allocate pinned rows");
        void* d = nullptr;
        PLK_MCUDA(m, cudaHostGetDevicePointer(&d, m->host, 0), "pinned rows");
        m->host_dev = static_cast<char*>(d);
        m->host_bytes = want;
    }
    if (!m->fail) {
        PLK_MCUDA(m, cudaMalloc(&m->fail, sizeof(int)), "allocate flag");
        PLK_MCUDA(m, cudaMemsetAsync(m->fail, 0, sizeof(int), m->stream), "clear flag");
    }
    if (rows > m->n_cap) {
        for (auto* v : {&m->n_act, &m->n_dz}) {
            for (auto* q : *v) cudaFree(q);
            v->clear();
        }
        cudaFree(m->loss_part); cudaFree(m->y_dev); cudaFree(m->xin); cudaFree(m->tin);
        m->loss_part = m->y_dev = m->xin = m->tin = nullptr;
        m->n_cap = 0;
        PLK_MCUDA(m, cudaMalloc(&m->loss_part, rows / kGM * kNetCtas * sizeof(float)), "allocate losses");
        PLK_MCUDA(m, cudaMalloc(&m->y_dev, (size_t)rows * m->dims.back() * sizeof(float)), "allocate outputs");
        PLK_MCUDA(m, cudaMalloc(&m->xin, (size_t)rows * m->dims.front() * sizeof(float)), "allocate inputs");
        PLK_MCUDA(m, cudaMalloc(&m->tin, (size_t)rows * m->dims.back() * sizeof(float)), "allocate targets");
        m->n_cap = rows;
    }
    if (train && m->n_act.empty()) {
        // all of them or none: a later pass takes what is there for whole, and a
        // smaller batch may fit where this one did not
        m->n_act.assign(n_layers(m), nullptr);
        m->n_dz.assign(n_layers(m), nullptr);
        cudaError_t e = cudaSuccess;
        for (int l = 0; e == cudaSuccess && l < n_layers(m); ++l) {
            e = cudaMalloc(&m->n_act[l], (size_t)m->n_cap * m->pdims[l] * sizeof(__nv_bfloat16));
            if (e == cudaSuccess) e = cudaMalloc(&m->n_dz[l], (size_t)m->n_cap * m->pdims[l + 1] * sizeof(__nv_bfloat16));
        }
        if (e != cudaSuccess) {
            for (auto* v : {&m->n_act, &m->n_dz}) {
                for (auto* q : *v) cudaFree(q);
                v->clear();
            }
            m->n_cap = 0;
            PLK_MCUDA(m, e, "allocate activations and gradients");
        }
    }
    return PLK_OK;
}

// One pass over `batch` rows: forward (t null), gradients, or an Adam step.
// The loss is in the pinned block once the stream has drained (net_finish).
plk_status net_pass(plk_mlp* m, int batch, const float* x, const float* t, bool adam, float lr, float* y_dev) {
    plk_status s = net_ensure(m, batch, t != nullptr);
    if (s != PLK_OK) return s;
    const int L = n_layers(m);
    const size_t xb = (size_t)batch * m->dims.front() * sizeof(float), tb = (size_t)batch * m->dims.back() * sizeof(float);
    NetArgs n{};
    n.L = L;
    n.batch = batch;
    n.backward = t != nullptr;
    n.adam = adam;
    if (xb + tb <= kHostRows) {
        char* xs = m->host + 256;
        char* ts = xs + (xb + 255) / 256 * 256;
        std::memcpy(xs, x, xb);
        if (t) std::memcpy(ts, t, tb);
        n.x = reinterpret_cast<const float*>(m->host_dev + (xs - m->host));
        n.t = reinterpret_cast<const float*>(m->host_dev + (ts - m->host));
    } else {
        PLK_MCUDA(m, cudaMemcpyAsync(m->xin, x, xb, cudaMemcpyHostToDevice, m->stream), "upload inputs");
        if (t) PLK_MCUDA(m, cudaMemcpyAsync(m->tin, t, tb, cudaMemcpyHostToDevice, m->stream), "upload targets");
        n.x = m->xin;
        n.t = m->tin;
    }
    n.y = y_dev;
    n.loss_part = m->loss_part;
    n.loss = reinterpret_cast<float*>(m->host_dev);
    n.fail = m->fail;
    n.gave_up = reinterpret_cast<int*>(m->host_dev) + 1;
    reinterpret_cast<int*>(m->host)[1] = reinterpret_cast<int*>(m->host)[2] = 0;
    n.withhold = m->withhold;
    m->withhold = 0;
    n.p = m->p; n.g = m->g; n.m = m->m; n.v = m->v;
    int tiles = 0;
    for (int l = 0; l < L; ++l) {
        NetLayer& ly = n.layer[l];
        ly.in = m->dims[l]; ly.out = m->dims[l + 1]; ly.pin = m->pdims[l]; ly.pout = m->pdims[l + 1];
        ly.wf = m->wf[l]; ly.wt = m->wt[l];
        ly.bias = m->p + m->b_off[l];
        ly.w_off = m->w_off[l]; ly.b_off = m->b_off[l];
        if (t) { ly.act = m->n_act[l]; ly.dz = m->n_dz[l]; }
        ly.tiles_n = (ly.in + kUpN - 1) / kUpN;
        ly.tile0 = tiles;
        tiles += ly.tiles_n * ((ly.out + kGM - 1) / kGM);
    }
    const int row_ctas = (batch + kGM - 1) / kGM * kNetCtas;
    rows_kernel<<<row_ctas, kNetThreads, kRowsSmem, m->stream>>>(n);
    PLK_MCUDA(m, cudaGetLastError(), "row kernel");
    if (!t) return PLK_OK;
    if (n.adam) {
        ++m->step;
        n.lr = lr;
        n.b1 = 0.9f; n.b2 = 0.999f; n.eps = 1e-8f;
        n.c1 = 1.f - std::pow(n.b1, (float)m->step);
        n.c2 = 1.f - std::pow(n.b2, (float)m->step);
    }
    update_kernel<<<tiles, kNetThreads, kUpSmem, m->stream>>>(n, row_ctas);
    PLK_MCUDA(m, cudaGetLastError(), "update kernel");
    return PLK_OK;
}

// Waits for the last pass (`trained`: one with an Adam step) and gives its loss,
// or PLK_ERR_TIMEOUT where a kernel gave up, with the flag cleared for the next.
plk_status net_finish(plk_mlp* m, bool trained, const char* what, float* loss) {
    if (loss) *loss = NAN;
    PLK_MCUDA(m, cudaStreamSynchronize(m->stream), what);
    const volatile int* gave_up = reinterpret_cast<const volatile int*>(m->host) + 1;
    if (gave_up[0]) {
        if (trained) --m->step;  // no update was made
        PLK_MCUDA(m, cudaMemsetAsync(m->fail, 0, sizeof(int), m->stream), "clear flag");
        return mfail(m, PLK_ERR_TIMEOUT, std::string(what) + ": a bounded wait of the row kernel ran out");
    }
    if (gave_up[1])
        return mfail(m, PLK_ERR_TIMEOUT, std::string(what) + ": a bounded wait of the update kernel ran out" +
                                             (trained ? "; only a part of the weights was updated" : ""));
    if (loss) *loss = *reinterpret_cast<const volatile float*>(m->host);
    return PLK_OK;
}

plk_status refresh_bf16(plk_mlp* m) {
    if (m->narrow) return net_images(m);
    // BF16 copies of every layer's weights from the FP32 master
    std::vector<float> host(m->n_params);
    PLK_MCUDA(m, cudaMemcpy(host.data(), m->p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost), "read weights");
    for (int l = 0; l < n_layers(m); ++l) {
        const int in = m->dims[l], out = m->dims[l + 1], pin = m->pdims[l], pout = m->pdims[l + 1];
        std::vector<__nv_bfloat16> w((size_t)pout * pin, __float2bfloat16(0.f));
        for (int r = 0; r < out; ++r)
            for (int c = 0; c < in; ++c) w[(size_t)r * pin + c] = __float2bfloat16(host[m->w_off[l] + (size_t)r * in + c]);
        PLK_MCUDA(m, cudaMemcpy(m->wb[l], w.data(), w.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice),
                  "upload weights");
    }
    return PLK_OK;
}

// forward of `batch` rows already in m->xin; leaves layer outputs in pre/act
plk_status forward(plk_mlp* m, int batch) {
    const int bp = pad64(batch);
    const int L = n_layers(m);
    const int total = bp * m->pdims[0];
    to_bf16_padded<<<(total + 255) / 256, 256, 0, m->stream>>>(m->xin, batch, m->dims[0], m->act[0], bp, m->pdims[0]);
    PLK_MCUDA(m, cudaGetLastError(), "input conversion");
    for (int l = 0; l < L; ++l) {
        GemmArgs ga{};
        ga.A = m->act[l]; ga.sa_m = m->pdims[l]; ga.sa_k = 1;
        ga.B = m->wb[l]; ga.sb_n = m->pdims[l]; ga.sb_k = 1;
        ga.M = bp; ga.N = m->pdims[l + 1]; ga.K = m->pdims[l];
        ga.bias = m->p + m->b_off[l];
        ga.relu = l < L - 1;
        ga.Cf = m->pre[l + 1];
        ga.Cb = m->act[l + 1];
        ga.ldc = m->pdims[l + 1];
        // the padded output columns beyond the real width carry bias reads;
        // restrict N to the real width and keep the padding zero
        ga.N = m->dims[l + 1];
        PLK_MCUDA(m, cudaMemsetAsync(m->act[l + 1], 0, (size_t)bp * m->pdims[l + 1] * sizeof(__nv_bfloat16), m->stream),
                  "clear activations");
        PLK_MCUDA(m, cudaMemsetAsync(m->pre[l + 1], 0, (size_t)bp * m->pdims[l + 1] * sizeof(float), m->stream),
                  "clear activations");
        PLK_MCUDA(m, gemm(ga, m->stream), "forward GEMM");
    }
    return PLK_OK;
}

// gradients of the mean squared error into m->g; loss into m->loss
plk_status backward(plk_mlp* m, int batch) {
    const int bp = pad64(batch);
    const int L = n_layers(m);
    loss_kernel<<<1, 256, 0, m->stream>>>(m->pre[L], m->pdims[L], m->tin, batch, bp, m->dims[L], m->pdims[L], m->dz,
                                          m->loss);
    PLK_MCUDA(m, cudaGetLastError(), "loss kernel");
    __nv_bfloat16* dz = m->dz;
    __nv_bfloat16* dn = m->dz2;
    for (int l = L - 1; l >= 0; --l) {
        const int in = m->dims[l], out = m->dims[l + 1], pin = m->pdims[l], pout = m->pdims[l + 1];
        // dW[out x in] = dZ^T A_prev
        GemmArgs gw{};
        gw.A = dz; gw.sa_m = 1; gw.sa_k = pout;
        gw.B = m->act[l]; gw.sb_n = 1; gw.sb_k = pin;
        gw.M = out; gw.N = in; gw.K = batch;
        gw.Cf = m->g + m->w_off[l];
        gw.ldc = in;
        PLK_MCUDA(m, gemm(gw, m->stream), "weight-gradient GEMM");
        colsum_kernel<<<(out + 127) / 128, 128, 0, m->stream>>>(dz, batch, out, pout, m->g + m->b_off[l]);
        PLK_MCUDA(m, cudaGetLastError(), "bias gradient");
        if (l > 0) {
            // dA_prev[B x in] = dZ W, masked by ReLU of layer l's input
            GemmArgs gd{};
            gd.A = dz; gd.sa_m = pout; gd.sa_k = 1;
            gd.B = m->wb[l]; gd.sb_n = 1; gd.sb_k = pin;
            gd.M = bp; gd.N = in; gd.K = out;
            gd.mask = m->act[l]; gd.smask_m = pin;
            gd.Cb = dn;
            gd.ldc = pin;
            PLK_MCUDA(m, cudaMemsetAsync(dn, 0, (size_t)bp * pin * sizeof(__nv_bfloat16), m->stream), "clear gradients");
            PLK_MCUDA(m, gemm(gd, m->stream), "activation-gradient GEMM");
            std::swap(dz, dn);
        }
    }
    return PLK_OK;
}

// SplitMix64 stream for the initial weights
uint64_t sm64(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace

extern "C" {

plk_status plk_mlp_create(plk_mlp** out, int device, int n_in, int n_hidden, int n_hidden_layers, int n_out,
                          uint64_t seed) {
    if (!out) return report_error(PLK_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (n_in < 1 || n_hidden < 1 || n_hidden_layers < 0 || n_out < 1)
        return report_error(PLK_ERR_ARG, "bad network sizes");
    int nd = 0;
    if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) return report_error(PLK_ERR_NODEV, "no CUDA device");
    if (device < 0 || device >= nd) return report_error(PLK_ERR_ARG, "device index out of range");
    cudaSetDevice(device);
    plk_mlp* m = new (std::nothrow) plk_mlp();
    if (!m) return report_error(PLK_ERR_ALLOC, "host allocation failed");
    m->device = device;
    m->dims.push_back(n_in);
    for (int i = 0; i < n_hidden_layers; ++i) m->dims.push_back(n_hidden);
    m->dims.push_back(n_out);
    for (int d : m->dims) m->pdims.push_back(pad16(d));
    size_t off = 0;
    for (int l = 0; l + 1 < (int)m->dims.size(); ++l) {
        m->w_off.push_back(off);
        off += (size_t)m->dims[l + 1] * m->dims[l];
        m->b_off.push_back(off);
        off += m->dims[l + 1];
    }
    m->n_params = off;
    cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&m->p, off * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->g, off * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->m, off * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->v, off * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(float));
    m->narrow = (int)m->dims.size() - 1 <= kNetLayers && *std::max_element(m->pdims.begin(), m->pdims.end()) <= kNetWide;
    for (int l = 0; !m->narrow && e == cudaSuccess && l + 1 < (int)m->dims.size(); ++l) {
        __nv_bfloat16* w = nullptr;
        e = cudaMalloc(&w, (size_t)m->pdims[l + 1] * m->pdims[l] * sizeof(__nv_bfloat16));
        m->wb.push_back(w);
    }
    for (int l = 0; m->narrow && e == cudaSuccess && l + 1 < (int)m->dims.size(); ++l) {
        // zero past the last CTA's columns
        const size_t fb = net_image_elems(m->pdims[l + 1], m->pdims[l]) * sizeof(__nv_bfloat16);
        const size_t tb = net_image_elems(m->pdims[l], m->pdims[l + 1]) * sizeof(__nv_bfloat16);
        __nv_bfloat16 *f = nullptr, *w = nullptr;
        e = cudaMalloc(&f, fb);
        m->wf.push_back(f);
        if (e == cudaSuccess) e = cudaMalloc(&w, tb);
        m->wt.push_back(w);
        if (e == cudaSuccess) e = cudaMemset(f, 0, fb);
        if (e == cudaSuccess) e = cudaMemset(w, 0, tb);
    }
    if (m->narrow && e == cudaSuccess)
        e = cudaFuncSetAttribute(rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem);
    if (m->narrow && e == cudaSuccess)
        e = cudaFuncSetAttribute(update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpSmem);
    if (e != cudaSuccess) {
        delete m;
        return report_error(PLK_ERR_ALLOC, cudaGetErrorString(e));
    }
    // He-normal weights (Box-Muller on a SplitMix64 stream), zero biases
    std::vector<float> host(off, 0.f);
    uint64_t s = seed;
    for (int l = 0; l + 1 < (int)m->dims.size(); ++l) {
        const double sd = std::sqrt(2.0 / m->dims[l]);
        for (size_t i = 0; i < (size_t)m->dims[l + 1] * m->dims[l]; ++i) {
            const double u1 = ((sm64(s) >> 11) + 1.0) / 9007199254740993.0, u2 = (sm64(s) >> 11) / 9007199254740992.0;
            host[m->w_off[l] + i] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
        }
    }
    cudaMemcpy(m->p, host.data(), off * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(m->m, 0, off * sizeof(float));
    cudaMemset(m->v, 0, off * sizeof(float));
    plk_status st = refresh_bf16(m);
    if (st != PLK_OK) {
        report_error(st, m->err);
        delete m;
        return st;
    }
    *out = m;
    return PLK_OK;
}

void plk_mlp_destroy(plk_mlp* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    delete m;
}

const char* plk_mlp_last_error(const plk_mlp* m) { return m ? m->err.c_str() : plk_last_error(nullptr); }

int plk_mlp_n_params(const plk_mlp* m) { return m ? (int)m->n_params : 0; }

plk_status plk_mlp_get_params(const plk_mlp* m, float* out) {
    if (!m || !out) return PLK_ERR_ARG;
    cudaSetDevice(m->device);
    if (cudaMemcpy(out, m->p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess) return PLK_ERR_CUDA;
    return PLK_OK;
}

plk_status plk_mlp_set_params(plk_mlp* m, const float* in) {
    if (!m || !in) return PLK_ERR_ARG;
    PLK_MCUDA(m, cudaSetDevice(m->device), "cudaSetDevice");
    PLK_MCUDA(m, cudaMemcpy(m->p, in, m->n_params * sizeof(float), cudaMemcpyHostToDevice), "upload weights");
    return refresh_bf16(m);
}

plk_status plk_mlp_forward(plk_mlp* m, int batch, const float* x, float* y) {
    if (!m || batch < 1 || !x || !y) return m ? mfail(m, PLK_ERR_ARG, "bad arguments to plk_mlp_forward") : PLK_ERR_ARG;
    PLK_MCUDA(m, cudaSetDevice(m->device), "cudaSetDevice");
    plk_status s;
    if (m->narrow) {
        if ((s = net_ensure(m, batch, false)) != PLK_OK) return s;
        if ((s = net_pass(m, batch, x, nullptr, false, 0.0f, m->y_dev)) != PLK_OK) return s;
        PLK_MCUDA(m, cudaMemcpyAsync(y, m->y_dev, (size_t)batch * m->dims.back() * sizeof(float), cudaMemcpyDeviceToHost,
                                     m->stream), "download outputs");
        if ((s = net_finish(m, false, "forward", nullptr)) != PLK_OK) std::fill(y, y + (size_t)batch * m->dims.back(), NAN);
        return s;
    }
    if ((s = ensure_batch(m, batch)) != PLK_OK) return s;
    PLK_MCUDA(m, cudaMemcpyAsync(m->xin, x, (size_t)batch * m->dims.front() * sizeof(float), cudaMemcpyHostToDevice,
                                 m->stream), "upload inputs");
    if ((s = forward(m, batch)) != PLK_OK) return s;
    const int L = n_layers(m), out = m->dims[L];
    PLK_MCUDA(m, cudaMemcpy2DAsync(y, out * sizeof(float), m->pre[L], m->pdims[L] * sizeof(float), out * sizeof(float),
                                   batch, cudaMemcpyDeviceToHost, m->stream), "download outputs");
    PLK_MCUDA(m, cudaStreamSynchronize(m->stream), "forward");
    return PLK_OK;
}

plk_status plk_mlp_gradients(plk_mlp* m, int batch, const float* x, const float* t, float* grad, float* loss) {
    if (!m || batch < 1 || !x || !t) return m ? mfail(m, PLK_ERR_ARG, "bad arguments to plk_mlp_gradients") : PLK_ERR_ARG;
    PLK_MCUDA(m, cudaSetDevice(m->device), "cudaSetDevice");
    plk_status s;
    if (m->narrow) {
        if ((s = net_pass(m, batch, x, t, false, 0.0f, nullptr)) != PLK_OK) return s;
        if (grad)
            PLK_MCUDA(m, cudaMemcpyAsync(grad, m->g, m->n_params * sizeof(float), cudaMemcpyDeviceToHost, m->stream),
                      "download gradients");
        return net_finish(m, false, "gradients", loss);
    }
    if ((s = ensure_batch(m, batch)) != PLK_OK) return s;
    PLK_MCUDA(m, cudaMemcpyAsync(m->xin, x, (size_t)batch * m->dims.front() * sizeof(float), cudaMemcpyHostToDevice,
                                 m->stream), "upload inputs");
    PLK_MCUDA(m, cudaMemcpyAsync(m->tin, t, (size_t)batch * m->dims.back() * sizeof(float), cudaMemcpyHostToDevice,
                                 m->stream), "upload targets");
    if ((s = forward(m, batch)) != PLK_OK) return s;
    if ((s = backward(m, batch)) != PLK_OK) return s;
    if (grad)
        PLK_MCUDA(m, cudaMemcpyAsync(grad, m->g, m->n_params * sizeof(float), cudaMemcpyDeviceToHost, m->stream),
                  "download gradients");
    if (loss) PLK_MCUDA(m, cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream), "download loss");
    PLK_MCUDA(m, cudaStreamSynchronize(m->stream), "gradients");
    return PLK_OK;
}

plk_status plk_mlp_test_withhold(plk_mlp* m, int where) {
    if (!m) return PLK_ERR_ARG;
    if (!m->narrow || where < 1 || where > 2)
        return mfail(m, PLK_ERR_ARG, "plk_mlp_test_withhold: 1 or 2, networks up to 256 wide");
    m->withhold = where;
    return PLK_OK;
}

plk_status plk_mlp_train_step(plk_mlp* m, int batch, const float* x, const float* t, float lr, float* loss) {
    plk_status s;
    if (m && m->narrow && batch >= 1 && x && t) {
        PLK_MCUDA(m, cudaSetDevice(m->device), "cudaSetDevice");
        if ((s = net_pass(m, batch, x, t, true, lr, nullptr)) != PLK_OK) return s;
        return net_finish(m, true, "train step", loss);
    }
    if ((s = plk_mlp_gradients(m, batch, x, t, nullptr, nullptr)) != PLK_OK) return s;
    ++m->step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    for (int l = 0; l < n_layers(m); ++l) {
        const int in = m->dims[l], out = m->dims[l + 1];
        const int nw = in * out;
        adam_kernel<<<(nw + 255) / 256, 256, 0, m->stream>>>(m->p + m->w_off[l], m->g + m->w_off[l], m->m + m->w_off[l],
                                                            m->v + m->w_off[l], nw, lr, b1, b2, 1e-8f, c1, c2, m->wb[l],
                                                            out, in, m->pdims[l]);
        adam_kernel<<<(out + 255) / 256, 256, 0, m->stream>>>(m->p + m->b_off[l], m->g + m->b_off[l], m->m + m->b_off[l],
                                                             m->v + m->b_off[l], out, lr, b1, b2, 1e-8f, c1, c2,
                                                             nullptr, 0, 1, 0);
    }
    PLK_MCUDA(m, cudaGetLastError(), "Adam update");
    if (loss) PLK_MCUDA(m, cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream), "download loss");
    PLK_MCUDA(m, cudaStreamSynchronize(m->stream), "train step");
    return PLK_OK;
}

}  // extern "C"
