// Plan and dispatch of prune_any_kernel (plk_prune_any.cuh).
#include "plk_prune_any.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>

namespace plk {

namespace {

constexpr size_t kAnySmem = 227 * 1024;  // of a CTA, the kernel's static bytes among them
constexpr int kAnyWarps = 8;  // per CTA at most

// of vectors stored where that is faster
double stored_limit() {
    const char* e = getenv("PLK_STORED_BYTES");
    return e ? atof(e) : 8e9;
}

int any_sm_count() {
    static std::atomic<int> n{0};
    int v = n.load();
    if (v > 0) return v;
    int dev = 0, c = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0)
        c = 152;
    n.store(c);
    return c;
}

struct AnyPlan {
    dev::AnyLaunch launch{};
    int H = 0, blocks = 0;
    double cost = 0.0;  // estimated cycles of one op on the fullest SM
};

// H, warps per CTA and the tables' place for these counts; H = 0 where
// nothing fits.  smem(H, launch): the dynamic bytes of a CTA, fixed: its static
// ones; writes: the pass writes node states (NodeOut).
template <class Smem>
AnyPlan any_plan(int S, int C, bool fp64, int n_sites, int n_codes, int max_depth, int sms, size_t fixed, bool writes,
                 Smem smem) {
    AnyPlan best;
    const int tsz = fp64 ? 8 : 4;
    for (int H = 1; H <= 4; H *= 2) {
        if (C * H > 32 || H > S || (H == 1 && S > 8)) continue;
        const int R = (S + H - 1) / H, W = 32 / (C * H);
        const long long warps = ((long long)n_sites + W - 1) / W;
        const int per_sm = (int)((warps + sms - 1) / sms);
        AnyPlan p;
        p.H = H;
        p.launch.depth = std::max(max_depth, 1);
        // tip tables through the ring while they are of the size of P(t)
        p.launch.stage_tips = n_codes <= 2 * S + 8 ? 1 : 0;
        const int child = std::max(C * S * S, p.launch.stage_tips ? C * n_codes * S : 0);
        p.launch.child_elems = (child * tsz + 15) / 16 * 16 / tsz;
        // one CTA per SM while eight warps hold its sites: a table brought in
        // once then serves every warp of the SM
        const int want = std::max(1, std::min(kAnyWarps, per_sm));
        bool fits = false;
        // all tables resident (up to 8 states) while one CTA an SM is all
        // there is to run, or two fit; else the ring
        p.launch.slots = 0;
        p.launch.warps = want;
        if (S <= 8) {
            const size_t need = smem(H, p.launch);
            fits = need <= (per_sm <= kAnyWarps ? kAnySmem - fixed : kAnySmem / 2);
        }
        for (int slots = 3; slots >= 2 && !fits; --slots)
            for (int w = want; w >= 1 && !fits; --w) {
                if (slots == 3 && w < (want + 1) / 2) break;  // rather two slots than half the warps
                p.launch.slots = slots;
                p.launch.warps = w;
                fits = smem(H, p.launch) <= kAnySmem - fixed;
            }
        if (!fits) continue;
        p.blocks = (int)((warps + p.launch.warps - 1) / p.launch.warps);
        const int load = (p.blocks + sms - 1) / sms * p.launch.warps;  // warps of the fullest SM, whole CTAs
        if (fp64) {
            // the SM's FP64 pipe takes 16 cycles a warp instruction: the fullest SM's
            // warps (157 CTAs on 152 SMs are two on five of them) with what they
            // issue besides, against the latency of one warp's dependent ones.
            // By per_sm alone a last wave's rounding chose
            // four lanes a category for 90,000 sites (4 states, C = 4, 7 taxa: 646
            // us of conditional vectors, one lane 285).
            const double op = 16.0 * R * 2 * S;
            const double out = writes ? 16.0 * ((2 * C + 12) * ((W * S + 31) / 32) + S) : 0.0;
            const int beside = std::max(1, (int)((kAnySmem + 1024) / (smem(H, p.launch) + fixed + 1024)));  // CTAs an SM holds
            const int rounds = (p.blocks + beside * sms - 1) / (beside * sms);
            p.cost = std::max(rounds * (500.0 + 6.0 * op + out), load * (op + 100.0 + out));
        } else {
            // four schedulers, against the latency of one warp's op
            p.cost = std::max((per_sm + 3) / 4 * (1.5 * R * S + 100.0), 200.0 + 2.0 * R * S + 5.0 * S);
        }
        // more lanes a site: while the SM's one CTA holds them all, else for a clear
        // gain only (they cost instructions that are not counted)
        if (best.H == 0 || p.cost < (fp64 ? (load <= kAnyWarps ? 1.15 : 0.95) : 1.0) * best.cost) best = p;
    }
    return best;
}

// node_pass: a pass for the node states (of conditional vectors, or of messages)
AnyPlan up_plan(const PruneArgs& a, int S, bool fp64, bool node_pass, bool cond_nodes, int sms) {
    return any_plan(S, a.C, fp64, a.n_sites, a.n_codes, a.max_depth, sms,
                    dev::kSumStatic + (node_pass ? dev::kWeightStatic : 0), cond_nodes,
                    [&](int H, dev::AnyLaunch p) {
                        static double some;
                        p.nodes = cond_nodes ? &some : nullptr;  // only its presence counts
                        return dev::any_smem(S, H, fp64, p, a);
                    });
}
AnyPlan down_plan(const PreorderArgs& a, int S, bool fp64, int sms) {
    return any_plan(S, a.C, fp64, a.n_sites, a.n_codes, 0, sms, dev::kWeightStatic, true,
                    [&](int H, const dev::AnyLaunch& p) { return dev::any_down_smem(S, H, fp64, p, a); });
}

// Whether the kernels that store every vector (a thread per site; node states are
// normalised or formed by further kernels) are faster: where many sites meet few
// ops or many idle lanes (11 categories leave a third), a warp's start, its sums and
// its idle lanes here cost more than the vectors' way through L2.  Both times in
// microseconds, fitted to 3 to 30 taxa, 5,000 to 100,000 sites, 2 to 24 states and 1
// to 16 categories; FP32 up to 5 taxa, as this kernel is faster above.  lnL, FP64, 3
// taxa x 100,000, 2 states, C = 11: 288 us here and 93 there; 9 states, C = 9, 1,212
// and 495; 10 taxa x 100,000, 5 states, C = 4, 449 and 478.  By this rule the
// mean over all those shapes is 0.6 % (node states 0.8) above the better of the two, by
// this kernel alone 7 (16).  They hold all vectors, this pass none: up to 8 GB.
bool stored_faster(const PruneArgs& a, int S, bool fp64, int kind, const AnyPlan& up, const AnyPlan* down, int sms) {
    // [FP32, FP64][lnL, conditionals, marginals]: here: start, the plan's cost, warps,
    // warps x ops x states; there: start, latency of an op and of a product, issue of both
    static constexpr double kFit[2][3][9] = {
        {{21, 1.2, 0.37, 0.071, 32, 0.78, 3.6, 3.1, 1.2}, {50, 1.4, 0.28, 0.31, 68, 0, 0, 16, 2.8}, {53, 0.98, 0.26, 0.49, 69, 0.64, 3.5, 25, 3.6}},
        {{21, 0.35, 0.38, 0.31, 31, 0.99, 4.9, 6.2, 6.6}, {37, 0.42, 0.41, 0.39, 54, 0.74, 4.3, 16, 8.4}, {43, 0.33, 0.56, 0.65, 50, 2, 13, 22, 10}}};
    const double stored = (fp64 ? 8.0 : 4.0) * (kind == 2 ? 2 : 1) * a.n_ops * a.n_sites * a.C * S;
    if (stored > stored_limit() || a.n_sites < 64 * sms || (!fp64 && a.n_ops > 4)) return false;
    const double* f = kFit[fp64][kind];
    const double ops = a.n_ops, products = a.n_ops - 1;
    const double load = (up.blocks + sms - 1) / sms * up.launch.warps;
    const double here = f[0] + f[1] * ops * (up.cost + (down ? down->cost : 0.0)) / 1e3 + f[2] * load + f[3] * ops * load * S / 10;
    const double x = ((a.n_sites + 127) / 128 + sms - 1) / sms * a.C, SS = S * S / 100.0;
    const double there = f[4] + f[5] * ops * a.C + f[6] * products * a.C * SS + f[7] * ops * x * S / 100 + f[8] * products * x * SS;
    return here > 1.05 * there;
}

}  // namespace

int prune_any_blocks(const PruneArgs& a, int S, int precision, bool nodes, bool marginal, bool may_store) {
    const bool fp64 = precision == PLK_FP64;
    if (S < 2 || S > kMaxStates || a.C > kMaxCats || a.n_ops < 1) return 0;
    if (!fp64 && !nodes && ((S == 4 && a.C <= 8) || S == 20)) return 0;  // the tuned FP32 forms
    const int sms = any_sm_count();
    const AnyPlan p = up_plan(a, S, fp64, nodes, nodes && !marginal, sms);
    if (p.H == 0) return 0;
    AnyPlan down;
    if (marginal) {
        PreorderArgs d{};
        d.n_int = a.n_int; d.n_tips = a.n_tips; d.n_nodes = a.n_nodes; d.n_sites = a.n_sites; d.n_codes = a.n_codes;
        d.C = a.C;
        down = down_plan(d, S, fp64, sms);
        if (down.H == 0) return 0;
    }
    if (S == 4 && a.C <= 8 && !nodes) {
        // prune4_kernel, a thread per site in 128-thread CTAs (FP64 only: FP32 has
        // other forms), issues the same FP64 instructions, 32 per category and op,
        // with less around them once its CTAs fill the SMs.  Cycles an op of each,
        // fitted to both over 4 to 50 taxa, 200 to 100,000 sites and 1 to 8
        // categories (prune4_kernel pads those to 1, 4 or 8); `start`: what this
        // kernel takes longer to start and end, in ops.  C = 1, 120 taxa x
        // 30,625 sites: 332 us here and 411 there, 40,000 534 and 505.
        const long long blocks4 = (a.n_sites + 127) / 128;
        const double issue4 = (double)((blocks4 + sms - 1) / sms) * 4 * 16.0 * 32 * a.C;
        const double cost4 = a.C == 1 ? 1.3 * issue4 + 1200.0 : (1.35 * issue4 + 1000.0 * a.C) * (a.C == 2 ? 1.2 : 1.0);
        const double start = a.C / 8.0;
        if ((a.n_ops + start) * 1.2 * p.cost > a.n_ops * cost4) return 0;
    }
    if (!may_store) return p.blocks;
    // the stored forms of 4 states (prune4_kernel), up to 8 categories, padded to 4 or 8:
    // 4 taxa x 100,000, C = 4, conditionals 240 us here and 216 there, marginals 314 and
    // 294; C = 8 439 and 317, 586 and 475.  At 16,000 sites (C = 4) 65 and 76, 79 and 100
    const double warps = (double)a.n_sites * a.C / 32 / sms;  // of an SM, a lane a category
    if (fp64 && nodes && S == 4 && a.C >= 4 && a.C <= 8 && 8.0 * a.n_ops * a.n_sites * a.C * S <= stored_limit() &&
        (marginal ? warps > 40 && a.n_ops <= 12 : warps > 20))
        return 0;
    // FP32 conditionals of one category: a long chain of ops with the output's division
    // in each, 900 taxa x 50 961 us here and 802 there, x 500 1,044 and 881, x 3,000 1,438
    // and 1,564; 300 taxa level
    if (!fp64 && nodes && !marginal && S == 4 && a.C == 1 && a.n_ops > 300 && a.n_sites <= 8 * sms &&
        4.0 * a.n_ops * a.n_sites * S <= stored_limit())
        return 0;
    if (S != 4 || a.C > 8 || nodes)
        if (stored_faster(a, S, fp64, nodes ? (marginal ? 2 : 1) : 0, p, down.H ? &down : nullptr, sms)) return 0;
    return p.blocks;
}

cudaError_t launch_prune_any(const PruneArgs& a, int S, int precision, int* n_blocks, cudaStream_t st) {
    const bool fp64 = precision == PLK_FP64;
    AnyPlan p = up_plan(a, S, fp64, a.nodes || a.msg, a.nodes != nullptr, any_sm_count());
    if (p.H == 0) return cudaErrorInvalidConfiguration;
    p.launch.msg = a.msg;
    p.launch.nodes = a.nodes;
    *n_blocks = p.blocks;
    if (fp64)
        return S <= 12 ? launch_any64_lo(a, S, p.H, p.launch, p.blocks, st)
                       : launch_any64_hi(a, S, p.H, p.launch, p.blocks, st);
    return S <= 12 ? launch_any32_lo(a, S, p.H, p.launch, p.blocks, st)
                   : launch_any32_hi(a, S, p.H, p.launch, p.blocks, st);
}

cudaError_t launch_down_any(const PreorderArgs& a, void* msg, int precision, cudaStream_t st) {
    const bool fp64 = precision == PLK_FP64;
    AnyPlan p = down_plan(a, a.S, fp64, any_sm_count());
    if (p.H == 0) return cudaErrorInvalidConfiguration;
    p.launch.msg = msg;
    if (fp64)
        return a.S <= 12 ? launch_down64_lo(a, a.S, p.H, p.launch, p.blocks, st)
                         : launch_down64_hi(a, a.S, p.H, p.launch, p.blocks, st);
    return a.S <= 12 ? launch_down32_lo(a, a.S, p.H, p.launch, p.blocks, st)
                     : launch_down32_hi(a, a.S, p.H, p.launch, p.blocks, st);
}

}  // namespace plk
