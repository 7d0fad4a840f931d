// Device-side layout of a batch (plk_batch.cu, plk_nni.cu, plk_batch_api.cpp).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "plk_internal.h"

namespace plk {

// One alignment + tree + model of a batch; offsets into the concatenated
// device arrays.  Internal nodes are numbered n_tips + post-order rank.
struct BatchItemDev {
    long long codes_off;  // bytes into codes ([n_tips][site_stride])
    int ops_off, n_ops;   // into ops
    int node_off;         // into t_eff, child and P32 ([node_off + v][C][16])
    int tip_off;          // into tip32 ([tip_off + t][C][16][4])
    int n_tips, n_sites, site_stride;
    int model_off;        // doubles into model: lam[4] L[16] R[16] root_w[4] cat_rate[C] cat_w[C]
    int n_moves, move_out_off;  // NNI rearrangements of this tree, into the NNI output
    int n_int;            // internal nodes (the root is n_tips + n_int - 1)
    int stage_off, n_stages;  // into stages (streamed tables)
    int pad;
};
static_assert(sizeof(BatchItemDev) == 64, "BatchItemDev is 64 bytes");

struct BatchDev {
    int n_items, n_units, n_nodes_total, C;
    int max_depth, pad;
    const BatchItemDev* items;
    const uint8_t* codes;
    const Op* ops;
    const double* t_eff;      // [n_nodes_total]
    const int2* node_item;    // [n_nodes_total] (item, local node id)
    const int2* child;        // [n_nodes_total] (left, right) local ids, -1 = none
    const double* model;      // per item, see BatchItemDev::model_off
    float* P32;               // [n_nodes_total][C][16]
    float* tip32;             // [n_tips_total][C][16][4]
    float* P32p;              // paired layout of P32 (plk_prune4p.cuh), or null
    float* tip32p;            // paired layout of tip32, or null
    // streamed tables (plk_batch4w.cu, stream_program): per item's ops in their
    // order, its stages, every node's place, the tables; or null
    const Op* sops;           // as ops
    const int2* stages;       // (first unit, units) of every item's stages
    const int* where;         // [n_nodes_total] first unit of a node's tables, -1 for a root
    float* stream;            // [units][KP][32]
    int write_std, pad2;      // batch_pmat_kernel writes P32 / tip32 when non-zero
    const int2* units;        // [n_units] (item, tile index), largest trees first
    double* unit_sums;        // [n_units][2]
    const int* item_unit_ptr; // [n_items + 1]
    const int* item_units;    // units of each item in site order
    double* lnl;              // [n_items]
    int* counter;             // work-queue head, zeroed before each launch
    // NNI scoring and branch-length derivatives (plk_nni.cu)
    float* Pn;                // [n_nodes_total][KP][j][i][2], KP = ceil(C / 2)
    float* tipn;              // [n_tips_total][KP][code][i][2]
    const int4* kids;         // [internal nodes of all items] (left, right, first move or -1, 0), local ids
    float4* records;          // per item [warp tile][move or edge slot]: (hi, lo, exponent, -) or (d1 hi, lo, d2 hi, lo)
    const long long* rec_off; // [n_items] into records
    const int2* reduce_blocks;// (item, first output) of every CTA of the fold
    double* nni_out;          // [sum over items of n_moves]
    int scratch_int, pad3;    // max internal nodes of any item
    float4* scr;              // per warp: messages, then outside vectors, [2 scratch_int][32 lanes][2]
    int* scr_e;               // per warp: their exponents [2 scratch_int][sites of a warp]
};

inline int batch_model_stride(int C) { return 40 + 2 * C; }

// One form of the batch post-order kernel: sites per thread, tip codes staged
// in shared memory or read from global, categories in pairs on the FP32x2
// pipe (C = 2, 4, 8; reads P32p / tip32p) or one at a time; or the streamed
// form (in pairs, any C).
struct BatchForm {
    int spt = 1;
    bool codes_smem = false;
    bool paired = false;
    bool stream = false;
};
bool batch_form_valid(int C, const BatchForm& f);
size_t batch_smem_bytes(int C, const BatchForm& f, int max_ops, int max_tips, int max_depth);
int batch_occupancy(int C, const BatchForm& f, size_t smem);
cudaError_t launch_batch_pmat(const BatchDev& b, cudaStream_t st);
cudaError_t launch_batch_prune(const BatchDev& b, const BatchForm& f, int grid, size_t smem, cudaStream_t st);
cudaError_t launch_batch_reduce(const BatchDev& b, cudaStream_t st);

// The streamed form (plk_batch4w.cu) with per_sm CTAs of four warps an SM: their
// tensor-memory columns and stack entries in them, byte offsets in shared memory.
struct BatchStreamShape {
    int tmem_cols, levels;
    int ops_at, codes_at, over_at, ops_in_smem;
    size_t smem;  // 0: does not fit
};
BatchStreamShape batch_stream_shape(int C, int spt, int max_ops, int max_depth, int per_sm);
cudaError_t launch_batch_prune4w(const BatchDev& b, const BatchStreamShape& sh, int spt, int grid, cudaStream_t st);

// NNI scoring and branch-length derivatives (plk_nni.cu): work units of `warps`
// warps of down_sites_per_warp sites; the tables of an item in shared memory
// (in_smem) or read through L1.  The edge slots of an item: slot i = child
// i % 2 of internal node n_tips + i / 2.
struct BlenDev {
    float* ex;                 // [n_nodes_total][KP][m][2] exp(rho_km t), or null (NNI)
    const int* item_edge_off;  // [n_items] first slot of each item
    double* edge_out;          // [total slots][2] (d1, d2)
};
struct DownSize {              // warps per CTA; the largest item whose tables sit in shared memory
    int warps = 0, nodes = 0, tips = 0, ints = 0;
};
constexpr int kDownWarps = 12;  // per CTA at most
int down_sites_per_warp(int C);
int down_smem_bytes(int C, bool blen, bool in_smem, const DownSize& z);
// the most a CTA may have of them
size_t down_smem_limit(int C, bool blen, bool in_smem);
// resident CTAs per SM
int down_occupancy(int C, bool blen, bool in_smem, const DownSize& z);
cudaError_t launch_down_tables(const BatchDev& b, const BlenDev& bd, cudaStream_t st);
// units [unit0, unit1) on `grid` CTAs (the work-queue head zeroed before)
cudaError_t launch_down(const BatchDev& b, const BlenDev& bd, bool blen, bool in_smem, const DownSize& z, int unit0,
                        int unit1, int grid, cudaStream_t st);
cudaError_t launch_down_reduce(const BatchDev& b, const BlenDev& bd, bool blen, int blocks, cudaStream_t st);

// Summary statistics of every item (plk_features.cu): out[n_items][43].
constexpr int kNumFeatures = 43;
cudaError_t launch_features(const BatchDev& b, float* out, cudaStream_t st);

}  // namespace plk
