// Host-side interface of the persistent decode kernel (persist.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "comm.cuh"

namespace mb200 {
namespace persist {

constexpr int kMaxLayers = 112;  // layers per launch: their descriptors travel in the kernel parameters

struct Layer {
    const float *attn_norm, *q_norm, *k_norm, *ffn_norm, *router;
    const uint8_t *wq, *wk, *wv, *wo, *experts;
    __half *kv_k, *kv_v;
    size_t estride;
    uint32_t up_off, down_off;  // inside an expert's blob (the gate rows come first)
    int v_q6, down_q6;
};

// `passes` work items over warps [w0, w0 + nw): warp i takes per items, the first rem warps one more.
struct Split {
    int w0, nw, per, rem;
};

// Lane map of a matrix with `bpr` super-blocks per row: a pass of a warp is v = 2^lv blocks of 8 / v rows; ceil(bpr / v) passes
// cover the columns, the last one ragged where v does not divide bpr.
struct Map {
    int bpr, lv;
};

struct Params {
    int n_layers, attn;  // attn = 0: the MoE block alone (one layer)
    int H, EFF, QD, KD, n_heads, n_kv, gqa, qblocks, chunks, n_experts, k, expert_lo, expert_cnt;
    float eps, scale;
    const float *cos_t, *sin_t;
    const int *pos;
    float *hidden;             // attn = 1: before the first layer, after the last one
    const float *x, *residual; // attn = 0
    float *y, *act;
    // Exchange buffers of {value, tag} cells: what one CTA computes and the others need (attn = 1; the logits always)
    uint2 *c_q, *c_k, *c_v, *c_part, *c_ml, *c_attn, *c_h1, *c_act, *c_h0, *c_logit;
    int *ids_out;              // attn = 0: the selection in the reference's slot order
    float *wts_out;
    unsigned long long *ctr;   // arrivals, only grows: one per CTA and launch
    double inv_grid;
    int *err;
    int pdl;
    PushDesc push;  // world > 0: the block of one rank of an expert-sharded model, all-reduced over the ranks
    // geometry
    Map mH, mQ, mE;            // rows of H, QD and EFF columns
    Split sq, sk, sv, so;      // passes of the four projections
    int xc, off_row, off_misc, off_ring, ring_bytes;  // columns of the staged vector; byte offsets in shared memory
    Layer L[kMaxLayers];
};

// Fills in the geometry of P for its shape; false = a shape this kernel does not take.
bool plan(Params &P);
int launch(Params &P, cudaStream_t stream);  // MB200_OK or an error status
void init();
// Cells of the exchange buffers (attn = 1) in the order of Params; returns the bytes, fills the pointers in if base is given.
size_t cells(Params &P, uint8_t *base);

}  // namespace persist
}  // namespace mb200
