// Host-side interface of the persistent decode kernel (persist.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>


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
    int fold;  // the layer's expert block alone would be one launch with the norm inside: whose order of sums stage_vec follows
};

// `passes` work items over warps [w0, w0 + nw): warp i takes per items, the first rem warps one more.
struct Split {
    int w0, nw, per, rem;
};

// Lane map of a matrix with `bpr` super-blocks per row: a pass of a warp is v = 2^lv blocks of 8 / v rows; ceil(bpr / v) passes
// cover the columns, the last one ragged where v does not divide bpr. A row is summed in groups of 2^lt blocks.
struct Map {
    int bpr, lv, lt;
};

struct Head {
    int n_layers;
    int H, EFF, QD, KD, n_heads, n_kv, gqa, qblocks, chunks, n_experts, k;
    float eps, scale;
    const float *cos_t, *sin_t;
    const int *pos;
    float *hidden;  // before the first layer, after the last one
    // Exchange buffers of {value, tag} cells: what one CTA computes and the others need
    uint2 *c_q, *c_k, *c_v, *c_part, *c_ml, *c_attn, *c_h1, *c_act, *c_h0, *c_logit;
    unsigned long long *ctr;  // arrivals, only grows: one per CTA and launch
    double inv_grid;
    int *err;
    int pdl;
    // geometry
    Map mH, mQ, mE;         // rows of H, QD and EFF columns
    Split sq, sk, sv, sg;   // passes of Q, K, V; gate / up items
    uint32_t ipe, ipe_magic;   // gate / up items per expert, 2^32 / ipe rounded up
    int stages[6];             // of a warp's ring: H Q4_K, H Q6_K, QD, EFF Q4_K, EFF Q6_K, gate / up
    int xc, off_row, off_ring, ring_bytes;  // columns of the staged vector; byte offsets in shared memory
};

struct Params : Head {
    Layer L[kMaxLayers];
};

// Fills in the geometry of P for its shape; false = a shape this kernel does not take.
bool plan(Params &P);
int launch(Params &P, cudaStream_t stream);  // MB200_OK or an error status
// Bytes of the exchange buffers and the counter for a shape (H, EFF, QD, KD, n_heads, n_experts, k set); fills the pointers in if
// base is given. Zeroed once by the owner.
size_t scratch(Params &P, uint8_t *base);

}  // namespace persist
}  // namespace mb200
