// One launch for many layers of a decoded token: a persistent cooperative kernel, one CTA per SM (op order of
// src/forward.c:604-1117):
//   Q, K, V of RMSNorm(hidden) | q/k norm + RoPE + KV store + attention partials | merge of the partials | O + residual |
//   router logits of RMSNorm(hidden) | top-k, gate / up + SwiGLU of the routed experts | down, weighted sum + residual
//
// At batch 1 a layer streams 49 MB (30B-A3B shape) or 157 MB (235B-A22B shape), 7.6 / 24 us at the copy rate; as five to seven
// kernels it took 68 / 104 us, because every kernel paid for its launch, for instructions fetched cold, for staging its input
// and for the ramp of its weight stream. Here
//   * a warp owns whole rows: it copies them itself into a private ring of shared memory (1-D bulk copies), computes them and
//     writes the results. No roles, no partial sums across warps (but for the down projection);
//   * what a CTA needs of the others it polls for, value by value: results travel as 8-byte cells {value, tag} written with one
//     store, so there is no barrier, no fence and no second read (a device-wide barrier, arrival counter and poll, took 2.5 us,
//     and the read of the vector another one; a cell is with its reader about 1 us after it was written). A tag belongs to one
//     layer of one launch. A cell is overwritten only by a CTA that has results of every CTA that were computed after they had
//     read it: each operation's writers depend on all CTAs' rows of the O projection and of the down projection;
//   * weights depend on nobody: while a warp would wait it has the first 20 KB of its next rows on the way (160 KB per SM,
//     which is all of most operations), and K / V rows of the cache before q exists;
//   * the input vector of an operation is split by every CTA into two int8 levels as it arrives;
//   * a CTA's rows of the hidden vector stay in its shared memory: it updates them in both halves of every layer.
//
// Every sum is taken in the order of the kernels that do the same layer by layer (decode.cu: run_layer), so both give the same
// bits. A rounding of another order is no error, but deep models with close router logits magnify it to another expert: 48 layers of
// synthetic 30B weights ended in another token for two seeds of eleven. Kept are the groups of blocks and their trees in a row's sum,
// the thread mapping behind the norms and the router logits, the order of attention chunks, and the reference's expert slots.
//
// The top-k a CTA does for itself by counting: the rank of an expert is how many logits are larger; how many of those came before
// it in the reference's replace-the-minimum walk tells whether that accepted it, from which its slot follows. Only where equal
// logits meet is the walk itself run.
//
// The code of a layer is run once per layer: what counts is its size (270 KB with a copy of every step per operation, 134 KB as
// one loop over the operations) and that nothing lives in local memory, which the weight stream and 227 KB of shared memory
// leave no L1 for. Hence eight warps with 255 registers (sixteen with 128 spilled 2 KB a thread and took half as long again),
// several rows per warp in flight instead, thread_id() and cta_id() read anew by every step, and the launch's
// parameters, divisions already done, in shared memory.
//
// Measured, per token: 30B shape at position 4095 (48 layers) 1716 us, 8 layers of the 235B shape at 8191 639 us (layer by layer
// 3276 / 931; 1763 / 661 before the dot products took their scales by byte permutes). Where a layer's time goes, by clock stamps of
// warp 0, mean over CTAs and layers, 30B / 235B, taken before that change, when a layer was 35 / 67.5 us (now 34 / 65):
//   waits for the operation's input (its slowest writer, and 1 us from a store to its readers)   7.8 / 13.6 us
//   norm, router logit, split into levels                                                        4.3 /  6.0
//   selection, with the exchange of the logits                                                   2.0 /  1.9
//   query heads, attention partials                                                              4.4 /  7.8
//   rows: Q, K, V | O | gate, up | down                                        2.5, 1.6, 5.0, 3.0 / 5.5, 3.7, 13.6, 9.7
// (gate / up is at the copy rate at the 235B shape.) Tried and slower: two K / V tiles in flight per warp, the selection by
// repeated warp maxima (150 cycles a round), the next round of a wide vector requested ahead (all three: registers), units of two
// rows, the partials' merge with the chunk maxima taken by four warps.
//
// Every wait is bounded: a cell or a copy that does not come raises the abort flag of the CTA and the device error word, and
// the CTA leaves after its copies in flight.
#include "persist.cuh"

#include <cstdio>

#include "comm.cuh"
#include "q4k_policy.cuh"
#include "q6k_policy.cuh"

namespace mb200 {
int pdl_enabled();
bool moe_fused_covers(int H, int EFF, int k, bool down_q6);

namespace persist {
namespace {

constexpr int kWarps = 8, kWork = kWarps * 32;
constexpr int kStages = 5;         // ring stages per warp at most
constexpr int kPitch = 132;        // floats between heads of a warp's attention result
constexpr int kKPitch = 320, kVPitch = 272;  // bytes between K / V rows in shared memory: free of bank conflicts as each is read
constexpr int kVOff = 16 * kKPitch;          // of the V rows behind the K rows
constexpr int kMaxDownRows = 64;   // rows of the hidden vector per CTA
constexpr int kMaxK = kWarps;    // a warp per slot, or several
constexpr int kMaxExperts = 256;   // two threads per expert
constexpr int kMaxChunks = 160;    // of the attention's positions
constexpr uint32_t kPolls = 1u << 19;  // a fraction of a second
constexpr float kLog2e = 1.4426950408889634f;

extern __shared__ __align__(1024) uint8_t smem[];

// Read anew by every step (volatile): what follows from it is then not computed once, ahead of the loop over the layers, and kept
// in registers -- or in local memory -- all along.
__device__ __forceinline__ int thread_id()
{
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}
__device__ __forceinline__ int cta_id()
{
    int t;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(t));
    return t;
}

struct Misc {
    uint64_t bars[kWarps][kStages];
    uint64_t row_bar, ranked;
    uint32_t tag;                           // of the launch's first layer
    int pos, row_pend;                      // row_pend: parity of the router row on its way, or -1
    alignas(16) float red[3][12];          // partial sums of the norm and of the router logit (see stage_vec)
    float am[kWarps][16], al[kWarps][16];  // attention: running maximum / sum per warp and head
    float hid[kMaxDownRows];               // the CTA's rows of the hidden vector: it writes them in both of a layer's halves
    union {
        float part[kMaxK][kMaxDownRows];   // the down projection's rows, by rank of the expert
        struct {                           // before them: experts in the walk's order; the keys it accepts, and their order
            alignas(16) uint32_t acc_key[kMaxExperts + 4];
            uint8_t eid[kMaxExperts], by_rank[kMaxExperts];
            float red32[32];
        };
    };
    alignas(16) uint32_t key[kMaxExperts]; // ordered logits, in the order of the reference's walk
    uint32_t accepted[kMaxExperts / 16];   // a bit per candidate
    int top_id[kMaxK + 1], top_pos[kMaxK + 1];  // by rank: expert, place in the walk
    uint32_t top_key[kMaxK + 1];
    int walked, slot_pos[kMaxK];           // the walk itself was run; candidate per output slot
    int order[kMaxK];                      // by output slot: rank
    float swt[kMaxK];
    float rope[128], norm[2][128];         // cosines and sines of the position; this layer's q and k norm weights
    int abort_flag;
    Head head;                              // the launch's parameters, read from here by every step (see thread_id)
    int2 own[kWarps][4];                    // a warp's rows of each operation: first, count (gate / up: items)
    int own_qm[kWarps], own_slot[kWarps];   // which of Q, K, V; slot of the down projection
    // the CTA's rows of the hidden vector; its part of the attention (chunks in all, own head block and tiles); the head it merges
    int R0, rows, nc, kvh, qb, part_slot, tile0, tile1, merge_block, merge_head;
};
enum Op { kQKV, kO, kExperts, kDown };
// Shared memory: Misc, the staged vector (and the attention's fragments, the merge), the router row, the warps' rings.
constexpr int kX = (static_cast<int>(sizeof(Misc)) + 127) & ~127;
__device__ __forceinline__ Misc &misc() { return *reinterpret_cast<Misc *>(smem); }
__device__ __forceinline__ const volatile Head &head() { return misc().head; }
__device__ __forceinline__ uint8_t *ring() { return smem + head().off_ring + (thread_id() >> 5) * head().ring_bytes; }
__device__ __forceinline__ uint64_t *ring_bars() { return misc().bars[thread_id() >> 5]; }
__device__ __forceinline__ volatile int *gave_up() { return &misc().abort_flag; }

__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWork) : "memory"); }
// Every thread: true = somebody in the CTA has given up (the same answer for all of them). A barrier of the CTA.
__device__ __forceinline__ bool cta_aborted()
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.or.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(*gave_up())), "n"(kWork)
        : "memory");
    return r != 0;
}

// (Not left early when somebody gives up: copies in flight are always waited for.)
__device__ __forceinline__ void wait_copy(uint64_t *bar, uint32_t parity)
{
    uint32_t i = 0;
#pragma unroll 1
    while (!mbar_try_wait(bar, parity))
        if (++i == kWaitBudget) {
            *gave_up() = 1;
            break;
        }
}

// ---- cells ----
__device__ __forceinline__ uint4 ld_cells2(const uint2 *p)  // two cells
{
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_cells2(uint2 *p, float a, float b, uint32_t tag)
{
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(p), "r"(__float_as_uint(a)), "r"(tag), "r"(__float_as_uint(b)) : "memory");
}
// One cell, bounded wait (0 and the abort flag if it does not come).
__device__ __forceinline__ float wait_value(const uint2 *p, uint32_t tag)
{
#pragma unroll 1
    for (uint32_t i = 0; i < kPolls; i++) {
        const uint2 c = ld_cell(p);
        if (c.y == tag) return __uint_as_float(c.x);
        if (*gave_up()) return 0.0f;
    }
    *gave_up() = 1;
    return 0.0f;
}
// Four cells, 32 apart (a head's values of a lane), all requested at once.
__device__ __forceinline__ void wait_values4(const uint2 *p, uint32_t tag, float (&v)[4])
{
#pragma unroll 1
    for (uint32_t i = 0;; i++) {
        bool ok = true;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint2 c = ld_cell(p + 32 * u);
            v[u] = __uint_as_float(c.x);
            ok = ok && c.y == tag;
        }
        if (ok || *gave_up()) return;
        if (i == kPolls) *gave_up() = 1;
    }
}

// ---- the staged input vector of xc columns: two arrays of int8 levels in 16-byte chunks of 16 columns, swizzled so that both
// block types read them without bank conflicts; the scale of every 32 columns and the sum of every 16 ----
__device__ __forceinline__ int chunk_at(int j)
{
    const int b = (j >> 3) & 3;
    return j ^ (b ^ (b << 1));
}
__device__ __forceinline__ float *x_scale(int xc) { return reinterpret_cast<float *>(smem + kX + 2 * xc); }
__device__ __forceinline__ float *x_sum(int xc) { return reinterpret_cast<float *>(smem + kX + 2 * xc + xc / 8); }
__device__ __forceinline__ void stage_quad(int xc, const float4 t, int c0, int lane)
{
    const float v[4] = {t.x, t.y, t.z, t.w};
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    float sum = __fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3]));
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));  // 8 lanes = 32 columns
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const float sc = amax * (1.0f / 127.0f);
    // (the division never of 0: that takes its slow path, and whole blocks of activations are 0)
    const float inv = 127.0f / (amax > 0.0f ? amax : 1.0f);
    uint32_t p1, p2;
    stream::split_levels(v, sc, amax > 0.0f ? inv : 0.0f, p1, p2);
    const int at = chunk_at(c0 >> 4) * 16 + (c0 & 12);
    *reinterpret_cast<uint32_t *>(smem + kX + at) = p1;
    *reinterpret_cast<uint32_t *>(smem + kX + xc + at) = p2;
    if ((lane & 7) == 0) x_scale(xc)[c0 >> 5] = sc;
    if ((lane & 3) == 0) x_sum(xc)[c0 >> 4] = sum;
}
__device__ __forceinline__ void load_x(Q4::XRegs &r, int xc, int col, int g)
{
    const int j = col * 16 + g * 4;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int at = chunk_at(j + i) * 16;
        const uint4 a = *reinterpret_cast<const uint4 *>(smem + kX + at), b = *reinterpret_cast<const uint4 *>(smem + kX + xc + at);
        r.q1[4 * i] = a.x; r.q1[4 * i + 1] = a.y; r.q1[4 * i + 2] = a.z; r.q1[4 * i + 3] = a.w;
        r.q2[4 * i] = b.x; r.q2[4 * i + 1] = b.y; r.q2[4 * i + 2] = b.z; r.q2[4 * i + 3] = b.w;
    }
    const float2 s = *reinterpret_cast<const float2 *>(x_scale(xc) + (j >> 1));
    const float4 t = *reinterpret_cast<const float4 *>(x_sum(xc) + j);
    r.kl = s.x * (1.0f / 254.0f);
    r.kh = s.y * (1.0f / (254.0f * 16.0f));
    r.sxl = t.x + t.y;
    r.sxh = t.z + t.w;
}
__device__ __forceinline__ void load_x(Q6::XRegs &r, int xc, int col, int sub)
{
    const int j0 = col * 16 + (sub >> 1) * 8 + (sub & 1);
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const int j = j0 + 2 * g, at = chunk_at(j) * 16;
        const uint4 a = *reinterpret_cast<const uint4 *>(smem + kX + at), b = *reinterpret_cast<const uint4 *>(smem + kX + xc + at);
        r.q1[4 * g] = a.x; r.q1[4 * g + 1] = a.y; r.q1[4 * g + 2] = a.z; r.q1[4 * g + 3] = a.w;
        r.q2[4 * g] = b.x; r.q2[4 * g + 1] = b.y; r.q2[4 * g + 2] = b.z; r.q2[4 * g + 3] = b.w;
        r.k[g] = x_scale(xc)[j >> 1] * (1.0f / 254.0f);
        r.sx32[g] = 32.0f * x_sum(xc)[j];
    }
}

// A row is summed in the order of the streaming matvec: groups of blocks (four lanes a block) as a tree, lanes far apart first, then
// the groups one after the other. Pass by pass: 2^lv blocks side by side, groups of 2^lt of them (one, or several where the groups are
// small), a reduction per pass. Where a row is an even number of groups of eight (`paired`: lv 3, lt 2), a lane takes in two passes two
// blocks that the tree adds first and adds them itself, with two groups side by side in the warp: a reduction per two passes. A
// row's sum is in the lanes l with (l & result_lanes()) == 0, for the pass's row result_row().
struct Passes {
    int col, step;  // first block of the lane; of a pass
    bool paired;
    __device__ __forceinline__ Passes(int lv, int lt, int q)
    {
        paired = lv == 3 && lt == 2;
        col = paired ? (q & 3) + (q >> 2) * 8 : q & ((1 << lv) - 1);
        step = 1 << lv;
    }
    __device__ __forceinline__ int at(int c) const { return col + (paired ? (c >> 1) * 16 + (c & 1) * 4 : c * step); }
    __device__ __forceinline__ bool reduces(int c) const { return !paired || (c & 1); }
};
template <int RU>
__device__ __forceinline__ int result_lanes(int lv, int lt)
{
    return (((4 << lv) - 1) & ~((4 << lt) - 1)) | ((4 << lt) / RU - 1);
}
template <int RU>
__device__ __forceinline__ int result_row(int lt, int lane)
{
    return (lane & ((4 << lt) - 1)) >> (lt + (RU == 4 ? 0 : 1));
}
template <int RU>
__device__ __forceinline__ float tree_sum(const float (&a)[RU], int lt, int lane)
{
    int off = 2 << lt;
    float v;
    bool hi = (lane & off) != 0;
    if (RU == 4) {
        float k0 = hi ? a[2] : a[0], k1 = hi ? a[3] : a[1];
        k0 += __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[2], off);
        k1 += __shfl_xor_sync(0xffffffffu, hi ? a[1] : a[3], off);
        off >>= 1;
        hi = (lane & off) != 0;
        v = hi ? k1 : k0;
        v += __shfl_xor_sync(0xffffffffu, hi ? k0 : k1, off);
    } else {
        v = hi ? a[1] : a[0];
        v += __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[1], off);
    }
#pragma unroll
    for (int o = 16 / RU; o > 2; o >>= 1)
        if (o < off) v += __shfl_xor_sync(0xffffffffu, v, o);
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
        const float t = v + __shfl_xor_sync(0xffffffffu, v, o);
        v = o < off ? t : v;
    }
    return v;
}
__device__ __forceinline__ float add_groups(float sum, float s, int lv, int lt, int lane)
{
    if (lt == lv) return sum + s;
    const int first = (lane & ~((4 << lv) - 1)) | (lane & ((4 << lt) - 1)), end = 1 << (lv - lt);
#pragma unroll 1
    for (int j = 0; j < end; j += 4) {
        float t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) t[i] = __shfl_sync(0xffffffffu, s, first + ((j + i) * 4 << lt));
#pragma unroll
        for (int i = 0; i < 4; i++) sum = j + i < end ? sum + t[i] : sum;
    }
    return sum;
}

// Products that are not fused into what follows
__device__ __forceinline__ float4 times(const float4 a, const float4 b)
{
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}

// Stages K columns (every thread of the CTA calls it; K a multiple of 256): src holds floats, or cells if tag != 0. norm_w:
// RMS-normalised with it (K <= 16 kWork: the whole vector in registers). logit_cell (with norm_w): the row of shared memory at
// off_row times the normalised vector goes there with the tag, before the splitting starts. Returns whether the CTA has given up.
//
// The sums are added in the order of the kernels that do the same layer by layer, so that both give the same bits (a rounding of
// another order grows: where a router has two logits as close, another expert). Two orders exist. `fold`: the norm inside the
// matvec and the one-launch expert block, twelve warps of which thread t has the quads t, t + 384, ... and the logit takes the
// scale afterwards; here thread t does the work of threads t and, below 128, t + 256, from shared memory. Otherwise: a norm kernel
// of 1024 threads (column c in thread c mod 1024) and a router of 128 (quad q in thread q mod 128) on its result.
__device__ __forceinline__ bool stage_vec(const void *src, uint32_t tag, int K, const float *norm_w, float eps, uint2 *logit_cell, bool fold)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
    const int xc = head().xc, nq = K >> 2;
#pragma unroll 1
    for (int q0 = tid; q0 < nq || norm_w; q0 += kWork * 4) {
        float4 v[4], g[4];
        if (norm_w) {
#pragma unroll
            for (int u = 0; u < 4; u++)
                g[u] = q0 + u * kWork < nq ? __ldg(reinterpret_cast<const float4 *>(norm_w) + q0 + u * kWork) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (tag) {
            uint32_t todo = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                todo |= (q0 + u * kWork < nq ? 1u : 0u) << u;
            }
#pragma unroll 1
            for (uint32_t i = 0; todo; i++) {  // what has not come is asked for again
                uint4 a[4], b[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    a[u] = b[u] = make_uint4(0, 0, 0, 0);
                    if (todo >> u & 1) {
                        const uint2 *p = static_cast<const uint2 *>(src) + 4 * (q0 + u * kWork);
                        a[u] = ld_cells2(p);
                        b[u] = ld_cells2(p + 2);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (a[u].y == tag && a[u].w == tag && b[u].y == tag && b[u].w == tag) {
                        v[u] = make_float4(__uint_as_float(a[u].x), __uint_as_float(a[u].z), __uint_as_float(b[u].x), __uint_as_float(b[u].z));
                        todo &= ~(1u << u);
                    }
                if (*gave_up()) break;
                if (i == kPolls) *gave_up() = 1;
            }
            __syncwarp();
        } else {
#pragma unroll
            for (int u = 0; u < 4; u++)
                v[u] = q0 + u * kWork < nq ? __ldcg(static_cast<const float4 *>(src) + q0 + u * kWork) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (norm_w) {
            const float4 *row = reinterpret_cast<const float4 *>(smem + head().off_row);
            // (idle until gate / up is requested; before the first projections, where it is not, the row is)
            float4 *raw = reinterpret_cast<float4 *>(smem + (logit_cell || !fold ? head().off_ring : head().off_row)), *weighted = raw + nq;
            if (fold) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (q0 + u * kWork < nq) {
                        raw[q0 + u * kWork] = v[u];
                        if (logit_cell) weighted[q0 + u * kWork] = times(v[u], g[u]);
                    }
                cta_sync();
                float s[4] = {0.f, 0.f, 0.f, 0.f}, d[2] = {0.f, 0.f};  // s: the sum behind the scale; 2, 3: behind the logit's
#pragma unroll
                for (int u = 0; u < 3; u++) {
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const int q = tid + kWork * k + 384 * u;
                        if (q >= nq || (k && warp >= 4)) break;
                        const float4 x = raw[q];
                        s[k] = fmaf(x.x, x.x, s[k]); s[k] = fmaf(x.y, x.y, s[k]); s[k] = fmaf(x.z, x.z, s[k]); s[k] = fmaf(x.w, x.w, s[k]);
                        if (logit_cell) {
                            const float4 r = row[q], h = weighted[q];
                            s[2 + k] = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, s[2 + k]))));
                            d[k] = fmaf(r.x, h.x, d[k]); d[k] = fmaf(r.y, h.y, d[k]); d[k] = fmaf(r.z, h.z, d[k]); d[k] = fmaf(r.w, h.w, d[k]);
                        }
                    }
                }
                const float all = tree_sum<4>(s, 3, lane), dots = tree_sum<2>(d, 3, lane);
                const int k4 = result_row<4>(3, lane), k2 = result_row<2>(3, lane);
                if ((lane & result_lanes<4>(3, 3)) == 0 && (!(k4 & 1) || warp < 4)) M.red[k4 >> 1][warp + 8 * (k4 & 1)] = all;
                if ((lane & result_lanes<2>(3, 3)) == 0 && (!k2 || warp < 4)) M.red[2][warp + 8 * k2] = dots;
            } else {
                float s[4] = {0.f, 0.f, 0.f, 0.f};  // of four threads of the norm kernel
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    s[0] = fmaf(v[u].x, v[u].x, s[0]);
                    s[1] = fmaf(v[u].y, v[u].y, s[1]);
                    s[2] = fmaf(v[u].z, v[u].z, s[2]);
                    s[3] = fmaf(v[u].w, v[u].w, s[3]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int e = 0; e < 4; e++) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
                if ((lane & 7) == 0) M.red32[tid >> 3] = (s[0] + s[2]) + (s[1] + s[3]);
            }
            cta_sync();
            float t = 0.0f;
            if (fold) {  // lanes 30 and 31 of the last warp: the logit and the sum its scale takes
                const float *red = M.red[warp == kWarps - 1 && lane >= 30 ? 32 - lane : 0];
#pragma unroll
                for (int w = 0; w < 12; w++) t += red[w];
            } else {
                t = warp_sum(M.red32[lane]);
            }
            float scale = 1.0f / sqrtf(t / static_cast<float>(K) + eps);
            if (fold) {
                t = __shfl_sync(0xffffffffu, t, 30);
                if (logit_cell && tid == kWork - 1) st_cell(logit_cell, t * scale, tag);
                scale = __shfl_sync(0xffffffffu, scale, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = times(times(v[u], make_float4(scale, scale, scale, scale)), g[u]);
            if (logit_cell && !fold) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (q0 + u * kWork < nq) raw[q0 + u * kWork] = v[u];
                cta_sync();
                if (tid < 128) {
                    float d = 0.0f;
#pragma unroll 2
                    for (int q = tid; q < nq; q += 128) {
                        const float4 r = row[q], x = raw[q];
                        d = fmaf(r.x, x.x, d); d = fmaf(r.y, x.y, d); d = fmaf(r.z, x.z, d); d = fmaf(r.w, x.w, d);
                    }
                    d = warp_sum(d);
                    if (lane == 0) M.red[0][warp] = d;
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                    if (tid == 0) st_cell(logit_cell, (M.red[0][0] + M.red[0][1]) + (M.red[0][2] + M.red[0][3]), tag);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // ring or row were written as plain memory
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int q = q0 + u * kWork;
            if (q - lane >= nq) break;  // warp-uniform: a warp covers 128 columns
            stage_quad(xc, v[u], 4 * q, lane);
        }
        if (norm_w) break;
    }
    return cta_aborted();
}

// ---- a warp's private ring: it issues its own copies and consumes them, so one "full" barrier per stage is all it takes.
// `parity`: per stage, the parity of its next completion. ----
__device__ __forceinline__ void ring_wait(uint64_t *bars, int s, uint32_t &parity)
{
    wait_copy(&bars[s], (parity >> s) & 1);
    parity ^= 1u << s;
    __syncwarp();
}

// A warp's rows [r0, r0 + n) of a matrix, ur rows a unit (a stage of the ring).
__host__ __device__ __forceinline__ uint32_t stage_bytes_of(uint32_t unit_bytes) { return (unit_bytes + 47u) & ~15u; }
// One lane: the 16-byte-aligned span enclosing a unit's rows (the few extra bytes share a 16-byte granule with valid ones).
__device__ __forceinline__ void issue_unit(const uint8_t *w, int row, int rows, uint32_t row_bytes, uint8_t *dst, uint64_t *bar)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(w) + (size_t)row * row_bytes;
    const uintptr_t e = a + (size_t)rows * row_bytes;
    const uintptr_t a0 = a & ~static_cast<uintptr_t>(15);
    const uint32_t bytes = static_cast<uint32_t>(((e + 15) & ~static_cast<uintptr_t>(15)) - a0);
    mbar_expect_tx(bar, bytes);
    bulk_g2s(dst, reinterpret_cast<const void *>(a0), bytes, bar);
}
// Requests the first units, a lane each; returns the mask of stages in flight.
__device__ __forceinline__ uint32_t prefetch(const uint8_t *w, int r0, int n, uint32_t row_bytes, int log_ur, int stages)
{
    uint8_t *buf = ring();
    uint64_t *bars = ring_bars();
    const int lane = thread_id() & 31, ur = 1 << log_ur, count = min(stages, (n + ur - 1) >> log_ur);
    const uint32_t sb = stage_bytes_of(row_bytes << log_ur);
    if (lane < count) issue_unit(w, r0 + lane * ur, min(ur, n - lane * ur), row_bytes, buf + lane * sb, &bars[lane]);
    __syncwarp();
    return (1u << count) - 1;
}
// Those rows (first units requested by prefetch() with the same arguments) times the staged vector from super-block xcol on:
// dst[row] = value (with keep: added to keep[row], which takes the sum), as a cell if tag != 0. Returns the ring's parities.
template <class F, int RU>
__device__ __forceinline__ uint32_t matvec(const uint8_t *w, int bpr, int lv, int lt, int r0, int n, void *dst, uint32_t tag, float *keep,
                                        int xcol, int stages, uint32_t parity)
{
    uint8_t *buf = ring();
    uint64_t *bars = ring_bars();
    const int xc = head().xc;
    const int lane = thread_id() & 31, q = lane >> 2, sub = lane & 3;
    const int rpp = 8 >> lv, rq = q >> lv, one = result_lanes<RU>(lv, lt);
    const int groups = (bpr + (1 << lv) - 1) >> lv, ur = RU * rpp;
    const Passes P(lv, lt, q);
    const uint32_t row_bytes = bpr * F::kBlockBytes, sb = stage_bytes_of(ur * row_bytes);
    typename F::XRegs xr;
    int s = 0;
#pragma unroll 1
    for (int r = 0; r < n; r += ur) {
        ring_wait(bars, s, parity);
        uint32_t skew = 0;
        if (F::kBlockBytes % 16) skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(w) + (size_t)(r0 + r) * row_bytes) & 15u;
        const uint8_t *base = buf + s * sb + skew + rq * row_bytes;
        float sum = 0.0f, acc[RU];
#pragma unroll
        for (int i = 0; i < RU; i++) acc[i] = 0.0f;
#pragma unroll 1
        for (int c = 0; c < groups; c++) {
            const int col = P.at(c);
            const bool in = col < bpr;  // a ragged last pass
            const int at = in ? col : 0;
            if (groups > 1 || r == 0) load_x(xr, xc, xcol + at, sub);
#pragma unroll
            for (int i = 0; i < RU; i++) {
                if (i > 0 && r + i * rpp >= n) break;
                const float d = F::block_dot(base + (i * rpp) * row_bytes + at * F::kBlockBytes, sub, xr);
                acc[i] += in ? d : 0.0f;
            }
            if (P.reduces(c)) {
                sum = add_groups(sum, tree_sum<RU>(acc, lt, lane), lv, lt, lane);
#pragma unroll
                for (int i = 0; i < RU; i++) acc[i] = 0.0f;
            }
        }
        __syncwarp();
        const int nr = r + stages * ur;
        if (lane == 0 && nr < n) issue_unit(w, r0 + nr, min(ur, n - nr), row_bytes, buf + s * sb, &bars[s]);
        const int row = r + result_row<RU>(lt, lane) * rpp + rq;
        if ((lane & one) == 0 && row < n) {
            float o = sum;
            if (keep) keep[r0 + row] = o += keep[r0 + row];
            if (tag)
                st_cell(static_cast<uint2 *>(dst) + r0 + row, o, tag);
            else
                static_cast<float *>(dst)[r0 + row] = o;
        }
        if (++s == stages) s = 0;
    }
    return parity;
}

// Item range of work warp `gid` in a split; n = 0 if it has no part.
__device__ __forceinline__ void share(const volatile Split &sp, int gid, int &i0, int &n)
{
    const int i = gid - sp.w0;
    const bool in = i >= 0 && i < sp.nw;
    i0 = in ? i * sp.per + min(i, sp.rem) : 0;
    n = in ? sp.per + (i < sp.rem ? 1 : 0) : 0;
}

// ---- attention ----
__device__ __forceinline__ void mma16816(float (&c)[4], const uint4 &a, uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// A head's 128 values, four per lane at lane + 32 i: RMS norm with the weights M.norm[which] (unless !normed) and rotation by M.rope.
__device__ __forceinline__ float4 norm_rope(float4 v, int which, bool normed, float eps)
{
    const Misc &M = misc();
    const int lane = thread_id() & 31;
    const float *w = M.norm[which];
    const float ss = warp_sum(fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x))));
    if (normed) {
        const float f = 1.0f / sqrtf(ss * (1.0f / 128.0f) + eps);
        v.x = v.x * f * w[lane];
        v.y = v.y * f * w[lane + 32];
        v.z = v.z * f * w[lane + 64];
        v.w = v.w * f * w[lane + 96];
    }
    const float c0 = M.rope[lane], c1 = M.rope[lane + 32], s0 = M.rope[64 + lane], s1 = M.rope[96 + lane];
    return make_float4(v.x * c0 - v.z * s0, v.y * c1 - v.w * s1, v.x * s0 + v.z * c0, v.y * s1 + v.w * c1);
}

// K / V rows of a tile of 16 positions, a row per lane; only rows before `pos`: the cache has nothing yet at the others
__device__ __forceinline__ void load_kv(const __half *kv_k, const __half *kv_v, int tile, int pos, int n_kv, int kvh)
{
    const int lane = thread_id() & 31, r = lane & 15, rows = min(16, pos - tile * 16);
    uint8_t *buf = ring();
    uint64_t *bar = ring_bars();
    if (lane == 0) mbar_expect_tx(bar, 2 * rows * 256);
    __syncwarp();
    if (r < rows)
        bulk_g2s(buf + (lane < 16 ? r * kKPitch : kVOff + r * kVPitch), (lane < 16 ? kv_k : kv_v) + ((size_t)(tile * 16 + r) * n_kv + kvh) * 128,
                 256, bar);
}

// This warp's tiles (tile, tile + kWarps, ... < t1; the first has been requested into the ring) for the 16 query heads whose
// fragments are in shared memory at 0 (hi halves) and 4096 (lo): leaves the unnormalised result [16][kPitch] in the ring, the
// running maxima (log2 domain) and sums in M.am / M.al. The tile of the newest position takes its K and V from the projections
// and, with store, writes them to the cache. Returns the ring's parities.
__device__ __forceinline__ uint32_t attn_tiles(int tile, int t1, int pos, int n_kv, int kvh, __half *kv_k, __half *kv_v, bool store,
                                            const uint2 *c_k, const uint2 *c_v, uint32_t tag, bool k_normed, float eps,
                                            uint32_t parity)
{
    uint8_t *buf = ring();
    Misc &M = misc();
    const int lane = thread_id() & 31, warp = thread_id() >> 5, g = lane >> 2, t = lane & 3;
    uint64_t *bars = M.bars[warp];
    float O[16][4];
#pragma unroll
    for (int u = 0; u < 16; u++) O[u][0] = O[u][1] = O[u][2] = O[u][3] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    const uint8_t *ka = buf + g * kKPitch + t * 16;
    const uint32_t va = smem_u32(buf) + kVOff + ((lane & 7) + ((lane >> 3) & 1) * 8) * kVPitch + (lane >> 4) * 16;
#pragma unroll 1
    for (;;) {
        ring_wait(bars, 0, parity);
        if (tile == (pos >> 4)) {
            float kv[4], vv[4];
            wait_values4(c_k + kvh * 128 + lane, tag, kv);
            wait_values4(c_v + kvh * 128 + lane, tag, vv);
            __syncwarp();
            const float4 kr = norm_rope(make_float4(kv[0], kv[1], kv[2], kv[3]), 1, k_normed, eps);
            const float kn[4] = {kr.x, kr.y, kr.z, kr.w};
            const size_t row = ((size_t)pos * n_kv + kvh) * 128;
            uint8_t *kd = buf + (pos & 15) * kKPitch, *vd = buf + kVOff + (pos & 15) * kVPitch;
            // the rows behind it: their scores are masked, but a probability of 0 times what the ring held might be NaN
            for (int i = ((pos & 15) + 1) * 16 + lane; i < 256; i += 32)
                *reinterpret_cast<uint4 *>(buf + kVOff + (i >> 4) * kVPitch + (i & 15) * 16) = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int d = lane + 32 * i;
                const __half hk = __float2half_rn(kn[i]), hv = __float2half_rn(vv[i]);
                *reinterpret_cast<__half *>(kd + 2 * d) = hk;
                *reinterpret_cast<__half *>(vd + 2 * d) = hv;
                if (store) {
                    kv_k[row + d] = hk;
                    kv_v[row + d] = hv;
                }
            }
            __syncwarp();
        }
        float S[2][4];
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) S[n][e] = 0.0f;
#pragma unroll 1
        for (int jj = 0; jj < 4; jj++) {  // 32 dims, eight of a lane: two steps
            const uint8_t *f = smem + kX + (2 * jj * 32 + lane) * 16;
            const uint4 h0 = *reinterpret_cast<const uint4 *>(f), h1 = *reinterpret_cast<const uint4 *>(f + 512);
            const uint4 lo0 = *reinterpret_cast<const uint4 *>(f + 4096), lo1 = *reinterpret_cast<const uint4 *>(f + 4096 + 512);
            const uint4 b0 = *reinterpret_cast<const uint4 *>(ka + jj * 64), b1 = *reinterpret_cast<const uint4 *>(ka + 8 * kKPitch + jj * 64);
            mma16816(S[0], h0, b0.x, b0.y);
            mma16816(S[1], h0, b1.x, b1.y);
            mma16816(S[0], lo0, b0.x, b0.y);
            mma16816(S[1], lo0, b1.x, b1.y);
            mma16816(S[0], h1, b0.z, b0.w);
            mma16816(S[1], h1, b1.z, b1.w);
            mma16816(S[0], lo1, b0.z, b0.w);
            mma16816(S[1], lo1, b1.z, b1.w);
        }
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const bool in = tile * 16 + n * 8 + 2 * t + e <= pos;
                S[n][e] = in ? S[n][e] : -INFINITY;
                S[n][2 + e] = in ? S[n][2 + e] : -INFINITY;
                mx0 = fmaxf(mx0, S[n][e]);
                mx1 = fmaxf(mx1, S[n][2 + e]);
            }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        }
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);  // finite: a tile holds at least one position
        const float r0 = exp2f(m0 - n0), r1 = exp2f(m1 - n1);
        m0 = n0;
        m1 = n1;
        l0 *= r0;
        l1 *= r1;
#pragma unroll
        for (int u = 0; u < 16; u++) {
            O[u][0] *= r0;
            O[u][1] *= r0;
            O[u][2] *= r1;
            O[u][3] *= r1;
        }
#pragma unroll
        for (int n = 0; n < 2; n++) {
            S[n][0] = exp2f(S[n][0] - n0);
            S[n][1] = exp2f(S[n][1] - n0);
            S[n][2] = exp2f(S[n][2] - n1);
            S[n][3] = exp2f(S[n][3] - n1);
            l0 += S[n][0] + S[n][1];
            l1 += S[n][2] + S[n][3];
        }
        const uint4 pa = make_uint4(pack2(S[0][0], S[0][1]), pack2(S[0][2], S[0][3]), pack2(S[1][0], S[1][1]), pack2(S[1][2], S[1][3]));
#pragma unroll
        for (int u = 0; u < 16; u += 2) {
            uint32_t b[4];
            ldmatrix4_trans(va + u * 16, b);
            mma16816(O[u], pa, b[0], b[1]);
            mma16816(O[u + 1], pa, b[2], b[3]);
        }
        tile += kWarps;
        if (tile >= t1) break;
        __syncwarp();
        load_kv(kv_k, kv_v, tile, pos, n_kv, kvh);
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (t == 0) {
        M.am[warp][g] = m0;
        M.am[warp][g + 8] = m1;
        M.al[warp][g] = l0;
        M.al[warp][g + 8] = l1;
    }
    __syncwarp();
    float *ow = reinterpret_cast<float *>(buf);
#pragma unroll
    for (int u = 0; u < 16; u++) {
        *reinterpret_cast<float2 *>(ow + g * kPitch + 8 * u + 2 * t) = make_float2(O[u][0], O[u][1]);
        *reinterpret_cast<float2 *>(ow + (g + 8) * kPitch + 8 * u + 2 * t) = make_float2(O[u][2], O[u][3]);
    }
    return parity;
}

// The warps bring nh query heads (128 cells each) into the fragments (hi + lo halves of q * scale * log2 e); the other rows are zero.
__device__ __forceinline__ void q_fragments(const uint2 *c_q, uint32_t tag, int nh, bool q_normed, float eps, float sc)
{
    const int lane = thread_id() & 31;
#pragma unroll 1
    for (int h = thread_id() >> 5; h < 16; h += kWarps) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (h < nh) {
            wait_values4(c_q + h * 128 + lane, tag, v);
            __syncwarp();
            const float4 r = norm_rope(make_float4(v[0], v[1], v[2], v[3]), 0, q_normed, eps);
            v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = lane & 7;  // of the eight dims 32 i + 8 t .. + 7: the lower four in step 2 i, the others in the next
            const int at = ((2 * i + (e >> 2)) * 32 + (h & 7) * 4 + (lane >> 3)) * 16 + ((h >> 3) + (e & 2)) * 4 + (e & 1) * 2;
            const float s = v[i] * sc;
            const __half hi = __float2half_rn(s);
            *reinterpret_cast<__half *>(smem + kX + at) = hi;
            *reinterpret_cast<__half *>(smem + kX + 4096 + at) = __float2half_rn(s - __half2float(hi));
        }
    }
}

// The CTA's partial of nw warps: one head per warp, four dims per lane, into the cells of slot `slot`.
__device__ __forceinline__ void attn_partial(int nw, int nh, uint2 *c_part, uint2 *c_ml, int slot, uint32_t tag)
{
    Misc &M = misc();
    const int lane = thread_id() & 31;
#pragma unroll 1
    for (int h = thread_id() >> 5; h < nh; h += kWarps) {
        float m = -INFINITY, s = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) m = fmaxf(m, w < nw ? M.am[w][h] : -INFINITY);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            if (w >= nw) break;
            const float f = exp2f(M.am[w][h] - m);
            const float4 o = *reinterpret_cast<const float4 *>(smem + head().off_ring + w * head().ring_bytes + (h * kPitch + 4 * lane) * 4);
            s = fmaf(M.al[w][h], f, s);
            a.x = fmaf(o.x, f, a.x); a.y = fmaf(o.y, f, a.y); a.z = fmaf(o.z, f, a.z); a.w = fmaf(o.w, f, a.w);
        }
        uint2 *p = c_part + ((size_t)slot * 16 + h) * 128 + 4 * lane;
        st_cells2(p, a.x, a.y, tag);
        st_cells2(p + 2, a.z, a.w, tag);
        if (lane == 0) st_cells2(c_ml + ((size_t)slot * 16 + h) * 2, m, s, tag);
    }
}

// Merges the nc chunks' partials of one head (hq of head block b), cells of the result. Warp 0 has the chunks' maxima and sums, the
// others bring the partials into shared memory (the ring is idle); then a thread per dim adds them up in chunk order.
__device__ __forceinline__ void merge_head(int b, int hq, int nc, int chunks, const uint2 *c_part, const uint2 *c_ml, uint2 *dst, uint32_t tag)
{
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
    float *fm = reinterpret_cast<float *>(smem + kX), *fl = fm + kMaxChunks, *part = reinterpret_cast<float *>(smem + head().off_ring);
    if (warp == 0) {
        constexpr int kPer = kMaxChunks / 32;
        float m[kPer], l[kPer], mt = -INFINITY, lt = 0.0f;
#pragma unroll 1
        for (uint32_t i = 0;; i++) {
            bool ok = true;
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                m[u] = -INFINITY;
                l[u] = 0.0f;
                if (lane + 32 * u < nc) {
                    const uint4 v = ld_cells2(c_ml + (((size_t)b * chunks + lane + 32 * u) * 16 + hq) * 2);
                    m[u] = __uint_as_float(v.x);
                    l[u] = __uint_as_float(v.z);
                    ok = ok && v.y == tag && v.w == tag;
                }
            }
            if (ok || *gave_up()) break;
            if (i == kPolls) *gave_up() = 1;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kPer; u++) mt = fmaxf(mt, m[u]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            if (32 * u >= nc) break;
            const float f = exp2f(m[u] - mt);  // 0 beyond the last chunk
            fm[lane + 32 * u] = f;
            lt = fmaf(l[u], f, lt);            // chunk c in lane c mod 16
            lt = fmaf(__shfl_down_sync(0xffffffffu, l[u], 16), __shfl_down_sync(0xffffffffu, f, 16), lt);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) lt += __shfl_xor_sync(0xffffffffu, lt, o);
        if (lane == 0) *fl = lt > 0.0f ? 1.0f / lt : 0.0f;
    } else {
#pragma unroll 1
        for (int c0 = warp - 1; c0 < nc; c0 += 6 * (kWarps - 1)) {
            uint4 o0[6], o1[6];
#pragma unroll 1
            for (uint32_t i = 0;; i++) {
                bool ok = true;
#pragma unroll
                for (int u = 0; u < 6; u++) {
                    const uint2 *p = c_part + (((size_t)b * chunks + min(c0 + u * (kWarps - 1), nc - 1)) * 16 + hq) * 128 + 4 * lane;
                    o0[u] = ld_cells2(p);
                    o1[u] = ld_cells2(p + 2);
                    ok = ok && o0[u].y == tag && o0[u].w == tag && o1[u].y == tag && o1[u].w == tag;
                }
                if (ok || *gave_up()) break;
                if (i == kPolls) *gave_up() = 1;
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 6; u++) {
                const int c = c0 + u * (kWarps - 1);
                if (c >= nc) break;
                *reinterpret_cast<uint4 *>(part + c * 128 + 4 * lane) = make_uint4(o0[u].x, o0[u].z, o1[u].x, o1[u].z);
            }
        }
    }
    cta_sync();
    if (tid < 128) {
        float o = 0.0f;
        float p[8];
#pragma unroll
        for (int u = 0; u < 8; u++) p[u] = u < nc ? part[u * 128 + tid] : 0.0f;
#pragma unroll 1
        for (int c = 0; c < nc; c += 8) {  // (the weights beyond the last chunk are 0)
            const float4 f0 = *reinterpret_cast<const float4 *>(fm + c), f1 = *reinterpret_cast<const float4 *>(fm + c + 4);
            const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const float x = p[u];
                p[u] = c + 8 + u < nc ? part[(c + 8 + u) * 128 + tid] : 0.0f;
                o = fmaf(x, f[u], o);
            }
        }
        st_cell(dst + tid, o * *fl, tag);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the ring was written and read as plain memory
    cta_sync();
}

// ---- selection ----
__device__ __forceinline__ uint32_t ordered(float v)
{
    const uint32_t b = __float_as_uint(v + 0.0f);  // -0 counts as 0
    return min(b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u), 0xFFFFFFFEu);
}
__device__ __forceinline__ float unordered(uint32_t k) { return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xFFFFFFFFu)); }

// One thread: the reference's walk over the logits in (e % 32, e / 32) order (n <= 32 k: nothing is dropped before the merge),
// replacing the first minimum when strictly greater. M.slot_pos: candidate of each slot.
__device__ __noinline__ void walk(int n, int k)
{
    Misc &M = misc();
#pragma unroll 1
    for (int i = 0; i < k; i++) M.slot_pos[i] = -1;
#pragma unroll 1
    for (int p = 0; p < n; p++) {
        int at = 0;
        uint32_t least = 0xFFFFFFFFu;
#pragma unroll 1
        for (int i = 0; i < k; i++) {
            const uint32_t v = M.slot_pos[i] < 0 ? 0 : M.key[M.slot_pos[i]];
            if (v < least) {
                least = v;
                at = i;
            }
        }
        if (M.key[p] > least) M.slot_pos[at] = p;
    }
}

// The k largest of n logits (every thread of the CTA calls it): M.top_id, the largest first, and what select_weights() needs. False:
// the CTA has given up.
__device__ __forceinline__ bool select_experts(const uint2 *cells, uint32_t tag, int n, int k)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
    static_assert(kWork >= kMaxExperts, "a thread per logit");
    if (tid < kMaxExperts) {
        if (tid < n) {
            const int l = tid & 31, p = l * (n >> 5) + min(l, n & 31) + (tid >> 5);  // its place in the walk
            M.eid[p] = static_cast<uint8_t>(tid);
            M.key[p] = ordered(wait_value(cells + tid, tag));
        } else {
            M.key[tid] = 0;
        }
    }
    if (tid == 0) M.walked = 0;
    if (cta_aborted()) return false;
    {
        const int half = ((n + 7) >> 3) * 4, lo = (tid & 1) ? half : 0, hi = lo + half;  // keys beyond n are 0
#pragma unroll 1
        for (int p = tid >> 1, it = 0; p - (lane >> 1) < n; p += kWork / 2, it++) {  // warp-uniform; two threads per candidate
            const uint32_t me = M.key[p];
            uint32_t count = 0;  // of larger ones (an equal one before it counts: a key is never the largest integer); high half: before it
#pragma unroll 2
            for (int i = lo; i < hi; i += 4) {
                const uint4 o = *reinterpret_cast<const uint4 *>(&M.key[i]);
                const uint32_t c0 = i < p, c1 = i + 1 < p, c2 = i + 2 < p, c3 = i + 3 < p;
                count += (o.x + c0 > me ? (c0 << 16) + 1 : 0) + (o.y + c1 > me ? (c1 << 16) + 1 : 0) + (o.z + c2 > me ? (c2 << 16) + 1 : 0) +
                         (o.w + c3 > me ? (c3 << 16) + 1 : 0);
            }
            count += __shfl_xor_sync(0xffffffffu, count, 1);
            const int rank = count & 0xFFFF;
            const bool mine = p < n && !(tid & 1);
            if (mine && rank <= k) {
                M.top_id[rank] = M.eid[p];
                M.top_pos[rank] = p;
                M.top_key[rank] = me;
            }
            // the walk accepts what fewer than k before it are as large as
            const bool accept = mine && static_cast<int>(count >> 16) < k;
            const uint32_t bits = __ballot_sync(0xffffffffu, accept);
            if (lane == 0) M.accepted[it * kWarps + warp] = bits;
            if (!(tid & 1)) M.acc_key[p] = accept ? me : 0xFFFFFFFFu;  // (larger than any key)
        }
    }
    cta_sync();
    if (n > k && M.top_key[k - 1] == M.top_key[k]) {  // the same for the whole CTA
        cta_sync();
        if (tid == 0) {
            walk(n, k);
            for (int i = 0; i < k; i++) {
                M.top_id[i] = M.eid[M.slot_pos[i]];
                M.top_pos[i] = M.slot_pos[i];
                M.top_key[i] = M.key[M.slot_pos[i]];
            }
            M.walked = 1;
        }
        cta_sync();
    }
    return true;
}
// The reference's output slots of the selected (M.order) and their weights (M.swt): of the accepted candidates the i-th takes slot i,
// a later one that of the candidate it replaces, the one of rank i - k from below. Not needed before the down projection, hence in
// two parts. First, by all warps while their first weights are on the way: the ranks among the accepted.
__device__ __forceinline__ void rank_accepted(int n)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31;
    if (M.walked != 1) {
        const int half = ((n + 7) >> 3) * 4, lo = (tid & 1) ? half : 0, hi = lo + half;
#pragma unroll 1
        for (int p = tid >> 1; p - (lane >> 1) < n; p += kWork / 2) {
            const uint32_t me = M.acc_key[p];
            uint32_t count = 0;  // smaller ones; high half: equal ones
#pragma unroll 1
            for (int i = lo; i < hi; i += 4) {
                const uint4 o = *reinterpret_cast<const uint4 *>(&M.acc_key[i]);
                count += (o.x < me) + (o.y < me) + (o.z < me) + (o.w < me);
                count += ((o.x == me) + (o.y == me) + (o.z == me) + (o.w == me)) << 16;
            }
            count += __shfl_xor_sync(0xffffffffu, count, 1);
            if (!(tid & 1) && me != 0xFFFFFFFFu) {
                int t = __popc(M.accepted[p >> 4] & ((1u << (2 * (p & 15))) - 1u));
#pragma unroll 1
                for (int w = 0; w < p >> 4; w++) t += __popc(M.accepted[w]);
                M.by_rank[count & 0xFFFF] = static_cast<uint8_t>(t);
                if (count >> 17) M.walked = 2;  // equal ones among them: the walk itself
            }
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&M.ranked);
}
// Then, by one warp.
__device__ __forceinline__ void select_weights(int n, int k, uint32_t parity)
{
    Misc &M = misc();
    const int lane = thread_id() & 31;
    wait_copy(&M.ranked, parity);
    const int walked = *const_cast<volatile int *>(&M.walked);
    if (walked == 0) {
        const int m = __reduce_add_sync(0xffffffffu, lane * 16 < n ? __popc(M.accepted[lane]) : 0);
        if (lane < k) {  // the i-th largest: where its chain of replacements began (each of them came before what replaced it)
            int t = M.by_rank[max(m - 1 - lane, 0)];
#pragma unroll 1
            for (int i = 0; i < n && t >= k; i++) t = M.by_rank[t - k];
            M.order[t < k ? t : 0] = lane;  // (t >= k: only if the CTA has given up)
        }
    } else if (walked == 1) {
        if (lane < k) M.order[lane] = lane;
    } else {
        if (lane == 0) walk(n, k);
        __syncwarp();
        if (lane < k) {
#pragma unroll 1
            for (int i = 0; i < k; i++)
                if (M.top_pos[i] == M.slot_pos[lane]) M.order[lane] = i;
        }
    }
    __syncwarp();
    const float v = lane < k ? unordered(M.top_key[M.order[lane]]) : -INFINITY;
    float mx = v;
#pragma unroll
    for (int o = kMaxK / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = lane < k ? expf(v - mx) : 0.0f;
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kMaxK; i++) sum += __shfl_sync(0xffffffffu, e, i);  // (0 beyond the k-th)
    if (lane < k) M.swt[lane] = e / sum;
}

// ---- gate / up: items [i0, i0 + n), item i = a pass of gate rows and the same up rows of the i / ipe-th routed expert. Two items
// a stage: their four products hide one another's latency, and one reduction serves them (a warp has 3 to 11 items). ----
// Every lane calls it: lane 2 j + h requests half h (gate, up) of item i + j of the stage, j < 2.
__device__ __forceinline__ void issue_items(const uint8_t *experts, size_t estride, uint32_t up_off, int i, int end, int ipe, uint32_t magic,
                                            uint32_t half, bool mine, int j, int h, uint8_t *dst, uint64_t *bar)
{
    const int item = i + j, slot = __umulhi(item, magic);
    const bool in = mine && item < end;
    if (in && j == 0 && h == 0) mbar_expect_tx(bar, (i + 1 < end ? 4 : 2) * half);
    __syncwarp();
    if (in) bulk_g2s(dst + (2 * j + h) * half, experts + (size_t)misc().top_id[slot] * estride + (item - slot * ipe) * half + (h ? up_off : 0), half, bar);
}
// Writes SwiGLU's result as cells act[slot * EFF + row].
__device__ __forceinline__ uint32_t gate_up(const uint8_t *experts, size_t estride, uint32_t up_off, int i0, int n, int ipe, uint32_t magic,
                                            int bpr, int lv, int lt, int EFF, uint2 *act, uint32_t tag, int stages, uint32_t parity)
{
    uint8_t *buf = ring();
    uint64_t *bars = ring_bars();
    const int xc = head().xc;
    const int lane = thread_id() & 31, q = lane >> 2, sub = lane & 3;
    const int rpp = 8 >> lv, rq = q >> lv, one = result_lanes<4>(lv, lt);
    const int groups = (bpr + (1 << lv) - 1) >> lv, end = i0 + n;
    const Passes P(lv, lt, q);
    const uint32_t row_bytes = bpr * kQ4KBlock, half = rpp * row_bytes, sb = 4 * half;
    const int ij = (lane >> 1) & 1, ih = lane & 1, is = lane >> 2;  // of a request: item, half, stage
    issue_items(experts, estride, up_off, i0 + 2 * is, end, ipe, magic, half, is < stages, ij, ih, buf + is * sb, &bars[is < stages ? is : 0]);
    rank_accepted(head().n_experts);
    Q4::XRegs xr;
    int s = 0;
#pragma unroll 1
    for (int i = i0; i < end; i += 2) {
        ring_wait(bars, s, parity);
        const uint8_t *base = buf + s * sb + rq * row_bytes;
        float sum = 0.0f, acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // gate, up of the two items
#pragma unroll 1
        for (int c = 0; c < groups; c++) {
            const int col = P.at(c);
            const bool in = col < bpr;  // a ragged last pass
            const int at = in ? col : 0;
            if (groups > 1 || i == i0) load_x(xr, xc, at, sub);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (u == 2 && i + 1 >= end) break;
                const float d = Q4::block_dot(base + u * half + at * kQ4KBlock, sub, xr);
                acc[u] += in ? d : 0.0f;
            }
            if (P.reduces(c)) {
                sum = add_groups(sum, tree_sum<4>(acc, lt, lane), lv, lt, lane);
#pragma unroll
                for (int u = 0; u < 4; u++) acc[u] = 0.0f;
            }
        }
        __syncwarp();
        issue_items(experts, estride, up_off, i + 2 * stages, end, ipe, magic, half, lane < 4, ij, ih, buf + s * sb, &bars[s]);
        const float g = sum, u = __shfl_xor_sync(0xffffffffu, g, 1 << lt);  // which ^ 1: a quarter of a group's lanes away
        const int which = result_row<4>(lt, lane), item = i + (which >> 1);
        if ((lane & one) == 0 && !(which & 1) && item < end) {
            const int slot = __umulhi(item, magic);
            st_cell(act + slot * EFF + (item - slot * ipe) * rpp + rq, g / (1.0f + expf(-g)) * u, tag);
        }
        if (++s == stages) s = 0;
    }
    return parity;
}

__global__ void __launch_bounds__(kWork, 1) persist_kernel(const __grid_constant__ Params params)
{
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5, cta = cta_id(), grid = gridDim.x;
    Misc &M = misc();
    const volatile Head &P = M.head;
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(static_cast<const Head *>(&params));
        for (int i = tid; i < static_cast<int>(sizeof(Head) / 4); i += kWork) reinterpret_cast<uint32_t *>(&M.head)[i] = src[i];
    }
    if (tid < kWarps * kStages) mbar_init(&M.bars[0][0] + tid, 1);
    if (tid == kWork - 1) {
        mbar_init(&M.row_bar, 1);
        mbar_init(&M.ranked, kWarps);
        M.abort_flag = 0;
        M.row_pend = -1;
    }
    __syncthreads();
    // What a warp does in every layer, in shared memory: it is looked up once per operation
    if (lane == 0) {
        const int gid = warp * grid + cta;
        int i0, n, m = 0;
        share(P.sq, gid, i0, n);  // rows of one of the three matrices behind the first norm
        if (gid >= P.sk.w0) { m = 1; share(P.sk, gid, i0, n); }
        if (gid >= P.sv.w0) { m = 2; share(P.sv, gid, i0, n); }
        M.own[warp][kQKV] = make_int2(i0 << (3 - P.mH.lv), n << (3 - P.mH.lv));
        M.own_qm[warp] = m;
        share(P.sg, gid, i0, n);
        M.own[warp][kExperts] = make_int2(i0, n);
        // O, down: the CTA's rows of the hidden vector; down: shared by the warps of a slot
        const int R0 = static_cast<int>(static_cast<unsigned>(P.H) * cta / grid), R1 = static_cast<int>(static_cast<unsigned>(P.H) * (cta + 1) / grid);
        const int wps = kWarps / P.k, slot = warp / wps, part = warp - slot * wps, per = (R1 - R0 + wps - 1) / wps;
        M.own[warp][kO] = make_int2(R0 + (R1 - R0) * warp / kWarps, (R1 - R0) * (warp + 1) / kWarps - (R1 - R0) * warp / kWarps);
        M.own_slot[warp] = slot;
        M.R0 = R0;
        M.rows = R1 - R0;
        M.own[warp][kDown] = make_int2(R0 + part * per, slot < P.k ? max(0, min(per, R1 - R0 - part * per)) : 0);
    }
    mbar_fence_init();
    __syncthreads();
    auto has_row = [&] { return cta_id() < P.n_experts; };
    auto request_row = [&](int l) {
        mbar_expect_tx(&M.row_bar, P.H * 4);
        bulk_g2s(smem + P.off_row, params.L[l].router + (size_t)cta_id() * P.H, P.H * 4, &M.row_bar);
    };

    uint32_t parity = 0, pend = 0;  // pend: stages in flight while the CTA may still give up
    // One pass of the loop: an operation (there is one copy of every step's code), preceded by the request for its weights. The
    // pass before the first only requests.
#pragma unroll 1
    for (int l = -1, op = kDown;;) {
        const int tid = thread_id(), warp = tid >> 5, cta = cta_id();
        const uint32_t tag = M.tag + l;
        if (l >= 0) {
            const Layer &L = params.L[l];
            // ---- the input vector ----
            {
                const void *src = P.c_act;
                const float *norm_w = nullptr;
                uint32_t t = tag;
                int K = P.k * P.EFF;
                uint2 *logit = nullptr;
                if (op == kQKV) {
                    src = l == 0 ? static_cast<const void *>(P.hidden) : P.c_h0;
                    t = l == 0 ? 0 : tag - 1;
                    norm_w = L.attn_norm;
                    K = P.H;
                } else if (op == kO) {
                    src = P.c_attn;
                    K = P.QD;
                    if (tid == 0 && has_row()) {
                        M.row_pend = l & 1;
                        request_row(l);
                    }
                } else if (op == kExperts) {  // the router logit of this CTA's expert on the way
                    src = P.c_h1;
                    norm_w = L.ffn_norm;
                    K = P.H;
                    logit = has_row() ? P.c_logit + cta : nullptr;
                    if (has_row()) wait_copy(&M.row_bar, l & 1);
                    if (tid == 0) M.row_pend = -1;
                }
                // the norm weights of the heads: on their way while the vector is waited for
                const float *hw = tid < 128 ? L.q_norm : L.k_norm;
                float hn = 0.0f;
                if (op == kQKV && tid < 256 && hw) hn = __ldg(hw + (tid & 127));
                if (stage_vec(src, t, K, norm_w, P.eps, logit, op == kQKV || L.fold)) break;
                if (op == kQKV && tid < 256) M.norm[tid >> 7][tid & 127] = hn;
            }
            // ---- its rows ----
            if (op == kExperts) {
                if (!select_experts(P.c_logit, tag, P.n_experts, P.k)) break;
                const int2 own = M.own[warp][kExperts];
                parity = gate_up(L.experts, L.estride, L.up_off, own.x, own.y, P.ipe, P.ipe_magic, P.mH.bpr, P.mH.lv, P.mH.lt, P.EFF, P.c_act, tag,
                                 P.stages[5], parity);
                if (warp == kWarps - 1) select_weights(P.n_experts, P.k, l & 1);
            } else {
                const int2 own = M.own[warp][op];
                const int qm = M.own_qm[warp], slot = M.own_slot[warp];
                const uint8_t *w = qm == 0 ? L.wq : qm == 1 ? L.wk : L.wv;
                void *dst = qm == 0 ? P.c_q : qm == 1 ? P.c_k : P.c_v;
                float *keep = nullptr;
                const int R0 = M.R0;
                uint32_t t = tag;
                bool q6 = qm == 2 && L.v_q6;
                int bpr = P.mH.bpr, lv = P.mH.lv, lt = P.mH.lt, xcol = 0, kind = q6 ? 1 : 0;
                if (op == kO) {
                    w = L.wo;
                    dst = P.c_h1;
                    keep = M.hid - R0;
                    q6 = false;
                    bpr = P.mQ.bpr;
                    lv = P.mQ.lv;
                    lt = P.mQ.lt;
                    kind = 2;
                } else if (op == kDown) {
                    w = L.experts + (size_t)M.top_id[slot < P.k ? slot : 0] * L.estride + L.down_off;
                    dst = M.part[slot < P.k ? slot : 0] - R0;
                    t = 0;
                    q6 = L.down_q6;
                    bpr = P.mE.bpr;
                    lv = P.mE.lv;
                    lt = P.mE.lt;
                    kind = q6 ? 4 : 3;
                    xcol = slot * bpr;
                }
                if (q6)
                    parity = matvec<Q6, 2>(w, bpr, lv, lt, own.x, own.y, dst, t, keep, xcol, P.stages[kind], parity);
                else
                    parity = matvec<Q4, 4>(w, bpr, lv, lt, own.x, own.y, dst, t, keep, xcol, P.stages[kind], parity);
                pend = 0;
            }
            // ---- attention of this CTA's positions ----
            if (op == kQKV) {
                const int base = M.tile0, tile1 = M.tile1, tile0 = base + warp;
                if (base < tile1) {
                    const int kvh = M.kvh, qb = M.qb;
                    if (tile0 < tile1) {
                        load_kv(L.kv_k, L.kv_v, tile0, M.pos, P.n_kv, kvh);
                        pend = 1;
                    }
                    cta_sync();  // the staged vector has been read
                    const int nh = min(16, P.gqa - qb * 16);
                    q_fragments(P.c_q + (kvh * P.gqa + qb * 16) * 128, tag, nh, L.q_norm != nullptr, P.eps, P.scale * kLog2e);
                    if (cta_aborted()) break;
                    if (tile0 < tile1)
                        parity = attn_tiles(tile0, tile1, M.pos, P.n_kv, kvh, L.kv_k, L.kv_v, qb == 0, P.c_k, P.c_v, tag,
                                            L.k_norm != nullptr, P.eps, parity);
                    pend = 0;
                    cta_sync();
                    attn_partial(min(kWarps, tile1 - base), nh, P.c_part, P.c_ml, M.part_slot, tag);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the ring was written and read as plain memory
                }
            }
            cta_sync();  // the staged vector and the ring have been read
            if (op == kQKV && cta < P.n_heads) {
                merge_head(M.merge_block, M.merge_head, M.nc, P.chunks, P.c_part, P.c_ml, P.c_attn + cta * 128, tag);
            }
        }
        // ---- the next operation's weights; gate / up requests its own: they depend on the routing ----
        const int next = (op + 1) & 3, ln = l + (op == kDown ? 1 : 0);
        if (ln < P.n_layers && next != kExperts) {
            const Layer &L = params.L[ln];
            const int2 own = M.own[warp][next];
            const int qm = M.own_qm[warp];
            const uint8_t *w = qm == 0 ? L.wq : qm == 1 ? L.wk : L.wv;
            bool q6 = qm == 2 && L.v_q6;
            int bpr = P.mH.bpr, lv = P.mH.lv, kind = q6 ? 1 : 0;
            if (next == kO) {
                w = L.wo;
                q6 = false;
                bpr = P.mQ.bpr;
                lv = P.mQ.lv;
                kind = 2;
            } else if (next == kDown) {
                w = L.experts + (size_t)M.top_id[M.own_slot[warp] < P.k ? M.own_slot[warp] : 0] * L.estride + L.down_off;
                q6 = L.down_q6;
                bpr = P.mE.bpr;
                lv = P.mE.lv;
                kind = q6 ? 4 : 3;
            }
            pend = prefetch(w, own.x, own.y, bpr * (q6 ? kQ6KBlock : kQ4KBlock), (q6 ? 4 : 5) - lv, P.stages[kind]);
        }
        if (l < 0) {
            if (P.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
            if (tid == 0) {
                // arrivals of the launches before this one (nobody of this launch arrives before every CTA has read it: the last
                // layer needs the activations of all of them); the quotient by a multiplication, a 64-bit division is a hundred
                // instructions
                unsigned long long c;
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(P.ctr) : "memory");
                unsigned long long n = static_cast<unsigned long long>(__ull2double_rz(c) * P.inv_grid);
                const long long r = static_cast<long long>(c - n * grid);
                if (r < 0) n--;
                if (r >= grid) n++;
                M.tag = static_cast<uint32_t>(n) * 128u + 1u;
                const int pos = __ldcg(P.pos);
                M.pos = pos;
                const int tpc = ((pos >> 4) + P.chunks) / P.chunks, ab = cta / P.chunks, ac = cta - ab * P.chunks;  // tiles per chunk; ours
                M.nc = ((pos >> 4) + tpc) / tpc;
                M.kvh = ab / P.qblocks;
                M.qb = ab - M.kvh * P.qblocks;
                M.part_slot = cta;
                M.tile0 = ac * tpc;
                M.tile1 = ab < P.n_kv * P.qblocks ? min((ac + 1) * tpc, (pos >> 4) + 1) : 0;
                const int kv = cta / P.gqa, hq = cta - kv * P.gqa;
                M.merge_block = kv * P.qblocks + (hq >> 4);
                M.merge_head = hq & 15;
            }
            const int R0 = M.R0, rows = M.rows;
            if (tid < rows) M.hid[tid] = __ldcg(P.hidden + R0 + tid);
            if (tid < 128) M.rope[tid] = __ldcg(tid < 64 ? P.cos_t + tid : P.sin_t + tid - 64);
            __syncthreads();
        } else if (op == kDown) {
            const int R0 = M.R0, rows = M.rows;
            if (tid < rows) {
                float y = 0.0f;
#pragma unroll 4
                for (int i = 0; i < P.k; i++) y = fmaf(M.swt[i], M.part[M.order[i]][tid], y);  // in the order of the slots
                y += M.hid[tid];
                M.hid[tid] = y;
                if (ln < P.n_layers)
                    st_cell(P.c_h0 + R0 + tid, y, tag);
                else
                    P.hidden[R0 + tid] = y;
            }
            if (ln == P.n_layers) break;
        }
        op = next;
        l = ln;
    }
    if (P.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (cta_aborted()) {  // leave after the copies in flight
        const int tid = thread_id();
        if (tid == 0) atomicExch(P.err, MB200_ERR_TIMEOUT);
#pragma unroll 1
        for (int s = 0; s < kStages; s++)
            if (pend >> s & 1) mbar_wait(&M.bars[tid >> 5][s], (parity >> s) & 1);
        if (tid == 0 && M.row_pend >= 0) mbar_wait(&M.row_bar, M.row_pend);
    }
    __syncthreads();
    if (thread_id() == 0) asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(P.ctr) : "memory");
}

Split split(int w0, int nw, int passes) { return Split{w0, nw, passes / nw, passes % nw}; }
// 2^lt: the streaming matvec's column groups (stream::prepare): the largest power of two that divides the blocks of a row, and
// eight (the last group ragged) where that makes more groups than it has warps.
Map map_of(int cols)
{
    Map m{cols / 256, 0, 0};
    while (m.lt < 3 && !(m.bpr >> m.lt & 1)) m.lt++;
    if (m.bpr >> m.lt > stream::kConsumers) m.lt = 3;
    m.lv = m.lt < 2 && m.bpr >= 8 ? 3 : m.lt;  // a ragged last pass costs less than single blocks side by side
    if (m.lt == 3 && m.bpr % 16 == 0) m.lt = 2;  // paired: half of a group is added in the lanes
    return m;
}
int stage_rows(const Map &m, bool q6) { return (q6 ? 2 : 4) << (3 - m.lv); }
int stage_of(const Map &m, bool q6) { return stage_bytes_of(stage_rows(m, q6) * m.bpr * (q6 ? kQ6KBlock : kQ4KBlock)); }
constexpr int kSmemBytes = 227 * 1024;

}  // namespace

size_t scratch(Params &P, uint8_t *base)
{
    size_t o = 256;
    if (base) P.ctr = reinterpret_cast<unsigned long long *>(base);
    auto take = [&](uint2 *&p, size_t n) {
        if (base) p = reinterpret_cast<uint2 *>(base + o);
        o += (n * sizeof(uint2) + 255) & ~static_cast<size_t>(255);
    };
    const size_t grid = device_sms();
    take(P.c_q, P.QD);
    take(P.c_k, P.KD);
    take(P.c_v, P.KD);
    take(P.c_part, grid * 16 * 128);
    take(P.c_ml, grid * 16 * 2);
    take(P.c_attn, P.QD);
    take(P.c_h1, P.H);
    take(P.c_act, (size_t)P.k * P.EFF);
    take(P.c_h0, P.H);
    take(P.c_logit, P.n_experts);
    return o;
}

bool plan(Params &P)
{
    const int grid = device_sms();
    if (P.H % 256 || P.EFF % 256 || P.QD % 256 || P.H < 256 || P.EFF < 256 || P.QD < 256 || P.H > 16 * kWork) return false;
    if (P.k < 1 || P.k > kMaxK || P.n_experts < P.k || P.n_experts > min(grid, kMaxExperts) || P.n_experts > 32 * P.k) return false;
    if (P.n_layers < 1 || P.n_layers > kMaxLayers) return false;
    P.qblocks = (P.gqa + 15) / 16;
    const int blocks = P.n_kv * P.qblocks;
    if (blocks > grid || P.n_heads > grid) return false;
    P.chunks = grid / blocks;
    P.mH = map_of(P.H);
    P.mQ = map_of(P.QD);
    P.mE = map_of(P.EFF);
    const int warps = kWarps * grid, rpp = 8 >> P.mH.lv;
    // the O projection and the down projection must have rows for every CTA: what tells a writer that all have read
    if (P.H < grid || P.H / grid + 1 > kMaxDownRows) return false;
    // Q, K, V: warps by what the rows cost (Q6_K: 1.46 times the bytes and more arithmetic per byte)
    const double cq = P.QD, ck = P.KD, cv = P.KD * (P.L[0].v_q6 ? 1.8 : 1.0), sum = cq + ck + cv;
    int wk = static_cast<int>(warps * ck / sum), wv = static_cast<int>(warps * cv / sum);
    wk = wk < 1 ? 1 : wk;
    wv = wv < 1 ? 1 : wv;
    P.sq = split(0, warps - wk - wv, P.QD / rpp);
    P.sk = split(warps - wk - wv, wk, P.KD / rpp);
    P.sv = split(warps - wv, wv, P.KD / rpp);
    P.ipe = P.EFF / rpp;
    P.ipe_magic = static_cast<uint32_t>((1ull << 32) / P.ipe) + 1;
    P.sg = split(0, warps, P.k * P.ipe);
    P.xc = P.H > P.QD ? P.H : P.QD;
    if (P.k * P.EFF > P.xc) P.xc = P.k * P.EFF;
    if (P.xc < 4096) P.xc = 4096;  // the attention's fragments and the merge use the same 8 KB
    auto up = [](int v) { return (v + 127) & ~127; };
    P.off_row = up(kX + 2 * P.xc + P.xc / 8 + P.xc / 4);
    P.off_ring = up(P.off_row + P.H * 4);
    for (int l = 0; l < P.n_layers; l++) P.L[l].fold = moe_fused_covers(P.H, P.EFF, P.k, P.L[l].down_q6 != 0);
    P.ring_bytes = ((kSmemBytes - P.off_ring) / kWarps) & ~127;
    bool v6 = false, d4 = false, d6 = false;
    for (int l = 0; l < P.n_layers; l++) {
        v6 = v6 || P.L[l].v_q6;
        d6 = d6 || P.L[l].down_q6;
        d4 = d4 || !P.L[l].down_q6;
    }
    const int bytes[6] = {stage_of(P.mH, false), stage_of(P.mH, true), stage_of(P.mQ, false), stage_of(P.mE, false), stage_of(P.mE, true),
                          4 * rpp * P.mH.bpr * kQ4KBlock};
    const bool used[6] = {true, v6, true, d4, d6, true};
    for (int i = 0; i < 6; i++) {
        P.stages[i] = P.ring_bytes / bytes[i] < kStages ? P.ring_bytes / bytes[i] : kStages;
        if (used[i] && P.stages[i] < 1) return false;
    }
    return kVOff + 16 * kVPitch <= P.ring_bytes && 16 * kPitch * 4 <= P.ring_bytes && P.chunks <= kMaxChunks && P.chunks * 512 <= kWarps * P.ring_bytes;
}

int launch(Params &P, cudaStream_t stream)
{
    static bool done[kMaxDevices] = {false};
    static int pdl_ok = 1;  // cleared if the driver refuses cooperative + programmatic serialization together
    const int dev = current_device(), grid = device_sms();
    if (!done[dev]) {
        if (cudaFuncSetAttribute(persist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) {
            cudaGetLastError();
            return MB200_ERR_LAUNCH;
        }
        done[dev] = true;
    }
    P.inv_grid = 1.0 / grid;
    P.err = device_error_word();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kWork);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;  // the CTAs wait for one another: all must be resident
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    P.pdl = (pdl_enabled() && pdl_ok) ? 1 : 0;
    cfg.numAttrs = P.pdl ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, persist_kernel, P);
    if (e != cudaSuccess && P.pdl) {
        cudaGetLastError();
        pdl_ok = 0;
        P.pdl = 0;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, persist_kernel, P);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return MB200_ERR_LAUNCH;
    }
    return MB200_OK;
}

}  // namespace persist
}  // namespace mb200
