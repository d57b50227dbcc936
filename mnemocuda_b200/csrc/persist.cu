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
// The top-k a CTA does for itself by counting: the rank of an expert is how many logits are larger. Only where equal logits
// straddle the boundary does the reference's replace-the-minimum walk decide, and is then run.
//
// The code of a layer is run once per layer: what counts is its size (270 KB with a copy of every step per operation, 106 KB as
// one loop over the operations) and that nothing lives in local memory, which the weight stream and 227 KB of shared memory
// leave no L1 for. Hence eight warps with 255 registers (sixteen with 128 spilled 2 KB a thread: 2870 us instead of 1930 per token
// below), several rows per warp in flight instead, thread_id() and cta_id() read anew by every step, and the launch's
// parameters, divisions already done, in shared memory.
//
// Measured, per token: 30B shape at position 4095 (48 layers) 3240 -> 1643 us, 8 layers of the 235B shape at 8191 925 -> 629; a
// layer is 33 / 65 us. What bounds it: seven exchanges between all SMs (a value written is with its readers 1 us later, and they
// wait for the slowest CTA: 20 of the 33 us), then instruction issue of the products (Q6_K down: 9 us at the 235B shape,
// where gate / up runs at the copy rate). Tried and slower: two K / V tiles in flight per warp, the selection by repeated warp
// maxima (150 cycles a round), the next round of a wide vector requested ahead (all three: registers), units of two rows.
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

namespace persist {
namespace {

constexpr int kWarps = 8, kWork = kWarps * 32;
constexpr int kStages = 5;         // ring stages per warp at most
constexpr int kPitch = 132;        // floats between heads of a warp's attention result
constexpr int kKvPitch = 272;      // bytes between K / V rows in shared memory
constexpr int kMaxDownRows = 64;   // rows of the hidden vector per CTA
constexpr int kMaxK = kWarps;    // a warp per slot, or several
constexpr int kMaxExperts = 256;   // two threads per expert
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
    uint64_t row_bar;
    unsigned long long launch;
    float red[2][kWarps];
    float am[kWarps][16], al[kWarps][16];  // attention: running maximum / sum per warp and head
    float hid[kMaxDownRows];               // the CTA's rows of the hidden vector: it writes them in both of a layer's halves
    float part[kMaxK][kMaxDownRows];
    alignas(16) uint32_t key[kMaxExperts]; // ordered logits
    int top_id[kMaxK + 1];
    uint32_t top_key[kMaxK + 1];
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
    float sum = (v[0] + v[1]) + (v[2] + v[3]);
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));  // 8 lanes = 32 columns
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const float sc = amax * (1.0f / 127.0f);
    const float inv = amax > 0.0f ? __fdividef(127.0f, amax) : 0.0f, inv2 = inv * 254.0f;
    // adding 1.5 * 2^23 rounds to the nearest integer and leaves it in the low bits: no conversions, which run at an eighth of
    // the FMA rate
    constexpr float kRound = 12582912.0f;
    uint32_t a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float ai = fmaf(v[i], inv, kRound);
        a[i] = __float_as_uint(ai);
        b[i] = __float_as_uint(fmaf(fmaf(-(ai - kRound), sc, v[i]), inv2, kRound));  // |remainder| <= sc / 2: at most 127
    }
    const uint32_t p1 = __byte_perm(__byte_perm(a[0], a[1], 0x0040), __byte_perm(a[2], a[3], 0x0040), 0x5410);
    const uint32_t p2 = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
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

// Stages K columns (every thread of the CTA calls it; K a multiple of 256): src holds floats, or cells if tag != 0. norm_w:
// RMS-normalised with it. logit_cell: the row of shared memory at off_row times the (normalised) vector goes there with
// the tag, before the splitting starts. With either of them K <= 16 kWork: the whole vector in registers. Returns whether the CTA
// has given up.
__device__ __forceinline__ bool stage_vec(const void *src, uint32_t tag, int K, const float *norm_w, float eps, uint2 *logit_cell)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
    const bool whole = norm_w || logit_cell;
    const int xc = head().xc;
#pragma unroll 1
    for (int base = tid * 4; base < K || whole; base += kWork * 16) {
        float4 v[4], g[4];
        if (norm_w) {
#pragma unroll
            for (int u = 0; u < 4; u++)
                g[u] = base + u * kWork * 4 < K ? __ldg(reinterpret_cast<const float4 *>(norm_w + base + u * kWork * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (tag) {
            uint32_t todo = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                todo |= (base + u * kWork * 4 < K ? 1u : 0u) << u;
            }
#pragma unroll 1
            for (uint32_t i = 0; todo; i++) {  // what has not come is asked for again
                uint4 a[4], b[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    a[u] = b[u] = make_uint4(0, 0, 0, 0);
                    if (todo >> u & 1) {
                        const uint2 *p = static_cast<const uint2 *>(src) + base + u * kWork * 4;
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
                v[u] = base + u * kWork * 4 < K ? __ldcg(reinterpret_cast<const float4 *>(static_cast<const float *>(src) + base + u * kWork * 4))
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (whole) {
            float ss = 0.0f, dot = 0.0f;
            if (norm_w) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    ss = fmaf(v[u].x, v[u].x, fmaf(v[u].y, v[u].y, fmaf(v[u].z, v[u].z, fmaf(v[u].w, v[u].w, ss))));
                    v[u].x *= g[u].x; v[u].y *= g[u].y; v[u].z *= g[u].z; v[u].w *= g[u].w;
                }
            }
            if (logit_cell) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (base + u * kWork * 4 < K) {
                        const float4 r = *reinterpret_cast<const float4 *>(smem + head().off_row + (base + u * kWork * 4) * 4);
                        dot = fmaf(v[u].x, r.x, fmaf(v[u].y, r.y, fmaf(v[u].z, r.z, fmaf(v[u].w, r.w, dot))));
                    }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ss += __shfl_xor_sync(0xffffffffu, ss, o);
                dot += __shfl_xor_sync(0xffffffffu, dot, o);
            }
            if (lane == 0) {
                M.red[0][warp] = ss;
                M.red[1][warp] = dot;
            }
            cta_sync();
            float t = 0.0f;
#pragma unroll
            for (int w = 0; w < kWarps; w++) t += M.red[0][w];  // fixed order: the same scale on every thread and CTA
            const float scale = norm_w ? 1.0f / sqrtf(t / static_cast<float>(K) + eps) : 1.0f;
            if (logit_cell && tid == 0) {
                float d = 0.0f;
#pragma unroll
                for (int w = 0; w < kWarps; w++) d += M.red[1][w];
                st_cell(logit_cell, d * scale, tag);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) { v[u].x *= scale; v[u].y *= scale; v[u].z *= scale; v[u].w *= scale; }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int c0 = base + u * kWork * 4;
            if (c0 - lane * 4 >= K) break;  // warp-uniform: a warp covers 128 columns
            stage_quad(xc, v[u], c0, lane);
        }
        if (whole) break;
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
__device__ __forceinline__ uint32_t matvec(const uint8_t *w, int bpr, int lv, int r0, int n, void *dst, uint32_t tag, float *keep, int xcol,
                                        int stages, uint32_t parity)
{
    uint8_t *buf = ring();
    uint64_t *bars = ring_bars();
    const int xc = head().xc;
    const int lane = thread_id() & 31, q = lane >> 2, sub = lane & 3;
    const int v = 1 << lv, rpp = 8 >> lv, cq = q & (v - 1), rq = q >> lv, W = 4 << lv;
    const int groups = (bpr + v - 1) >> lv, ur = RU * rpp;
    const uint32_t row_bytes = bpr * F::kBlockBytes, sb = stage_bytes_of(ur * row_bytes);
    typename F::XRegs xr;
    int s = 0;
#pragma unroll 1
    for (int r = 0; r < n; r += ur) {
        ring_wait(bars, s, parity);
        uint32_t skew = 0;
        if (F::kBlockBytes % 16) skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(w) + (size_t)(r0 + r) * row_bytes) & 15u;
        const uint8_t *base = buf + s * sb + skew + rq * row_bytes;
        float acc[RU];
#pragma unroll
        for (int i = 0; i < RU; i++) acc[i] = 0.0f;
#pragma unroll 1
        for (int c = 0; c < groups; c++) {
            const int col = (c << lv) + cq;
            const bool in = col < bpr;  // a ragged last group
            const int at = in ? col : 0;
            if (groups > 1 || r == 0) load_x(xr, xc, xcol + at, sub);
#pragma unroll
            for (int i = 0; i < RU; i++) {
                if (i > 0 && r + i * rpp >= n) break;
                const float d = F::block_dot(base + (i * rpp) * row_bytes + at * F::kBlockBytes, sub, xr);
                acc[i] += in ? d : 0.0f;
            }
        }
        __syncwarp();
        const int nr = r + stages * ur;
        if (lane == 0 && nr < n) issue_unit(w, r0 + nr, min(ur, n - nr), row_bytes, buf + s * sb, &bars[s]);
        int which;
        const float sum = stream::packed_sum<RU, false>(acc, W, lane, which);
        const int row = r + which * rpp + rq;
        if ((lane & (W / RU - 1)) == 0 && row < n) {
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
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4])
{
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
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
    const float ss = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
    if (normed) {
        const float f = 1.0f / sqrtf(ss * (1.0f / 128.0f) + eps);
        v.x *= f * w[lane];
        v.y *= f * w[lane + 32];
        v.z *= f * w[lane + 64];
        v.w *= f * w[lane + 96];
    }
    const float c0 = M.rope[lane], c1 = M.rope[lane + 32], s0 = M.rope[64 + lane], s1 = M.rope[96 + lane];
    return make_float4(v.x * c0 - v.z * s0, v.y * c1 - v.w * s1, v.x * s0 + v.z * c0, v.y * s1 + v.w * c1);
}

// K / V rows of a tile of 16 positions, a row per lane
__device__ __forceinline__ void load_kv(const __half *kv_k, const __half *kv_v, int tile, int pos, int n_kv, int kvh)
{
    const int lane = thread_id() & 31;
    uint8_t *buf = ring();
    uint64_t *bar = ring_bars();
    if (lane == 0) mbar_expect_tx(bar, 32 * 256);
    __syncwarp();
    const int p = min(tile * 16 + (lane & 15), pos);
    bulk_g2s(buf + lane * kKvPitch, (lane < 16 ? kv_k : kv_v) + ((size_t)p * n_kv + kvh) * 128, 256, bar);
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
    const uint32_t kbase = smem_u32(buf), vbase = kbase + 16 * kKvPitch;
    const uint32_t ka = kbase + (lane & 7) * kKvPitch + (lane >> 3) * 16;
    const uint32_t va = vbase + ((lane & 7) + ((lane >> 3) & 1) * 8) * kKvPitch + (lane >> 4) * 16;
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
            uint8_t *kd = buf + (pos & 15) * kKvPitch;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int d = lane + 32 * i;
                const __half hk = __float2half_rn(kn[i]), hv = __float2half_rn(vv[i]);
                *reinterpret_cast<__half *>(kd + 2 * d) = hk;
                *reinterpret_cast<__half *>(kd + 16 * kKvPitch + 2 * d) = hv;
                if (store) {
                    kv_k[row + d] = hk;
                    kv_v[row + d] = hv;
                }
            }
            __syncwarp();
        }
        float S[2][4], T[2][4];  // hi and lo halves of Q: independent chains
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) S[n][e] = T[n][e] = 0.0f;
#pragma unroll 1
        for (int jj = 0; jj < 4; jj++) {
            const uint8_t *f = smem + kX + (2 * jj * 32 + lane) * 16;
            const uint4 h0 = *reinterpret_cast<const uint4 *>(f), h1 = *reinterpret_cast<const uint4 *>(f + 512);
            const uint4 lo0 = *reinterpret_cast<const uint4 *>(f + 4096), lo1 = *reinterpret_cast<const uint4 *>(f + 4096 + 512);
#pragma unroll
            for (int n = 0; n < 2; n++) {
                uint32_t b[4];
                ldmatrix4<false>(ka + n * 8 * kKvPitch + jj * 64, b);
                mma16816(S[n], h0, b[0], b[1]);
                mma16816(T[n], lo0, b[0], b[1]);
                mma16816(S[n], h1, b[2], b[3]);
                mma16816(T[n], lo1, b[2], b[3]);
            }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const bool in = tile * 16 + n * 8 + 2 * t + e <= pos;
                S[n][e] = in ? S[n][e] + T[n][e] : -INFINITY;
                S[n][2 + e] = in ? S[n][2 + e] + T[n][2 + e] : -INFINITY;
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
            ldmatrix4<true>(va + u * 16, b);
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
            const int d = lane + 32 * i, kk = d & 15;
            const int at = ((d >> 4) * 32 + (h & 7) * 4 + ((kk & 7) >> 1)) * 16 + ((h >> 3) + 2 * (kk >> 3)) * 4 + (kk & 1) * 2;
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

// Merges the nc chunks' partials of one head (hq of head block b): the CTA's warps over the chunks; cells of the result.
__device__ __forceinline__ void merge_head(int b, int hq, int nc, int chunks, const uint2 *c_part, const uint2 *c_ml, uint2 *dst, uint32_t tag)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
    float m = -INFINITY, s = 0.0f;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int c0 = warp; c0 < nc; c0 += 5 * kWarps) {
        uint4 ms[5], o0[5], o1[5];
#pragma unroll 1
        for (uint32_t i = 0;; i++) {
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 5; u++) {
                const size_t slot = ((size_t)b * chunks + min(c0 + u * kWarps, nc - 1)) * 16 + hq;
                ms[u] = ld_cells2(c_ml + slot * 2);
                o0[u] = ld_cells2(c_part + slot * 128 + 4 * lane);
                o1[u] = ld_cells2(c_part + slot * 128 + 4 * lane + 2);
                ok = ok && ms[u].y == tag && ms[u].w == tag && o0[u].y == tag && o0[u].w == tag && o1[u].y == tag && o1[u].w == tag;
            }
            if (ok || *gave_up()) break;
            if (i == kPolls) *gave_up() = 1;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 5; u++) {
            if (c0 + u * kWarps >= nc) break;
            const float mu = __uint_as_float(ms[u].x), mn = fmaxf(m, mu), fo = exp2f(m - mn), fn = exp2f(mu - mn);
            s = s * fo + __uint_as_float(ms[u].z) * fn;
            a.x = a.x * fo + __uint_as_float(o0[u].x) * fn;
            a.y = a.y * fo + __uint_as_float(o0[u].z) * fn;
            a.z = a.z * fo + __uint_as_float(o1[u].x) * fn;
            a.w = a.w * fo + __uint_as_float(o1[u].z) * fn;
            m = mn;
        }
    }
    float *buf = reinterpret_cast<float *>(smem + kX);  // [kWarps][128]
    *reinterpret_cast<float4 *>(buf + warp * 128 + 4 * lane) = a;
    if (lane == 0) {
        M.red[0][warp] = m;
        M.red[1][warp] = s;
    }
    cta_sync();
    if (tid < 128) {
        float mt = -INFINITY, st = 0.0f, o = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) mt = fmaxf(mt, M.red[0][w]);
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const float f = exp2f(M.red[0][w] - mt);  // 0 for a warp without a chunk
            st = fmaf(M.red[1][w], f, st);
            o = fmaf(buf[w * 128 + tid], f, o);
        }
        st_cell(dst + tid, o / st, tag);
    }
    cta_sync();
}

// ---- selection ----
__device__ __forceinline__ uint32_t ordered(float v)
{
    const uint32_t b = __float_as_uint(v + 0.0f);  // -0 counts as 0
    return min(b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u), 0xFFFFFFFEu);
}
__device__ __forceinline__ float unordered(uint32_t k) { return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xFFFFFFFFu)); }

// One thread: the reference's walk (n <= 32 k: nothing is dropped before the merge) over the logits in (e % 32, e / 32) order,
// replacing the first minimum when strictly greater.
__device__ __noinline__ void walk(int n, int k)
{
    Misc &M = misc();
#pragma unroll 1
    for (int i = 0; i < k; i++) {
        M.top_id[i] = 0;
        M.top_key[i] = 0;
    }
#pragma unroll 1
    for (int l = 0; l < 32; l++)
#pragma unroll 1
        for (int e = l; e < n; e += 32) {
            int at = 0;
#pragma unroll 1
            for (int i = 1; i < k; i++)
                if (M.top_key[i] < M.top_key[at]) at = i;
            if (M.key[e] > M.top_key[at]) {
                M.top_key[at] = M.key[e];
                M.top_id[at] = e;
            }
        }
}

// The k largest of n logits (every thread of the CTA calls it): lane i < k of every warp returns the i-th expert, M.top_key
// keeps their logits. -1: the CTA has given up.
__device__ __forceinline__ int select_experts(const uint2 *cells, uint32_t tag, int n, int k)
{
    Misc &M = misc();
    const int tid = thread_id(), lane = tid & 31;
    static_assert(kWork >= kMaxExperts, "a thread per logit");
    if (tid < kMaxExperts) M.key[tid] = tid < n ? ordered(wait_value(cells + tid, tag)) : 0;
    if (cta_aborted()) return -1;
    {
        const int half = ((n + 7) >> 3) * 4, lo = (tid & 1) ? half : 0, hi = lo + half;  // keys beyond n are 0
#pragma unroll 1
        for (int e = tid >> 1; e - (lane >> 1) < n; e += kWork / 2) {  // warp-uniform; two threads per expert
            const uint32_t me = M.key[e];
            int rank = 0;
#pragma unroll 4
            for (int i = lo; i < hi; i += 4) {  // an equal one before it counts as larger (a key is never the largest integer)
                const uint4 o = *reinterpret_cast<const uint4 *>(&M.key[i]);
                rank += (o.x + (i < e) > me) + (o.y + (i + 1 < e) > me) + (o.z + (i + 2 < e) > me) + (o.w + (i + 3 < e) > me);
            }
            rank += __shfl_xor_sync(0xffffffffu, rank, 1);
            if (rank <= k && e < n && !(tid & 1)) {
                M.top_id[rank] = e;
                M.top_key[rank] = me;
            }
        }
    }
    cta_sync();
    if (n > k && M.top_key[k - 1] == M.top_key[k]) {  // the same for the whole CTA
        cta_sync();
        if (tid == 0) walk(n, k);
        cta_sync();
    }
    return M.top_id[lane < k ? lane : 0];
}
// One warp, later (the requests for the experts do not need them): the weights of the selected, to M.swt.
__device__ __forceinline__ void select_weights(int k)
{
    Misc &M = misc();
    const int lane = thread_id() & 31;
    const float v = lane < k ? unordered(M.top_key[lane]) : -INFINITY;
    float mx = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = lane < k ? expf(v - mx) : 0.0f;
    const float sum = warp_sum(e);
    if (lane < k) M.swt[lane] = e / sum;
}

// ---- gate / up: items [i0, i0 + n), item i = a pass of gate rows and the same up rows of the i / ipe-th routed expert. Two items
// a stage: their four products hide one another's latency, and one reduction serves them (a warp has 3 to 11 items). ----
// Every lane calls it: lane 2 j + h requests half h (gate, up) of item i + j of the stage, j < 2.
__device__ __forceinline__ void issue_items(const uint8_t *experts, size_t estride, uint32_t up_off, int id, int i, int end, int ipe, uint32_t magic,
                                            uint32_t half, bool mine, int j, int h, uint8_t *dst, uint64_t *bar)
{
    const int item = i + j, slot = __umulhi(item, magic);
    const int ex = __shfl_sync(0xffffffffu, id, slot & 31);
    const bool in = mine && item < end;
    if (in && j == 0 && h == 0) mbar_expect_tx(bar, (i + 1 < end ? 4 : 2) * half);
    __syncwarp();
    if (in) bulk_g2s(dst + (2 * j + h) * half, experts + (size_t)ex * estride + (item - slot * ipe) * half + (h ? up_off : 0), half, bar);
}
// id: lane i holds the i-th routed expert. Writes SwiGLU's result as cells act[slot * EFF + row].
__device__ __forceinline__ uint32_t gate_up(const uint8_t *experts, size_t estride, uint32_t up_off, int id, int i0, int n, int ipe, uint32_t magic,
                                            int bpr, int lv, int EFF, uint2 *act, uint32_t tag, int stages, uint32_t parity)
{
    uint8_t *buf = ring();
    uint64_t *bars = ring_bars();
    const int xc = head().xc;
    const int lane = thread_id() & 31, q = lane >> 2, sub = lane & 3;
    const int v = 1 << lv, rpp = 8 >> lv, cq = q & (v - 1), rq = q >> lv, W = 4 << lv;
    const int groups = (bpr + v - 1) >> lv, end = i0 + n;
    const uint32_t row_bytes = bpr * kQ4KBlock, half = rpp * row_bytes, sb = 4 * half;
    const int ij = (lane >> 1) & 1, ih = lane & 1, is = lane >> 2;  // of a request: item, half, stage
    issue_items(experts, estride, up_off, id, i0 + 2 * is, end, ipe, magic, half, is < stages, ij, ih, buf + is * sb, &bars[is < stages ? is : 0]);
    Q4::XRegs xr;
    int s = 0;
#pragma unroll 1
    for (int i = i0; i < end; i += 2) {
        ring_wait(bars, s, parity);
        const uint8_t *base = buf + s * sb + rq * row_bytes;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // gate, up of the two items
#pragma unroll 1
        for (int c = 0; c < groups; c++) {
            const int col = (c << lv) + cq;
            const bool in = col < bpr;  // a ragged last group
            const int at = in ? col : 0;
            if (groups > 1 || i == i0) load_x(xr, xc, at, sub);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (u == 2 && i + 1 >= end) break;
                const float d = Q4::block_dot(base + u * half + at * kQ4KBlock, sub, xr);
                acc[u] += in ? d : 0.0f;
            }
        }
        __syncwarp();
        issue_items(experts, estride, up_off, id, i + 2 * stages, end, ipe, magic, half, lane < 4, ij, ih, buf + s * sb, &bars[s]);
        int which;
        const float g = stream::packed_sum<4, false>(acc, W, lane, which);
        const float u = __shfl_xor_sync(0xffffffffu, g, W >> 2);  // which ^ 1: a quarter of the row's lanes away
        const int item = i + (which >> 1);
        if ((lane & (W / 4 - 1)) == 0 && !(which & 1) && item < end) {
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
        M.abort_flag = 0;
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
    const bool has_row = cta < P.n_experts;
    auto request_row = [&](int l) {
        mbar_expect_tx(&M.row_bar, P.H * 4);
        bulk_g2s(smem + P.off_row, params.L[l].router + (size_t)cta_id() * P.H, P.H * 4, &M.row_bar);
    };
    int row_pend = has_row ? 0 : -1;  // parity of the router row on its way
    if (has_row && tid == 0) request_row(0);

    uint32_t parity = 0, pend = 0, tag = 0;  // pend: stages in flight while the CTA may still give up
    int pos = 0, id = 0;                     // id: lane i holds the i-th routed expert
    bool ok = true;
    // One pass of the loop: an operation (there is one copy of every step's code), preceded by the request for its weights. The
    // pass before the first only requests.
#pragma unroll 1
    for (int it = -1, l = 0, op = kDown;; it++) {
        const int tid = thread_id(), lane = tid & 31, warp = tid >> 5, cta = cta_id();
        if (it >= 0) {
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
                } else if (op == kExperts) {  // the router logit of this CTA's expert on the way
                    src = P.c_h1;
                    norm_w = L.ffn_norm;
                    K = P.H;
                    logit = has_row ? P.c_logit + cta : nullptr;
                    if (has_row) wait_copy(&M.row_bar, l & 1);
                    row_pend = -1;
                }
                // the norm weights of the heads: on their way while the vector is waited for
                const float *hw = tid < 128 ? L.q_norm : L.k_norm;
                float hn = 0.0f;
                if (op == kQKV && tid < 256 && hw) hn = __ldg(hw + (tid & 127));
                ok = !stage_vec(src, t, K, norm_w, P.eps, logit);
                if (!ok) break;
                if (op == kQKV && tid < 256) M.norm[tid >> 7][tid & 127] = hn;
            }
            // ---- its rows ----
            if (op == kExperts) {
                if (has_row && l + 1 < P.n_layers) {
                    row_pend = (l + 1) & 1;
                    if (tid == 0) request_row(l + 1);
                }
                id = select_experts(P.c_logit, tag, P.n_experts, P.k);
                ok = id >= 0;
                if (!ok) break;
                const int2 own = M.own[warp][kExperts];
                parity = gate_up(L.experts, L.estride, L.up_off, id, own.x, own.y, P.ipe, P.ipe_magic, P.mH.bpr, P.mH.lv, P.EFF, P.c_act, tag,
                                 P.stages[5], parity);
                if (warp == kWarps - 1) select_weights(P.k);
            } else {
                const int2 own = M.own[warp][op];
                const int qm = M.own_qm[warp], slot = M.own_slot[warp];
                const uint8_t *w = qm == 0 ? L.wq : qm == 1 ? L.wk : L.wv;
                void *dst = qm == 0 ? P.c_q : qm == 1 ? P.c_k : P.c_v;
                float *keep = nullptr;
                const int R0 = M.R0;
                uint32_t t = tag;
                bool q6 = qm == 2 && L.v_q6;
                int bpr = P.mH.bpr, lv = P.mH.lv, xcol = 0, kind = q6 ? 1 : 0;
                if (op == kO) {
                    w = L.wo;
                    dst = P.c_h1;
                    keep = M.hid - R0;
                    q6 = false;
                    bpr = P.mQ.bpr;
                    lv = P.mQ.lv;
                    kind = 2;
                } else if (op == kDown) {
                    w = L.experts + (size_t)__shfl_sync(0xffffffffu, id, slot & 31) * L.estride + L.down_off;
                    dst = M.part[slot < P.k ? slot : 0] - R0;
                    t = 0;
                    q6 = L.down_q6;
                    bpr = P.mE.bpr;
                    lv = P.mE.lv;
                    kind = q6 ? 4 : 3;
                    xcol = slot * bpr;
                }
                if (q6)
                    parity = matvec<Q6, 2>(w, bpr, lv, own.x, own.y, dst, t, keep, xcol, P.stages[kind], parity);
                else
                    parity = matvec<Q4, 4>(w, bpr, lv, own.x, own.y, dst, t, keep, xcol, P.stages[kind], parity);
                pend = 0;
            }
            // ---- attention of this CTA's positions ----
            if (op == kQKV) {
                const int base = M.tile0, tile1 = M.tile1, tile0 = base + warp;
                if (base < tile1) {
                    const int kvh = M.kvh, qb = M.qb;
                    if (tile0 < tile1) {
                        load_kv(L.kv_k, L.kv_v, tile0, pos, P.n_kv, kvh);
                        pend = 1;
                    }
                    cta_sync();  // the staged vector has been read
                    const int nh = min(16, P.gqa - qb * 16);
                    q_fragments(P.c_q + (kvh * P.gqa + qb * 16) * 128, tag, nh, L.q_norm != nullptr, P.eps, P.scale * kLog2e);
                    ok = !cta_aborted();
                    if (!ok) break;
                    if (tile0 < tile1)
                        parity = attn_tiles(tile0, tile1, pos, P.n_kv, kvh, L.kv_k, L.kv_v, qb == 0, P.c_k, P.c_v, tag,
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
        const int next = (op + 1) & 3, ln = l + (op == kDown && it >= 0 ? 1 : 0);
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
                w = L.experts + (size_t)__shfl_sync(0xffffffffu, id, M.own_slot[warp] & 31) * L.estride + L.down_off;
                q6 = L.down_q6;
                bpr = P.mE.bpr;
                lv = P.mE.lv;
                kind = q6 ? 4 : 3;
            }
            pend = prefetch(w, own.x, own.y, bpr * (q6 ? kQ6KBlock : kQ4KBlock), (q6 ? 4 : 5) - lv, P.stages[kind]);
        }
        if (it < 0) {
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
                M.launch = n;
            }
            __syncthreads();
            tag = static_cast<uint32_t>(M.launch) * 128u + 1u;
            pos = __ldcg(P.pos);
            if (tid == 0) {
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
        } else if (op == kDown) {
            const int R0 = M.R0, rows = M.rows;
            if (tid < rows) {
                float y = 0.0f;
#pragma unroll 4
                for (int i = 0; i < P.k; i++) y = fmaf(M.swt[i], M.part[i][tid], y);
                y += M.hid[tid];
                M.hid[tid] = y;
                if (ln < P.n_layers)
                    st_cell(P.c_h0 + R0 + tid, y, tag);
                else
                    P.hidden[R0 + tid] = y;
            }
            if (ln == P.n_layers) break;
            tag++;
        }
        op = next;
        l = ln;
    }
    if (P.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!ok) {  // given up: leave after the copies in flight
        if (tid == 0) atomicExch(P.err, MB200_ERR_TIMEOUT);
#pragma unroll 1
        for (int s = 0; s < kStages; s++)
            if (pend >> s & 1) mbar_wait(&M.bars[warp][s], (parity >> s) & 1);
        if (row_pend >= 0) mbar_wait(&M.row_bar, row_pend);
    }
    __syncthreads();
    if (tid == 0) asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(P.ctr) : "memory");
}

Split split(int w0, int nw, int passes) { return Split{w0, nw, passes / nw, passes % nw}; }
Map map_of(int cols)
{
    Map m{cols / 256, 0};
    while (m.lv < 3 && !(m.bpr >> m.lv & 1)) m.lv++;
    if (m.lv < 2 && m.bpr >= 8) m.lv = 3;  // a ragged last group costs less than single blocks side by side
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
    return 32 * kKvPitch <= P.ring_bytes && 16 * kPitch * 4 <= P.ring_bytes;
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
