// One launch for many layers of a decoded token: a persistent cooperative kernel, one CTA per SM (op order of
// src/forward.c:604-1117):
//   Q, K, V of RMSNorm(hidden) | q/k norm + RoPE + KV store + attention partials | merge of the partials | O + residual |
//   router logits of RMSNorm(hidden) | top-k, gate / up + SwiGLU of the routed experts | down, weighted sum + residual
// and, with the last three alone, the MoE block.
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
//   * weights depend on nobody: while a warp would wait it has the first ~11 KB of its next rows on the way (180 KB per SM,
//     which is all of most operations), and K / V rows of the cache before q exists;
//   * the input vector of an operation is split by every CTA into two int8 levels as it arrives.
//
// The top-k a CTA does for itself by counting: the rank of an expert is how many logits are larger. The MoE block returns ids,
// weights and activations in the reference's slots, which follow from its replace-the-minimum walk: slots_of() has the closed
// form (see topk.cuh), evaluated while the first weights are on their way. Equal logits where it matters take the walk itself.
//
// The code of a layer is run once per layer: what counts is that it stays in the instruction caches (with everything inlined it
// was 270 KB, and a layer took longer than the separate kernels). So every step is a function, one copy each, whose arguments
// are plain values -- a reference to the parameter block or to a struct would be read through memory, behind the weight
// stream -- and which finds its shared memory by offsets; loops over run-time counts are not unrolled.
//
// Every wait is bounded: a cell or a copy that does not come raises the abort flag of the CTA and the device error word, and
// the CTA leaves after its copies in flight.
#include "persist.cuh"

#include <cstdio>

#include "q4k_policy.cuh"
#include "q6k_policy.cuh"

namespace mb200 {
int pdl_enabled();

namespace persist {
namespace {

constexpr int kWarps = 16, kWork = kWarps * 32;
constexpr int kStages = 5;         // ring stages per warp at most
constexpr int kPitch = 132;        // floats between heads of a warp's attention result
constexpr int kKvPitch = 272;      // bytes between K / V rows in shared memory
constexpr int kMaxDownRows = 64;   // rows of the hidden vector per CTA
constexpr int kMaxK = 16;
constexpr int kMaxExperts = 256;   // two threads per expert
constexpr uint32_t kPolls = 1u << 19;  // a fraction of a second
constexpr float kLog2e = 1.4426950408889634f;

extern __shared__ __align__(1024) uint8_t smem[];

struct Misc {
    uint64_t bars[kWarps][kStages];
    uint64_t row_bar;
    unsigned long long launch;
    float red[2][kWarps];
    float am[kWarps][16], al[kWarps][16];  // attention: running maximum / sum per warp and head
    float part[kMaxK][kMaxDownRows];
    uint32_t key[kMaxExperts];             // ordered logits
    int arrival[kMaxExperts], byrank[kMaxExperts];
    int top_id[kMaxK + 1], slot_of_rank[kMaxK];
    uint32_t top_key[kMaxK + 1];
    int sid[kMaxK], slot[kMaxK];
    float swt[kMaxK];
    int accepted, tie, abort_flag;
};

__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWork) : "memory"); }
// Every thread: true = somebody in the CTA has given up (the same answer for all of them). A barrier of the CTA.
__device__ __forceinline__ bool cta_aborted(const volatile int *flag)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.or.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(*flag)), "n"(kWork)
        : "memory");
    return r != 0;
}

__device__ __noinline__ void wait_slow(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
#pragma unroll 1
    for (uint32_t i = 0; i < kWaitBudget; i++)
        if (*abort_flag || mbar_try_wait(bar, parity)) return;
    *abort_flag = 1;
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
__device__ __forceinline__ float wait_value(const uint2 *p, uint32_t tag, volatile int *abort_flag)
{
#pragma unroll 1
    for (uint32_t i = 0; i < kPolls; i++) {
        const uint2 c = ld_cell(p);
        if (c.y == tag) return __uint_as_float(c.x);
        if (*abort_flag) return 0.0f;
    }
    *abort_flag = 1;
    return 0.0f;
}
// Four cells, 32 apart (a head's values of a lane), all requested at once.
__device__ __forceinline__ void wait_values4(const uint2 *p, uint32_t tag, volatile int *abort_flag, float (&v)[4])
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
        if (ok || *abort_flag) return;
        if (i == kPolls) *abort_flag = 1;
    }
}

// ---- the staged input vector of xc columns: two arrays of int8 levels in 16-byte chunks of 16 columns, swizzled so that both
// block types read them without bank conflicts; the scale of every 32 columns and the sum of every 16 ----
__device__ __forceinline__ int chunk_at(int j)
{
    const int b = (j >> 3) & 3;
    return j ^ (b ^ (b << 1));
}
__device__ __forceinline__ float *x_scale(int xc) { return reinterpret_cast<float *>(smem + 2 * xc); }
__device__ __forceinline__ float *x_sum(int xc) { return reinterpret_cast<float *>(smem + 2 * xc + xc / 8); }
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
    *reinterpret_cast<uint32_t *>(smem + at) = p1;
    *reinterpret_cast<uint32_t *>(smem + xc + at) = p2;
    if ((lane & 7) == 0) x_scale(xc)[c0 >> 5] = sc;
    if ((lane & 3) == 0) x_sum(xc)[c0 >> 4] = sum;
}
__device__ __forceinline__ void load_x(Q4::XRegs &r, int xc, int col, int g)
{
    const int j = col * 16 + g * 4;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int at = chunk_at(j + i) * 16;
        const uint4 a = *reinterpret_cast<const uint4 *>(smem + at), b = *reinterpret_cast<const uint4 *>(smem + xc + at);
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
        const uint4 a = *reinterpret_cast<const uint4 *>(smem + at), b = *reinterpret_cast<const uint4 *>(smem + xc + at);
        r.q1[4 * g] = a.x; r.q1[4 * g + 1] = a.y; r.q1[4 * g + 2] = a.z; r.q1[4 * g + 3] = a.w;
        r.q2[4 * g] = b.x; r.q2[4 * g + 1] = b.y; r.q2[4 * g + 2] = b.z; r.q2[4 * g + 3] = b.w;
        r.k[g] = x_scale(xc)[j >> 1] * (1.0f / 254.0f);
        r.sx32[g] = 32.0f * x_sum(xc)[j];
    }
}

