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

// Stages K columns (every thread of the CTA calls it; K a multiple of 256): src holds floats, or cells if tag != 0. norm_w:
// RMS-normalised with it. logit_cell: the row of shared memory at off_row times the (normalised) vector goes there with
// logit_tag, before the splitting starts. With either of them K <= 8192: the whole vector in registers. Returns whether the CTA
// has given up.
__device__ __noinline__ bool stage_vec(const void *src, uint32_t tag, int K, const float *norm_w, float eps, int off_row,
                                       uint2 *logit_cell, uint32_t logit_tag, int xc, int off_misc)
{
    Misc &M = *reinterpret_cast<Misc *>(smem + off_misc);
    volatile int *abort_flag = &M.abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool whole = norm_w || logit_cell;
#pragma unroll 1
    for (int base = tid * 4; base < K || whole; base += kWork * 16) {
        float4 v[4], g[4];
        if (norm_w) {
#pragma unroll
            for (int u = 0; u < 4; u++)
                g[u] = base + u * kWork * 4 < K ? __ldg(reinterpret_cast<const float4 *>(norm_w + base + u * kWork * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (tag) {
#pragma unroll 1
            for (uint32_t i = 0;; i++) {
                bool ok = true;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    uint4 a = make_uint4(0, tag, 0, tag), b = a;
                    if (base + u * kWork * 4 < K) {
                        const uint2 *p = static_cast<const uint2 *>(src) + base + u * kWork * 4;
                        a = ld_cells2(p);
                        b = ld_cells2(p + 2);
                    }
                    ok = ok && a.y == tag && a.w == tag && b.y == tag && b.w == tag;
                    v[u] = make_float4(__uint_as_float(a.x), __uint_as_float(a.z), __uint_as_float(b.x), __uint_as_float(b.z));
                }
                if (ok || *abort_flag) break;
                if (i == kPolls) *abort_flag = 1;
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
                        const float4 r = *reinterpret_cast<const float4 *>(smem + off_row + (base + u * kWork * 4) * 4);
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
                st_cell(logit_cell, d * scale, logit_tag);
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
    return cta_aborted(abort_flag);
}

// ---- a warp's private ring: it issues its own copies and consumes them, so one "full" barrier per stage is all it takes.
// `parity`: per stage, the parity of its next completion. ----
__device__ __forceinline__ void ring_wait(uint64_t *bars, int s, uint32_t &parity, volatile int *abort_flag)
{
    if (!mbar_try_wait(&bars[s], (parity >> s) & 1)) wait_slow(&bars[s], (parity >> s) & 1, abort_flag);
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
__device__ __noinline__ uint32_t prefetch(const uint8_t *w, int r0, int n, uint32_t row_bytes, int ur, uint8_t *buf, int ring_bytes,
                                          uint64_t *bars)
{
    const uint32_t sb = stage_bytes_of(ur * row_bytes);
    const int lane = threadIdx.x & 31;
    const int stages = min(kStages, ring_bytes / static_cast<int>(sb)), count = min(stages, n > 0 ? (n + ur - 1) / ur : 0);
    if (lane < count) issue_unit(w, r0 + lane * ur, min(ur, n - lane * ur), row_bytes, buf + lane * sb, &bars[lane]);
    __syncwarp();
    return (1u << count) - 1;
}
// Those rows (first units requested by prefetch() with the same arguments) times the staged vector from super-block xcol on:
// dst[row] = value (+ add[row - r0]), as a cell if tag != 0. Returns the ring's parities.
template <class F, int RU>
__device__ __noinline__ uint32_t matvec(const uint8_t *w, int bpr, int lv, int r0, int n, void *dst, uint32_t tag, const float *add, int xcol,
                                        int xc, uint8_t *buf, int ring_bytes, uint64_t *bars, uint32_t parity, volatile int *abort_flag)
{
    const int lane = threadIdx.x & 31, q = lane >> 2, sub = lane & 3;
    const int v = 1 << lv, rpp = 8 >> lv, cq = q & (v - 1), rq = q >> lv, W = 4 << lv;
    const int groups = (bpr + v - 1) >> lv, ur = RU * rpp;
    const uint32_t row_bytes = bpr * F::kBlockBytes, sb = stage_bytes_of(ur * row_bytes);
    const int stages = min(kStages, ring_bytes / static_cast<int>(sb));
    typename F::XRegs xr;
    int s = 0;
#pragma unroll 1
    for (int r = 0; r < n; r += ur) {
        ring_wait(bars, s, parity, abort_flag);
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
            const float o = sum + (add ? add[row] : 0.0f);
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
__device__ __forceinline__ void share(const Split &sp, int gid, int &i0, int &n)
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

// A head's 128 values, four per lane at lane + 32 i: RMS norm (w may be null) and rotation.
__device__ __noinline__ float4 norm_rope(float4 v, const float *w, float eps, const float *cos_t, const float *sin_t)
{
    const int lane = threadIdx.x & 31;
    const float ss = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
    if (w) {
        const float f = 1.0f / sqrtf(ss * (1.0f / 128.0f) + eps);
        v.x *= f * __ldg(w + lane);
        v.y *= f * __ldg(w + lane + 32);
        v.z *= f * __ldg(w + lane + 64);
        v.w *= f * __ldg(w + lane + 96);
    }
    const float c0 = __ldcg(cos_t + lane), c1 = __ldcg(cos_t + lane + 32), s0 = __ldcg(sin_t + lane), s1 = __ldcg(sin_t + lane + 32);
    return make_float4(v.x * c0 - v.z * s0, v.y * c1 - v.w * s1, v.x * s0 + v.z * c0, v.y * s1 + v.w * c1);
}

// K / V rows of a tile of 16 positions, a row per lane
__device__ __forceinline__ void load_kv(const __half *kv_k, const __half *kv_v, int tile, int pos, int n_kv, int kvh, uint8_t *buf, uint64_t *bar)
{
    const int lane = threadIdx.x & 31;
    if (lane == 0) mbar_expect_tx(bar, 32 * 256);
    __syncwarp();
    const int p = min(tile * 16 + (lane & 15), pos);
    bulk_g2s(buf + lane * kKvPitch, (lane < 16 ? kv_k : kv_v) + ((size_t)p * n_kv + kvh) * 128, 256, bar);
}

// This warp's tiles (tile, tile + 16, ... < t1; the first has been requested into the ring) for the 16 query heads whose
// fragments are in shared memory at 0 (hi halves) and 4096 (lo): leaves the unnormalised result [16][kPitch] in the ring, the
// running maxima (log2 domain) and sums in M.am / M.al. The tile of the newest position takes its K and V from the projections
// and, with store, writes them to the cache. Returns the ring's parities.
__device__ __noinline__ uint32_t attn_tiles(int tile, int t1, int pos, int n_kv, int kvh, __half *kv_k, __half *kv_v, bool store,
                                            const uint2 *c_k, const uint2 *c_v, uint32_t tag, const float *k_norm, float eps,
                                            const float *cos_t, const float *sin_t, uint8_t *buf, uint32_t parity, int off_misc)
{
    Misc &M = *reinterpret_cast<Misc *>(smem + off_misc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
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
        ring_wait(bars, 0, parity, &M.abort_flag);
        if (tile == (pos >> 4)) {
            float kv[4], vv[4];
            wait_values4(c_k + kvh * 128 + lane, tag, &M.abort_flag, kv);
            wait_values4(c_v + kvh * 128 + lane, tag, &M.abort_flag, vv);
            __syncwarp();
            const float4 kr = norm_rope(make_float4(kv[0], kv[1], kv[2], kv[3]), k_norm, eps, cos_t, sin_t);
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
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
            const uint8_t *f = smem + (2 * jj * 32 + lane) * 16;
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
        load_kv(kv_k, kv_v, tile, pos, n_kv, kvh, buf, &bars[0]);
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

// Warp h (< nh) brings query head h0 + h into the fragments (hi + lo halves of q * scale * log2 e); the others' rows are zero.
__device__ __noinline__ void q_fragments(const uint2 *c_q, uint32_t tag, bool live, const float *q_norm, float eps, const float *cos_t,
                                         const float *sin_t, float sc, int off_misc)
{
    Misc &M = *reinterpret_cast<Misc *>(smem + off_misc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
        wait_values4(c_q + lane, tag, &M.abort_flag, v);
        __syncwarp();
        const float4 r = norm_rope(make_float4(v[0], v[1], v[2], v[3]), q_norm, eps, cos_t, sin_t);
        v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = lane + 32 * i, kk = d & 15;
        const int at = ((d >> 4) * 32 + (warp & 7) * 4 + ((kk & 7) >> 1)) * 16 + ((warp >> 3) + 2 * (kk >> 3)) * 4 + (kk & 1) * 2;
        const float s = v[i] * sc;
        const __half hi = __float2half_rn(s);
        *reinterpret_cast<__half *>(smem + at) = hi;
        *reinterpret_cast<__half *>(smem + 4096 + at) = __float2half_rn(s - __half2float(hi));
    }
}

// The CTA's partial of nw warps: one head per warp, four dims per lane, into the cells of slot `slot`.
__device__ __noinline__ void attn_partial(int nw, uint2 *c_part, uint2 *c_ml, int slot, uint32_t tag, int off_misc, int off_ring, int ring_bytes)
{
    Misc &M = *reinterpret_cast<Misc *>(smem + off_misc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float m = -INFINITY, s = 0.0f;
#pragma unroll 1
    for (int w = 0; w < nw; w++) m = fmaxf(m, M.am[w][warp]);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int w = 0; w < nw; w++) {
        const float f = exp2f(M.am[w][warp] - m);
        const float4 o = *reinterpret_cast<const float4 *>(smem + off_ring + w * ring_bytes + (warp * kPitch + 4 * lane) * 4);
        s = fmaf(M.al[w][warp], f, s);
        a.x = fmaf(o.x, f, a.x); a.y = fmaf(o.y, f, a.y); a.z = fmaf(o.z, f, a.z); a.w = fmaf(o.w, f, a.w);
    }
    uint2 *p = c_part + ((size_t)slot * 16 + warp) * 128 + 4 * lane;
    st_cells2(p, a.x, a.y, tag);
    st_cells2(p + 2, a.z, a.w, tag);
    if (lane == 0) st_cells2(c_ml + ((size_t)slot * 16 + warp) * 2, m, s, tag);
}

// Merges the nc chunks' partials of one head (hq of head block b): the CTA's warps over the chunks; cells of the result.
__device__ __noinline__ void merge_head(int b, int hq, int nc, int chunks, const uint2 *c_part, const uint2 *c_ml, uint2 *dst, uint32_t tag, int off_misc)
{
    Misc &M = *reinterpret_cast<Misc *>(smem + off_misc);
    volatile int *abort_flag = &M.abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float m = -INFINITY, s = 0.0f;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int c0 = warp; c0 < nc; c0 += 3 * kWarps) {
        uint4 ms[3], o0[3], o1[3];
#pragma unroll 1
        for (uint32_t i = 0;; i++) {
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const size_t slot = ((size_t)b * chunks + min(c0 + u * kWarps, nc - 1)) * 16 + hq;
                ms[u] = ld_cells2(c_ml + slot * 2);
                o0[u] = ld_cells2(c_part + slot * 128 + 4 * lane);
                o1[u] = ld_cells2(c_part + slot * 128 + 4 * lane + 2);
                ok = ok && ms[u].y == tag && ms[u].w == tag && o0[u].y == tag && o0[u].w == tag && o1[u].y == tag && o1[u].w == tag;
            }
            if (ok || *abort_flag) break;
            if (i == kPolls) *abort_flag = 1;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 3; u++) {
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
    float *buf = reinterpret_cast<float *>(smem);  // [16][128]
    *reinterpret_cast<float4 *>(buf + warp * 128 + 4 * lane) = a;
    if (lane == 0) {
        M.red[0][warp] = m;
        M.red[1][warp] = s;
    }
    cta_sync();
    if (tid < 128) {
        float mt = -INFINITY, st = 0.0f, o = 0.0f;
#pragma unroll 1
        for (int w = 0; w < kWarps; w++) mt = fmaxf(mt, M.red[0][w]);
#pragma unroll 1
        for (int w = 0; w < kWarps; w++) {
            const float f = exp2f(M.red[0][w] - mt);  // 0 for a warp without a chunk
            st = fmaf(M.red[1][w], f, st);
            o = fmaf(buf[w * 128 + tid], f, o);
        }
        st_cell(dst + tid, o / st, tag);
    }
    cta_sync();
}

}  // namespace
}  // namespace persist
}  // namespace mb200
