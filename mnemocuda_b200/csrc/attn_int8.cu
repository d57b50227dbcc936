// Decode attention over the INT8 KV cache on tensor cores (reference src/kernels.cu:1382-1480, 1536-1546).
//
// Grid (KV head x block of 16 query heads, chunk of positions); every K / V byte is read once for all query heads of
// the block. The cache is 128 + 4 bytes per row, so the kernel is HBM-bound once the arithmetic is on
// mma.sync.m16n8k16: 64 heads / 4 KV heads / 32768 positions take 21 us (5.3 us at the copy rate; 136 with fp32 FMAs and a
// five-step warp reduction per position and head). What is left is latency: a CTA has eight warps, 20 % of the issue slots are
// used, and the merges of the warps, the cluster and the last CTA come one after the other behind barriers and a ticket.
//   * int8 values become fp16 exactly (0x6400 | (v + 128) is 1152 + v); q and the probabilities are carried as
//     hi + lo fp16 pairs (22 bits), accumulation is fp32, so nothing is rounded beyond fp32 arithmetic's own size. A head's q
//     is brought into fp16's range by a power of two of its own, which its scores take back.
//   * The K scale multiplies the score. The V scale is folded into the probability: the accumulators hold
//     sum p * (vs / vmax) * v with vmax the largest V scale the warp has met, so the fp16 pair never leaves its range
//     whatever the scales are; vmax multiplies back at the end.
//   * Two CTAs of a cluster (consecutive chunks) exchange their partial results through distributed shared memory, each
//     merging eight of the sixteen heads; what is left are 18 instead of 36 partials per head block, merged by the last
//     CTA of each half to arrive (ticket). A cluster of two always fits the SMs; larger ones do not divide them.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <stdio.h>

#include "common.cuh"

namespace mb200 {
int pdl_enabled();

namespace {
namespace cg = cooperative_groups;

constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kHD = 128;      // head dimension
constexpr int kTile = 16;     // positions per warp step
constexpr int kPitch = 132;   // floats between heads in the shared-memory results (4 x 33: conflict-free stores)
constexpr int kMaxGroups = 64;   // (KV head, query-head block) pairs per launch
constexpr int kMaxSlots = 256;   // (group, cluster) pairs per launch
constexpr float kLog2e = 1.4426950408889634f;

struct Work {  // library-resident workspace (2.1 MB per device)
    float part[kMaxSlots * 16 * kHD];
    float ml[kMaxSlots * 2 * 16];
    int tickets[kMaxGroups * 2];
};
__device__ Work g_work;

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// (a, b) as fp16 plus what that rounding dropped
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 back = __half22float2(h);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = pack2(a - back.x, b - back.y);
}
__device__ __forceinline__ float exp2_fast(float x)  // the hardware's 2^x, 0 for -inf; its error (2 ulp) is exp2f's
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two of the four (int8 + 128) bytes of w -> two fp16: sel 0x4140 = bytes 0, 1; 0x4342 = bytes 2, 3
__device__ __forceinline__ uint32_t to_half2(uint32_t w, uint32_t sel)
{
    const uint32_t t = __byte_perm(w, 0x64646464u, sel);
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&t), __half2half2(__ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t *>(&r);
}

// Fragments (g = lane / 4, t = lane % 4):
//  Q K^T:  the 16 k of step j are dims 32 t + 4 j + {0,1 | 2,3}: a thread's share of a K row is 32 contiguous bytes
//  P V:    k = position in the tile, column g of output tile u = dim 16 g + u: 16 contiguous bytes of four V rows
template <int CL>
__global__ void __launch_bounds__(kThreads, 1)
attn_int8_kernel(const float *q, const int8_t *__restrict__ kv_k, const int8_t *__restrict__ kv_v, const float *k_scales,
                 const float *v_scales, float *out, int n_kv_heads, int gqa, int seq_len, float scale, int tiles_per_chunk)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint4 *afrag = reinterpret_cast<uint4 *>(smem_raw);           // [2 hi/lo][8 steps][32 lanes]
    float *osm = reinterpret_cast<float *>(smem_raw + 8192);      // [8 warps][16 heads][kPitch]; later the CTA's partial in [0]
    float *msm = osm + kWarps * 16 * kPitch;                      // [8][16] running maxima (log2 domain)
    float *lsm = msm + kWarps * 16;                               // [8][16] sums
    float *cml = lsm + kWarps * 16;                               // [2][16] the CTA's max and sum
    __shared__ int is_last;
    __shared__ float head_scale[16];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int qb = (gqa + 15) / 16;
    const int kvh = blockIdx.x / qb, blk = blockIdx.x % qb;
    const int h0 = kvh * gqa + blk * 16, nh = min(16, gqa - blk * 16);
    const int p_begin = min(seq_len, static_cast<int>(blockIdx.y) * tiles_per_chunk * kTile);
    const int p_end = min(seq_len, p_begin + tiles_per_chunk * kTile);
    const size_t row_stride = (size_t)n_kv_heads * kHD;
    const int8_t *kbase = kv_k + (size_t)kvh * kHD + 32 * t;
    const int8_t *vbase = kv_v + (size_t)kvh * kHD + 16 * g;
    const float *sbase = (lane < 16 ? k_scales : v_scales) + kvh;  // lanes 0-15: K scales of the tile, 16-31: V scales

    struct Tile {
        uint4 k[2][2], v[4];
        float sc;
    };
    const int n_tiles = (p_end - p_begin + kTile - 1) / kTile, last = max(p_end - 1, 0);
    auto load = [&](int tile, Tile &x) {
        const int base = p_begin + tile * kTile;
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
            const uint4 *src = reinterpret_cast<const uint4 *>(kbase + (size_t)min(base + nt * 8 + g, last) * row_stride);
            x.k[nt][0] = __ldcg(src);
            x.k[nt][1] = __ldcg(src + 1);
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
            x.v[r] = __ldcg(reinterpret_cast<const uint4 *>(vbase + (size_t)min(base + 2 * t + (r & 1) + (r >> 1) * 8, last) * row_stride));
        x.sc = __ldcg(sbase + (size_t)min(base + (lane & 15), last) * n_kv_heads);
    };
    Tile cur, nxt;
    if (warp < n_tiles) load(warp, cur);

    // Q fragments, hi + lo of q * scale * log2 e times a power of two that brings the head's largest to 2^12: a warp per head, lane
    // (t, j) has the four dims 32 t + 4 j .. + 3 of step j. The scores take the power back (head_scale).
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int h = warp + kWarps * i;
        const float sc = scale * kLog2e;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (h < nh) r = __ldcg(reinterpret_cast<const float4 *>(q + (size_t)(h0 + h) * kHD) + lane);
        r.x *= sc; r.y *= sc; r.z *= sc; r.w *= sc;
        const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fmaxf(fabsf(r.z), fabsf(r.w)))));
        const uint32_t e = min(max(top >> 23, 13u), 253u);  // its exponent; the power and its inverse stay normal
        const float up = __uint_as_float((266u - e) << 23);
        uint32_t hi[2], lo[2];
        split2(r.x * up, r.y * up, hi[0], lo[0]);
        split2(r.z * up, r.w * up, hi[1], lo[1]);
        uint32_t *f = reinterpret_cast<uint32_t *>(afrag + (lane & 7) * 32 + warp * 4 + (lane >> 3)) + i;
        f[0] = hi[0];  // rows g, g + 8 of k 2t, 2t + 1; of k 2t + 8, 2t + 9
        f[2] = hi[1];
        f[8 * 32 * 4] = lo[0];
        f[8 * 32 * 4 + 2] = lo[1];
        if (lane == 0) head_scale[h] = __uint_as_float((e - 12u) << 23);
    }
    __syncthreads();
    const float f0 = head_scale[g], f1 = head_scale[g + 8];

    float O[16][4];
#pragma unroll
    for (int u = 0; u < 16; u++) O[u][0] = O[u][1] = O[u][2] = O[u][3] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f, vmax = 0.0f;
    for (int tile = warp; tile < n_tiles; tile += kWarps) {
        const int base = p_begin + tile * kTile;
        if (tile + kWarps < n_tiles) load(tile + kWarps, nxt);
        // four independent accumulator chains (two position halves x hi / lo), added at the end
        float S[2][4], Sl[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++) S[nt][e] = Sl[nt][e] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint4 ah = afrag[j * 32 + lane], al = afrag[(8 + j) * 32 + lane];
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                const uint4 kk = cur.k[nt][j >> 2];
                const uint32_t u = ((j & 3) == 0 ? kk.x : (j & 3) == 1 ? kk.y : (j & 3) == 2 ? kk.z : kk.w) ^ 0x80808080u;
                const uint32_t b0 = to_half2(u, 0x4140), b1 = to_half2(u, 0x4342);
                mma16816(S[nt], ah.x, ah.y, ah.z, ah.w, b0, b1);
                mma16816(Sl[nt], al.x, al.y, al.z, al.w, b0, b1);
            }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, vs[4], vt = 0.0f;
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int i = nt * 8 + 2 * t + e;
                const float ks = __shfl_sync(0xffffffffu, cur.sc, i);
                vs[nt * 2 + e] = __shfl_sync(0xffffffffu, cur.sc, 16 + i);
                const bool in = base + i < p_end;
                S[nt][e] = in ? (S[nt][e] + Sl[nt][e]) * (ks * f0) : -INFINITY;
                S[nt][2 + e] = in ? (S[nt][2 + e] + Sl[nt][2 + e]) * (ks * f1) : -INFINITY;
                mx0 = fmaxf(mx0, S[nt][e]);
                mx1 = fmaxf(mx1, S[nt][2 + e]);
                vt = fmaxf(vt, fabsf(vs[nt * 2 + e]));
            }
        }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            vt = fmaxf(vt, __shfl_xor_sync(0xffffffffu, vt, o));
        }
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1), nv = fmaxf(vmax, vt);
        const float r0 = exp2_fast(m0 - n0), r1 = exp2_fast(m1 - n1);  // 2^-inf = 0 on the first tile
        const float vinv = nv > 0.0f ? 1.0f / nv : 0.0f;
        const float rv = vmax * vinv;
        m0 = n0;
        m1 = n1;
        vmax = nv;
        l0 *= r0;
        l1 *= r1;
        const float o0 = r0 * rv, o1 = r1 * rv;
        if (__any_sync(0xffffffffu, o0 != 1.0f || o1 != 1.0f)) {  // the running maxima settle after a few tiles
#pragma unroll
            for (int u = 0; u < 16; u++) {
                O[u][0] *= o0;
                O[u][1] *= o0;
                O[u][2] *= o1;
                O[u][3] *= o1;
            }
        }
        uint32_t ph[4], pl[4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
            const float p0 = exp2_fast(S[nt][0] - n0), p1 = exp2_fast(S[nt][1] - n0);
            const float p2 = exp2_fast(S[nt][2] - n1), p3 = exp2_fast(S[nt][3] - n1);
            l0 += p0 + p1;
            l1 += p2 + p3;
            const float va = vs[nt * 2] * vinv, vb = vs[nt * 2 + 1] * vinv;
            split2(p0 * va, p1 * vb, ph[nt * 2], pl[nt * 2]);          // row g,     positions 8 nt + 2t, 2t + 1
            split2(p2 * va, p3 * vb, ph[nt * 2 + 1], pl[nt * 2 + 1]);  // row g + 8
        }
        const uint32_t vw[4][4] = {{cur.v[0].x, cur.v[0].y, cur.v[0].z, cur.v[0].w}, {cur.v[1].x, cur.v[1].y, cur.v[1].z, cur.v[1].w},
                                   {cur.v[2].x, cur.v[2].y, cur.v[2].z, cur.v[2].w}, {cur.v[3].x, cur.v[3].y, cur.v[3].z, cur.v[3].w}};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            // bytes of rows 2t and 2t + 1 (and of 2t + 8, 2t + 9) interleaved: one dim's pair side by side
            const uint32_t a = vw[0][w] ^ 0x80808080u, b = vw[1][w] ^ 0x80808080u;
            const uint32_t c = vw[2][w] ^ 0x80808080u, d = vw[3][w] ^ 0x80808080u;
            const uint32_t ab[2] = {__byte_perm(a, b, 0x5140), __byte_perm(a, b, 0x7362)};
            const uint32_t cd[2] = {__byte_perm(c, d, 0x5140), __byte_perm(c, d, 0x7362)};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t sel = (i & 1) ? 0x4342 : 0x4140;
                const uint32_t b0 = to_half2(ab[i >> 1], sel), b1 = to_half2(cd[i >> 1], sel);
                mma16816(O[4 * w + i], ph[0], ph[1], ph[2], ph[3], b0, b1);
                mma16816(O[4 * w + i], pl[0], pl[1], pl[2], pl[3], b0, b1);
            }
        }
        cur = nxt;
    }
    // ---- the warps' shares to shared memory ----
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (t == 0) {
        msm[warp * 16 + g] = m0;
        msm[warp * 16 + g + 8] = m1;
        lsm[warp * 16 + g] = l0;
        lsm[warp * 16 + g + 8] = l1;
    }
    {
        float *ow = osm + warp * 16 * kPitch;  // dim d of a head sits at (d / 32) * 33 + d % 32
#pragma unroll
        for (int u = 0; u < 16; u++) {
            ow[g * kPitch + 33 * t + u] = O[u][0] * vmax;        // dim 16 (2t) + u
            ow[g * kPitch + 33 * t + 16 + u] = O[u][1] * vmax;   // dim 16 (2t + 1) + u
            ow[(g + 8) * kPitch + 33 * t + u] = O[u][2] * vmax;
            ow[(g + 8) * kPitch + 33 * t + 16 + u] = O[u][3] * vmax;
        }
    }
    __syncthreads();
    // ---- the CTA's partial: thread -> head tid / 16, dims 8 (tid % 16) .. + 7 ----
    const int head = tid >> 4, d0 = (tid & 15) * 8;
    const int at = (d0 >> 5) * 33 + (d0 & 31);
    float M = -INFINITY, L = 0.0f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < kWarps; w++) M = fmaxf(M, msm[w * 16 + head]);
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const float mw = msm[w * 16 + head];
        const float f = (mw == -INFINITY) ? 0.0f : exp2_fast(mw - M);
        L = fmaf(lsm[w * 16 + head], f, L);
        const float *ow = osm + (w * 16 + head) * kPitch + at;
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = fmaf(ow[i], f, acc[i]);
    }
    auto store_out = [&](float *dst, const float (&v)[8], float f) {
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0] * f, v[1] * f, v[2] * f, v[3] * f);
        *reinterpret_cast<float4 *>(dst + 4) = make_float4(v[4] * f, v[5] * f, v[6] * f, v[7] * f);
    };
    int rank = 0;
    bool mine = true;  // this thread's (head, dims) belong to this CTA's share of the merge
    if (CL > 1) {
        // post the partial (each thread overwrites only what it alone has read), then merge heads [8 rank, 8 rank + 8)
        cg::cluster_group cl = cg::this_cluster();
        rank = static_cast<int>(cl.block_rank());
#pragma unroll
        for (int i = 0; i < 8; i++) osm[head * kPitch + at + i] = acc[i];
        if ((tid & 15) == 0) {
            cml[head] = M;
            cml[16 + head] = L;
        }
        cl.sync();
        mine = (head >> 3) == rank;
        if (mine) {
            const float *po = cl.map_shared_rank(osm, rank ^ 1), *pm = cl.map_shared_rank(cml, rank ^ 1);
            const float Mo = pm[head], Lo = pm[16 + head], Mt = fmaxf(M, Mo);
            const float fa = (M == -INFINITY) ? 0.0f : exp2_fast(M - Mt), fb = (Mo == -INFINITY) ? 0.0f : exp2_fast(Mo - Mt);
            L = L * fa + Lo * fb;
            M = Mt;
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = acc[i] * fa + po[head * kPitch + at + i] * fb;
        }
        cl.sync();  // the partner has read this CTA's shared memory
    }
    const int S = gridDim.y / CL;  // partials per head block
    if (S == 1) {
        if (mine && head < nh) store_out(out + (size_t)(h0 + head) * kHD + d0, acc, L > 0.0f ? 1.0f / L : 0.0f);
        return;
    }
    const size_t slot = (size_t)blockIdx.x * S + blockIdx.y / CL;
    if (mine) {
        store_out(g_work.part + (slot * 16 + head) * kHD + d0, acc, 1.0f);
        if ((tid & 15) == 0) {
            g_work.ml[(slot * 2 + 0) * 16 + head] = M;
            g_work.ml[(slot * 2 + 1) * 16 + head] = L;
        }
    }
    __syncthreads();
    if (tid == 0) {  // one fence for the CTA: the barrier orders the other threads' stores before it
        __threadfence();
        is_last = atomicAdd(&g_work.tickets[blockIdx.x * 2 + rank], 1) == S - 1;
        __threadfence();
    }
    __syncthreads();
    if (!is_last) return;
    if (mine && head < nh) {
        const size_t s0 = (size_t)blockIdx.x * S;
        float Mt = -INFINITY;
        for (int c0 = 0; c0 < S; c0 += 8) {  // eight partials' loads in flight at a time
            float mv[8];
#pragma unroll
            for (int u = 0; u < 8; u++) mv[u] = __ldcg(g_work.ml + ((s0 + min(c0 + u, S - 1)) * 2) * 16 + head);
#pragma unroll
            for (int u = 0; u < 8; u++) Mt = fmaxf(Mt, mv[u]);
        }
        float Lt = 0.0f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int c0 = 0; c0 < S; c0 += 8) {
            float mv[8], lv[8];
            float4 a[8], b[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const size_t sl = s0 + min(c0 + u, S - 1);
                mv[u] = __ldcg(g_work.ml + (sl * 2) * 16 + head);
                lv[u] = __ldcg(g_work.ml + (sl * 2 + 1) * 16 + head);
                a[u] = __ldcg(reinterpret_cast<const float4 *>(g_work.part + (sl * 16 + head) * kHD + d0));
                b[u] = __ldcg(reinterpret_cast<const float4 *>(g_work.part + (sl * 16 + head) * kHD + d0 + 4));
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const float f = (c0 + u >= S || mv[u] == -INFINITY) ? 0.0f : exp2_fast(mv[u] - Mt);
                Lt = fmaf(lv[u], f, Lt);
                o[0] = fmaf(a[u].x, f, o[0]); o[1] = fmaf(a[u].y, f, o[1]); o[2] = fmaf(a[u].z, f, o[2]); o[3] = fmaf(a[u].w, f, o[3]);
                o[4] = fmaf(b[u].x, f, o[4]); o[5] = fmaf(b[u].y, f, o[5]); o[6] = fmaf(b[u].z, f, o[6]); o[7] = fmaf(b[u].w, f, o[7]);
            }
        }
        store_out(out + (size_t)(h0 + head) * kHD + d0, o, Lt > 0.0f ? 1.0f / Lt : 0.0f);
    }
    if (tid == 0) g_work.tickets[blockIdx.x * 2 + rank] = 0;  // ready for the next launch
}

constexpr int kSmem = 8192 + (kWarps * 16 * kPitch + 2 * kWarps * 16 + 32) * 4;

template <int CL>
void launch(const float *q, const int8_t *k, const int8_t *v, const float *ks, const float *vs, float *out, int groups, int chunks,
            int n_kv_heads, int gqa, int seq_len, float scale, cudaStream_t stream)
{
    const int tiles = (seq_len + kTile - 1) / kTile;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups, chunks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = CL;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, attn_int8_kernel<CL>, q, k, v, ks, vs, out, n_kv_heads, gqa, seq_len, scale, (tiles + chunks - 1) / chunks);
}

}  // namespace

void attn_int8_init()
{
    static bool done[kMaxDevices] = {false};
    const int dev = current_device();
    if (done[dev]) return;
    cudaFuncSetAttribute(attn_int8_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    cudaFuncSetAttribute(attn_int8_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    done[dev] = true;
}

// false = a shape or alignment this kernel does not take (nothing launched)
bool attn_int8_tc(const float *q, const void *k, const void *v, const float *ks, const float *vs, float *out, int n_heads_q,
                  int n_kv_heads, int gqa, int seq_len, float scale, cudaStream_t stream)
{
    const uintptr_t addr = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                           reinterpret_cast<uintptr_t>(out);
    if (gqa < 1 || n_heads_q != n_kv_heads * gqa || (addr & 15)) return false;
    const int groups = n_kv_heads * ((gqa + 15) / 16);
    if (groups > kMaxGroups) return false;
    attn_int8_init();
    // one CTA per SM; a chunk of fewer positions than one tile per warp would only add partial results to merge
    const int tiles = (seq_len + kTile - 1) / kTile;
    int chunks = device_sms() / groups;
    if (chunks > (tiles + kWarps - 1) / kWarps) chunks = (tiles + kWarps - 1) / kWarps;
    if (chunks > kMaxSlots / groups) chunks = kMaxSlots / groups;
    const int8_t *k8 = static_cast<const int8_t *>(k), *v8 = static_cast<const int8_t *>(v);
    if (chunks < 2) {
        launch<1>(q, k8, v8, ks, vs, out, groups, 1, n_kv_heads, gqa, seq_len, scale, stream);
    } else {
        launch<2>(q, k8, v8, ks, vs, out, groups, chunks & ~1, n_kv_heads, gqa, seq_len, scale, stream);
    }
    return true;
}

}  // namespace mb200
