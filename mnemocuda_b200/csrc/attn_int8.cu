// Decode attention over the INT8 KV cache on tensor cores (reference src/kernels.cu:1382-1480, 1536-1546).
//
// Grid (KV head x block of 16 query heads, chunk of positions); every K / V byte is read once for all query heads of
// the block. The cache is 128 + 4 bytes per row, so the kernel is HBM-bound once the arithmetic is on
// mma.sync.m16n8k16: 64 heads / 4 KV heads / 32768 positions take 15.0 us in a chain of calls, 15.7 one call at a time (5.3 us at the copy rate; 21.5 and 20.9
// with eight warps that held a tile ahead in registers, 136 with fp32 FMAs and a five-step warp reduction per position and head), 32 / 8 heads
// 18.0 in a chain (31.2). By clock
// stamps, 64 / 4 at 32768: 3 us until q is in fragments (while the first tiles stream), 7.2 the tiles (the MMAs alone are 5), then one
// after the other the merges of the warps (1.1), the cluster (0.5) and, behind a ticket (1.3), the last CTA (1.2).
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

constexpr int kWarps = 12, kThreads = kWarps * 32, kFewTiles = 4;
constexpr int kStages = 2;    // tiles on their way per warp
constexpr int kHD = 128;      // head dimension
constexpr int kTile = 16;     // positions per warp step
constexpr int kRow = 144;     // bytes between K / V rows of a stage: 16-byte reads of eight lanes hit all banks
constexpr int kStageBytes = 2 * kTile * kRow + 2 * kTile * 4;  // K rows, V rows, K scales, V scales
constexpr int kPitch = 132;   // floats between heads in the shared-memory results (4 x 33: conflict-free stores)
constexpr int kMaxGroups = 64;   // (KV head, query-head block) pairs per launch
constexpr int kBatch = 20;     // partials a merging thread has on their way
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
    asm(
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
// PACK: at most eight query heads per KV head; rows g are their q and probabilities' hi halves, rows g + 8 the lo ones, one MMA for both.
// FEW: a single CTA per head block, whose first kFewTiles warps have a tile at most. All twelve warps' results stored and merged
// cost 64 / 4 heads at 64 positions 4.1 instead of 3.5 us, 32 / 8 heads 3.1 instead of 2.9.
template <int CL, bool PACK, bool FEW>
__global__ void __launch_bounds__(kThreads, 1)
attn_int8_kernel(const float *q, const int8_t *__restrict__ kv_k, const int8_t *__restrict__ kv_v, const float *k_scales,
                 const float *v_scales, float *out, int n_kv_heads, int gqa, int seq_len, float scale, int tiles_per_chunk)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int HB = PACK ? 8 : 16, kMergers = HB * 16;  // heads of a CTA; threads that merge, sixteen per head
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint4 *afrag = reinterpret_cast<uint4 *>(smem_raw);           // [2 hi/lo][8 steps][32 lanes]
    float *msm = reinterpret_cast<float *>(smem_raw + 8192);      // [warps][16] running maxima (log2 domain)
    float *lsm = msm + kWarps * 16;                               // [warps][16] sums
    float *cml = lsm + kWarps * 16;                               // [2][16] the CTA's max and sum
    uint8_t *rings = reinterpret_cast<uint8_t *>(cml + 32);       // [warps][stages]
    float *osm = reinterpret_cast<float *>(rings);                // then [warps][16 heads][kPitch]; last the CTA's partial in [0]
    __shared__ int is_last;
    __shared__ float head_scale[16];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int qb = (gqa + 15) / 16;
    const int kvh = blockIdx.x / qb, blk = blockIdx.x % qb;
    const int h0 = kvh * gqa + blk * 16, nh = min(16, gqa - blk * 16);
    const int p_begin = min(seq_len, static_cast<int>(blockIdx.y) * tiles_per_chunk * kTile);
    const int p_end = min(seq_len, p_begin + tiles_per_chunk * kTile);
    const size_t row_stride = (size_t)n_kv_heads * kHD;
    const int n_tiles = (p_end - p_begin + kTile - 1) / kTile, last = max(p_end - 1, 0);
    // A warp's tiles go through a ring of its own, requested two tiles ahead (one tile ahead in registers, every step waited for
    // memory): lane copies 16 bytes of rows lane / 8 + 4 i, and the K scale (lanes 0-15) or V scale of row lane % 16.
    uint8_t *ring = rings + warp * kStages * kStageBytes;
    const int8_t *ksrc = kv_k + (size_t)kvh * kHD + 16 * (lane & 7), *vsrc = kv_v + (size_t)kvh * kHD + 16 * (lane & 7);
    const float *ssrc = (lane < 16 ? k_scales : v_scales) + kvh;
    const uint32_t dst = smem_u32(ring) + (lane >> 3) * kRow + 16 * (lane & 7), sdst = smem_u32(ring) + 2 * kTile * kRow + 4 * lane;
    auto request = [&](int tile, int stage) {
        if (tile < n_tiles) {
            const int base = p_begin + tile * kTile;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const size_t row = (size_t)min(base + (lane >> 3) + 4 * i, last) * row_stride;
                const uint32_t to = dst + stage * kStageBytes + 4 * i * kRow;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(ksrc + row) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + kTile * kRow), "l"(vsrc + row) : "memory");
            }
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sdst + stage * kStageBytes),
                         "l"(ssrc + (size_t)min(base + (lane & 15), last) * n_kv_heads)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // q comes before the tiles: behind 150 KB of them it took 4 us.
    constexpr int kQ = (HB + kWarps - 1) / kWarps;
    float4 qr[kQ];
#pragma unroll
    for (int i = 0; i < kQ; i++) {
        const int h = warp + kWarps * i;
        qr[i] = h < nh ? __ldcg(reinterpret_cast<const float4 *>(q + (size_t)(h0 + h) * kHD) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    request(warp, 0);

    // Q fragments, hi + lo of q * scale * log2 e times a power of two that brings the head's largest to 2^12: a warp per head, lane
    // (t, j) has the four dims 32 t + 4 j .. + 3 of step j. The scores take the power back (head_scale).
#pragma unroll
    for (int i = 0; i < kQ; i++) {
        const int h = warp + kWarps * i;
        if (h >= HB) break;
        const float sc = scale * kLog2e;
        float4 r = qr[i];
        r.x *= sc; r.y *= sc; r.z *= sc; r.w *= sc;
        const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fmaxf(fabsf(r.z), fabsf(r.w)))));
        const uint32_t e = min(max(top >> 23, 13u), 253u);  // its exponent; the power and its inverse stay normal
        const float up = __uint_as_float((266u - e) << 23);
        uint32_t hi[2], lo[2];
        split2(r.x * up, r.y * up, hi[0], lo[0]);
        split2(r.z * up, r.w * up, hi[1], lo[1]);
        // rows g, g + 8 of k 2t, 2t + 1; of k 2t + 8, 2t + 9
        uint32_t *f = reinterpret_cast<uint32_t *>(afrag + (lane & 7) * 32 + (h & 7) * 4 + (lane >> 3)) + (h >> 3);
        uint32_t *fl = f + (PACK ? 1 : 8 * 32 * 4);
        f[0] = hi[0];
        f[2] = hi[1];
        fl[0] = lo[0];
        fl[2] = lo[1];
        if (lane == 0) head_scale[h] = __uint_as_float((e - 12u) << 23);
    }
    __syncthreads();
    // Requests beyond what the memory system takes hold up the warp that makes them: only the first tile's come before the fragments.
#pragma unroll
    for (int i = 1; i < kStages; i++) request(warp + kWarps * i, i);
    const float f0 = head_scale[g], f1 = PACK ? 0.0f : head_scale[g + 8];

    float O[16][4];
#pragma unroll
    for (int u = 0; u < 16; u++) O[u][0] = O[u][1] = O[u][2] = O[u][3] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f, vmax = 0.0f, vinv = 0.0f;
    int stage = 0;
    for (int tile = warp; tile < n_tiles; tile += kWarps) {
        const int base = p_begin + tile * kTile;
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        __syncwarp();
        const uint8_t *st = ring + stage * kStageBytes;
        const uint8_t *krow = st + g * kRow + 32 * t, *vrow = st + kTile * kRow + 2 * t * kRow + 16 * g;
        const float2 *scales = reinterpret_cast<const float2 *>(st + 2 * kTile * kRow) + t;  // of positions 2t, 2t + 1; four apart: 8 further
        const float2 ks[2] = {scales[0], scales[4]}, vs2[2] = {scales[8], scales[12]};
        uint4 kq[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int i = 0; i < 2; i++) kq[nt][i] = *reinterpret_cast<const uint4 *>(krow + nt * 8 * kRow + 16 * i);
        // four independent accumulator chains (two position halves x hi / lo), added at the end
        float S[2][4], Sl[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++) S[nt][e] = Sl[nt][e] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint4 ah = afrag[j * 32 + lane], al = PACK ? ah : afrag[(8 + j) * 32 + lane];
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                const uint4 kk = kq[nt][j >> 2];
                const uint32_t u = ((j & 3) == 0 ? kk.x : (j & 3) == 1 ? kk.y : (j & 3) == 2 ? kk.z : kk.w) ^ 0x80808080u;
                const uint32_t b0 = to_half2(u, 0x4140), b1 = to_half2(u, 0x4342);
                mma16816(PACK && (j & 1) ? Sl[nt] : S[nt], ah.x, ah.y, ah.z, ah.w, b0, b1);
                if (!PACK) mma16816(Sl[nt], al.x, al.y, al.z, al.w, b0, b1);
            }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, vt = 0.0f;
        const float vs[4] = {vs2[0].x, vs2[0].y, vs2[1].x, vs2[1].y};
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float k = e ? ks[nt].y : ks[nt].x;
                const bool in = base + nt * 8 + 2 * t + e < p_end;
                if (PACK) {
                    S[nt][e] = in ? ((S[nt][e] + Sl[nt][e]) + (S[nt][2 + e] + Sl[nt][2 + e])) * (k * f0) : -INFINITY;
                } else {
                    S[nt][e] = in ? (S[nt][e] + Sl[nt][e]) * (k * f0) : -INFINITY;
                    S[nt][2 + e] = in ? (S[nt][2 + e] + Sl[nt][2 + e]) * (k * f1) : -INFINITY;
                    mx1 = fmaxf(mx1, S[nt][2 + e]);
                }
                mx0 = fmaxf(mx0, S[nt][e]);
                vt = fmaxf(vt, fabsf(vs[nt * 2 + e]));
            }
        }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            if (!PACK) mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            vt = fmaxf(vt, __shfl_xor_sync(0xffffffffu, vt, o));
        }
        // What the accumulators are relative to, a head's maximum and the largest V scale, follows only when it falls behind by more
        // than 2^8 and 2^4: products stay below 2^12, inside fp16's range, and most tiles need not touch the 64 accumulators.
        const bool up0 = mx0 > m0 + 8.0f, up1 = !PACK && mx1 > m1 + 8.0f, upv = vt > 16.0f * vmax;
        if (__any_sync(0xffffffffu, up0 || up1 || upv)) {
            const float n0 = up0 ? mx0 : m0, n1 = up1 ? mx1 : m1, nv = upv ? vt : vmax;
            const float r0 = n0 == m0 ? 1.0f : exp2_fast(m0 - n0), r1 = n1 == m1 ? 1.0f : exp2_fast(m1 - n1);  // 2^-inf = 0 on the first tile
            vinv = nv > 0.0f ? 1.0f / nv : 0.0f;
            const float rv = nv == vmax ? 1.0f : vmax * vinv, o0 = r0 * rv, o1 = r1 * rv;
            m0 = n0;
            m1 = n1;
            vmax = nv;
            l0 *= r0;
            l1 *= r1;
#pragma unroll
            for (int u = 0; u < 16; u++) {
                O[u][0] *= o0;
                O[u][1] *= o0;
                O[u][2] *= PACK ? o0 : o1;
                O[u][3] *= PACK ? o0 : o1;
            }
        }
        uint32_t ph[4], pl[4];  // rows g: positions 8 nt + 2t, 2t + 1 in 2 nt; rows g + 8 in 2 nt + 1
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
            const float va = vs[nt * 2] * vinv, vb = vs[nt * 2 + 1] * vinv;
            const float p0 = exp2_fast(S[nt][0] - m0), p1 = exp2_fast(S[nt][1] - m0);
            l0 += p0 + p1;
            if (PACK) {
                split2(p0 * va, p1 * vb, ph[nt * 2], ph[nt * 2 + 1]);
            } else {
                const float p2 = exp2_fast(S[nt][2] - m1), p3 = exp2_fast(S[nt][3] - m1);
                l1 += p2 + p3;
                split2(p0 * va, p1 * vb, ph[nt * 2], pl[nt * 2]);
                split2(p2 * va, p3 * vb, ph[nt * 2 + 1], pl[nt * 2 + 1]);
            }
        }
        uint32_t vw[4][4];  // rows 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint4 v = *reinterpret_cast<const uint4 *>(vrow + ((r & 1) + (r >> 1) * 8) * kRow);
            vw[r][0] = v.x; vw[r][1] = v.y; vw[r][2] = v.z; vw[r][3] = v.w;
        }
#pragma unroll
        for (int w = 0; w < 4; w++) {
            // bytes of rows 2t and 2t + 1 (and of 2t + 8, 2t + 9) interleaved: one dim's pair side by side
            const uint32_t a = vw[0][w] ^ 0x80808080u, a2 = vw[1][w] ^ 0x80808080u;
            const uint32_t c = vw[2][w] ^ 0x80808080u, d = vw[3][w] ^ 0x80808080u;
            const uint32_t ab[2] = {__byte_perm(a, a2, 0x5140), __byte_perm(a, a2, 0x7362)};
            const uint32_t cd[2] = {__byte_perm(c, d, 0x5140), __byte_perm(c, d, 0x7362)};
            uint32_t b[8];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t sel = (i & 1) ? 0x4342 : 0x4140;
                b[2 * i] = to_half2(ab[i >> 1], sel);
                b[2 * i + 1] = to_half2(cd[i >> 1], sel);
                mma16816(O[4 * w + i], ph[0], ph[1], ph[2], ph[3], b[2 * i], b[2 * i + 1]);
            }
            if (!PACK)
#pragma unroll
                for (int i = 0; i < 4; i++) mma16816(O[4 * w + i], pl[0], pl[1], pl[2], pl[3], b[2 * i], b[2 * i + 1]);
        }
        __syncwarp();  // all lanes have read the stage
        request(tile + kWarps * kStages, stage);
        if (++stage == kStages) stage = 0;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the rings become the warps' results
    // ---- the warps' shares to shared memory ----
    const bool shares = !FEW || warp < n_tiles;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (t == 0 && shares) {
        msm[warp * 16 + g] = m0;
        lsm[warp * 16 + g] = l0;
        if (!PACK) {
            msm[warp * 16 + g + 8] = m1;
            lsm[warp * 16 + g + 8] = l1;
        }
    }
    if (shares) {
        float *ow = osm + warp * 16 * kPitch;  // dim d of a head sits at (d / 32) * 33 + d % 32
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const float a = PACK ? O[u][0] + O[u][2] : O[u][0], b = PACK ? O[u][1] + O[u][3] : O[u][1];
            ow[g * kPitch + 33 * t + u] = a * vmax;        // dim 16 (2t) + u
            ow[g * kPitch + 33 * t + 16 + u] = b * vmax;   // dim 16 (2t + 1) + u
            if (!PACK) {
                ow[(g + 8) * kPitch + 33 * t + u] = O[u][2] * vmax;
                ow[(g + 8) * kPitch + 33 * t + 16 + u] = O[u][3] * vmax;
            }
        }
    }
    __syncthreads();
    // ---- the CTA's partial: thread -> head tid / 16, dims 8 (tid % 16) .. + 7 ----
    const int head = (tid & (kMergers - 1)) >> 4, d0 = (tid & 15) * 8;
    const bool merges = tid < kMergers;
    const int at = (d0 >> 5) * 33 + (d0 & 31);
    float M = -INFINITY, L = 0.0f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (merges) {
        constexpr int W = FEW ? kFewTiles : kWarps;
#pragma unroll
        for (int w = 0; w < W; w++)
            if (!FEW || w < n_tiles) M = fmaxf(M, msm[w * 16 + head]);
#pragma unroll
        for (int w = 0; w < W; w++) {
            if (FEW && w >= n_tiles) break;
            const float mw = msm[w * 16 + head];
            const float f = (mw == -INFINITY) ? 0.0f : exp2_fast(mw - M);
            L = fmaf(lsm[w * 16 + head], f, L);
            const float *ow = osm + (w * 16 + head) * kPitch + at;
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = fmaf(ow[i], f, acc[i]);
        }
    }
    auto store_out = [&](float *to, const float (&v)[8], float f) {
        *reinterpret_cast<float4 *>(to) = make_float4(v[0] * f, v[1] * f, v[2] * f, v[3] * f);
        *reinterpret_cast<float4 *>(to + 4) = make_float4(v[4] * f, v[5] * f, v[6] * f, v[7] * f);
    };
    if (CL == 1) {
        if (merges && head < nh) store_out(out + (size_t)(h0 + head) * kHD + d0, acc, L > 0.0f ? 1.0f / L : 0.0f);
        return;
    }
    // post the partial, then merge half of the heads each
    cg::cluster_group cl = cg::this_cluster();
    const int rank = static_cast<int>(cl.block_rank());
    float *post = reinterpret_cast<float *>(afrag);  // [heads][128], 8 KB: the fragments have been read
    if (merges) {
        store_out(post + head * kHD + d0, acc, 1.0f);
        if ((tid & 15) == 0) {
            cml[head] = M;
            cml[16 + head] = L;
        }
    }
    cl.sync();
    const int S = gridDim.y / CL;  // partials per head block
    const size_t slot = (size_t)blockIdx.x * S + blockIdx.y / CL;
    if (merges && head / (HB / 2) == rank) {
        const float *po = cl.map_shared_rank(post, rank ^ 1) + head * kHD + d0, *pm = cl.map_shared_rank(cml, rank ^ 1);
        const float4 pa = *reinterpret_cast<const float4 *>(po), pb = *reinterpret_cast<const float4 *>(po + 4);
        const float other[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
        const float Mo = pm[head], Lo = pm[16 + head], Mt = fmaxf(M, Mo);
        const float fa = (M == -INFINITY) ? 0.0f : exp2_fast(M - Mt), fb = (Mo == -INFINITY) ? 0.0f : exp2_fast(Mo - Mt);
        L = L * fa + Lo * fb;
        M = Mt;
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = acc[i] * fa + other[i] * fb;
        if (S == 1) {
            if (head < nh) store_out(out + (size_t)(h0 + head) * kHD + d0, acc, L > 0.0f ? 1.0f / L : 0.0f);
        } else {
            store_out(g_work.part + (slot * 16 + head) * kHD + d0, acc, 1.0f);
            if ((tid & 15) == 0) {
                g_work.ml[(slot * 2 + 0) * 16 + head] = M;
                g_work.ml[(slot * 2 + 1) * 16 + head] = L;
            }
        }
    }
    // This CTA has read the partner's shared memory; it leaves when the partner has read its own.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    auto partner_done = [] { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); };
    if (S == 1) {
        partner_done();
        return;
    }
    __syncthreads();
    if (tid == 0) {  // one release for the CTA: the barrier orders the other threads' stores before it
        int ticket;
        asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(ticket) : "l"(&g_work.tickets[blockIdx.x * 2 + rank]) : "memory");
        is_last = ticket == S - 1;
    }
    __syncthreads();
    if (!is_last) {
        partner_done();
        return;
    }
    // ---- the last CTA of this half of the heads: a warp per head, four dims per thread, kBatch partials' loads in flight ----
    const int mh = HB / 2 * rank + warp;
    if (warp < HB / 2 && mh < nh) {
        const size_t s0 = (size_t)blockIdx.x * S;
        const float *part = g_work.part + (s0 * 16 + mh) * kHD + 4 * lane;
        auto fetch = [&](float4 (&v)[kBatch], int c0) {
#pragma unroll
            for (int u = 0; u < kBatch; u++)
                v[u] = c0 + u < S ? __ldcg(reinterpret_cast<const float4 *>(part + (size_t)(c0 + u) * 16 * kHD)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 v[kBatch];
        fetch(v, 0);
        float *weight = osm + warp * kPitch;  // of the partials (the results have been merged)
        float m[kMaxSlots / 64], l[kMaxSlots / 64], Mt = -INFINITY, Lt = 0.0f;
#pragma unroll
        for (int i = 0; i < kMaxSlots / 64; i++) {
            const int c = lane + 32 * i;
            m[i] = c < S ? __ldcg(g_work.ml + ((s0 + c) * 2) * 16 + mh) : -INFINITY;
            l[i] = c < S ? __ldcg(g_work.ml + ((s0 + c) * 2 + 1) * 16 + mh) : 0.0f;
            Mt = fmaxf(Mt, m[i]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) Mt = fmaxf(Mt, __shfl_xor_sync(0xffffffffu, Mt, o));
#pragma unroll
        for (int i = 0; i < kMaxSlots / 64; i++) {
            const int c = lane + 32 * i;
            const float f = m[i] == -INFINITY ? 0.0f : exp2_fast(m[i] - Mt);
            if (c < S) weight[c] = f;
            Lt = fmaf(l[i], f, Lt);
        }
        Lt = warp_sum(Lt);
        __syncwarp();
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int c0 = 0; c0 < S; c0 += kBatch) {
            if (c0) fetch(v, c0);
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                const float f = c0 + u < S ? weight[c0 + u] : 0.0f;
                o.x = fmaf(v[u].x, f, o.x);
                o.y = fmaf(v[u].y, f, o.y);
                o.z = fmaf(v[u].z, f, o.z);
                o.w = fmaf(v[u].w, f, o.w);
            }
        }
        const float inv = Lt > 0.0f ? 1.0f / Lt : 0.0f;
        *reinterpret_cast<float4 *>(out + (size_t)(h0 + mh) * kHD + 4 * lane) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    }
    if (tid == 0) g_work.tickets[blockIdx.x * 2 + rank] = 0;  // ready for the next launch
    partner_done();
}

constexpr int kRingBytes = kWarps * kStages * kStageBytes, kResultBytes = kWarps * 16 * kPitch * 4;
constexpr int kSmem = 8192 + (2 * kWarps * 16 + 32) * 4 + (kRingBytes > kResultBytes ? kRingBytes : kResultBytes);
static_assert(kSmem <= 227 * 1024, "shared memory budget");

template <int CL, bool FEW>
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
    cudaLaunchKernelEx(&cfg, gqa <= 8 ? attn_int8_kernel<CL, true, FEW> : attn_int8_kernel<CL, false, FEW>, q, k, v, ks, vs, out, n_kv_heads, gqa, seq_len, scale, (tiles + chunks - 1) / chunks);
}

}  // namespace

void attn_int8_init()
{
    static bool done[kMaxDevices] = {false};
    const int dev = current_device();
    if (done[dev]) return;
    for (auto kernel : {attn_int8_kernel<1, false, false>, attn_int8_kernel<1, true, false>, attn_int8_kernel<1, false, true>, attn_int8_kernel<1, true, true>,
                        attn_int8_kernel<2, false, false>, attn_int8_kernel<2, true, false>})
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
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
        auto run = tiles <= kFewTiles ? launch<1, true> : launch<1, false>;
        run(q, k8, v8, ks, vs, out, groups, 1, n_kv_heads, gqa, seq_len, scale, stream);
    } else {
        launch<2, false>(q, k8, v8, ks, vs, out, groups, chunks & ~1, n_kv_heads, gqa, seq_len, scale, stream);
    }
    return true;
}

}  // namespace mb200
