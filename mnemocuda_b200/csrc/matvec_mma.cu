// Q4_K and Q5_K matvecs y = W x on the integer tensor path (mma.sync m16n8k32, u8 x s8 -> s32), for rows of whole super-blocks up to
// 8192 columns; the streaming kernel (stream_matvec.cuh) has the rest.
//
// Arithmetic as there (q4k_policy.cuh): x is split once per CTA into two int8 levels per 32 columns, the dot products of the
// nibbles with both levels are exact integers, and they are scaled in fp32. What differs is who multiplies. An MMA takes 16
// rows x 32 bytes of nibbles; its eight result columns are four sub-blocks x two levels: B holds a sub-block's levels in its
// two columns, at the k of its nibbles, and zeros elsewhere, so four MMAs into the same accumulators leave each lane both
// levels of one sub-block of two rows, which is what it then scales. 16 rows of a super-block take 8 MMAs and 150 other
// instructions, the streaming kernel's dp4a two times 205; the launch's fixed work is smaller too.
//
// What bounds it: in a chain of launches, the way from one y to the next x: of 6.1 us at 8192 x 4096, 0.65 from the end of the
// grid to the next one's wait, 1.3 for x and its levels, 0.5 a stage of 14 rows (a warp's own chain of loads, MMAs and scaling),
// 0.35 for the last sums; the weights arrive meanwhile. So a CTA whose weights fit takes at most half of an SM (113 KB of
// shared memory, 96 registers a thread, at which Q4_K with two super-blocks a warp spills 4 bytes): under programmatic dependent launch the next launch's CTA starts beside it and
// has its weights in shared memory when y is done. Chains of 16 launches against the streaming kernel: 8192 x 4096 8.1 -> 6.1 us,
// 4096 x 4096 6.4 -> 4.1, 6144 x 2048 5.1 -> 3.7, 512 x 2048 3.7 -> 2.7, 50000 x 4096 26.5 -> 20.0 (5.7 TB/s);
// up to 4096 columns no size of 1 to 50000 rows was slower, with or without dependent launches (wider ones: see launch()), and the error
// against 64 bits is the same.
// Up to 4096 columns a warp keeps the levels of its one or two super-blocks in registers with two CTAs on an SM; with three
// or four, up to 8192, a CTA needs the SM's registers for itself and has all of x asked for before it splits any of it (in two rounds one
// after the other 4096 x 8192 took 6.9 us, 512 x 8192 5.0): 4096 x 8192 9.6 -> 6.5 us, 2048 x 6144 6.1 -> 4.5, 512 x 8192 5.4 -> 4.6. With six
// (4096 x 12288: 12.3 us against 12.0) and with levels read again for each stage (1000 x 16384: 8.7 against 8.4) it is no faster.
// Q5_K, with 160 instructions more a unit to put the fifth bits in their places: 8192 x 4096 10.1 -> 8.3 us, 512 x 2048 3.8 -> 2.8,
// 5461 x 2816 6.7 -> 6.2, 30000 x 4096 21.0 -> 18.7.
//
// Stages: whole rows, one bulk copy each (a copy per row costs the requesting warp 60 ns a row); a warp takes 16 rows of one
// to four super-block columns, the last warp requests the stages and adds the columns' sums in ascending order.
#include "q4k_policy.cuh"
#include "tcgen.cuh"

namespace mb200 {
namespace {

constexpr int kWarps = 8, kMvThreads = (kWarps + 1) * 32, kXThreads = kWarps * 32;
constexpr int kXCols = 128 / kWarps;  // columns of x a thread splits: 4096 in a round
constexpr int kMvStages = 6;
constexpr int kMvMaxCols = 4 * kWarps * 256;
constexpr int kHalfSm = 113 * 1024, kWholeSm = 226 * 1024;  // half: (228 KB - 2 x 1 KB) / 2
constexpr int kHalfTiles = 3;        // a CTA with more stages than these takes the whole SM
// x comes in behind whatever weights its SM has asked for before: 97 KB of them cost it 0.7 us. So of a ring in the whole SM
// no more than kAheadBytes are requested before x is here, and the next launch starts when it is (4096 x 4096: 5.1 us with the
// next launch at once, 4.4 so), unless the launch is so small that starting the next one is what takes its time
// (512 x 2048, 4.6 KB a CTA: 2.67 at once, 3.04 with x; 2048 x 1536, 12 KB: 2.68, 2.76; 4096 x 2304, 36 KB: 4.04, 3.99).
constexpr int kAheadBytes = 80 * 1024, kEarlyBytes = 20 * 1024;

// Q4_K and Q5_K: a block's d, dmin and scales, Q5_K's fifth bits, the nibbles
struct T4 {
    static constexpr int kBlock = kQ4KBlock, kQs = 16;
    static constexpr bool kFifth = false;
};
struct T5 {
    static constexpr int kBlock = 176, kQs = 48;
    static constexpr bool kFifth = true;
};

struct MvArgs {
    const uint8_t *w;
    const float *x;
    float *y;
    int per, rem;  // rows / CTAs, rows % CTAs
    int bpr;       // super-blocks of a row
    int cols;      // warps side by side on a row: warp column c takes super-blocks c, c + cols, ...
    int rows;      // rows of a stage, at most 16 per warp of a column
    int stages;
    int ahead;     // stages requested before x is here
    int early;     // 1: the next launch may start at once
    int odd;       // 1: lanes of odd rows start with the other half of a super-block
    int pdl;
    // shared memory: mbarriers, levels of x, scale per sub-block, sums of sub-blocks, sums of a stage [stage][column][row], stages
    int s1, sum, part, stage0, stage_bytes, total;
    int *err;
};
constexpr int kZero = 2 * kMvStages * 8, kX = kZero + 32;  // 16 zero bytes; the levels of x
constexpr int kXBlock = 8 * 64 + 4 * 64;                    // of a super-block: [sub-block][level][32], and those of even sub-blocks negated

__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A lane's share of one row: sub-blocks t and t + 4, with the integers of both levels.
struct XLane {
    float k0, k1, sx0, sx1;  // scale / 254 (Q4_K: an odd sub-block's nibbles count sixteen times: / 16) and sum of x
};
__device__ __forceinline__ float scaled(float sc0, float m0, float sc1, float m1, uint32_t dd, int a0, int b0, int a1, int b1, const XLane &x)
{
    const float2 d = __half22float2(*reinterpret_cast<const __half2 *>(&dd));
    float p = sc0 * (x.k0 * static_cast<float>(a0 * 254 + b0));
    p = fmaf(sc1, x.k1 * static_cast<float>(a1 * 254 + b1), p);
    return fmaf(d.x, p, -d.y * fmaf(m1, x.sx1, m0 * x.sx0));
}
// kXCols columns of x from c0 on -> two int8 levels, v ~= sc * (a + b / 254), where XFrag reads them
template <class T>
__device__ __forceinline__ void split_x(const float (&v)[kXCols], int c0, bool valid, int lane, uint8_t *smem, const MvArgs &P)
{
    constexpr int kLanes = 32 / kXCols;  // of a sub-block
    float amax = fabsf(v[0]), sum = v[0];
#pragma unroll
    for (int i = 1; i < kXCols; i++) {
        amax = fmaxf(amax, fabsf(v[i]));
        sum += v[i];
    }
#pragma unroll
    for (int i = 1; i < kLanes; i *= 2) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, i));
        sum += __shfl_xor_sync(0xffffffffu, sum, i);
    }
    const float sc = amax * (1.0f / 127.0f), inv = amax > 0.0f ? 127.0f / amax : 0.0f;
    uint32_t p1[kXCols / 4], p2[kXCols / 4];
#pragma unroll
    for (int i = 0; i < kXCols / 4; i++) {
        const float q[4] = {v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]};
        stream::split_levels(q, sc, inv, p1[i], p2[i]);
    }
    if (!valid) return;
    const int chunk = c0 >> 5;
    uint8_t *to = smem + kX + (chunk >> 3) * kXBlock + (c0 & 31);
#pragma unroll
    for (int i = 0; i < kXCols / 8; i++) {
        *reinterpret_cast<uint2 *>(to + (chunk & 7) * 64 + 8 * i) = make_uint2(p1[2 * i], p1[2 * i + 1]);
        *reinterpret_cast<uint2 *>(to + (chunk & 7) * 64 + 32 + 8 * i) = make_uint2(p2[2 * i], p2[2 * i + 1]);
        if (!T::kFifth && !(chunk & 1)) {
            *reinterpret_cast<uint2 *>(to + 512 + (chunk & 6) * 32 + 8 * i) = make_uint2(__vneg4(p1[2 * i]), __vneg4(p1[2 * i + 1]));
            *reinterpret_cast<uint2 *>(to + 512 + (chunk & 6) * 32 + 32 + 8 * i) = make_uint2(__vneg4(p2[2 * i]), __vneg4(p2[2 * i + 1]));
        }
    }
    if (lane % kLanes == 0) {
        reinterpret_cast<float *>(smem + P.s1)[chunk] = sc * (!T::kFifth && (chunk & 1) ? 1.0f / (254.0f * 16.0f) : 1.0f / 254.0f);
        reinterpret_cast<float *>(smem + P.sum)[chunk] = sum;
    }
}

// A lane's levels of one super-block: [half][8 bytes of the lane's 16][word]. The lane's k belong to sub-blocks j (low
// nibbles) and j + 1 (high nibbles); only the columns of these sub-blocks' levels hold them.
// Q4_K: low nibbles . x = bytes . x + high nibbles . (-x): one mask a word of weights.
template <class T>
struct XFrag {
    uint4 low[2], high[2];
    XLane l;
    __device__ __forceinline__ void load(const uint8_t *smem, const MvArgs &P, int sb, int g, int t)
    {
        const int j = 2 * (t >> 1), at = kX + sb * kXBlock + (g & 1) * 32 + (t & 1) * 16;
        const bool is_lo = (g >> 1) == j, is_hi = (g >> 1) == j + 1;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            low[h] = *reinterpret_cast<const uint4 *>(smem + (is_lo ? at + (4 * h + j) * 64 : kZero));
            high[h] = *reinterpret_cast<const uint4 *>(smem + (!T::kFifth && is_lo ? at + 512 + (4 * h + j) * 32 : is_hi ? at + (4 * h + j) * 64 + 64 : kZero));
        }
        const float *s1 = reinterpret_cast<const float *>(smem + P.s1) + sb * 8 + t, *xs = reinterpret_cast<const float *>(smem + P.sum) + sb * 8 + t;
        l = {s1[0], s1[4], xs[0], xs[4]};
    }
};

// four nibbles and, from bit i of `bits` on, their fifth bits
__device__ __forceinline__ uint32_t five(uint32_t w, uint32_t bits, int i)
{
    // (a multiplication spreads them: bit k of four goes to bit 8 k + 4)
    const uint32_t m = i & 4 ? ((bits >> (i & 8)) & 0xF0u) * 0x00204081u : ((bits >> (i & 8)) & 0xFu) * 0x02040810u;
    return (w & 0x0F0F0F0Fu) | (m & 0x10101010u);
}

// The lane's part of 16 rows of one super-block: of rows g and g + 8.
template <class T>
__device__ __forceinline__ void dot16(const uint8_t *pa, const uint8_t *pb, int t, bool turned, const XFrag<T> &x, float &va, float &vb)
{
    // 64 bytes of a row over its four lanes; with rows a multiple of 128 bytes apart, the odd ones the other 64 first
    const int o = T::kQs + 16 * t + (turned ? 64 : 0), o1 = T::kQs + 16 * t + (turned ? 0 : 64);
    const uint4 a0 = *reinterpret_cast<const uint4 *>(pa + o), b0 = *reinterpret_cast<const uint4 *>(pb + o);
    const uint4 a1 = *reinterpret_cast<const uint4 *>(pa + o1), b1 = *reinterpret_cast<const uint4 *>(pb + o1);
    const uint4 ha = *reinterpret_cast<const uint4 *>(pa), hb = *reinterpret_cast<const uint4 *>(pb);
    int c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    constexpr uint32_t kHi = 0xF0F0F0F0u;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint4 u = (h == 0) != turned ? a0 : a1, v = (h == 0) != turned ? b0 : b1;
        if (T::kFifth) {
            const uint2 fa = *reinterpret_cast<const uint2 *>(pa + 16 + 16 * h + 8 * (t >> 1)), fb = *reinterpret_cast<const uint2 *>(pb + 16 + 16 * h + 8 * (t >> 1));
            const int sh = 16 * (t & 1);
            const uint32_t al = fa.x >> sh, ah = fa.y >> sh, bl = fb.x >> sh, bh = fb.y >> sh;
            imma(c[h], five(u.x, al, 0), five(v.x, bl, 0), five(u.y, al, 4), five(v.y, bl, 4), x.low[h].x, x.low[h].y);
            imma(c[h], five(u.x >> 4, ah, 0), five(v.x >> 4, bh, 0), five(u.y >> 4, ah, 4), five(v.y >> 4, bh, 4), x.high[h].x, x.high[h].y);
            imma(c[h], five(u.z, al, 8), five(v.z, bl, 8), five(u.w, al, 12), five(v.w, bl, 12), x.low[h].z, x.low[h].w);
            imma(c[h], five(u.z >> 4, ah, 8), five(v.z >> 4, bh, 8), five(u.w >> 4, ah, 12), five(v.w >> 4, bh, 12), x.high[h].z, x.high[h].w);
        } else {
            imma(c[h], u.x, v.x, u.y, v.y, x.low[h].x, x.low[h].y);
            imma(c[h], u.x & kHi, v.x & kHi, u.y & kHi, v.y & kHi, x.high[h].x, x.high[h].y);
            imma(c[h], u.z, v.z, u.w, v.w, x.low[h].z, x.low[h].w);
            imma(c[h], u.z & kHi, v.z & kHi, u.w & kHi, v.w & kHi, x.high[h].z, x.high[h].w);
        }
    }
    // scales and mins of sub-blocks t and t + 4 of both rows side by side: [scale, min] of row g, [scale, min] of row g + 8
    const uint32_t q = __byte_perm(__byte_perm(ha.y, ha.z, 0x40 + 0x11 * t), __byte_perm(hb.y, hb.z, 0x40 + 0x11 * t), 0x5410);
    const uint32_t w = __byte_perm(ha.w, hb.w, 0x4400 + 0x1111 * t);
    const uint32_t s0 = q & 0x3F3F3F3Fu, s1 = ((q >> 2) & 0x30303030u) | (__byte_perm(w, w >> 4, 0x7250) & 0x0F0F0F0Fu);
    va = scaled(byte_float(s0, 0), byte_float(s0, 1), byte_float(s1, 0), byte_float(s1, 1), ha.x, c[0][0], c[0][1], c[1][0], c[1][1], x.l);
    vb = scaled(byte_float(s0, 2), byte_float(s0, 3), byte_float(s1, 2), byte_float(s1, 3), hb.x, c[0][2], c[0][3], c[1][2], c[1][3], x.l);
}

// NB: super-blocks a warp takes side by side
template <class T, int NB>
__global__ void __launch_bounds__(kMvThreads, NB <= 2 ? 2 : 1) matvec_mma_kernel(const __grid_constant__ MvArgs P)
{
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + kMvStages;
    float *part = reinterpret_cast<float *>(smem + P.part);
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int cta = blockIdx.x;
    const int first = cta * P.per + min(cta, P.rem), n_rows = P.per + (cta < P.rem ? 1 : 0);
    const int S = P.stages, pitch = P.bpr * T::kBlock;

    if (warp == kWarps) {
        // ---- requests the stages, adds up their sums ----
        const uint32_t row_bytes = P.bpr * T::kBlock;
        const uint8_t *w = P.w + (size_t)first * row_bytes;
        const bool leader = elect_lane();
        int req = 0;  // rows requested
        auto request = [&](int slot) {
            const int rows = min(P.rows, n_rows - req);
            if (leader) {
                mbar_expect_tx(&full[slot], rows * row_bytes);
                bulk_g2s(smem + P.stage0 + slot * P.stage_bytes, w + (size_t)req * row_bytes, rows * row_bytes, &full[slot]);
            }
            req += rows;
        };
        if (leader) {  // the lane that arrives on the barriers below, before the CTA's first barrier
            *reinterpret_cast<uint4 *>(smem + kZero) = make_uint4(0u, 0u, 0u, 0u);
            for (int s = 0; s < S; s++) {
                mbar_init(&full[s], 1);
                mbar_init(&empty[s], kWarps);
            }
            mbar_fence_init();
        }
        if (P.pdl && P.early) stream::grid_dep_launch();
        for (int s = 0; s < P.ahead && req < n_rows; s++) request(s);
        __syncthreads();
        for (int s = P.ahead; s < S && req < n_rows; s++) request(s);
        if (P.pdl) stream::grid_dep_wait();  // y may still be in use by the upstream kernel
        int slot = 0, phase = 0;
        for (int row = 0; row < n_rows; row += P.rows) {
            const int rows = min(P.rows, n_rows - row);
            if (!mbar_wait(&empty[slot], phase)) {  // (a warp whose wait ran out has left: this one runs out too)
                if (lane == 0) atomicExch(P.err, MB200_ERR_TIMEOUT);
                return;
            }
            const float *pt = part + slot * P.cols * P.rows;
            float *y = P.y + first + row;
            for (int r = lane; r < rows; r += 32) {
                float v = 0.0f;
#pragma unroll 4
                for (int c = 0; c < P.cols; c++) v += pt[c * P.rows + r];
                y[r] = v;
            }
            __syncwarp();
            if (req < n_rows) request(slot);
            if (++slot == S) {
                slot = 0;
                phase ^= 1;
            }
        }
        return;
    }

    // ---- the levels of x ----
    if (P.pdl) {
        // x may be cold; asked for here, it waits in the L2 for the upstream kernel's end
        for (int c = threadIdx.x * 32; c < P.bpr * 256; c += kXThreads * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(P.x + c));
        stream::grid_dep_wait();  // x is produced by the upstream kernel
    }
    {
        const int K = P.bpr * 256;
        const bool vec_ok = (reinterpret_cast<uintptr_t>(P.x) & 15) == 0;
        constexpr int kRounds = NB <= 2 ? 1 : 2, kRound = kXThreads * kXCols;  // all of x is asked for before any of it is split
        const int c0 = threadIdx.x * kXCols;
        float v[kRounds][kXCols];
#pragma unroll
        for (int n = 0; n < kRounds; n++) {
            const float *from = P.x + n * kRound + c0;
#pragma unroll
            for (int i = 0; i < kXCols; i += 4) {
                float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (n * kRound + c0 < K) {
                    if (vec_ok)
                        q = __ldcg(reinterpret_cast<const float4 *>(from + i));
                    else
                        q = make_float4(__ldcg(from + i), __ldcg(from + i + 1), __ldcg(from + i + 2), __ldcg(from + i + 3));
                }
                v[n][i] = q.x, v[n][i + 1] = q.y, v[n][i + 2] = q.z, v[n][i + 3] = q.w;
            }
        }
        // (reads x: not before it has arrived)
        if (P.pdl && !P.early && c0 < K && __float_as_uint(v[0][0]) != 0x7fc12345u) stream::grid_dep_launch();
#pragma unroll
        for (int n = 0; n < kRounds; n++)
            if (n * kRound + c0 - lane * kXCols < K) split_x<T>(v[n], n * kRound + c0, n * kRound + c0 < K, lane, smem, P);
    }
    __syncthreads();

    // ---- products ----
    const int g = lane >> 2, t = lane & 3;
    int col = warp, tile = 0;  // the warp's column and its first row of a stage
    while (col >= P.cols) {
        col -= P.cols;
        tile += 16;
    }
    const bool turned = P.odd & g & 1;
    const bool all = col + (NB - 1) * P.cols < P.bpr;
    XFrag<T> x[NB];
    int at[NB];  // the warp's super-blocks in a row; a row's last ones may not go round
#pragma unroll
    for (int n = 0; n < NB; n++) {
        const int sb = min(col + n * P.cols, P.bpr - 1);
        x[n].load(smem, P, sb, g, t);
        at[n] = sb * T::kBlock;
    }
    int slot = 0, phase = 0;
    for (int row = 0; row < n_rows; row += P.rows) {
        const int left = min(P.rows, n_rows - row) - tile;  // rows from the warp's first on
        if (!mbar_wait(&full[slot], phase)) return;
        if (left > 0) {
            const uint8_t *st = smem + P.stage0 + slot * P.stage_bytes + tile * pitch;
            const uint8_t *ra = st + min(g, left - 1) * pitch, *rb = st + min(g + 8, left - 1) * pitch;
            float va[NB], vb[NB];
#pragma unroll
            for (int n = 0; n < NB; n++) dot16<T>(ra + at[n], rb + at[n], t, turned, x[n], va[n], vb[n]);
#pragma unroll
            for (int n = 1; n < NB; n++)
                if (n + 1 < NB || all) {
                    va[0] += va[n];
                    vb[0] += vb[n];
                }
            // sub-blocks of a row over four lanes: even lanes go on with row g, odd lanes with row g + 8
            float v = ((t & 1) ? vb[0] : va[0]) + __shfl_xor_sync(0xffffffffu, (t & 1) ? va[0] : vb[0], 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            const int r = tile + g + 8 * t;
            if (t < 2 && r < P.rows) part[(slot * P.cols + col) * P.rows + r] = v;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == S) {
            slot = 0;
            phase ^= 1;
        }
    }
}

// The shared memory of `stages` stages of `rows` rows of `row_bytes`
int fit(MvArgs &P, int row_bytes, int rows, int stages)
{
    P.rows = rows;
    P.stages = stages;
    P.s1 = kX + P.bpr * kXBlock;
    P.sum = P.s1 + P.bpr * 32;
    P.part = P.sum + P.bpr * 32;
    P.stage0 = (P.part + stages * P.cols * rows * 4 + 127) & ~127;
    P.stage_bytes = rows * row_bytes;
    P.total = P.stage0 + stages * P.stage_bytes;
    return P.total;
}

template <class T>
void init()
{
    cudaFuncSetAttribute(matvec_mma_kernel<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
    cudaFuncSetAttribute(matvec_mma_kernel<T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
    cudaFuncSetAttribute(matvec_mma_kernel<T, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
    cudaFuncSetAttribute(matvec_mma_kernel<T, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
}

}  // namespace

void matvec_mma_init()
{
    static bool done[kMaxDevices] = {false};
    const int dev = current_device();
    if (done[dev]) return;
    init<T4>();
    init<T5>();
    done[dev] = true;
}

namespace {

template <class T>
bool launch(const void *weights, const float *x, float *y, int n_rows, int n_cols, cudaStream_t stream, const char *where)
{
    if (n_rows < 1 || n_cols < 256 || n_cols % 256 || n_cols > kMvMaxCols || (reinterpret_cast<uintptr_t>(weights) & 15)) return false;
    // By columns alone: the streaming kernel adds in another order, and a row's bits must not depend on how many rows the call has (a
    // tensor split by rows over ranks gives what the whole one gives). Q4_K is faster here at every width for 700 rows or more and for fewer
    // no slower but at 4352 columns (512 rows: 4.04 us against 3.93). Q5_K is slower at 4352 and 4608 columns (4.57 against 4.23, 20000
    // rows 18.0 either way), where the streaming kernel splits x in one round; beyond it is 1.2 to 1.45 times as fast at 1024 to 4096 rows and,
    // from 6400 columns on, up to 0.5 us slower below 300.
    if (T::kFifth && n_cols > 2 * kWarps * 256 && n_cols <= 4608) return false;
    matvec_mma_init();
    MvArgs P{};
    P.w = static_cast<const uint8_t *>(weights);
    P.x = x;
    P.y = y;
    P.bpr = n_cols / 256;
    const int nb = P.bpr <= kWarps ? 1 : P.bpr <= 2 * kWarps ? 2 : P.bpr <= 3 * kWarps ? 3 : 4;
    P.cols = (P.bpr + nb - 1) / nb;
    const int row_bytes = P.bpr * T::kBlock;
    P.odd = row_bytes % 128 == 0;
    const int sms = device_sms(), grid = n_rows < sms ? n_rows : sms;
    P.per = n_rows / grid;
    P.rem = n_rows % grid;
    // As few stages of the same size as fit: all of them in half an SM, or a ring in the whole of it. (8192 x 4096, 56 rows a
    // CTA: 7.0 us with three of four stages in half an SM, where the fourth comes behind the next launch's; 6.1 in the whole.)
    const int rows = P.per + (P.rem ? 1 : 0), most = kWarps / P.cols * 16, tiles = (rows + most - 1) / most;
    if (nb > 2 || tiles > kHalfTiles || fit(P, row_bytes, (rows + tiles - 1) / tiles, tiles) > kHalfSm) {
        int s = kMvStages;
        while (s > 3 && fit(P, row_bytes, most, s) > kWholeSm) s--;
        for (int n = tiles; fit(P, row_bytes, (rows + n - 1) / n, n < s ? n : s) > kWholeSm;) n++;
    }
    P.ahead = P.total <= kHalfSm ? P.stages : P.stage_bytes > kAheadBytes ? 1 : kAheadBytes / P.stage_bytes;
    P.early = rows * row_bytes <= kEarlyBytes;
    P.pdl = stream::pdl_mode();
    P.err = device_error_word();

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kMvThreads);
    cfg.dynamicSmemBytes = P.total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = P.pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, nb == 1 ? matvec_mma_kernel<T, 1> : nb == 2 ? matvec_mma_kernel<T, 2> : nb == 3 ? matvec_mma_kernel<T, 3> : matvec_mma_kernel<T, 4>, P);
    MB200_CHECK_LAUNCH(where);
    return true;
}

}  // namespace

bool matvec_q4k_mma(const void *weights, const float *x, float *y, int n_rows, int n_cols, cudaStream_t stream, const char *where)
{
    return launch<T4>(weights, x, y, n_rows, n_cols, stream, where);
}
bool matvec_q5k_mma(const void *weights, const float *x, float *y, int n_rows, int n_cols, cudaStream_t stream, const char *where)
{
    return launch<T5>(weights, x, y, n_rows, n_cols, stream, where);
}

}  // namespace mb200
