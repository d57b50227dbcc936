// Weights -> pairs of fp16 (hi, lo) for the tensor cores, in packed fp16 arithmetic.
//
// A Q4_K weight is w = s * n - b with n a small integer and s = d * scale, b = dmin * min of the sub-block. With a unit u, a
// power of two chosen per sub-block so that no |w| of it exceeds 2048 u, s1 = s and b1 = b rounded to multiples of u make
// hi = s1 * n - b1 an integer multiple of u of at most 11 bits: one HFMA2 computes it EXACTLY for two weights.
// lo = (s - s1) * n - (b - b1), the rest, is at most 8 u and is rounded to fp16 once. A Q6_K weight is w = s * (q - 32), s of 18
// bits: with s = s1 + s2 in fp16 halves, hi is the rounded product with s1, and lo what that rounding left (one HFMA2, exact) plus
// the product with s2, rounded once. Converting an fp32 weight, converting back, subtracting and converting the remainder took ten
// instructions per two weights (the producers of the grouped GEMM were issue-bound on exactly that); these are three and four.
// Error of hi + lo, root mean square over the weights of synthetic blocks: Q4_K 7e-7, Q6_K 2e-8 of the weights' (a second half
// rounded from fp32: 1e-8 and 0). Results against fp64, six shapes from 1024 x 256 to 4096 x 1536, are as far off as with that,
// 0.6 to 2.3e-5: fp32 accumulation decides. (A Q4_K lo from operands 16 + n, one instruction less, has 1.3e-6, a Q6_K lo from a
// rounded s alike; results at 1024 x 256 were then 10 % further off. The exact ones cost 3 % of the time.)
//
// What is left is getting n out of the packed bits, on the integer pipe, which has half the FMA pipe's rate. A nibble shifted
// to bits 6..9 of a 16-bit half and OR-ed with 0x4C00 is 16 + n: one shift and one LOP3 for two weights, no byte permute and
// no subtraction, because the 16 goes into the addend exactly (16 s1 + b1 is a multiple of u below 2^11 u as well). The two
// weights are then bytes 0 and 2 (1 and 3) of a word: inside every four columns the order is 0, 2, 1, 3, and the
// activations are laid out the same way (k_order).
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace mb200 {

__device__ __forceinline__ uint32_t dup_half(float v)
{
    const __half2 h = __float2half2_rn(v);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b)
{
    const __half2 r = __hadd2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b)
{
    const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c)
{
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b),
                              *reinterpret_cast<const __half2 *>(&c));
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t hfms2(uint32_t a, uint32_t b, uint32_t c)  // a b - c
{
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b),
                              __hneg2(*reinterpret_cast<const __half2 *>(&c)));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// 1.5 * 2^23 * u with u = 2^(exponent of t - DROP): adding and subtracting it rounds to a multiple of u
template <int DROP>
__device__ __forceinline__ float round_magic(float t)
{
    return __uint_as_float((__float_as_uint(t) & 0x7F800000u) + (static_cast<uint32_t>(23 - DROP) << 23) + 0x00400000u);
}

// Position of column k in the operand layout: columns 1 and 2 of every four change places.
__host__ __device__ constexpr int k_order(int k) { return (k & ~3) | ((k & 1) << 1) | ((k >> 1) & 1); }

// d * v for an integer v of at most 23 bits: v in the mantissa of 2^23, one FMA (c = -2^23 d) instead of a conversion
__device__ __forceinline__ float mul_small(float d, float c, uint32_t v) { return fmaf(d, __uint_as_float(0x4B000000u | v), c); }

// One Q4_K sub-block's scale and min as the packed factors of hi and lo for operands 16 + n.
struct SplitQ4 {
    uint32_t s1, c1, rs, cr;
    __device__ __forceinline__ void set(float s, float b)
    {
        // 16 |s1| + |b1| <= 2^11 u, so that it is an fp16 number too: 16 |s| + |b| stays 1/128 below, which is more than the 8.5 u
        // that rounding may add
        const float M = round_magic<10>(fmaf(16.0f, fabsf(s), fabsf(b)) * 1.0078125f);
        const float s1f = (s + M) - M, b1f = (b + M) - M, rsf = s - s1f;
        s1 = dup_half(s1f);
        rs = dup_half(rsf);
        c1 = dup_half(fmaf(-16.0f, s1f, -b1f));
        cr = dup_half(b1f - b);
    }
};
// 32 weights whose nibbles are the low (HIGH = false) or high nibbles of 8 words, two per register in k_order
template <bool HIGH>
__device__ __forceinline__ void split_q4(const uint32_t (&w)[8], const SplitQ4 &f, uint32_t (&hi)[16], uint32_t (&lo)[16])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t v0 = ((HIGH ? w[i] << 2 : w[i] << 6) & 0x03C003C0u) | 0x4C004C00u;
        const uint32_t v1 = ((HIGH ? w[i] >> 6 : w[i] >> 2) & 0x03C003C0u) | 0x4C004C00u;
        hi[2 * i] = hfma2(v0, f.s1, f.c1);
        lo[2 * i] = hfma2(hadd2(v0, 0xCC00CC00u), f.rs, f.cr);  // - 16
        hi[2 * i + 1] = hfma2(v1, f.s1, f.c1);
        lo[2 * i + 1] = hfma2(hadd2(v1, 0xCC00CC00u), f.rs, f.cr);
    }
}

struct SplitQ6 {
    uint32_t s1, rs;
    __device__ __forceinline__ void set(float s)
    {
        s1 = dup_half(s);
        rs = dup_half(s - __half2float(__ushort_as_half(static_cast<unsigned short>(s1))));  // exact: s has 18 bits
    }
};
// 32 weights q - 32: q = the nibble of `l` at bit 4 (LHI = false: at bit 0) | two bits of `h` at bit HB, << 4, of each byte.
// q goes to bits 4..9 of a half: 64 + q. The first 16 weights have scale f[0], the others f[1].
template <bool LHI, int HB>
__device__ __forceinline__ void split_q6(const uint32_t *l, const uint32_t *h, const SplitQ6 (&f)[2], uint32_t (&hi)[16],
                                         uint32_t (&lo)[16])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t h0 = ((h[i] << (8 - HB)) & 0x03000300u) | 0x54005400u, h1 = ((h[i] >> HB) & 0x03000300u) | 0x54005400u;
        const uint32_t q0 = ((LHI ? l[i] : l[i] << 4) & 0x00F000F0u) | h0, q1 = ((LHI ? l[i] >> 8 : l[i] >> 4) & 0x00F000F0u) | h1;
        const uint32_t v0 = hadd2(q0, 0xD600D600u), v1 = hadd2(q1, 0xD600D600u);  // - 96
        hi[2 * i] = hmul2(v0, f[i >> 2].s1);
        lo[2 * i] = hfma2(v0, f[i >> 2].rs, hfms2(v0, f[i >> 2].s1, hi[2 * i]));
        hi[2 * i + 1] = hmul2(v1, f[i >> 2].s1);
        lo[2 * i + 1] = hfma2(v1, f[i >> 2].rs, hfms2(v1, f[i >> 2].s1, hi[2 * i + 1]));
    }
}

// ---- Q6_K blocks in shared memory ----
// A block is 210 bytes at a 2-byte alignment: no tensor map fits it and 16-byte copies would have to carry up to 14 bytes of
// skew. A warp copies the 53 aligned words that hold it (two words per lane; the last word's spare bytes share it with valid
// ones); a row's thread then reads its words, which start 0 or 2 bytes into the first (`skew`).
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src)  // 4 bytes, shared <- global, both 4-byte aligned
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar)  // one arrival when this thread's copies so far have landed
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void copy_q6k_row(uint32_t dst_lane, const uint8_t *blk, int lane)  // dst_lane: the row's slot + 4 lane
{
    const uint8_t *a = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(blk) & ~static_cast<uintptr_t>(3)) + 4 * lane;
    cp_async4(dst_lane, a);
    if (lane < 53 - 32) cp_async4(dst_lane + 128, a + 128);
}
struct RawQ6 {  // half a block: 128 weights
    uint32_t ql[16], qh[8], sc[2];
    float d;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t skew, int half)
    {
        const uint32_t sel = skew ? 0x5432u : 0x3210u;
        const uint32_t *wp = reinterpret_cast<const uint32_t *>(row);
        uint32_t prev = wp[16 * half];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t nx = wp[16 * half + i + 1];
            ql[i] = __byte_perm(prev, nx, sel);
            prev = nx;
        }
        prev = wp[32 + 8 * half];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t nx = wp[32 + 8 * half + i + 1];
            qh[i] = __byte_perm(prev, nx, sel);
            prev = nx;
        }
        const uint32_t a = wp[48 + 2 * half], b = wp[49 + 2 * half], c = wp[50 + 2 * half];
        sc[0] = __byte_perm(a, b, sel);
        sc[1] = __byte_perm(b, c, sel);
        d = __half2float(__ushort_as_half(static_cast<unsigned short>(skew ? wp[52] >> 16 : wp[52])));
    }
};

}  // namespace mb200
