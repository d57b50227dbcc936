// Weights -> small integers in fp16 for the tensor cores, in packed fp16 arithmetic.
//
// A Q4_K weight is d * (scale * n) - dmin * min, a Q6_K weight d * (scale * (q - 32)): apart from d and dmin, which belong to a whole
// super-block of a row, integers. scale * n is at most 945 and exact in fp16; scale * (q - 32) has 12 bits and a sign and is hi, the
// rounded product, plus lo, what that left (-1, 0 or 1). The grouped GEMM multiplies these and applies d and dmin to its sums, so
// no weight is ever rounded.
//
// A field of at most 10 bits, masked out of a 16-bit half, IS an fp16 number: a subnormal, n * 2^-24, or 2^4 times that for a field
// that starts at bit 4. So a nibble needs one AND -- the low ones of bytes 0, 2, the high ones of bytes 0, 2, both again after one
// shift by 8 for bytes 1, 3 -- and one HMUL2 by 16 * scale or scale gives scale * n * 2^-20: nine instructions for eight weights, where
// fp16 halves of the scaled weight took twenty (its unit per sub-block, operands 16 + n, two FMAs, a subtraction). The two bits of a
// Q6_K weight are shifted beside its nibble and OR-ed in (11 integer instructions for eight weights, on the pipe that has half the
// FMA pipe's rate), 32 is subtracted, and a product and an FMA give hi and lo.
//
// The two weights of a register are bytes 0 and 2 (1 and 3) of a word: inside every four columns the order is 0, 2, 1, 3, and the
// activations are laid out the same way (k_order).
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace mb200 {

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
__device__ __forceinline__ uint32_t hfms2(uint32_t a, uint32_t b, uint32_t c)  // a b - c
{
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b),
                              __hneg2(*reinterpret_cast<const __half2 *>(&c)));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// Position of column k in the operand layout: columns 1 and 2 of every four change places.
__host__ __device__ constexpr int k_order(int k) { return (k & ~3) | ((k & 1) << 1) | ((k >> 1) & 1); }

constexpr float kIntScale = 1048576.0f;  // 2^20: what an operand of the integer forms has to be multiplied by

// The two scales of a 64-column group (sc2: two bytes, the low nibbles' first) as factors of their masked nibbles.
struct ScaleQ4 {
    uint32_t lo, hi;
    __device__ __forceinline__ explicit ScaleQ4(uint32_t sc2)
    {
        const uint32_t s = hmul2(__byte_perm(sc2, 0u, 0x4140), 0x74007400u);  // sc 2^-24 -> 2^-10
        const uint32_t t = hmul2(s, 0x64007400u);                             // 2^4 sc (low nibbles), sc
        lo = __byte_perm(t, 0u, 0x1010);
        hi = __byte_perm(t, 0u, 0x3232);
    }
};
// 32 + 32 weights scale * n * 2^-20, of the low and of the high nibbles of 8 words, two per register in k_order
__device__ __forceinline__ void int_q4(const uint32_t (&w)[8], const ScaleQ4 &f, uint32_t (&lo)[16], uint32_t (&hi)[16])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t v = w[i] >> 8;
        lo[2 * i] = hmul2(w[i] & 0x000F000Fu, f.lo);
        lo[2 * i + 1] = hmul2(v & 0x000F000Fu, f.lo);
        hi[2 * i] = hmul2(w[i] & 0x00F000F0u, f.hi);
        hi[2 * i + 1] = hmul2(v & 0x00F000F0u, f.hi);
    }
}

// ---- Q6_K blocks in shared memory ----
// A block is 210 bytes at a 2-byte alignment. Groups of rows make a tensor map (encode_q6k_groups); where the address or the number of
// rows rules that out, a warp copies the 53 aligned words that hold it (two words per lane; the last word's spare bytes share it with valid
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
// N words of a row that may begin two bytes into the first (HALF, half = 2)
template <bool HALF, int N>
__device__ __forceinline__ void q6k_words(const uint32_t *p, int half, uint32_t (&v)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = p[i];
    if (HALF) {
        const uint32_t last = p[N], sel = half ? 0x5432u : 0x3210u;
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = __byte_perm(v[i], i < N - 1 ? v[i + 1] : last, sel);
    }
}
struct RawQ6 {  // half a block: 128 weights
    uint32_t ql[16], qh[8], sc[2];
    float d;
    template <bool HALF>
    __device__ __forceinline__ void load(const uint8_t *row, int half, int h)
    {
        const uint32_t *wp = reinterpret_cast<const uint32_t *>(row);
        q6k_words<HALF>(wp + 16 * h, half, ql);
        q6k_words<HALF>(wp + 32 + 8 * h, half, qh);
        q6k_words<HALF>(wp + 48 + 2 * h, half, sc);
        d = __half2float(__ushort_as_half(static_cast<unsigned short>(half ? wp[52] >> 16 : wp[52])));
    }
};
// A quarter of a block, from a slot of shared memory in which the block begins `skew` bytes (even, below 16) from the start: 32 bytes
// of ql and the qh bytes of the same half. Quarter u covers columns 128 (u / 2) + 32 (u % 2) + {0..31},
// from the low nibbles, and 64 more, from the high ones.
struct QuarterQ6 {
    uint32_t ql[8], qh[8], sc[2];  // sc: the two scales of the low nibbles (bytes 0, 1), of the high ones
    float d;
    template <bool HALF>
    __device__ __forceinline__ void load(const uint8_t *row, int half, int u)
    {
        const uint32_t *wp = reinterpret_cast<const uint32_t *>(row);
        const uint32_t sel = half ? 0x5432u : 0x3210u;
        q6k_words<HALF>(wp + 8 * u, half, ql);
        q6k_words<HALF>(wp + 32 + 8 * (u >> 1), half, qh);
        const uint32_t a = wp[48 + 2 * (u >> 1)], b = wp[49 + 2 * (u >> 1)], c = HALF ? wp[50 + 2 * (u >> 1)] : 0u;
        const uint32_t sel2 = sel >> (u & 1 ? 8 : 0);  // bytes 2, 3 for the odd quarters
        sc[0] = __byte_perm(a, b, sel2);
        sc[1] = __byte_perm(b, c, sel2);
        d = __half2float(__ushort_as_half(static_cast<unsigned short>(half ? wp[52] >> 16 : wp[52])));
    }
};
// 16 + 16 weights of a quarter, from words 4 `part` .. + 3: scale * (q - 32) * 2^-20, eight registers of hi halves and eight of lo ones, of
// the low nibbles (`low`) and the high ones (`high`)
__device__ __forceinline__ void int_q6(const QuarterQ6 &raw, int part, int odd, uint32_t (&low)[16], uint32_t (&high)[16])
{
    // int8 + 128 in the low bits of 1024; minus 1152; the low nibbles' times 2^4, which the high ones carry
    auto scale = [&](uint32_t sc) { return hadd2(__byte_perm(sc ^ 0x8080u, 0x64646464u, part ? 0x4141 : 0x4040), 0xE480E480u); };
    const uint32_t fl = hmul2(scale(raw.sc[0]), 0x4C004C00u), fh = scale(raw.sc[1]);
    const int left = 4 - 2 * odd, right = 4 + 2 * odd;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w0 = raw.ql[4 * part + i], w1 = w0 >> 8, h0 = raw.qh[4 * part + i] << left, h1 = raw.qh[4 * part + i] >> right;
        const uint32_t a0 = hadd2((w0 & 0x000F000Fu) | (h0 & 0x00300030u), 0x80208020u);
        const uint32_t a1 = hadd2((w1 & 0x000F000Fu) | (h1 & 0x00300030u), 0x80208020u);
        const uint32_t b0 = hadd2((w0 & 0x00F000F0u) | (h0 & 0x03000300u), 0x82008200u);
        const uint32_t b1 = hadd2((w1 & 0x00F000F0u) | (h1 & 0x03000300u), 0x82008200u);
        low[2 * i] = hmul2(a0, fl);
        low[2 * i + 1] = hmul2(a1, fl);
        high[2 * i] = hmul2(b0, fh);
        high[2 * i + 1] = hmul2(b1, fh);
        low[8 + 2 * i] = hfms2(a0, fl, low[2 * i]);
        low[8 + 2 * i + 1] = hfms2(a1, fl, low[2 * i + 1]);
        high[8 + 2 * i] = hfms2(b0, fh, high[2 * i]);
        high[8 + 2 * i + 1] = hfms2(b1, fh, high[2 * i + 1]);
    }
}

// ---- weights rounded to fp16 once (the dense GEMM, whose accumulators run through all of K) ----
// scale * n and scale * q - 32 scale are exact in fp32 out of one FMA whose factors are fp16 (Blackwell's mixed-precision FMA runs at the
// rate of the fp32 one), d and the min follow in fp32, then one rounding. The masked fields are fp16 numbers as they are (above), so a
// weight costs the integer pipe 1.1 instructions instead of the 1.9 of bytes permuted into fp32 mantissas; that pipe has half the
// rate (Q4_K 512 x 512 x 8192 in tiles of 128: 30.2 instead of 33.4 us).

// a * b + c, a and b the low or high halves of their registers
template <bool AH, bool BH>
__device__ __forceinline__ float mixed_fma(uint32_t a, uint32_t b, float c)
{
    float r;
    const unsigned short x = static_cast<unsigned short>(AH ? a >> 16 : a), y = static_cast<unsigned short>(BH ? b >> 16 : b);
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(r) : "h"(x), "h"(y), "f"(c));
    return r;
}
// (a, b) * (f, f) + (c, c)
__device__ __forceinline__ void fma_pair(float &a, float &b, float f, float c)
{
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmov.b64 z, {%3, %3};\n\t"
        "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a), "+f"(b)
        : "f"(f), "f"(c));
}
__device__ __forceinline__ uint32_t pack_halves(float lo, float hi)
{
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// two bytes of up to 10 bits each as fp16 numbers
__device__ __forceinline__ uint32_t small_half2(uint32_t two_bytes)
{
    return hadd2(__byte_perm(two_bytes, 0x64646464u, 0x4140), 0xE400E400u);  // 1024 + v - 1024
}
// 32 weights d * sc * n + c (sc in the low half), n the low or high nibbles of 8 words, in column order
template <bool HIGH>
__device__ __forceinline__ void round_q4(const uint32_t (&w)[8], uint32_t sc, float d, float c, uint32_t (&o)[16])
{
    constexpr uint32_t mask = HIGH ? 0x00F000F0u : 0x000F000Fu;
    const float f = d * (HIGH ? 1048576.0f : 16777216.0f);  // a masked nibble is n 2^-20 or n 2^-24
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t even = w[i] & mask, odd = (w[i] >> 8) & mask;
        float v[4] = {mixed_fma<false, false>(even, sc, 0.0f), mixed_fma<false, false>(odd, sc, 0.0f),
                      mixed_fma<true, false>(even, sc, 0.0f), mixed_fma<true, false>(odd, sc, 0.0f)};
        fma_pair(v[0], v[1], f, c);
        fma_pair(v[2], v[3], f, c);
        o[2 * i] = pack_halves(v[0], v[1]);
        o[2 * i + 1] = pack_halves(v[2], v[3]);
    }
}
// 32 weights d * sc * (q - 32) of half a block, thirty-two-group 2 c + h. Here a byte permuted into the mantissa of 2.0f (v = 2 + q / 64) and
// one FMA per weight, s (q - 32) = 64 s v - 160 s, take less: the exact integers above have 12 bits, a second multiplication, and do not
// share their shifts between the nibbles as the grouped GEMM's do (Q6_K 512 x 512 x 8192: 34.3 instead of 30.5 us in tiles of 64).
__device__ __forceinline__ void round_q6(const RawQ6 &raw, int c, int h, uint32_t (&o)[16])
{
    float a[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float s = raw.d * static_cast<float>(static_cast<int8_t>(raw.sc[c] >> (16 * h + 8 * i)));
        a[i] = 64.0f * s;
        b[i] = -160.0f * s;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t l = c ? raw.ql[8 * h + i] >> 4 : raw.ql[8 * h + i];
        const uint32_t hb = c == 0 ? (h == 0 ? raw.qh[i] << 4 : raw.qh[i] << 2) : (h == 0 ? raw.qh[i] : raw.qh[i] >> 2);
        const uint32_t n = (l & 0x0F0F0F0Fu) | (hb & 0x30303030u);
        const float s = a[i >> 2], m = b[i >> 2];
        o[2 * i] = pack_halves(fmaf(s, __uint_as_float(__byte_perm(n, 0x40000000u, 0x7044)), m), fmaf(s, __uint_as_float(__byte_perm(n, 0x40000000u, 0x7144)), m));
        o[2 * i + 1] = pack_halves(fmaf(s, __uint_as_float(__byte_perm(n, 0x40000000u, 0x7244)), m), fmaf(s, __uint_as_float(__byte_perm(n, 0x40000000u, 0x7344)), m));
    }
}

}  // namespace mb200
