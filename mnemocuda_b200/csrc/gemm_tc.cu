// Prefill GEMM on 5th-generation tensor cores (tcgen05 + TMEM), sm_100a:
//     out[t][n] = sum_k  f16(X[t][k]) * dequant(W)[n][k]        X: fp16 [M x K], W: Q4_K or Q6_K [N x K], out: fp32 [M x N]
//
// The reference's "tensor-core GEMM" (src/gemm_q4k.cu:201-266) is an int8 mma.sync experiment that
// quantises activations to Q8_1 and is only ever run at batch 1; its numerics are not validated.
// The semantics implemented here are the ones the reference's dequant defines: fp32 dequant(W),
// fp16 activations, fp32 accumulation (W rounded to fp16 for the tensor core: 2.8e-4 relative L2).
//
// Mapping. The weight rows are the UMMA M dimension (128 rows per CTA), the tokens the UMMA N
// dimension (256 per CTA), K is walked in chunks of 64 (one 128-byte swizzle row of fp16):
//   D[n (128 TMEM lanes)][t (256 TMEM columns)] += A[n][k] * B[t][k]
//   * B (activations) arrives by TMA (cp.async.bulk.tensor.2d, 128-byte swizzle, no multicast);
//   * A (weights) is produced in the kernel: two groups of 8 warps (even / odd K chunks, so one
//     group's latency hides behind the other's) read the raw GGUF blocks from global memory,
//     rebuild w = d*sc*q - dmin*m (Q4_K) / d*sc*(q-32) (Q6_K) in fp32, round to fp16 and store
//     the tile in the same K-major 128-byte-swizzled layout TMA would have produced;
//   * one elected thread issues tcgen05.mma (kind::f16, M128 N256 K16), accumulators live in
//     TMEM (256 columns), tcgen05.commit signals the stage free / the accumulator complete;
//   * the 16 producer warps read the accumulator back with tcgen05.ld and store out[t][n]
//     (coalesced over n).
// 4-stage ring (48 KB per stage); every mbarrier wait is bounded; TMEM is always released.
#include <cstdio>

#include "tcgen.cuh"

namespace mb200 {

EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

namespace {

constexpr int kBN = 128;   // weight rows per CTA (UMMA M)
// tokens per CTA (UMMA N) is a template parameter BT: 256 for the dense GEMM, 64 for the grouped
// per-expert form (about 32 tokens per expert in the benchmark's routing)
constexpr int kBK = 64;    // K per stage: 64 fp16 = one 128-byte swizzle row
constexpr int kDequantWarps = 16;
constexpr int kThreads = (2 + kDequantWarps) * 32;  // warp 0: TMA, warp 1: MMA + TMEM, warps 2..17: dequant (+ epilogue)
constexpr int kABytes = kBN * kBK * 2;               // 16 KB
template <int BT, int HL = 0>
struct Cfg {
    static constexpr int kBBytes = BT * kBK * 2;  // 32 KB (BT = 256) / 8 KB (BT = 64)
    static constexpr int kATotal = kABytes * (HL ? 2 : 1), kBTotal = kBBytes * (HL == 2 ? 2 : 1);
    static constexpr int kStageBytes = kATotal + kBTotal;
    static constexpr int kStages = (192 * 1024) / kStageBytes;  // 192 KB of operands in flight
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr int kTmemCols = BT;  // power of two >= 32
    // Instruction descriptor: fp16 x fp16 -> fp32, both operands K-major, M = kBN, N = BT.
    static constexpr uint32_t kIdesc =
        (1u << 4) | (static_cast<uint32_t>(BT >> 3) << 17) | (static_cast<uint32_t>(kBN >> 4) << 24);
};

#ifdef MB200_TRACE
__device__ long long g_gemm_trace[256];
#endif

struct GemmParams {
    const uint8_t *w;   // dense: the matrix; grouped: expert 0's blob + offset of the matrix inside a blob
    float *out;         // [rows of X][N]
    int M, N, K, bpr;   // M: rows of X (dense: tokens; grouped: routed (token, expert) pairs, expert-sorted)
    int q6;             // 0: Q4_K, 1: Q6_K
    int *err;
    // grouped form: CTA x = expert * tiles_per_expert + row tile; the expert's tokens are rows
    // [seg_off[e], seg_off[e] + seg_cnt[e]) of X
    const int *seg_off, *seg_cnt;
    int tiles_per_expert;  // 0 = dense
    size_t expert_stride;
    int x_lo_row0;         // HL = 2: the lo halves of the activations are rows x_lo_row0 .. of the same tensor map
};

// ---- one thread's 32 weights of a 64-wide K chunk, as fp32 ----------------------
// Q4_K: thread (row, h): chunk c of block b holds qs[32c..32c+31]; low nibbles are k-local 0..31
// (sub-block 2c), high nibbles 32..63 (sub-block 2c+1)  (reference src/kernels.cu:114-136).
// `raw` is the whole 144-byte block in registers (header + 8 x 16 bytes of qs), fetched one block
// ahead of its use so the global-memory latency hides behind four K chunks of work.
struct RawQ4 {
    uint4 hdr;
    uint4 q[2][2];  // the two chunks of the block this producer group handles (c = grp, grp + 2), 32 bytes each
};
__device__ __forceinline__ void load_raw_q4k(RawQ4 &raw, const uint8_t *blk, int grp)
{
    raw.hdr = __ldg(reinterpret_cast<const uint4 *>(blk));
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint8_t *q = blk + 16 + 32 * (grp + 2 * i);
        raw.q[i][0] = __ldg(reinterpret_cast<const uint4 *>(q));
        raw.q[i][1] = __ldg(reinterpret_cast<const uint4 *>(q + 16));
    }
}
// 32 weights of chunk c = grp + 2*I: low (h = 0) or high (h = 1) nibbles of its 32 bytes
template <int I>
__device__ __forceinline__ void dequant32_q4k(const RawQ4 &raw, int grp, int h, float (&wv)[32])
{
    const uint4 hdr = raw.hdr;
    uint32_t sc2, m2;
    q4k_scale_pair(hdr.y, hdr.z, hdr.w, grp + 2 * I, sc2, m2);
    const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
    const float sc = static_cast<float>(h ? (sc2 >> 8) : (sc2 & 0xFFu));
    const float mn = static_cast<float>(h ? (m2 >> 8) : (m2 & 0xFFu));
    // A masked nibble byte dropped into byte 2 of 2.0f (0x40000000) is v = 2 + n/64 -- an int->float
    // convert for the price of one byte permute:  w = d*sc*n - dmin*m = (64*d*sc) * v - (128*d*sc + dmin*m).
    // The cancellation costs ~8 of fp32's 24 bits; fp16 needs 11.
    const float a = 64.0f * (dd.x * sc);
    const float b = -(2.0f * a + dd.y * mn);
    const uint32_t qs[8] = {raw.q[I][0].x, raw.q[I][0].y, raw.q[I][0].z, raw.q[I][0].w,
                            raw.q[I][1].x, raw.q[I][1].y, raw.q[I][1].z, raw.q[I][1].w};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t word = (h ? (qs[i] >> 4) : qs[i]) & 0x0F0F0F0Fu;
        wv[4 * i + 0] = fmaf(a, __uint_as_float(__byte_perm(word, 0x40000000u, 0x7054)), b);
        wv[4 * i + 1] = fmaf(a, __uint_as_float(__byte_perm(word, 0x40000000u, 0x7154)), b);
        wv[4 * i + 2] = fmaf(a, __uint_as_float(__byte_perm(word, 0x40000000u, 0x7254)), b);
        wv[4 * i + 3] = fmaf(a, __uint_as_float(__byte_perm(word, 0x40000000u, 0x7354)), b);
    }
}

// Q6_K: a 64-wide K chunk c (0..3) of block b covers half hh = c >> 1 and the two thirty-two-groups
// g = 2*(c&1) + {0,1} of that half (value order 128hh + 32g + l). Thread h takes group
// g = 2*(c&1) + h, positions l = 0..31, i.e. k-local 32h + l  (reference src/kernels.cu:455-484).
// Its raw bytes -- 32 of ql, 32 of qh, two scales, d -- are fetched one chunk ahead of their use
// as aligned words (a Q6_K block is only 2-byte aligned: nine words + a funnel shift give eight).
struct RawQ6 {
    uint32_t ql[8], qh[8];
    unsigned short scb, dbits;
};
__device__ __forceinline__ void load_words_2b(const uint8_t *p, uint32_t (&w)[8])
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *base = reinterpret_cast<const uint32_t *>(a & ~static_cast<uintptr_t>(3));
    const uint32_t sh = static_cast<uint32_t>(a & 3) * 8;
    uint32_t t[9];
#pragma unroll
    for (int i = 0; i < 9; i++) t[i] = __ldg(base + i);  // the ninth word still lies inside the 210-byte block
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = __funnelshift_r(t[i], t[i + 1], sh);
}
__device__ __forceinline__ void load_raw_q6k(RawQ6 &raw, const uint8_t *blk, int c, int h)
{
    const int hh = c >> 1, g = 2 * (c & 1) + h;
    load_words_2b(blk + 64 * hh + 32 * (g & 1), raw.ql);
    load_words_2b(blk + 128 + 32 * hh, raw.qh);
    raw.scb = __ldg(reinterpret_cast<const unsigned short *>(blk + 192 + 8 * hh + 2 * g));
    raw.dbits = __ldg(reinterpret_cast<const unsigned short *>(blk + 208));
}
__device__ __forceinline__ void dequant32_q6k(const RawQ6 &raw, int c, int h, float (&wv)[32])
{
    const int g = 2 * (c & 1) + h;
    const float d = __half2float(__ushort_as_half(raw.dbits));
    const float s0 = d * static_cast<float>(static_cast<int8_t>(raw.scb & 0xFF));
    const float s1 = d * static_cast<float>(static_cast<int8_t>(raw.scb >> 8));
    const int lo_shift = 4 * (g >> 1), hi_shift = 2 * g;
    // q = lo4 | hi2 << 4 rebuilt four bytes at a time; a byte dropped into byte 2 of 2.0f (0x40000000) is
    // v = 2 + q/64, so  w = s*(q - 32) = (64 s) * v - 160 s  is one byte permute and one FMA per weight.
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t lo = (raw.ql[i] >> lo_shift) & 0x0F0F0F0Fu;
        const uint32_t hi = ((raw.qh[i] >> hi_shift) & 0x03030303u) << 4;
        const uint32_t q4 = lo | hi;
        const float s = i < 4 ? s0 : s1;
        const float a = 64.0f * s, b = -160.0f * s;
        wv[4 * i + 0] = fmaf(a, __uint_as_float(__byte_perm(q4, 0x40000000u, 0x7044)), b);
        wv[4 * i + 1] = fmaf(a, __uint_as_float(__byte_perm(q4, 0x40000000u, 0x7144)), b);
        wv[4 * i + 2] = fmaf(a, __uint_as_float(__byte_perm(q4, 0x40000000u, 0x7244)), b);
        wv[4 * i + 3] = fmaf(a, __uint_as_float(__byte_perm(q4, 0x40000000u, 0x7344)), b);
    }
}

template <int BT, int HL>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap xmap,
                                                               const __grid_constant__ GemmParams P)
{
    using C = Cfg<BT, HL>;
    constexpr int kStages = C::kStages, kStageBytes = C::kStageBytes, kBBytes = C::kBBytes, kTmemCols = C::kTmemCols;
    constexpr int kATotal = C::kATotal, kBTotal = C::kBTotal;
    constexpr uint32_t kIdesc = C::kIdesc;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);  // not through an integer: stays a shared-memory pointer
    uint8_t *stage_base = smem;                                    // kStages x (A 16 KB | B 32 KB), 1024-byte aligned
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kStages * kStageBytes);
    uint64_t *empty = full + kStages;
    uint64_t *acc_full = empty + kStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#ifdef MB200_TRACE
    const long long tr0 = clock64();
#define GSTAMP(slot) do { if (blockIdx.x == 0 && blockIdx.y == 0 && lane == 0) g_gemm_trace[slot] = clock64() - tr0; } while (0)
#else
#define GSTAMP(name) do {} while (0)
#endif
    // dense: weight tile blockIdx.x, token tile blockIdx.y. grouped: blockIdx.x = (expert, weight tile),
    // tokens = the expert's slice of X; a CTA whose token tile lies beyond the slice has nothing to do.
    const int expert = P.tiles_per_expert ? blockIdx.x / P.tiles_per_expert : 0;
    const int n0 = (P.tiles_per_expert ? blockIdx.x % P.tiles_per_expert : blockIdx.x) * kBN;  // first weight row
    const int seg0 = P.tiles_per_expert ? P.seg_off[expert] : 0;
    const int seg_n = P.tiles_per_expert ? P.seg_cnt[expert] : P.M;
    if (static_cast<int>(blockIdx.y) * BT >= seg_n) return;  // before any barrier / TMEM use: uniform for the CTA
    const int t0 = seg0 + blockIdx.y * BT;   // first row of X for this CTA
    const int t_end = seg0 + seg_n;          // rows of X past this belong to someone else
    const uint8_t *wbase = P.w + (size_t)expert * P.expert_stride;
    const int n_kb = P.K / kBK;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < kStages; s++) {
            mbar_init(&full[s], kDequantWarps / 2 + 1);  // the 8 warps of one producer group + the TMA thread's expect_tx arrival
            mbar_init(&empty[s], 1);                 // tcgen05.commit
        }
        mbar_init(acc_full, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (warp <= 2) GSTAMP(warp);

    if (warp == 0) {
        // ---------------- TMA producer: activations ----------------
        if (lane == 0) {
            int s = 0, ph = 0;
            for (int kb = 0; kb < n_kb; kb++) {
                if (kb >= kStages && !mbar_wait(&empty[s], ph ^ 1)) {
                    *abort_flag = 1;
                    break;
                }
                uint8_t *b_tile = stage_base + s * kStageBytes + kATotal;
                mbar_expect_tx(&full[s], kBTotal);
                tma_load_2d(b_tile, &xmap, kb * kBK, t0, &full[s]);
                if (HL == 2) tma_load_2d(b_tile + kBBytes, &xmap, kb * kBK, P.x_lo_row0 + t0, &full[s]);
                if (++s == kStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: the warp runs converged (tcgen.cuh) ----------------
        const uint32_t leader = elect_lane(), tm = warp_uniform(tmem_base), s0 = warp_uniform(smem_u32(stage_base));
        int s = 0, ph = 0;
        for (int kb = 0; kb < n_kb; kb++) {
            if (!mbar_wait(&full[s], ph)) *abort_flag = 1;
            if (__any_sync(0xffffffffu, *abort_flag)) break;
            tc_fence_after();
            const uint32_t a_addr = s0 + s * kStageBytes;
            const uint64_t da = smem_desc_sw128(a_addr), db = smem_desc_sw128(a_addr + kATotal);
            if (leader) {
#pragma unroll
                for (int kk = 0; kk < kBK / 16; kk++)  // 16 fp16 = 32 bytes = 2 descriptor units per K step
                    umma_f16(tm, da + 2 * kk, db + 2 * kk, kIdesc, (kb | kk) != 0);
                umma_commit(&empty[s]);  // the stage may be refilled once these MMAs have read it
            }
            __syncwarp();
            if (++s == kStages) {
                s = 0;
                ph ^= 1;
            }
        }
        if (leader) umma_commit(acc_full);  // all MMAs done: the accumulator is complete
    } else {
        // ---------------- dequant producers: weights -> fp16, swizzled K-major ----------------
        const int dt = tid - 64;        // 0..511
        const int grp = dt >> 8;        // producer group: K chunks kb = grp, grp + 2, ...
        const int r = (dt & 255) >> 1, h = dt & 1;  // weight row of the tile; low / high nibbles (k-local 32h ..)
        const int n = n0 + r;
        const bool row_ok = n < P.N;
        const size_t blk_bytes = P.q6 ? kQ6KBlock : kQ4KBlock;
        const uint8_t *row = wbase + (size_t)(row_ok ? n : 0) * P.bpr * blk_bytes;
        bool stop = false;
        // store this thread's 32 weights of K chunk kb into the A tile of its stage and publish it
        auto publish = [&](const float (&wv)[32], int kb) {
            const int s = kb % kStages, use = kb / kStages;
            if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1)) *abort_flag = 1;
            uint8_t *a_row = stage_base + s * kStageBytes + r * 128;
#pragma unroll
            for (int j = 0; j < 4; j++) {  // four 16-byte chunks of 8 fp16: logical chunk 4h + j, XOR-swizzled by the row
                uint32_t pk[4], pl[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float w0 = row_ok ? wv[8 * j + 2 * e] : 0.0f, w1 = row_ok ? wv[8 * j + 2 * e + 1] : 0.0f;
                    const __half2 hv = __floats2half2_rn(w0, w1);
                    pk[e] = *reinterpret_cast<const uint32_t *>(&hv);
                    if (HL) {  // what the fp16 rounding dropped, as a second fp16
                        const float2 back = __half22float2(hv);
                        const __half2 lv = __floats2half2_rn(w0 - back.x, w1 - back.y);
                        pl[e] = *reinterpret_cast<const uint32_t *>(&lv);
                    }
                }
                const int chunk = (4 * h + j) ^ (r & 7);
                *reinterpret_cast<uint4 *>(a_row + chunk * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                if (HL) *reinterpret_cast<uint4 *>(a_row + kABytes + chunk * 16) = make_uint4(pl[0], pl[1], pl[2], pl[3]);
            }
            proxy_fence_async();  // generic-proxy stores above must be visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if (*abort_flag) stop = true;
        };
        if (P.q6) {
            RawQ6 cur, nxt;
            load_raw_q6k(cur, row + (size_t)(grp >> 2) * blk_bytes, grp & 3, h);
            for (int kb = grp; kb < n_kb && !stop; kb += 2) {
                if (kb + 2 < n_kb) load_raw_q6k(nxt, row + (size_t)((kb + 2) >> 2) * blk_bytes, (kb + 2) & 3, h);  // one chunk ahead
                float wv[32];
                dequant32_q6k(cur, kb & 3, h, wv);
                publish(wv, kb);
                cur = nxt;
            }
        } else {
            RawQ4 cur, nxt;
            load_raw_q4k(cur, row, grp);
            for (int b = 0; b < P.bpr && !stop; b++) {
                if (b + 1 < P.bpr) load_raw_q4k(nxt, row + (size_t)(b + 1) * kQ4KBlock, grp);  // one block ahead
                float wv[32];
                dequant32_q4k<0>(cur, grp, h, wv);
                publish(wv, 4 * b + grp);
                if (!stop) {
                    dequant32_q4k<1>(cur, grp, h, wv);
                    publish(wv, 4 * b + grp + 2);
                }
                cur = nxt;
            }
        }
        // ---------------- epilogue: every producer warp; a warp may only touch TMEM lanes 32*(warp%4).. ----------------
        {
            const int quarter = warp & 3;
            const int part = (warp - 2) >> 2;  // 4 warps share a lane quarter and split the 8 column chunks
            if (!mbar_wait(acc_full, 0)) *abort_flag = 1;
            tc_fence_after();
            if (warp == 2) GSTAMP(12);
            if (!*abort_flag) {
                const int nrow = n0 + quarter * 32 + lane;
#pragma unroll 1
                for (int c0 = part * 32; c0 < BT; c0 += 128) {
                    if (t0 + c0 >= t_end) break;
                    uint32_t v[32];
                    tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c0, v);
                    if (nrow < P.N) {
                        float *o = P.out + (size_t)(t0 + c0) * P.N + nrow;
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (t0 + c0 + j < t_end) o[(size_t)j * P.N] = __uint_as_float(v[j]);
                    }
                }
            }
        }
    }
    if (warp == 2) GSTAMP(13);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
    if (tid == 0 && *abort_flag) atomicExch(P.err, MB200_ERR_TIMEOUT);
}

// ---- dense Q4_K form with the weight operand in TENSOR MEMORY -------------------------------------------
// In the kernel above each 64-wide K chunk moves 96 KB through shared memory (the producers' 16 KB of fp16
// weights in, the same 16 KB out to the tensor core, 32 KB of activations in by TMA and out again), which at
// 128 B per clock is 750 cycles against 524 for the MMAs, and every CTA pulls its 256-token activation tile
// from L2 again (256 MB per 512 x 8192 x 4096 GEMM: about 10 TB/s at the rate the tensor cores could go).
// Here the dequantised weights never touch shared memory: a producer thread owns one weight row (= one TMEM
// lane), dequantises its 64 weights of a K chunk into 32 registers of packed fp16 and writes them with
// tcgen05.st into a 32-column TMEM stage, from where the MMA takes its A operand. Shared memory carries only
// the activations (six 32 KB stages). The tile shape is a
// parameter (kAtmSlabs M = 128 slabs of weight rows x kAtmBT tokens): 1 x 256 is what is built -- 2 x 128, which
// halves the activation traffic from L2 (the next limit: 256 MB per GEMM), was measured slower (55 vs 34 us)
// because every weight is then dequantised twice as often and the producers become the bottleneck.
constexpr int kAtmBT = 256;                              // tokens per CTA (UMMA N)
constexpr int kAtmSlabs = 1;                             // M = 128 slabs of weight rows per CTA
constexpr int kAtmRows = kAtmSlabs * kBN;
constexpr int kAtmGroups = 4 / kAtmSlabs;                // producer groups; group g dequantises chunks kb = g (mod kAtmGroups)
constexpr int kAtmAStages = 6, kAtmBStages = 6;  // one ring: equal by construction
static_assert(kAtmAStages == kAtmBStages, "the weight and activation stages share their barriers");
constexpr int kAtmBBytes = kAtmBT * kBK * 2;             // 32 KB
constexpr int kAtmACols = kBK / 2;                       // 32 columns: 64 fp16 per row
constexpr int kAtmAccCols = kAtmSlabs * kAtmBT;          // 256
constexpr int kAtmTmemCols = 512;                        // 256 accumulator + 6 x 32 operand columns -> next power of two
constexpr int kAtmSmemBytes = kAtmBStages * kAtmBBytes + 1024 + 512;
constexpr uint32_t kAtmIdesc = Cfg<kAtmBT, 0>::kIdesc;
static_assert(kAtmAccCols + kAtmAStages * kAtmSlabs * kAtmACols <= kAtmTmemCols, "tensor memory budget");

__global__ void __launch_bounds__(kThreads, 1) gemm_tc_atm_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                 const __grid_constant__ GemmParams P)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);  // not through an integer: stays a shared-memory pointer
    // one ring: stage s holds the weights of a chunk in TMEM and its activations in shared memory
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kAtmBStages * kAtmBBytes);
    uint64_t *empty = full + kAtmBStages;
    uint64_t *acc_full = empty + kAtmBStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * kAtmRows, t0 = blockIdx.y * kAtmBT, t_end = P.M;
    if (t0 >= P.M) return;
    const int n_kb = P.K / kBK;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < kAtmBStages; s++) {
            mbar_init(&full[s], 4 * kAtmSlabs + 1);  // the warps (slabs x four lane quarters) of a producer group + the TMA thread
            mbar_init(&empty[s], 1);                 // tcgen05.commit
        }
        mbar_init(acc_full, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kAtmTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a0 = tmem_base + kAtmAccCols;  // operand stages behind the accumulator columns

    if (warp == 0) {
        if (lane == 0) {  // ---- TMA: activations ----
            int s = 0, ph = 0;
            for (int kb = 0; kb < n_kb; kb++) {
                if (kb >= kAtmBStages && !mbar_wait(&empty[s], ph ^ 1)) {
                    *abort_flag = 1;
                    break;
                }
                mbar_expect_tx(&full[s], kAtmBBytes);
                tma_load_2d(smem + s * kAtmBBytes, &xmap, kb * kBK, t0, &full[s]);
                if (++s == kAtmBStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp runs converged (tcgen.cuh) ----
        const uint32_t leader = elect_lane(), tm = warp_uniform(tmem_base), b0 = warp_uniform(smem_u32(smem));
        int s = 0, ph = 0;
        for (int kb = 0; kb < n_kb; kb++) {
            if (!mbar_wait(&full[s], ph)) *abort_flag = 1;
            if (__any_sync(0xffffffffu, *abort_flag)) break;
            tc_fence_after();
            const uint64_t db = smem_desc_sw128(b0 + s * kAtmBBytes);
            const uint32_t ta = tm + kAtmAccCols + s * (kAtmSlabs * kAtmACols);
            if (leader) {
#pragma unroll
                for (int kk = 0; kk < kBK / 16; kk++)  // 16 fp16 of K = 8 operand columns = 2 descriptor units
#pragma unroll
                    for (int sl = 0; sl < kAtmSlabs; sl++)
                        umma_f16_ta(tm + sl * kAtmBT, ta + sl * kAtmACols + 8 * kk, db + 2 * kk, kAtmIdesc, (kb | kk) != 0);
                umma_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == kAtmBStages) {
                s = 0;
                ph ^= 1;
            }
        }
        if (leader) umma_commit(acc_full);
    } else {
        // ---- producers: lane quarter q = warp % 4 (a warp may only touch TMEM lanes 32 q ..), idx = (warp - 2) / 4,
        // slab = idx % slabs, group par = idx / slabs: the thread owns row 128 slab + 32 q + lane of the tile and
        // the K chunks kb = par (mod groups): chunks par, par + groups, ... of every block of its row ----
        const int quarter = warp & 3, idx = (warp - 2) >> 2, slab = idx % kAtmSlabs, par = idx / kAtmSlabs;
        const int r = slab * kBN + quarter * 32 + lane, n = n0 + r;
        const bool row_ok = n < P.N;
        const uint8_t *row = P.w + (size_t)(row_ok ? n : 0) * P.bpr * kQ4KBlock;
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        constexpr int kPer = 4 / kAtmGroups;  // chunks of a block this thread dequantises
        struct Raw {
            uint4 hdr;
            uint4 q[kPer][2];
        } cur, nxt;
        auto load_raw = [&](Raw &raw, const uint8_t *blk) {
            raw.hdr = __ldg(reinterpret_cast<const uint4 *>(blk));
#pragma unroll
            for (int i = 0; i < kPer; i++) {
                const uint8_t *q = blk + 16 + 32 * (par + kAtmGroups * i);
                raw.q[i][0] = __ldg(reinterpret_cast<const uint4 *>(q));
                raw.q[i][1] = __ldg(reinterpret_cast<const uint4 *>(q + 16));
            }
        };
        load_raw(cur, row);
        bool stop = false;
        for (int b = 0; b < P.bpr && !stop; b++) {
            if (b + 1 < P.bpr) load_raw(nxt, row + (size_t)(b + 1) * kQ4KBlock);  // one block ahead
#pragma unroll
            for (int I = 0; I < kPer; I++) {
                // 64 weights of chunk c = par + groups I: low nibbles of its 32 bytes are k-local 0..31 (sub-block 2c),
                // high nibbles 32..63 (sub-block 2c + 1)
                uint32_t sc2, m2;
                q4k_scale_pair(cur.hdr.y, cur.hdr.z, cur.hdr.w, par + kAtmGroups * I, sc2, m2);
                const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&cur.hdr.x));
                const float live = row_ok ? 1.0f : 0.0f;  // rows past the matrix contribute zeros
                const float a_lo = live * 64.0f * (dd.x * static_cast<float>(sc2 & 0xFFu));
                const float a_hi = live * 64.0f * (dd.x * static_cast<float>(sc2 >> 8));
                const float b_lo = -(2.0f * a_lo + live * dd.y * static_cast<float>(m2 & 0xFFu));
                const float b_hi = -(2.0f * a_hi + live * dd.y * static_cast<float>(m2 >> 8));
                const uint32_t qs[8] = {cur.q[I][0].x, cur.q[I][0].y, cur.q[I][0].z, cur.q[I][0].w,
                                        cur.q[I][1].x, cur.q[I][1].y, cur.q[I][1].z, cur.q[I][1].w};
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint32_t lo = qs[i] & 0x0F0F0F0Fu, hi = (qs[i] >> 4) & 0x0F0F0F0Fu;
                    // a nibble byte dropped into byte 2 of 2.0f is 2 + n / 64: w = (64 d sc) v - (128 d sc + dmin m)
                    const float l0 = fmaf(a_lo, __uint_as_float(__byte_perm(lo, 0x40000000u, 0x7054)), b_lo);
                    const float l1 = fmaf(a_lo, __uint_as_float(__byte_perm(lo, 0x40000000u, 0x7154)), b_lo);
                    const float l2 = fmaf(a_lo, __uint_as_float(__byte_perm(lo, 0x40000000u, 0x7254)), b_lo);
                    const float l3 = fmaf(a_lo, __uint_as_float(__byte_perm(lo, 0x40000000u, 0x7354)), b_lo);
                    const float h0 = fmaf(a_hi, __uint_as_float(__byte_perm(hi, 0x40000000u, 0x7054)), b_hi);
                    const float h1 = fmaf(a_hi, __uint_as_float(__byte_perm(hi, 0x40000000u, 0x7154)), b_hi);
                    const float h2 = fmaf(a_hi, __uint_as_float(__byte_perm(hi, 0x40000000u, 0x7254)), b_hi);
                    const float h3 = fmaf(a_hi, __uint_as_float(__byte_perm(hi, 0x40000000u, 0x7354)), b_hi);
                    const __half2 p0 = __floats2half2_rn(l0, l1), p1 = __floats2half2_rn(l2, l3);
                    const __half2 p2 = __floats2half2_rn(h0, h1), p3 = __floats2half2_rn(h2, h3);
                    pk[2 * i] = *reinterpret_cast<const uint32_t *>(&p0);       // k = 4 i, 4 i + 1
                    pk[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&p1);   // k = 4 i + 2, 4 i + 3
                    pk[16 + 2 * i] = *reinterpret_cast<const uint32_t *>(&p2);  // k = 32 + 4 i ...
                    pk[16 + 2 * i + 1] = *reinterpret_cast<const uint32_t *>(&p3);
                }
                const int kb = 4 * b + par + kAtmGroups * I, s = kb % kAtmAStages, use = kb / kAtmAStages;
                if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1)) *abort_flag = 1;
                if (*abort_flag) {
                    stop = true;
                    break;
                }
                tc_fence_after();  // the MMAs that read this stage are complete: the overwrite is ordered after them
                tmem_st32(tmem_a0 + lane_addr + (s * kAtmSlabs + slab) * kAtmACols, pk);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
            cur = nxt;
        }
        // ---- epilogue: the warp reads its lane quarter of its slab's accumulator, its group's share of the token columns ----
        {
            if (!mbar_wait(acc_full, 0)) *abort_flag = 1;
            tc_fence_after();
            if (!*abort_flag) {
                const int nrow = n0 + r;
                constexpr int kShare = kAtmBT / kAtmGroups;
#pragma unroll 1
                for (int c0 = par * kShare; c0 < (par + 1) * kShare; c0 += 32) {
                    if (t0 + c0 >= t_end) break;
                    uint32_t v[32];
                    tmem_ld32(tmem_base + lane_addr + slab * kAtmBT + c0, v);
                    if (nrow < P.N) {
                        float *o = P.out + (size_t)(t0 + c0) * P.N + nrow;
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (t0 + c0 + j < t_end) o[(size_t)j * P.N] = __uint_as_float(v[j]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, kAtmTmemCols);
    if (tid == 0 && *abort_flag) atomicExch(P.err, MB200_ERR_TIMEOUT);
}

// X: fp16 [rows_x][K] row-major. Launches gemm_tc_kernel<BT> over grid (weight tiles [x experts], token tiles).
template <int BT, int HL = 0>
int launch_gemm_bt(GemmParams &P, const void *x_f16, int rows_x, dim3 grid, cudaStream_t stream, const char *where)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc) {
        fprintf(stderr, "[mnemo_b200] %s: cuTensorMapEncodeTiled is not available\n", where);
        return MB200_ERR_LAUNCH;
    }
    CUtensorMap xmap;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(P.K), static_cast<cuuint64_t>(rows_x)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(P.K) * 2};
    const cuuint32_t box[2] = {kBK, BT};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x_f16), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        fprintf(stderr, "[mnemo_b200] %s: tensor map for X could not be encoded\n", where);
        return MB200_ERR_ARG;
    }
    static bool attr_done[kMaxDevices] = {false};  // the opt-in is a per-device attribute
    if (!attr_done[current_device()]) {
        cudaFuncSetAttribute(gemm_tc_kernel<BT, HL>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BT, HL>::kSmemBytes);
        attr_done[current_device()] = true;
    }
    P.bpr = P.K / 256;
    P.err = device_error_word();
    gemm_tc_kernel<BT, HL><<<grid, kThreads, Cfg<BT, HL>::kSmemBytes, stream>>>(xmap, P);
    return cudaGetLastError() == cudaSuccess ? MB200_OK : MB200_ERR_LAUNCH;
}

// The dense Q4_K form with the weight operand in tensor memory (gemm_tc_atm_kernel).
int launch_gemm_atm(GemmParams &P, const void *x_f16, int rows_x, dim3 grid, cudaStream_t stream, const char *where)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc) {
        fprintf(stderr, "[mnemo_b200] %s: cuTensorMapEncodeTiled is not available\n", where);
        return MB200_ERR_LAUNCH;
    }
    CUtensorMap xmap;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(P.K), static_cast<cuuint64_t>(rows_x)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(P.K) * 2};
    const cuuint32_t box[2] = {kBK, kAtmBT};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x_f16), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        fprintf(stderr, "[mnemo_b200] %s: tensor map for X could not be encoded\n", where);
        return MB200_ERR_ARG;
    }
    static bool attr_done[kMaxDevices] = {false};
    if (!attr_done[current_device()]) {
        cudaFuncSetAttribute(gemm_tc_atm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtmSmemBytes);
        attr_done[current_device()] = true;
    }
    P.bpr = P.K / 256;
    P.err = device_error_word();
    gemm_tc_atm_kernel<<<grid, kThreads, kAtmSmemBytes, stream>>>(xmap, P);
    return cudaGetLastError() == cudaSuccess ? MB200_OK : MB200_ERR_LAUNCH;
}

int launch_gemm(const void *w, const void *x_f16, float *out, int M, int N, int K, int q6, cudaStream_t stream,
                const char *where)
{
    if (!w || !x_f16 || !out || M < 1 || N < 1 || K < 1) return MB200_ERR_ARG;
    if (K % 256 != 0) {
        fprintf(stderr, "[mnemo_b200] %s: K=%d must be a multiple of 256\n", where, K);
        return MB200_ERR_UNSUPPORTED;
    }
    if ((reinterpret_cast<uintptr_t>(x_f16) & 15) || (!q6 && (reinterpret_cast<uintptr_t>(w) & 15)) ||
        (q6 && (reinterpret_cast<uintptr_t>(w) & 1)))
        return MB200_ERR_ARG;
    GemmParams P{};
    P.w = static_cast<const uint8_t *>(w);
    P.out = out;
    P.M = M;
    P.N = N;
    P.K = K;
    P.q6 = q6;
    if (M <= 64)
        return launch_gemm_bt<64>(P, x_f16, M, dim3((N + kBN - 1) / kBN, 1), stream, where);
    if (!q6) return launch_gemm_atm(P, x_f16, M, dim3((N + kAtmRows - 1) / kAtmRows, (M + kAtmBT - 1) / kAtmBT), stream, where);
    return launch_gemm_bt<256>(P, x_f16, M, dim3((N + kBN - 1) / kBN, (M + 255) / 256), stream, where);
}

}  // namespace

void gemm_init()
{
    cudaFuncSetAttribute(gemm_tc_kernel<256, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<256>::kSmemBytes);
    cudaFuncSetAttribute(gemm_tc_kernel<64, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<64>::kSmemBytes);
    cudaFuncSetAttribute(gemm_tc_atm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtmSmemBytes);
    (void)encode_tiled();
}

}  // namespace mb200

using namespace mb200;

extern "C" {

int mb200_gemm_q4k_f16(const void *w, const void *x_f16, float *out, int M, int N, int K, cudaStream_t stream)
{
    return launch_gemm(w, x_f16, out, M, N, K, 0, stream, "mb200_gemm_q4k_f16");
}

int mb200_gemm_q6k_f16(const void *w, const void *x_f16, float *out, int M, int N, int K, cudaStream_t stream)
{
    return launch_gemm(w, x_f16, out, M, N, K, 1, stream, "mb200_gemm_q6k_f16");
}

}  // extern "C"

#ifdef MB200_TRACE
extern "C" void mb200_gemm_trace_read(void *dst)
{
    cudaMemcpyFromSymbol(dst, mb200::g_gemm_trace, sizeof(long long) * 256, 0, cudaMemcpyDeviceToDevice);
}
#endif
