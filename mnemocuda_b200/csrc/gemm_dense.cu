// Dense prefill GEMM on 5th-generation tensor cores:
//     out[t][n] = sum_k  f16(X[t][k]) * dequant(W)[n][k]        X: fp16 [M x K], W: Q4_K or Q6_K [N x K], out: fp32 [M x N]
// fp32 dequant(W) rounded to fp16 once (2.8e-4 relative L2), fp16 activations, fp32 accumulation.
// (The reference's "tensor-core GEMM", src/gemm_q4k.cu:201-266, is an int8 mma.sync experiment at batch 1.)
//
// The weight rows are the UMMA M dimension (128 per CTA, one TMEM lane each), the tokens the N dimension (BT per CTA), K goes in
// chunks of 64. Per CTA: a warp that loads activations (TMA, 128-byte swizzle), a warp that issues the MMAs, one or two that
// bring raw super-blocks into a shared-memory ring (Q4_K: TMA, rows of 144-byte blocks make a tensor map; Q6_K: 4-byte
// cp.async walking along the rows, as 210-byte blocks fit no tensor map), and 16 warps that dequantise a row per thread and
// store the fp16 operand straight into TMEM. A stage of the ring is a chunk: 32 TMEM columns of weights and BT x 128 bytes of
// activations behind one pair of barriers.
//
// What bounds a tile is one of: the dequant warps (about 300 cycles per chunk and SM whatever BT is), the activation tile's
// way from L2 (BT x 128 bytes per chunk at 42 bytes per cycle and SM), a fixed 6000 cycles of launch, ramp and epilogue. So BT
// and the number of K splits are chosen per shape (plan()): wide tiles where there are enough of them to fill the SMs, narrow
// ones -- every weight then dequantised more than once, on SMs that would otherwise idle -- where there are not, and for still
// smaller shapes the CTAs of a cluster share the K range of a tile and add their accumulators through distributed shared
// memory, in rank order (deterministic). At the large end two CTAs share a tile of 256 rows x 256 tokens (cta_group::2): each
// dequantises its own rows and loads half of the activations, which makes the MMAs the bound (512 x 8192 x 4096: the tensor pipe
// is busy 66 % of the launch's cycles, ramp and epilogue included).
//
// Measured: Q4_K 512 x 8192 x 4096 35 us (clock-throttled in a loop: 21 us of cycles at 1.92 GHz), 2048 x 8192 x 4096 135,
// 200 x 4096 x 4096 12.8, 16 x 4096 x 4096 8.4 (host-bound); Q6_K 512 x 8192 x 4096 42.8, 130 x 7795 x 5120 37.1,
// 33 x 2022 x 2560 12.4. (Weights through shared memory, one tile size and no K split: 1.2 to 4 times as long.)
#include <cooperative_groups.h>

#include <cstdio>

#include "dequant.cuh"
#include "tcgen.cuh"

namespace mb200 {
int pdl_enabled();

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
namespace cg = cooperative_groups;

constexpr int kRows = 128;   // weight rows per tile (UMMA M)
constexpr int kGroups = 4;   // dequant groups of 4 warps
constexpr int kQ6Pitch = 212;  // bytes between rows of a Q6_K stage: 53 words, odd, so 32 rows hit 32 banks
constexpr int kMaxSplit = 8;

struct Params {
    const uint8_t *w;
    float *out;
    int M, N, bpr;
    int pdl;
    int *err;
};

template <int QT, int BT, bool PAIR>
struct Cfg {
    static constexpr int kDq0 = QT == 4 ? 3 : 4, kThreads = (kDq0 + 4 * kGroups) * 32;
    static constexpr int kXRows = PAIR ? BT / 2 : BT;
    static constexpr int kStages = BT == 256 ? (PAIR ? 8 : 5) : BT == 128 ? 8 : 14;  // what TMEM (BT + 32 columns each) and shared memory hold
    static constexpr int kXBytes = kXRows * 128;
    static constexpr int kWBytes = QT == 4 ? kRows * kQ4KBlock : kRows * kQ6Pitch;
    static constexpr int kWStages = QT == 6 && BT == 256 && !PAIR ? 2 : 3;
    static constexpr int kOffW = kStages * kXBytes;
    static constexpr int kOffBar = kOffW + kWStages * kWBytes;
    static constexpr int kSmem = kOffBar + 512 + 1024 /* alignment */;
    static_assert(kSmem <= 227 * 1024 && BT + 32 * kStages <= 512, "shared memory / tensor memory budget");
};

// See the grouped GEMM: a wait that runs out raises the abort flag, after which no wait of the CTA waits any more.
__device__ __noinline__ void wait_slow(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    for (uint32_t i = 0; i < kWaitBudget; i++)
        if (*abort_flag || mbar_try_wait(bar, parity)) return;
    *abort_flag = 1;
}
__device__ __forceinline__ void wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    if (!mbar_try_wait(bar, parity)) wait_slow(bar, parity, abort_flag);
}

// 32 weights -> 16 registers of fp16 pairs. A small integer in byte 2 of 2.0f (0x40000000) is v = 2 + n / 64: an int -> float
// conversion for one byte permute; w = s n - b = (64 s) v - (128 s + b) in fp32, rounded to fp16 once.
__device__ __forceinline__ void pack_f16(const uint32_t (&n)[8], const float (&a)[2], const float (&b)[2], uint32_t (&o)[16])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float s = a[i >> 2], c = b[i >> 2];
        const float w0 = fmaf(s, __uint_as_float(__byte_perm(n[i], 0x40000000u, 0x7044)), c);
        const float w1 = fmaf(s, __uint_as_float(__byte_perm(n[i], 0x40000000u, 0x7144)), c);
        const float w2 = fmaf(s, __uint_as_float(__byte_perm(n[i], 0x40000000u, 0x7244)), c);
        const float w3 = fmaf(s, __uint_as_float(__byte_perm(n[i], 0x40000000u, 0x7344)), c);
        const __half2 p0 = __floats2half2_rn(w0, w1), p1 = __floats2half2_rn(w2, w3);
        o[2 * i] = *reinterpret_cast<const uint32_t *>(&p0);
        o[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&p1);
    }
}

template <int QT, int BT, bool PAIR>
__global__ void __launch_bounds__((Cfg<QT, BT, PAIR>::kThreads), 1) gemm_dense_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                                const __grid_constant__ CUtensorMap wmap,
                                                                                const Params P)
{
    using C = Cfg<QT, BT, PAIR>;
    constexpr int S = C::kStages, WS = C::kWStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);  // not through an integer: stays a shared-memory pointer
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + C::kOffBar), *empty = full + S;
    uint64_t *wfull = empty + S, *wempty = wfull + WS, *acc_full = wempty + WS, *pfull = acc_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(pfull + S);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * kRows, t0 = blockIdx.y * BT;
    const int split = blockIdx.z, splits = gridDim.z;
    const int b0 = P.bpr * split / splits, nb = P.bpr * (split + 1) / splits - b0;  // this CTA's super-blocks
    const int units = 2 * nb;  // half super-blocks: two chunks each
    // Chunk order, the same for every role: round j takes units 4 j + g, g < G (G = 4, or 2 in a last round); chunk 0 of
    // each, then chunk 1.

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 4 + 1);  // the four warps of a dequant group + the X loader's expect_tx arrival
            mbar_init(&empty[s], 1);     // tcgen05.commit
            mbar_init(&pfull[s], 1);     // PAIR: the other CTA's stage is full
        }
        for (int s = 0; s < WS; s++) {
            mbar_init(&wfull[s], QT == 4 ? 1 : 64);  // TMA: the expect_tx arrival; cp.async: every thread of the two warps
            mbar_init(&wempty[s], 8);                // the two groups that share a super-block
        }
        mbar_init(acc_full, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc<PAIR>(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    if (PAIR) cg::this_cluster().sync();  // the partner's barriers are initialised
    tc_fence_after();
    const int rank = PAIR ? static_cast<int>(blockIdx.x & 1) : 0;
    if (P.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {  // ---- activations ----
            if (P.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");  // X may come from the kernel upstream
            int s = 0, ph = 1;
            for (int j = 0; j < units; j += kGroups) {
                const int G = min(kGroups, units - j);
                for (int cgi = 0; cgi < 2 * G; cgi++) {
                    wait(&empty[s], ph, abort_flag);  // passes at once while the stage has not been used
                    const int k = 256 * b0 + (cgi < G ? 128 * (j + cgi) : 128 * (j + cgi - G) + 64);
                    mbar_expect_tx(&full[s], C::kXBytes);
                    tma_load_2d(smem + s * C::kXBytes, &xmap, k, t0 + rank * C::kXRows, &full[s]);
                    if (++s == S) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp runs converged, one lane's instructions take effect (tcgen.cuh) ----
        const uint32_t leader = elect_lane(), tm = warp_uniform(tmem), x0 = warp_uniform(smem_u32(smem));
        constexpr uint32_t idesc = umma_idesc_f16(PAIR ? 2 * kRows : kRows, BT);
        int s = 0, ph = 0;
        for (int kb = 0; kb < 2 * units; kb++) {
            wait(&full[s], ph, abort_flag);
            if (PAIR && rank == 0) wait(&pfull[s], ph, abort_flag);
            tc_fence_after();
            __syncwarp();
            const uint64_t db = smem_desc_sw128(x0 + s * C::kXBytes);
            const uint32_t a = tm + BT + 32 * s;
            if (leader) {
                if (PAIR && rank == 1) {  // tell the first CTA, which issues for both
                    tc_fence_before();
                    mbar_arrive_cta0(&pfull[s]);
                } else {
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {  // 16 fp16 of K = 8 operand columns = 2 descriptor units
                        if (PAIR)
                            umma2_f16_ta(tm, a + 8 * kk, db + 2 * kk, idesc, (kb | kk) != 0);
                        else
                            umma_f16_ta(tm, a + 8 * kk, db + 2 * kk, idesc, (kb | kk) != 0);
                    }
                    if (PAIR)
                        umma2_commit(&empty[s]);
                    else
                        umma_commit(&empty[s]);
                }
            }
            __syncwarp();
            if (++s == S) {
                s = 0;
                ph ^= 1;
            }
        }
        if (leader) {
            if (!PAIR)
                umma_commit(acc_full);
            else if (rank == 0)
                umma2_commit(acc_full);
        }
        __syncwarp();
    } else if (warp < C::kDq0) {
        // ---- raw weights: 128 rows x one super-block per stage; they never depend on the kernel upstream ----
        if (QT == 6 || lane == 0) {
            int s = 0, ph = 1;
            for (int b = 0; b < nb; b++) {
                wait(&wempty[s], ph, abort_flag);
                uint8_t *dst = smem + C::kOffW + s * C::kWBytes;
                if (QT == 4) {
                    mbar_expect_tx(&wfull[s], C::kWBytes);
                    tma_load_2d(dst, &wmap, (b0 + b) * kQ4KBlock, n0, &wfull[s]);  // rows past N arrive as zeros
                } else {
                    const int r0 = (warp - 2) * 64, rows = min(64, P.N - n0 - r0);  // rows past N are not stored in the end
                    const uint8_t *blk = P.w + ((size_t)(n0 + r0) * P.bpr + b0 + b) * kQ6KBlock;
                    uint32_t d = smem_u32(dst) + r0 * kQ6Pitch + 4 * lane;
#pragma unroll 4
                    for (int r = 0; r < rows; r++) {
                        copy_q6k_row(d, blk, lane);
                        blk += (size_t)P.bpr * kQ6KBlock;
                        d += kQ6Pitch;
                    }
                    cp_async_arrive(&wfull[s]);
                }
                if (++s == WS) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (QT == 6) asm volatile("cp.async.wait_all;" ::: "memory");
        }
    } else {
        // ---- dequant: thread = row r of the tile; group g ----
        const int q = warp & 3, g = (warp - C::kDq0) >> 2, r = 32 * q + lane;
        const uint32_t lane_addr = static_cast<uint32_t>(32 * q) << 16;
        auto stage_free = [&](int it) {
            const int s = it % S;
            if (it >= S) wait(&empty[s], ((it / S) - 1) & 1, abort_flag);
            __syncwarp();
            tc_fence_after();
            return tmem + BT + 32 * s + lane_addr;
        };
        auto publish = [&](int it) {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[it % S]);
        };
        uint32_t row_addr = 0;  // Q6_K: low bits of the row's address
        if (QT == 6) row_addr = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(P.w)) + ((uint32_t)(n0 + r) * (uint32_t)P.bpr + b0) * kQ6KBlock;
        for (int j = 0; j < units; j += kGroups) {
            const int G = min(kGroups, units - j), u = j + g;
            if (g >= G) break;
            const int sb = u >> 1, half = u & 1, ws = sb % WS;
            wait(&wfull[ws], (sb / WS) & 1, abort_flag);
            __syncwarp();
            const uint8_t *blk = smem + C::kOffW + ws * C::kWBytes;
            uint32_t o[16], n8[8];
            if (QT == 4) {
                blk += r * kQ4KBlock;
                const uint4 hdr = *reinterpret_cast<const uint4 *>(blk);
                uint4 qv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) qv[i] = *reinterpret_cast<const uint4 *>(blk + 16 + 64 * half + 16 * i);
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[ws]);
                const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int it = 2 * j + c * G + g;
                    uint32_t sc2, m2, ta = 0;
                    q4k_scale_pair(hdr.y, hdr.z, hdr.w, 2 * half + c, sc2, m2);
                    const uint32_t wq[8] = {qv[2 * c].x, qv[2 * c].y, qv[2 * c].z, qv[2 * c].w,
                                            qv[2 * c + 1].x, qv[2 * c + 1].y, qv[2 * c + 1].z, qv[2 * c + 1].w};
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float a = 64.0f * (dd.x * static_cast<float>(h ? sc2 >> 8 : sc2 & 0xFFu));
                        const float b = -(2.0f * a + dd.y * static_cast<float>(h ? m2 >> 8 : m2 & 0xFFu));
#pragma unroll
                        for (int i = 0; i < 8; i++) n8[i] = (h ? wq[i] >> 4 : wq[i]) & 0x0F0F0F0Fu;
                        const float av[2] = {a, a}, bv[2] = {b, b};
                        pack_f16(n8, av, bv, o);
                        if (h == 0) ta = stage_free(it);
                        tmem_st16(ta + 16 * h, o);
                    }
                    publish(it);
                }
            } else {
                RawQ6 raw;
                raw.load(blk + r * kQ6Pitch, (row_addr + sb * kQ6KBlock) & 2u, half);
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[ws]);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int it = 2 * j + c * G + g;
                    uint32_t ta = 0;
#pragma unroll
                    for (int h = 0; h < 2; h++) {  // thirty-two-group 2 c + h of the half, two scales
                        float av[2], bv[2];
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const float s = raw.d * static_cast<float>(static_cast<int8_t>(raw.sc[c] >> (16 * h + 8 * i)));
                            av[i] = 64.0f * s;
                            bv[i] = -160.0f * s;
                        }
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const uint32_t l = c ? raw.ql[8 * h + i] >> 4 : raw.ql[8 * h + i];
                            const uint32_t hb = c == 0 ? (h == 0 ? raw.qh[i] << 4 : raw.qh[i] << 2) : (h == 0 ? raw.qh[i] : raw.qh[i] >> 2);
                            n8[i] = (l & 0x0F0F0F0Fu) | (hb & 0x30303030u);
                        }
                        pack_f16(n8, av, bv, o);
                        if (h == 0) ta = stage_free(it);
                        tmem_st16(ta + 16 * h, o);
                    }
                    publish(it);
                }
            }
        }
        // ---- epilogue: group g takes its share of the token columns ----
        wait(acc_full, 0, abort_flag);
        __syncwarp();
        tc_fence_after();
        if (P.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");  // out may still be in use upstream
        constexpr int kShare = BT / kGroups;
        float *red = reinterpret_cast<float *>(smem);  // [BT][128]: the activation ring, read for the last time by now
#pragma unroll 1
        for (int c0 = g * kShare; c0 < (g + 1) * kShare; c0 += 16) {
            if (t0 + c0 >= P.M) break;
            uint32_t v[16];
            tmem_ld16(tmem + lane_addr + c0, v);
            if (splits > 1) {
#pragma unroll
                for (int i = 0; i < 16; i++) red[(c0 + i) * kRows + r] = __uint_as_float(v[i]);
            } else if (n0 + r < P.N) {
                float *dst = P.out + (size_t)(t0 + c0) * P.N + n0 + r;
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (t0 + c0 + i < P.M) dst[(size_t)i * P.N] = __uint_as_float(v[i]);
            }
        }
    }
    if (splits > 1) {
        // ---- the cluster adds its partial tiles: rank k does every splits-th token ----
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        if (warp >= C::kDq0) {
            const int i = tid - C::kDq0 * 32, r = i & 127;
            const float *red = reinterpret_cast<const float *>(smem);
            const float *peer[kMaxSplit];
#pragma unroll
            for (int p = 0; p < kMaxSplit; p++) peer[p] = cl.map_shared_rank(red, p < splits ? p : 0);
            const int tokens = min(BT, P.M - t0);
            for (int t = split + splits * (i >> 7); t < tokens; t += splits * 4) {
                float v[kMaxSplit];
#pragma unroll
                for (int p = 0; p < kMaxSplit; p++) v[p] = p < splits ? peer[p][t * kRows + r] : 0.0f;
                float acc = v[0];
#pragma unroll
                for (int p = 1; p < kMaxSplit; p++) acc += v[p];
                if (n0 + r < P.N) P.out[(size_t)(t0 + t) * P.N + n0 + r] = acc;
            }
        }
        cl.sync();  // nobody leaves while its shared memory is being read
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cg::this_cluster().sync();  // neither leaves while the other may still signal it
    if (warp == 1) tmem_dealloc<PAIR>(tmem, 512);
    if (tid == 0 && *abort_flag) atomicExch(P.err, MB200_ERR_TIMEOUT);
}

struct Plan {
    int bt, splits;
    bool pair;
};
// The cheapest form by the cost model of the file's head, in SM cycles: whole waves of tiles, a tile being 6000 cycles plus its
// chunks, and 2500 for adding up splits. Ties go to the wider tile.
Plan plan(int M, int N, int K)
{
    const int sms = device_sms(), bpr = K / 256, row_tiles = (N + kRows - 1) / kRows;
    Plan best{256, 1, false};
    long best_cost = -1;
    auto offer = [&](int bt, int s, bool pair, int per) {
        const long tiles = (long)(pair ? row_tiles + (row_tiles & 1) : row_tiles) * ((M + bt - 1) / bt) * s;
        if (s > 1 && tiles > sms) return;
        const long cost = (tiles + sms - 1) / sms * (6000 + 4L * ((bpr + s - 1) / s) * per + (s > 1 ? 2500 : 0));
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = {bt, s, pair};
        }
    };
    offer(256, 1, true, 530);
    for (int bt = 256; bt >= 64; bt /= 2)
        for (int s = 1; s <= kMaxSplit && s <= bpr; s *= 2) offer(bt, s, false, 3 * bt > 300 ? 3 * bt : 300);
    return best;
}

template <int QT, int BT, bool PAIR>
void attr()
{
    static bool done[kMaxDevices] = {false};  // the opt-in is a per-device attribute
    if (done[current_device()]) return;
    cudaFuncSetAttribute(gemm_dense_kernel<QT, BT, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<QT, BT, PAIR>::kSmem);
    done[current_device()] = true;
}

template <int QT, int BT, bool PAIR>
int launch(const Params &P, const CUtensorMap &wmap, const void *x, int K, int splits, cudaStream_t stream)
{
    using C = Cfg<QT, BT, PAIR>;
    CUtensorMap xmap;
    if (!encode_f16_rows(&xmap, x, K, P.M, C::kXRows)) return MB200_ERR_ARG;
    attr<QT, BT, PAIR>();
    const int row_tiles = (P.N + kRows - 1) / kRows;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(PAIR ? row_tiles + (row_tiles & 1) : row_tiles, (P.M + BT - 1) / BT, splits);
    cfg.blockDim = dim3(C::kThreads);
    cfg.dynamicSmemBytes = C::kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = PAIR ? 2 : 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = splits;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = P.pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_dense_kernel<QT, BT, PAIR>, xmap, wmap, P) == cudaSuccess ? MB200_OK : MB200_ERR_LAUNCH;
}

template <int QT>
int launch_gemm(const void *w, const void *x_f16, float *out, int M, int N, int K, cudaStream_t stream, const char *where)
{
    if (!w || !x_f16 || !out || M < 1 || N < 1 || K < 1) return MB200_ERR_ARG;
    if (K % 256 != 0) {
        fprintf(stderr, "[mnemo_b200] %s: K=%d must be a multiple of 256\n", where, K);
        return MB200_ERR_UNSUPPORTED;
    }
    if ((reinterpret_cast<uintptr_t>(x_f16) & 15) || (reinterpret_cast<uintptr_t>(w) & (QT == 4 ? 15 : 1))) return MB200_ERR_ARG;
    Params P{static_cast<const uint8_t *>(w), out, M, N, K / 256, pdl_enabled(), device_error_word()};
    CUtensorMap wmap = {};
    if (QT == 4 && !encode_q4k_rows(&wmap, w, P.bpr, N, 1, 0, kRows)) {
        fprintf(stderr, "[mnemo_b200] %s: a tensor map could not be encoded\n", where);
        return MB200_ERR_ARG;
    }
    const Plan p = plan(M, N, K);
    if (p.pair) return launch<QT, 256, true>(P, wmap, x_f16, K, 1, stream);
    if (p.bt == 64) return launch<QT, 64, false>(P, wmap, x_f16, K, p.splits, stream);
    if (p.bt == 128) return launch<QT, 128, false>(P, wmap, x_f16, K, p.splits, stream);
    return launch<QT, 256, false>(P, wmap, x_f16, K, p.splits, stream);
}

}  // namespace

void gemm_init()
{
    attr<4, 64, false>();
    attr<4, 128, false>();
    attr<4, 256, false>();
    attr<4, 256, true>();
    attr<6, 64, false>();
    attr<6, 128, false>();
    attr<6, 256, false>();
    attr<6, 256, true>();
    (void)encode_tiled();
}

}  // namespace mb200

using namespace mb200;

extern "C" {

int mb200_gemm_q4k_f16(const void *w, const void *x_f16, float *out, int M, int N, int K, cudaStream_t stream)
{
    return launch_gemm<4>(w, x_f16, out, M, N, K, stream, "mb200_gemm_q4k_f16");
}

int mb200_gemm_q6k_f16(const void *w, const void *x_f16, float *out, int M, int N, int K, cudaStream_t stream)
{
    return launch_gemm<6>(w, x_f16, out, M, N, K, stream, "mb200_gemm_q6k_f16");
}

}  // extern "C"
