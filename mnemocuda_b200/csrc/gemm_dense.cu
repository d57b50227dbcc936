// Dense prefill GEMM on 5th-generation tensor cores:
//     out[t][n] = sum_k  f16(X[t][k]) * dequant(W)[n][k]        X: fp16 [M x K], W: Q4_K or Q6_K [N x K], out: fp32 [M x N]
// fp32 dequant(W) rounded to fp16 once (2.8e-4 relative L2), fp16 activations, fp32 accumulation.
// (The reference's "tensor-core GEMM", src/gemm_q4k.cu:201-266, is an int8 mma.sync experiment at batch 1.)
//
// The weight rows are the UMMA M dimension (128 per CTA, one TMEM lane each), the tokens the N dimension (BT per CTA), K goes in
// chunks of 64. Per CTA: a warp that loads activations (TMA, 128-byte swizzle), a warp that issues the MMAs, one that brings raw
// super-blocks into a shared-memory ring (TMA: rows of 144-byte Q4_K blocks make a tensor map, of 210-byte Q6_K blocks 1 to 8 rows
// together do; a Q6_K tensor off its 16 bytes, or with rows left over, by two warps of 4-byte cp.async), and 16 warps that
// dequantise a row per thread and store the fp16 operand straight into TMEM. A stage of the ring is a chunk: 32 TMEM columns of weights
// and BT x 128 bytes of activations behind one pair of barriers.
//
// What bounds a tile is one of: the dequant warps (370 to 480 cycles per chunk and SM at up to 128 tokens), the activation tile's
// way from L2 and the MMAs (590 at 256), and a start and an end of 2 to 7 us, the longer the wider the tile and the fuller the GPU.
// So BT and the number of K splits are chosen per shape (plan()): wide tiles where there are enough of them to fill the SMs, narrow
// ones -- every weight then dequantised more than once, on SMs that would otherwise idle -- where there are not, and for still
// smaller shapes the CTAs of a cluster share the K range of a tile and add their accumulators through distributed shared
// memory, in rank order (deterministic). At the large end two CTAs may share a tile of 256 rows x 256 tokens (cta_group::2): each
// dequantises its own rows and loads half of the activations.
//
// Measured (in brackets: shapes placed by the cycles of the SMs alone, Q6_K by cp.async, loaders in one-thread branches, byte permutes for
// Q4_K): Q4_K 512 x 8192 x 4096 28.2 us in a burst (28.9), 33.6 under the power cap in a loop (34.2); 2048 x 8192 x 4096 110 (113),
// 197 x 4096 x 4096 11.7 (12.8), 197 x 2048 x 2048 7.1 (16.0), 512 x 512 x 8192 10.6 (17.3), 8 x 2048 x 2048 3.5 (7.8); Q6_K 512 x 8192 x 4096
// 29.7 (35.9), 197 x 8192 x 4096 18.4 (30.9), 197 x 4096 x 1536 7.4 (11.0), 8 x 8192 x 4096 12.5 (16.9).
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
    int group;  // Q6_K: rows a tensor map takes together (encode_q6k_groups), 0: by cp.async
    int pdl;
    int *err;
};

template <int QT, int BT, bool PAIR>
struct Cfg {
    static constexpr int kDq0 = QT == 4 ? 3 : 4, kThreads = (kDq0 + 4 * kGroups) * 32;
    static constexpr int kXRows = PAIR ? BT / 2 : BT;
    static constexpr int kStages = BT == 256 ? (PAIR ? 8 : 5) : BT == 128 ? 8 : 14;  // what TMEM (BT + 32 columns each) and shared memory hold
    static constexpr int kXBytes = kXRows * 128;
    static constexpr int kWBytes = QT == 4 ? kRows * kQ4KBlock : kRows * kQ6Slot;
    static constexpr int kWStages = QT == 6 && BT == 256 && !PAIR ? 2 : 3;
    // A dequant group takes every second super-block. Barriers of its own for every second round of the ring's stages, so that it waits
    // for every phase of those it uses: on a stage's one barrier it would miss every second phase, and the parity of the one before the
    // missed one lets it pass (super-block 4 at once if 2 lands before 1).
    static constexpr int kWBars = 2 * kWStages;
    static_assert(kWBars % (kGroups / 2) == 0, "a group meets every phase of the barriers it waits on");
    static constexpr int kOffW = kStages * kXBytes;
    static constexpr int kOffBar = kOffW + kWStages * kWBytes;
    static constexpr int kSmem = kOffBar + 512 + 1024 /* alignment */;
    static_assert(kSmem <= 227 * 1024 && BT + 32 * kStages <= 512, "shared memory / tensor memory budget");
};

// The S partial tiles [token][128 rows] of a cluster, in rank order: rank `split` takes every S-th token, a warp a token, a lane four
// rows, up to eight 16-byte loads in flight (with one of four bytes at a time Q6_K 8 x 2048 x 2048 took 10.6 instead of 8.5 us).
template <int S, int BT>
__device__ __forceinline__ void add_splits(cg::cluster_group cl, uint8_t *smem, const Params &P, int split, int n0, int t0, int w, int lane)
{
    constexpr int U = 8 / S, kStep = S * 4 * kGroups;
    const float4 *peer[S];
#pragma unroll
    for (int p = 0; p < S; p++) peer[p] = cl.map_shared_rank(reinterpret_cast<const float4 *>(smem), p) + lane;
    const int tokens = min(BT, P.M - t0), n = n0 + 4 * lane;
    const bool vec = n + 3 < P.N && (P.N & 3) == 0 && (reinterpret_cast<uintptr_t>(P.out) & 15) == 0;
    for (int t = split + S * w; t < tokens; t += U * kStep) {
        float4 v[U][S];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int p = 0; p < S; p++)
                if (t + u * kStep < tokens) v[u][p] = peer[p][(t + u * kStep) * (kRows / 4)];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (t + u * kStep >= tokens) break;
            float4 a = v[u][0];
#pragma unroll
            for (int p = 1; p < S; p++) {
                a.x += v[u][p].x;
                a.y += v[u][p].y;
                a.z += v[u][p].z;
                a.w += v[u][p].w;
            }
            float *o = P.out + (size_t)(t0 + t + u * kStep) * P.N + n;
            if (vec) {
                *reinterpret_cast<float4 *>(o) = a;
            } else {
                if (n < P.N) o[0] = a.x;
                if (n + 1 < P.N) o[1] = a.y;
                if (n + 2 < P.N) o[2] = a.z;
                if (n + 3 < P.N) o[3] = a.w;
            }
        }
    }
}

template <int QT, int BT, bool PAIR>
__global__ void __launch_bounds__((Cfg<QT, BT, PAIR>::kThreads), 1) gemm_dense_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                                const __grid_constant__ CUtensorMap wmap,
                                                                                const Params P)
{
    using C = Cfg<QT, BT, PAIR>;
    constexpr int S = C::kStages, WS = C::kWStages, WB = C::kWBars;
    static_assert(8 * (3 * S + 2 * WB + 1) + 8 <= 512, "barriers");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);  // not through an integer: stays a shared-memory pointer
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + C::kOffBar), *empty = full + S;
    uint64_t *wfull = empty + S, *wempty = wfull + WB, *acc_full = wempty + WB, *pfull = acc_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(pfull + S);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = static_cast<int>(warp_uniform(tid >> 5));
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
        for (int s = 0; s < WB; s++) {
            mbar_init(&wfull[s], QT == 4 || P.group ? 1 : 64);  // TMA: the expect_tx arrival; cp.async: every thread of the two warps
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
    const uint32_t tmem = warp_uniform(*tmem_slot), leader = elect_lane();

    // Loaders and issuer run converged through their loops, one lane's copies and MMAs take effect (tcgen.cuh).
    if (warp == 0) {
        // ---- activations ----
        if (P.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");  // X may come from the kernel upstream
        int s = 0;
        uint32_t ph = 1;
        for (int j = 0; j < units; j += kGroups) {
            const int G = min(kGroups, units - j);
            for (int cgi = 0; cgi < 2 * G; cgi++) {
                wait(&empty[s], ph, abort_flag);  // passes at once while the stage has not been used
                __syncwarp();
                const int k = 256 * b0 + (cgi < G ? 128 * (j + cgi) : 128 * (j + cgi - G) + 64);
                if (leader) {
                    mbar_expect_tx(&full[s], C::kXBytes);
                    tma_load_2d(smem + s * C::kXBytes, &xmap, k, t0 + rank * C::kXRows, &full[s]);
                }
                if (++s == S) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        constexpr uint32_t idesc = umma_idesc_f16(PAIR ? 2 * kRows : kRows, BT);
        const uint32_t full0 = warp_uniform(smem_u32(full)), desc0 = desc_lo(warp_uniform(smem_u32(smem)));
        const uint32_t to_empty = 8 * S, to_pfull = 8 * static_cast<uint32_t>(pfull - full);
        int s = 0;
        uint32_t ph = 0;
        for (int kb = 0; kb < 2 * units; kb++) {
            const uint32_t bar = full0 + 8 * s;
            wait(bar, ph, abort_flag);
            if (PAIR && rank == 0) wait(bar + to_pfull, ph, abort_flag);
            tc_fence_after();
            __syncwarp();
            const uint32_t db = desc0 + s * (C::kXBytes / 16), a = tmem + BT + 32 * s;
            if (leader) {
                if (PAIR && rank == 1) {  // tell the first CTA, which issues for both
                    tc_fence_before();
                    mbar_arrive_cta0(&pfull[s]);
                } else {
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {  // 16 fp16 of K = 8 operand columns = 2 descriptor units
                        if (PAIR)
                            umma2_f16_ta(tmem, a + 8 * kk, desc64(db + 2 * kk), idesc, (kb | kk) != 0);
                        else
                            umma_f16_ta(tmem, a + 8 * kk, desc64(db + 2 * kk), idesc, (kb | kk) != 0);
                    }
                    if (PAIR)
                        umma2_commit(&empty[s]);
                    else
                        umma_commit(bar + to_empty);
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
        if (warp == 2 || !P.group) {
            int s = 0, f = 0, e = 0;  // stage; barrier of this super-block, of the one that had the stage before
            uint32_t ph = 0;
            for (int b = 0; b < nb; b++) {
                if (b >= WS) {
                    wait(&wempty[e], ph, abort_flag);
                    if (++e == WB) {
                        e = 0;
                        ph ^= 1;
                    }
                }
                __syncwarp();
                uint8_t *dst = smem + C::kOffW + s * C::kWBytes;
                if (QT == 4 || P.group) {
                    if (leader) {
                        mbar_expect_tx(&wfull[f], C::kWBytes);
                        if (QT == 4) {
                            tma_load_2d(dst, &wmap, (b0 + b) * kQ4KBlock, n0, &wfull[f]);  // rows past N arrive as zeros
                        } else {
                            for (int j = 0; j < P.group; j++)
                                tma_load_2d(dst + (j * kRows / P.group) * kQ6Slot, &wmap, ((j * P.bpr + b0 + b) * kQ6KBlock) & ~15, n0 / P.group,
                                            &wfull[f]);
                        }
                    }
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
                    cp_async_arrive(&wfull[f]);
                }
                if (++s == WS) s = 0;
                if (++f == WB) f = 0;
            }
            if (QT == 6 && !P.group) asm volatile("cp.async.wait_all;" ::: "memory");
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
        // Q6_K: where the row's blocks lie in a stage, and the bytes (mod 16) by which they are off
        const uint8_t *row = nullptr;
        uint32_t row_addr = 0;
        if (QT == 6) {
            const int rg = P.group ? r & (P.group - 1) : 0;
            row = smem + C::kOffW + (P.group ? (rg * (kRows / P.group) + r / P.group) * kQ6Slot : r * kQ6Pitch);
            row_addr = P.group ? (uint32_t)(rg * P.bpr + b0) * kQ6KBlock
                               : (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(P.w)) + ((uint32_t)(n0 + r) * (uint32_t)P.bpr + b0) * kQ6KBlock) & 3u;
        }
        const uint32_t off_mask = P.group ? 15u : 3u;
        for (int j = 0; j < units; j += kGroups) {
            const int G = min(kGroups, units - j), u = j + g;
            if (g >= G) break;
            const int sb = u >> 1, half = u & 1, ws = sb % WS, wb = sb % WB;
            wait(&wfull[wb], (sb / WB) & 1, abort_flag);
            __syncwarp();
            const uint8_t *blk = smem + C::kOffW + ws * C::kWBytes;
            uint32_t o[16];
            if (QT == 4) {
                blk += r * kQ4KBlock;
                const uint4 hdr = *reinterpret_cast<const uint4 *>(blk);
                uint4 qv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) qv[i] = *reinterpret_cast<const uint4 *>(blk + 16 + 64 * half + 16 * i);
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[wb]);
                const float d = __half2float(__ushort_as_half(static_cast<unsigned short>(hdr.x)));
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int it = 2 * j + c * G + g;
                    uint32_t sc2, m2, ta = 0;
                    q4k_scale_pair(hdr.y, hdr.z, hdr.w, 2 * half + c, sc2, m2);
                    const uint32_t sc = small_half2(sc2), m = small_half2(m2), minus_dmin = (hdr.x >> 16) ^ 0x8000u;
                    const uint32_t wq[8] = {qv[2 * c].x, qv[2 * c].y, qv[2 * c].z, qv[2 * c].w,
                                            qv[2 * c + 1].x, qv[2 * c + 1].y, qv[2 * c + 1].z, qv[2 * c + 1].w};
                    round_q4<false>(wq, sc, d, mixed_fma<false, false>(m, minus_dmin, 0.0f), o);
                    ta = stage_free(it);
                    tmem_st16(ta, o);
                    round_q4<true>(wq, sc >> 16, d, mixed_fma<true, false>(m, minus_dmin, 0.0f), o);
                    tmem_st16(ta + 16, o);
                    publish(it);
                }
            } else {
                const uint32_t off = (row_addr + sb * kQ6KBlock) & off_mask;
                const uint8_t *words = row + ws * C::kWBytes + (off & 12u);
                RawQ6 raw;
                if (__any_sync(0xffffffffu, off & 2u)) raw.load<true>(words, off & 2u, half); else raw.load<false>(words, 0, half);
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[wb]);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int it = 2 * j + c * G + g;
                    uint32_t ta = 0;
#pragma unroll
                    for (int h = 0; h < 2; h++) {  // thirty-two-group 2 c + h of the half, two scales
                        round_q6(raw, c, h, o);
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
            switch (splits) {
                case 2: add_splits<2, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane); break;
                case 3: add_splits<3, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane); break;
                case 4: add_splits<4, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane); break;
                case 5: add_splits<5, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane); break;
                case 6: add_splits<6, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane); break;
                default: add_splits<8, BT>(cl, smem, P, split, n0, t0, warp - C::kDq0, lane);
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

template <int QT, int BT, bool PAIR>
void attr()
{
    static bool done[kMaxDevices] = {false};  // the opt-in is a per-device attribute
    if (done[current_device()]) return;
    cudaFuncSetAttribute(gemm_dense_kernel<QT, BT, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<QT, BT, PAIR>::kSmem);
    done[current_device()] = true;
}

// CTAs that run at a time when clusters of `s` have to find room in one GPC each: 148, 148, 135, 132, 130, 132, -, 120 for one CTA per SM.
// By size of the cluster, for the current device, which a call asks for once: asking is a call of the runtime.
const int *clustered_ctas()
{
    static int known[kMaxDevices][kMaxSplit + 1] = {};
    int *n = known[current_device()];
    for (int s = n[kMaxSplit] ? kMaxSplit + 1 : 1; s <= kMaxSplit; s++) {
        attr<4, 64, false>();
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMaxSplit, 1, s);
        cfg.blockDim = dim3(Cfg<4, 64, false>::kThreads);
        cfg.dynamicSmemBytes = Cfg<4, 64, false>::kSmem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = s;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, gemm_dense_kernel<4, 64, false>, &cfg) != cudaSuccess) cudaGetLastError();
        n[s] = clusters > 0 ? clusters * s : device_sms() / s * s;
    }
    return n;
}

struct Plan {
    int bt, splits;
    bool pair;
};
// The cheapest form by a cost model in ns, fitted to 21 shapes x all forms of either type (1.5 % above the best form on average, 17 % at
// most; by SM cycles and 148 CTAs for whatever clusters it was up to 2.2 times the best: 128 CTAs in clusters of eight are two waves).
// A wave costs its longest tile -- super-blocks by token tile -- plus a start and an end that grow with the tile and with how much
// of the GPU is started; adding up splits comes on top.
Plan plan(int qt, int M, int N, int K)
{
    static const struct {
        int sb, fixed, fill;
    } kCost[2][4] = {{{740, 0, 3500}, {780, 1800, 3200}, {1190, 3600, 3600}, {1180, 3600, 3600}},    // Q4_K: 64, 128, 256 tokens, a pair
                     {{810, 0, 4400}, {960, 800, 4600}, {1210, 3100, 5200}, {1200, 3100, 5200}}};  // Q6_K
    const int sms = device_sms(), bpr = K / 256, row_tiles = (N + kRows - 1) / kRows;
    const int *ctas = clustered_ctas();
    Plan best{256, 1, true};
    long best_cost = -1;
    auto offer = [&](int form, int s) {
        const bool pair = form == 3;
        const int bt = pair ? 256 : 64 << form, rows = pair ? row_tiles + (row_tiles & 1) : row_tiles;
        const long tiles = (long)rows * ((M + bt - 1) / bt) * s, room = ctas[pair ? 2 : s];
        if (s > 1 && tiles > room) return;
        const auto &c = kCost[qt == 6][form];
        const long cost = (tiles + room - 1) / room * ((long)(bpr + s - 1) / s * c.sb + c.fixed + c.fill * (tiles < sms ? tiles : sms) / sms) +
                          (s > 1 ? 1250 + 50 * s : 0);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = {bt, s, pair};
        }
    };
    offer(3, 1);
    for (int form = 2; form >= 0; form--)
        for (int s : {1, 2, 3, 4, 5, 6, 8})
            if (s <= bpr) offer(form, s);
    return best;
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
    Params P{static_cast<const uint8_t *>(w), out, M, N, K / 256, 0, pdl_enabled(), device_error_word()};
    CUtensorMap wmap = {};
    if (QT == 6 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
        P.group = q6k_group(P.bpr);
        if (N % P.group) P.group = 0;
    }
    if ((QT == 4 && !encode_q4k_rows(&wmap, w, P.bpr, N, 1, 0, kRows)) || (P.group && !encode_q6k_groups(&wmap, w, P.bpr, P.group, N, 1, 0, kRows))) {
        fprintf(stderr, "[mnemo_b200] %s: a tensor map could not be encoded\n", where);
        return MB200_ERR_ARG;
    }
    const Plan p = plan(QT, M, N, K);
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
    (void)clustered_ctas();
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
