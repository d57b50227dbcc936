// tcgen05 / TMEM / TMA instruction wrappers shared by the tensor-core kernels.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace mb200 {

// PAIR = true: the cta_group::2 forms, for the two CTAs of a cluster that work on one M = 256 tile (both execute them).
template <bool PAIR = false>
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols)
{
    if (PAIR) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <bool PAIR = false>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    if (PAIR)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
    else
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// kind::f16 instruction descriptor: fp16 x fp16 -> fp32, both operands K-major, M x N
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n)
{
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
// The instruction takes its operands from uniform registers, and how the issuing code looks to the compiler decides the rate.
// A warp that stays converged through the loop and its barrier waits, with all MMAs of a step inside one
// `if (leader)` (leader from elect_lane(), addresses from warp_uniform()), issues an M128 x N32 x K16 every 16.6 cycles, the
// tensor core's own rate. With the whole loop inside a one-thread branch every operand is moved to a uniform register for
// every instruction: 94 cycles, whatever N <= 128; with the leader as a predicate of each instruction: 50-60.
__device__ __forceinline__ uint32_t elect_lane()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p;
}
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
// A operand in tensor memory (128 lanes = rows, two fp16 per 32-bit column), B operand through a shared-memory descriptor.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same over two CTAs, issued by the first: M = 256, each CTA holds its 128 rows of A and D in its own TMEM and half of B's
// N rows in its shared memory (same addresses in both).
__device__ __forceinline__ void umma2_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 consecutive 32-bit columns of this thread's TMEM lane (lane = 32 * (warp % 4) + lane id)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st1(uint32_t taddr, uint32_t r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(r) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint32_t bar)  // bar: address in shared memory
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) { umma_commit(smem_u32(bar)); }
__device__ __forceinline__ void umma2_commit(uint64_t *bar)  // arrives at this barrier of both CTAs
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "h"(static_cast<unsigned short>(3))
                 : "memory");
}
// Arrives at the same barrier in CTA 0 of the cluster. What it announces is tensor memory and TMA-written shared memory, ordered
// by the tcgen05 fences and the barriers it was seen through; a .release.cluster arrive would wait for every store of the
// thread to be visible cluster-wide first, 1000 cycles and more.
__device__ __forceinline__ void mbar_arrive_cta0(uint64_t *bar)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// tmem_ld16 in two steps, so that two loads are under way together; the values must not be touched between them
__device__ __forceinline__ void tmem_ld16_start(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16_finish(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst_smem, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst_smem)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst_smem, const CUtensorMap *map, int x, int y, int z, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst_smem)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(void *dst_smem, const CUtensorMap *map, int x, int y, int z, int w, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            smem_u32(dst_smem)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor: K-major tile, 128-byte swizzle, rows of 128 bytes, 8-row
// groups 1024 bytes apart (SBO); the tile base is 1024-byte aligned (base offset 0).
// Its low half (start address in 16-byte units, leading-dimension offset unused for swizzled K-major) may be added to as it is, 32 bits.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint64_t desc64(uint32_t lo)
{
    constexpr uint32_t hi = (1024u >> 4)    // stride-dimension offset
                            | (1u << 14)    // descriptor version (sm_100)
                            | (2u << 29);   // SWIZZLE_128B
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Waits inside the GEMMs. After one that ran out (bounded_wait.cuh) the roles run through their loops on whatever the buffers hold (all
// addresses stay in bounds) and the kernel reports the timeout. (try_wait with a time limit sleeps in between: 10 % slower.)
// Asking costs issue slots that the dequantising warps need: PATIENT waits (the loaders', which run stages ahead) pause in between.
template <bool PATIENT = false>
__device__ __forceinline__ void wait(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    bounded_wait([=] { return mbar_try_wait(bar, parity); }, [] { if (PATIENT) __nanosleep(100); }, abort_flag);
}
template <bool PATIENT = false>
__device__ __forceinline__ void wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    wait<PATIENT>(smem_u32(bar), parity, abort_flag);
}

constexpr int kQ6Slot = 240;  // bytes of a Q6_K block in a stage: 15 x 16, an odd number, so that the rows of a warp spread over all banks

// ---- host: tensor maps ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled();  // the driver's cuTensorMapEncodeTiled, or null (gemm_dense.cu)

// fp16 [rows][K] row-major, boxes of box_rows rows x 64 columns with the 128-byte swizzle
inline bool encode_f16_rows(CUtensorMap *map, const void *x, int K, size_t rows, int box_rows)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Q4_K matrices of `mats` equal tensors mat_stride bytes apart as one byte tensor (block column, row[, tensor]); boxes of
// box_rows rows x one 144-byte block. A block column starts at a multiple of 144 = 9 x 16 bytes.
inline bool encode_q4k_rows(CUtensorMap *map, const void *w, int bpr, size_t rows, int mats, size_t mat_stride, int box_rows)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(bpr) * kQ4KBlock, rows, static_cast<cuuint64_t>(mats)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(bpr) * kQ4KBlock, mat_stride};
    const cuuint32_t box[3] = {kQ4KBlock, static_cast<cuuint32_t>(box_rows), 1}, estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, mat_stride ? 3 : 2, const_cast<void *>(w), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Q6_K: rows of 210-byte blocks have no stride a tensor map can take, but 1, 2, 4 or 8 rows together are a multiple of 16 bytes. Row j of
// every such group is a box of its own, from the last multiple of 16 before its block: all of the box's rows are off by the same bytes.
inline int q6k_group(int bpr) { return bpr % 8 == 0 ? 1 : bpr % 4 == 0 ? 2 : bpr % 2 == 0 ? 4 : 8; }
inline bool encode_q6k_groups(CUtensorMap *map, const void *w, int bpr, int group, int rows, int mats, size_t mat_stride, int box_rows)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t bytes = static_cast<cuuint64_t>(bpr) * kQ6KBlock * group;
    const cuuint64_t dims[3] = {bytes, static_cast<cuuint64_t>(rows / group), static_cast<cuuint64_t>(mats)}, strides[2] = {bytes, mat_stride};
    const cuuint32_t box[3] = {kQ6Slot, static_cast<cuuint32_t>(box_rows / group), 1}, estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, mat_stride ? 3 : 2, const_cast<void *>(w), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace mb200
