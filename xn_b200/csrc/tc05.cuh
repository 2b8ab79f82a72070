// Building blocks of the tensor-memory kernels: mbarriers, TMA loads, shared-memory matrix descriptors, tcgen05 MMA /
// commit / tensor-memory transfers, and the host-side tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "wait.cuh"

namespace xn {

constexpr int BM = 128;        // rows of A per tile = TMEM lanes
constexpr int BKB = 128;       // bytes of K per stage = one 128-byte swizzle atom
constexpr int UMMA_KB = 32;    // bytes of K per tcgen05.mma (32 x 8-bit or 16 x 16-bit)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// Pull a tensor map (a kernel parameter) into the TMA unit's descriptor cache: the first copy that names it then
// does not start with a fetch of the descriptor.
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_only(uint64_t *b, unsigned bytes) {  // no arrival
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t *b, unsigned parity, const WaitCtx &w) {
    return mbar_wait_bounded(smem_u32(b), parity, w);
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// One thread of a converged warp, chosen with elect.sync.  The roles that issue TMA copies and MMAs run under it rather
// than under `lane == 0`: only then does the compiler know that a single thread is active, and feeds these instructions'
// uniform-register operands directly instead of through a loop over the active lanes.  Issue cost of tcgen05.mma
// (M = 128, K = 32 bytes), in cycles per MMA at N = 16 / 64 / 128 / 192 / 256: 118 / 118 / 118 / 118 / 129 under
// `lane == 0`, 66 / 68 / 72 / 97 / 129 under elect.sync with the descriptors' constant high words (the tensor pipe itself
// needs N / 2).
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }  // known to be uniform

// Shared-memory matrix descriptors, low words; the high word is the same for every operand here:
//   bits 32-45 stride byte offset 1024 (between 8-row groups), bit 46 descriptor version, bits 61-63 SWIZZLE_128B.
// To advance along k add (bytes >> 4) to the low word.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
// K-major tile, 128-byte swizzle (the leading byte offset is unused).
__device__ __forceinline__ uint32_t smem_desc(const void *tile) { return (smem_u32(tile) & 0x3FFFFu) >> 4; }
// MN-major operand (the [K, N] right-hand side of a plain `matmul`, n contiguous): the tile is a row of 64-column blocks,
// each block = BK k-rows of 128 bytes as TMA writes them with the 128-byte swizzle.  Within a block the 8-row groups along
// k are 1024 bytes apart (stride byte offset), the blocks along n `block_bytes` apart (leading byte offset).
__device__ __forceinline__ uint32_t smem_desc_mn(const void *tile, unsigned block_bytes) {
    return ((smem_u32(tile) & 0x3FFFFu) >> 4) | (block_bytes >> 4) << 16;
}

// Instruction descriptor: D = f32, A/B formats, both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t instr_desc(int a_fmt, int b_fmt, int n) {
    return (1u << 4) | ((uint32_t)a_fmt << 7) | ((uint32_t)b_fmt << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(BM >> 4) << 24);
}

template <bool F8>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t a_desc, uint32_t b_desc, uint32_t idesc, uint32_t acc) {
    if (F8)
        asm volatile(
            "{\n.reg .pred p;\n.reg .b64 a, b;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p;\n}" ::"r"(tmem_d),
            "r"(a_desc), "r"(b_desc), "r"(idesc), "r"(acc), "n"(DESC_HI)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\n.reg .b64 a, b;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}" ::"r"(tmem_d),
            "r"(a_desc), "r"(b_desc), "r"(idesc), "r"(acc), "n"(DESC_HI)
            : "memory");
}
__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint32_t a_desc, uint32_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 a, b;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, p;\n}" ::"r"(tmem_d),
        "r"(a_desc), "r"(b_desc), "r"(idesc), "r"(acc), "n"(DESC_HI)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// issue only: the caller waits once for all its loads
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- host side: tensor maps (tmap.cu) ----
// 2-D row-major [rows, k] tensor with `elem` bytes per element and a row pitch of ld elements; box = 128 bytes of k by
// box_rows rows, 128-byte swizzle, out-of-range reads give zeros.
int make_map(CUtensorMap *map, const void *base, int elem, size_t rows, size_t k, size_t ld, int box_rows);
// The same with `batch` matrices batch_stride elements apart (box covers one of them); *batch_inner: see tmap.cu.
int make_map3(CUtensorMap *map, const void *base, int elem, size_t rows, size_t k, size_t ld, int box_rows, size_t batch,
              size_t batch_stride, int *batch_inner);
// [k, n] operand with n contiguous, 16-bit elements; box 64 n x 64 k.
int make_map_mn(CUtensorMap *map, const void *base, size_t n, size_t k, size_t ld, size_t batch, size_t batch_stride,
                int *batch_inner);

}  // namespace xn
