// 5th-generation tensor core (tcgen05) helpers for sm_100a: tensor memory
// allocation, shared-memory matrix descriptors, the BF16 x BF16 -> FP32 MMA,
// commits to mbarriers, tensor-memory loads, and tiled TMA loads.
//
// Shared-memory operand layouts (16-byte units "u", CB = elements per row of
// a staged box: 32 bf16 = 64 B rows with 64-byte swizzle, 64 bf16 = 128 B
// rows with 128-byte swizzle; the TMA writes exactly these layouts):
//   K-major  (rows = M or N, K contiguous):  8-row atoms of CB elements,
//            atom stride SBO = 8 * row bytes; one MMA (K = 16) reads 32 bytes
//            of every row, the next K step starts 32 bytes further.
//   MN-major (rows = K, M or N contiguous): CB-element groups (LBO apart),
//            8-row atoms SBO = 8 * row bytes apart; one MMA reads 16 rows,
//            the next K step starts 16 rows further.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace fmvd {
namespace umma {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Swizzle code of the descriptor's layout field for a row of 'row_bytes'.
__host__ __device__ constexpr uint32_t layout_code(int row_bytes) { return row_bytes == 128 ? 2u : 4u; }

// Shared-memory matrix descriptor (version 1, base offset 0, legacy LBO
// mode): start, leading and stride byte offsets in 16-byte units.  Kept as two
// words: the start address (below 256 KB, so it never carries out of its
// field) is in the lower one, and moving an operand by b bytes adds b / 16.
struct Desc {
    uint32_t lo, hi;
    __device__ __forceinline__ Desc operator+(uint32_t bytes) const { return Desc{lo + bytes / 16, hi}; }
};
__device__ __forceinline__ Desc make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, int row_bytes)
{
    return Desc{(saddr >> 4) | ((lbo_bytes >> 4) << 16),
                (sbo_bytes >> 4) | (1u << 14) /* descriptor version for sm_100 */ | (layout_code(row_bytes) << 29)};
}

// Instruction descriptor of kind::f16: BF16 A and B, FP32 accumulator,
// M x N tile, operand majors (0 = K-major, 1 = MN-major).
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, int a_mn_major, int b_mn_major)
{
    return (1u << 4)                        // D format F32
           | (1u << 7)                      // A format BF16
           | (1u << 10)                     // B format BF16
           | ((uint32_t)a_mn_major << 15)   // A major
           | ((uint32_t)b_mn_major << 16)   // B major
           | ((uint32_t)(N >> 3) << 17)     // N / 8
           | ((uint32_t)(M >> 4) << 24);    // M / 16
}

// ---- tensor memory (one warp, all lanes) ----------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- MMA (a whole, converged warp; an elected lane issues) -------------------
// The role's code runs on every lane, so that descriptors and addresses stay
// warp-uniform, and elect.sync picks the lane that issues.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, Desc a, Desc b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),
        "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The mbarrier receives one arrival when every MMA the elected lane issued before
// has completed (and released its shared-memory operands).
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
        : "memory");
}
// This thread's warp, as a value the compiler knows to be the same on all lanes.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// ---- 32-byte global accesses (p on a 32-byte boundary) -----------------------
__device__ __forceinline__ void ldg32(const void *p, uint32_t (&r)[8])
{
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(p));
}
__device__ __forceinline__ void stg32(void *p, const uint32_t (&r)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// ---- tensor memory -> registers (warp w reads lanes 32 (w % 4) ..) ---------
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++)
        v[i] = __uint_as_float(r[i]);
}

// ---- mbarriers and TMA -------------------------------------------------------
__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded wait: false after max_spins polls.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity, int max_spins = 1 << 24)
{
    for (int i = 0; i < max_spins; i++) {
        if (bar_try_wait(bar, parity))
            return true;
        if (i > 64)
            __nanosleep(32);
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                            uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_addr(bar))
        : "memory");
}

} // namespace umma
} // namespace fmvd
