// Building blocks shared by the tcgen05 kernels (grouped expert GEMMs, router-logits GEMM):
// mbarrier waits with a bound, shared-memory / instruction descriptors of K-major
// SWIZZLE_128B operands, tcgen05.mma / commit / ld wrappers, and the tensor-map encoder.
#pragma once
#include "moe_internal.cuh"
#include <cuda.h>

namespace lumen {
namespace tc {

constexpr int SUB_BYTES = 128 * 128;  // [128 rows x 64 k] f16, 128-byte rows, SWIZZLE_128B
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait. Returns false when another role aborted or the limit expired
// (in which case it raises the abort flag itself).
struct AbortCtl {
    volatile uint32_t* flag;  // CTA-wide abort flag in shared memory
    uint64_t limit_ns;
};
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const AbortCtl& ac) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t i = 0;; ++i) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*ac.flag) return false;
            if (globaltimer_ns() - t0 > ac.limit_ns) {
                *ac.flag = 1u;
                return false;
            }
        }
    }
}

// A role that gives up does not leave while its copies are on their way into shared memory: of the phases up to number n - 1
// that it has asked for on the ring of barriers at bar0, every step-th, those that the ring can still hold, each complete or the
// limit over (a phase that other roles have a part in may stay incomplete for good).
__host__ __device__ constexpr int first_to_land(int n, int stages, int step) {
    return n <= 0 ? n : n > stages ? n - stages + step - 1 : (n - 1) % step;
}
static_assert(first_to_land(0, 4, 2) == 0 && first_to_land(1, 4, 2) == 0 && first_to_land(2, 4, 2) == 1 && first_to_land(3, 4, 2) == 0, "");
static_assert(first_to_land(4, 4, 2) == 1 && first_to_land(5, 4, 2) == 2 && first_to_land(48, 4, 2) == 45, "");  // 45 and 47
static_assert(first_to_land(0, 4, 1) == 0 && first_to_land(3, 4, 1) == 0 && first_to_land(9, 4, 1) == 5, "");
__device__ __forceinline__ void let_land(uint32_t bar0, int stages, int n, int step = 1) {
    const uint64_t t0 = globaltimer_ns();
    for (int q = first_to_land(n, stages, step); q < n; q += step)
        while (!mbar_try(bar0 + (q % stages) * 8, (q / stages) & 1) && globaltimer_ns() - t0 < 1000000ull) {
        }
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
    // K-major, SWIZZLE_128B: 8-row groups 1024 B apart (SBO), LBO unused (1), descriptor version 1
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// One lane of a converged warp, the form in which the tcgen05 instructions are issued: the code around
// them stays warp-uniform, so descriptors and addresses live in uniform registers. (Issued from a branch taken by
// lane 0 alone, every tcgen05.mma cost ~95 cycles of operand moves, more than the product itself up
// to 128 columns.)
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ uint32_t make_idesc(int n, bool bf16) {
    const uint32_t fmt = bf16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// 32-byte store (the address must be 32-byte aligned): one whole sector per lane, where a lane's
// piece of a row is all a warp instruction writes of that row
__device__ __forceinline__ void st_global_v8(void* p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
// Orders later uses of registers that an earlier tcgen05.ld fills after the wait for that load (the
// loads are asynchronous; when a load is issued ahead of the wait, arithmetic on its registers must
// not be scheduled above the wait).
__device__ __forceinline__ void tmem_ld_fence8(uint32_t (&r)[8]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])::"memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 2-D tiled copy global -> shared (SWIZZLE_128B box), completion counted in bytes on `bar`
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// contiguous copy global -> shared (16-byte aligned, a multiple of 16 bytes), completion counted in bytes on `bar`
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// test hooks: the phase at hand expects this many bytes more (no arrival)
__device__ __forceinline__ void mbar_expect_more(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

}  // namespace tc

// [rows, cols] f16 row-major -> tensor map with a (64 x box_rows) box and the 128-byte swizzle;
// x (the column) of every copy is a multiple of 64 elements = 128 bytes.
cudaError_t make_tmap_f16(const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out);
// the same for an f16 array of nd <= 5 dimensions (innermost first; strides in bytes, from the second dimension on)
cudaError_t make_tmap_f16_nd(const void* base, int nd, const uint64_t* dims, const uint64_t* strides, const uint32_t* box, CUtensorMap* out,
                             CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B);

}  // namespace lumen
