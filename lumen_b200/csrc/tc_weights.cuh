// Arithmetic that the tcgen05 prefill kernels on CTA pairs (prefill_pair.cu) and on single CTAs (prefill_tc.cu) share: the results of an
// expert-parallel call are one GPU's to the bit because both take their SwiGLU from here and unpack weights as here
// (prefill_tc.cu has store_weights written out, see dequant_store there; tests compare the two forms' outputs).
#pragma once
#include "mma_frag.cuh"
#include "tc_common.cuh"

namespace lumen {
namespace tc {

__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Eight weights of a row, scale folded in with one rounding, to 16 bytes of an operand. Q4_0: w0 holds their nibbles; Q8_0: w0 elements
// 4t.., w1 elements 16+4t.. of the block. scale: the block's f16 scale in both halves. Issued for every weight of a call, so its
// instructions are counted: 1 shift, 4 logic, 4 subtract, 4 multiply, 1 store with a constant offset.
template <int Q>
__device__ __forceinline__ void store_weights(uint32_t addr, uint32_t w0, uint32_t w1, uint32_t scale, const UnpackConst& k) {
    uint32_t l0, l1, h0, h1;
    if constexpr (Q == Q4_0) {
        const uint32_t x = w0, y = x >> 8;
        l0 = hsub2_u32(lop_and_or(x, 0x000F000Fu, k.or_a), k.sub_a);
        h0 = hsub2_u32(lop_and_or(x, 0x00F000F0u, k.or_b), k.sub_b);
        l1 = hsub2_u32(lop_and_or(y, 0x000F000Fu, k.or_a), k.sub_a);
        h1 = hsub2_u32(lop_and_or(y, 0x00F000F0u, k.or_b), k.sub_b);
    } else {
        // bytes biased by 128 -> unsigned; 0x64xx = 1024 + xx; subtract 1152.
        const uint32_t x = w0 ^ k.or_b, y = w1 ^ k.or_b;
        l0 = hsub2_u32(prmt(x, k.or_a, 0x4240u), k.sub_a);
        l1 = hsub2_u32(prmt(x, k.or_a, 0x4341u), k.sub_a);
        h0 = hsub2_u32(prmt(y, k.or_a, 0x4240u), k.sub_a);
        h1 = hsub2_u32(prmt(y, k.or_a, 0x4341u), k.sub_a);
    }
    sts128(addr, hmul2_u32(l0, scale), hmul2_u32(h0, scale), hmul2_u32(l1, scale), hmul2_u32(h1, scale));
}

// SwiGLU (cuda/shaders/moe_expert.cu:47-50), g / (1 + e^-g) * u, on the approximate exp2 and reciprocal units: their error
// (~2^-21) is far below the f16 rounding of the result that follows. The epilogue of a wide tile is exposed, so its
// instructions count; the range fix-ups of the library forms are not needed here (e^-g = inf gives 0, as it should; a
// reciprocal below 2^-126 may flush to 0).
__device__ __forceinline__ float swiglu_fast(float g, float u) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r * u;
}

}  // namespace tc
}  // namespace lumen
