// Register-level pieces that the mma.sync mat-vec kernels share: shared-memory access by 32-bit address, f16 halves, the multiply.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

namespace mlxn {

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// Loads at a compile-time offset from a register address (the offset travels in the instruction: no address arithmetic)
template <uint32_t OFF> __device__ __forceinline__ uint32_t lds32i(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}
template <uint32_t OFF> __device__ __forceinline__ uint32_t lds_u16i(uint32_t addr) {
    uint32_t v;
    asm volatile("{ .reg .u16 t; ld.shared.u16 t, [%1+%2]; cvt.u32.u16 %0, t; }" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}
template <uint32_t OFF> __device__ __forceinline__ void lds64i(uint32_t addr, uint32_t &a, uint32_t &b) {
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2+%3];" : "=r"(a), "=r"(b) : "r"(addr), "n"(OFF));
}
template <uint32_t OFF> __device__ __forceinline__ void lds128i(uint32_t addr, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d) {
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr), "n"(OFF));
}
template <uint32_t OFF> __device__ __forceinline__ void lds128i(uint32_t addr, uint32_t (&v)[4]) { lds128i<OFF>(addr, v[0], v[1], v[2], v[3]); }
// The f16 in the low / high half of a 32-bit word, as f32
__device__ __forceinline__ float f16lo_to_float(uint32_t w) {
    float f;
    asm("{ .reg .f16 l, h; mov.b32 {l, h}, %1; cvt.f32.f16 %0, l; }" : "=f"(f) : "r"(w));
    return f;
}
__device__ __forceinline__ float f16hi_to_float(uint32_t w) {
    float f;
    asm("{ .reg .f16 l, h; mov.b32 {l, h}, %1; cvt.f32.f16 %0, h; }" : "=f"(f) : "r"(w));
    return f;
}
// f(integral_constant<int, I>) for I = 0 .. N - 1: loop bodies whose shared-memory offsets must be compile-time constants
template <int I, int N, class F> __device__ __forceinline__ void static_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t a) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(a) : "memory");
}

// D = A (16 x 16, row) * B (16 x 8, col) + C, f16 operands, f32 accumulate.  Lane (g = lane / 4, t = lane % 4):
// a0 = A[g][2t, 2t+1], a1 = A[g+8][2t, 2t+1], a2 = A[g][2t+8, 2t+9], a3 = A[g+8][2t+8, 2t+9];
// b0 = B[2t, 2t+1][g], b1 = B[2t+8, 2t+9][g]; c0 = C[g][2t], c1 = C[g][2t+1], c2 = C[g+8][2t], c3 = C[g+8][2t+1].
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

}  // namespace mlxn
