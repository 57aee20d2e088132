// Packed 32-bit float operations (two floats in a 64-bit register). Each half is rounded on its own, so a packed operation has
// the bits of two scalar ones; it takes one issue slot for both.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>

namespace qtb {

__device__ __forceinline__ unsigned long long pack_f32x2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack_f32x2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long mul_f32x2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long widen_half2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack_f32x2(f.x, f.y);
}
// acc + x y, two F16 products added to two floats: the product of two F16 numbers is exact in F32, so this has the bits of fma_f32x2 on the widened operands,
// without widening them (which, like packed operations, only the heavy half of the FMA pipe does, two cycles an instruction); two instructions, one cycle each.
__device__ __forceinline__ unsigned long long fma_half2_mixed(uint32_t x, uint32_t y, unsigned long long acc) {
    unsigned long long r;
    asm("{\n\t.reg .b16 xl, xu, yl, yu;\n\t.reg .f32 a, b;\n\tmov.b32 {xl, xu}, %1;\n\tmov.b32 {yl, yu}, %2;\n\tmov.b64 {a, b}, %3;\n\tfma.rn.f32.f16 a, xl, yl, a;\n\tfma.rn.f32.f16 b, xu, yu, b;\n\tmov.b64 %0, {a, b};\n\t}"
        : "=l"(r)
        : "r"(x), "r"(y), "l"(acc));
    return r;
}
__device__ __forceinline__ unsigned long long widen_bf162(uint32_t h) { return pack_f32x2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)); }

__device__ __forceinline__ unsigned long long shfl_xor_f32x2(unsigned long long v, int mask) { return __shfl_xor_sync(0xffffffffu, v, mask); }

// One halving step over the thread bit `mask` for the first n of N values: threads with the bit clear keep the first half of
// them, the others the second half, each added to the partner's copy (addition commutes, so both halves have the bits of the
// sum in either order).
template <int N>
__device__ __forceinline__ void halve_f32x2(unsigned long long (&v)[N], int n, int mask, bool upper) {
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
        if (k < n / 2) {
            const unsigned long long keep = upper ? v[k + n / 2] : v[k], send = upper ? v[k] : v[k + n / 2];
            v[k] = add_f32x2(keep, shfl_xor_f32x2(send, mask));
        }
    }
}

}  // namespace qtb
