// What the float kernels on the tensor cores share (gemm_f32_tc.cu, attention_f32_tc.cuh): a float as three bfloat16 numbers, x = h + m + l
// exactly, pairs of floats, and short loads and stores of tensor memory.
#pragma once

#include "float_pairs.cuh"
#include "ptx.cuh"

namespace bg {

// Two floats into their three parts, two bfloat16 a word (the first one low): exact for multiples of 2^-133, parts that are not numbers for
// what is infinite, not a number, or next to the largest float.
__device__ __forceinline__ unsigned gt_pack(unsigned long long v) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(high2(v)), "f"(low2(v)));
    return r;
}
__device__ __forceinline__ unsigned long long gt_unpack(unsigned p) {
    return (unsigned long long)(p << 16) | ((unsigned long long)(p & 0xffff0000u) << 32);
}
__device__ __forceinline__ void gt_split(unsigned long long v, unsigned& h, unsigned& m, unsigned& l) {
    const unsigned long long minus = pair2(-1.0f, -1.0f);
    h = gt_pack(v);
    const unsigned long long r = fma2(gt_unpack(h), minus, v);
    m = gt_pack(r);
    const unsigned long long q = fma2(gt_unpack(m), minus, r);
    l = __byte_perm((unsigned)q, (unsigned)(q >> 32), 0x7632);
}
// Both floats times a power of two (one by one: packed, the multiplication makes float attention slower by a tenth).
__device__ __forceinline__ unsigned long long gt_up(unsigned long long v, float up) { return pair2(low2(v) * up, high2(v) * up); }
__device__ __forceinline__ unsigned long long gt_add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Loads and stores of tensor memory; the caller waits.
__device__ __forceinline__ void gt_ld8(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void gt_ld16(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void gt_st4(unsigned taddr, const unsigned (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// The registers of a thread of this warpgroup, from HAS at launch to WANTS.
template <int HAS, int WANTS>
__device__ __forceinline__ void gt_regs() {
    if constexpr (WANTS > HAS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(WANTS));
    if constexpr (WANTS < HAS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(WANTS));
}

}  // namespace bg
