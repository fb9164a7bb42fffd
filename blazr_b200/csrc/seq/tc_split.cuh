// tc_split.cuh -- products of f32 operands on the tensor cores of one SM: every operand in three bf16 parts (x = x1 + x2 + x3, 24 bits), a product as
// the six tcgen05.mma products that matter, smallest first (seq_attn_tc.cu says why).  Wrappers, splits and operand descriptors.
#pragma once
#include "tc_pair.cuh"

namespace tcsplit {

using namespace tcpair;

__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void commit_one(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                 "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void ld16(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void async_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// packed pairs of f32 (one instruction for both)
__device__ __forceinline__ uint64_t pk(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// two values -> three packed bf16 pairs (low half = a); a value without finite parts has a NaN among them
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(b), "f"(a));
    float ra, rb, sa_, sb_;
    const uint64_t minus1 = pk(-1.f, -1.f);
    upk(fma2(pk(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xFFFF0000u)), minus1, pk(a, b)), ra, rb);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(rb), "f"(ra));
    upk(fma2(pk(__uint_as_float(p2 << 16), __uint_as_float(p2 & 0xFFFF0000u)), minus1, pk(ra, rb)), sa_, sb_);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p3) : "f"(sb_), "f"(sa_));
}
// a pair of values -> three packed bf16 pairs by truncation (toward zero, either sign): 8 + 8 + 8 significant bits, no conversion instruction
__device__ __forceinline__ void cut2(float x, float y, uint64_t minus1, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const float x1 = __uint_as_float(__float_as_uint(x) & 0xFFFF0000u), y1 = __uint_as_float(__float_as_uint(y) & 0xFFFF0000u);
    float rx, ry, sx, sy;
    upk(fma2(pk(x1, y1), minus1, pk(x, y)), rx, ry);
    const float x2 = __uint_as_float(__float_as_uint(rx) & 0xFFFF0000u), y2 = __uint_as_float(__float_as_uint(ry) & 0xFFFF0000u);
    upk(fma2(pk(x2, y2), minus1, pk(rx, ry)), sx, sy);
    p1 = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    p2 = __byte_perm(__float_as_uint(rx), __float_as_uint(ry), 0x7632);
    p3 = __byte_perm(__float_as_uint(sx), __float_as_uint(sy), 0x7632);
}
__device__ __forceinline__ void sts8(uint32_t addr, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory"); }
// mn-major operand, 128-byte swizzle: rows (k) of 128 bytes = 64 consecutive mn, 8-row groups 1024 bytes apart, the next 64 mn `lbo` bytes on
__device__ __forceinline__ uint64_t desc_mn128(uint32_t a, uint32_t lbo) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

}  // namespace tcsplit
