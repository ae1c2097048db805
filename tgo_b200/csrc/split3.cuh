// True float32 products on the tensor cores: a float32 number is the sum of three bfloat16 numbers
// (hi + mid + lo, 8 bits each, every rest exact), a product of two such sums is nine products that the
// tensor cores form exactly, and the three smallest of them (mid lo, lo mid, lo lo: below 2^-26 of
// the whole) are left out. What is not finite has no such sum: hi is then infinite or NaN and the rests
// NaN, so that the result is not finite either, which the callers look for.
#pragma once
#include "tcgen.cuh"

// The three parts of two neighbouring numbers, each part's two packed in one word. A number that rounds
// past the largest bfloat16 gets an infinite hi.
__device__ __forceinline__ void s3_split2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = tg_pack(a, b);
    const float ra = a - __uint_as_float(hi << 16), rb = b - __uint_as_float(hi & 0xffff0000u);
    mid = tg_pack(ra, rb);
    lo = tg_pack(ra - __uint_as_float(mid << 16), rb - __uint_as_float(mid & 0xffff0000u));
}
// Eight neighbouring numbers: a 16-byte piece of each part.
__device__ __forceinline__ void s3_split8(const float (&v)[8], uint4& hi, uint4& mid, uint4& lo) {
    s3_split2(v[0], v[1], hi.x, mid.x, lo.x);
    s3_split2(v[2], v[3], hi.y, mid.y, lo.y);
    s3_split2(v[4], v[5], hi.z, mid.z, lo.z);
    s3_split2(v[6], v[7], hi.w, mid.w, lo.w);
}
__device__ __forceinline__ void s3_store16(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Generic stores to shared memory, made visible to the products that read them.
__device__ __forceinline__ void s3_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
