// True float32 products on the tensor cores: a float32 number is the sum of three bfloat16 numbers
// (hi + mid + lo, 8 bits each, every rest exact), a product of two such sums is nine products that the
// tensor cores form exactly, and the three smallest of them (mid lo, lo mid, lo lo: below 2^-26 of
// the whole) are left out. What is not finite has no such sum: hi is then infinite or NaN and the rests
// NaN, so that the result is not finite either, which the callers look for. bfloat16 numbers end at 2^-133, so that
// what is below 2^-110 would keep fewer bits: numbers are taken S3_UP times before they are cut (every float32
// number then has all of its parts), and what they were multiplied into S3_DOWN times for each of them after.
#pragma once
#include "tcgen.cuh"

#define S3_UP 0x1p24f
#define S3_DOWN 0x1p-24f

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
// Whether one of two packed bfloat16 numbers is infinite or NaN.
__device__ __forceinline__ bool s3_odd2(uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ bool s3_odd8(uint4 w) { return s3_odd2(w.x) || s3_odd2(w.y) || s3_odd2(w.z) || s3_odd2(w.w); }
// The parts of S3_UP v, every part finite, for products whose masked terms must stay zero: what is not finite, or not S3_UP
// times, is taken for 0, and a number that rounds past the largest bfloat16 has its hi cut instead. Bit 0 of the result:
// there was a number that is not finite; bit 1: one that is too large.
__device__ __noinline__ int s3_mend8(const float* v, uint32_t* hi, uint32_t* mid, uint32_t* lo) {
    const float inf = __int_as_float(0x7f800000);
    int odd = 0;
    for (int i = 0; i < 8; ++i) {
        float x = v[i] * S3_UP;
        if (!(fabsf(x) < inf)) {
            odd |= fabsf(v[i]) < inf ? 2 : 1;
            x = 0.f;
        }
        uint32_t h = __float_as_uint(__bfloat162float(__float2bfloat16_rn(x)));
        if ((h & 0x7f800000u) == 0x7f800000u) h = __float_as_uint(x) & 0xffff0000u;
        const float r = x - __uint_as_float(h);
        const uint32_t m = __float_as_uint(__bfloat162float(__float2bfloat16_rn(r)));
        const uint32_t l = __float_as_uint(__bfloat162float(__float2bfloat16_rn(r - __uint_as_float(m))));
        const int at = 16 * (i & 1);
        hi[i >> 1] = at ? hi[i >> 1] | h : h >> 16;
        mid[i >> 1] = at ? mid[i >> 1] | m : m >> 16;
        lo[i >> 1] = at ? lo[i >> 1] | l : l >> 16;
    }
    return odd;
}
// ... of numbers that are bfloat16 numbers already.
__device__ __forceinline__ bool s3_finite8(uint4& v) {
    if (!s3_odd8(v)) return false;
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if ((w[i] & 0x7f80u) == 0x7f80u) w[i] &= 0xffff0000u;
        if ((w[i] & 0x7f800000u) == 0x7f800000u) w[i] &= 0xffffu;
    }
    v = make_uint4(w[0], w[1], w[2], w[3]);
    return true;
}
__device__ __forceinline__ void s3_store16(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Generic stores to shared memory, made visible to the products that read them.
__device__ __forceinline__ void s3_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// A 16-byte piece's place in a tile of 128-byte rows with the 128-byte swizzle.
__device__ __forceinline__ uint32_t s3_place(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); }
// S3_UP times R eights to their places dst[r], dst[r] + step, dst[r] + 2 step with every part finite; true: a number was not
// finite, or too large (2^103 and more), and lies there as 0. Of the latter the smallest row goes to *too_large. One test for
// all of them, so that their chains of conversions run side by side.
template <int R>
__device__ __forceinline__ bool s3_put(const float (&v)[R][8], const uint32_t (&dst)[R], uint32_t step, const int (&row)[R], int* too_large) {
    uint4 part[R][3];
    // the rest of what is not finite, or rounds to infinity, is not finite: 0 times it is not 0
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
    uint32_t any = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float up[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) up[i] = v[r][i] * S3_UP;
        s3_split8(up, part[r][0], part[r][1], part[r][2]);
        __nv_bfloat162 a = __hmul2(*(const __nv_bfloat162*)&part[r][1].x, zero), b = __hmul2(*(const __nv_bfloat162*)&part[r][1].y, zero);
        a = __hfma2(*(const __nv_bfloat162*)&part[r][1].z, zero, a);
        b = __hfma2(*(const __nv_bfloat162*)&part[r][1].w, zero, b);
        any |= (*(const uint32_t*)&a | *(const uint32_t*)&b) & 0x7fff7fffu;
    }
    bool odd = false;
    if (any) {
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            float f[8];
            uint32_t w[3][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                f[i] = v[0][i];
#pragma unroll
                for (int q = 1; q < R; ++q) f[i] = r == q ? v[q][i] : f[i];
            }
            uint32_t to = dst[0];
            int at = row[0];
#pragma unroll
            for (int q = 1; q < R; ++q) {
                to = r == q ? dst[q] : to;
                at = r == q ? row[q] : at;
            }
            const int what = s3_mend8(f, w[0], w[1], w[2]);
            if (what & 2) atomicMin(too_large, at);
            odd = what != 0 || odd;
#pragma unroll
            for (int q = 0; q < 3; ++q) s3_store16(to + q * step, make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]));
        }
        return odd;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) s3_store16(dst[r] + q * step, part[r][q]);
    return false;
}
__device__ __forceinline__ bool s3_put8(const float (&v)[8], uint32_t dst, uint32_t step, int row, int* too_large) {
    float f[1][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[0][i] = v[i];
    const uint32_t to[1] = {dst};
    const int at[1] = {row};
    return s3_put<1>(f, to, step, at, too_large);
}
// D += A B^T over 16 KSTEPS of k and every kept pair of parts, the smallest first. Part p of A starts a_part * p
// after da and a k-step a_k after the one before (descriptor units of 16 bytes); AP, BP: parts there are (1: the
// numbers are bfloat16 numbers themselves). One thread issues.
template <int AP, int BP, int KSTEPS>
__device__ __forceinline__ void s3_products(uint32_t d, uint64_t da, uint32_t a_part, uint32_t a_k, uint64_t db, uint32_t b_part,
                                            uint32_t b_k, uint32_t idesc, bool more) {
    uint32_t acc = more ? 1u : 0u;
#pragma unroll
    for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int p = 0; p < AP; ++p) {
            const int q = sum - p;
            if (q < 0 || q >= BP) continue;
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) {
                tg_mma(d, da + (uint64_t)(a_part * p + a_k * k), db + (uint64_t)(b_part * q + b_k * k), idesc, acc);
                acc = 1u;
            }
        }
}
