// Register-tiled float32 products from shared memory, for the chunk-wise recurrences: an output
// tile [4 TY RM][4 TX RN] over TY x TX threads, A and B both k-major in shared memory. Thread (ty,
// tx) owns rows 4 (r TY + ty) .. + 3 and columns 4 (c TX + tx) .. + 3 for r < RM, c < RN, so that a
// warp's 16-byte reads meet neighbouring places; two columns share a packed FMA (fma.rn.f32x2, each
// half rounded as a single FMA is).
#pragma once
#include "common.cuh"

__device__ __forceinline__ unsigned long long ft_pair(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 ft_split(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

template <int RM, int RN, int TY, int TX>
struct FmaTile {
    unsigned long long acc[4 * RM][2 * RN];
    int ty, tx;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 4 * RM; ++i)
#pragma unroll
            for (int j = 0; j < 2 * RN; ++j) acc[i][j] = 0ull;
    }
    __device__ __forceinline__ int row(int i) const { return 4 * ((i >> 2) * TY + ty) + (i & 3); }
    __device__ __forceinline__ int col(int c) const { return 4 * (c * TX + tx); }
    // acc += sum over k < n of A[k][row] B[k][col]
    __device__ __forceinline__ void add(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb, int n) {
        const float* a0 = A + 4 * ty;
        const float* b0 = B + 4 * tx;
#pragma unroll 4
        for (int k = 0; k < n; ++k, a0 += lda, b0 += ldb) {
            unsigned long long b[2 * RN];
#pragma unroll
            for (int c = 0; c < RN; ++c) {
                const ulonglong2 v = *(const ulonglong2*)(b0 + 4 * c * TX);
                b[2 * c] = v.x;
                b[2 * c + 1] = v.y;
            }
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const float4 v = *(const float4*)(a0 + 4 * r * TY);
                const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const unsigned long long aa = ft_pair(a[i], a[i]);
#pragma unroll
                    for (int j = 0; j < 2 * RN; ++j)
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[4 * r + i][j]) : "l"(aa), "l"(b[j]));
                }
            }
        }
    }
    __device__ __forceinline__ void scale_row(int i, float f) {
#pragma unroll
        for (int j = 0; j < 2 * RN; ++j) {
            const float2 v = ft_split(acc[i][j]);
            acc[i][j] = ft_pair(v.x * f, v.y * f);
        }
    }
    __device__ __forceinline__ float4 get(int i, int c) const {
        const float2 a = ft_split(acc[i][2 * c]), b = ft_split(acc[i][2 * c + 1]);
        return make_float4(a.x, a.y, b.x, b.y);
    }
};

__device__ __forceinline__ void ft_copy16(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ft_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ft_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
