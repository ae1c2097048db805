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
    // acc += sum over k0 <= k < n, k <= row of A[k][row] B[k][col], for the triangle of a chunk (RM = 1): a
    // term past a row is not added at all, since 0 times a value that is not finite is not 0. (Where every
    // value is finite `add` over the whole is the faster: a chunk's outputs 134 us against 139.)
    __device__ __forceinline__ void add_triangle(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb,
                                                 int k0, int n) {
        static_assert(RM == 1, "one run of rows a thread");
        const float* a0 = A + (size_t)k0 * lda + 4 * ty;
        const float* b0 = B + (size_t)k0 * ldb + 4 * tx;
#pragma unroll 2
        for (int k = k0; k < n; ++k, a0 += lda, b0 += ldb) {
            unsigned long long b[2 * RN];
#pragma unroll
            for (int c = 0; c < RN; ++c) {
                const ulonglong2 v = *(const ulonglong2*)(b0 + 4 * c * TX);
                b[2 * c] = v.x;
                b[2 * c + 1] = v.y;
            }
            const float4 v = *(const float4*)a0;
            const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (k > 4 * ty + i) continue;
                const unsigned long long aa = ft_pair(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 2 * RN; ++j)
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(b[j]));
            }
        }
    }
    // The same over channels k0 .. k0 + n - 1 of a tile that was laid down across its rows: column c of
    // channel k stands at c ^ 4 ((k >> SHIFT) & 7) (ft_swizzle), in A and, with BSWZ, in B. n and k0 are
    // multiples of 1 << SHIFT.
    template <int SHIFT, bool BSWZ>
    __device__ __forceinline__ void add_swizzled(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb,
                                                 int k0, int n) {
#pragma unroll 1
        for (int kb = 0; kb < n; kb += 1 << SHIFT) {
            const int x = 4 * (((k0 + kb) >> SHIFT) & 7);
            const float* b0 = B + (size_t)kb * ldb;
            const float* a0 = A + (size_t)kb * lda;
#pragma unroll
            for (int k = 0; k < (1 << SHIFT); ++k, a0 += lda, b0 += ldb) {
                unsigned long long b[2 * RN];
#pragma unroll
                for (int c = 0; c < RN; ++c) {
                    const ulonglong2 v = *(const ulonglong2*)(b0 + (BSWZ ? (4 * (c * TX + tx)) ^ x : 4 * (c * TX + tx)));
                    b[2 * c] = v.x;
                    b[2 * c + 1] = v.y;
                }
#pragma unroll
                for (int r = 0; r < RM; ++r) {
                    const float4 v = *(const float4*)(a0 + ((4 * (r * TY + ty)) ^ x));
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

// Where column c of channel k stands in a tile of channel rows that threads fill from row-major memory: a
// warp then stores four rows x eight runs of 1 << shift channels without meeting a bank twice (rows of
// 64 + 4 floats), and groups of four columns stay together.
__device__ __forceinline__ int ft_swizzle(int c, int k, int shift) { return c ^ (4 * ((k >> shift) & 7)); }

__device__ __forceinline__ bool ft_not_finite(float4 v) {
    const float inf = __int_as_float(0x7f800000);
    return !(fabsf(v.x) < inf && fabsf(v.y) < inf && fabsf(v.z) < inf && fabsf(v.w) < inf);
}
__device__ __forceinline__ void ft_copy16(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ft_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ft_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
