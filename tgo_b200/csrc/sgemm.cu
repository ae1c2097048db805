// y[M,N] = x[M,K] . w[N,K]^T in true float32: plain FMA, no tensor cores, no reduced-
// precision mode. Every output element is one running sum over k = 0..K-1 in that order,
// whatever tile it falls in, so a row's result does not depend on which other rows are in
// the batch. This is the matrix product of the float32 path of the whole model.
//
// Bound by the FMA pipes (128 lanes an SM). A thread owns 8 x 8, 8 x 4 or 2 x 4 outputs in
// registers, so that a k costs it 16-byte reads of shared memory for a few outputs each; two
// neighbouring columns go through one packed FMA (fma.rn.f32x2, each half rounded as a single
// FMA is), which leaves issue slots for the reads (scalar FMA: 5 to 25 % slower). Steps of 16 k
// come in by asynchronous 4-byte copies that lay them down k-major, two steps ahead.
// MEASURED (B200, K = 2048; a 64 x 64 tile with 4 x 4 outputs a thread, loads and products in
// turn, in brackets): 557 x 12288 outputs 597 us, 47 of 74 TFLOP/s (1272 us); 557 x 2048 134 us
// (250); 100 x 12288 191 us (344); 3 x 32768 132 us (429); 1 x 2048 54 us (167): a single sum's
// chain of 2048 FMA. ncu: FMA pipes 64 % busy, the rest waits for reads of shared memory.
#include "common.cuh"

#define SG_BK 16
#define SG_STAGES 3

__device__ __forceinline__ unsigned long long sg_pair(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void sg_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// A step's 16 k of ROWS rows on their way into shared memory, k-major; k and rows past the end
// are zeros (a product with them leaves a sum as it is).
template <int ROWS, int THREADS>
__device__ __forceinline__ void sg_load(float (*s)[ROWS + 4], const float* __restrict__ p, int row0, int rows,
                                        int k0, int K) {
    constexpr int N = ROWS * SG_BK / THREADS;
    static_assert(ROWS * SG_BK % THREADS == 0, "a thread copies as many as every other");
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int idx = threadIdx.x + i * THREADS;
        const int r = idx / SG_BK, k = idx % SG_BK;
        const bool ok = row0 + r < rows && k0 + k < K;
        const float* src = ok ? p + (size_t)(row0 + r) * K + k0 + k : p;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                     ::"r"((uint32_t)__cvta_generic_to_shared(&s[k][r])), "l"(src), "r"(ok ? 4 : 0) : "memory");
    }
}

// Thread (ty, tx) owns rows 4 ty .. 4 ty + 3 of every run of 4 BM / TM rows and columns 4 tx ..
// 4 tx + 3 of every run of 4 BN / TN: a warp's 16-byte reads then hit neighbouring places.
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
sgemm_tn_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                int M, int N, int K) {
    constexpr int TY = BM / TM, TX = BN / TN, THREADS = TX * TY;
    constexpr int RM = TM < 4 ? TM : 4;                  // rows a thread owns side by side
    constexpr int XF = SG_BK * (BM + 4), WF = SG_BK * (BN + 4);
    extern __shared__ __align__(16) float sg_smem[];         // [SG_STAGES][XF + WF]
    auto xs = [&](int st) { return (float (*)[BM + 4])(sg_smem + st * (XF + WF)); };
    auto ws = [&](int st) { return (float (*)[BN + 4])(sg_smem + st * (XF + WF) + XF); };
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    auto load = [&](int st, int k0) {
        if (k0 < K) {
            sg_load<BM, THREADS>(xs(st), x, m0, M, k0, K);
            sg_load<BN, THREADS>(ws(st), w, n0, N, k0, K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < SG_STAGES - 1; ++st) load(st, st * SG_BK);
    int st = 0;
    for (int k0 = 0; k0 < K; k0 += SG_BK) {
        asm volatile("cp.async.wait_group %0;" ::"n"(SG_STAGES - 2) : "memory");
        __syncthreads();                                 // this step's k are there, the last step's place is free
        load(st == 0 ? SG_STAGES - 1 : st - 1, k0 + (SG_STAGES - 1) * SG_BK);
        float (*xb)[BM + 4] = xs(st);
        float (*wb)[BN + 4] = ws(st);
        st = st + 1 == SG_STAGES ? 0 : st + 1;
        // the next k's values are read while the present ones multiply
        float a[2][TM];
        unsigned long long b[2][TN / 2];
        auto read = [&](int f, int kk) {
#pragma unroll
            for (int i = 0; i < TM; i += RM) {
                const float* p = &xb[kk][i * TY + ty * RM];
                if (RM == 4) {
                    const float4 v = *(const float4*)p;
                    a[f][i] = v.x; a[f][i + (RM > 1 ? 1 : 0)] = v.y;
                    a[f][i + (RM > 2 ? 2 : 0)] = v.z; a[f][i + (RM > 3 ? 3 : 0)] = v.w;
                } else {
#pragma unroll
                    for (int r = 0; r < RM; ++r) a[f][i + r] = p[r];
                }
            }
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const ulonglong2 v = *(const ulonglong2*)&wb[kk][j * TX + tx * 4];
                b[f][j / 2] = v.x;
                b[f][j / 2 + 1] = v.y;
            }
        };
        read(0, 0);
#pragma unroll
        for (int kk = 0; kk < SG_BK; ++kk) {
            if (kk + 1 < SG_BK) read((kk + 1) & 1, kk + 1);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const unsigned long long aa = sg_pair(a[kk & 1][i], a[kk & 1][i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) sg_fma2(acc[i][j], aa, b[kk & 1][j]);
            }
        }
    }
    const bool vec_out = N % 4 == 0 && ((uintptr_t)y & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + (i / RM) * RM * TY + ty * RM + i % RM;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int gn = n0 + j * TX + tx * 4;
            float v[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][j / 2]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][j / 2 + 1]));
            float* dst = y + (size_t)gm * N + gn;
            if (vec_out && gn + 4 <= N) *(float4*)dst = make_float4(v[0], v[1], v[2], v[3]);
            else
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (gn + c < N) dst[c] = v[c];
        }
    }
}

template <int BM, int BN, int TM, int TN>
static int sg_go(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return TGO_E_BAD_ARG;
    constexpr int threads = (BM / TM) * (BN / TN);
    constexpr size_t smem = (size_t)SG_STAGES * SG_BK * (BM + BN + 8) * sizeof(float);
    static bool sized[64] = {};                          // per device: the attribute is set there
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
    if (!sized[dev]) {
        e = cudaFuncSetAttribute(sgemm_tn_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        sized[dev] = true;
    }
    sgemm_tn_kernel<BM, BN, TM, TN><<<grid, threads, smem, stream>>>(x, w, y, M, N, K);
    return launch_status();
}

// For tests and tuning: the tile instead of the choice by size (0 gives the choice back).
static int sg_forced = 0;
TGO_API void tgo_sgemm_force_tile(int tile) { sg_forced = tile; }

TGO_API int tgo_sgemm_tn(const float* x, const float* w, float* y, int M, int N, int K,
                         cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return TGO_E_BAD_ARG;
    const int sms = tgo_multiprocessors();
    // The tile: a round (as many tiles as SMs) costs `fixed` once and `round` each, in us at K = 2048,
    // fitted to the times of 15 products of 1 to 1200 rows (64 x 128: 123 us for one round, 597 for
    // six; 64 x 64: 88, 133 for two, 688 for twelve; 16 x 64: 54, 132 for four, 1450 for forty-six).
    // 128 x 128 tiles were never the fastest (785 us where 64 x 128 took 597).
    int pick = sg_forced;
    if (!pick) {
        static const struct { int bm, bn; double fixed, round; } tiles[3] = {
            {64, 128, 25.0, 97.0}, {64, 64, 30.0, 55.0}, {16, 64, 22.0, 32.0}};
        double best = -1.0;
        for (int i = 0; i < 3; ++i) {
            const long long n = (long long)((M + tiles[i].bm - 1) / tiles[i].bm) * ((N + tiles[i].bn - 1) / tiles[i].bn);
            const double cost = tiles[i].fixed + (double)((n + sms - 1) / sms) * tiles[i].round;
            if (best < 0 || cost < best) { best = cost; pick = i + 1; }
        }
    }
    switch (pick) {
        case 1: return sg_go<64, 128, 8, 8>(x, w, y, M, N, K, stream);
        case 2: return sg_go<64, 64, 8, 4>(x, w, y, M, N, K, stream);
        default: return sg_go<16, 64, 2, 4>(x, w, y, M, N, K, stream);
    }
}
