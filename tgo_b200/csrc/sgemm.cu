// y[M,N] = x[M,K] . w[N,K]^T in true float32, no reduced-precision mode: the matrix product of the
// float32 path of the whole model. An output's arithmetic depends on N, K and w's alignment alone, so
// a row's result does not depend on which other rows are in the batch. Two forms: plain FMA, here, for short or
// ragged K; and three bfloat16 parts a number on the tensor cores, below.
//
// Plain FMA: every output element is one running sum over k = 0..K-1 in that order, whatever tile
// it falls in. Bound by the FMA pipes (128 lanes an SM). A thread owns 8 x 8, 8 x 4 or 2 x 4 outputs in
// registers, so that a k costs it 16-byte reads of shared memory for a few outputs each; two
// neighbouring columns go through one packed FMA (fma.rn.f32x2, each half rounded as a single
// FMA is), which leaves issue slots for the reads (scalar FMA: 5 to 25 % slower). Steps of 16 k
// come in by asynchronous 4-byte copies that lay them down k-major, two steps ahead.
// MEASURED (B200, ten calls in a row), sizes that come here: K = 250, 557 x 12288 outputs 84 us, 41 of 74 TFLOP/s, 557 x
// 2048 22, 1 x 2048 10.5; K = 128, 557 x 12288 47, 1 x 2048 6.5; K = 2050, whose rows are not whole 16 bytes, 557 x 12288 626,
// 1 x 2048 56: a single sum's chain of 2050 FMA. At K = 2048 a 64 x 64 tile with 4 x 4 outputs a thread, loads and products in
// turn, took 1272 for 557 x 12288 (597). ncu: FMA pipes 64 % busy, the rest waits for reads of shared memory.
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

// For tests and tuning: the plain kernel, with this tile, instead of the choice by size (0 gives the choice back).
static int sg_forced = 0;
TGO_API void tgo_sgemm_force_tile(int tile) { sg_forced = tile; }

// ------------------------------------------------------------- the same on the tensor cores
// K of at least SP_MIN_K and rows of whole 16 bytes: each float32 number as three bfloat16 parts and six of
// their nine products on tcgen05 (split3.cuh). A CTA takes 128 rows of w (the accumulator's lanes) and NT
// rows of x (its columns), a k-block of 64 at a time, in five warpgroups:
//   warps 0..7    add each k-block's products, which they read from tensor memory, to float32 sums in registers;
//   warps 8..15   make w's three parts from float32 tiles in shared memory and lay them down in tensor memory,
//                 a lane a row (two stages);
//   warp 16       TMA loads of the parts of x, which a small kernel has laid out before (two k-blocks deep);
//   warp 17       products, w from tensor memory: x's lo with w's hi; mid with mid, hi; hi with lo, mid, hi, into
//                 one of two accumulators;
//   warp 18       TMA loads of w, three k-blocks deep.
// An accumulator holds ONE k-block: the tensor cores cut a sum's low bits at every step where an FMA rounds,
// so a long sum there would lean towards zero; four steps at the sum's size and a rounded addition
// per k-block err less than a chain of 64 FMA (MEASURED against 64 bits, 2-norms, normal numbers:
// K = 2048 1.3e-7 for the chain's 8.1e-7, K = 6144 1.9e-7 for 1.4e-6).
// Both sides are taken SP_UP times and an output SP_DOWN times: bfloat16 numbers end at 2^-133, so that the parts
// of 1e-36 as it stands hold no more than its first 15 bits (MEASURED error 2.7e-5; at 1e-38 2.7e-3), while 24 powers
// of two higher every float32 number has all of its parts.
// An output's arithmetic is the same whatever tile it falls in and whatever rows are beside it. An output
// that is not finite (an input that is not, or is more than 2^103, or a sum past 2^80) is made again as the plain
// kernel makes it: a block that has one makes its whole tile by FMA over tiles in shared memory (sp_plain) and writes
// the outputs that were not finite. MEASURED, K = 2048, both launches: all of 557 x 2048 215 us (36 where all are finite; 8900
// by a thread an output; 131 by the plain kernel), of 557 x 12288 1250 (136; 53000; 598), of one row x 2048 162 (28; 165; 60).
// Bound by shared memory and the tensor pipe side by side at many rows (a k-block at NT = 128: 1660 and 1540
// cycles), by the issue of 24 products a k-block at few. With w's parts in shared memory, made by the warps that
// sum, and the products issued by a lane that no elect.sync had chosen, a k-block took 2500 cycles at any NT.
// MEASURED (B200, flushed L2, both launches; the plain kernel in brackets): 557 rows, K = 2048: 12288
// outputs 132 us (601), 3072 42 (193), 2048 36 (131); K = 6144, 2048 outputs 81 (375); 100 x 12288 48 (188);
// 3 x 32768 about 75 (145); 1 x 2048 26 (59).
#include "split3.cuh"

#define SP_BK 64
#define SP_UP 0x1p24f
#define SP_DOWN 0x1p-48f
#define SP_MIN_K 256                                     // 256 x 256: 11.3 us for 12.3; K = 128: 11.3 for 10.2
#define SP_THREADS 640                                   // warp 19 only fills up the last warpgroup
#define SP_W_BYTES (128 * SP_BK * 4)                     // a k-block of w: two tiles of 32 columns
#define SP_W_STAGES 3
#define SP_X_RING (2 * 3 * SP_ACC * SP_BK * 2)                // two k-blocks of the three parts
#define SP_SMEM (1024 + SP_W_STAGES * SP_W_BYTES + SP_X_RING + 512)
#define SP_ACC 160                                       // columns of an accumulator: two, then two stages of w's parts
#define SP_PARTS 96

__device__ int sgemm_error_flag = 0;

// parts [3][M][Kp] of x [M][K]: eight numbers a thread
__global__ void __launch_bounds__(256)
sgemm_split_kernel(const float* __restrict__ x, bf16* __restrict__ parts, int M, int K, int Kp, int vec) {
    pdl_wait();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int runs = Kp / 8;
    if (i >= (long long)M * runs) return;
    const long long row = i / runs;
    const int k = (int)(i % runs) * 8;
    const float* p = x + row * K + k;
    float v[8];
    if (vec && k + 8 <= K) {
        const float4 a = ((const float4*)p)[0], b = ((const float4*)p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = k + j < K ? p[j] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= SP_UP;
    uint4 part[3];
    s3_split8(v, part[0], part[1], part[2]);
#pragma unroll
    for (int j = 0; j < 3; ++j) *(uint4*)(parts + ((size_t)j * M + row) * Kp + k) = part[j];
}

// acc[0 .. N - 1] += N columns of tensor memory
template <int N> __device__ __forceinline__ void sp_add(uint32_t t, float* acc) {
    if constexpr (N >= 32) {
        uint32_t r[32];
        tg_ld32(t, r);
        tg_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] += __uint_as_float(r[i]);
        sp_add<N - 32>(t + 32, acc + 32);
    } else if constexpr (N == 16) {
        uint32_t r[16];
        tg_ld16(t, r);
        tg_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] += __uint_as_float(r[i]);
    }
}

// How many of the 256 threads that sum.
__device__ __forceinline__ uint32_t sp_count(bool yes) {
    uint32_t n;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.popc.u32 %0, 1, 256, p;\n\t}" : "=r"(n) : "r"((uint32_t)yes) : "memory");
    return n;
}

// The registers (96 a thread at launch) go where they are used: 256 x (SP_SUM_REGS + SP_PART_REGS) + 128 x 40
// is not more than 640 x 96.
#define SP_SUM_REGS 128
#define SP_PART_REGS 88
template <int N> __device__ __forceinline__ void sp_regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void sp_regs_less() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// The tile's outputs as sgemm_tn_kernel makes them, by the 256 threads that sum: NT / 16 x 8 outputs a thread, steps of 16 k
// two ahead. Those that were finite stay.
template <int NT>
__device__ __forceinline__ void sp_plain(float* tile, const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N,
                                         int K, int m0, int n0) {
    constexpr int R = NT / 16, XF = SG_BK * (NT + 4), WF = SG_BK * (128 + 4);
    static_assert(3 * (XF + WF) * (int)sizeof(float) <= SP_W_STAGES * SP_W_BYTES + SP_X_RING, "the rings' place");
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    unsigned long long acc[R][4];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    auto load = [&](int st, int k0) {
        if (k0 < K) {
            float* to = tile + st * (XF + WF);
            sg_load<NT, 256>((float (*)[NT + 4])to, x, m0, M, k0, K);
            sg_load<128, 256>((float (*)[132])(to + XF), w, n0, N, k0, K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, 0);
    load(1, SG_BK);
    int st = 0;
    for (int k0 = 0; k0 < K; k0 += SG_BK) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        asm volatile("bar.sync 1, 256;" ::: "memory");   // this step's k are there, the last step's place is free
        load(st == 0 ? 2 : st - 1, k0 + 2 * SG_BK);
        const float* xb = tile + st * (XF + WF) + ty;
        const float* wb = tile + st * (XF + WF) + XF + 4 * tx;
        st = st == 2 ? 0 : st + 1;
#pragma unroll 2
        for (int kk = 0; kk < SG_BK; ++kk, xb += NT + 4, wb += 132) {
            const ulonglong2 b0 = *(const ulonglong2*)wb, b1 = *(const ulonglong2*)(wb + 64);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const unsigned long long aa = sg_pair(xb[16 * i], xb[16 * i]);
                sg_fma2(acc[i][0], aa, b0.x); sg_fma2(acc[i][1], aa, b0.y);
                sg_fma2(acc[i][2], aa, b1.x); sg_fma2(acc[i][3], aa, b1.y);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty + 16 * i, n = n0 + 64 * (j >> 1) + 4 * tx + 2 * (j & 1);
            float v[2];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][j]));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float* to = y + (size_t)m * N + n + c;
                if (m < M && n + c < N && !(fabsf(*to) < __int_as_float(0x7f800000))) *to = v[c];
            }
        }
}

// Grid (tiles of x's rows, tiles of w's rows): the CTAs that read the same rows of w run side by side.
// Every wait has a time limit; TMEM is freed on every path.
template <int NT>
__global__ void __launch_bounds__(SP_THREADS, 1)
sgemm_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    constexpr int X_TILE = NT * SP_BK * 2, CW = NT / 2;
    static_assert(NT % 32 == 0 && NT <= SP_ACC && 2 * SP_ACC + 2 * SP_PARTS <= 512, "tensor memory");
    extern __shared__ unsigned char sp_raw[];
    unsigned char* wt = (unsigned char*)(((uintptr_t)sp_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* xt = wt + SP_W_STAGES * SP_W_BYTES;
    uint64_t* w_full = (uint64_t*)(xt + SP_X_RING);            // [SP_W_STAGES]
    uint64_t* w_empty = w_full + SP_W_STAGES;                  // [SP_W_STAGES]
    uint64_t* p_full = w_empty + SP_W_STAGES;                  // [2]
    uint64_t* acc_full = p_full + 2;                           // [2]: a k-block's products are made, its operands read
    uint64_t* acc_empty = acc_full + 2;                        // [2]
    uint64_t* settled = acc_empty + 2;
    uint64_t* x_full = settled + 1;                            // [2]
    uint32_t* tmem_slot = (uint32_t*)(x_full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * NT, n0 = blockIdx.y * 128, kbs = (K + SP_BK - 1) / SP_BK;
    if (threadIdx.x == 0) {
        for (int i = 0; i < SP_W_STAGES; ++i) { tg_init(&w_full[i], 1); tg_init(&w_empty[i], 8); }
        for (int i = 0; i < 2; ++i) {
            tg_init(&p_full[i], 8);
            tg_init(&acc_full[i], 1);
            tg_init(&acc_empty[i], 8);
            tg_init(&x_full[i], 1);
        }
        tg_init(settled, 1);
        tg_init_done();
    }
    if (warp == 17) tg_alloc512(tmem_slot);
    tg_before();
    __syncthreads();
    tg_after();
    const uint32_t tmem = *tmem_slot, lanes = (uint32_t)((warp & 3) * 32) << 16;
    pdl_wait();

    if (warp < 8) {
        sp_regs_more<SP_SUM_REGS>();
        float acc[CW];
#pragma unroll
        for (int i = 0; i < CW; ++i) acc[i] = 0.f;
        const uint32_t cols = tmem + lanes + (uint32_t)((warp >> 2) * CW);
        bool ok = true;
        for (int kb = 0; kb < kbs; ++kb) {
            ok = __all_sync(0xffffffffu, tg_wait(&acc_full[kb & 1], (kb >> 1) & 1, &sgemm_error_flag, 4));
            if (!ok) break;
            tg_after();
            sp_add<CW>(cols + (uint32_t)((kb & 1) * SP_ACC), acc);
            tg_before();
            __syncwarp();
            if (lane == 0) tg_arrive(&acc_empty[kb & 1]);
        }
        const int n = n0 + (warp & 3) * 32 + lane, mb = m0 + (warp >> 2) * CW;
        bool odd = false;
        if (ok && n < N) {
            float* yo = y + (size_t)mb * N + n;
#pragma unroll
            for (int i = 0; i < CW; ++i)
                if (mb + i < M) {
                    yo[(size_t)i * N] = acc[i] * SP_DOWN;
                    odd = odd || !(fabsf(acc[i]) < __int_as_float(0x7f800000));
                }
        }
        // every copy has landed and been read once the last products are there: the rings are free
        __syncwarp();
        const uint32_t waits = sp_count(!ok), odds = sp_count(odd);
        if (!waits && odds) sp_plain<NT>((float*)wt, x, w, y, M, N, K, m0, n0);
    } else if (warp < 16) {
        sp_regs_less<SP_PART_REGS>();
        // a lane a row of w; warps 8..11 take the first 32 k of a k-block, 12..15 the others
        const int row = (warp & 3) * 32 + lane, half = (warp - 8) >> 2;
        const uint32_t src = tg_smem(wt) + (uint32_t)(half * (SP_W_BYTES / 2) + row * 128);
        const uint32_t dst = tmem + lanes + 2 * SP_ACC + 16 * half;
        bool ok = true;
        for (int kb = 0; kb < kbs; ++kb) {
            const int s = kb % SP_W_STAGES;
            ok = __all_sync(0xffffffffu, tg_wait(&w_full[s], (kb / SP_W_STAGES) & 1, &sgemm_error_flag, 5));
            if (!ok) break;
            uint32_t part[3][16];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float4 v;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                             : "r"(src + (uint32_t)(s * SP_W_BYTES + ((c ^ (row & 7)) << 4))) : "memory");
                s3_split2(v.x * SP_UP, v.y * SP_UP, part[0][2 * c], part[1][2 * c], part[2][2 * c]);
                s3_split2(v.z * SP_UP, v.w * SP_UP, part[0][2 * c + 1], part[1][2 * c + 1], part[2][2 * c + 1]);
            }
            __syncwarp();
            if (lane == 0) tg_arrive(&w_empty[s]);
            // the k-block before the last has been multiplied: its parts' place is free
            if (kb > 1) ok = __all_sync(0xffffffffu, tg_wait(&acc_full[kb & 1], ((kb >> 1) & 1) ^ 1, &sgemm_error_flag, 1));
            if (!ok) break;
            tg_after();
#pragma unroll
            for (int q = 0; q < 3; ++q) tg_st16(dst + (uint32_t)((kb & 1) * SP_PARTS + 32 * q), part[q]);
            tg_wait_st();
            tg_before();
            __syncwarp();
            if (lane == 0) tg_arrive(&p_full[kb & 1]);
        }
    } else {
        sp_regs_less<40>();
        if (warp == 16 && lane == 0) {
            bool ok = true;
            uint32_t it = 0;
            for (; it < (uint32_t)kbs; ++it) {
                const uint32_t s = it & 1;
                if (it > 1) ok = tg_wait(&acc_full[s], ((it >> 1) & 1) ^ 1, &sgemm_error_flag, 2);
                if (!ok) break;
                tg_expect(&x_full[s], 3 * X_TILE);
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    tg_load_2d(xt + (3 * s + p) * X_TILE, &map_x, (int)it * SP_BK, p * M + m0, &x_full[s]);
            }
            if (!ok) tg_settle_copies(x_full, 2, it, &sgemm_error_flag, 2);
        } else if (warp == 18 && lane == 0) {
            bool ok = true;
            uint32_t it = 0;
            for (; it < (uint32_t)kbs; ++it) {
                const uint32_t s = it % SP_W_STAGES;
                ok = tg_wait(&w_empty[s], ((it / SP_W_STAGES) & 1) ^ 1, &sgemm_error_flag, 6);
                if (!ok) break;
                tg_expect(&w_full[s], SP_W_BYTES);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    tg_load_2d(wt + s * SP_W_BYTES + h * (SP_W_BYTES / 2), &map_w, (int)it * SP_BK + 32 * h, n0, &w_full[s]);
            }
            if (!ok) tg_settle_copies(w_full, SP_W_STAGES, it, &sgemm_error_flag, 6);
        } else if (warp == 17) {
            const uint32_t idesc = tg_idesc(NT);
            const bool leader = tg_elect();
            bool ok = true;
            for (int kb = 0; kb < kbs; ++kb) {
                const uint32_t par = (kb >> 1) & 1;
                ok = tg_wait(&acc_empty[kb & 1], par ^ 1, &sgemm_error_flag, 3) && tg_wait(&x_full[kb & 1], par, &sgemm_error_flag, 3) &&
                     tg_wait(&p_full[kb & 1], par, &sgemm_error_flag, 3);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                tg_after();
                if (leader) {
                    const uint32_t d = tmem + (uint32_t)(SP_ACC * (kb & 1)), a = tmem + (uint32_t)(2 * SP_ACC + SP_PARTS * (kb & 1));
                    const uint64_t dx = tg_desc(xt + 3 * (kb & 1) * X_TILE);
#pragma unroll
                    for (int p = 2; p >= 0; --p)
#pragma unroll
                        for (int q = 2 - p; q >= 0; --q)
#pragma unroll
                            for (int k = 0; k < SP_BK / 16; ++k)
                                tg_mma_ts(d, a + (uint32_t)(32 * q + 8 * k), dx + (uint64_t)(p * (X_TILE >> 4) + 2 * k), idesc, p < 2 || k > 0 ? 1u : 0u);
                    tg_commit(&acc_full[kb & 1]);
                }
                __syncwarp();
            }
            if (!ok && leader) tg_settle_products(settled, &sgemm_error_flag, 3);
            __syncwarp();
        }
    }
    tg_before();
    __syncthreads();
    if (warp == 17) {
        tg_after();
        tg_free512(tmem);
    }
}

template <int NT>
static int sp_go(const CUtensorMap& map, const CUtensorMap& map_w, const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    static bool sized[64] = {};                          // per device: the attribute is set there
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
    if (!sized[dev]) {
        e = cudaFuncSetAttribute(sgemm_tc_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SP_SMEM);
        if (e != cudaSuccess) return (int)e;
        sized[dev] = true;
    }
    const dim3 grid((M + NT - 1) / NT, (N + 127) / 128);
    if (grid.y > 65535) return TGO_E_BAD_ARG;
    return tgo_launch_pdl(sgemm_tc_kernel<NT>, grid, dim3(SP_THREADS), SP_SMEM, stream, map, map_w, x, w, y, M, N, K);
}

// Bytes of workspace a product needs for the parts of x; 0: it is made by the plain kernel and needs
// none. The rule does not look at M, so that a row's result does not depend on the rows beside it.
TGO_API int tgo_sgemm_part_bytes(const float* w, int K, int N) {
    if (sg_forced || K < SP_MIN_K || K % 4 || (uintptr_t)w % 16 || (N + 127) / 128 > 65535) return 0;
    return 3 * 2 * ((K + 7) / 8 * 8);                    // a row of x
}

TGO_API int tgo_sgemm_error(int* value) { return (int)cudaMemcpyFromSymbol(value, sgemm_error_flag, sizeof(int)); }

static int sp_forced = 0;
TGO_API void tgo_sgemm_force_columns(int nt) { sp_forced = nt; }

// As tgo_sgemm_tn; parts: tgo_sgemm_part_bytes bytes a row of x, 16-byte aligned.
TGO_API int tgo_sgemm_split(const float* x, const float* w, float* y, int M, int N, int K, bf16* parts, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const int Kp = (K + 7) / 8 * 8;
    if (!tgo_sgemm_part_bytes(w, K, N) || !parts || (uintptr_t)parts % 16 || M > 0x7fffffff / 3 - 256) return TGO_E_BAD_ARG;
    // The tile: a round (as many tiles as SMs) takes that long for a k-block, in ns (K = 6144, 1 to 557 rows).
    static const struct { int nt, ns; } tiles[5] = {{160, 1250}, {128, 1060}, {96, 900}, {64, 770}, {32, 590}};
    const int sms = tgo_multiprocessors();
    int nt = sp_forced;
    if (!nt) {
        long long best = -1;
        for (int i = 0; i < 5; ++i) {
            const long long n = (long long)((M + tiles[i].nt - 1) / tiles[i].nt) * ((N + 127) / 128);
            const long long cost = (n + sms - 1) / sms * tiles[i].ns;
            if (best < 0 || cost < best) { best = cost; nt = tiles[i].nt; }
        }
    }
    CUtensorMap map, map_w;
    if (!tg_map(&map, parts, 3LL * M, Kp, Kp, nt) || !tg_map_f32(&map_w, w, N, K, K, 128)) return TGO_E_BAD_ARG;
    const long long runs = (long long)M * (Kp / 8);
    const int vec = K % 4 == 0 && (uintptr_t)x % 16 == 0;
    if ((runs + 255) / 256 > 0x7fffffffLL) return TGO_E_BAD_ARG;
    const int rc = tgo_launch_pdl(sgemm_split_kernel, dim3((unsigned)((runs + 255) / 256)), dim3(256), 0, stream, x, parts, M, K, Kp, vec);
    if (rc) return rc;
    switch (nt) {
        case 160: return sp_go<160>(map, map_w, x, w, y, M, N, K, stream);
        case 128: return sp_go<128>(map, map_w, x, w, y, M, N, K, stream);
        case 96: return sp_go<96>(map, map_w, x, w, y, M, N, K, stream);
        case 64: return sp_go<64>(map, map_w, x, w, y, M, N, K, stream);
        default: return sp_go<32>(map, map_w, x, w, y, M, N, K, stream);
    }
}

TGO_API int tgo_sgemm_tn(const float* x, const float* w, float* y, int M, int N, int K,
                         cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return TGO_E_BAD_ARG;
    const int sms = tgo_multiprocessors();
    // The tile: a round (as many tiles as SMs) costs `fixed` once and `round` each, in us at K = 2048,
    // fitted to the times of 15 products of 1 to 1200 rows (64 x 128: 123 us for one round, 597 for
    // six; 64 x 64: 88, 133 for two, 688 for twelve; 16 x 64: 54, 132 for four, 1450 for forty-six).
    // 128 x 128 tiles were never the fastest (785 us where 64 x 128 took 597). For K = 64, 128, 250 and 2050, 1 to 1200 rows and
    // 64 to 12288 outputs the choice is the fastest of the three tiles or at most 2 us behind it (1200 x 12288, K = 2050: 1304 of 1302).
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
