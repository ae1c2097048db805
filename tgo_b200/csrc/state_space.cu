// A selective state-space mixer's recurrent part (the form known as Mamba-2): a short causal
// convolution per channel with its last inputs kept per request, and the scan
//
//   dt_t = softplus(raw_t + dt_bias_h)                      per head h, float32
//   S_t  = exp(-exp(A_log_h) dt_t) S_(t-1) + dt_t B_t x_t^T      S is [N, P], float32
//   y_t  = S_t^T C_t + D_h x_t
//
// over each request's tokens of the step, from and into the request's float32 state. Head h
// reads B and C of group floor(h / (H / G)). Everything after the convolution's input is
// float32 whatever the storage type of the projections.
//
// A second scan (the form known as Mamba-1) has a decay of its own for every channel and state,
// and B and C shared by all channels:
//
//   dt_t    = softplus(raw_t + dt_bias)                     per channel c
//   S[c, n] = exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n       S is [channels, N], float32
//   y_c     = (sum_n S[c, n] C_n + D_c x_c) * silu(z_c)
//
// A request's state row (float32, `state_stride` floats apart) holds the scan's state
// [H][N][P] (or [channels][N]) at `ssm_offset` and the convolution's last taps - 1 inputs [taps - 1][C] (oldest
// first) at `conv_offset`.
#include "split3.cuh"

// ------------------------------------------------------------------------- convolution
// y[t][c] = silu(bias[c] + sum_j w[c][j] x[t - (taps - 1 - j)][c]); inputs before the step's
// first token come from the request's kept inputs, zeros before the request's start (a fresh
// state row is zero). x is a column view [T, C] in the storage type; y [T, C] float32 or in the
// storage type (TY).
template <typename T, typename TY>
__global__ void __launch_bounds__(256)
causal_conv_act_kernel(const T* __restrict__ x, long long x_stride, const float* __restrict__ w,
                       const float* __restrict__ bias, TY* __restrict__ y, int C, int taps,
                       const int* __restrict__ seq_ids, const int* __restrict__ q_start,
                       const int* __restrict__ state_slots, const float* __restrict__ state,
                       long long state_stride, long long conv_offset) {
    pdl_wait();
    const int t = blockIdx.x;
    const int b = seq_ids[t];
    const int r = t - q_start[b];                       // place among the request's tokens
    const float* kept = state + (size_t)state_slots[b] * state_stride + conv_offset;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        float a = bias ? bias[c] : 0.f;
        for (int j = 0; j < taps; ++j) {
            const int back = taps - 1 - j;               // how many tokens before this one
            float v;
            if (back <= r) v = to_f32(x[(size_t)(t - back) * x_stride + c]);
            else v = kept[(size_t)(taps - 1 - (back - r)) * C + c];
            a = fmaf(w[(size_t)c * taps + j], v, a);
        }
        y[(size_t)t * C + c] = from_f32<TY>(a / (1.f + expf(-a)));
    }
}

// The same with eight channels a thread (16-byte loads of x) and TOK consecutive tokens, whose
// rows are asked for before the first is used, the window of inputs in registers: for up to four
// taps, C, the row stride and x's address as multiples of eight elements. `kept4`: the kept rows
// can be read 16 bytes at a time. One token a thread where the step has only single tokens.
#define CV_TOK 8
__device__ __forceinline__ void cv_widen(float* v, uint4 q) {
    const uint32_t* w = (const uint32_t*)&q;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)(w + k));
        v[2 * k] = f.x;
        v[2 * k + 1] = f.y;
    }
}
__device__ __forceinline__ void cv_load8(float* v, const float* p) {
    const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void cv_store(bf16* p, const float* v) {
    uint4 q;
    uint32_t* w = (uint32_t*)&q;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        w[k] = *(const uint32_t*)&b;
    }
    *(uint4*)p = q;
}
__device__ __forceinline__ void cv_store(float* p, const float* v) {
    *(float4*)p = make_float4(v[0], v[1], v[2], v[3]);
    *(float4*)(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

template <typename TY, int TAPS, int TOK>
__global__ void __launch_bounds__(128)
causal_conv_act_x8_kernel(const bf16* __restrict__ x, long long x_stride, const float* __restrict__ w,
                          const float* __restrict__ bias, TY* __restrict__ y, int Tn, int C,
                          const int* __restrict__ seq_ids, const int* __restrict__ q_start,
                          const int* __restrict__ state_slots, const float* __restrict__ state,
                          long long state_stride, long long conv_offset, int kept4) {
    pdl_wait();
    const int c = 8 * (blockIdx.y * blockDim.x + threadIdx.x), t_lo = blockIdx.x * TOK;
    if (c >= C) return;
    uint4 rows[TOK];
#pragma unroll
    for (int u = 0; u < TOK; ++u)
        rows[u] = *(const uint4*)(x + (size_t)(t_lo + u < Tn ? t_lo + u : Tn - 1) * x_stride + c);
    float wt[8 * TAPS], bs[8], win[TAPS][8];             // win[j] meets tap j; the last is the token's own
#pragma unroll
    for (int q = 0; q < TAPS; ++q) cv_load8(wt + 8 * q, w + (size_t)c * TAPS + 8 * q);    // [channel][tap]
    if (bias) {
        cv_load8(bs, bias + c);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) bs[i] = 0.f;
    }
    int q_at = -1, first = 0;
#pragma unroll
    for (int u = 0; u < TOK; ++u) {
        const int t = t_lo + u;
        if (t >= Tn) break;
        const int b = seq_ids[t];
        if (u == 0 || b != q_at) {                       // a window from the start: rows of the step, then kept ones
            q_at = b;
            first = q_start[b];
            const float* kept = state + (size_t)state_slots[b] * state_stride + conv_offset;
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j) {
                const int back = TAPS - 1 - j, r = t - first;
                if (back <= r) {
                    cv_widen(win[j], *(const uint4*)(x + (size_t)(t - back) * x_stride + c));
                } else {
                    const float* k = kept + (size_t)(TAPS - 1 - (back - r)) * C + c;
                    if (kept4) {
                        cv_load8(win[j], k);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) win[j][i] = k[i];
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j)
#pragma unroll
                for (int i = 0; i < 8; ++i) win[j][i] = win[j + 1][i];
        }
        cv_widen(win[TAPS - 1], rows[u]);
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float a = bs[i];
#pragma unroll
            for (int j = 0; j < TAPS; ++j) a = fmaf(wt[i * TAPS + j], win[j][i], a);
            o[i] = __fdividef(a, 1.f + __expf(-a));
        }
        cv_store(y + (size_t)t * C + c, o);
    }
}

// After the convolution has run: the kept inputs of every request become the last taps - 1
// of (kept inputs, then the step's inputs). A thread per (request, channel).
template <typename T>
__global__ void __launch_bounds__(256)
causal_conv_keep_kernel(const T* __restrict__ x, long long x_stride, int C, int taps,
                        const int* __restrict__ q_start, const int* __restrict__ state_slots,
                        float* __restrict__ state, long long state_stride, long long conv_offset) {
    pdl_wait();
    const int b = blockIdx.x;
    const int t0 = q_start[b], n = q_start[b + 1] - t0;
    float* kept = state + (size_t)state_slots[b] * state_stride + conv_offset;
    const int keep = taps - 1;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        // ascending i reads kept[n + i] before any later write could reach it (n + i >= i)
        for (int i = 0; i < keep; ++i) {
            const int at = n + i;                        // place in (kept, then new)
            const float v = at < keep ? kept[(size_t)at * C + c]
                                      : to_f32(x[(size_t)(t0 + at - keep) * x_stride + c]);
            kept[(size_t)i * C + c] = v;
        }
    }
}

// y_dtype: float32, or the storage type. `keep` 0 leaves the kept inputs where they are (the
// channel scan below moves them on itself).
TGO_API int tgo_causal_conv_act(const void* x, long long x_stride, int dtype, const float* w,
                                const float* bias, void* y, int y_dtype, int T, int B, int C, int taps,
                                const int* seq_ids, const int* q_start, const int* state_slots,
                                float* state, long long state_stride, long long conv_offset, int keep,
                                cudaStream_t stream) {
    if (T <= 0 || B <= 0) return 0;
    if (C <= 0 || taps <= 0 || taps > 64 || state_stride < conv_offset + (long long)(taps - 1) * C)
        return TGO_E_BAD_ARG;
    const int cy = (C + 255) / 256 > 64 ? 64 : (C + 255) / 256;
    int rc;
#define CONV_GO(TT, TY)                                                                                    \
    tgo_launch_pdl(causal_conv_act_kernel<TT, TY>, dim3(T, cy), dim3(256), 0, stream, (const TT*)x, x_stride, w, \
                   bias, (TY*)y, C, taps, seq_ids, q_start, state_slots, (const float*)state, state_stride, \
                   conv_offset)
    const int kept4 = state_stride % 4 == 0 && conv_offset % 4 == 0 && (uintptr_t)state % 16 == 0;
#define CONV_X8_AT(TY, TAPS, TOK)                                                                          \
    tgo_launch_pdl(causal_conv_act_x8_kernel<TY, TAPS, TOK>, dim3((T + TOK - 1) / TOK, (C / 8 + 127) / 128),       \
                   dim3(128), 0, stream, (const bf16*)x, x_stride, w, bias, (TY*)y, T, C, seq_ids, q_start,      \
                   state_slots, (const float*)state, state_stride, conv_offset, kept4)
#define CONV_X8(TY, TAPS) (T == B ? CONV_X8_AT(TY, TAPS, 1) : CONV_X8_AT(TY, TAPS, CV_TOK))
#define CONV_TAPS(TY) (taps == 1 ? CONV_X8(TY, 1) : taps == 2 ? CONV_X8(TY, 2) : taps == 3 ? CONV_X8(TY, 3) : CONV_X8(TY, 4))
    if (dtype == TGO_BF16 && (y_dtype == TGO_F32 || y_dtype == TGO_BF16) && taps <= 4 && C % 8 == 0 &&
        x_stride % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)w % 16 == 0 &&
        (uintptr_t)bias % 16 == 0)
        rc = y_dtype == TGO_F32 ? CONV_TAPS(float) : CONV_TAPS(bf16);
    else if (dtype == TGO_BF16 && y_dtype == TGO_F32) rc = CONV_GO(bf16, float);
    else if (dtype == TGO_BF16 && y_dtype == TGO_BF16) rc = CONV_GO(bf16, bf16);
    else if (dtype == TGO_F32 && y_dtype == TGO_F32) rc = CONV_GO(float, float);
    else return TGO_E_BAD_ARG;
#undef CONV_GO
#undef CONV_X8
#undef CONV_X8_AT
#undef CONV_TAPS
    if (rc || taps == 1 || !keep) return rc;
    if (dtype == TGO_BF16)
        return tgo_launch_pdl(causal_conv_keep_kernel<bf16>, dim3(B, cy), dim3(256), 0, stream, (const bf16*)x,
                              x_stride, C, taps, q_start, state_slots, state, state_stride, conv_offset);
    return tgo_launch_pdl(causal_conv_keep_kernel<float>, dim3(B, cy), dim3(256), 0, stream, (const float*)x,
                          x_stride, C, taps, q_start, state_slots, state, state_stride, conv_offset);
}

// -------------------------------------------------------------------------------- scan
// A block per (request, head, 32 columns of P). 256 threads: thread (column c = tid / 8,
// slice s = tid % 8) keeps rows n = 32 i + 4 s + j (j = 0..3) of its column of S in registers
// for the whole walk over the request's tokens; a token's y[c] is the sum of the eight
// slices' partial sums (three shuffles, the same order for every token). The tokens' B, C, x
// and dt come through shared memory SS_TOK at a time, two buffers: the next tokens load while
// these are walked; B and C are read four rows at a time. The order of every sum depends on
// the sizes alone, so a token's result does not depend on how the tokens were cut or batched
// beyond the state's own history, which is the same sequence of updates whatever the cut.
#define SS_TOK 16
#define SS_COLS 32

// a 4-byte asynchronous copy into shared memory (zeros when !valid)
__device__ __forceinline__ void ss_copy4(float* dst, const float* src, bool valid) {
    const int n = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n));
}

template <typename T, int NI>
__global__ void __launch_bounds__(256)
selective_scan_kernel(const float* __restrict__ xbc, int C, const T* __restrict__ dt_raw,
                      long long dt_stride, const float* __restrict__ dt_bias,
                      const float* __restrict__ A_log, const float* __restrict__ D,
                      float* __restrict__ y, int H, int G, int N, int P,
                      const int* __restrict__ q_start, const int* __restrict__ state_slots,
                      float* __restrict__ state, long long state_stride, long long ssm_offset) {
    constexpr int NP = NI * 8;                           // N rounded up to whole rounds of 32
    extern __shared__ __align__(16) float smem[];
    // per buffer: B [SS_TOK][NP], C [SS_TOK][NP], x [SS_TOK][SS_COLS], dt [SS_TOK], decay [SS_TOK]
    constexpr int BUF = 2 * SS_TOK * NP + SS_TOK * SS_COLS + 2 * SS_TOK;
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * SS_COLS;
    const int g = h / (H / G);
    const int inner = H * P;
    const int col = threadIdx.x >> 3, s = threadIdx.x & 7;
    const int c = c0 + col;
    const bool live = c < P;
    const int t0 = q_start[b], n_tok = q_start[b + 1] - t0;
    float* Sg = state + (size_t)state_slots[b] * state_stride + ssm_offset + (size_t)h * N * P;
    // the state comes and goes through shared memory, so that global memory sees whole rows
    // of 32 columns (the staging buffers are idle then; [N][33] floats fit in them)
    float S[NI];
    for (int i = threadIdx.x; i < N * SS_COLS; i += 256) {
        const int n = i / SS_COLS, cc = i % SS_COLS;
        smem[n * (SS_COLS + 1) + cc] = c0 + cc < P ? Sg[(size_t)n * P + c0 + cc] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int n = 32 * (i >> 2) + 4 * s + (i & 3);
        S[i] = n < N ? smem[n * (SS_COLS + 1) + col] : 0.f;
    }
    __syncthreads();
    const float A = expf(A_log[h]);
    const float Dh = D ? D[h] : 0.f;
    const float bias = dt_bias ? dt_bias[h] : 0.f;
    auto stage = [&](int base, int buf) {
        float* Bs = smem + buf * BUF;
        float* Cs = Bs + SS_TOK * NP;
        float* xs = Cs + SS_TOK * NP;
        float* dts = xs + SS_TOK * SS_COLS;
        float* das = dts + SS_TOK;
        const int nt = n_tok - base < SS_TOK ? n_tok - base : SS_TOK;
        for (int i = threadIdx.x; i < nt * NP; i += 256) {
            const int r = i / NP, n = i % NP;
            const float* row = xbc + (size_t)(t0 + base + r) * C + inner + (size_t)g * N;
            ss_copy4(Bs + i, n < N ? row + n : xbc, n < N);
            ss_copy4(Cs + i, n < N ? row + (size_t)G * N + n : xbc, n < N);
        }
        for (int i = threadIdx.x; i < nt * SS_COLS; i += 256) {
            const int r = i / SS_COLS, cc = i % SS_COLS;
            const bool ok = c0 + cc < P;
            ss_copy4(xs + i, ok ? xbc + (size_t)(t0 + base + r) * C + (size_t)h * P + c0 + cc : xbc, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::);
        if (threadIdx.x < nt) {
            const float z = to_f32(dt_raw[(size_t)(t0 + base + threadIdx.x) * dt_stride + h]) + bias;
            const float dt = z > 20.f ? z : log1pf(expf(z));
            dts[threadIdx.x] = dt;
            das[threadIdx.x] = expf(-A * dt);
        }
    };
    stage(0, 0);
    for (int base = 0, buf = 0; base < n_tok; base += SS_TOK, buf ^= 1) {
        const int nt = n_tok - base < SS_TOK ? n_tok - base : SS_TOK;
        if (base + SS_TOK < n_tok) {
            stage(base + SS_TOK, buf ^ 1);                // the buffer the last pass left
            asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        const float* Bs = smem + buf * BUF;
        const float* Cs = Bs + SS_TOK * NP;
        const float* xs = Cs + SS_TOK * NP;
        const float* dts = xs + SS_TOK * SS_COLS;
        const float* das = dts + SS_TOK;
        for (int r = 0; r < nt; ++r) {
            const float x = xs[r * SS_COLS + col];
            const float dx = dts[r] * x, da = das[r];
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i4 = 0; i4 < NI / 4; ++i4) {
                const float4 bq = *(const float4*)(Bs + r * NP + 32 * i4 + 4 * s);
                const float4 cq = *(const float4*)(Cs + r * NP + 32 * i4 + 4 * s);
                S[4 * i4 + 0] = fmaf(da, S[4 * i4 + 0], dx * bq.x);
                S[4 * i4 + 1] = fmaf(da, S[4 * i4 + 1], dx * bq.y);
                S[4 * i4 + 2] = fmaf(da, S[4 * i4 + 2], dx * bq.z);
                S[4 * i4 + 3] = fmaf(da, S[4 * i4 + 3], dx * bq.w);
                part[0] = fmaf(S[4 * i4 + 0], cq.x, part[0]);
                part[1] = fmaf(S[4 * i4 + 1], cq.y, part[1]);
                part[2] = fmaf(S[4 * i4 + 2], cq.z, part[2]);
                part[3] = fmaf(S[4 * i4 + 3], cq.w, part[3]);
            }
            float sum = (part[0] + part[1]) + (part[2] + part[3]);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            if (s == 0 && live) y[(size_t)(t0 + base + r) * inner + (size_t)h * P + c] = sum + Dh * x;
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int n = 32 * (i >> 2) + 4 * s + (i & 3);
        if (n < N) smem[n * (SS_COLS + 1) + col] = S[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N * SS_COLS; i += 256) {
        const int n = i / SS_COLS, cc = i % SS_COLS;
        if (c0 + cc < P) Sg[(size_t)n * P + c0 + cc] = smem[n * (SS_COLS + 1) + cc];
    }
}

template <typename T, int NI>
static int launch_scan(const float* xbc, int C, const T* dt_raw, long long dt_stride,
                       const float* dt_bias, const float* A_log, const float* D, float* y, int B,
                       int H, int G, int N, int P, const int* q_start, const int* state_slots,
                       float* state, long long state_stride, long long ssm_offset,
                       cudaStream_t stream) {
    const size_t smem = 2 * ((size_t)2 * SS_TOK * NI * 8 + SS_TOK * SS_COLS + 2 * SS_TOK) * sizeof(float);
    auto kernel = selective_scan_kernel<T, NI>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return tgo_launch_pdl(kernel, dim3(B, H, (P + SS_COLS - 1) / SS_COLS), dim3(256),
                          smem, stream, xbc, C, dt_raw, dt_stride, dt_bias, A_log, D, y, H, G, N, P,
                          q_start, state_slots, state, state_stride, ssm_offset);
}

template <typename T>
static int scan_by_size(const float* xbc, int C, const T* dt_raw, long long dt_stride,
                        const float* dt_bias, const float* A_log, const float* D, float* y, int B,
                        int H, int G, int N, int P, const int* q_start, const int* state_slots,
                        float* state, long long state_stride, long long ssm_offset,
                        cudaStream_t stream) {
#define SS_GO(NI) launch_scan<T, NI>(xbc, C, dt_raw, dt_stride, dt_bias, A_log, D, y, B, H, G, N, P, \
                                     q_start, state_slots, state, state_stride, ssm_offset, stream)
    const int ni = (N + 7) / 8;
    if (ni <= 4) return SS_GO(4);
    if (ni <= 8) return SS_GO(8);
    if (ni <= 16) return SS_GO(16);
    return SS_GO(32);
#undef SS_GO
}

// xbc float32 [T, C], C = H P + 2 G N: the convolution's output (x, then B, then C of every
// group); dt_raw a column view [T, H] in the storage type; y float32 [T, H P].
TGO_API int tgo_selective_scan(const float* xbc, int C, const void* dt_raw, long long dt_stride,
                               int dtype, const float* dt_bias, const float* A_log, const float* D,
                               float* y, int B, int H, int G, int N, int P, const int* q_start,
                               const int* state_slots, float* state, long long state_stride,
                               long long ssm_offset, cudaStream_t stream) {
    if (B <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || N <= 0 || N > 256 || P <= 0 || H > 65535 ||
        C != H * P + 2 * G * N || state_stride < ssm_offset + (long long)H * N * P)
        return TGO_E_BAD_ARG;
    if (dtype == TGO_BF16)
        return scan_by_size<bf16>(xbc, C, (const bf16*)dt_raw, dt_stride, dt_bias, A_log, D, y, B, H, G, N,
                                  P, q_start, state_slots, state, state_stride, ssm_offset, stream);
    if (dtype == TGO_F32)
        return scan_by_size<float>(xbc, C, (const float*)dt_raw, dt_stride, dt_bias, A_log, D, y, B, H, G, N,
                                   P, q_start, state_slots, state, state_stride, ssm_offset, stream);
    return TGO_E_BAD_ARG;
}

// ------------------------------------------------------------------- scan over prompt portions
// The recurrence written out over chunks of up to SD_CHUNK tokens of one request, so that chunks of
// every head run side by side. With L_i the logarithm of the product of the decays up to and with
// token i of the chunk (n tokens), v_j = dt_j x_j:
//
//   y_i = exp(L_i) S^T C_i + sum_{j<=i} exp(L_i - L_j) (C_i . B_j) v_j + D x_i
//   S  <- exp(L_n) S + sum_j exp(L_n - L_j) B_j v_j^T
//
// Four launches: steps (dt and L of every token; L in 64 bits, so that the differences of large
// sums lose nothing), summaries (the sum of S's line), a scan over the chunks, which leaves the
// state before each chunk in its summary's place, and outputs. MEASURED (B200, 2048 tokens, 64 heads of 64 x 128):
// 711 us by the walk above, 224 with float32 products in register tiles of packed FMA (summaries 52, scan over the
// chunks 32, outputs 132), 151 with their parts on the tensor cores (31, 32, 84); errors against 64 bits, means of 15
// draws: outputs 0.9e-7 (1.1e-7 by FMA), state 8.4e-8 (8.7e-8).
// The workspace is a state's size a chunk and head; a call whose workspace does not hold all heads takes
// them in groups, one after the other over the same memory (heads do not meet; the sums are the same).
// The walk stays for the float32 engine, whose sums do not depend on how a prompt is cut, for
// steps of few tokens a request, and for other sizes.
#define SD_CHUNK 64

// The request and tokens of chunk `ci` (chunks are numbered request after request): false past the
// last. One warp.
__device__ __forceinline__ bool sd_find(const int* __restrict__ q_start, int B, int ci, int& b, int& tok0, int& n, int& nth) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int b0 = 0; b0 < B; b0 += 32) {
        const int r = b0 + lane;
        const int s = r < B ? q_start[r] : 0, len = r < B ? q_start[r + 1] - s : 0;
        const int c = (len + SD_CHUNK - 1) / SD_CHUNK;
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += a;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, ci < before + incl);
        if (hit) {
            const int src = __ffs(hit) - 1;
            nth = ci - before - __shfl_sync(0xffffffffu, incl - c, src);
            const int start = __shfl_sync(0xffffffffu, s, src), all = __shfl_sync(0xffffffffu, len, src);
            b = b0 + src;
            tok0 = start + nth * SD_CHUNK;
            n = all - nth * SD_CHUNK < SD_CHUNK ? all - nth * SD_CHUNK : SD_CHUNK;
            return true;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    return false;
}

// chunks [chunks][4]: first token, tokens, request, place among the request's chunks (tokens 0: none).
// dts, cum [chunks][H][SD_CHUNK].
template <typename T>
__global__ void __launch_bounds__(256)
ssd_steps_kernel(const T* __restrict__ dt_raw, long long dt_stride, const float* __restrict__ dt_bias,
                 const float* __restrict__ A_log, int H, const int* __restrict__ q_start, int B,
                 int4* __restrict__ chunks, float* __restrict__ dts, double* __restrict__ cum) {
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ci = blockIdx.x;
    int b = 0, tok0 = 0, n = 0, nth = 0;
    if (!sd_find(q_start, B, ci, b, tok0, n, nth)) n = 0;
    if (blockIdx.y == 0 && threadIdx.x == 0) chunks[ci] = make_int4(tok0, n, b, nth);
    const int h = blockIdx.y * 8 + warp;
    if (n == 0 || h >= H) return;
    const float A = expf(A_log[h]), bias = dt_bias ? dt_bias[h] : 0.f;
    double l[2];
    float dt[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {                        // tokens 2 lane, 2 lane + 1
        const int t = 2 * lane + i;
        dt[i] = 0.f;
        if (t < n) {
            const float z = to_f32(dt_raw[(size_t)(tok0 + t) * dt_stride + h]) + bias;
            dt[i] = z > 20.f ? z : log1pf(expf(z));
        }
        // A decay below 2^-369 is 0 in 32 bits, beside whatever it is multiplied by: held at exp(-256), so that
        // differences of sums stay numbers where A is infinite. (NaN stays NaN.)
        l[i] = t < n ? -(double)A * (double)dt[i] : 0.0;
        if (l[i] < -256.0) l[i] = -256.0;
    }
    double incl = l[0] + l[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += a;
    }
    const double before = __shfl_up_sync(0xffffffffu, incl, 1);
    const size_t at = ((size_t)ci * H + h) * SD_CHUNK + 2 * lane;
    *(float2*)(dts + at) = make_float2(dt[0], dt[1]);
    *(double2*)(cum + at) = make_double2((lane ? before : 0.0) + l[0], incl);
}

// ---- the products, in true float32 on the tensor cores (split3.cuh): three bfloat16 parts a number
// A block takes a chunk's rows of several heads of one group, whose B and C are the same, 128 of their channels ("a
// pair": two heads of 64, or one of 128) at a time: channels are the accumulators' lanes, tokens or states their
// columns, so that every operand is laid down as it lies in memory and a warp's results leave as whole lines.
// Sixteen warps lay parts down and write results, one issues. In the outputs A = exp(L_i - L_j) dt_j (C . B) has D on
// its diagonal, so that x goes in as it is and nothing is read for the results. Bound by the chains of conversions (about 2500
// cycles a stage of 64 x 128 numbers for eight warps) and not by the products, 50 cycles each. Zeros of A times a value that is not finite are not
// zero: such a number is laid down as 0, which leaves what does not depend on it as it is, bit for bit, and a
// block that met one makes plain sums too (SD_PLAIN of a column a thread; MEASURED: 2048 tokens, 64 heads of 64 x 128, all NaN 1180 us, all finite 157; 2820
// by a thread a sum) and writes those that are not finite. A
// finite number too large for its parts (2^103 and more), or an A whose C . B is (2^80), is 0 there too: the plain sums of its row
// and the rows after it are written whatever they are, of its head if it is not one of B or C. So are those in the place of a result
// that the products made overflow.
#define SD_THREADS 512
#define SD_HALF 256                   // of the outputs: one half lays the states and values down, the other A
#define SD_HEADS 16                   // heads a block takes at most
#define SD_TILE 8192                  // 64 rows of 64 bfloat16 numbers
#define SD_PLAIN 16                   // plain sums a thread makes side by side

__device__ int ssd_error_flag = 0;

__device__ __forceinline__ bool sd_not_finite(float x) { return !(fabsf(x) < __int_as_float(0x7f800000)); }
__device__ __forceinline__ void sd_eight(float (&f)[8], float4 a, float4 b, float w, bool ok) {
    f[0] = ok ? a.x * w : 0.f; f[1] = ok ? a.y * w : 0.f; f[2] = ok ? a.z * w : 0.f; f[3] = ok ? a.w * w : 0.f;
    f[4] = ok ? b.x * w : 0.f; f[5] = ok ? b.y * w : 0.f; f[6] = ok ? b.z * w : 0.f; f[7] = ok ? b.w * w : 0.f;
}
// A warp's share of an operand is laid down.
__device__ __forceinline__ void sd_full(uint64_t* bar) {
    s3_fence();
    tg_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) tg_arrive(bar);
}
// For a whole warp: the phase of a barrier is over.
__device__ __forceinline__ bool sd_wait(uint64_t* bar, uint32_t phase, int code) {
    const bool ok = __all_sync(0xffffffffu, tg_wait(bar, phase, &ssd_error_flag, code));
    tg_after();
    return ok;
}
// Barrier of THREADS threads that leave together: whether no wait of theirs has run out.
template <int THREADS> __device__ __forceinline__ bool sd_sync(bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                 "bar.red.and.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)ok), "n"(THREADS) : "memory");
    return r != 0;
}
// A chunk's B or C, 64 rows of N states: asked for, then laid down (rows of tokens, N / 64 tiles a part).
template <int N> struct SdRows {
    static constexpr int RUNS = SD_CHUNK * (N / 8) / SD_THREADS;
    float4 v[RUNS][2];
    __device__ __forceinline__ void load(const float* __restrict__ rows, int C, int n) {
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            const int i = threadIdx.x + j * SD_THREADS, r = i / (N / 8);
            const float4* src = (const float4*)(rows + (size_t)(r < n ? r : 0) * C + (i % (N / 8)) * 8);
            v[j][0] = src[0];
            v[j][1] = src[1];
        }
    }
    __device__ __forceinline__ bool put(uint32_t tile, int n, int* too_large) const {
        float f[RUNS][8];
        uint32_t dst[RUNS];
        int row[RUNS];
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            const int i = threadIdx.x + j * SD_THREADS, r = i / (N / 8), piece = i % (N / 8);
            sd_eight(f[j], v[j][0], v[j][1], 1.f, r < n);
            dst[j] = tile + (piece >> 3) * SD_TILE + s3_place(r, piece & 7);
            row[j] = r;
        }
        return s3_put<RUNS>(f, dst, N / 64 * SD_TILE, row, too_large);
    }
};
// x of a pair: 64 rows of 128 channels of neighbouring heads (channels past `width` are zeros), a row and head times
// its weight; two tiles of 64 channels a part.
template <int THREADS> struct SdPair {
    static constexpr int RUNS = SD_CHUNK * 16 / THREADS;
    float4 v[RUNS][2];
    __device__ __forceinline__ void load(const float* __restrict__ rows, int C, int n, int width) {
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            const int i = threadIdx.x + j * THREADS, r = i / 16, c = (i % 16) * 8;
            const float4* src = (const float4*)(rows + (size_t)(r < n ? r : 0) * C + (c < width ? c : 0));
            v[j][0] = src[0];
            v[j][1] = src[1];
        }
    }
    // weights [128 / P][SD_CHUNK]; null: none. too_large: a place for each of the heads
    template <int P> __device__ __forceinline__ bool put(uint32_t tile, int n, int width, const float (*weights)[SD_CHUNK], int* too_large) const {
        bool odd = false;
        const int head = threadIdx.x % 16 * 8 / P;       // the same in every turn
#pragma unroll
        for (int j0 = 0; j0 < RUNS; j0 += 2) {
            float f[2][8];
            uint32_t dst[2];
            int row[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int i = threadIdx.x + (j0 + j) * THREADS, r = i / 16, piece = i % 16;
                const bool in = r < n && piece * 8 < width;
                sd_eight(f[j], v[j0 + j][0], v[j0 + j][1], in && weights ? weights[head][r] : 1.f, in);
                dst[j] = tile + (piece >> 3) * SD_TILE + s3_place(r, piece & 7);
                row[j] = r;
            }
            odd = s3_put<2>(f, dst, 2 * SD_TILE, row, too_large + head) || odd;
        }
        return odd;
    }
};

// The plain sums of a block that met a number which is not finite or too large. Not inlined: the products' chains take 2 to 4 % longer beside them.
template <int N, int P>
__device__ __noinline__ void sd_plain_summaries(float* Bf, const float* __restrict__ rows, const float* __restrict__ br, int C, int h0, int hb, int n,
                                                const float* __restrict__ dts, const double* __restrict__ cum, const int* too_large, float* U) {
    // Bf [64][N]
    float* Wf = Bf + SD_CHUNK * N;                   // [hb][64]
    for (int i = threadIdx.x; i < n * N; i += SD_THREADS + 32) Bf[i] = br[(size_t)(i / N) * C + i % N];
    for (int i = threadIdx.x; i < hb * SD_CHUNK; i += SD_THREADS + 32) {
        const int end = i / SD_CHUNK * SD_CHUNK + n - 1;
        Wf[i] = i % SD_CHUNK < n ? dts[i] * expf((float)(cum[end] - cum[i])) : 0.f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < hb * (N / SD_PLAIN) * P; i += SD_THREADS + 32) {
        const int l = i / (N / SD_PLAIN * P), m = i / P % (N / SD_PLAIN) * SD_PLAIN, c = i % P;
        const bool plain = min(too_large[l], too_large[SD_HEADS]) < SD_CHUNK;
        float sum[SD_PLAIN] = {};
#pragma unroll 4
        for (int j = 0; j < n; ++j) {
            const float v = rows[(size_t)j * C + (h0 + l) * P + c] * Wf[l * SD_CHUNK + j];
#pragma unroll
            for (int r = 0; r < SD_PLAIN; ++r) sum[r] = fmaf(Bf[j * N + m + r], v, sum[r]);
        }
#pragma unroll
        for (int r = 0; r < SD_PLAIN; ++r) {
            float* to = U + (size_t)(l * N + m + r) * P + c;
            if (plain || sd_not_finite(sum[r]) || sd_not_finite(*to)) *to = sum[r];
        }
    }
}

// Shared memory: B's parts (N / 64 tiles a part), two buffers of a pair's weighted values (two tiles a part).
template <int N, int P>
__global__ void __launch_bounds__(SD_THREADS + 32, 1)
ssd_summaries_kernel(const float* __restrict__ xbc, int C, int H, int G, int first, int hb, const int4* __restrict__ chunks,
                     const float* __restrict__ dts, const double* __restrict__ cum, float* __restrict__ U) {
    constexpr int HP = 128 / P, NB = N / 64, STAGE = 6 * SD_TILE;
    extern __shared__ unsigned char sd_raw[];
    unsigned char* sB = (unsigned char*)(((uintptr_t)sd_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sV = sB + 3 * NB * SD_TILE;
    __shared__ float ws[2][HP][SD_CHUNK];
    __shared__ __align__(8) uint64_t bars[5];
    __shared__ uint32_t tmem_slot;
    __shared__ int too_large[SD_HEADS + 1];              // a head's x; B
    uint64_t *v_full = bars, *v_done = bars + 2, *settled = bars + 4;
    pdl_wait();
    const int4 ch = chunks[blockIdx.x];
    const int n = ch.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n == 0) return;
    const int nh = gridDim.y * hb, l0 = blockIdx.y * hb, h0 = first + l0, pairs = (hb + HP - 1) / HP;
    const float* rows = xbc + (size_t)ch.x * C;
    const size_t at = (size_t)blockIdx.x * nh + l0;      // the workspace holds the nh heads from `first` on
    if (warp == 0) tg_alloc<4 * N>(&tmem_slot);
    if (threadIdx.x <= SD_HEADS) too_large[threadIdx.x] = SD_CHUNK;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) { tg_init(&v_full[i], SD_THREADS / 32); tg_init(&v_done[i], 1); }
        tg_init(settled, 1);
        tg_init_done();
    }
    tg_before();
    __syncthreads();
    tg_after();
    const uint32_t tmem = tmem_slot;
    bool odd = false, ok = true;
    if (warp == SD_THREADS / 32) {
        const bool leader = tg_elect();
        for (int q = 0; q < pairs; ++q) {
            ok = sd_wait(&v_full[q & 1], (q >> 1) & 1, 1);
            if (!ok) break;
            if (leader) {
#pragma unroll
                for (int x = 0; x < 2; ++x)              // either half of the tokens for itself: the sums err less
                    s3_products<3, 3, SD_CHUNK / 32>(tmem + (uint32_t)(N * (2 * (q & 1) + x)), tg_desc_mn(sV + (q & 1) * STAGE, SD_TILE) + 256u * x,
                                                     2 * SD_TILE >> 4, 128, tg_desc_mn(sB, SD_TILE) + 256u * x, NB * SD_TILE >> 4, 128,
                                                     tg_idesc(N, true, true), false);
                tg_commit(&v_done[q & 1]);
            }
            __syncwarp();
        }
        if (!ok && leader) tg_settle_products(settled, &ssd_error_flag, 1);
    } else {
        SdRows<N> b;
        b.load(rows + H * P + (h0 / (H / G)) * N, C, n);
        SdPair<SD_THREADS> x;
        x.load(rows + h0 * P, C, n, min(hb, HP) * P);
        odd = b.put(tg_smem(sB), n, &too_large[SD_HEADS]);
        for (int q = 0; q <= pairs; ++q) {
            if (q < pairs) {
                const int heads = min(HP, hb - q * HP);
                // the buffers' products of the pair before the last have been waited for below
                if (threadIdx.x < heads * SD_CHUNK) {
                    const int e = threadIdx.x / SD_CHUNK, j = threadIdx.x % SD_CHUNK;
                    const size_t o = (at + q * HP + e) * SD_CHUNK;
                    ws[q & 1][e][j] = j < n ? dts[o + j] * expf((float)(cum[o + n - 1] - cum[o + j])) : 0.f;
                }
                ok = sd_sync<SD_THREADS>(ok);
                if (!ok) break;
                odd = x.put<P>(tg_smem(sV) + (q & 1) * STAGE, n, heads * P, ws[q & 1], &too_large[q * HP]) || odd;
                sd_full(&v_full[q & 1]);
                if (q + 1 < pairs) x.load(rows + (h0 + (q + 1) * HP) * P, C, n, min(HP, hb - (q + 1) * HP) * P);
            }
            if (q > 0) {                                 // the pair before this one
                const int d = q - 1, row = (warp & 3) * 32 + lane, l = d * HP + row / P;
                ok = sd_wait(&v_done[d & 1], (d >> 1) & 1, 2);
                constexpr int COLS = N / 4;              // states a warp
                const int n0 = (warp >> 2) * COLS;
                const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(2 * N * (d & 1) + n0);
                float* dst = U + ((at + l) * N + n0) * P + row % P;
#pragma unroll
                for (int c = 0; c < COLS; c += 16, dst += 16 * P) {
                    uint32_t r0[16], r1[16];
                    tg_ld16(t + c, r0);
                    tg_ld16(t + (uint32_t)(N + c), r1);
                    tg_wait_ld();
                    if (ok && l < hb)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float sum = (__uint_as_float(r0[i]) + __uint_as_float(r1[i])) * (S3_DOWN * S3_DOWN);
                            odd = odd || sd_not_finite(sum);
                            dst[i * P] = sum;
                        }
                }
                tg_before();                             // before the next products into this buffer
            }
        }
    }
    ok = __syncthreads_and(ok);
    if (__syncthreads_or(odd) && ok) {                   // plain sums
        sd_plain_summaries<N, P>((float*)sB, rows, rows + H * P + (h0 / (H / G)) * N, C, h0, hb, n, dts + at * SD_CHUNK, cum + at * SD_CHUNK, too_large, U + at * N * P);
    }
    tg_before();
    __syncthreads();
    if (warp == 0) {
        tg_after();
        tg_free<4 * N>(tmem_slot);
    }
}

// grid (requests, heads, ceil(N P / 1024)): a thread four neighbouring elements of the state
__global__ void __launch_bounds__(256)
ssd_scan_kernel(int H, int NP, const int* __restrict__ q_start, const int* __restrict__ state_slots,
                const double* __restrict__ cum, float* __restrict__ U, float* __restrict__ state, long long state_stride,
                long long offset) {
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y;
    const int e = 4 * (blockIdx.z * blockDim.x + threadIdx.x);
    const int n_tok = q_start[b + 1] - q_start[b];
    __shared__ int s_first;
    if (threadIdx.x < 32) {                              // chunks of the requests before this one
        int first = 0;
        for (int r = threadIdx.x; r < b; r += 32) first += (q_start[r + 1] - q_start[r] + SD_CHUNK - 1) / SD_CHUNK;
        first = __reduce_add_sync(0xffffffffu, first);
        if (threadIdx.x == 0) s_first = first;
    }
    __syncthreads();
    if (e >= NP || n_tok <= 0) return;
    const int chunks = (n_tok + SD_CHUNK - 1) / SD_CHUNK;
    const size_t first = ((size_t)s_first * H + h);
    float4* sp = (float4*)(state + (size_t)state_slots[b] * state_stride + offset + (size_t)h * NP + e);
    float4 s = *sp;
    const size_t step = (size_t)H * NP / 4;
    float4* ub = (float4*)(U + first * NP + e);
    const double* total = cum + first * SD_CHUNK;        // a chunk's whole decay stands at its last token
    constexpr int X = 8;
    float4 u[X], w[X];
#pragma unroll
    for (int x = 0; x < X; ++x) u[x] = x < chunks ? ub[(size_t)x * step] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int cb = 0; cb < chunks; cb += X) {
#pragma unroll
        for (int x = 0; x < X; ++x)
            w[x] = cb + X + x < chunks ? ub[(size_t)(cb + X + x) * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int x = 0; x < X; ++x) {
            const int c = cb + x;
            if (c >= chunks) break;
            ub[(size_t)c * step] = s;
            const int last = c == chunks - 1 ? n_tok - 1 - c * SD_CHUNK : SD_CHUNK - 1;
            const float g = expf((float)total[(size_t)c * H * SD_CHUNK + last]);
            s.x = fmaf(g, s.x, u[x].x); s.y = fmaf(g, s.y, u[x].y); s.z = fmaf(g, s.z, u[x].z); s.w = fmaf(g, s.w, u[x].w);
        }
#pragma unroll
        for (int x = 0; x < X; ++x) u[x] = w[x];
    }
    *sp = s;
}

// Shared memory: C's parts; B's, over which a pair's A come to lie (24 KB a head); two buffers that the states (64 of
// them x 128 channels a stage) and the values of a pair go through in turn.
template <int N, int P> __host__ __device__ constexpr int sd_a_bytes() {
    return 3 * (N / 64 > 128 / P ? N / 64 : 128 / P) * SD_TILE;
}
template <int N, int P> __host__ __device__ constexpr int sd_out_bytes() { return 3 * (N / 64) * SD_TILE + sd_a_bytes<N, P>() + 2 * 6 * SD_TILE; }

template <int N, int P>
__device__ __noinline__ void sd_plain_outputs(float* Cf, const float* __restrict__ rows, const float* __restrict__ brow, const float* __restrict__ crow,
                                              int C, int H, int h0, int hb, int n, const float* __restrict__ D, const double (*ls)[SD_CHUNK],
                                              const float (*ds)[SD_CHUNK], const float (*el)[SD_CHUNK], const int* plain_from,
                                              const float* __restrict__ U, float* y) {
    // Cf [64][N]
    float* Bf = Cf + SD_CHUNK * N;                   // [64][N + 1]
    float* Sf = Bf + SD_CHUNK * (N + 1);             // [64][65]
    for (int x = threadIdx.x; x < n * N; x += SD_THREADS + 32) {
        Cf[x] = crow[(size_t)(x / N) * C + x % N];
        Bf[x / N * (N + 1) + x % N] = brow[(size_t)(x / N) * C + x % N];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n * SD_CHUNK; x += SD_THREADS + 32) {
        const int i = x / SD_CHUNK, j = x % SD_CHUNK;
        float sum = 0.f;
        for (int m = 0; j <= i && m < N; ++m) sum = fmaf(Cf[i * N + m], Bf[j * (N + 1) + m], sum);
        Sf[i * (SD_CHUNK + 1) + j] = sum;
    }
    __syncthreads();
    for (int x = threadIdx.x; x < hb * (SD_CHUNK / SD_PLAIN) * P; x += SD_THREADS + 32) {
        const int l = x / (SD_CHUNK / SD_PLAIN * P), i = x / P % (SD_CHUNK / SD_PLAIN) * SD_PLAIN, c = x % P;
        if (i >= n) continue;                        // of rows past n the sums are made and not written
        const float* Uc = U + (size_t)l * N * P + c;
        const float* xc = rows + (h0 + l) * P + c;
        const int plain = min(plain_from[l], plain_from[SD_HEADS]);
        const float Dh = D ? D[h0 + l] : 0.f;
        float sum[SD_PLAIN] = {};
#pragma unroll 4
        for (int m = 0; m < N; ++m) {
            const float u = Uc[(size_t)m * P];
#pragma unroll
            for (int r = 0; r < SD_PLAIN; ++r) sum[r] = fmaf(Cf[(i + r) * N + m], u, sum[r]);
        }
#pragma unroll
        for (int r = 0; r < SD_PLAIN; ++r) sum[r] *= el[l][i + r];
        for (int j = 0; j < min(n, i + SD_PLAIN); ++j) {
            const float v = ds[l][j] * xc[(size_t)j * C];
#pragma unroll
            for (int r = 0; r < SD_PLAIN; ++r)
                if (j <= i + r) sum[r] = fmaf(Sf[(i + r) * (SD_CHUNK + 1) + j] * expf((float)(ls[l][i + r] - ls[l][j])), v, sum[r]);
        }
#pragma unroll
        for (int r = 0; r < SD_PLAIN; ++r) {
            if (i + r >= n) break;
            const float last = fmaf(Dh, xc[(size_t)(i + r) * C], sum[r]);
            float* to = y + (size_t)(i + r) * H * P + (h0 + l) * P + c;
            if (i + r >= plain || sd_not_finite(last) || sd_not_finite(*to)) *to = last;
        }
    }
}

template <int N, int P>
__global__ void __launch_bounds__(SD_THREADS + 32, 1)
ssd_outputs_kernel(const float* __restrict__ xbc, int C, int H, int G, int first, int hb, const float* __restrict__ D,
                   const int4* __restrict__ chunks, const float* __restrict__ dts, const double* __restrict__ cum,
                   const float* __restrict__ U, float* __restrict__ y) {
    constexpr int HP = 128 / P, HALVES = N / 64, STAGES = HALVES + 1, STAGE = 6 * SD_TILE;
    extern __shared__ unsigned char sd_raw[];
    unsigned char* sC = (unsigned char*)(((uintptr_t)sd_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sB = sC + 3 * HALVES * SD_TILE;
    unsigned char* sA = sB;
    unsigned char* sR = sB + sd_a_bytes<N, P>();         // [2]
    __shared__ double ls[SD_HEADS][SD_CHUNK];
    __shared__ float ds[SD_HEADS][SD_CHUNK], el[SD_HEADS][SD_CHUNK];
    __shared__ int plain_from[SD_HEADS + 1];             // the first row whose plain sums are written whatever they are: a head's; all heads'
    __shared__ __align__(8) uint64_t bars[13];
    __shared__ uint32_t tmem_slot;
    uint64_t *cb_full = bars, *s_done = bars + 1, *r_full = bars + 2 /* [2] */, *r_done = bars + 4 /* [2] */;
    // y_done, one a buffer: a warp hands over A of pair q before it waits for the products of pair q - 1, so that those
    // of q may be made first; the next phase of the same barrier, pair q + 1's, needs the warp's y_free of q - 1.
    uint64_t *y_done = bars + 6 /* [2] */, *a_full = bars + 8, *y_free = bars + 9 /* [2] */, *settled = bars + 11, *a_done = bars + 12;
    pdl_wait();
    const int4 ch = chunks[blockIdx.x];
    const int n = ch.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n == 0) return;
    const int nh = gridDim.y * hb, l0 = blockIdx.y * hb, h0 = first + l0, pairs = (hb + HP - 1) / HP;
    const float* rows = xbc + (size_t)ch.x * C;
    const float* brow = rows + H * P + (h0 / (H / G)) * N;
    const float* crow = brow + (size_t)G * N;
    const size_t at = (size_t)blockIdx.x * nh + l0;
    if (warp == 0) tg_alloc512(&tmem_slot);
    if (threadIdx.x == 0) {
        tg_init(cb_full, SD_THREADS / 32);
        tg_init(s_done, 1);
        for (int i = 0; i < 2; ++i) { tg_init(&r_full[i], SD_HALF / 32); tg_init(&r_done[i], 1); tg_init(&y_done[i], 1); tg_init(&y_free[i], SD_HALF / 32); }
        tg_init(a_full, SD_HALF / 32);
        tg_init(a_done, 1);
        tg_init(settled, 1);
        tg_init_done();
    }
    if (threadIdx.x <= SD_HEADS) plain_from[threadIdx.x] = SD_CHUNK;
    for (int i = threadIdx.x; i < hb * SD_CHUNK; i += SD_THREADS + 32) {
        const double l = cum[at * SD_CHUNK + i];
        (&ls[0][0])[i] = l;
        (&ds[0][0])[i] = dts[at * SD_CHUNK + i];
        (&el[0][0])[i] = expf((float)l);
    }
    tg_before();
    __syncthreads();
    tg_after();
    // columns: a pair's 256 begin at 256 (q & 1): C S by halves of the states (0, 64), A v of either head (128, 192).
    // C . B by halves lies in the second pair's first 128 until the first pair's A are made.
    const uint32_t tmem = tmem_slot, lanes = (uint32_t)((warp & 3) * 32) << 16;
    bool odd = false, ok = true;
    if (warp == SD_THREADS / 32) {
        // ---------------------------------------------------------- issuer
        const bool leader = tg_elect();
        ok = sd_wait(cb_full, 0, 3);
        if (ok && leader) {                              // rows 64.. of the accumulators are nobody's
#pragma unroll
            for (int x = 0; x < HALVES; ++x)
                s3_products<3, 3, 4>(tmem + 256u + 64u * x, tg_desc(sC + x * SD_TILE), HALVES * SD_TILE >> 4, 2, tg_desc(sB + x * SD_TILE),
                                     HALVES * SD_TILE >> 4, 2, tg_idesc(64), false);
            tg_commit(s_done);
        }
        __syncwarp();
        for (int q = 0, stage = 0; q < pairs && ok; ++q) {
            const uint32_t to = tmem + 256u * (q & 1);
            if (q > 1) ok = sd_wait(&y_free[q & 1], ((q >> 1) & 1) ^ 1, 3);      // the results of the pair before the last are out
            for (int x = 0; x < STAGES && ok; ++x, ++stage) {
                unsigned char* buf = sR + (stage & 1) * STAGE;
                ok = sd_wait(&r_full[stage & 1], (stage >> 1) & 1, 3);
                if (ok && x == 1) ok = sd_wait(a_full, q & 1, 3);
                if (!ok) break;
                if (leader) {
                    if (x != 1)
                        s3_products<3, 3, 4>(to + 64u * (x >> 1), tg_desc_mn(buf, SD_TILE), 2 * SD_TILE >> 4, 128,
                                             tg_desc(sC + (x >> 1) * SD_TILE), HALVES * SD_TILE >> 4, 2, tg_idesc(64, false, true), false);
                    else
#pragma unroll
                        for (int e = 0; e < HP; ++e)     // both heads' lanes, of which e's are read
                            s3_products<3, 3, 4>(to + 128u + 64u * e, tg_desc_mn(buf, SD_TILE), 2 * SD_TILE >> 4, 128,
                                                 tg_desc(sA + 3 * e * SD_TILE), SD_TILE >> 4, 2, tg_idesc(64, false, true), false);
                    tg_commit(&r_done[stage & 1]);
                    if (x == 1) tg_commit(a_done);
                    if (x == STAGES - 1) tg_commit(&y_done[q & 1]);
                }
                __syncwarp();
            }
        }
        if (!ok && leader) tg_settle_products(settled, &ssd_error_flag, 3);
    } else {
        {
            SdRows<N> c, b;
            c.load(crow, C, n);
            b.load(brow, C, n);
            odd = c.put(tg_smem(sC), n, &plain_from[SD_HEADS]);
            odd = b.put(tg_smem(sB), n, &plain_from[SD_HEADS]) || odd;
        }
        sd_full(cb_full);
        if (warp < SD_HALF / 32) {
            // ------------------------------------------------------ the states and values of the pairs
            // the states of a pair's heads [N][P] each: a stage is 64 states x 128 channels. The values come second, so
            // that A v is made while the other states are laid down.
            constexpr int RUNS = 64 * 16 / SD_HALF;
            float4 p[RUNS][2];
            auto ask = [&](int q, int x) {
#pragma unroll
                for (int j = 0; j < RUNS; ++j) {
                    const int i = threadIdx.x + j * SD_HALF, m = 64 * x + i / 16, c = (i % 16) * 8;
                    const int l = min(q * HP + c / P, hb - 1);
                    const float4* src = (const float4*)(U + ((at + l) * N + m) * P + c % P);
                    p[j][0] = src[0];
                    p[j][1] = src[1];
                }
            };
            ask(0, 0);
            SdPair<SD_HALF> v;
            for (int q = 0, stage = 0; q < pairs && ok; ++q) {
                const int heads = min(HP, hb - q * HP), width = heads * P;
                for (int x = 0; x < STAGES && ok; ++x, ++stage) {
                    if (stage > 1) ok = sd_wait(&r_done[stage & 1], ((stage >> 1) & 1) ^ 1, 4);
                    if (!ok) break;
                    const uint32_t buf = tg_smem(sR) + (stage & 1) * STAGE;
                    if (x != 1) {
#pragma unroll
                        for (int j0 = 0; j0 < RUNS; j0 += 2) {
                            float f[2][8];
                            uint32_t dst[2];
                            const int row[2] = {0, 0};   // every row sees the states
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                const int i = threadIdx.x + (j0 + j) * SD_HALF, piece = i % 16;
                                sd_eight(f[j], p[j0 + j][0], p[j0 + j][1], 1.f, piece * 8 < width);
                                dst[j] = buf + (piece >> 3) * SD_TILE + s3_place(i / 16, piece & 7);
                            }
                            odd = s3_put<2>(f, dst, 2 * SD_TILE, row, &plain_from[q * HP + threadIdx.x % 16 * 8 / P]) || odd;
                        }
                    } else {
                        odd = v.template put<P>(buf, n, width, nullptr, &plain_from[q * HP]) || odd;
                    }
                    sd_full(&r_full[stage & 1]);
                    if (x == 0) v.load(rows + (h0 + q * HP) * P, C, n, width);
                    else if (x + 1 < STAGES) ask(q, 1);
                    else if (q + 1 < pairs) ask(q + 1, 0);
                }
            }
        } else {
            // ------------------------------------------------------ A of the pairs, and their results
            const int tid = threadIdx.x - SD_HALF, ai = tid / 4, aj = tid % 4 * 8;       // two eights of every A: aj, aj + 32
            ok = sd_sync<SD_HALF>(sd_wait(s_done, 0, 6));
            float s[16];
            {                                            // C . B out of tensor memory, a row to four threads
                float* st = (float*)sB;                  // B's parts have been read
                if ((warp & 3) < 2) {
                    const int i = (warp & 3) * 32 + lane, j0 = (warp >> 2 & 1) * 32;
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        uint32_t s0[16], s1[16];
                        tg_ld16(tmem + lanes + 256u + (uint32_t)(j0 + c), s0);
                        if (HALVES > 1) tg_ld16(tmem + lanes + 320u + (uint32_t)(j0 + c), s1);
                        tg_wait_ld();
#pragma unroll
                        for (int x = 0; x < 16; ++x)
                            st[i * (SD_CHUNK + 1) + j0 + c + x] = (__uint_as_float(s0[x]) + (HALVES > 1 ? __uint_as_float(s1[x]) : 0.f)) * (S3_DOWN * S3_DOWN);
                    }
                }
                sd_sync<SD_HALF>(ok);
#pragma unroll
                for (int x = 0; x < 16; ++x) s[x] = st[ai * (SD_CHUNK + 1) + aj + (x & 7) + (x >> 3) * 32];
                sd_sync<SD_HALF>(ok);
            }
            for (int q = 0; q <= pairs && ok; ++q) {
                if (q > 0) ok = sd_wait(a_done, (q - 1) & 1, 5);     // A's place is free
                if (!ok) break;
                if (q < pairs) {
                    for (int e = 0; e < min(HP, hb - q * HP); ++e) {
                        const double* l = ls[q * HP + e];
                        const float* dt = ds[q * HP + e];
                        const double li = l[ai];
                        const float Dh = D ? D[h0 + q * HP + e] : 0.f;
                        float f[2][8];
#pragma unroll
                        for (int x = 0; x < 16; ++x) {
                            const int j = aj + (x & 7) + (x >> 3) * 32;
                            const float a = s[x] * (expf((float)(li - l[j])) * dt[j]);       // 0 to infinity past the diagonal
                            f[x >> 3][x & 7] = j > ai || ai >= n ? 0.f : j == ai ? a + Dh : a;
                        }
                        const uint32_t tile = tg_smem(sA) + (uint32_t)(3 * e * SD_TILE);
                        const uint32_t dst[2] = {tile + s3_place(ai, aj / 8), tile + s3_place(ai, aj / 8 + 4)};
                        const int at_row[2] = {ai, ai};
                        if (s3_put<2>(f, dst, SD_TILE, at_row, &plain_from[q * HP + e])) {
                            atomicMin(&plain_from[q * HP + e], ai);
                            odd = true;
                        }
                    }
                    sd_full(a_full);
                }
                if (q > 0) {
                    const int d = q - 1, row = (warp & 3) * 32 + lane, l = d * HP + row / P, i0 = (warp >> 2 & 1) * 32;
                    ok = sd_wait(&y_done[d & 1], (d >> 1) & 1, 5);
                    if (!ok) break;
                    const uint32_t t = tmem + lanes + 256u * (d & 1) + (uint32_t)i0;
                    float* dst = y + (size_t)(ch.x + i0) * H * P + (h0 + l) * P + row % P;
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        uint32_t a[16], p0[16], p1[16];
                        tg_ld16(t + 128u + 64u * (row / P) + c, a);
                        tg_ld16(t + c, p0);
                        if (HALVES > 1) tg_ld16(t + 64u + c, p1);
                        tg_wait_ld();
                        if (l < hb)
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                if (i0 + c + i < n) {
                                    const float far = __uint_as_float(p0[i]) + (HALVES > 1 ? __uint_as_float(p1[i]) : 0.f);
                                    const float sum = fmaf(far * (S3_DOWN * S3_DOWN), el[l][i0 + c + i], __uint_as_float(a[i]) * (S3_DOWN * S3_DOWN));
                                    odd = odd || sd_not_finite(sum);
                                    dst[(size_t)(c + i) * H * P] = sum;
                                }
                    }
                    sd_full(&y_free[d & 1]);
                }
            }
        }
    }
    ok = __syncthreads_and(ok);
    if (__syncthreads_or(odd) && ok) {                   // plain sums: a token past a row is not added at all
        sd_plain_outputs<N, P>((float*)sC, rows, brow, crow, C, H, h0, hb, n, D, ls, ds, el, plain_from, U + at * N * P, y + (size_t)ch.x * H * P);
    }
    tg_before();
    __syncthreads();
    if (warp == 0) {
        tg_after();
        tg_free512(tmem_slot);
    }
}

// The code a wait of the chunks' products left when it ran out (0: none did). Synchronises.
TGO_API int tgo_ssd_error(int* value) { return (int)cudaMemcpyFromSymbol(value, ssd_error_flag, sizeof(int)); }

TGO_API int tgo_ssd_chunk_tokens() { return SD_CHUNK; }
template <int N, int P>
static int ssd_go(const float* xbc, int C, const bf16* dt_raw, long long dt_stride, const float* dt_bias, const float* A_log,
                  const float* D, float* y, int T, int B, int H, int G, const int* q_start, const int* state_slots,
                  float* state, long long state_stride, long long offset, float* ws, int each, int hb, cudaStream_t stream) {
    constexpr size_t s1 = 1024 + (3 * (N / 64) + 2 * 6) * SD_TILE, s3 = 1024 + sd_out_bytes<N, P>();
    static_assert(s1 >= 1024 + SD_CHUNK * (N + SD_HEADS) * sizeof(float), "the plain sums' tiles");
    static_assert(s3 >= 1024 + SD_CHUNK * (2 * N + 1 + SD_CHUNK + 1) * sizeof(float), "the plain sums' tiles");
    static bool sized[64] = {};                          // per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
    if (!sized[dev]) {
        if ((e = cudaFuncSetAttribute(ssd_summaries_kernel<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1)) != cudaSuccess) return (int)e;
        if ((e = cudaFuncSetAttribute(ssd_outputs_kernel<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3)) != cudaSuccess) return (int)e;
        sized[dev] = true;
    }
    const int n_chunks = T / SD_CHUNK + B;               // at least as many as there are
    for (int h0 = 0; h0 < H; h0 += each) {
        const int nh = H - h0 < each ? H - h0 : each;
        float* U = ws;
        double* cum = (double*)(U + (size_t)n_chunks * nh * N * P);
        float* dts = (float*)(cum + (size_t)n_chunks * nh * SD_CHUNK);
        int4* chunks = (int4*)(dts + (size_t)n_chunks * nh * SD_CHUNK);
        int rc = tgo_launch_pdl(ssd_steps_kernel<bf16>, dim3(n_chunks, (nh + 7) / 8), dim3(256), 0, stream, dt_raw + h0, dt_stride,
                                dt_bias ? dt_bias + h0 : dt_bias, A_log + h0, nh, q_start, B, chunks, dts, cum);
        if (rc) return rc;
        rc = tgo_launch_pdl(ssd_summaries_kernel<N, P>, dim3(n_chunks, nh / hb), dim3(SD_THREADS + 32), s1, stream, xbc, C, H, G, h0,
                            hb, (const int4*)chunks, (const float*)dts, (const double*)cum, U);
        if (rc) return rc;
        rc = tgo_launch_pdl(ssd_scan_kernel, dim3(B, nh, (N * P / 4 + 255) / 256), dim3(256), 0, stream, nh, N * P, q_start,
                            state_slots, (const double*)cum, U, state, state_stride, offset + (long long)h0 * N * P);
        if (rc) return rc;
        rc = tgo_launch_pdl(ssd_outputs_kernel<N, P>, dim3(n_chunks, nh / hb), dim3(SD_THREADS + 32), s3, stream, xbc, C, H, G, h0, hb, D,
                            (const int4*)chunks, (const float*)dts, (const double*)cum, (const float*)U, y);
        if (rc) return rc;
    }
    return 0;
}

// 1 if the chunked scan takes these sizes and places (places as addresses); bfloat16 engine only.
TGO_API int tgo_ssd_takes(const void* xbc, const void* y, const void* state, long long state_stride, long long offset, int H,
                          int G, int N, int P) {
    return H > 0 && H <= 65535 && G > 0 && H % G == 0 && (N == 64 || N == 128) && (P == 64 || P == 128) &&
           (uintptr_t)xbc % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)state % 16 == 0 && state_stride % 4 == 0 &&
           offset % 4 == 0;
}

// Heads taken at a time, and 65536 times the heads of a block, where the workspace may have `ws_floats` floats: (T /
// tgo_ssd_chunk_tokens() + B) times (h (N P + 3 tgo_ssd_chunk_tokens()) + 4) for h heads at a time (a summary, the steps' sizes and
// logarithms, and what each chunk is). 0: not one head.
// Heads a block: as many of a group as leave a block a multiprocessor, so that B and C are laid down once for them.
// Heads at a time: about as many each time as the workspace makes needful, in whole blocks. What they take of the
// workspace gives the same answer again.
TGO_API int tgo_ssd_heads(int T, int B, int H, int G, int N, int P, long long ws_floats) {
    if (T <= 0 || B <= 0 || H <= 0 || H > 65535 || G <= 0 || H % G) return 0;
    const int n_chunks = T / SD_CHUNK + B, group = H / G;                // at least as many as there are
    long long most = (ws_floats / n_chunks - 4) / (N * P + 3 * SD_CHUNK);
    if (most <= 0) return 0;
    if (most > H) most = H;
    int answer = 0;
    for (int d = 1; d <= group && d <= most && d <= SD_HEADS; ++d) {
        if (group % d) continue;
        const int blocks = H / d, at_once = (int)(most / d), goes = (blocks + at_once - 1) / at_once;
        const int each = (blocks + goes - 1) / goes;
        if (d <= 128 / P || (long long)n_chunks * each >= tgo_multiprocessors()) answer = each * d + 65536 * d;
    }
    return answer;
}

// As tgo_selective_scan with dt_raw in bfloat16; ws: ws_floats floats, 16-byte aligned, shared out as tgo_ssd_heads says.
TGO_API int tgo_ssd_scan(const float* xbc, int C, const void* dt_raw, long long dt_stride, const float* dt_bias,
                         const float* A_log, const float* D, float* y, int T, int B, int H, int G, int N, int P,
                         const int* q_start, const int* state_slots, float* state, long long state_stride,
                         long long ssm_offset, float* ws, long long ws_floats, cudaStream_t stream) {
    if (B <= 0 || T <= 0) return 0;
    const int heads = tgo_ssd_heads(T, B, H, G, N, P, ws_floats), each = heads % 65536, hb = heads / 65536;
    if (!tgo_ssd_takes(xbc, y, state, state_stride, ssm_offset, H, G, N, P) || C != H * P + 2 * G * N ||
        state_stride < ssm_offset + (long long)H * N * P || !ws || (uintptr_t)ws % 16 || !heads)
        return TGO_E_BAD_ARG;
#define SD_GO(N, P)                                                                                                    \
    return ssd_go<N, P>(xbc, C, (const bf16*)dt_raw, dt_stride, dt_bias, A_log, D, y, T, B, H, G, q_start, state_slots, state, \
                        state_stride, ssm_offset, ws, each, hb, stream)
    if (N == 128) { if (P == 64) SD_GO(128, 64); SD_GO(128, 128); }
    if (P == 64) SD_GO(64, 64);
    SD_GO(64, 128);
#undef SD_GO
}

// ---------------------------------------------------------------------- scan per channel
// A block per (request, CS_WALK / L channels) whose threads have two roles and work on different
// tiles of TOK tokens at the same time. The walking warps: L lanes share a channel and lane l keeps states
// l * NS .. l * NS + NS - 1 of it in registers for the whole walk over the request's tokens. Four
// tokens are taken together: their decays do not depend on the state, so only one FMA per state
// and token is a chain, and the four sums over n are joined by a transposing exchange in the
// quad (three shuffles for four tokens) and, for L > 4, by shuffles over the quads, the same
// order for every token. Tokens past the end of a tile have dt = 0 and leave the state as it is.
// The serving warps: while tile k is walked it puts tile k + 1 into shared memory (dt through
// softplus once per (token, channel), beside dt * x; B and C as float32 rows), asks for tile
// k + 2's inputs, and finishes tile k - 1 (D x added, times silu(z), stored). `a2` is A log2(e).
//
// The walk ends with the convolution's kept inputs: the last taps - 1 of (kept, then the
// step's raw inputs `conv_in`), which the convolution has read before this kernel starts.
#define CS_WALK 128              // walking threads
// serving threads: 256 where a tile has a (token, channel) pair for each, else 128
#define CS_SERVE(TOK, L) ((TOK) * (CS_WALK / (L)) % 256 == 0 ? 256 : 128)

// One step of one state: 2^e S + add. A state that decays slowly is multiplied by nearly 1
// thousands of times, and an exponential that is off by the same fraction of a unit in the last
// place each time adds up; the float32 engine therefore takes the change S (2^e - 1), whose
// rounding is relative to the change, while the decay is slow.
template <typename T> __device__ __forceinline__ float cs_step(float S, float e, float add);
template <> __device__ __forceinline__ float cs_step<bf16>(float S, float e, float add) {
    float d;                                             // a decay below 2^-126 is none
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(e));
    return fmaf(d, S, add);
}
template <> __device__ __forceinline__ float cs_step<float>(float S, float e, float add) {
    if (e < -0.5f) return fmaf(exp2f(e), S, add);
    return S + fmaf(expm1f(e * 0.69314718055994531f), S, add);
}

// softplus and silu: the library's functions in the float32 engine; in the bfloat16 engine the
// special-function unit's exponential, logarithm and reciprocal (float32, a few units in the
// last place), with log(1 + e) by its series where e is small.
template <typename T> __device__ __forceinline__ float cs_softplus(float v);
template <> __device__ __forceinline__ float cs_softplus<float>(float v) { return v > 20.f ? v : log1pf(expf(v)); }
template <> __device__ __forceinline__ float cs_softplus<bf16>(float v) {
    const float e = __expf(v);
    const float small = e * fmaf(e, fmaf(e, fmaf(e, -0.25f, 0.33333334f), -0.5f), 1.f);
    return v > 20.f ? v : e < 0.03f ? small : __logf(1.f + e);
}
template <typename T> __device__ __forceinline__ float cs_silu(float z);
template <> __device__ __forceinline__ float cs_silu<float>(float z) { return z / (1.f + expf(-z)); }
template <> __device__ __forceinline__ float cs_silu<bf16>(float z) { return __fdividef(z, 1.f + __expf(-z)); }

// The kept inputs of one channel of one request.
template <typename T>
__device__ __forceinline__ void cs_keep(float* kept, const T* __restrict__ conv_in, long long conv_in_stride,
                                        int c, int C, int taps, int t0, int n_tok) {
    const int keep = taps - 1;
    // ascending i reads kept[n_tok + i] before any later write could reach it
    for (int i = 0; i < keep; ++i) {
        const int at = n_tok + i;                        // place in (kept, then new)
        kept[(size_t)i * C + c] = at < keep ? kept[(size_t)at * C + c]
                                            : to_f32(conv_in[(size_t)(t0 + at - keep) * conv_in_stride + c]);
    }
}

template <typename T, int L, int NS, int TOK>
__global__ void __launch_bounds__(CS_WALK + CS_SERVE(TOK, L))
channel_scan_kernel(const T* __restrict__ x, long long x_stride, const T* __restrict__ z, long long z_stride,
                    const float* __restrict__ dt_raw, long long dt_stride, const float* __restrict__ dt_bias,
                    const float* __restrict__ a2, const T* __restrict__ bm, const T* __restrict__ cm,
                    long long bc_stride, const float* __restrict__ D, T* __restrict__ y, int C, int N,
                    const int* __restrict__ q_start, const int* __restrict__ state_slots,
                    float* __restrict__ state, long long state_stride, long long ssm_offset,
                    const T* __restrict__ conv_in, long long conv_in_stride, int taps, long long conv_offset) {
    constexpr int CH = CS_WALK / L;                      // channels of this block
    constexpr int NP = L * NS;                           // N rounded up
    constexpr int SERVE = CS_SERVE(TOK, L);
    constexpr int PER = TOK * CH / SERVE;                // (token, channel) pairs a serving thread loads
    constexpr int RSTEP = SERVE / CH;                 // tokens between a thread's pairs
    constexpr int PBC = TOK * NP / SERVE;
    static_assert(TOK * CH % SERVE == 0 && TOK * NP % SERVE == 0, "tile");
    extern __shared__ __align__(16) float cs_smem[];
    float* s_b = cs_smem;                                // [2][TOK][NP]
    float* s_c = s_b + 2 * TOK * NP;                  // [2][TOK][NP]
    float2* s_dt = (float2*)(s_c + 2 * TOK * NP);     // [2][TOK][CH + 1]: dt, dt x
    float* s_y = (float*)(s_dt + 2 * TOK * (CH + 1)); // [2][TOK][CH + 1]
    pdl_wait();
    const int b = blockIdx.x, c0 = blockIdx.y * CH;
    const int t0 = q_start[b], n_tok = q_start[b + 1] - t0;
    const int n_tiles = (n_tok + TOK - 1) / TOK;
    float* row = state + (size_t)state_slots[b] * state_stride;
    if (threadIdx.x < CS_WALK) {
        // ---- walking
        const int tid = threadIdx.x;
        const int lane_l = tid % L, wch = tid / L, wc = c0 + wch, n0 = lane_l * NS;
        const bool live = wc < C;
        float S[NS], A[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const bool ok = live && n0 + i < N;
            S[i] = ok ? row[ssm_offset + (size_t)wc * N + n0 + i] : 0.f;
            A[i] = ok ? a2[(size_t)wc * N + n0 + i] : 0.f;
        }
        const bool odd = tid & 1, high = tid & 2;
        __syncthreads();                                 // tile 0 is in shared memory
        for (int k = 0; k < n_tiles; ++k) {
            const int nt = n_tok - k * TOK < TOK ? n_tok - k * TOK : TOK;
            const float2* dts = s_dt + (k & 1) * TOK * (CH + 1) + wch;
            const float* bs = s_b + (k & 1) * TOK * NP + n0;
            const float* cs = s_c + (k & 1) * TOK * NP + n0;
            float* ys = s_y + (k & 1) * TOK * (CH + 1) + wch;
            for (int r = 0; r < nt; r += 4) {
                float part[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float2 dd = dts[(r + u) * (CH + 1)];
                    const float* br = bs + (r + u) * NP;
                    const float* cr = cs + (r + u) * NP;
                    float p = 0.f, p2 = 0.f;
#pragma unroll
                    for (int i = 0; i < NS; i += 4) {
                        const float4 bq = *(const float4*)(br + i), cq = *(const float4*)(cr + i);
                        S[i] = cs_step<T>(S[i], dd.x * A[i], dd.y * bq.x);
                        S[i + 1] = cs_step<T>(S[i + 1], dd.x * A[i + 1], dd.y * bq.y);
                        S[i + 2] = cs_step<T>(S[i + 2], dd.x * A[i + 2], dd.y * bq.z);
                        S[i + 3] = cs_step<T>(S[i + 3], dd.x * A[i + 3], dd.y * bq.w);
                        p = fmaf(S[i], cq.x, p);
                        p2 = fmaf(S[i + 1], cq.y, p2);
                        p = fmaf(S[i + 2], cq.z, p);
                        p2 = fmaf(S[i + 3], cq.w, p2);
                    }
                    part[u] = p + p2;
                }
                // four sums over the quad, transposed: lane q of a quad ends with token r + q
                const float s0 = odd ? part[0] : part[1], s1 = odd ? part[2] : part[3];
                float k0 = odd ? part[1] : part[0], k1 = odd ? part[3] : part[2];
                k0 += __shfl_xor_sync(0xffffffffu, s0, 1);
                k1 += __shfl_xor_sync(0xffffffffu, s1, 1);
                const float s2 = high ? k0 : k1;
                float sum = high ? k1 : k0;
                sum += __shfl_xor_sync(0xffffffffu, s2, 2);
#pragma unroll
                for (int o = 4; o < L; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane_l < 4) ys[(r + (tid & 3)) * (CH + 1)] = sum;
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (live && n0 + i < N) row[ssm_offset + (size_t)wc * N + n0 + i] = S[i];
        return;
    }
    // ---- serving: channel lc, tokens lt + RSTEP i of a tile
    const int tid = threadIdx.x - CS_WALK;
    const int lcl = tid % CH, lc = c0 + lcl, lt = tid / CH;
    const bool lok = lc < C;
    const float bias = (lok && dt_bias) ? dt_bias[lc] : 0.f;
    const float skip = (lok && D) ? D[lc] : 0.f;
    const T zero = from_f32<T>(0.f);
    T xn[PER], bn[PBC], cn[PBC];                         // raw, so that nothing waits for them here
    float dn[PER];
    auto fetch = [&](int k) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = k * TOK + lt + RSTEP * i;
            const bool ok = lok && r < n_tok;
            const size_t t = (size_t)(t0 + r);
            xn[i] = ok ? x[t * x_stride + lc] : zero;
            dn[i] = ok ? dt_raw[t * dt_stride + lc] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < PBC; ++i) {
            const int q = tid + SERVE * i;
            const int r = k * TOK + q / NP, n = q % NP;
            const bool ok = n < N && r < n_tok;
            bn[i] = ok ? bm[(size_t)(t0 + r) * bc_stride + n] : zero;
            cn[i] = ok ? cm[(size_t)(t0 + r) * bc_stride + n] : zero;
        }
    };
    auto stage = [&](int k) {                            // what fetch(k) has brought
        float2* dts = s_dt + (k & 1) * TOK * (CH + 1);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = lt + RSTEP * i;
            const float dt = k * TOK + r < n_tok ? cs_softplus<T>(dn[i] + bias) : 0.f;
            dts[r * (CH + 1) + lcl] = make_float2(dt, dt * to_f32(xn[i]));
        }
#pragma unroll
        for (int i = 0; i < PBC; ++i) {
            s_b[(k & 1) * TOK * NP + tid + SERVE * i] = to_f32(bn[i]);
            s_c[(k & 1) * TOK * NP + tid + SERVE * i] = to_f32(cn[i]);
        }
    };
    T xr[PER], zr[PER];
    auto recall = [&](int k) {                           // x and z of a walked tile, ahead of their use
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = k * TOK + lt + RSTEP * i;
            const bool ok = lok && r < n_tok;
            xr[i] = ok ? x[(size_t)(t0 + r) * x_stride + lc] : zero;
            zr[i] = ok ? z[(size_t)(t0 + r) * z_stride + lc] : zero;
        }
    };
    auto finish = [&](int k) {                           // the walked tile k: gate and store
        const float* ys = s_y + (k & 1) * TOK * (CH + 1);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = lt + RSTEP * i;
            if (lok && k * TOK + r < n_tok)
                y[(size_t)(t0 + k * TOK + r) * C + lc] =
                    from_f32<T>(fmaf(skip, to_f32(xr[i]), ys[r * (CH + 1) + lcl]) * cs_silu<T>(to_f32(zr[i])));
        }
    };
    fetch(0);
    stage(0);
    if (n_tiles > 1) fetch(1);
    __syncthreads();
    for (int k = 0; k < n_tiles; ++k) {
        if (k > 0) recall(k - 1);
        if (k + 1 < n_tiles) stage(k + 1);
        if (k + 2 < n_tiles) fetch(k + 2);
        if (k > 0) finish(k - 1);
        __syncthreads();
    }
    if (n_tiles > 0) {
        recall(n_tiles - 1);
        finish(n_tiles - 1);
    }
    if (conv_in && tid < CH && c0 + tid < C)
        cs_keep(row + conv_offset, conv_in, conv_in_stride, c0 + tid, C, taps, t0, n_tok);
}

// A step in which every request brings one token: nothing to stage, a thread takes NS states of
// one channel of one request (L lanes a channel, four states a 16-byte access where they lie
// that way), the lanes join their sums and the first of them gates and stores.
template <typename T, int L, int NS, bool VEC>
__global__ void __launch_bounds__(128)
channel_scan_single_kernel(const T* __restrict__ x, long long x_stride, const T* __restrict__ z, long long z_stride,
                           const float* __restrict__ dt_raw, long long dt_stride, const float* __restrict__ dt_bias,
                           const float* __restrict__ a2, const T* __restrict__ bm, const T* __restrict__ cm,
                           long long bc_stride, const float* __restrict__ D, T* __restrict__ y, int C, int N,
                           const int* __restrict__ q_start, const int* __restrict__ state_slots,
                           float* __restrict__ state, long long state_stride, long long ssm_offset,
                           const T* __restrict__ conv_in, long long conv_in_stride, int taps, long long conv_offset) {
    constexpr int CH = 128 / L;
    pdl_wait();
    const int b = blockIdx.x, lane_l = threadIdx.x % L, n0 = lane_l * NS;
    const int c = blockIdx.y * CH + threadIdx.x / L;
    const bool live = c < C;
    const int t = q_start[b];
    float* row = state + (size_t)state_slots[b] * state_stride;
    float* Sg = row + ssm_offset + (size_t)(live ? c : 0) * N + n0;
    const float* Ag = a2 + (size_t)(live ? c : 0) * N + n0;
    float S[NS], A[NS];
    if (VEC) {
#pragma unroll
        for (int i = 0; i < NS; i += 4) {
            const bool ok = live && n0 + i < N;          // N % 4 == 0: the four are in or out together
            const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 s4 = ok ? *(const float4*)(Sg + i) : zero4, a4 = ok ? *(const float4*)(Ag + i) : zero4;
            S[i] = s4.x; S[i + 1] = s4.y; S[i + 2] = s4.z; S[i + 3] = s4.w;
            A[i] = a4.x; A[i + 1] = a4.y; A[i + 2] = a4.z; A[i + 3] = a4.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const bool ok = live && n0 + i < N;
            S[i] = ok ? Sg[i] : 0.f;
            A[i] = ok ? Ag[i] : 0.f;
        }
    }
    const float xv = live ? to_f32(x[(size_t)t * x_stride + c]) : 0.f;
    const float zv = live ? to_f32(z[(size_t)t * z_stride + c]) : 0.f;
    const float dv = live ? dt_raw[(size_t)t * dt_stride + c] + (dt_bias ? dt_bias[c] : 0.f) : 0.f;
    const float dt = cs_softplus<T>(dv), dx = dt * xv;
    float p = 0.f, p2 = 0.f;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        const bool in = n0 + i < N;
        const float bv = in ? to_f32(bm[(size_t)t * bc_stride + n0 + i]) : 0.f;
        const float cv = in ? to_f32(cm[(size_t)t * bc_stride + n0 + i]) : 0.f;
        S[i] = cs_step<T>(S[i], dt * A[i], dx * bv);
        if (i & 1) p2 = fmaf(S[i], cv, p2); else p = fmaf(S[i], cv, p);
    }
    if (VEC) {
#pragma unroll
        for (int i = 0; i < NS; i += 4)
            if (live && n0 + i < N) *(float4*)(Sg + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (live && n0 + i < N) Sg[i] = S[i];
    }
    float sum = p + p2;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane_l || !live) return;
    const float skip = D ? D[c] : 0.f;
    y[(size_t)t * C + c] = from_f32<T>(fmaf(skip, xv, sum) * cs_silu<T>(zv));
    if (conv_in) cs_keep(row + conv_offset, conv_in, conv_in_stride, c, C, taps, t, 1);
}

template <typename T, int L, int NS>
static int launch_channel_scan(const void* x, long long x_stride, const void* z, long long z_stride,
                               const float* dt_raw, long long dt_stride, const float* dt_bias, const float* a2,
                               const void* bm, const void* cm, long long bc_stride, const float* D, void* y, int Tn,
                               int B, int C, int N, const int* q_start, const int* state_slots, float* state,
                               long long state_stride, long long ssm_offset, const void* conv_in,
                               long long conv_in_stride, int taps, long long conv_offset, cudaStream_t stream) {
    constexpr int CH = CS_WALK / L, NP = L * NS;
#define CS_LAUNCH(KERNEL, GRID, BLOCK, SMEM)                                                                  \
    tgo_launch_pdl(KERNEL, GRID, dim3(BLOCK), SMEM, stream, (const T*)x, x_stride, (const T*)z, z_stride,     \
                   dt_raw, dt_stride, dt_bias, a2, (const T*)bm, (const T*)cm, bc_stride, D, (T*)y, C, N, q_start, \
                   state_slots, state, state_stride, ssm_offset, (const T*)conv_in, conv_in_stride, taps, conv_offset)
    if (Tn == B) {                                       // every request brings one token
        const dim3 grid(B, (C + 128 / L - 1) / (128 / L));
        const bool vec = N % 4 == 0 && state_stride % 4 == 0 && ssm_offset % 4 == 0 && (uintptr_t)state % 16 == 0 &&
                         (uintptr_t)a2 % 16 == 0;
        if (vec) return CS_LAUNCH((channel_scan_single_kernel<T, L, NS, true>), grid, 128, 0);
        return CS_LAUNCH((channel_scan_single_kernel<T, L, NS, false>), grid, 128, 0);
    }
    constexpr int TOK = NP <= 32 ? 64 : 32;              // tokens a tile: what shared memory has room for
    const size_t smem = (size_t)2 * TOK * (2 * NP + 3 * (CH + 1)) * sizeof(float);
    auto kernel = channel_scan_kernel<T, L, NS, TOK>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return CS_LAUNCH(kernel, dim3(B, (C + CH - 1) / CH), CS_WALK + CS_SERVE(TOK, L), smem);
#undef CS_LAUNCH
}

// x, z column views [T, C], bm, cm column views [T, N] (row stride bc_stride) and conv_in a
// column view [T, C] (null: no kept inputs to move on), all in the storage type; dt_raw float32
// [T, C] (strided); a2 float32 [C, N]; y [T, C] in the storage type. A request's state [C][N] lies
// at `ssm_offset` of its state row, its kept inputs [taps - 1][C] at `conv_offset`.
TGO_API int tgo_channel_scan(const void* x, long long x_stride, const void* z, long long z_stride, int dtype,
                             const float* dt_raw, long long dt_stride, const float* dt_bias, const float* a2,
                             const void* bm, const void* cm, long long bc_stride, const float* D, void* y, int T,
                             int B, int C, int N, const int* q_start, const int* state_slots, float* state,
                             long long state_stride, long long ssm_offset, const void* conv_in,
                             long long conv_in_stride, int taps, long long conv_offset, cudaStream_t stream) {
    if (B <= 0 || T <= 0) return 0;
    if (C <= 0 || N <= 0 || N > 256 || T < B || (dtype != TGO_BF16 && dtype != TGO_F32) ||
        state_stride < ssm_offset + (long long)C * N || (C + 3) / 4 > 65535 ||
        (conv_in && (taps < 1 || state_stride < conv_offset + (long long)(taps - 1) * C)))
        return TGO_E_BAD_ARG;
#define CS_GO(L, NS)                                                                                          \
    (dtype == TGO_BF16                                                                                        \
         ? launch_channel_scan<bf16, L, NS>(x, x_stride, z, z_stride, dt_raw, dt_stride, dt_bias, a2, bm, cm,  \
                                            bc_stride, D, y, T, B, C, N, q_start, state_slots, state, state_stride, \
                                            ssm_offset, conv_in, conv_in_stride, taps, conv_offset, stream)   \
         : launch_channel_scan<float, L, NS>(x, x_stride, z, z_stride, dt_raw, dt_stride, dt_bias, a2, bm, cm, \
                                             bc_stride, D, y, T, B, C, N, q_start, state_slots, state, state_stride, \
                                             ssm_offset, conv_in, conv_in_stride, taps, conv_offset, stream))
    if (N <= 16) return CS_GO(4, 4);
    if (N <= 32) return CS_GO(4, 8);
    if (N <= 64) return CS_GO(8, 8);
    if (N <= 128) return CS_GO(16, 8);
    return CS_GO(32, 8);
#undef CS_GO
}
