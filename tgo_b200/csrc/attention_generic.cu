// Paged causal attention, one warp per (token, head), any head size up to 256 (rows whose
// values lie inside the keys: up to 1152) and any
// storage type. It is the float32 path's attention and the fallback of the bfloat16
// path for head sizes that the tensor-core kernels do not take.
//
// The query at position p of request b reads keys lo..p, lo = max(0, p - window + 1)
// (window 0: lo = 0), through the request's block table. Keys are taken 32 at a time
// starting at lo, so the order of every sum depends on (p, window) alone: the result
// for a position is bit-identical however the tokens were cut into steps or batched.
//
// Keys are dh wide and values dv wide (two cache planes with rows of their own when they
// differ). With `sinks` (float32, one number per query head) the softmax's denominator also
// holds exp(sink_h): a key that is always seen, is not scaled and has no value.
// `softcap` > 0 bounds every score: s <- softcap * tanh(s / softcap), after the scale.
// A value row starts `v_row` elements after the one before it: dv for a plane of values; the
// key rows' width when a value is the first dv channels of its key row (one cache plane that
// serves as both, v_cache = k_cache).
// `keep_first` > 0 (with a window): the first keep_first keys of the request stay visible to
// every later query, at their true positions, beside the window. The keys are then walked as
// one list (the kept ones that lie before the window, then the window), 32 at a time, so the
// order of the sums still depends on (p, window, keep_first) alone.
// `dist_bias` (float32 [n_dist][H]): dist_bias[min(p - j, n_dist - 1)][h] is added to the
// scaled score of key j, unscaled (a learned bias by distance).
// `gate` ([T, >= H] in the storage type, rows gate_stride apart): the output of head h at token t
// is multiplied by the logistic function of gate[t][h].
#include "common.cuh"

#define AG_MAX_DH 256            // rows up to this wide take the instance with 8 sums a lane
#define AG_MAX_WIDE 640          // wider ones, up to this, the instance with 20
#define AG_MAX_WIDEST 1152       // and up to this (a latent of 1024 with its rotated part), 36
#define AG_WARPS 4

template <typename T, int NACC>
__global__ void attention_generic_kernel(
    const T* __restrict__ q, long long q_stride, T* __restrict__ out, long long out_stride,
    int H, int Hkv, int dh, int dv, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
    int page_size, const int* __restrict__ block_tables, int max_blocks,
    const int* __restrict__ seq_ids, const int* __restrict__ positions, float scale, int window,
    const float* __restrict__ sinks, float softcap, int v_row, int keep_first,
    const float* __restrict__ dist_bias, int n_dist, const T* __restrict__ gate, long long gate_stride) {
    extern __shared__ float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int h = blockIdx.y * AG_WARPS + warp;
    if (h >= H) return;
    float* qs = smem + warp * dh;
    const int p = positions[t];
    const int b = p >= 0 ? seq_ids[t] : 0;
    const int kvh = h / (H / Hkv);
    const int* bt = block_tables + (size_t)b * max_blocks;
    const T* qv = q + (size_t)t * q_stride + (size_t)h * dh;
    for (int i = lane; i < dh; i += 32) qs[i] = to_f32(qv[i]);
    __syncwarp();

    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    float m = -INFINITY, l = 0.f;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;

    const int nkept = keep_first < lo ? keep_first : lo;       // kept keys that lie before the window
    const int nkeys = p >= 0 ? nkept + (p - lo + 1) : 0;
    for (int vbase = 0; vbase < nkeys; vbase += 32) {
        const int vj = vbase + lane;
        const int j = vj < nkept ? vj : lo + (vj - nkept);
        const int nvalid = (nkeys - vbase) < 32 ? (nkeys - vbase) : 32;
        float s = -INFINITY;
        if (vj < nkeys) {
            const int page = bt[j / page_size];
            const T* kr = k_cache + (((size_t)page * Hkv + kvh) * page_size + (j % page_size)) * dh;
            float a = 0.f;
            for (int d = 0; d < dh; ++d) a += qs[d] * to_f32(kr[d]);
            s = a * scale;
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            if (dist_bias) s += dist_bias[(size_t)((p - j) < n_dist ? (p - j) : n_dist - 1) * H + h];
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);          // m = -inf the first time: corr = 0
        const float w = vj < nkeys ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(w);
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] *= corr;
        for (int jj = 0; jj < nvalid; ++jj) {
            const float wj = __shfl_sync(0xffffffffu, w, jj);
            const int kj = (vbase + jj) < nkept ? vbase + jj : lo + (vbase + jj - nkept);
            const int page = bt[kj / page_size];
            const T* vr = v_cache + (((size_t)page * Hkv + kvh) * page_size + (kj % page_size)) * v_row;
#pragma unroll
            for (int i = 0; i < NACC; ++i) {
                const int d = lane + 32 * i;
                if (d < dv) acc[i] += wj * to_f32(vr[d]);
            }
        }
        m = m_new;
    }
    if (sinks && p >= 0) {                         // the sink joins the denominator last
        const float sk = sinks[h];
        const float m_new = fmaxf(m, sk);
        const float corr = expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] *= corr;
    }
    T* o = out + (size_t)t * out_stride + (size_t)h * dv;
    float inv = l > 0.f ? 1.f / l : 0.f;           // position < 0: no keys, zeros out
    if (gate) inv *= 1.f / (1.f + expf(-to_f32(gate[(size_t)t * gate_stride + h])));
#pragma unroll
    for (int i = 0; i < NACC; ++i) {
        const int d = lane + 32 * i;
        if (d < dv) o[d] = from_f32<T>(acc[i] * inv);
    }
}

// ------------------------------------------------------------- prompt portions, every earlier key
// The same sums in the same order, for steps that bring several tokens a request and see every
// earlier key (window 0: the keys are then cut into the same 32 for every query). A block takes
// AGT_Q query rows (the heads of one kv head x consecutive tokens of one request) and brings each 32
// keys and values into shared memory once for all of them, float32 ones by asynchronous copies one tile ahead; a
// warp owns AGT_R rows, a lane one key for the scores and 4 NV channels for the sums. Tiles whose every key all
// of a warp's rows see go side by side through the softmax and without a test a key. Bound by reads of shared memory
// (a 16-byte read of a key row feeds 4 AGT_R FMA). The first `n_blocks` blocks of a kv head take the first run of tokens of one
// request among their AGT_Q / G tokens; where requests meet inside those, the runs that begin there go
// to the blocks behind them, so that no request waits for another's keys.
// The caller picks this kernel from four tokens a request on (bits do not depend on it): MEASURED
// (B200, 301 + 256 tokens of 16/4 heads of 128, float32): a warp a query 772 us, this 75 (139 with each tile waited
// for, each row's sums by themselves and the weights by shuffles); 64 tokens beside
// fifteen single ones of 1000 keys, 16/4 heads of 128: 946 and 93 us (302; 1258 when a block walked the requests
// that meet in it in turn), 8/8 heads of 64: 556 and 101 (178; 2691). 32 rows a block and not 16: fewer blocks take a short
// prompt, but keys come half as often (and groups of up to 32 heads fit): 20 calls in a row, with the 16 rows of the form before in
// brackets, 20 tokens of 16/4 heads of 128 16.6 us (18.6), 33 of 8/8 of 64 18.6 (16.5), 128 29 (49) and 27 (35), 64 after 1000
// 146 (329) and 115 (222); 32/1 heads of 64, a warp a query before: 4 tokens 10.4 (8.3), 8 10.9 (10.4), 20 12.4 (18).
#define AGT_WARPS 8
#define AGT_R 4
#define AGT_Q (AGT_WARPS * AGT_R)
#define AGT_MAX_SMEM ((int)((2 * (32 * (AG_MAX_DH + 4) + 32 * AG_MAX_DH) + AGT_Q * (AG_MAX_DH + 32)) * sizeof(float)))

__device__ __forceinline__ float4 ag_load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 ag_load4(const bf16* p) {
    const uint2 v = *(const uint2*)p;
    const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&v.x), b = __bfloat1622float2(*(const __nv_bfloat162*)&v.y);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Four numbers of a row of the cache to shared memory as float32; zeros where !ok. float32 rows on their way when it returns.
__device__ __forceinline__ void agt_copy4(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void agt_copy4(float* dst, const bf16* src, bool ok) {
    *(float4*)dst = ok ? ag_load4(src) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// The request of a token, -1 for one that brings nothing.
__device__ __forceinline__ int agt_request(const int* __restrict__ positions, const int* __restrict__ seq_ids, int t) {
    return positions[t] >= 0 ? seq_ids[t] : -1;
}

// The token where the k-th run begins that does not begin with a block's tokens, or -1. The whole block calls.
__device__ __forceinline__ int agt_run(int k, int nt, int Tn, const int* __restrict__ positions, const int* __restrict__ seq_ids) {
    __shared__ int s_before[AGT_WARPS], s_at;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int base = 0, seen = 0; base < Tn; base += 32 * AGT_WARPS) {
        const int t = base + threadIdx.x;
        const bool begins = t < Tn && t % nt && agt_request(positions, seq_ids, t) != agt_request(positions, seq_ids, t - 1);
        const unsigned ballot = __ballot_sync(0xffffffffu, begins);
        if (lane == 0) s_before[warp] = __popc(ballot);
        const int n = __syncthreads_count(begins);
        if (k < seen + n) {
            int rank = seen + __popc(ballot & ((1u << lane) - 1u));
            for (int w = 0; w < warp; ++w) rank += s_before[w];
            if (begins && rank == k) s_at = t;
            __syncthreads();
            return s_at;
        }
        seen += n;
        __syncthreads();                                 // s_before is written again
    }
    return -1;
}

template <typename T, int NV>
__global__ void __launch_bounds__(32 * AGT_WARPS, NV == 1 ? 2 : 1)
attention_generic_tiles_kernel(const T* __restrict__ q, long long q_stride, T* __restrict__ out, long long out_stride,
                               int Tn, int n_blocks, int H, int Hkv, int dh, int dv, const T* __restrict__ k_cache,
                               const T* __restrict__ v_cache, int page_size, const int* __restrict__ block_tables,
                               int max_blocks, const int* __restrict__ seq_ids, const int* __restrict__ positions,
                               float scale, const float* __restrict__ sinks, float softcap, int v_row,
                               const float* __restrict__ dist_bias, int n_dist, const T* __restrict__ gate,
                               long long gate_stride) {
    extern __shared__ __align__(16) float agt_smem[];
    const int ldk = dh + 4;                              // 16-byte reads of 8 rows hit 8 different places
    const int buf_floats = 32 * (ldk + dv);              // keys [32][ldk], then values [32][dv]; two of them
    float* qs = agt_smem + 2 * buf_floats;               // [AGT_Q][dh]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* ws = qs + AGT_Q * dh + warp * AGT_R * 32;     // the warp's weights [AGT_R][32]
    const int G = H / Hkv, kvh = blockIdx.y;
    const int nt = AGT_Q / G;                            // tokens of a block (G <= AGT_Q)
    for (int run = blockIdx.x;; run += gridDim.x - n_blocks) {       // a first run, or the others a block has to take
        const int t0 = run < n_blocks ? run * nt : agt_run(run - n_blocks, nt, Tn, positions, seq_ids);
        if (t0 < 0) return;
        const int b = agt_request(positions, seq_ids, t0);
        int t_end = t0 + 1, p_last = positions[t0];
        for (; t_end % nt && t_end < Tn && agt_request(positions, seq_ids, t_end) == b; ++t_end) p_last = max(p_last, positions[t_end]);
        const int nq = (t_end - t0) * G;
        for (int i = threadIdx.x; i < AGT_Q * dh; i += blockDim.x) {
            const int r = i / dh;
            qs[i] = r < nq ? to_f32(q[(size_t)(t0 + r / G) * q_stride + (size_t)(kvh * G + r % G) * dh + i % dh]) : 0.f;
        }
        float m[AGT_R], l[AGT_R];
        float4 acc[AGT_R][NV];
        int tok[AGT_R], pos[AGT_R];
#pragma unroll
        for (int r = 0; r < AGT_R; ++r) {
            const int row = warp * AGT_R + r;
            m[r] = -INFINITY;
            l[r] = 0.f;
            tok[r] = row < nq ? t0 + row / G : t_end;
            pos[r] = tok[r] < t_end ? positions[tok[r]] : -1;
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[r][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const int* bt = block_tables + (size_t)(b < 0 ? 0 : b) * max_blocks;
        int pos_min = pos[0];
#pragma unroll
        for (int r = 1; r < AGT_R; ++r) pos_min = min(pos_min, pos[r]);
        // AGT_WARPS threads a key: its place is looked up once
        auto load = [&](int k0, int buf) {
            if (k0 <= p_last) {
                const int r = threadIdx.x / AGT_WARPS, j = k0 + r, c0 = (threadIdx.x % AGT_WARPS) * 4;
                const bool ok = j <= p_last;
                const size_t row = ok ? ((size_t)bt[j / page_size] * Hkv + kvh) * page_size + j % page_size : 0;
                const T *kr = k_cache + row * dh, *vr = v_cache + row * v_row;
                float *kd = agt_smem + buf * buf_floats + r * ldk, *vd = agt_smem + buf * buf_floats + 32 * ldk + r * dv;
                for (int c = c0; c < dh; c += 4 * AGT_WARPS) agt_copy4(kd + c, kr + c, ok);
                for (int c = c0; c < dv; c += 4 * AGT_WARPS) agt_copy4(vd + c, vr + c, ok);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        __syncthreads();                                 // the last run's keys have been read
        load(0, 0);
        for (int k0 = 0, buf = 0; k0 <= p_last; k0 += 32, buf ^= 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();                             // this tile is there, the last one has been read
            load(k0 + 32, buf ^ 1);
            const float* ks = agt_smem + buf * buf_floats;
            const float* vs = ks + 32 * ldk;
            if (warp * AGT_R >= nq) continue;            // none of the run's rows are this warp's
            float a[AGT_R], w[AGT_R];
#pragma unroll
            for (int r = 0; r < AGT_R; ++r) a[r] = 0.f;
#pragma unroll 4
            for (int d = 0; d < dh; d += 4) {
                const float4 k4 = *(const float4*)(ks + lane * ldk + d);
#pragma unroll
                for (int r = 0; r < AGT_R; ++r) {
                    const float4 q4 = *(const float4*)(qs + (warp * AGT_R + r) * dh + d);
                    a[r] = fmaf(q4.x, k4.x, a[r]);
                    a[r] = fmaf(q4.y, k4.y, a[r]);
                    a[r] = fmaf(q4.z, k4.z, a[r]);
                    a[r] = fmaf(q4.w, k4.w, a[r]);
                }
            }
            if (k0 + 31 <= pos_min) {                    // every row sees every key
                float m_new[AGT_R], sum[AGT_R];
#pragma unroll
                for (int r = 0; r < AGT_R; ++r) {
                    const int p = pos[r], j = k0 + lane;
                    float s = a[r] * scale;
                    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
                    if (dist_bias) s += dist_bias[(size_t)((p - j) < n_dist ? (p - j) : n_dist - 1) * H + kvh * G + (warp * AGT_R + r) % G];
                    a[r] = m_new[r] = s;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < AGT_R; ++r) m_new[r] = fmaxf(m_new[r], __shfl_xor_sync(0xffffffffu, m_new[r], o));
#pragma unroll
                for (int r = 0; r < AGT_R; ++r) {
                    m_new[r] = fmaxf(m[r], m_new[r]);
                    sum[r] = w[r] = expf(a[r] - m_new[r]);
                    ws[r * 32 + lane] = w[r];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < AGT_R; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
#pragma unroll
                for (int r = 0; r < AGT_R; ++r) {
                    const float corr = expf(m[r] - m_new[r]);
                    l[r] = l[r] * corr + sum[r];
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        acc[r][i].x *= corr; acc[r][i].y *= corr; acc[r][i].z *= corr; acc[r][i].w *= corr;
                    }
                    m[r] = m_new[r];
                }
                __syncwarp();
#pragma unroll 2
                for (int j0 = 0; j0 < 32; j0 += 4) {
                    float4 w4[AGT_R];
#pragma unroll
                    for (int r = 0; r < AGT_R; ++r) w4[r] = *(const float4*)(ws + r * 32 + j0);
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                        for (int i = 0; i < NV; ++i) {
                            const float4 v4 = (lane + 32 * i) * 4 < dv ? *(const float4*)(vs + (j0 + jj) * dv + (lane + 32 * i) * 4)
                                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int r = 0; r < AGT_R; ++r) {
                                const float wj = jj == 0 ? w4[r].x : jj == 1 ? w4[r].y : jj == 2 ? w4[r].z : w4[r].w;
                                acc[r][i].x = fmaf(wj, v4.x, acc[r][i].x);
                                acc[r][i].y = fmaf(wj, v4.y, acc[r][i].y);
                                acc[r][i].z = fmaf(wj, v4.z, acc[r][i].z);
                                acc[r][i].w = fmaf(wj, v4.w, acc[r][i].w);
                            }
                        }
                }
                __syncwarp();                            // the weights have been read
                continue;
            }
            int most = 0;
#pragma unroll
            for (int r = 0; r < AGT_R; ++r) {
                const int p = pos[r], j = k0 + lane;
                w[r] = 0.f;
                if (k0 > p) continue;                    // the same for the whole warp
                float s = -INFINITY;
                if (j <= p) {
                    s = a[r] * scale;
                    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
                    if (dist_bias) s += dist_bias[(size_t)((p - j) < n_dist ? (p - j) : n_dist - 1) * H + kvh * G + (warp * AGT_R + r) % G];
                }
                const float m_new = fmaxf(m[r], warp_max(s));
                const float corr = expf(m[r] - m_new);
                w[r] = j <= p ? expf(s - m_new) : 0.f;
                l[r] = l[r] * corr + warp_sum(w[r]);
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    acc[r][i].x *= corr; acc[r][i].y *= corr; acc[r][i].z *= corr; acc[r][i].w *= corr;
                }
                m[r] = m_new;
                const int n = p - k0 + 1 < 32 ? p - k0 + 1 : 32;
                most = n > most ? n : most;
            }
            for (int jj = 0; jj < most; ++jj) {
                float4 v4[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    v4[i] = (lane + 32 * i) * 4 < dv ? *(const float4*)(vs + jj * dv + (lane + 32 * i) * 4)
                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int r = 0; r < AGT_R; ++r) {
                    const float wj = __shfl_sync(0xffffffffu, w[r], jj);
                    if (k0 + jj > pos[r]) continue;      // past this row's keys: nothing is added, not even 0 x NaN
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        acc[r][i].x = fmaf(wj, v4[i].x, acc[r][i].x);
                        acc[r][i].y = fmaf(wj, v4[i].y, acc[r][i].y);
                        acc[r][i].z = fmaf(wj, v4[i].z, acc[r][i].z);
                        acc[r][i].w = fmaf(wj, v4[i].w, acc[r][i].w);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < AGT_R; ++r) {
            if (tok[r] >= t_end) continue;
            const int h = kvh * G + (warp * AGT_R + r) % G;
            if (sinks && pos[r] >= 0) {                  // the sink joins the denominator last
                const float sk = sinks[h];
                const float m_new = fmaxf(m[r], sk);
                const float corr = expf(m[r] - m_new);
                l[r] = l[r] * corr + expf(sk - m_new);
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    acc[r][i].x *= corr; acc[r][i].y *= corr; acc[r][i].z *= corr; acc[r][i].w *= corr;
                }
            }
            float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
            if (gate) inv *= 1.f / (1.f + expf(-to_f32(gate[(size_t)tok[r] * gate_stride + h])));
            T* o = out + (size_t)tok[r] * out_stride + (size_t)h * dv;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int d = (lane + 32 * i) * 4;
                if (d >= dv) continue;
                o[d] = from_f32<T>(acc[r][i].x * inv);
                o[d + 1] = from_f32<T>(acc[r][i].y * inv);
                o[d + 2] = from_f32<T>(acc[r][i].z * inv);
                o[d + 3] = from_f32<T>(acc[r][i].w * inv);
            }
        }
        if (run < n_blocks) return;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                 // the run's queries, keys and values have been read
    }
}

// 1 if the tiled kernel takes the step: heads of a group within a block's rows, widths of whole
// 16-byte (8-byte in bfloat16) pieces up to 256.
TGO_API int tgo_attention_generic_tiles_takes(int H, int Hkv, int dh, int dv, int v_row) {
    return Hkv > 0 && H % Hkv == 0 && H / Hkv <= AGT_Q && dh > 0 && dh <= AG_MAX_DH && dh % 4 == 0 && dv > 0 &&
           dv <= AG_MAX_DH && dv % 4 == 0 && v_row >= dv && v_row % 4 == 0;
}

TGO_API int tgo_attention_generic_tiles(const void* q, long long q_stride, void* out, long long out_stride, int dtype,
                                        int T, int H, int Hkv, int dh, int dv, const void* k_cache,
                                        const void* v_cache, int page_size, const int* block_tables, int n_seqs,
                                        int max_blocks, const int* seq_ids, const int* positions, float scale,
                                        const float* sinks, float softcap, int v_row, const float* dist_bias, int n_dist,
                                        const void* gate, long long gate_stride, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (v_row <= 0) v_row = dv;
    if (!tgo_attention_generic_tiles_takes(H, Hkv, dh, dv, v_row) || Hkv > 65535 || page_size <= 0 || n_seqs <= 0 ||
        max_blocks <= 0 || !(softcap >= 0.f) || (dist_bias && n_dist <= 0) || ((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15) ||
        (dtype != TGO_BF16 && dtype != TGO_F32))
        return TGO_E_BAD_ARG;
    // a block for the first run of every nt tokens, and as many as there are requests for the others
    const int nt = AGT_Q / (H / Hkv), n_blocks = (T + nt - 1) / nt;
    const dim3 grid(n_blocks + (n_seqs < T ? n_seqs : T), Hkv);
    const size_t smem = (size_t)(2 * 32 * (dh + 4 + dv) + AGT_Q * (dh + 32)) * sizeof(float);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
#define AGT_GO(TT, NV)                                                                                         \
    do {                                                                                                        \
        static int sized[64] = {};                       /* per device: the shared memory asked for there */    \
        if (sized[dev] < (int)smem) {                                                                           \
            e = cudaFuncSetAttribute(attention_generic_tiles_kernel<TT, NV>,                                    \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, AGT_MAX_SMEM);                \
            if (e != cudaSuccess) return (int)e;                                                                \
            sized[dev] = AGT_MAX_SMEM;                                                                          \
        }                                                                                                       \
        attention_generic_tiles_kernel<TT, NV><<<grid, 32 * AGT_WARPS, smem, stream>>>(                         \
            (const TT*)q, q_stride, (TT*)out, out_stride, T, n_blocks, H, Hkv, dh, dv, (const TT*)k_cache,      \
            (const TT*)v_cache, page_size, block_tables, max_blocks, seq_ids, positions, scale, sinks, softcap, \
            v_row, dist_bias, n_dist, (const TT*)gate, gate_stride);                                            \
    } while (0)
    if (dtype == TGO_BF16) { if (dv > 128) AGT_GO(bf16, 2); else AGT_GO(bf16, 1); }
    else { if (dv > 128) AGT_GO(float, 2); else AGT_GO(float, 1); }
#undef AGT_GO
    return launch_status();
}

TGO_API int tgo_attention_generic(const void* q, long long q_stride, void* out,
                                  long long out_stride, int dtype, int T, int H, int Hkv, int dh, int dv,
                                  const void* k_cache, const void* v_cache, int page_size,
                                  const int* block_tables, int max_blocks, const int* seq_ids,
                                  const int* positions, float scale, int window,
                                  const float* sinks, float softcap, int v_row, int keep_first,
                                  const float* dist_bias, int n_dist, const void* gate, long long gate_stride,
                                  cudaStream_t stream) {
    if (T <= 0) return 0;
    if (v_row <= 0) v_row = dv;
    if (dh <= 0 || dh > AG_MAX_WIDEST || dv <= 0 || dv > AG_MAX_WIDEST || H <= 0 || Hkv <= 0 || H % Hkv ||
        page_size <= 0 || max_blocks <= 0 || window < 0 || v_row < dv || !(softcap >= 0.f) || keep_first < 0 ||
        (dist_bias && n_dist <= 0))
        return TGO_E_BAD_ARG;
    const bool wide = dv > AG_MAX_DH, widest = dv > AG_MAX_WIDE;
    const dim3 grid(T, (H + AG_WARPS - 1) / AG_WARPS);
    const size_t smem = (size_t)AG_WARPS * dh * sizeof(float);
#define AG_GO(TT, NACC)                                                                            \
    attention_generic_kernel<TT, NACC><<<grid, AG_WARPS * 32, smem, stream>>>(                         \
        (const TT*)q, q_stride, (TT*)out, out_stride, H, Hkv, dh, dv, (const TT*)k_cache,              \
        (const TT*)v_cache, page_size, block_tables, max_blocks, seq_ids, positions, scale, window,   \
        sinks, softcap, v_row, keep_first, dist_bias, n_dist, (const TT*)gate, gate_stride)
    if (dtype == TGO_BF16) {
        if (widest) AG_GO(bf16, AG_MAX_WIDEST / 32); else if (wide) AG_GO(bf16, AG_MAX_WIDE / 32); else AG_GO(bf16, AG_MAX_DH / 32);
    } else if (dtype == TGO_F32) {
        if (widest) AG_GO(float, AG_MAX_WIDEST / 32); else if (wide) AG_GO(float, AG_MAX_WIDE / 32); else AG_GO(float, AG_MAX_DH / 32);
    } else
        return TGO_E_BAD_ARG;
#undef AG_GO
    return launch_status();
}
