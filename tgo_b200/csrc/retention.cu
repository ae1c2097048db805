// Retention: linear attention with one fixed decay per head, no softmax and no denominator.
// Per request and head a float32 state S [dk][dv] is carried from token to token:
//
//   S_t = decay * S_(t-1) + k_t v_t^T,      o_t = S_t^T q_t
//
// q and k are rotated (half-split pairs, from the step's cos/sin table) as they are loaded,
// and k is then multiplied by k_scale; all of it in float32, whatever the storage type of the
// projections. A step's tokens of one request are taken in chunks of up to RT_CHUNK tokens:
// inside a chunk (local index i, j; n tokens)
//
//   o_i = sum_{j<=i} decay^(i-j) (q_i . k_j) v_j  +  decay^(i+1) S^T q_i
//   S  <- decay^n S + sum_j decay^(n-1-j) k_j v_j^T
//
// which is the recurrence written out; a single token (a decode step) is a chunk of one.
// The columns of S are independent, so a block owns a slice of dv columns of one
// (request, head): grid (requests, heads, slices). The powers of the decay come from a table
// made by repeated multiplication.
#include "split3.cuh"

#define RT_CHUNK 32
#define RT_THREADS 256

// What q, k and v go through as they are read (a parameter of every kernel here):
// 0 nothing, 1 SiLU, in float32.
template <typename T>
__device__ __forceinline__ float taken(T x, int act) {
    const float f = to_f32(x);
    return act == 1 ? f / (1.f + expf(-f)) : f;
}

template <typename T>
__device__ __forceinline__ float rotated(const T* __restrict__ x, const float* __restrict__ cs,
                                         int i, int rot, int act) {
    const int half = rot >> 1;
    if (i < half) return taken(x[i], act) * cs[i] - taken(x[i + half], act) * cs[half + i];
    if (i < rot) return taken(x[i], act) * cs[i - half] + taken(x[i - half], act) * cs[i];
    return taken(x[i], act);
}

template <typename T>
__global__ void __launch_bounds__(RT_THREADS)
retention_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ k,
                 long long k_stride, const T* __restrict__ v, long long v_stride,
                 float* __restrict__ out, int H, int dk, int dv, int vs,
                 const float* __restrict__ decay, float k_scale, int act, const float* __restrict__ rope,
                 int rot, const int* __restrict__ q_start, const int* __restrict__ state_slots,
                 float* __restrict__ state) {
    extern __shared__ float smem[];
    const int dkp = dk + 1;
    float* Qs = smem;                               // [RT_CHUNK][dk + 1]
    float* Ks = Qs + RT_CHUNK * dkp;                // [RT_CHUNK][dk + 1]
    float* Vs = Ks + RT_CHUNK * dkp;                // [RT_CHUNK][vs]
    float* As = Vs + RT_CHUNK * vs;                 // [RT_CHUNK][RT_CHUNK + 1]
    float* Ss = As + RT_CHUNK * (RT_CHUNK + 1);     // [dk][vs]
    float* pw = Ss + (size_t)dk * vs;               // [RT_CHUNK + 1]
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y;
    const int c0 = blockIdx.z * vs;
    const int nc = (dv - c0) < vs ? (dv - c0) : vs;
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 <= t0) return;
    const float g = decay[h];
    float* Sg = state + (((size_t)state_slots[b] * H + h) * dk) * dv + c0;
    for (int i = threadIdx.x; i < dk * vs; i += RT_THREADS) {
        const int d = i / vs, c = i % vs;
        Ss[i] = c < nc ? Sg[(size_t)d * dv + c] : 0.f;
    }
    if (threadIdx.x == 0) {
        float x = 1.f;
        for (int i = 0; i <= RT_CHUNK; ++i) {
            pw[i] = x;
            x *= g;
        }
    }
    for (int ts = t0; ts < t1; ts += RT_CHUNK) {
        const int n = (t1 - ts) < RT_CHUNK ? (t1 - ts) : RT_CHUNK;
        __syncthreads();
        for (int i = threadIdx.x; i < n * dk; i += RT_THREADS) {
            const int r = i / dk, d = i % dk;
            const size_t t = (size_t)(ts + r);
            const float* cs = rope ? rope + t * rot : nullptr;
            const T* qr = q + t * q_stride + (size_t)h * dk;
            const T* kr = k + t * k_stride + (size_t)h * dk;
            Qs[r * dkp + d] = cs ? rotated(qr, cs, d, rot, act) : taken(qr[d], act);
            Ks[r * dkp + d] = (cs ? rotated(kr, cs, d, rot, act) : taken(kr[d], act)) * k_scale;
        }
        for (int i = threadIdx.x; i < n * vs; i += RT_THREADS) {
            const int r = i / vs, c = i % vs;
            Vs[i] = c < nc ? taken(v[(size_t)(ts + r) * v_stride + (size_t)h * dv + c0 + c], act) : 0.f;
        }
        __syncthreads();
        // A[i][j] = decay^(i-j) q_i . k_j for j <= i
        for (int idx = threadIdx.x; idx < n * n; idx += RT_THREADS) {
            const int i = idx / n, j = idx % n;
            float a = 0.f;
            if (j <= i) {
                const float* qi = Qs + i * dkp;
                const float* kj = Ks + j * dkp;
                for (int d = 0; d < dk; ++d) a += qi[d] * kj[d];
                a *= pw[i - j];
            }
            As[i * (RT_CHUNK + 1) + j] = a;
        }
        __syncthreads();
        // o_i[c] = sum_j A[i][j] v_j[c] + decay^(i+1) sum_d q_i[d] S[d][c]
        for (int idx = threadIdx.x; idx < n * vs; idx += RT_THREADS) {
            const int i = idx / vs, c = idx % vs;
            if (c >= nc) continue;
            const float* qi = Qs + i * dkp;
            float far = 0.f;
            for (int d = 0; d < dk; ++d) far += qi[d] * Ss[d * vs + c];
            float near = 0.f;
            const float* ai = As + i * (RT_CHUNK + 1);
            for (int j = 0; j <= i; ++j) near += ai[j] * Vs[j * vs + c];
            out[((size_t)(ts + i) * H + h) * dv + c0 + c] = near + pw[i + 1] * far;
        }
        __syncthreads();
        // S[d][c] = decay^n S[d][c] + sum_j decay^(n-1-j) k_j[d] v_j[c]
        for (int idx = threadIdx.x; idx < dk * vs; idx += RT_THREADS) {
            const int d = idx / vs, c = idx % vs;
            float a = 0.f;
            for (int j = 0; j < n; ++j) a += pw[n - 1 - j] * Ks[j * dkp + d] * Vs[j * vs + c];
            Ss[idx] = pw[n] * Ss[idx] + a;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < dk * vs; i += RT_THREADS) {
        const int d = i / vs, c = i % vs;
        if (c < nc) Sg[(size_t)d * dv + c] = Ss[i];
    }
}

static inline size_t retention_smem(int dk, int vs) {
    return ((size_t)2 * RT_CHUNK * (dk + 1) + (size_t)RT_CHUNK * vs + (size_t)RT_CHUNK * (RT_CHUNK + 1) +
            (size_t)dk * vs + RT_CHUNK + 1) * sizeof(float);
}

// q, k: [T, >= H*dk] rows (strided), v: [T, >= H*dv]; out float32 [T, H*dv]; state float32
// [slots, H, dk, dv]; decay float32 [H] on the device; rope [T, rot] (cos then sin) or null.
TGO_API int tgo_retention(const void* q, long long q_stride, const void* k, long long k_stride,
                          const void* v, long long v_stride, int dtype, float* out, int B, int H,
                          int dk, int dv, const float* decay, float k_scale, int act, const float* rope,
                          int rot, const int* q_start, const int* state_slots, float* state,
                          cudaStream_t stream) {
    if (B <= 0) return 0;
    if (H <= 0 || dk <= 0 || dv <= 0 || rot < 0 || rot > dk || (rot & 1) || H > 65535)
        return TGO_E_BAD_ARG;
    int vs = 32;                                    // columns of the state a block owns
    while (vs > 8 && retention_smem(dk, vs) > 200 * 1024) vs >>= 1;
    const size_t smem = retention_smem(dk, vs);
    if (smem > 200 * 1024) return TGO_E_BAD_ARG;
    const dim3 grid(B, H, (dv + vs - 1) / vs), block(RT_THREADS);
    if (grid.z > 65535) return TGO_E_BAD_ARG;
    if (dtype == TGO_BF16) {
        auto kern = retention_kernel<bf16>;
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return tgo_launch_pdl(kern, grid, block, smem, stream, (const bf16*)q, q_stride,
                              (const bf16*)k, k_stride, (const bf16*)v, v_stride, out, H, dk, dv, vs,
                              decay, k_scale, act, rope, rot, q_start, state_slots, state);
    }
    if (dtype == TGO_F32) {
        auto kern = retention_kernel<float>;
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return tgo_launch_pdl(kern, grid, block, smem, stream, (const float*)q, q_stride,
                              (const float*)k, k_stride, (const float*)v, v_stride, out, H, dk, dv,
                              vs, decay, k_scale, act, rope, rot, q_start, state_slots, state);
    }
    return TGO_E_BAD_ARG;
}

// ------------------------------------------------------------------ a step of single tokens
// One token a request: o = decay S^T q + (q . k) v and S <- decay S + k v^T straight from and
// to global memory, a block per (request, head, 32 columns of S), every element of S read
// once and written once.
#define RD_THREADS 128
template <typename T>
__global__ void __launch_bounds__(RD_THREADS)
retention_decode_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ k,
                        long long k_stride, const T* __restrict__ v, long long v_stride,
                        float* __restrict__ out, int H, int dk, int dv,
                        const float* __restrict__ decay, float k_scale, int act,
                        const float* __restrict__ rope, int rot,
                        const int* __restrict__ state_slots, float* __restrict__ state) {
    extern __shared__ float smem[];
    float* qs = smem;                 // [dk]
    float* ks = qs + dk;              // [dk]
    float* red = ks + dk;             // [RD_THREADS / 32][32]
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, rg = threadIdx.x >> 5;
    const int c = blockIdx.z * 32 + lane;
    const size_t t = (size_t)b;
    const float* cs = rope ? rope + t * rot : nullptr;
    const T* qr = q + t * q_stride + (size_t)h * dk;
    const T* kr = k + t * k_stride + (size_t)h * dk;
    for (int d = threadIdx.x; d < dk; d += RD_THREADS) {
        qs[d] = cs ? rotated(qr, cs, d, rot, act) : taken(qr[d], act);
        ks[d] = (cs ? rotated(kr, cs, d, rot, act) : taken(kr[d], act)) * k_scale;
    }
    __syncthreads();
    const float g = decay[h];
    const float vc = c < dv ? taken(v[t * v_stride + (size_t)h * dv + c], act) : 0.f;
    float* Sg = state + (((size_t)state_slots[b] * H + h) * dk) * dv;
    float far = 0.f, qk = 0.f;
    constexpr int RG = RD_THREADS / 32;
    // eight rows of the state a thread and turn: all their loads first (the stores into the
    // same array would otherwise hold every next load back), then the arithmetic and the stores
    for (int d0 = rg; d0 < dk; d0 += RG * 8) {
        float sv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int d = d0 + u * RG;
            sv[u] = (d < dk && c < dv) ? Sg[(size_t)d * dv + c] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int d = d0 + u * RG;
            if (d < dk) {
                qk += qs[d] * ks[d];
                if (c < dv) {
                    far += qs[d] * sv[u];
                    Sg[(size_t)d * dv + c] = g * sv[u] + ks[d] * vc;
                }
            }
        }
    }
    __shared__ float qk_part[RG];
    red[rg * 32 + lane] = far;
    if (lane == 0) qk_part[rg] = qk;        // every lane of a row group holds the same part
    __syncthreads();
    if (rg == 0 && c < dv) {
        float f = 0.f, a = 0.f;
#pragma unroll
        for (int x = 0; x < RG; ++x) {
            f += red[x * 32 + lane];
            a += qk_part[x];
        }
        out[(t * H + h) * dv + c] = g * f + a * vc;
    }
}

// --------------------------------------------------------------- prompt portions, by chunks
// The tokens of a step are cut into chunks of up to RC_CHUNK tokens of one request (a list
// the host makes: first token row and count of each chunk). Three launches, every chunk of
// every head in parallel in the first and the third:
//
//   summaries   U_c = sum_j decay^(n-1-j) k_j v_j^T                [dk, dv] per (chunk, head)
//   scan        per request and head, chunk after chunk: P_c = S; S <- decay^n S + U_c (the
//               state before each chunk replaces its summary; the last S is the new state)
//   outputs     o_i = sum_{j<=i} decay^(i-j) (q_i . k_j) v_j + decay^(i+1) P_c^T q_i
#define RC_CHUNK 64
#define RC_THREADS 256
#define RC_VS 64                      // columns of V and of the state taken at a time

template <typename T>
__device__ __forceinline__ void load_rotated(float* dst, int ld, const T* __restrict__ x, long long stride,
                                             int h, int dk, const float* __restrict__ rope, int rot,
                                             int tok0, int n, float mul, int act) {
    // four elements a turn, their loads first: a row of the chunk is short, and a loop that
    // waits for every element's loads in turn is bound by their latency
    for (int i0 = threadIdx.x; i0 < n * dk; i0 += 4 * RC_THREADS) {
        float val[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * RC_THREADS;
            if (i < n * dk) {
                const int r = i / dk, d = i % dk;
                const size_t t = (size_t)(tok0 + r);
                const T* row = x + t * stride + (size_t)h * dk;
                val[u] = (rope ? rotated(row, rope + t * rot, d, rot, act) : taken(row[d], act)) * mul;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * RC_THREADS;
            if (i < n * dk) dst[(i / dk) * ld + i % dk] = val[u];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(RC_THREADS)
retention_summaries_kernel(const T* __restrict__ k, long long k_stride, const T* __restrict__ v,
                           long long v_stride, int H, int dk, int dv,
                           const float* __restrict__ decay, float k_scale, int act,
                           const float* __restrict__ rope, int rot,
                           const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_ntok,
                           float* __restrict__ U) {
    extern __shared__ float smem[];
    const int ldk = dk + 1;
    float* Ks = smem;                         // [RC_CHUNK][dk + 1], rows times decay^(n-1-j)
    float* Vs = Ks + RC_CHUNK * ldk;          // [RC_CHUNK][RC_VS]
    float* pw = Vs + RC_CHUNK * RC_VS;        // [RC_CHUNK + 1]
    pdl_wait();
    const int ci = blockIdx.x, h = blockIdx.y;
    const int tok0 = chunk_tok0[ci], n = chunk_ntok[ci];
    if (threadIdx.x == 0) {
        float x = 1.f;
        const float g = decay[h];
        for (int i = 0; i <= RC_CHUNK; ++i) { pw[i] = x; x *= g; }
    }
    load_rotated(Ks, ldk, k, k_stride, h, dk, rope, rot, tok0, n, k_scale, act);
    __syncthreads();
    for (int i = threadIdx.x; i < n * dk; i += RC_THREADS) Ks[(i / dk) * ldk + i % dk] *= pw[n - 1 - i / dk];
    float* Uo = U + ((size_t)ci * H + h) * dk * dv;
    for (int c0 = 0; c0 < dv; c0 += RC_VS) {
        const int nc = dv - c0 < RC_VS ? dv - c0 : RC_VS;
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < n * RC_VS; i += RC_THREADS) {
            const int r = i / RC_VS, c = i % RC_VS;
            Vs[i] = c < nc ? taken(v[(size_t)(tok0 + r) * v_stride + (size_t)h * dv + c0 + c], act) : 0.f;
        }
        __syncthreads();
        // U[d][c] over 4 x 4 register tiles: tiles of rows d0.., columns cc..
        const int tiles_c = RC_VS / 4, tiles_d = (dk + 3) / 4;
        for (int tile = threadIdx.x; tile < tiles_d * tiles_c; tile += RC_THREADS) {
            const int d0 = (tile / tiles_c) * 4, cc = (tile % tiles_c) * 4;
            float acc[4][4] = {};
            for (int j = 0; j < n; ++j) {
                const float4 vv = *(const float4*)(Vs + j * RC_VS + cc);
                float kk[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) kk[x] = d0 + x < dk ? Ks[j * ldk + d0 + x] : 0.f;
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[x][0] += kk[x] * vv.x; acc[x][1] += kk[x] * vv.y;
                    acc[x][2] += kk[x] * vv.z; acc[x][3] += kk[x] * vv.w;
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    if (d0 + x < dk && cc + y < nc) Uo[(size_t)(d0 + x) * dv + c0 + cc + y] = acc[x][y];
        }
    }
}

// grid (requests, heads, ceil(dk * dv / 256)): a thread an element of the state
__global__ void retention_scan_kernel(int H, int dk, int dv, const float* __restrict__ decay,
                                      const int* __restrict__ q_start,
                                      const int* __restrict__ state_slots,
                                      const int* __restrict__ chunk_first, float* __restrict__ U,
                                      float* __restrict__ state) {
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y;
    const int e = blockIdx.z * blockDim.x + threadIdx.x;
    if (e >= dk * dv) return;
    const int n_tok = q_start[b + 1] - q_start[b];
    if (n_tok <= 0) return;
    const int chunks = (n_tok + RC_CHUNK - 1) / RC_CHUNK;
    const float g = decay[h];
    float gfull = 1.f;
    for (int i = 0; i < RC_CHUNK; ++i) gfull *= g;
    float* sp = state + ((size_t)state_slots[b] * H + h) * dk * dv + e;
    float s = *sp;
    const int c0 = chunk_first[b];
    const size_t step = (size_t)H * dk * dv;
    float* ub = U + ((size_t)c0 * H + h) * dk * dv + e;
    for (int cb = 0; cb < chunks; cb += 16) {        // sixteen summaries loaded ahead of their use
        float u[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) u[x] = cb + x < chunks ? ub[(size_t)(cb + x) * step] : 0.f;
#pragma unroll
        for (int x = 0; x < 16; ++x) {
            const int c = cb + x;
            if (c < chunks) {
                ub[(size_t)c * step] = s;
                float gn = gfull;
                if (c == chunks - 1) {
                    gn = 1.f;
                    for (int i = 0; i < n_tok - c * RC_CHUNK; ++i) gn *= g;
                }
                s = gn * s + u[x];
            }
        }
    }
    *sp = s;
}

template <typename T>
__global__ void __launch_bounds__(RC_THREADS)
retention_outputs_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ k,
                         long long k_stride, const T* __restrict__ v, long long v_stride,
                         float* __restrict__ out, int H, int dk, int dv,
                         const float* __restrict__ decay, float k_scale, int act,
                         const float* __restrict__ rope, int rot,
                         const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_ntok,
                         const float* __restrict__ P) {
    extern __shared__ float smem[];
    const int ldk = dk + 1, lda = RC_CHUNK + 1;
    float* Qs = smem;                          // [RC_CHUNK][dk + 1]
    float* Ks = Qs + RC_CHUNK * ldk;           // [RC_CHUNK][dk + 1]
    float* As = Ks + RC_CHUNK * ldk;           // [RC_CHUNK][RC_CHUNK + 1]
    float* Vs = As + RC_CHUNK * lda;           // [RC_CHUNK][RC_VS]
    float* Ss = Vs + RC_CHUNK * RC_VS;         // [dk][RC_VS]
    float* pw = Ss + (size_t)dk * RC_VS;       // [RC_CHUNK + 1]
    pdl_wait();
    const int ci = blockIdx.x, h = blockIdx.y;
    const int tok0 = chunk_tok0[ci], n = chunk_ntok[ci];
    if (threadIdx.x == 0) {
        float x = 1.f;
        const float g = decay[h];
        for (int i = 0; i <= RC_CHUNK; ++i) { pw[i] = x; x *= g; }
    }
    load_rotated(Qs, ldk, q, q_stride, h, dk, rope, rot, tok0, n, 1.f, act);
    load_rotated(Ks, ldk, k, k_stride, h, dk, rope, rot, tok0, n, k_scale, act);
    __syncthreads();
    // A[i][j] = decay^(i-j) q_i . k_j (j <= i), 4 x 4 tiles
    {
        const int tiles = RC_CHUNK / 4;
        for (int tile = threadIdx.x; tile < tiles * tiles; tile += RC_THREADS) {
            const int i0 = (tile / tiles) * 4, j0 = (tile % tiles) * 4;
            if (i0 >= n || j0 >= n) continue;
            float acc[4][4] = {};
            if (j0 <= i0 + 3) {
                for (int d = 0; d < dk; ++d) {
                    float qq[4], kk[4];
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        qq[x] = Qs[(i0 + x) * ldk + d];
                        kk[x] = Ks[(j0 + x) * ldk + d];
                    }
#pragma unroll
                    for (int x = 0; x < 4; ++x)
#pragma unroll
                        for (int y = 0; y < 4; ++y) acc[x][y] += qq[x] * kk[y];
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int i = i0 + x, j = j0 + y;
                    As[i * lda + j] = (j <= i && i < n) ? acc[x][y] * pw[i - j] : 0.f;
                }
        }
    }
    const float* Pc = P + ((size_t)ci * H + h) * dk * dv;
    for (int c0 = 0; c0 < dv; c0 += RC_VS) {
        const int nc = dv - c0 < RC_VS ? dv - c0 : RC_VS;
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < n * RC_VS; i += RC_THREADS) {
            const int r = i / RC_VS, c = i % RC_VS;
            Vs[i] = c < nc ? taken(v[(size_t)(tok0 + r) * v_stride + (size_t)h * dv + c0 + c], act) : 0.f;
        }
#pragma unroll 8
        for (int i = threadIdx.x; i < dk * RC_VS; i += RC_THREADS) {
            const int d = i / RC_VS, c = i % RC_VS;
            Ss[i] = c < nc ? Pc[(size_t)d * dv + c0 + c] : 0.f;
        }
        __syncthreads();
        const int tiles_c = RC_VS / 4, tiles_i = (n + 3) / 4;
        for (int tile = threadIdx.x; tile < tiles_i * tiles_c; tile += RC_THREADS) {
            const int i0 = (tile / tiles_c) * 4, cc = (tile % tiles_c) * 4;
            float near[4][4] = {}, far[4][4] = {};
            const int jmax = i0 + 3 < n - 1 ? i0 + 3 : n - 1;
            for (int j = 0; j <= jmax; ++j) {
                const float4 vv = *(const float4*)(Vs + j * RC_VS + cc);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float a = As[(i0 + x) * lda + j];        // rows >= n were zeroed or unused
                    near[x][0] += a * vv.x; near[x][1] += a * vv.y; near[x][2] += a * vv.z; near[x][3] += a * vv.w;
                }
            }
            for (int d = 0; d < dk; ++d) {
                const float4 ss = *(const float4*)(Ss + d * RC_VS + cc);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float qq = Qs[(i0 + x) * ldk + d];
                    far[x][0] += qq * ss.x; far[x][1] += qq * ss.y; far[x][2] += qq * ss.z; far[x][3] += qq * ss.w;
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    if (i0 + x < n && cc + y < nc)
                        out[((size_t)(tok0 + i0 + x) * H + h) * dv + c0 + cc + y] =
                            near[x][y] + pw[i0 + x + 1] * far[x][y];
        }
    }
}

// ------------------------------------------------ the same, for heads of 64 or 128 key channels
// The products in true float32 on the tensor cores: each number as three bfloat16 parts (split3.cuh), values that
// are bfloat16 numbers already as one. A block makes 128 columns of V: channels of V are the accumulators' lanes,
// tokens (or key channels) their columns, so that every operand is laid down as it lies in memory and a warp's results
// leave as whole lines.
//   summaries   U^T = V^T K: K's scaled and rotated rows and V, one product of 64 tokens;
//   scan        four neighbouring elements a thread, eight summaries asked for while the eight before
//               them are used: bound by memory (every summary read once, every state written once);
//   outputs     Q and K once for up to two slices: Q K^T by halves of 64 channels; P comes 64 channels x 128 columns
//               at a time through two buffers, P^T Q^T; A = decay^(i-j) Q K^T goes back to shared memory as
//               parts (over K's), V^T A^T; out = decay^(i+1) (Q P) + A V. A warp of its own issues the products while
//               sixteen lay the next operands down. (One slice a block, halves of Q, K and P one after the
//               other, two blocks an SM: 167 us.)
// Zeros of A times a value that is not finite are not zero: such a number is laid down as 0, which leaves what does
// not depend on it as it is, bit for bit, and a block that met one makes plain sums too (RF_PLAIN of a column a
// thread; MEASURED, all three launches: 4096 tokens, 16 heads of 128 x 256, all NaN 1400 us, all finite 206; 3050 by a thread a sum) and
// writes those that are not finite. A finite number too large for its parts (2^103 and more), or an A whose
// Q K^T is (2^80), is 0 there too: the plain sums of its row and the rows after it are written whatever they are, in its slice if it
// is one of V or P. So are those in the place of a result that the products made overflow.
// MEASURED (B200, 4096 tokens, 16 heads of 128 x 256, bfloat16 rows; register tiles of packed FMA in brackets):
// summaries 51 us (122), scan 40, outputs 121 us (190). The summaries are bound by the bytes of U; a block of the outputs
// by its chain: loads 5000 cycles, parts of Q and K 3000, 168 products of 75 cycles, results 2300.
#define RF_SLICE 128
#define RF_TILE 8192                  // 64 rows of 64 bfloat16 numbers
#define RF_LOOP_LD 129                // rows of the plain sums' tiles
#define RF_PLAIN 16                   // plain sums a thread makes side by side

__device__ int retention_error_flag = 0;

// Eight channels of a row as they lie, and their values after the activation. Asked for first and turned
// later, so that several are under way at once.
template <typename T> struct Raw8;
template <> struct Raw8<bf16> { uint4 u; };
template <> struct Raw8<float> { float4 a, b; };
__device__ __forceinline__ void load8(Raw8<bf16>& w, const bf16* __restrict__ x) { w.u = *(const uint4*)x; }
__device__ __forceinline__ void load8(Raw8<float>& w, const float* __restrict__ x) {
    w.a = ((const float4*)x)[0];
    w.b = ((const float4*)x)[1];
}
__device__ __forceinline__ void taken8(const Raw8<bf16>& raw, int act, float (&f)[8]) {
    const uint32_t w[4] = {raw.u.x, raw.u.y, raw.u.z, raw.u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __bfloat1622float2(*(const __nv_bfloat162*)&w[i]);
        f[2 * i] = v.x;
        f[2 * i + 1] = v.y;
    }
    if (act == 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] / (1.f + expf(-f[i]));
}
__device__ __forceinline__ void taken8(const Raw8<float>& raw, int act, float (&f)[8]) {
    f[0] = raw.a.x; f[1] = raw.a.y; f[2] = raw.a.z; f[3] = raw.a.w;
    f[4] = raw.b.x; f[5] = raw.b.y; f[6] = raw.b.z; f[7] = raw.b.w;
    if (act == 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] / (1.f + expf(-f[i]));
}

// Two runs of eight channels of a row that a rotation turns into each other, or two runs that it leaves as they are:
// pair p of DK / 16; rot is a multiple of 16.
template <typename T> struct Pair8 {
    Raw8<T> x, y;
    float4 c0, c1, s0, s1;
    int lo, hi;
    bool turned;
    __device__ __forceinline__ void load(const T* __restrict__ row, const float* __restrict__ cs, int p, int rot) {
        turned = cs && 16 * p < rot;
        lo = turned ? 8 * p : 16 * p;
        hi = turned ? lo + (rot >> 1) : lo + 8;
        load8(x, row + lo);
        load8(y, row + hi);
        if (turned) {
            c0 = *(const float4*)(cs + lo); c1 = *(const float4*)(cs + lo + 4);
            s0 = *(const float4*)(cs + hi); s1 = *(const float4*)(cs + hi + 4);
        }
    }
    __device__ __forceinline__ void values(int act, float (&f)[8], float (&g)[8]) const {
        taken8(x, act, f);
        taken8(y, act, g);
        if (!turned) return;
        const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const float n[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float a = f[i], b = g[i];
            f[i] = a * c[i] - b * n[i];
            g[i] = b * c[i] + a * n[i];
        }
    }
};

// The powers of the decay, 0 .. RC_CHUNK, by repeated multiplication.
__device__ __forceinline__ void rf_powers(float* pw, float g) {
    if (threadIdx.x == 0) {
        float x = 1.f;
        for (int i = 0; i <= RC_CHUNK; ++i) { pw[i] = x; x *= g; }
    }
}

// Columns c0 .. c0 + 127 of the chunk's values, asked for and then laid down (rows of tokens, two tiles of 64 columns a
// part); rows past n and columns past dv are zeros. True: a thread's are not all finite.
template <int THREADS> __device__ constexpr int rf_v_runs() { return RC_CHUNK * (RF_SLICE / 8) / THREADS; }
template <typename T, int THREADS>
__device__ __forceinline__ void rf_ask_v(Raw8<T> (&raw)[rf_v_runs<THREADS>()], const T* __restrict__ v, long long v_stride, int h,
                                         int dv, int c0, int tok0, int n) {
#pragma unroll
    for (int j = 0; j < rf_v_runs<THREADS>(); ++j) {
        const int i = threadIdx.x + j * THREADS, r = i / (RF_SLICE / 8), c = (i % (RF_SLICE / 8)) * 8;
        load8(raw[j], v + (size_t)(tok0 + (r < n ? r : 0)) * v_stride + (size_t)h * dv + (c0 + c < dv ? c0 + c : 0));
    }
}
template <typename T, int VP, int THREADS>
__device__ __forceinline__ bool rf_put_v(uint32_t tile, const Raw8<T> (&raw)[rf_v_runs<THREADS>()], int dv, int c0, int n, int act, int* too_large) {
    bool odd = false;
#pragma unroll
    for (int j = 0; j < rf_v_runs<THREADS>(); ++j) {
        const int i = threadIdx.x + j * THREADS, r = i / (RF_SLICE / 8), piece = i % (RF_SLICE / 8);
        const bool ok = r < n && c0 + 8 * piece < dv;
        const uint32_t dst = tile + (piece >> 3) * RF_TILE + s3_place(r, piece & 7);
        if constexpr (VP == 1) {
            uint4 w = ok ? raw[j].u : make_uint4(0u, 0u, 0u, 0u);
            odd = s3_finite8(w) || odd;
            s3_store16(dst, w);
        } else {
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (ok) taken8(raw[j], act, f);
            odd = s3_put8(f, dst, 2 * RF_TILE, r, too_large) || odd;
        }
    }
    return odd;
}
// The parts of eight numbers to their place in three tiles `step` bytes apart; `from`: the first row that what is too large counts for.
__device__ __forceinline__ bool rf_put8(uint32_t tile, uint32_t step, int row, int piece, const float (&f)[8], int from, int* too_large) {
    return s3_put8(f, tile + s3_place(row, piece), step, from, too_large);
}
// The value of column c of a token, as the plain sums take it.
template <typename T>
__device__ __forceinline__ float rf_value(const T* __restrict__ v, long long v_stride, size_t t, int h, int dv, int c, int act) {
    return taken(v[t * v_stride + (size_t)h * dv + c], act);
}
__device__ __forceinline__ bool rf_not_finite(float x) { return !(fabsf(x) < __int_as_float(0x7f800000)); }
// A block's products are there (`phase` of their barrier), for all threads or for none.
__device__ __forceinline__ bool rf_made(uint64_t* bar, uint32_t phase, int code) {
    const bool ok = __syncthreads_and(tg_wait(bar, phase, &retention_error_flag, code));
    tg_after();
    return ok;
}

// The plain sums of a block that met a number which is not finite or too large.
template <typename T, int DK>
__device__ __forceinline__ void rf_plain_summaries(float* Kf, const T* __restrict__ k, long long k_stride, const T* __restrict__ v, long long v_stride,
                                                int H, int dv, float k_scale, int act, const float* __restrict__ rope, int rot, int tok0, int n,
                                                int h, int first, int ns, const float* pw, const int* too_large, float* Uo) {
    load_rotated(Kf, RF_LOOP_LD, k, k_stride, h, DK, rope, rot, tok0, n, k_scale, act);
    __syncthreads();
    for (int i = threadIdx.x; i < DK / RF_PLAIN * RF_SLICE * ns; i += RC_THREADS) {
        const int d = i / (RF_SLICE * ns) * RF_PLAIN, c = first + i % (RF_SLICE * ns);
        if (c >= dv) continue;
        const bool plain = min(too_large[(c - first) / RF_SLICE], too_large[2]) < RC_CHUNK;
        float s[RF_PLAIN] = {};
#pragma unroll 4
        for (int j = 0; j < n; ++j) {
            const float x = rf_value(v, v_stride, (size_t)(tok0 + j), h, dv, c, act);
#pragma unroll
            for (int r = 0; r < RF_PLAIN; ++r) s[r] = fmaf(Kf[j * RF_LOOP_LD + d + r] * pw[n - 1 - j], x, s[r]);
        }
#pragma unroll
        for (int r = 0; r < RF_PLAIN; ++r) {
            float* to = Uo + (size_t)(d + r) * dv + c;
            if (plain || rf_not_finite(s[r]) || rf_not_finite(*to)) *to = s[r];
        }
    }
}

// VP: parts a value has (1: bfloat16 rows without an activation). A block makes the columns of up to two slices.
template <typename T, int DK, int VP>
__global__ void __launch_bounds__(RC_THREADS, VP == 1 ? 2 : 1)
retention_summaries_tc_kernel(const T* __restrict__ k, long long k_stride, const T* __restrict__ v, long long v_stride,
                              int H, int dv, const float* __restrict__ decay, float k_scale, int act,
                              const float* __restrict__ rope, int rot, const int* __restrict__ chunk_tok0,
                              const int* __restrict__ chunk_ntok, int slices, float* __restrict__ U) {
    constexpr int KB = DK / 64;                          // tiles of a part of K
    extern __shared__ unsigned char rf_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)rf_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sV = base + 3 * KB * RF_TILE;         // K's parts, then either slice's of V
    __shared__ float pw[RC_CHUNK + 1];
    __shared__ __align__(8) uint64_t bars[2];            // one a slice
    __shared__ uint32_t tmem_slot;
    __shared__ int too_large[3];                         // either slice's V; K
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) tg_alloc<2 * DK>(&tmem_slot);
    if (threadIdx.x == 0) { tg_init(&bars[0], 1); tg_init(&bars[1], 1); tg_init_done(); }
    if (threadIdx.x < 3) too_large[threadIdx.x] = RC_CHUNK;
    pdl_wait();
    const int ci = blockIdx.x, h = blockIdx.y, first = blockIdx.z * slices * RF_SLICE;
    const int n = chunk_ntok[ci], tok0 = n > 0 ? chunk_tok0[ci] : 0;      // rows past n read the first one
    const int ns = min(slices, (dv - first + RF_SLICE - 1) / RF_SLICE);
    Raw8<T> vr[rf_v_runs<RC_THREADS>()];
    rf_ask_v<T, RC_THREADS>(vr, v, v_stride, h, dv, first, tok0, n);
    rf_powers(pw, decay[h]);
    tg_before();
    __syncthreads();
    tg_after();
    const uint32_t tmem = tmem_slot;
    bool odd = false;
    constexpr int PAIRS = RC_CHUNK * (DK / 16) / RC_THREADS;
    Pair8<T> kr[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
        const int i = threadIdx.x + j * RC_THREADS, r = i / (DK / 16);
        const size_t t = (size_t)(tok0 + (r < n ? r : 0));
        kr[j].load(k + t * k_stride + (size_t)h * DK, rope ? rope + t * rot : nullptr, i % (DK / 16), rot);
    }
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
        const int r = (threadIdx.x + j * RC_THREADS) / (DK / 16);
        float f[8], g[8];
        kr[j].values(act, f, g);
        const float w = r < n ? pw[n - 1 - r] : 0.f;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            f[x] = r < n ? f[x] * k_scale * w : 0.f;
            g[x] = r < n ? g[x] * k_scale * w : 0.f;
        }
        odd = rf_put8(tg_smem(base) + (uint32_t)(kr[j].lo / 64 * RF_TILE), KB * RF_TILE, r, (kr[j].lo / 8) & 7, f, r, &too_large[2]) || odd;
        odd = rf_put8(tg_smem(base) + (uint32_t)(kr[j].hi / 64 * RF_TILE), KB * RF_TILE, r, (kr[j].hi / 8) & 7, g, r, &too_large[2]) || odd;
    }
    for (int s = 0; s < ns; ++s) {
        unsigned char* sv = sV + s * 2 * VP * RF_TILE;
        odd = rf_put_v<T, VP, RC_THREADS>(tg_smem(sv), vr, dv, first + s * RF_SLICE, n, act, &too_large[s]) || odd;
        if (s + 1 < ns) rf_ask_v<T, RC_THREADS>(vr, v, v_stride, h, dv, first + (s + 1) * RF_SLICE, tok0, n);
        s3_fence();
        odd = __syncthreads_or(odd);
        if (warp == 0 && tg_elect()) {
            s3_products<VP, 3, RC_CHUNK / 16>(tmem + (uint32_t)(DK * s), tg_desc_mn(sv, RF_TILE), 2 * RF_TILE >> 4, 128,
                                              tg_desc_mn(base, RF_TILE), KB * RF_TILE >> 4, 128, tg_idesc(DK, true, true), false);
            tg_commit(&bars[s]);
        }
        __syncwarp();
    }
    bool ok = true;
    for (int s = 0; s < ns && ok; ++s) ok = rf_made(&bars[s], 0, 1);
    float* Uo = U + ((size_t)ci * H + h) * DK * dv;
    if (ok) {
        const int d0 = (warp >> 2) * (DK / 2);
        float nan = 0.f;
        for (int s = 0; s < ns; ++s) {
            const int c = first + s * RF_SLICE + (warp & 3) * 32 + lane;
#pragma unroll
            for (int x = 0; x < DK / 2; x += 32) {
                uint32_t r[32];
                tg_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(DK * s + d0 + x), r);
                tg_wait_ld();
                float* dst = Uo + (size_t)(d0 + x) * dv + c;
                if (c < dv)
#pragma unroll
                    for (int i = 0; i < 32; ++i, dst += dv) {
                        const float sum = __uint_as_float(r[i]) * (VP == 1 ? S3_DOWN : S3_DOWN * S3_DOWN);
                        nan = fmaf(sum, 0.f, nan);       // 0 as long as all are finite
                        *dst = sum;
                    }
            }
        }
        if (__syncthreads_or(odd || nan != 0.f)) {
            rf_plain_summaries<T, DK>((float*)base, k, k_stride, v, v_stride, H, dv, k_scale, act, rope, rot, tok0, n, h, first, ns, pw, too_large, Uo);
        }
    } else {
        for (int s = 0; s < ns; ++s) tg_wait(&bars[s], 0, &retention_error_flag, 1);      // products that may still be under way
    }
    tg_before();
    __syncthreads();
    if (warp == 0) {
        tg_after();
        tg_free<2 * DK>(tmem);
    }
}

// grid (requests, heads, ceil(dk dv / 1024)): a thread four neighbouring elements of the state
__global__ void __launch_bounds__(256)
retention_scan4_kernel(int H, int dkdv, const float* __restrict__ decay, const int* __restrict__ q_start,
                       const int* __restrict__ state_slots, const int* __restrict__ chunk_first, float* __restrict__ U,
                       float* __restrict__ state) {
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y;
    const int e = 4 * (blockIdx.z * blockDim.x + threadIdx.x);
    const int n_tok = q_start[b + 1] - q_start[b];
    if (e >= dkdv || n_tok <= 0) return;
    const int chunks = (n_tok + RC_CHUNK - 1) / RC_CHUNK, last = n_tok - (chunks - 1) * RC_CHUNK;
    const float g = decay[h];
    float gfull = 1.f, glast = 1.f;
    for (int i = 0; i < RC_CHUNK; ++i) {
        gfull *= g;
        if (i < last) glast *= g;
    }
    float4* sp = (float4*)(state + ((size_t)state_slots[b] * H + h) * dkdv + e);
    float4 s = *sp;
    const size_t step = (size_t)H * dkdv / 4;
    float4* ub = (float4*)(U + ((size_t)chunk_first[b] * H + h) * dkdv + e);
    constexpr int N = 8;
    float4 u[N], w[N];
#pragma unroll
    for (int x = 0; x < N; ++x) u[x] = x < chunks ? ub[(size_t)x * step] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int cb = 0; cb < chunks; cb += N) {
#pragma unroll
        for (int x = 0; x < N; ++x)
            w[x] = cb + N + x < chunks ? ub[(size_t)(cb + N + x) * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int x = 0; x < N; ++x) {
            const int c = cb + x;
            if (c >= chunks) break;
            ub[(size_t)c * step] = s;
            const float gn = c == chunks - 1 ? glast : gfull;
            s.x = gn * s.x + u[x].x; s.y = gn * s.y + u[x].y; s.z = gn * s.z + u[x].z; s.w = gn * s.w + u[x].w;
        }
#pragma unroll
        for (int x = 0; x < N; ++x) u[x] = w[x];
    }
    *sp = s;
}

// Shared memory: Q's parts (a part DK / 64 tiles), two buffers of P's (64 channels x 128 columns, two tiles a part),
// K's parts, over which A's and one slice's values come to lie (24 KB more than K at DK = 128).
#define RF_OUT_THREADS 512           // and a warp that issues the products
template <int DK> __host__ __device__ constexpr int rf_out_k() { return 3 * (DK / 64) * RF_TILE + 2 * 6 * RF_TILE; }
template <int DK> __host__ __device__ constexpr int rf_out_bytes() { return rf_out_k<DK>() + 9 * RF_TILE; }

template <typename T, int DK>
__device__ __forceinline__ void rf_plain_outputs(float* Qf, const T* __restrict__ q, long long q_stride, const T* __restrict__ k, long long k_stride,
                                              const T* __restrict__ v, long long v_stride, float* __restrict__ out, int H, int dv, float k_scale,
                                              int act, const float* __restrict__ rope, int rot, int tok0, int n, int h, int first, int ns,
                                              const float* pw, const int* plain_from, const float* __restrict__ Pc) {
    // Qf [64][RF_LOOP_LD], then K's
    float* Kf = Qf + RC_CHUNK * RF_LOOP_LD;
    float* Af = Kf + RC_CHUNK * RF_LOOP_LD;          // [64][65]
    load_rotated(Qf, RF_LOOP_LD, q, q_stride, h, DK, rope, rot, tok0, n, 1.f, act);
    load_rotated(Kf, RF_LOOP_LD, k, k_stride, h, DK, rope, rot, tok0, n, k_scale, act);
    __syncthreads();
    for (int x = threadIdx.x; x < n * RC_CHUNK; x += RF_OUT_THREADS + 32) {
        const int i = x / RC_CHUNK, j = x % RC_CHUNK;
        float s = 0.f;
        for (int d = 0; j <= i && d < DK; ++d) s = fmaf(Qf[i * RF_LOOP_LD + d], Kf[j * RF_LOOP_LD + d], s);
        Af[i * (RC_CHUNK + 1) + j] = j <= i ? s * pw[i - j] : 0.f;
    }
    __syncthreads();
    for (int x = threadIdx.x; x < RC_CHUNK / RF_PLAIN * RF_SLICE * ns; x += RF_OUT_THREADS + 32) {
        const int i = x / (RF_SLICE * ns) * RF_PLAIN, c = first + x % (RF_SLICE * ns);
        if (c >= dv || i >= n) continue;             // of rows past n the sums are made and not written
        const int plain = min(plain_from[(c - first) / RF_SLICE], plain_from[2]);
        float s[RF_PLAIN] = {};
#pragma unroll 4
        for (int d = 0; d < DK; ++d) {
            const float p = Pc[(size_t)d * dv + c];
#pragma unroll
            for (int r = 0; r < RF_PLAIN; ++r) s[r] = fmaf(Qf[(i + r) * RF_LOOP_LD + d], p, s[r]);
        }
#pragma unroll
        for (int r = 0; r < RF_PLAIN; ++r) s[r] *= pw[i + r + 1];
#pragma unroll 4
        for (int j = 0; j < min(n, i + RF_PLAIN); ++j) {
            const float y = rf_value(v, v_stride, (size_t)(tok0 + j), h, dv, c, act);
#pragma unroll
            for (int r = 0; r < RF_PLAIN; ++r)
                if (j <= i + r) s[r] = fmaf(Af[(i + r) * (RC_CHUNK + 1) + j], y, s[r]);
        }
#pragma unroll
        for (int r = 0; r < RF_PLAIN; ++r) {
            float* to = out + ((size_t)(tok0 + i + r) * H + h) * dv + c;
            if (i + r < n && (i + r >= plain || rf_not_finite(s[r]) || rf_not_finite(*to))) *to = s[r];
        }
    }
}

template <typename T, int DK, int VP>
__global__ void __launch_bounds__(RF_OUT_THREADS + 32, 1)
retention_outputs_tc_kernel(const T* __restrict__ q, long long q_stride, const T* __restrict__ k, long long k_stride,
                            const T* __restrict__ v, long long v_stride, float* __restrict__ out, int H, int dv,
                            const float* __restrict__ decay, float k_scale, int act, const float* __restrict__ rope,
                            int rot, const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_ntok, int slices,
                            const float* __restrict__ P) {
    constexpr int HALVES = DK / 64, THREADS = RF_OUT_THREADS;
    extern __shared__ unsigned char rf_raw[];
    unsigned char* sQ = (unsigned char*)(((uintptr_t)rf_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sP = sQ + 3 * HALVES * RF_TILE;       // [2]
    unsigned char* sK = sQ + rf_out_k<DK>();
    unsigned char* sA = sK;
    unsigned char* sV = sK + 3 * RF_TILE;
    __shared__ float pw[RC_CHUNK + 1];
    __shared__ __align__(8) uint64_t bars[9];
    __shared__ uint32_t tmem_slot;
    __shared__ int plain_from[3];                        // the first row whose plain sums are written whatever they are: a slice's; both
    uint64_t *s_done = bars, *p_done = bars + 1 /* [2] */, *v_done = bars + 3;
    uint64_t *qk_full = bars + 4, *p_full = bars + 5 /* [2] */, *a_full = bars + 7, *v_full = bars + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) tg_alloc512(&tmem_slot);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 9; ++i) tg_init(&bars[i], i < 4 ? 1 : THREADS / 32);
        plain_from[0] = plain_from[1] = plain_from[2] = RC_CHUNK;
        tg_init_done();
    }
    pdl_wait();
    const int ci = blockIdx.x, h = blockIdx.y, first = blockIdx.z * slices * RF_SLICE;
    const int n = chunk_ntok[ci], tok0 = n > 0 ? chunk_tok0[ci] : 0;      // rows past n read the first one
    const int ns = min(slices, (dv - first + RF_SLICE - 1) / RF_SLICE), stages = ns * HALVES;
    const float* Pc = P + ((size_t)ci * H + h) * DK * dv;
    // columns: Q K^T by halves (0, 64); P Q of slice s and half x at 128 + 64 (2 s + x); A V of slice s at 384 + 64 s
    bool odd = false, ok = true;
    if (warp == THREADS / 32) {
        // ---------------------------------------------------------- issuer
        tg_before();
        __syncthreads();
        tg_after();
        const uint32_t tmem = tmem_slot;
        const bool leader = tg_elect();
        auto wait = [&](uint64_t* bar, uint32_t phase) {
            ok = __all_sync(0xffffffffu, ok && tg_wait(bar, phase, &retention_error_flag, 6));
            tg_after();
            return ok;
        };
        if (wait(qk_full, 0) && leader) {                // rows 64.. of the accumulators are nobody's
#pragma unroll
            for (int x = 0; x < HALVES; ++x)
                s3_products<3, 3, 4>(tmem + 64u * x, tg_desc(sQ + x * RF_TILE), HALVES * RF_TILE >> 4, 2, tg_desc(sK + x * RF_TILE),
                                     HALVES * RF_TILE >> 4, 2, tg_idesc(64), false);
            tg_commit(s_done);
        }
        __syncwarp();
        auto values = [&](int s) {
            if (leader) {
                s3_products<VP, 3, 4>(tmem + 384u + 64u * s, tg_desc_mn(sV, RF_TILE), 2 * RF_TILE >> 4, 128, tg_desc(sA), RF_TILE >> 4, 2,
                                      tg_idesc(64, false, true), false);
                tg_commit(v_done);
            }
            __syncwarp();
        };
        for (int stage = 0; stage < stages && ok; ++stage) {
            const int b = stage & 1, x = stage % HALVES;
            if (wait(&p_full[b], (stage >> 1) & 1) && leader) {
                s3_products<3, 3, 4>(tmem + 128u + 64u * (2 * (stage / HALVES) + x), tg_desc_mn(sP + b * 6 * RF_TILE, RF_TILE),
                                     2 * RF_TILE >> 4, 128, tg_desc(sQ + x * RF_TILE), HALVES * RF_TILE >> 4, 2, tg_idesc(64, false, true), false);
                tg_commit(&p_done[b]);
            }
            __syncwarp();
            if (stage == HALVES - 1 && ok && wait(a_full, 0)) values(0);
        }
        if (ns > 1 && ok && wait(v_full, 0)) values(1);
    } else {
        // ---------------------------------------------------------- parts and results
        // Q and K
        constexpr int PAIRS = 2 * RC_CHUNK * (DK / 16) / THREADS;
        Pair8<T> run[PAIRS];
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
            const int i = threadIdx.x + j * THREADS, r = (i / (DK / 16)) % RC_CHUNK;
            const size_t t = (size_t)(tok0 + (r < n ? r : 0));
            run[j].load(i / (RC_CHUNK * (DK / 16)) ? k + t * k_stride + (size_t)h * DK : q + t * q_stride + (size_t)h * DK,
                        rope ? rope + t * rot : nullptr, i % (DK / 16), rot);
        }
        // P: a stage is 64 channels x 128 columns (the halves of a slice one after the other), eight columns a thread and run
        float4 p[2][2];
        auto ask_p = [&](int stage) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int i = threadIdx.x + j * THREADS, d = 64 * (stage % HALVES) + i / 16, c = first + stage / HALVES * RF_SLICE + (i % 16) * 8;
                const float4* src = (const float4*)(Pc + (size_t)d * dv + (c < dv ? c : 0));
                p[j][0] = src[0];
                p[j][1] = src[1];
            }
        };
        ask_p(0);
        rf_powers(pw, decay[h]);
        tg_before();
        __syncthreads();
        tg_after();
        const uint32_t tmem = tmem_slot, lanes = (uint32_t)((warp & 3) * 32) << 16;
        auto full = [&](uint64_t* bar) {                     // a warp's share of an operand is laid down
            s3_fence();
            tg_before();
            __syncwarp();
            if (lane == 0) tg_arrive(bar);
        };
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
            const int i = threadIdx.x + j * THREADS, r = (i / (DK / 16)) % RC_CHUNK;
            const bool key = i / (RC_CHUNK * (DK / 16));
            float f[8], g[8];
            run[j].values(act, f, g);
            const float w = r >= n ? 0.f : key ? k_scale : 1.f;
            if (r >= n || key)
#pragma unroll
                for (int x = 0; x < 8; ++x) { f[x] = r >= n ? 0.f : f[x] * w; g[x] = r >= n ? 0.f : g[x] * w; }
            const uint32_t tile = tg_smem(key ? sK : sQ);
            odd = rf_put8(tile + (uint32_t)(run[j].lo / 64 * RF_TILE), HALVES * RF_TILE, r, (run[j].lo / 8) & 7, f, r, &plain_from[2]) || odd;
            odd = rf_put8(tile + (uint32_t)(run[j].hi / 64 * RF_TILE), HALVES * RF_TILE, r, (run[j].hi / 8) & 7, g, r, &plain_from[2]) || odd;
        }
        full(qk_full);
        Raw8<T> vr[rf_v_runs<THREADS>()];
        for (int stage = 0; stage < stages; ++stage) {
            const int b = stage & 1;
            unsigned char* buf = sP + b * 6 * RF_TILE;
            if (stage > 1) ok = __all_sync(0xffffffffu, tg_wait(&p_done[b], ((stage >> 1) & 1) ^ 1, &retention_error_flag, 1));
            if (!ok) break;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int i = threadIdx.x + j * THREADS, d = i / 16, piece = i % 16;
                float f[8] = {p[j][0].x, p[j][0].y, p[j][0].z, p[j][0].w, p[j][1].x, p[j][1].y, p[j][1].z, p[j][1].w};
                if (first + stage / HALVES * RF_SLICE + piece * 8 >= dv)
#pragma unroll
                    for (int x = 0; x < 8; ++x) f[x] = 0.f;
                odd = rf_put8(tg_smem(buf) + (uint32_t)((piece >> 3) * RF_TILE), 2 * RF_TILE, d, piece & 7, f, 0, &plain_from[stage / HALVES]) || odd;
            }
            if (stage + 1 < stages) ask_p(stage + 1);
            if (stage == HALVES - 1) rf_ask_v<T, THREADS>(vr, v, v_stride, h, dv, first, tok0, n);
            full(&p_full[b]);
            if (stage != HALVES - 1) continue;
            // beside the first slice: A's parts (a lane a token, 16 earlier tokens a warp) and the slice's values
            ok = __all_sync(0xffffffffu, tg_wait(s_done, 0, &retention_error_flag, 2));
            if (!ok) break;
            tg_after();
            if ((warp & 3) < 2) {
                const int i = (warp & 3) * 32 + lane, j0 = (warp >> 2) * 16;
                uint32_t s0[16], s1[16];
                tg_ld16(tmem + lanes + (uint32_t)j0, s0);
                if (HALVES > 1) tg_ld16(tmem + lanes + 64u + (uint32_t)j0, s1);
                tg_wait_ld();
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    float f[8];
#pragma unroll
                    for (int x = 0; x < 8; ++x) {
                        const int gap = i - (j0 + 8 * y + x);
                        const float s = __uint_as_float(s0[8 * y + x]) + (HALVES > 1 ? __uint_as_float(s1[8 * y + x]) : 0.f);
                        f[x] = gap >= 0 ? s * (S3_DOWN * S3_DOWN) * pw[gap >= 0 ? gap : 0] : 0.f;
                    }
                    if (rf_put8(tg_smem(sA), RF_TILE, i, (j0 >> 3) + y, f, i, &plain_from[2])) {
                        atomicMin(&plain_from[2], i);
                        odd = true;
                    }
                }
            }
            odd = rf_put_v<T, VP, THREADS>(tg_smem(sV), vr, dv, first, n, act, &plain_from[0]) || odd;
            if (ns > 1) rf_ask_v<T, THREADS>(vr, v, v_stride, h, dv, first + RF_SLICE, tok0, n);
            full(a_full);
        }
        if (ok) ok = __all_sync(0xffffffffu, tg_wait(v_done, 0, &retention_error_flag, 3));      // and with it all that was issued before
        tg_after();
        if (ok && ns > 1) {
            odd = rf_put_v<T, VP, THREADS>(tg_smem(sV), vr, dv, first + RF_SLICE, n, act, &plain_from[1]) || odd;
            full(v_full);
        }
        if (ok) {
            const int i0 = (warp >> 2) * 16;
            float nan = 0.f;
            for (int s = 0; s < ns && ok; ++s) {
                if (s > 0) ok = __all_sync(0xffffffffu, tg_wait(v_done, 1, &retention_error_flag, 4));
                tg_after();
                const int c = first + s * RF_SLICE + (warp & 3) * 32 + lane;
                uint32_t a[16], p0[16], p1[16];
                tg_ld16(tmem + lanes + 384u + 64u * s + (uint32_t)i0, a);
                tg_ld16(tmem + lanes + 128u + 128u * s + (uint32_t)i0, p0);
                if (HALVES > 1) tg_ld16(tmem + lanes + 192u + 128u * s + (uint32_t)i0, p1);
                tg_wait_ld();
                float* dst = out + ((size_t)(tok0 + i0) * H + h) * dv + c;
                if (c < dv && ok)
#pragma unroll
                    for (int i = 0; i < 16; ++i, dst += (size_t)H * dv)
                        if (i0 + i < n) {
                            const float far = __uint_as_float(p0[i]) + (HALVES > 1 ? __uint_as_float(p1[i]) : 0.f);
                            const float sum = fmaf(far * (S3_DOWN * S3_DOWN), pw[i0 + i + 1],
                                                   __uint_as_float(a[i]) * (VP == 1 ? S3_DOWN : S3_DOWN * S3_DOWN));
                            nan = fmaf(sum, 0.f, nan);   // 0 as long as all are finite
                            *dst = sum;
                        }
            }
            odd = odd || nan != 0.f;
        }
    }
    ok = __syncthreads_and(ok);
    odd = __syncthreads_or(odd);
    if (!ok) {                                           // products that may still be under way
        for (int x = 0; x < 8; ++x) tg_wait(&bars[x >> 1], x & 1, &retention_error_flag, 5);
    } else if (odd) {                                    // plain sums: a term past a row is not added at all
        rf_plain_outputs<T, DK>((float*)sQ, q, q_stride, k, k_stride, v, v_stride, out, H, dv, k_scale, act, rope, rot, tok0, n, h, first, ns, pw,
                                plain_from, Pc);
    }
    tg_before();
    __syncthreads();
    if (warp == 0) {
        tg_after();
        tg_free512(tmem_slot);
    }
}

template <typename T, int DK, int VP>
static int retention_tc(const T* q, long long q_stride, const T* k, long long k_stride, const T* v, long long v_stride,
                           float* out, int B, int H, int dv, const float* decay, float k_scale, int act,
                           const float* rope, int rot, const int* q_start, const int* state_slots, float* state,
                           int chunks, const int* chunk_tok0, const int* chunk_ntok, const int* chunk_first,
                           float* scratch, cudaStream_t stream) {
    constexpr size_t s1 = 1024 + (size_t)(3 * (DK / 64) + 4 * VP) * RF_TILE, s3 = 1024 + rf_out_bytes<DK>();
    static_assert(s1 >= 1024 + RC_CHUNK * RF_LOOP_LD * sizeof(float), "the plain sums' tiles");
    static_assert(s3 >= 1024 + RC_CHUNK * (2 * RF_LOOP_LD + RC_CHUNK + 1) * sizeof(float), "the plain sums' tiles");
    auto k1 = retention_summaries_tc_kernel<T, DK, VP>;
    auto k3 = retention_outputs_tc_kernel<T, DK, VP>;
    static bool sized[64] = {};                          // per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
    if (!sized[dev]) {
        if ((e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1)) != cudaSuccess) return (int)e;
        if ((e = cudaFuncSetAttribute(k3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3)) != cudaSuccess) return (int)e;
        sized[dev] = true;
    }
    // Two slices a block, which share Q's and K's parts, unless blocks of one are all on the chip at once. MEASURED, bfloat16,
    // one slice and two, us: 4 heads of 128 x 256, 1024 tokens (128 blocks of one) 21.5 and 26.6, 1536 (192) 33.5 and 27.6; 16 of
    // them, 256 tokens (128) 22.4 and 27.4, 512 (256) 35.5 and 29.3, 4096 264 and 202; 2 of 64 x 512, 1024 (128) 17.4 and 20.9,
    // 1536 (192) 25.8 and 21.8.
    const int slices = (dv + RF_SLICE - 1) / RF_SLICE, per = (long long)chunks * H * slices > tgo_multiprocessors() ? 2 : 1;
    const int z = (slices + per - 1) / per;
    int rc = tgo_launch_pdl(k1, dim3(chunks, H, z), dim3(RC_THREADS), s1, stream, k, k_stride, v, v_stride, H, dv,
                            decay, k_scale, act, rope, rot, chunk_tok0, chunk_ntok, per, scratch);
    if (rc) return rc;
    rc = tgo_launch_pdl(retention_scan4_kernel, dim3(B, H, (DK * dv / 4 + 255) / 256), dim3(256), 0, stream, H, DK * dv,
                        decay, q_start, state_slots, chunk_first, scratch, state);
    if (rc) return rc;
    return tgo_launch_pdl(k3, dim3(chunks, H, z), dim3(RF_OUT_THREADS + 32), s3, stream, q, q_stride, k, k_stride, v, v_stride, out,
                          H, dv, decay, k_scale, act, rope, rot, chunk_tok0, chunk_ntok, per, (const float*)scratch);
}

// The code a wait of the chunks' products left when it ran out (0: none did). Synchronises.
TGO_API int tgo_retention_error(int* value) { return (int)cudaMemcpyFromSymbol(value, retention_error_flag, sizeof(int)); }

static inline size_t summaries_smem(int dk) {
    return ((size_t)RC_CHUNK * (dk + 1) + (size_t)RC_CHUNK * RC_VS + RC_CHUNK + 1) * sizeof(float);
}
static inline size_t outputs_smem(int dk) {
    return ((size_t)2 * RC_CHUNK * (dk + 1) + (size_t)RC_CHUNK * (RC_CHUNK + 1) + (size_t)RC_CHUNK * RC_VS +
            (size_t)dk * RC_VS + RC_CHUNK + 1) * sizeof(float);
}

TGO_API int tgo_retention_chunk_tokens() { return RC_CHUNK; }

// 1 if the chunked kernels (and the single-token kernel) take these sizes.
TGO_API int tgo_retention_chunked_supports(int H, int dk, int dv) {
    return (H > 0 && H <= 65535 && dk > 0 && dv > 0 && outputs_smem(dk) <= 200 * 1024) ? 1 : 0;
}

template <typename T>
static int retention_chunked(const T* q, long long q_stride, const T* k, long long k_stride, const T* v,
                             long long v_stride, float* out, int B, int H, int dk, int dv, const float* decay,
                             float k_scale, int act, const float* rope, int rot, const int* q_start,
                             const int* state_slots, float* state, int chunks, const int* chunk_tok0,
                             const int* chunk_ntok, const int* chunk_first, float* scratch, int single,
                             cudaStream_t stream) {
    if (single) {
        const size_t smem = ((size_t)2 * dk + RD_THREADS) * sizeof(float);
        return tgo_launch_pdl(retention_decode_kernel<T>, dim3(B, H, (dv + 31) / 32), dim3(RD_THREADS), smem,
                              stream, q, q_stride, k, k_stride, v, v_stride, out, H, dk, dv, decay, k_scale, act,
                              rope, rot, state_slots, state);
    }
    // rows that can be read eight channels at a time, rotated halves of whole eights
    auto whole = [&](const void* p, long long stride) { return (uintptr_t)p % 16 == 0 && stride * sizeof(T) % 16 == 0; };
    if ((dk == 64 || dk == 128) && dv % 8 == 0 && rot % 16 == 0 && whole(q, q_stride) && whole(k, k_stride) &&
        whole(v, v_stride) && (uintptr_t)rope % 16 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)scratch % 16 == 0) {
#define RF_GO(DK, VP)                                                                                                \
    return retention_tc<T, DK, VP>(q, q_stride, k, k_stride, v, v_stride, out, B, H, dv, decay, k_scale, act, rope,  \
                                   rot, q_start, state_slots, state, chunks, chunk_tok0, chunk_ntok, chunk_first, scratch, stream)
        if constexpr (sizeof(T) == 2)
            if (act == 0) {
                if (dk == 128) RF_GO(128, 1);
                RF_GO(64, 1);
            }
        if (dk == 128) RF_GO(128, 3);
        RF_GO(64, 3);
#undef RF_GO
    }
    const size_t s1 = summaries_smem(dk), s3 = outputs_smem(dk);
    auto k1 = retention_summaries_kernel<T>;
    auto k3 = retention_outputs_kernel<T>;
    if (s1 > 48 * 1024) cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
    if (s3 > 48 * 1024) cudaFuncSetAttribute(k3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3);
    int rc = tgo_launch_pdl(k1, dim3(chunks, H), dim3(RC_THREADS), s1, stream, k, k_stride, v, v_stride, H, dk,
                            dv, decay, k_scale, act, rope, rot, chunk_tok0, chunk_ntok, scratch);
    if (rc) return rc;
    rc = tgo_launch_pdl(retention_scan_kernel, dim3(B, H, (dk * dv + 255) / 256), dim3(256), 0, stream, H, dk,
                        dv, decay, q_start, state_slots, chunk_first, scratch, state);
    if (rc) return rc;
    return tgo_launch_pdl(k3, dim3(chunks, H), dim3(RC_THREADS), s3, stream, q, q_stride, k, k_stride, v,
                          v_stride, out, H, dk, dv, decay, k_scale, act, rope, rot, chunk_tok0, chunk_ntok,
                          (const float*)scratch);
}

// As tgo_retention, by chunks. chunk_tok0 / chunk_ntok: the chunks (at most
// tgo_retention_chunk_tokens() tokens of one request each, a request's chunks in order and
// next to each other); chunk_first [B]: index of each request's first chunk; scratch: float32
// [chunks, H, dk, dv]. single != 0: every request brings one token (no chunk lists needed).
TGO_API int tgo_retention_chunked(const void* q, long long q_stride, const void* k, long long k_stride,
                                  const void* v, long long v_stride, int dtype, float* out, int B, int H,
                                  int dk, int dv, const float* decay, float k_scale, int act, const float* rope,
                                  int rot, const int* q_start, const int* state_slots, float* state,
                                  int chunks, const int* chunk_tok0, const int* chunk_ntok,
                                  const int* chunk_first, float* scratch, int single, cudaStream_t stream) {
    if (B <= 0) return 0;
    if (!tgo_retention_chunked_supports(H, dk, dv) || rot < 0 || rot > dk || (rot & 1) ||
        (!single && (chunks <= 0 || !chunk_tok0 || !chunk_ntok || !chunk_first || !scratch)))
        return TGO_E_BAD_ARG;
    if (dtype == TGO_BF16)
        return retention_chunked<bf16>((const bf16*)q, q_stride, (const bf16*)k, k_stride, (const bf16*)v,
                                       v_stride, out, B, H, dk, dv, decay, k_scale, act, rope, rot, q_start,
                                       state_slots, state, chunks, chunk_tok0, chunk_ntok, chunk_first, scratch,
                                       single, stream);
    if (dtype == TGO_F32)
        return retention_chunked<float>((const float*)q, q_stride, (const float*)k, k_stride, (const float*)v,
                                        v_stride, out, B, H, dk, dv, decay, k_scale, act, rope, rot, q_start,
                                        state_slots, state, chunks, chunk_tok0, chunk_ntok, chunk_first,
                                        scratch, single, stream);
    return TGO_E_BAD_ARG;
}
