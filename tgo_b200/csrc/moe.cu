// A routed feed-forward (mixture of experts): every token goes to the `top` experts with the
// largest router logits, weighted by the softmax over those logits alone.
//
//   logits     Wr x + br in float32 (Wr, br float32; x in the storage type)
//   pick       the top experts (ties: the lower index), their weights, and a count per expert
//   plan       expert e's (token, choice) pairs get places offsets[e] .. offsets[e+1]-1; the
//              places are cut into row tiles of one expert each
//              (steps of few tokens: pick, plan and scatter are one block's work)
//   scatter    pair -> place (within an expert the order is whatever the atomics give; a
//              pair's result does not depend on its place)
//   up         hidden[place] = act(x Wg_e^T) * (x Wu_e^T) for the token of the pair at `place`
//   down       y[pair] = hidden[place] Wd_e^T, float32
//   combine    out[t] = sum_j weight[t][j] y[t top + j] (+ extra[t]), j in order, all float32
//
// The products are tiled: float32 storage takes plain-FMA tiles with float32 sums over k in
// order; bfloat16 storage runs on tcgen05 (float32 accumulators in tensor memory, operands by
// TMA) when the widths are multiples of 8 (16-byte chunks), and takes the plain tiles otherwise. Either way a row's result does not depend on which tile or batch
// it falls in.
//
// Variants, each a parameter: `score_mode` 1 takes the softmax over ALL router logits; the choice
// is by that score plus a per-expert `correction`, the weights are the chosen experts' scores
// (without the correction) divided by their sum (+ 1e-20). The last router outputs past the
// `E_real` experts that have matrices are identity experts: their output is the token's input
// row itself; they get no place and no tile, the combine adds weight * x for them.
// `score_mode` 2 takes the logistic function of each logit as its score; with `groups` > 1 the
// experts are that many equal runs of neighbours, a run's strength is the sum of its two largest
// choice scores (`run_best` 2) or its largest alone (`run_best` 1), and only experts of the `keep`
// strongest runs can be chosen; without `renorm` the weights are the chosen scores themselves; `route_scale` multiplies the weights. One more
// router row after all experts (`gate_out`) gives a logistic gate per token that multiplies
// `extra` in the combine. Experts without a gate matrix (wg null) are W_down act(W_up x);
// activation 3 is the square of relu.
#include "tcgen.cuh"

#define MOE_TM 64                // rows of a tile of the plain products
#define MOE_TILE 128             // rows of one expert a planned tile holds at most
#define MOE_TN 64
#define MOE_TK 16

// ------------------------------------------------------------------------------ logits
// A block takes ML_TOK tokens and ML_EXP router rows (experts); its eight warps share the width,
// four channels a thread and 1024 a round, so that the loads of a few tokens are all in flight
// at once. A warp's 32 sums are joined by a transposing exchange (lane i ends with pair i), the
// warps' through shared memory in warp order: the order of a sum depends on the width alone.
// out [T, rows]; the last row may have no bias (the gate of a shared expert). Block 0 also zeroes
// the experts' counts.
#define ML_TOK 8
#define ML_EXP 4
template <typename T> struct Load4;
template <> struct Load4<bf16> {
    static __device__ __forceinline__ float4 get(const bf16* p) {
        const uint2 v = *(const uint2*)p;
        const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&v.x);
        const float2 b = __bfloat1622float2(*(const __nv_bfloat162*)&v.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
template <> struct Load4<float> {
    static __device__ __forceinline__ float4 get(const float* p) { return *(const float4*)p; }
};

template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
moe_logits_kernel(const T* __restrict__ x, long long x_stride, const float* __restrict__ wr,
                  const float* __restrict__ br, int Tn, int d, int rows, int E, float* __restrict__ out,
                  int* __restrict__ counts, int E_real) {
    __shared__ float s_part[8][32];
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < E_real; i += 256) counts[i] = 0;
    const int e0 = blockIdx.y * ML_EXP, t0 = blockIdx.x * ML_TOK;
    // tokens and rows past the end repeat the last one: their sums are not stored
    const T* xr[ML_TOK];
    const float* w[ML_EXP];
#pragma unroll
    for (int j = 0; j < ML_TOK; ++j) xr[j] = x + (size_t)(t0 + j < Tn ? t0 + j : Tn - 1) * x_stride;
#pragma unroll
    for (int k = 0; k < ML_EXP; ++k) w[k] = wr + (size_t)(e0 + k < rows ? e0 + k : rows - 1) * d;
    float a[32];                                         // a[4 j + k]: token j, row k
#pragma unroll
    for (int q = 0; q < 32; ++q) a[q] = 0.f;
    if (VEC) {
        for (int i = 4 * threadIdx.x; i < d; i += 1024) {
            float4 wv[ML_EXP], xv[ML_TOK];
#pragma unroll
            for (int k = 0; k < ML_EXP; ++k) wv[k] = *(const float4*)(w[k] + i);
#pragma unroll
            for (int j = 0; j < ML_TOK; ++j) xv[j] = Load4<T>::get(xr[j] + i);
#pragma unroll
            for (int j = 0; j < ML_TOK; ++j)
#pragma unroll
                for (int k = 0; k < ML_EXP; ++k) {
                    float v = a[4 * j + k];
                    v = fmaf(wv[k].x, xv[j].x, v);
                    v = fmaf(wv[k].y, xv[j].y, v);
                    v = fmaf(wv[k].z, xv[j].z, v);
                    a[4 * j + k] = fmaf(wv[k].w, xv[j].w, v);
                }
        }
    } else {
        for (int i = threadIdx.x; i < d; i += 256) {
            float wv[ML_EXP];
#pragma unroll
            for (int k = 0; k < ML_EXP; ++k) wv[k] = w[k][i];
#pragma unroll
            for (int j = 0; j < ML_TOK; ++j) {
                const float v = to_f32(xr[j][i]);
#pragma unroll
                for (int k = 0; k < ML_EXP; ++k) a[4 * j + k] = fmaf(wv[k], v, a[4 * j + k]);
            }
        }
    }
    // 32 sums over 32 lanes: with each round a lane keeps half of its values, lane i ends with sum i
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < o; ++q) {
            const float give = up ? a[q] : a[q + o], have = up ? a[q + o] : a[q];
            a[q] = have + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    s_part[warp][lane] = a[0];
    __syncthreads();
    if (warp == 0) {
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) v += s_part[q][lane];
        const int t = t0 + lane / 4, e = e0 + lane % 4;
        if (t < Tn && e < rows) out[(size_t)t * rows + e] = v + ((br && e < E) ? br[e] : 0.f);
    }
}

// -------------------------------------------------------------------------------- pick
// One warp picks one token's experts. lg [E + 1], sc [E] and gs [groups] are the warp's own
// shared memory; `z` the token's logits.
__device__ __forceinline__ void moe_pick(const float* __restrict__ z, float* lg, float* sc, float* gs,
                                         int t, int E, int top, int* __restrict__ ids,
                                         float* __restrict__ wts, int* counts, int score_mode,
                                         const float* __restrict__ correction, int E_real,
                                         float* __restrict__ gate_out, int groups, int keep, int renorm,
                                         float route_scale, int run_best) {
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < E + (gate_out ? 1 : 0); e += 32) lg[e] = z[e];
    __syncwarp();
    if (gate_out && lane == 0) gate_out[t] = 1.f / (1.f + expf(-lg[E]));
    float first = 0.f, sum = 0.f, mine = 0.f;
    int mine_e = 0;
    // the largest of n values in shared memory below `limit` and its index (ties: the lower index),
    // the same in every lane; with nothing above -inf the index is `fallback`
    auto largest = [&](const float* v, int n, int fallback, float limit, float& best) {
        float mine_v = -INFINITY;
        int be = 0x7fffffff;
        for (int e = lane; e < n; e += 32) {
            const float x = v[e];
            if (x > mine_v && x < limit) { mine_v = x; be = e; }
        }
        // a float's bits, reordered so that they compare as integers
        const unsigned raw = __float_as_uint(mine_v);
        const unsigned key = (raw & 0x80000000u) ? ~raw : raw | 0x80000000u;
        const unsigned top_key = __reduce_max_sync(0xffffffffu, key);
        best = __uint_as_float((top_key & 0x80000000u) ? top_key & 0x7fffffffu : ~top_key);
        const unsigned bi = __reduce_min_sync(0xffffffffu, key == top_key ? (unsigned)be : 0x7fffffffu);
        return (int)bi < n ? (int)bi : fallback;
    };
    if (score_mode != 0) {
        // scores: the softmax over every logit, or each logit's logistic; the choice adds the correction
        float mx = 0.f, den = 1.f;
        if (score_mode == 1) {
            mx = -INFINITY;
            for (int e = lane; e < E; e += 32) mx = fmaxf(mx, lg[e]);
            mx = warp_max(mx);
            den = 0.f;
            for (int e = lane; e < E; e += 32) {
                const float w = expf(lg[e] - mx);
                sc[e] = w;
                den += w;
            }
            den = warp_sum(den);
        }
        for (int e = lane; e < E; e += 32) {
            const float sv = score_mode == 1 ? sc[e] / den : 1.f / (1.f + expf(-lg[e]));
            sc[e] = sv;
            lg[e] = sv + (correction ? correction[e] : 0.f);
        }
        __syncwarp();
        if (groups > 1) {
            const int size = E / groups;
            for (int g = lane; g < groups; g += 32) {
                float a = -INFINITY, c = -INFINITY;      // the two largest of the run
                for (int e = g * size; e < (g + 1) * size; ++e) {
                    const float v = lg[e];
                    if (v > a) { c = a; a = v; } else if (v > c) { c = v; }
                }
                gs[g] = size > 1 && run_best > 1 ? a + c : a;
            }
            __syncwarp();
            // the weakest groups - keep runs go: mark the strongest with +inf, then close the others
            for (int j = 0; j < keep; ++j) {
                float best;
                const int bg = largest(gs, groups, groups, INFINITY, best);
                __syncwarp();                            // every lane has read gs
                if (lane == 0 && bg < groups) gs[bg] = INFINITY;
                __syncwarp();
            }
            for (int e = lane; e < E; e += 32)
                if (gs[e / size] != INFINITY) lg[e] = -INFINITY;
            __syncwarp();
        }
        for (int j = 0; j < top; ++j) {
            float best;
            const int be = largest(lg, E, j, INFINITY, best);
            const float w = sc[be];
            sum += w;
            if (lane == j) { mine = w; mine_e = be; }
            __syncwarp();                                // every lane has read lg
            if (lane == 0) lg[be] = -INFINITY;
            __syncwarp();
        }
        if (lane < top) {
            ids[(size_t)t * top + lane] = mine_e;
            wts[(size_t)t * top + lane] = (renorm ? mine / (sum + 1e-20f) : mine) * route_scale;
            if (mine_e < E_real) atomicAdd(&counts[mine_e], 1);
        }
        return;
    }
    for (int j = 0; j < top; ++j) {
        float best;
        const int be = largest(lg, E, j, INFINITY, best);
        if (j == 0) first = best;
        const float w = expf(best - first);
        sum += w;
        if (lane == j) { mine = w; mine_e = be; }
        __syncwarp();
        if (lane == 0) lg[be] = -INFINITY;
        __syncwarp();
    }
    if (lane < top) {
        ids[(size_t)t * top + lane] = mine_e;
        wts[(size_t)t * top + lane] = mine / sum * route_scale;
        if (mine_e < E_real) atomicAdd(&counts[mine_e], 1);
    }
}

#define MOE_PW 4
__global__ void __launch_bounds__(32 * MOE_PW)
moe_pick_kernel(const float* __restrict__ logits, int rows, int Tn, int E, int top, int* __restrict__ ids,
                float* __restrict__ wts, int* __restrict__ counts, int score_mode,
                const float* __restrict__ correction, int E_real, float* __restrict__ gate_out, int groups,
                int keep, int renorm, float route_scale, int run_best) {
    extern __shared__ float smem[];                      // [MOE_PW][2 E + 1 + groups]
    pdl_wait();
    const int warp = threadIdx.x >> 5, t = blockIdx.x * MOE_PW + warp;
    if (t >= Tn) return;
    float* lg = smem + (size_t)warp * (2 * E + 1 + groups);
    moe_pick(logits + (size_t)t * rows, lg, lg + E + 1, lg + 2 * E + 1, t, E, top, ids, wts, counts, score_mode,
             correction, E_real, gate_out, groups, keep, renorm, route_scale, run_best);
}

// -------------------------------------------------------------------------------- plan
// One warp: offsets [E + 1], tiles (expert, first place, rows) and their count in tile_info[0]; the
// fill counters go back to zero. A lane takes a run of experts, the places and tiles before it by
// a running sum over the lanes.
__device__ __forceinline__ void moe_plan(const int* counts, int E, int* __restrict__ offsets, int* fill,
                                         int* __restrict__ tile_info, int* __restrict__ tiles, int max_tiles) {
    const int lane = threadIdx.x & 31, per = (E + 31) / 32;
    const int e_lo = lane * per < E ? lane * per : E, e_hi = e_lo + per < E ? e_lo + per : E;
    int c = 0, nt = 0;
    for (int e = e_lo; e < e_hi; ++e) {
        c += counts[e];
        nt += (counts[e] + MOE_TILE - 1) / MOE_TILE;
    }
    int at = c, tile = nt;                               // inclusive sums over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, at, o), b = __shfl_up_sync(0xffffffffu, tile, o);
        if (lane >= o) { at += a; tile += b; }
    }
    if (lane == 31) {
        offsets[E] = at;
        tile_info[0] = tile < max_tiles ? tile : max_tiles;
    }
    at -= c;
    tile -= nt;
    for (int e = e_lo; e < e_hi; ++e) {
        const int n = counts[e];
        offsets[e] = at;
        fill[e] = 0;
        for (int r = 0; r < n; r += MOE_TILE, ++tile) {
            if (tile >= max_tiles) break;
            tiles[3 * tile] = e;
            tiles[3 * tile + 1] = at + r;
            tiles[3 * tile + 2] = n - r < MOE_TILE ? n - r : MOE_TILE;
        }
        at += n;
    }
}

__global__ void __launch_bounds__(32)
moe_plan_kernel(const int* __restrict__ counts, int E, int* __restrict__ offsets, int* __restrict__ fill,
                int* __restrict__ tile_info, int* __restrict__ tiles, int max_tiles) {
    pdl_wait();
    moe_plan(counts, E, offsets, fill, tile_info, tiles, max_tiles);
}

// A step of few tokens: pick, plan and scatter by one block, the counts and fill counters in
// shared memory.
#define MOE_FEW_WARPS 32
__global__ void __launch_bounds__(32 * MOE_FEW_WARPS)
moe_route_few_kernel(const float* __restrict__ logits, int rows, int Tn, int E, int top, int* __restrict__ ids,
                     float* __restrict__ wts, int score_mode, const float* __restrict__ correction, int E_real,
                     float* __restrict__ gate_out, int groups, int keep, int renorm, float route_scale,
                     int run_best, int* __restrict__ offsets, int* __restrict__ perm, int* __restrict__ place,
                     int* __restrict__ tile_info, int* __restrict__ tiles, int max_tiles) {
    extern __shared__ float smem[];                      // [warps][2 E + 1 + groups], counts, fill
    const int per = 2 * E + 1 + groups;
    int* counts = (int*)(smem + (size_t)MOE_FEW_WARPS * per);
    int* fill = counts + E_real;
    const int warp = threadIdx.x >> 5, n = 32 * MOE_FEW_WARPS;
    for (int i = threadIdx.x; i < E_real; i += n) counts[i] = 0;
    pdl_wait();
    __syncthreads();
    float* lg = smem + (size_t)warp * per;
    for (int t = warp; t < Tn; t += MOE_FEW_WARPS) {
        moe_pick(logits + (size_t)t * rows, lg, lg + E + 1, lg + 2 * E + 1, t, E, top, ids, wts, counts, score_mode,
                 correction, E_real, gate_out, groups, keep, renorm, route_scale, run_best);
        __syncwarp();
    }
    __syncthreads();                                     // ids are in memory for the whole block
    if (warp == 0) moe_plan(counts, E_real, offsets, fill, tile_info, tiles, max_tiles);
    __syncthreads();
    for (int p = threadIdx.x; p < Tn * top; p += n) {
        const int e = ids[p];
        if (e >= E_real) { place[p] = -1; continue; }
        const int at = offsets[e] + atomicAdd(&fill[e], 1);
        perm[at] = p;
        place[p] = at;
    }
}

__global__ void moe_scatter_kernel(const int* __restrict__ ids, int pairs,
                                   const int* __restrict__ offsets, int* __restrict__ fill,
                                   int* __restrict__ perm, int* __restrict__ place, int E_real) {
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pairs) return;
    const int e = ids[p];
    if (e >= E_real) { place[p] = -1; return; }          // an identity expert: no matrices, no place
    const int at = offsets[e] + atomicAdd(&fill[e], 1);
    perm[at] = p;
    place[p] = at;
}

// ----------------------------------------------------------------------------- products
__device__ __forceinline__ float moe_act(float z, int act) {
    if (act == 1) return z > 0.f ? z : 0.f;
    if (act == 3) return z > 0.f ? z * z : 0.f;
    if (act == 2) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return z / (1.f + expf(-z));
}

// hidden[place][f] = act(x_tok . Wg[e][f]) * (x_tok . Wu[e][f]); Wg, Wu [E, ff, d]. Without a
// gate matrix (wg null): act(x_tok . Wu[e][f]).
template <typename T>
__global__ void __launch_bounds__(256)
moe_up_kernel(const T* __restrict__ x, long long x_stride, const T* __restrict__ wg,
              const T* __restrict__ wu, T* __restrict__ hidden, int d, int ff, int top, int act,
              const int* __restrict__ perm, const int* __restrict__ tile_info,
              const int* __restrict__ tiles) {
    __shared__ float xs[MOE_TK][MOE_TM + 4];
    __shared__ float gs[MOE_TK][MOE_TN + 4];
    __shared__ float us[MOE_TK][MOE_TN + 4];
    __shared__ int toks[MOE_TM];
    pdl_wait();
    if ((int)blockIdx.y >= tile_info[0]) return;
    const int e = tiles[3 * blockIdx.y], skip = MOE_TM * blockIdx.z;     // z: which half of the planned tile
    const int r0 = tiles[3 * blockIdx.y + 1] + skip, rows = min(tiles[3 * blockIdx.y + 2] - skip, MOE_TM);
    if (rows <= 0) return;
    const int n0 = blockIdx.x * MOE_TN;
    if (threadIdx.x < MOE_TM) toks[threadIdx.x] = threadIdx.x < rows ? perm[r0 + threadIdx.x] / top : -1;
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const T* wge = wg + (size_t)e * ff * d;
    const T* wue = wu + (size_t)e * ff * d;
    float ag[4][4], au[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ag[i][j] = au[i][j] = 0.f;
    for (int k0 = 0; k0 < d; k0 += MOE_TK) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int idx = threadIdx.x + r * 256;
            const int row = idx / MOE_TK, kk = idx % MOE_TK;
            const int gk = k0 + kk, gn = n0 + row;
            const int tok = toks[row];
            xs[kk][row] = (tok >= 0 && gk < d) ? to_f32(x[(size_t)tok * x_stride + gk]) : 0.f;
            const bool in = gn < ff && gk < d;
            gs[kk][row] = (in && wg) ? to_f32(wge[(size_t)gn * d + gk]) : 0.f;
            us[kk][row] = in ? to_f32(wue[(size_t)gn * d + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < MOE_TK; ++kk) {
            float a[4], g[4], u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) { g[j] = gs[kk][tx * 4 + j]; u[j] = us[kk][tx * 4 + j]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    ag[i][j] = fmaf(a[i], g[j], ag[i][j]);
                    au[i][j] = fmaf(a[i], u[j], au[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = ty * 4 + i;
        if (row >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < ff)
                hidden[(size_t)(r0 + row) * ff + gn] =
                    from_f32<T>(wg ? moe_act(ag[i][j], act) * au[i][j] : moe_act(au[i][j], act));
        }
    }
}

// y[pair][n] = hidden[place] . Wd[e][n]; Wd [E, d, ff]; y float32 [pairs, d].
template <typename T>
__global__ void __launch_bounds__(256)
moe_down_kernel(const T* __restrict__ hidden, const T* __restrict__ wd, float* __restrict__ y, int d,
                int ff, const int* __restrict__ perm, const int* __restrict__ tile_info,
                const int* __restrict__ tiles) {
    __shared__ float hs[MOE_TK][MOE_TM + 4];
    __shared__ float ws[MOE_TK][MOE_TN + 4];
    pdl_wait();
    if ((int)blockIdx.y >= tile_info[0]) return;
    const int e = tiles[3 * blockIdx.y], skip = MOE_TM * blockIdx.z;     // z: which half of the planned tile
    const int r0 = tiles[3 * blockIdx.y + 1] + skip, rows = min(tiles[3 * blockIdx.y + 2] - skip, MOE_TM);
    if (rows <= 0) return;
    const int n0 = blockIdx.x * MOE_TN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const T* wde = wd + (size_t)e * d * ff;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < ff; k0 += MOE_TK) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int idx = threadIdx.x + r * 256;
            const int row = idx / MOE_TK, kk = idx % MOE_TK;
            const int gk = k0 + kk, gn = n0 + row;
            hs[kk][row] = (row < rows && gk < ff) ? to_f32(hidden[(size_t)(r0 + row) * ff + gk]) : 0.f;
            ws[kk][row] = (gn < d && gk < ff) ? to_f32(wde[(size_t)gn * ff + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < MOE_TK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = hs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = ty * 4 + i;
        if (row >= rows) continue;
        const int pair = perm[r0 + row];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < d) y[(size_t)pair * d + gn] = acc[i][j];
        }
    }
}

// ------------------------------------------------------------- products on the tensor cores
// Persistent: one CTA an SM walks (planned tile, column tile) items, columns fastest, so that the
// tiles of one expert run at the same time and its matrices come from memory once. MODE 1: A rows
// are x rows gathered by token, B is Wg[e] and Wu[e] side by side ([N, K] each, bn rows of both
// make one operand of 2 bn columns), the result act(gate) * up goes to hidden[place] in bfloat16.
// MODE 2: the form without a gate, B is Wu[e] alone and the result act(up). MODE 0: A rows are
// hidden[place], B is Wd[e], the result goes to y[pair] in float32.
//   warps 0, 6  TMA into a ring of stages. Warp 6: the B boxes. Warp 0: A, a box for a whole tile
//               or boxes of 32 rows where its rows lie in place order, else a lane four rows (gather4); rows
//               past a part tile's are not fetched, their sums are never stored;
//   warp 1      issues the products (a thread), 128 x n x 16 each, into two accumulators in turn;
//   warps 2..5  accumulator -> activation -> staged, so that a store covers whole 64- or 128-byte
//               pieces of rows, while the next item's products run.
// Bound by the weights' way from memory for a few rows an expert (each read once; a stage is
// 32 KB of them, four in flight an SM) and by the operands' way into the SM (about 70 bytes a
// cycle) for full tiles. MEASURED (B200, 32 experts, top 4, ff 768 of width 2048, gated; mma.sync
// tiles of 64 x 64 fed by cp.async before): 2048 tokens, up 76 us (250; 91 with one warp to ask for all) and down 40
// (135), 680 and 640 TFLOP/s with the copy of x's rows before them 8 us; 64 tokens, from a flushed L2, 48 us (71)
// and 24 (25), 4.2 TB/s of weights.
#define MT_BK 64
#define MT_A_BYTES (MOE_TILE * MT_BK * 2)
#define MT_RING (192 * 1024)
#define MT_STAGE_OUT 4096                  // per epilogue warp: 32 rows x 128 bytes on their way out
#define MT_SMEM (MT_RING + 4 * MT_STAGE_OUT + 1024 + 256)
#define MT_THREADS 224

__device__ int moe_error_flag = 0;

// act of the products' results. SiLU as z / (1 + e^-z) for z >= 0 and z e^z / (1 + e^z) below, so that the
// divisor lies in [1, 2] and the quotient needs no scaling: the hardware's reciprocal and one correction by the
// remainder. (With a plain division, whose rare cases are a branch an element, the up product of 64 tokens
// took 64 us instead of 51, that of 2048 103 instead of 90.)
__device__ __forceinline__ float moe_act_tile(float z, int act) {
    if (act != 0) return moe_act(z, act);
    const float e = expf(-fabsf(z)), d = 1.f + e, n = z >= 0.f ? z : z * e;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = n * r;
    return z < __int_as_float(0x7f800000) ? fmaf(fmaf(-q, d, n), r, q) : z;
}

template <int MODE>
__global__ void __launch_bounds__(MT_THREADS, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_tile, const __grid_constant__ CUtensorMap map_b0,
              const __grid_constant__ CUtensorMap map_b1, bf16* __restrict__ hidden, float* __restrict__ y, int N,
              int K, int bn, int top, int act, int gather, const int* __restrict__ perm,
              const int* __restrict__ tile_info, const int* __restrict__ tiles) {
    constexpr bool UP = MODE != 0, GATED = MODE == 1;
    const int nm = GATED ? 2 * bn : bn;                        // columns of a product
    const int stage_bytes = MT_A_BYTES + nm * MT_BK * 2;
    const int stages = min(MT_RING / stage_bytes, 8);
    extern __shared__ unsigned char moe_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)moe_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* out_stage = base + MT_RING;                 // [4][MT_STAGE_OUT]
    uint64_t* full = (uint64_t*)(out_stage + 4 * MT_STAGE_OUT);
    uint64_t* empty = full + 8;
    uint64_t* acc_full = empty + 8;                            // [2]
    uint64_t* acc_empty = acc_full + 2;                        // [2]
    uint64_t* settled = acc_empty + 2;                         // after a wait ran out
    uint32_t* tmem_slot = (uint32_t*)(settled + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; ++i) { tg_init(&full[i], 2); tg_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { tg_init(&acc_full[i], 1); tg_init(&acc_empty[i], 4); }
        tg_init(settled, 1);
        tg_init_done();
    }
    if (warp == 1) tg_alloc512(tmem_slot);
    tg_before();
    __syncthreads();
    tg_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    const int n_nt = (N + bn - 1) / bn, total = tile_info[0] * n_nt, kbs = (K + MT_BK - 1) / MT_BK;

    if (warp == 0 || warp == 6) {
        // ---- rows (warp 0) and matrices (warp 6): a warp starts a copy about every 80 cycles
        uint32_t it = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
            const int tile = w / n_nt, n0 = (w % n_nt) * bn;
            const int e = tiles[3 * tile], r0 = tiles[3 * tile + 1], rows = tiles[3 * tile + 2];
            // more than three boxes of 32 rows come as one of 128: the rows after an expert's are the next one's, whose
            // sums nobody stores
            const bool whole = !gather && rows > 96;
            int src[4] = {0, 0, 0, 0};
            if (gather && warp == 0)
#pragma unroll
                for (int j = 0; j < 4; ++j) src[j] = perm[r0 + min(4 * lane + j, rows - 1)] / top;
            const int groups = gather ? (rows + 3) / 4 : whole ? 1 : (rows + 31) / 32, group_bytes = gather ? 512 : whole ? MT_A_BYTES : 4096;
            for (int kb = 0; kb < kbs; ++kb, ++it) {
                const int s = it % stages;
                ok = __all_sync(0xffffffffu, tg_wait(&empty[s], ((it / stages) & 1) ^ 1, &moe_error_flag, 1));
                if (!ok) break;
                unsigned char* st = base + (size_t)s * stage_bytes;
                if (warp == 6) {
                    if (lane == 0) {
                        tg_expect(&full[s], (uint32_t)(nm * MT_BK * 2));
                        tg_load_2d(st + MT_A_BYTES, &map_b0, kb * MT_BK, e * N + n0, &full[s]);
                        if (GATED) tg_load_2d(st + MT_A_BYTES + bn * MT_BK * 2, &map_b1, kb * MT_BK, e * N + n0, &full[s]);
                    }
                    __syncwarp();
                    continue;
                }
                if (lane == 0) tg_expect(&full[s], (uint32_t)(groups * group_bytes));
                __syncwarp();
                if (whole) {
                    if (lane == 0) tg_load_2d(st, &map_tile, kb * MT_BK, r0, &full[s]);
                } else if (!gather) {
                    if (lane < groups) tg_load_2d(st + lane * 4096, &map_a, kb * MT_BK, r0 + 32 * lane, &full[s]);
                } else if (lane < groups) {
                    tg_gather4(st + lane * 512, &map_a, kb * MT_BK, src[0], src[1], src[2], src[3], &full[s]);
                }
            }
        }
        if (!ok) tg_settle_copies(full, stages, it, &moe_error_flag, 1);
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tg_idesc(nm);
            uint32_t it = 0, n = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x, ++n) {
                const uint32_t buf = n & 1u, d = tmem + 256u * buf;
                ok = tg_wait(&acc_empty[buf], ((n >> 1) & 1u) ^ 1u, &moe_error_flag, 2);
                if (!ok) break;
                tg_after();
                for (int kb = 0; kb < kbs; ++kb, ++it) {
                    const int s = it % stages;
                    ok = tg_wait(&full[s], (it / stages) & 1, &moe_error_flag, 3);
                    if (!ok) break;
                    tg_after();
                    unsigned char* st = base + (size_t)s * stage_bytes;
                    const uint64_t da = tg_desc(st), db = tg_desc(st + MT_A_BYTES);
#pragma unroll
                    for (int k = 0; k < MT_BK / 16; ++k) tg_mma(d, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tg_commit(&empty[s]);
                }
                tg_commit(&acc_full[buf]);
            }
            if (!ok) tg_settle_products(settled, &moe_error_flag, 3);
        }
    } else {
        const int quarter = warp & 3;                          // tensor-memory lanes this warp may read
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t stage = tg_smem(out_stage + (warp - 2) * MT_STAGE_OUT);
        uint32_t n = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok; w += gridDim.x, ++n) {
            const int tile = w / n_nt, n0 = (w % n_nt) * bn;
            const int r0 = tiles[3 * tile + 1], rows = tiles[3 * tile + 2];
            const int pair = !UP && row < rows ? perm[r0 + row] : 0;
            const uint32_t buf = n & 1u, acc = tmem + 256u * buf + lane_base;
            ok = __all_sync(0xffffffffu, tg_wait(&acc_full[buf], (n >> 1) & 1u, &moe_error_flag, 4));
            tg_after();
            const bool any = ok && quarter * 32 < rows;        // the same for the whole warp
            for (int c = 0; any && c < bn && n0 + c < N; c += 32) {
                uint32_t a[32];
                tg_ld32(acc + c, a);
                if (UP) {
                    uint32_t u[GATED ? 32 : 1];
                    if constexpr (GATED) tg_ld32(acc + bn + c, u);
                    tg_wait_ld();
                    float v[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        v[i] = moe_act_tile(__uint_as_float(a[i]), act) * (GATED ? __uint_as_float(u[GATED ? i : 0]) : 1.f);
                    // 64 bytes a row, pieces of 16 shifted by row so that neither side meets a bank twice
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(stage + (uint32_t)(lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4))),
                                     "r"(tg_pack(v[8 * q], v[8 * q + 1])), "r"(tg_pack(v[8 * q + 2], v[8 * q + 3])),
                                     "r"(tg_pack(v[8 * q + 4], v[8 * q + 5])), "r"(tg_pack(v[8 * q + 6], v[8 * q + 7])) : "memory");
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int r = i * 8 + (lane >> 2), q = lane & 3;
                        uint4 x;
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                                     : "r"(stage + (uint32_t)(r * 64 + ((q ^ ((r >> 1) & 3)) << 4))) : "memory");
                        if (quarter * 32 + r < rows && n0 + c + q * 8 < N)
                            *(uint4*)(hidden + (size_t)(r0 + quarter * 32 + r) * N + n0 + c + q * 8) = x;
                    }
                } else {
                    tg_wait_ld();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(stage + (uint32_t)(lane * 128 + ((q ^ (lane & 7)) << 4))),
                                     "r"(a[4 * q]), "r"(a[4 * q + 1]), "r"(a[4 * q + 2]), "r"(a[4 * q + 3]) : "memory");
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = i * 4 + (lane >> 3), q = lane & 7;
                        uint4 x;
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                                     : "r"(stage + (uint32_t)(r * 128 + ((q ^ (r & 7)) << 4))) : "memory");
                        const int to = __shfl_sync(0xffffffffu, pair, r);
                        if (quarter * 32 + r < rows && n0 + c + q * 4 < N) *(uint4*)(y + (size_t)to * N + n0 + c + q * 4) = x;
                    }
                }
                __syncwarp();
            }
            tg_before();
            __syncwarp();
            if (lane == 0) tg_arrive(&acc_empty[buf]);
        }
    }
    tg_before();
    __syncthreads();
    if (warp == 1) {
        tg_after();
        tg_free512(tmem);
    }
}

// xg[place] = x[token of the pair at `place`]: a block a place, 16 bytes a thread and turn.
__global__ void __launch_bounds__(128)
moe_gather_kernel(const bf16* __restrict__ x, long long x_stride, bf16* __restrict__ xg, int d, int top, int E,
                  const int* __restrict__ perm, const int* __restrict__ offsets) {
    pdl_wait();
    if ((int)blockIdx.x >= offsets[E]) return;           // identity experts' pairs have no place
    const uint4* src = (const uint4*)(x + (size_t)(perm[blockIdx.x] / top) * x_stride);
    uint4* dst = (uint4*)(xg + (size_t)blockIdx.x * d);
    for (int c = threadIdx.x; c < d / 8; c += 128) dst[c] = src[c];
}

// The column tile: a round of items costs its k-blocks at the slower of their products (2 cycles a
// column) and of their bytes (70 a cycle) and 200 cycles each, and about 1500 cycles; the number of planned
// tiles is the device's to know, `m_est` what evenly spread tokens would make. MEASURED (B200, 104 sizes: 8
// shapes of experts, 1 to 2048 tokens, every width): the widths picked are 2.6 % behind the best. Without
// the cycles a k-block, rounding to whole rounds picked 32 columns for 16 experts of 1536 x 4096 and 8 to 64
// tokens: 108 to 173 us where 96 columns take 81 to 85 (mma.sync tiles: 82 to 131).
static int moe_tc_width(int N, int K, int E, int pairs, bool gated, int sms) {
    const int per = pairs / E;
    const double m_est = pairs <= E ? pairs : per < 128 ? E : E * ((per + 64) / 128 + 0.5);
    const double a_bytes = (per < 1 ? 4.0 : per < 128 ? per : 128.0) * 128.0;
    const int f = gated ? 2 : 1, kbs = (K + MT_BK - 1) / MT_BK;
    double best = -1.0;
    int bn = 32;
    for (int w = 256 / f; w >= 32; w -= 32) {
        const double items = m_est * ((N + w - 1) / w);
        const double math = 2.0 * w * f, feed = (a_bytes + 128.0 * w * f) / 70.0;
        const double rounds = items <= sms ? 1.0 : items > 4.0 * sms ? items / sms : (double)(long long)(items / sms + 0.999);
        const double cost = rounds * (kbs * (200.0 + (math > feed ? math : feed)) + 1500.0);
        if (best < 0 || cost < best) { best = cost; bn = w; }
    }
    return bn;
}

// The rule itself: columns of a tile of products with E experts' matrices [N, K] (gated: two of them).
TGO_API int tgo_moe_tile_width(int N, int K, int E, int pairs, int gated, int sms) {
    return N > 0 && K > 0 && E > 0 && sms > 0 ? moe_tc_width(N, K, E, pairs, gated != 0, sms) : 0;
}

template <int MODE>
static int moe_tc_launch(const void* a, long long a_rows, long long a_stride, const void* b0, const void* b1, void* hidden,
                         float* y, int N, int K, int E, int pairs, int top, int act, bool gather,
                         const int* perm, const int* tile_info, const int* tiles, cudaStream_t stream) {
    static bool sized[64] = {};                                // per device
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return (int)err;
    if (dev < 0 || dev >= 64 || (long long)E * N > 0x7fffffffll) return TGO_E_BAD_ARG;
    if (!sized[dev]) {
        err = cudaFuncSetAttribute(moe_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM);
        if (err != cudaSuccess) return (int)err;
        sized[dev] = true;
    }
    const int bn = moe_tc_width(N, K, E, pairs, MODE == 1, tgo_multiprocessors());
    CUtensorMap ma, mt, m0, m1;
    if (!tg_map(&ma, a, a_rows, K, a_stride, gather ? 1 : 32) || !tg_map(&mt, a, a_rows, K, a_stride, MOE_TILE) || !tg_map(&m0, b0, (long long)E * N, K, K, bn) ||
        !tg_map(&m1, b1 ? b1 : b0, (long long)E * N, K, K, bn))
        return TGO_E_BAD_ARG;
    return tgo_launch_pdl(moe_tc_kernel<MODE>, dim3(tgo_multiprocessors()), dim3(MT_THREADS), MT_SMEM, stream, ma, mt, m0, m1, (bf16*)hidden, y,
                          N, K, bn, top, act, gather ? 1 : 0, perm, tile_info, tiles);
}

// out[t][c] = sum_j wts[t][j] y[t top + j][c] + extra_gate[t] * extra[t][c]; a pair whose
// expert is an identity expert (ids >= E_real; `ids` null: there are none) contributes
// wts * x[t][c] instead. `beside` [T, d] (TB: float32 or bfloat16; null: none) is added too, and
// with `accumulate` (float32 out) the whole is added to out: a block whose mixer and feed-forward read the
// same rows has both results put into the stream by this one pass.
template <typename T, typename TB, typename TO>
__global__ void moe_combine_kernel(const float* __restrict__ y, const float* __restrict__ wts,
                                   const float* __restrict__ extra, TO* __restrict__ out, int d,
                                   int top, const int* __restrict__ ids, int E_real,
                                   const T* __restrict__ x, long long x_stride,
                                   const float* __restrict__ extra_gate,
                                   const TB* __restrict__ beside, int accumulate, int vec) {
    pdl_wait();
    const int t = blockIdx.x;
    const float eg = extra_gate ? extra_gate[t] : 1.f;
    if (vec) {                                           // four columns a thread
        for (int c = 4 * (blockIdx.y * blockDim.x + threadIdx.x); c < d; c += 4 * blockDim.x * gridDim.y) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 ex = extra ? *(const float4*)(extra + (size_t)t * d + c) : a;
            const float4 bs = beside ? Load4<TB>::get(beside + (size_t)t * d + c) : a;
            const float4 o = accumulate ? *(const float4*)((const float*)out + (size_t)t * d + c) : a;
#pragma unroll 4
            for (int j = 0; j < top; ++j) {
                const size_t pair = (size_t)t * top + j;
                const float w = wts[pair];
                const float4 v = (ids && ids[pair] >= E_real) ? Load4<T>::get(x + (size_t)t * x_stride + c)
                                                              : *(const float4*)(y + pair * d + c);
                a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y);
                a.z = fmaf(w, v.z, a.z); a.w = fmaf(w, v.w, a.w);
            }
            if (extra) {
                a.x = fmaf(eg, ex.x, a.x); a.y = fmaf(eg, ex.y, a.y);
                a.z = fmaf(eg, ex.z, a.z); a.w = fmaf(eg, ex.w, a.w);
            }
            if (beside) { a.x += bs.x; a.y += bs.y; a.z += bs.z; a.w += bs.w; }
            if (accumulate) { a.x += o.x; a.y += o.y; a.z += o.z; a.w += o.w; }
            if constexpr (sizeof(TO) == 4) *(float4*)(out + (size_t)t * d + c) = a;
            else *(uint2*)(out + (size_t)t * d + c) = make_uint2(tg_pack(a.x, a.y), tg_pack(a.z, a.w));
        }
        return;
    }
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < d; c += blockDim.x * gridDim.y) {
        float a = 0.f;
        for (int j = 0; j < top; ++j) {
            const size_t pair = (size_t)t * top + j;
            const float v = (ids && ids[pair] >= E_real) ? to_f32(x[(size_t)t * x_stride + c]) : y[pair * d + c];
            a = fmaf(wts[pair], v, a);
        }
        if (extra) a = fmaf(eg, extra[(size_t)t * d + c], a);
        if (beside) a += to_f32(beside[(size_t)t * d + c]);
        if (accumulate) a += to_f32(out[(size_t)t * d + c]);
        out[(size_t)t * d + c] = from_f32<TO>(a);
    }
}

TGO_API int tgo_moe_tile_rows() { return MOE_TILE; }

// Reads (and waits for the device to reach) the code a wait that ran out left; 0: none did.
TGO_API int tgo_moe_error(int* value) { return (int)cudaMemcpyFromSymbol(value, moe_error_flag, sizeof(int)); }

// ids, place int32 [T top]; wts float32 [T top]; logits float32 [T, router rows]; counts, fill
// int32 [E]; offsets int32 [E + 1]; perm int32 [T top]; tile_info int32 [1]; tiles int32
// [3 max_tiles].
#define MOE_FEW_TOKENS 128
TGO_API int tgo_moe_route(const void* x, long long x_stride, int dtype, const float* wr,
                          const float* br, int T, int d, int E, int top, float* logits, int* ids, float* wts,
                          int* counts, int* fill, int* offsets, int* perm, int* place,
                          int* tile_info, int* tiles, int max_tiles, int score_mode,
                          const float* correction, int E_real, float* gate_out, int groups, int keep,
                          int renorm, float route_scale, int run_best, int* launches, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (d <= 0 || E <= 0 || E > 2048 || top <= 0 || top > 32 || top > E || max_tiles <= 0 ||
        E_real < 0 || E_real > E || score_mode < 0 || score_mode > 2 || groups < 1 || E % groups ||
        keep < 1 || keep > groups || (long long)keep * (E / groups) < top || (groups > 1 && score_mode == 0) ||
        run_best < 1 || run_best > 2 || (dtype != TGO_BF16 && dtype != TGO_F32))
        return TGO_E_BAD_ARG;
    const int rows = E + (gate_out ? 1 : 0);
    const dim3 lgrid((T + ML_TOK - 1) / ML_TOK, (rows + ML_EXP - 1) / ML_EXP);
    const bool vec = d % 4 == 0 && x_stride % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)wr % 16 == 0;
#define LOGITS_GO(TT, V)                                                                                    \
    tgo_launch_pdl(moe_logits_kernel<TT, V>, lgrid, dim3(256), 0, stream, (const TT*)x, x_stride, wr, br, T, d, \
                   rows, E, logits, counts, E_real)
    int rc = dtype == TGO_BF16 ? (vec ? LOGITS_GO(bf16, true) : LOGITS_GO(bf16, false))
                               : (vec ? LOGITS_GO(float, true) : LOGITS_GO(float, false));
#undef LOGITS_GO
    if (rc) return rc;
    const size_t per = (size_t)(2 * E + 1 + groups) * sizeof(float);
    const size_t few = MOE_FEW_WARPS * per + (size_t)2 * E_real * sizeof(int);
    if (T <= MOE_FEW_TOKENS && few <= 200 * 1024) {
        if (few > 48 * 1024)
            cudaFuncSetAttribute(moe_route_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few);
        *launches = 2;
        return tgo_launch_pdl(moe_route_few_kernel, dim3(1), dim3(32 * MOE_FEW_WARPS), few, stream,
                              (const float*)logits, rows, T, E, top, ids, wts, score_mode, correction, E_real,
                              gate_out, groups, keep, renorm, route_scale, run_best, offsets, perm, place, tile_info,
                              tiles, max_tiles);
    }
    *launches = 4;
    const size_t smem = MOE_PW * per;
    if (smem > 48 * 1024)                                // more than about 1000 router outputs
        cudaFuncSetAttribute(moe_pick_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    rc = tgo_launch_pdl(moe_pick_kernel, dim3((T + MOE_PW - 1) / MOE_PW), dim3(32 * MOE_PW), smem, stream,
                        (const float*)logits, rows, T, E, top, ids, wts, counts, score_mode, correction, E_real,
                        gate_out, groups, keep, renorm, route_scale, run_best);
    if (rc) return rc;
    rc = tgo_launch_pdl(moe_plan_kernel, dim3(1), dim3(32), 0, stream, (const int*)counts, E_real, offsets, fill,
                        tile_info, tiles, max_tiles);
    if (rc) return rc;
    const int pairs = T * top;
    return tgo_launch_pdl(moe_scatter_kernel, dim3((pairs + 255) / 256), dim3(256), 0, stream,
                          (const int*)ids, pairs, (const int*)offsets, fill, perm, place, E_real);
}

// x [T, d] rows (stride x_stride); wg, wu [E, ff, d]; wd [E, d, ff]; hidden [T top, ff] in the
// storage type; y float32 [T top, d]; extra float32 [T, d] or null; out [T, d], float32 or (no
// accumulation) bfloat16. xg: null, or
// [T top, d] in the storage type, 16-byte aligned: room for the rows of x in place order.
TGO_API int tgo_moe_experts(const void* x, long long x_stride, int dtype, const void* wg,
                            const void* wu, const void* wd, void* hidden, float* y,
                            const float* wts, const float* extra, void* out, int T, int d, int ff,
                            int top, int act, const int* perm, const int* offsets, void* xg, const int* tile_info,
                            const int* tiles, int max_tiles, const int* ids, int E_real,
                            const float* extra_gate, const void* beside, int beside_dtype,
                            int accumulate, int out_dtype, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (d <= 0 || ff <= 0 || top <= 0 || max_tiles <= 0 || max_tiles > 65535 || act < 0 || act > 3)
        return TGO_E_BAD_ARG;
    const int comb_vec = d % 4 == 0 && x_stride % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0 &&
                         (uintptr_t)extra % 16 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)beside % 16 == 0;
    const int comb_y = comb_vec && d > 512 ? (d / 512 < 16 ? d / 512 : 16) : 1;
    if ((beside && beside_dtype != TGO_F32 && beside_dtype != TGO_BF16) ||
        (out_dtype != TGO_F32 && (out_dtype != TGO_BF16 || accumulate)))
        return TGO_E_BAD_ARG;
#define MOE_COMBINE_OF(TT, TB, TO)                                                                         \
    tgo_launch_pdl(moe_combine_kernel<TT, TB, TO>, dim3(T, comb_y), dim3(128), 0, stream, (const float*)y, wts, extra,  \
                   (TO*)out, d, top, ids, E_real, (const TT*)x, x_stride, extra_gate, (const TB*)beside, accumulate,     \
                   comb_vec)
#define MOE_COMBINE(TT)                                                                                               \
    (out_dtype == TGO_BF16 ? (beside && beside_dtype == TGO_BF16 ? MOE_COMBINE_OF(TT, bf16, bf16) : MOE_COMBINE_OF(TT, float, bf16)) \
                           : beside && beside_dtype == TGO_BF16 ? MOE_COMBINE_OF(TT, bf16, float) : MOE_COMBINE_OF(TT, float, float))
    const dim3 g1((ff + MOE_TN - 1) / MOE_TN, max_tiles, MOE_TILE / MOE_TM), g2((d + MOE_TN - 1) / MOE_TN, max_tiles, MOE_TILE / MOE_TM);
    int rc;
    const bool chunks = d % 8 == 0 && ff % 8 == 0 && x_stride % 8 == 0 && (uintptr_t)x % 16 == 0 &&
                        (uintptr_t)wg % 16 == 0 && (uintptr_t)wu % 16 == 0 && (uintptr_t)wd % 16 == 0 &&
                        (uintptr_t)hidden % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)xg % 16 == 0 && E_real > 0;
    if (dtype == TGO_BF16 && chunks) {
        const int pairs = T * top;
        const void* a = x;
        long long a_rows = T, a_stride = x_stride;
        if (xg) {
            rc = tgo_launch_pdl(moe_gather_kernel, dim3(pairs), dim3(128), 0, stream, (const bf16*)x, x_stride, (bf16*)xg, d,
                                top, E_real, perm, offsets);
            if (rc) return rc;
            a = xg; a_rows = pairs; a_stride = d;
        }
        rc = wg ? moe_tc_launch<1>(a, a_rows, a_stride, wg, wu, hidden, nullptr, ff, d, E_real, pairs, top, act, !xg, perm, tile_info, tiles, stream)
                : moe_tc_launch<2>(a, a_rows, a_stride, wu, nullptr, hidden, nullptr, ff, d, E_real, pairs, top, act, !xg, perm, tile_info, tiles, stream);
        if (rc) return rc;
        rc = moe_tc_launch<0>(hidden, pairs, ff, wd, nullptr, nullptr, y, d, ff, E_real, pairs, top, act, false, perm, tile_info, tiles, stream);
        if (rc) return rc;
        return MOE_COMBINE(bf16);
    }
    if (dtype == TGO_BF16) {
        rc = tgo_launch_pdl(moe_up_kernel<bf16>, g1, dim3(256), 0, stream, (const bf16*)x, x_stride,
                            (const bf16*)wg, (const bf16*)wu, (bf16*)hidden, d, ff, top, act, perm, tile_info,
                            tiles);
        if (rc) return rc;
        rc = tgo_launch_pdl(moe_down_kernel<bf16>, g2, dim3(256), 0, stream, (const bf16*)hidden,
                            (const bf16*)wd, y, d, ff, perm, tile_info, tiles);
        if (rc) return rc;
        return MOE_COMBINE(bf16);
    }
    if (dtype != TGO_F32) return TGO_E_BAD_ARG;
    rc = tgo_launch_pdl(moe_up_kernel<float>, g1, dim3(256), 0, stream, (const float*)x, x_stride,
                        (const float*)wg, (const float*)wu, (float*)hidden, d, ff, top, act, perm, tile_info,
                        tiles);
    if (rc) return rc;
    rc = tgo_launch_pdl(moe_down_kernel<float>, g2, dim3(256), 0, stream, (const float*)hidden,
                        (const float*)wd, y, d, ff, perm, tile_info, tiles);
    if (rc) return rc;
    return MOE_COMBINE(float);
#undef MOE_COMBINE
#undef MOE_COMBINE_OF
}
