// Paged causal attention over one wide row a token (a compressed latent and its rotated part; the
// values are its first dv channels) for prompt portions, on the tcgen05 tensor cores: what
// attention_tc.cu does for heads of 128, with rows too wide for its plan.
//
// A work item is 128 query rows (all H heads of 128 / H consecutive tokens of one request: there is
// one key/value head) and one part of up to 256 value channels: the sums of 512 value channels
// would take all of tensor memory, so two items make S for the same rows and each keeps its half
// (1.5 times the products of a kernel that could keep both). Tensor memory: S0, S1 (128 columns each,
// P lies over S) and O (256). Shared memory: the item's Q (nine blocks of 128 rows x 64 channels for
// rows of 576: 147 KB), and two rings of 16 KB slots: K blocks of 128 keys x 64 channels, V blocks of
// 32 keys x 256 channels of the same rows, fetched again when P is ready (keeping them would need
// 64 KB more). Per key tile of 128 the products take 3328 cycles (36 of 64, 8 of 128) and 208 KB come
// into the SM: both near what it can do.
//   warp 0      draws items (longest first) from a counter, asks TMA for Q, publishes a record;
//   warps 12..14, 10 and 15  ask for K and for V, a warp a slot of its ring, a page and block a lane (a warp starts a
//               copy about every 80 cycles, and a key tile in pages of 16 takes 72 of K and 32 of V: one warp each, 138 us);
//   warps 1, 11   issue S = Q K^T and O += P V, a thread each;
//   warps 2..9  softmax, two threads a row, as in attention_tc.cu (lazily moved maximum).
// Rows of V that nobody may read are zeroed by warps 10 and 15, each in its slot, once they have landed (P is zero there, but the
// cache may hold anything).
//
// MEASURED (B200, 2048 tokens of 16 heads, rows of 576, values of 512; mma.sync tiles of eight warps in
// brackets): 118 us (511), 617 TFLOP/s of the products an ideal kernel would make.
//
// Every wait has a time limit (about two seconds), after which the CTA stops issuing, waits, with the same
// limit, for its copies and products under way, frees its tensor memory and returns. No cluster, no
// multicast.
#include "tcgen.cuh"

#define LT_THREADS 512
#define LT_BLOCK 16384                   // 128 rows x 64 channels, or 32 rows x 256
#define LT_MAX_BLOCKS 9                  // blocks of Q: rows up to 576 wide
#define LT_K_SLOTS 3
#define LT_V_SLOTS 2
#define LT_TILES ((LT_MAX_BLOCKS + LT_K_SLOTS + LT_V_SLOTS) * LT_BLOCK)
#define LT_MISC 3072
#define LT_SMEM (LT_TILES + LT_MISC)     // all 227 KB: the tiles start where the block's memory does

__device__ int lt_error_flag = 0;

struct LtItem {
    int valid, tok0, n_rows, p0, n_it, t_lo, key_lo, key_hi, seq, part;
    int pad[6];
};

__device__ __forceinline__ bool lt_bar_or(bool pred) {   // barrier of the 256 softmax threads
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                 "bar.red.or.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)pred) : "memory");
    return r != 0;
}
__device__ __forceinline__ float lt_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void lt_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(tg_smem(dst)), "l"(map), "r"(tg_smem(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}

// A warp that gives up waits for the last copies into its own slot; `count` uses of the ring have gone by.
__device__ __forceinline__ void lt_settle_slot(uint64_t* full, uint32_t slots, uint32_t slot, uint32_t count, int* err, int code) {
    if (count <= slot) return;
    const uint32_t last = count - 1 - (count - 1 - slot) % slots;
    tg_wait(&full[slot], (last / slots) & 1u, err, code);
}

__global__ void __launch_bounds__(LT_THREADS, 1)
attention_latent_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const __grid_constant__ CUtensorMap map_v, bf16* __restrict__ out, long long out_stride,
                           int page_size, const int* __restrict__ block_tables, int max_blocks,
                           const int* __restrict__ positions, const int* __restrict__ seq_ids,
                           const int* __restrict__ tile_tok0, const int* __restrict__ tile_ntok, int n_tiles, int H,
                           int blocks, int dv, float scale_log2, int window, const float* __restrict__ sinks,
                           unsigned int* __restrict__ ticket) {
    extern __shared__ __align__(1024) unsigned char base[];
    unsigned char* sQ = base;
    unsigned char* sK = sQ + LT_MAX_BLOCKS * LT_BLOCK;
    unsigned char* sV = sK + LT_K_SLOTS * LT_BLOCK;
    uint64_t* bars = (uint64_t*)(base + LT_TILES);
    uint64_t* q_full = bars;             // [1]
    uint64_t* q_empty = bars + 1;        // [1]
    uint64_t* k_full = bars + 2;         // [3]
    uint64_t* k_empty = bars + 5;        // [3]
    uint64_t* v_full = bars + 8;         // [2]
    uint64_t* v_empty = bars + 10;       // [2]
    uint64_t* v_ok = bars + 12;          // [2]: rows nobody may read are zero
    uint64_t* s_full = bars + 14;        // [2]
    uint64_t* p_full = bars + 16;        // [2]
    uint64_t* p_free = bars + 18;        // [2]
    uint64_t* o_free = bars + 20;        // [1]
    uint64_t* o_done = bars + 21;        // [1]
    uint64_t* settled = bars + 22;       // [2]: after a wait ran out, one an issuer
    uint32_t* tmem_slot = (uint32_t*)(bars + 24);
    LtItem* ring = (LtItem*)(bars + 26);                 // [2]
    float* s_xm = (float*)(ring + 2);                    // [2][2 halves][128 rows]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int parts = (dv + 255) / 256, n_items = n_tiles * parts;
    const int ppt = 128 / page_size;                     // pages of a key tile
    const int box_rows = (128 / H) * H;                  // rows of a Q box
    if (tg_smem(base) & 1023u) {                         // the plan leaves no room to move the tiles
        if (tid == 0) atomicExch(&lt_error_flag, 9);
        return;
    }
    if (tid == 0) {
        tg_init(q_full, 1);
        tg_init(q_empty, 15);
        for (int i = 0; i < LT_K_SLOTS; ++i) { tg_init(&k_full[i], 1); tg_init(&k_empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            tg_init(&v_full[i], 1); tg_init(&v_empty[i], 1); tg_init(&v_ok[i], 1);
            tg_init(&s_full[i], 1); tg_init(&p_full[i], 8); tg_init(&p_free[i], 1); tg_init(&settled[i], 1);
        }
        tg_init(o_free, 8);
        tg_init(o_done, 1);
        tg_init_done();
    }
    if (warp == 1) tg_alloc512(tmem_slot);
    tg_before();
    __syncthreads();
    tg_after();
    const uint32_t tmem = *tmem_slot, tm_o = tmem + 256u;
    int* const err = &lt_error_flag;

    if (warp == 0) {
        // ---------------------------------------------------------- items and Q
        bool ok = true;
        for (uint32_t n = 0; ok; ++n) {
            LtItem* rec = &ring[n & 1u];
            // the products with the last item's Q have run, and everybody has read its record
            ok = __all_sync(0xffffffffu, tg_wait(q_empty, (n & 1u) ^ 1u, err, 1));
            if (!ok) {
                tg_settle_copies(q_full, 1, n, err, 1);
                break;
            }
            int item = 0;
            if (lane == 0) item = (int)atomicAdd(ticket, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= n_items) {
                if (lane == 0) {
                    rec->valid = 0;
                    tg_arrive(q_full);
                }
                break;
            }
            const int tile = n_tiles - 1 - item / parts;     // longest first: later tiles read more keys
            const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
            const int p0 = positions[tok0], seq = seq_ids[tok0];
            const int key_lo = (window > 0 && p0 - window + 1 > 0) ? p0 - window + 1 : 0, key_hi = p0 + ntok;
            const int t_lo = key_lo / 128, n_it = p0 < 0 ? 0 : (key_hi + 127) / 128 - t_lo;
            if (lane == 0) {
                rec->valid = 1; rec->tok0 = tok0; rec->n_rows = ntok * H; rec->p0 = p0; rec->n_it = n_it;
                rec->t_lo = t_lo; rec->key_lo = key_lo; rec->key_hi = key_hi; rec->seq = seq; rec->part = item % parts;
                if (n_it > 0) {
                    // a box spans a full tile's tokens: later rows are other tokens' (never stored) or zeros
                    tg_expect(q_full, (uint32_t)blocks * (uint32_t)box_rows * 128u);
                    for (int c = 0; c < blocks; ++c) lt_load_3d(sQ + c * LT_BLOCK, &map_q, 64 * c, 0, tok0, q_full);
                } else {
                    tg_arrive(q_full);
                }
            }
            __syncwarp();
        }
    } else if (warp >= 12 && warp < 12 + LT_K_SLOTS) {
        // ---------------------------------------------------------- K
        bool ok = true;
        uint32_t g = 0;
        for (uint32_t n = 0; ok; ++n) {
            ok = __all_sync(0xffffffffu, tg_wait(q_full, n & 1u, err, 2));
            if (!ok) break;
            const LtItem rec = ring[n & 1u];
            if (!rec.valid) break;
            __syncwarp();
            if (lane == 0) tg_arrive(q_empty);
            const int* bt = block_tables + (size_t)rec.seq * max_blocks;
            for (int it = 0; it < rec.n_it && ok; ++it) {
                const int j = rec.t_lo + it;
                int first = j * ppt, last = first + ppt;
                while (first < last && (first + 1) * page_size <= rec.key_lo) ++first;
                while (last > first && (last - 1) * page_size >= rec.key_hi) --last;
                const bool mine = lane < last - first;
                const int row = mine ? bt[first + lane] * page_size : 0;
                const int at = (first + lane - j * ppt) * page_size * 128;
                for (int c = 0; c < blocks; ++c, ++g) {
                    const uint32_t s = g % LT_K_SLOTS, ph = (g / LT_K_SLOTS) & 1u;
                    if (s != (uint32_t)(warp - 12)) continue;
                    ok = __all_sync(0xffffffffu, tg_wait(&k_empty[s], ph ^ 1u, err, 3));
                    if (!ok) break;
                    if (lane == 0) tg_expect(&k_full[s], (uint32_t)(last - first) * (uint32_t)page_size * 128u);
                    __syncwarp();
                    if (mine) tg_load_2d(sK + s * LT_BLOCK + at, &map_k, 64 * c, row, &k_full[s]);
                }
            }
        }
        if (!ok) lt_settle_slot(k_full, LT_K_SLOTS, warp - 12, g, err, 3);
    } else if (warp == 10 || warp == 15) {
        // ---------------------------------------------------------- V
        bool ok = true;
        uint32_t g = 0;
        const int vrows = page_size < 32 ? page_size : 32, vboxes = 32 / vrows;      // boxes of a slot's rows
        for (uint32_t n = 0; ok; ++n) {
            ok = __all_sync(0xffffffffu, tg_wait(q_full, n & 1u, err, 4));
            if (!ok) break;
            const LtItem rec = ring[n & 1u];
            if (!rec.valid) break;
            __syncwarp();
            if (lane == 0) tg_arrive(q_empty);
            const int* bt = block_tables + (size_t)rec.seq * max_blocks;
            const int width = min(256, dv - 256 * rec.part), cols = width / 64;
            for (int it = 0; it < rec.n_it && ok; ++it) {
                for (int q = 0; q < 4; ++q) {
                    const int k0 = (rec.t_lo + it) * 128 + 32 * q;
                    if (k0 >= rec.key_hi || k0 + 32 <= rec.key_lo) continue;         // P is zero there
                    const uint32_t s = g % LT_V_SLOTS, ph = (g / LT_V_SLOTS) & 1u;
                    if (s != (warp == 15 ? 1u : 0u)) {   // the other warp's
                        ++g;
                        continue;
                    }
                    ok = __all_sync(0xffffffffu, tg_wait(&v_empty[s], ph ^ 1u, err, 5));
                    if (!ok) break;
                    ++g;
                    unsigned char* slot = sV + s * LT_BLOCK;
                    // boxes whose rows somebody may read: [b_lo, b_hi)
                    int b_lo = 0, b_hi = vboxes;
                    while (k0 + (b_lo + 1) * vrows <= rec.key_lo) ++b_lo;
                    while (k0 + (b_hi - 1) * vrows >= rec.key_hi) --b_hi;
                    if (lane == 0) tg_expect(&v_full[s], (uint32_t)((b_hi - b_lo) * vrows * cols * 128));
                    __syncwarp();
                    const int count = (b_hi - b_lo) * cols;
                    if (lane < count) {
                        const int c = lane / (b_hi - b_lo), b = b_lo + lane % (b_hi - b_lo);
                        const int key = k0 + b * vrows;
                        tg_load_2d(slot + c * 4096 + b * vrows * 128, &map_v, 256 * rec.part + 64 * c,
                                   bt[key / page_size] * page_size + key % page_size, &v_full[s]);
                    }
                    if (k0 < rec.key_lo || k0 + 32 > rec.key_hi) {
                        ok = __all_sync(0xffffffffu, tg_wait(&v_full[s], ph, err, 6));
                        if (!ok) break;
                        const int key = k0 + lane;
                        if (key < rec.key_lo || key >= rec.key_hi)
                            for (int c = 0; c < cols; ++c)
#pragma unroll
                                for (int x = 0; x < 8; ++x)
                                    *(uint4*)(slot + c * 4096 + lane * 128 + x * 16) = make_uint4(0u, 0u, 0u, 0u);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) tg_arrive(&v_ok[s]);
                    }
                }
            }
        }
        if (!ok) lt_settle_slot(v_full, LT_V_SLOTS, warp == 15 ? 1 : 0, g, err, 5);
    } else if (warp == 1) {
        // ---------------------------------------------------------- issuer of S = Q K^T
        if (lane == 0) {
            const uint32_t idesc = tg_idesc(128);
            uint32_t g = 0, t = 0;                       // K slots and key tiles so far
            bool ok = true;
            for (uint32_t n = 0; ok; ++n) {
                ok = tg_wait(q_full, n & 1u, err, 7);
                if (!ok) break;
                const LtItem* rec = &ring[n & 1u];
                if (!rec->valid) break;
                const int n_it = rec->n_it;
                for (int it = 0; it < n_it && ok; ++it, ++t) {
                    const uint32_t sb = t & 1u;
                    ok = tg_wait(&p_free[sb], ((t >> 1) & 1u) ^ 1u, err, 8);        // the P in this buffer has been multiplied
                    for (int c = 0; c < blocks && ok; ++c, ++g) {
                        const uint32_t s = g % LT_K_SLOTS;
                        ok = tg_wait(&k_full[s], (g / LT_K_SLOTS) & 1u, err, 8);
                        if (!ok) break;
                        tg_after();
                        const uint64_t dq = tg_desc(sQ + c * LT_BLOCK), dk = tg_desc(sK + s * LT_BLOCK);
#pragma unroll
                        for (int k = 0; k < 4; ++k) tg_mma(tmem + 128u * sb, dq + 2 * k, dk + 2 * k, idesc, (c > 0 || k > 0) ? 1u : 0u);
                        tg_commit(&k_empty[s]);
                    }
                    if (ok) tg_commit(&s_full[sb]);
                }
                tg_commit(q_empty);                      // the item's products with Q have run
            }
            if (!ok) tg_settle_products(&settled[0], err, 8);
        }
    } else if (warp == 11) {
        // ---------------------------------------------------------- issuer of O += P V
        if (lane == 0) {
            uint32_t g = 0, t = 0, okph = 0;
            bool ok = true;
            for (uint32_t n = 0; ok; ++n) {
                ok = tg_wait(q_full, n & 1u, err, 10);
                if (!ok) break;
                const LtItem rec = ring[n & 1u];
                if (!rec.valid) break;
                tg_arrive(q_empty);
                const uint32_t idesc = tg_idesc(min(256, dv - 256 * rec.part), true);
                uint32_t acc = 0;
                for (int it = 0; it < rec.n_it && ok; ++it, ++t) {
                    const uint32_t sb = t & 1u;
                    if (it == 0) ok = tg_wait(o_free, (n & 1u) ^ 1u, err, 11);      // the last item's O is out
                    ok = ok && tg_wait(&p_full[sb], (t >> 1) & 1u, err, 12);
                    for (int q = 0; q < 4 && ok; ++q) {
                        const int k0 = (rec.t_lo + it) * 128 + 32 * q;
                        if (k0 >= rec.key_hi || k0 + 32 <= rec.key_lo) continue;
                        const uint32_t s = g % LT_V_SLOTS;
                        ok = tg_wait(&v_full[s], (g / LT_V_SLOTS) & 1u, err, 13);
                        ++g;
                        if (ok && (k0 < rec.key_lo || k0 + 32 > rec.key_hi)) {
                            ok = tg_wait(&v_ok[s], (okph >> s) & 1u, err, 14);
                            okph ^= 1u << s;
                        }
                        if (!ok) break;
                        tg_after();
                        const uint64_t dv_ = tg_desc_mn(sV + s * LT_BLOCK, 4096u);
#pragma unroll
                        for (int k = 0; k < 2; ++k) {    // 16 keys = two groups of eight rows = 2048 bytes
                            tg_mma_ts(tm_o, tmem + 128u * sb + 16u * q + 8u * k, dv_ + (uint64_t)(128 * k), idesc, acc);
                            acc = 1u;
                        }
                        tg_commit(&v_empty[s]);
                    }
                    if (!ok) break;
                    tg_commit(&p_free[sb]);
                    tg_commit(o_done);
                }
            }
            if (!ok) tg_settle_products(&settled[1], err, 12);
        }
    } else {
        // ---------------------------------------------------------- softmax
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        uint32_t t = 0;
        for (uint32_t n = 0;; ++n) {
            if (ok) ok = tg_wait(q_full, n & 1u, err, 15);
            if (lt_bar_or(!ok)) break;                   // a wait ran out somewhere: all 256 leave together
            const LtItem rec = ring[n & 1u];
            if (!rec.valid) break;
            __syncwarp();
            if (lane == 0) tg_arrive(q_empty);
            const int n_rows = rec.n_rows, p0 = rec.p0, n_it = rec.n_it;
            const int width = min(256, dv - 256 * rec.part), oc = width / 2;
            const bool row_ok = row < n_rows;
            const int head = (row_ok ? row : 0) % H;
            bf16* dst = out + (size_t)(rec.tok0 + (row_ok ? row : 0) / H) * out_stride + (size_t)head * dv + 256 * rec.part + oc * half;
            if (n_it == 0) {                             // a request that brings nothing: zeros out
                if (row_ok)
                    for (int i = 0; i < oc; i += 8) *(uint4*)(dst + i) = make_uint4(0u, 0u, 0u, 0u);
                __syncwarp();
                if (lane == 0) tg_arrive(o_free);
                continue;
            }
            const int pos = row_ok ? p0 + row / H : -1;
            const int vis_lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
            const int last_row = quarter * 32 + 31;
            const int pos_min = p0 + quarter * 32 / H, pos_max = p0 + (last_row < n_rows ? last_row : n_rows - 1) / H;
            const int vis_max = (window > 0 && pos_max - window + 1 > 0) ? pos_max - window + 1 : 0;
            float m_used = -INFINITY, l = 0.f;
            for (int it = 0; it < n_it; ++it, ++t) {
                const uint32_t sb = t & 1u, tm_s = tmem + 128u * sb;
                const int kbase = (rec.t_lo + it) * 128 + 64 * half;
                if (ok) ok = tg_wait(&s_full[sb], (t >> 1) & 1u, err, 16);
                tg_after();
                float sc[64];
                {
                    uint32_t r0[32], r1[32];
                    tg_ld32(tm_s + lane_base + 64u * half, r0);
                    tg_ld32(tm_s + lane_base + 64u * half + 32u, r1);
                    tg_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) { sc[i] = __uint_as_float(r0[i]); sc[32 + i] = __uint_as_float(r1[i]); }
                }
                const bool full = last_row < n_rows && kbase + 63 <= pos_min && kbase >= vis_max;
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                if (full) {
#pragma unroll
                    for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sc[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 64; ++i) {
                        const int key = kbase + i;
                        sc[i] = (key <= pos && key >= vis_lo) ? sc[i] : -INFINITY;
                        mx4[i & 3] = fmaxf(mx4[i & 3], sc[i]);
                    }
                }
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
                float* xm = s_xm + sb * 256;
                xm[half * 128 + row] = mx;
                if (lt_bar_or(!ok)) { ok = false; break; }   // both halves have read their S
                mx = fmaxf(mx, xm[(half ^ 1) * 128 + row]);
                const float m_new = fmaxf(m_used, mx);
                const bool grow = m_new > m_used + 8.f || (m_used == -INFINITY && m_new != -INFINITY);
                const bool rescale = __any_sync(0xffffffffu, grow);
                float corr = 1.f;
                if (rescale) {
                    corr = m_new == -INFINITY ? 1.f : exp2f(m_used - m_new);
                    m_used = m_new;
                }
                const float base_m = m_used == -INFINITY ? 0.f : m_used;
                float sum4[4] = {0.f, 0.f, 0.f, 0.f};
                {
                    uint32_t r[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float a = lt_ex2(fmaf(sc[2 * i], scale_log2, -base_m));
                        const float b = lt_ex2(fmaf(sc[2 * i + 1], scale_log2, -base_m));
                        sum4[i & 3] += a + b;
                        r[i] = tg_pack(a, b);
                    }
                    tg_st32(tm_s + lane_base + 32u * half, r);
                }
                l = l * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
                if (it > 0) {
                    if (ok) ok = tg_wait(o_done, (t - 1u) & 1u, err, 17);            // the previous P V is in O
                    tg_after();
                    if (rescale)
                        for (int c = 0; c < oc; c += 32) {
                            uint32_t r[32];
                            tg_ld32(tm_o + lane_base + (uint32_t)(oc * half + c), r);
                            tg_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
                            tg_st32(tm_o + lane_base + (uint32_t)(oc * half + c), r);
                        }
                }
                tg_wait_st();
                tg_before();
                const bool warp_ok = __all_sync(0xffffffffu, ok);
                if (lane == 0 && warp_ok) tg_arrive(&p_full[sb]);
            }
            if (!ok) break;                              // decided at a barrier: the same for all 256
            ok = tg_wait(o_done, (t - 1u) & 1u, err, 18);    // the item's last P V
            tg_after();
            // the buffer of the tile before the last: its readers passed that tile's barrier
            float* xl = s_xm + (t & 1u) * 256;
            xl[half * 128 + row] = l;
            if (lt_bar_or(!ok)) break;
            l += xl[(half ^ 1) * 128 + row];
            float f = 1.f;
            if (sinks) {                                 // the sink joins the denominator last
                const float sk = sinks[head] * 1.4426950408889634f, mn = fmaxf(m_used, sk);
                f = exp2f(m_used - mn);
                l = l * f + exp2f(sk - mn);
            }
            const float inv = l > 0.f ? f / l : 0.f;
            for (int c = 0; c < oc; c += 32) {
                uint32_t r[32];
                tg_ld32(tm_o + lane_base + (uint32_t)(oc * half + c), r);
                tg_wait_ld();
                if (row_ok)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 v;
                        v.x = tg_pack(__uint_as_float(r[8 * i]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
                        v.y = tg_pack(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
                        v.z = tg_pack(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
                        v.w = tg_pack(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
                        *(uint4*)(dst + c + i * 8) = v;
                    }
            }
            tg_before();
            __syncwarp();
            if (lane == 0) tg_arrive(o_free);
        }
    }
    tg_before();
    __syncthreads();
    if (warp == 1) {
        tg_after();
        tg_free512(tmem);
    }
}

// Reads (and waits for the device to reach) the code a wait that ran out left; 0: none did.
TGO_API int tgo_attention_latent_tc_error(int* value) { return (int)cudaMemcpyFromSymbol(value, lt_error_flag, sizeof(int)); }

// 1 if the kernel takes the shape: one key/value head, up to 128 query heads, rows up to 576 wide whose
// first dv channels (whole blocks of 64) are the values, pages of 8, 16, 32, 64 or 128 tokens.
TGO_API int tgo_attention_latent_tc_supports(int H, int dk, int dv, int page_size) {
    const bool p_ok = page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128;
    return H >= 1 && H <= 128 && dv >= 64 && dv % 64 == 0 && dk >= dv && dk <= 64 * LT_MAX_BLOCKS && dk % 8 == 0 && p_ok;
}

// q: n_tokens rows of q_stride elements, the first H * dk columns the heads; out: H * dv columns a
// row; cache [n_pages, 1, page_size, dk] bfloat16; tiles of up to 128 / H consecutive tokens of one
// request (tile_tok0, tile_ntok); scale > 0; window 0: every earlier key; sinks [H] or null.
// counters: an int that this launch alone uses, zeroed here.
TGO_API int tgo_attention_latent_tc(const void* q, long long q_stride, int n_tokens, void* out, long long out_stride,
                                    const void* cache, int n_pages, int page_size, const int* block_tables,
                                    int max_blocks, const int* positions, const int* seq_ids, const int* tile_tok0,
                                    const int* tile_ntok, int n_tiles, int H, int dk, int dv, float scale, int window,
                                    const float* sinks, int* counters, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (n_tokens <= 0 || !tgo_attention_latent_tc_supports(H, dk, dv, page_size) || n_pages <= 0 || max_blocks <= 0 ||
        window < 0 || !tile_tok0 || !tile_ntok || !counters || q_stride % 8 || out_stride % 8 || ((uintptr_t)q % 16) ||
        ((uintptr_t)out % 16) || ((uintptr_t)cache % 16) || !(scale > 0.f) ||
        (long long)n_pages * page_size > 0x7fffffffll || (long long)n_tiles * 2 > 0x7fffffffll)
        return TGO_E_BAD_ARG;
    CUtensorMap mq, mk, mv;
    const long long rows = (long long)n_pages * page_size;
    if (!tg_map(&mk, cache, rows, dk, dk, page_size) || !tg_map(&mv, cache, rows, dk, dk, page_size < 32 ? page_size : 32) ||
        !tg_map_heads(&mq, q, n_tokens, H, dk, q_stride, 128 / H))
        return TGO_E_BAD_ARG;
    static int sms_of[64] = {};                          // per device, and that the attribute is set there
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return TGO_E_BAD_ARG;
    if (!sms_of[dev]) {
        e = cudaFuncSetAttribute(attention_latent_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM);
        if (e != cudaSuccess) return (int)e;
        int n = 0;
        if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)e;
        sms_of[dev] = n;
    }
    if ((e = cudaMemsetAsync(counters, 0, sizeof(int), stream)) != cudaSuccess) return (int)e;
    const int items = n_tiles * ((dv + 255) / 256), sms = sms_of[dev];
    attention_latent_tc_kernel<<<dim3(items < sms ? items : sms), LT_THREADS, LT_SMEM, stream>>>(
        mq, mk, mv, (bf16*)out, out_stride, page_size, block_tables, max_blocks, positions, seq_ids, tile_tok0, tile_ntok,
        n_tiles, H, (dk + 63) / 64, dv, scale * 1.4426950408889634f, window, sinks, (unsigned int*)counters);
    return launch_status();
}
