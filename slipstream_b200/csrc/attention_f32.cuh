// Paged, ragged, causal grouped-query attention with float32 operands and arithmetic on CUDA cores, tiled for prompt
// portions and split over the keys where there are few query tiles (decode steps).  Masks, sinks, soft caps, gates, kept
// first keys and `across` as in attention_simt.cuh.
//
// Rows are (token, query head of a kv head's group) pairs, so a group shares every tile of keys and values.  A block takes
// RT rows of one request and walks tiles of 32 keys that start at multiples of 32 from the request's first token, copied
// ahead by cp.async (keys into one of two buffers, values while the scores are formed); a thread forms 4 x (RT / 16) scores
// and (RT / 8) x 4 ceil(D / 64) outputs in registers.
//
// The order of the arithmetic behind one row is the same however the prompt was cut, whatever else is in the step and
// however many blocks share a row's keys: keys fall into slices of AF_SLICE from the request's first token, every slice has
// a softmax of its own (32 keys at a time, in order), and a row's slices are joined in order (af_join).  A block that
// walks all slices of its rows joins them in registers; with more than one block to a row (gridDim.z) every slice's
// maximum, sum and output go to scratch memory and attn_f32_join_kernel joins them, with the same operations.
//
// Bound by issue: 70 % of its instructions are the multiply-adds, and three blocks of four warps an SM issue on about half
// of the cycles.  Against attention_simt.cuh (a tile of 16 tokens of one query head, keys in series, no copies ahead):
// 777 tokens of two requests, one behind 300 cached ones, 28 heads of 128 on 4: 551 -> 209 us.  Decode steps with heads of up
// to 128 have a kernel of their own (attn_f32_decode_kernel).
#pragma once

#include "common.cuh"
#include "mma_sync.cuh"

#define AF_BN 32
#define AF_SLICE 128
#define AF_THREADS 128

struct AttnF32Args {
    const float* q;
    int64_t q_stride;
    float* out;
    int64_t out_stride;
    const float* kv;
    const int32_t* tables;
    int max_blocks;
    const int32_t* tile_req;  // tiles of 64 rows (first row in tile_q0), or null: a decode step, ceil(G / RT) tiles a request
    const int32_t* tile_q0;
    const int32_t* q_start;
    const int32_t* seq_lens;
    int n_requests;
    int n_q, n_kv, page_size;
    int64_t num_pages;
    float scale;
    int window;
    int* err;
    const float* gate;
    float softcap;
    const float* sinks;
    int keep, across;
    float* part;      // [rows][output heads][max_slices][D]; null where a row has one block
    float2* part_ml;  // [rows][output heads][max_slices]: a slice's maximum and sum
    int max_slices;
    int n_rows;
};

// The factors with which a row's state (maximum m, sum l) and a slice's take part in their union, which replaces (m, l).
__device__ __forceinline__ float2 af_join(float& m, float& l, float slice_m, float slice_l) {
    const float top = fmaxf(m, slice_m);
    const float a = m == -INFINITY ? 0.f : expf(__fsub_rn(m, top)), b = slice_m == -INFINITY ? 0.f : expf(__fsub_rn(slice_m, top));
    l = __fadd_rn(__fmul_rn(l, a), __fmul_rn(slice_l, b));
    m = top;
    return make_float2(a, b);
}
__device__ __forceinline__ float af_mix(float total, float2 f, float slice) {
    return __fadd_rn(__fmul_rn(total, f.x), __fmul_rn(slice, f.y));
}
__device__ __forceinline__ float af_finish(float v, float l, const float* gate) {
    v *= l > 0.f ? 1.0f / l : 0.f;
    return gate ? gated<false>(v, *gate) : v;
}

template <int D, int RT>
constexpr int af_smem_bytes() {
    return (RT * (D + 4) + 2 * AF_BN * (D + 4) + AF_BN * D + AF_BN * (RT + 4) + 2 * RT) * 4;
}

template <int D, int RT>
__global__ void __launch_bounds__(AF_THREADS, D <= 128 ? 3 : 1) attn_f32_kernel(const AttnF32Args g) {
    constexpr int KS = D + 4, PS = RT + 4;             // row strides in shared memory: rows 16 bytes further round the banks
    constexpr int KPT = RT * AF_BN / AF_THREADS / 4, TX = AF_BN / KPT, TY = AF_THREADS / TX;  // scores: rows ty + TY i (i < 4), keys tx + TX j
    constexpr int RP = RT / (AF_THREADS / 16), NC = (D + 63) / 64;     // outputs: rows py RP + i, elements 4 (px + 16 c) .. + 3
    extern __shared__ __align__(16) float af_smem[];
    float* Qs = af_smem;
    float* Ks = Qs + RT * KS;
    float* Vs = Ks + 2 * AF_BN * KS;
    float* Ps = Vs + AF_BN * D;   // [key][row]
    float* alpha_s = Ps + AF_BN * PS; // by row: the factor of what was summed before the tile, and the maximum so far
    float* max_s = alpha_s + RT;

    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x;
    // the kv head runs fastest and a request's later tiles, which see more keys, come first: the longest blocks start first
    const int G = g.n_q / g.n_kv, n_heads = g.across ? g.n_kv * g.n_kv : g.n_kv, u = blockIdx.x % n_heads;
    const int block = ((int)gridDim.x - 1 - (int)blockIdx.x) / n_heads;
    const HeadPair hp = head_pair(u, g.n_kv, g.across);
    int r, row0;
    if (g.tile_req != nullptr) {
        constexpr int SUB = 64 / RT;  // blocks of a tile of the list
        r = g.tile_req[block / SUB];
        row0 = g.tile_q0[block / SUB] + (block % SUB) * RT;
    } else {
        const int per_request = (G + RT - 1) / RT;
        r = block / per_request;
        row0 = (block % per_request) * RT;
    }
    const int qs = g.q_start[r], q_len = g.q_start[r + 1] - qs, seq_len = g.seq_lens[r];
    const int rows = min(RT, q_len * G - row0);
    if (rows <= 0) return;  // a padding tile of a captured step (uniform over the block)
    const int pos0 = seq_len - q_len, p_first = pos0 + row0 / G, p_max = pos0 + (row0 + rows - 1) / G;
    const int lo_min = key_floor(p_first, g.window);
    const int32_t* table = g.tables + (int64_t)r * g.max_blocks;

    // this block's slices, and the tiles of its walk that fall into them: n1 kept ones from a1 on, then those from a2 on
    const KeyTiles walk = key_tiles(lo_min, p_max, g.keep, AF_BN);
    constexpr int TPS = AF_SLICE / AF_BN;
    const int s_first = walk.kept > 0 ? 0 : walk.first / TPS, s_count = p_max < 0 ? 0 : p_max / AF_SLICE + 1 - s_first;
    const int per = (s_count + (int)gridDim.z - 1) / (int)gridDim.z;
    const int t_begin = (s_first + (int)blockIdx.z * per) * TPS, t_end = min(s_first + s_count, s_first + ((int)blockIdx.z + 1) * per) * TPS;
    const int a1 = t_begin, n1 = max(0, min(walk.kept, t_end) - a1);
    const int a2 = max(walk.first, t_begin), n2 = max(0, min(p_max / AF_BN + 1, t_end) - a2);
    const int n_tiles = s_count > 0 ? n1 + n2 : 0;
    const bool alone = g.part == nullptr;
    if (!alone && n_tiles == 0) return;
    auto tile_at = [&](int j) { return j < n1 ? a1 + j : a2 + (j - n1); };

    for (int idx = tid; idx < RT * (D / 4); idx += AF_THREADS) {
        const int row = idx / (D / 4), d4 = idx - row * (D / 4);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows) {
            const float* src = g.q + (int64_t)(qs + (row0 + row) / G) * g.q_stride + (int64_t)(hp.key * G + (row0 + row) % G) * D + d4 * 4;
            v = make_float4(src[0], src[1], src[2], src[3]);
        }
        *reinterpret_cast<float4*>(&Qs[row * KS + d4 * 4]) = v;
    }
    constexpr int TPR = AF_THREADS / AF_BN;  // threads that copy a key and its value; rows outside [lo_min, p_max] that are not kept are zero
    // (the page of the tile after is looked up a tile ahead)
    const int copy_row = tid / TPR;
    auto page_of = [&](int j) -> int64_t {
        const int key = tile_at(j) * AF_BN + copy_row;
        if (j >= n_tiles || !((key >= lo_min || key < g.keep) && key <= p_max)) return -1;
        return table[key / g.page_size];
    };
    int64_t next_page = page_of(0);
    int64_t value_at = -1;  // where the value of the key that was fetched last stands
    auto fetch_key = [&](int j) {
        int64_t page = next_page;
        next_page = page_of(j + 1);
        if (page >= g.num_pages) {
            if (tid % TPR == 0) atomicOr(g.err, SS_ERR_PAGE_RANGE);
            page = -1;
        }
        const bool live = page >= 0;
        const int64_t off = live ? (int64_t)((tile_at(j) * AF_BN + copy_row) % g.page_size) * D : 0;
        const float* src = g.kv + (live ? ((page * 2 + 0) * g.n_kv + hp.key) * g.page_size * (int64_t)D + off : 0);
        value_at = live ? ((page * 2 + 1) * g.n_kv + hp.value) * g.page_size * (int64_t)D + off : -1;
        float* dst = Ks + ((j & 1) * AF_BN + copy_row) * KS;
#pragma unroll
        for (int d = (tid % TPR) * 4; d < D; d += 4 * TPR) cp_async16(dst + d, src + (live ? d : 0), live);
    };
    auto fetch_value = [&]() {
        const bool live = value_at >= 0;
        const float* src = g.kv + (live ? value_at : 0);
#pragma unroll
        for (int d = (tid % TPR) * 4; d < D; d += 4 * TPR) cp_async16(Vs + copy_row * D + d, src + (live ? d : 0), live);
    };

    const int tx = tid % TX, ty = tid / TX, px = tid & 15, py = tid >> 4;
    float m[4];
    float acc[RP][NC * 4], l[RP], tot[RP][NC * 4], tot_m[RP], tot_l[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        // a sink: one more term exp(sinks[h]) in the row's denominator, with neither key nor value, added one time
        const bool sink = g.sinks != nullptr;
        tot_m[i] = sink ? g.sinks[hp.key * G + (row0 + py * RP + i) % G] : -INFINITY;
        tot_l[i] = sink ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < NC * 4; ++c) tot[i][c] = 0.f;
    }
    if (n_tiles > 0) fetch_key(0);
    cp_async_commit();

    for (int j = 0; j < n_tiles; ++j) {
        const int kt = tile_at(j), buf = j & 1;
        const bool opens = j == 0 || tile_at(j - 1) / TPS != kt / TPS, closes = j + 1 == n_tiles || tile_at(j + 1) / TPS != kt / TPS;
        cp_async_wait<0>();
        __syncthreads();  // the tile's keys are there, and everyone is done with the values before it
        fetch_value();
        cp_async_commit();
        if (j + 1 < n_tiles) fetch_key(j + 1);
        cp_async_commit();

        // ---- scores
        float s[4][KPT];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < KPT; ++k) s[i][k] = 0.f;
        const float* kb = Ks + buf * AF_BN * KS;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            float4 q4[4], k4[KPT];
#pragma unroll
            for (int i = 0; i < 4; ++i) q4[i] = *reinterpret_cast<const float4*>(&Qs[(ty + TY * i) * KS + d]);
#pragma unroll
            for (int k = 0; k < KPT; ++k) k4[k] = *reinterpret_cast<const float4*>(&kb[(tx + TX * k) * KS + d]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < KPT; ++k) {
                    s[i][k] = fmaf(q4[i].x, k4[k].x, s[i][k]);
                    s[i][k] = fmaf(q4[i].y, k4[k].y, s[i][k]);
                    s[i][k] = fmaf(q4[i].z, k4[k].z, s[i][k]);
                    s[i][k] = fmaf(q4[i].w, k4[k].w, s[i][k]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = ty + TY * i, pos = pos0 + (row0 + row) / G, lowest = key_floor(pos, g.window);
            float sc[KPT], top = -INFINITY;
#pragma unroll
            for (int k = 0; k < KPT; ++k) {
                const int key = kt * AF_BN + tx + TX * k;
                const bool ok = row < rows && key <= pos && (key >= lowest || key < g.keep);
                const float x = __fmul_rn(s[i][k], g.scale);
                sc[k] = ok ? (g.softcap > 0.f ? __fmul_rn(g.softcap, tanhf(x / g.softcap)) : x) : -INFINITY;
                top = fmaxf(top, sc[k]);
            }
#pragma unroll
            for (int o = TX / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float before = opens ? -INFINITY : m[i];
            const float now = fmaxf(before, top);
#pragma unroll
            for (int k = 0; k < KPT; ++k)
                Ps[(tx + TX * k) * PS + row] = sc[k] == -INFINITY ? 0.f : expf(__fsub_rn(sc[k], now));  // (a NaN has no part in `now`, and stays)
            if (tx == 0) {
                alpha_s[row] = before == -INFINITY ? 0.f : expf(__fsub_rn(before, now));
                max_s[row] = now;
            }
            m[i] = now;
        }
        cp_async_wait<1>();  // the values; the next keys may still be under way
        __syncthreads();

        // ---- outputs
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const float a = opens ? 0.f : alpha_s[py * RP + i];
            l[i] = opens ? 0.f : __fmul_rn(l[i], a);
#pragma unroll
            for (int c = 0; c < NC * 4; ++c) acc[i][c] = opens ? 0.f : __fmul_rn(acc[i][c], a);
        }
        const float* vb = Vs;
#pragma unroll 4
        for (int k = 0; k < AF_BN; ++k) {
            float p[RP];
            if constexpr (RP == 2) {
                const float2 t = *reinterpret_cast<const float2*>(&Ps[k * PS + py * RP]);
                p[0] = t.x; p[1] = t.y;
            } else {
#pragma unroll
                for (int i = 0; i < RP; i += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(&Ps[k * PS + py * RP + i]);
                    p[i] = t.x; p[i + 1] = t.y; p[i + 2] = t.z; p[i + 3] = t.w;
                }
            }
#pragma unroll
            for (int i = 0; i < RP; ++i) l[i] = __fadd_rn(l[i], p[i]);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if ((px + 16 * c) * 4 >= D) break;
                const float4 v = *reinterpret_cast<const float4*>(&vb[k * D + (px + 16 * c) * 4]);
#pragma unroll
                for (int i = 0; i < RP; ++i) {
                    acc[i][c * 4 + 0] = fmaf(p[i], v.x, acc[i][c * 4 + 0]);
                    acc[i][c * 4 + 1] = fmaf(p[i], v.y, acc[i][c * 4 + 1]);
                    acc[i][c * 4 + 2] = fmaf(p[i], v.z, acc[i][c * 4 + 2]);
                    acc[i][c * 4 + 3] = fmaf(p[i], v.w, acc[i][c * 4 + 3]);
                }
            }
        }
        if (!closes) continue;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const int row = py * RP + i;
            const float slice_m = max_s[row];
            if (alone) {
                const float2 f = af_join(tot_m[i], tot_l[i], slice_m, l[i]);
#pragma unroll
                for (int c = 0; c < NC * 4; ++c) tot[i][c] = af_mix(tot[i][c], f, acc[i][c]);
            } else if (row < rows) {
                const int64_t at = ((int64_t)(qs + (row0 + row) / G) * (n_heads * G) + u * G + (row0 + row) % G) * g.max_slices + kt / TPS;
                if (px == 0) g.part_ml[at] = make_float2(slice_m, l[i]);
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if ((px + 16 * c) * 4 < D)
                        *reinterpret_cast<float4*>(&g.part[at * D + (px + 16 * c) * 4]) =
                            make_float4(acc[i][c * 4], acc[i][c * 4 + 1], acc[i][c * 4 + 2], acc[i][c * 4 + 3]);
            }
        }
    }
    if (!alone) return;
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = py * RP + i;
        if (row >= rows) break;
        const int64_t t = qs + (row0 + row) / G;
        const int h = (row0 + row) % G;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if ((px + 16 * c) * 4 >= D) break;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = (px + 16 * c) * 4 + e;
                g.out[t * g.out_stride + (int64_t)(u * G + h) * D + d] =
                    af_finish(tot[i][c * 4 + e], tot_l[i], g.gate ? g.gate + t * g.q_stride + (int64_t)(hp.key * G + h) * D + d : nullptr);
            }
        }
    }
}

// One token a request: a block takes AFD_RT rows of a request and a slice of keys (gridDim.z blocks deal a request's slices
// out among them), whose keys and values it fetches in one go.  The scores of the slice's tiles are formed side by side, a
// warp to 16 keys; a tile's maximum so far is that of the tiles before it and its own, whoever formed them, so the
// exponentials, the sums (a thread to 4 rows and 2 elements) and the joins are those of attn_f32_kernel, bit for bit.
//
// BOTH: keys and values have buffers of their own and travel together, one block an SM: for a grid of one wave, whose time
// is the latency of its loads.  Otherwise values follow into the keys' buffer and three blocks an SM cover for each other.
//
// Bound by shared memory: a load brings 128 bytes a cycle to an SM's registers, also where lanes share a word, so a slice's
// scores take 3,700 cycles and its outputs as many, beside 3,000 in which its 131 KB arrive.  (Products of 4 x 4 a thread, on
// two warps, need half of that and run longer all the same: 439 us where these take 359, a warp has no other beside it.)
// With its join, against attn_f32_kernel (four tiles of a slice one after another), us, requests of equal length replayed from a
// graph, 12 heads of 128 on 2: four of 2,000 tokens 28 -> 11 (33.8 -> 17.0 behind a layer's products); 28 on 4: 20 of 800 80 -> 27, 20 of
// 16,000 1,080 -> 356 (the memory takes 180), 200 of 300 135 -> 85, one of 100 17.8 -> 8.8; 14 of 64 on 2: 256 of 1,000 239 -> 104.
// Groups of more than 8 heads, whose keys come once for every 8, against tiles of 16 rows: heads of 128 on 1, 64 requests of 800
// tokens, 9 heads 58 -> 35, 24 109 -> 49, 64 168 -> 125, 128 302 -> 228.
#define AFD_RT 8
#define AFD_THREADS 256
#define AFD_PS 8

template <int D, bool BOTH>
constexpr int afd_smem_bytes() {
    return (AFD_RT * (D + 4) + (BOTH ? 2 : 1) * AF_SLICE * (D + 4) + AF_SLICE * AFD_PS + (8 + AF_SLICE / AF_BN + 2) * AFD_RT) * 4;
}

template <int D, bool BOTH>
__global__ void __launch_bounds__(AFD_THREADS, BOTH ? 1 : 3) attn_f32_decode_kernel(const AttnF32Args g) {
    static_assert(AF_SLICE == 128 && AF_BN == 32 && D <= 128, "eight warps of 16 keys, 128 threads a half of the rows");
    constexpr int KS = D + 4, TPS = AF_SLICE / AF_BN, C4 = D / 4;
    extern __shared__ __align__(16) float afd_smem[];
    float* Qs = afd_smem;
    float* Ks = Qs + AFD_RT * KS;
    float* Vs = BOTH ? Ks + AF_SLICE * KS : Ks;
    float* Ps = Ks + (BOTH ? 2 : 1) * AF_SLICE * KS;  // [key][row]
    float* top_s = Ps + AF_SLICE * AFD_PS;            // [warp][row]: the largest score of the warp's 16 keys
    float* alpha_s = top_s + 8 * AFD_RT;              // [tile][row]: the factor of what was summed before the tile
    float* ml_s = alpha_s + TPS * AFD_RT;              // [row]: maximum and sum of the only slice

    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = g.n_q / g.n_kv, n_heads = g.across ? g.n_kv * g.n_kv : g.n_kv, u = blockIdx.x % n_heads;
    const int per_request = (G + AFD_RT - 1) / AFD_RT, block = blockIdx.x / n_heads;
    const HeadPair hp = head_pair(u, g.n_kv, g.across);
    const int r = block / per_request, row0 = (block % per_request) * AFD_RT, rows = min(AFD_RT, G - row0);
    pdl_wait();
    const int token = g.q_start[r], token_end = g.q_start[r + 1], seq_len = g.seq_lens[r];
    const int q_len = token_end - token;
    if (q_len <= 0) return;  // a padding request of a captured step
    const int pos = seq_len - q_len, lowest = key_floor(pos, g.window);
    const int32_t* table = g.tables + (int64_t)r * g.max_blocks;
    const KeyTiles walk = key_tiles(lowest, pos, g.keep, AF_BN);
    const int s_first = walk.kept > 0 ? 0 : walk.first / TPS, s_end = pos < 0 ? 0 : pos / AF_SLICE + 1;
    const bool alone = g.part == nullptr;  // no request has a second slice
    if (!alone && s_first + (int)blockIdx.z >= s_end) return;

    const int64_t to_value = (int64_t)(g.n_kv + hp.value - hp.key) * g.page_size * D;  // from a key to its value
    const int tx = lane & 7, ty = lane >> 3;              // scores: keys 16 warp + tx (+ 8), rows ty (+ 4)
    const int half = tid >> 6 & 1, d = (tid & 63) * 2;   // outputs: rows 4 half .. + 3, elements d and d + 1
    // the output of a row of which the only slice has maximum m, sum l and output v
    auto finish = [&](int row, float m, float l, float v0, float v1) {
        const int h = hp.key * G + row0 + row;
        float tot_m = g.sinks ? g.sinks[h] : -INFINITY, tot_l = g.sinks ? 1.f : 0.f;
        const float2 f = af_join(tot_m, tot_l, m, l);
        float* out = g.out + (int64_t)token * g.out_stride + (int64_t)(u * G + row0 + row) * D + d;
        const float* gate = g.gate ? g.gate + (int64_t)token * g.q_stride + (int64_t)h * D + d : nullptr;
        out[0] = af_finish(af_mix(0.f, f, v0), tot_l, gate);
        out[1] = af_finish(af_mix(0.f, f, v1), tot_l, gate ? gate + 1 : nullptr);
    };
    // (asked for in front of the keys, behind which it would queue)
    float4 query = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < AFD_RT * C4 && tid / C4 < rows) {
        const float* src = g.q + (int64_t)token * g.q_stride + (int64_t)(hp.key * G + row0 + tid / C4) * D + tid % C4 * 4;
        query = make_float4(src[0], src[1], src[2], src[3]);
    }
    bool first = true;
    for (int slice = s_first + (int)blockIdx.z; slice < s_end; slice += (int)gridDim.z) {
        int seen = 0;  // the tiles of the slice that hold a key in sight
#pragma unroll
        for (int t = 0; t < TPS; ++t)
            if (slice * TPS + t < walk.kept || (slice * TPS + t >= walk.first && slice * TPS + t <= pos / AF_BN)) seen |= 1 << t;
        if (seen == 0) continue;
        const bool mine = seen >> (warp / 2) & 1;
        // ---- keys (and values): a warp fetches the 16 whose scores it forms; those out of sight are zero
        int64_t key_at = -1;
        if (mine && lane < 16) {
            const int key = slice * AF_SLICE + warp * 16 + lane;
            if ((key >= lowest || key < g.keep) && key <= pos) {
                const int64_t page = table[key / g.page_size];
                if (page >= g.num_pages) atomicOr(g.err, SS_ERR_PAGE_RANGE);
                else if (page >= 0) key_at = ((page * 2 * g.n_kv + hp.key) * g.page_size + key % g.page_size) * D;
            }
        }
        auto fetch = [&](float* to, int64_t further) {
            // whole rows to an instruction where they fill its lanes, otherwise 8 lanes to a row (359 against 374 us for 20
            // requests behind 16,000 with heads of 128; 339 against 265 for 100 behind 700 with heads of 96)
            constexpr bool WHOLE = 32 % C4 == 0;
            constexpr int LANES = WHOLE ? C4 : 8, RPI = 32 / LANES;
            const int c0 = lane % LANES * 4;
#pragma unroll
            for (int i = 0; i < 16 / RPI; ++i) {
                const int64_t at = __shfl_sync(0xffffffffu, key_at, i * RPI + lane / LANES);
                const float* src = g.kv + (at >= 0 ? at + further + c0 : 0);
                float* dst = to + (warp * 16 + i * RPI + lane / LANES) * KS + c0;
#pragma unroll
                for (int c = 0; c < D; c += LANES * 4)
                    if (WHOLE || c + c0 < D) cp_async16(dst + c, src + c, at >= 0);
            }
        };
        if (!first) __syncthreads();  // everyone is done with the slice before
        if (mine) fetch(Ks, 0);
        cp_async_commit();
        if (BOTH && mine) fetch(Vs, to_value);
        cp_async_commit();
        if (first) {
            if (tid < AFD_RT * C4) *reinterpret_cast<float4*>(&Qs[tid / C4 * KS + tid % C4 * 4]) = query;
            __syncthreads();
            first = false;
        }
        cp_async_wait<1>();
        __syncwarp();

        // ---- scores
        float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        if (mine) {
            const float *q0 = Qs + ty * KS, *k0 = Ks + (warp * 16 + tx) * KS;
#pragma unroll (BOTH ? 8 : 4)
            for (int e = 0; e < D; e += 4) {
                float4 q4[2], k4[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    q4[i] = *reinterpret_cast<const float4*>(q0 + i * 4 * KS + e);
                    k4[i] = *reinterpret_cast<const float4*>(k0 + i * 8 * KS + e);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        s[i][k] = fmaf(q4[i].x, k4[k].x, s[i][k]);
                        s[i][k] = fmaf(q4[i].y, k4[k].y, s[i][k]);
                        s[i][k] = fmaf(q4[i].z, k4[k].z, s[i][k]);
                        s[i][k] = fmaf(q4[i].w, k4[k].w, s[i][k]);
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int key = slice * AF_SLICE + warp * 16 + tx + 8 * k;
                const bool ok = mine && ty + 4 * i < rows && key <= pos && (key >= lowest || key < g.keep);
                const float x = __fmul_rn(s[i][k], g.scale);
                s[i][k] = ok ? (g.softcap > 0.f ? __fmul_rn(g.softcap, tanhf(x / g.softcap)) : x) : -INFINITY;
                top = fmaxf(top, s[i][k]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            if (tx == 0) top_s[warp * AFD_RT + ty + 4 * i] = top;
        }
        __syncthreads();
        if (!BOTH && mine) fetch(Vs, to_value);  // (over the warp's own keys)
        if (!BOTH) cp_async_commit();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = ty + 4 * i;
            float before = -INFINITY, now = -INFINITY;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const float top = top_s[w * AFD_RT + row];
                if (w < (warp & ~1)) before = fmaxf(before, top);
                if (w <= (warp | 1)) now = fmaxf(now, top);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
                Ps[(warp * 16 + tx + 8 * k) * AFD_PS + row] = s[i][k] == -INFINITY ? 0.f : expf(__fsub_rn(s[i][k], now));  // (a NaN has no part in `now`, and stays)
            if (tx == 0 && !(warp & 1)) alpha_s[warp / 2 * AFD_RT + row] = before == -INFINITY ? 0.f : expf(__fsub_rn(before, now));
        }
        cp_async_wait<0>();
        __syncthreads();

        // ---- outputs: warps 0 to 3; meanwhile a lane of warp 4 to each row sums the probabilities
        float acc[4][2], l = 0.f;
        if (warp < 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.f;
            if (d < D)
                for (int t = 0; t < TPS; ++t) {
                    if (!(seen >> t & 1)) continue;
                    if (seen & ((1 << t) - 1)) {
                        const float4 a = *reinterpret_cast<const float4*>(&alpha_s[t * AFD_RT + half * 4]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            acc[0][e] = __fmul_rn(acc[0][e], a.x); acc[1][e] = __fmul_rn(acc[1][e], a.y);
                            acc[2][e] = __fmul_rn(acc[2][e], a.z); acc[3][e] = __fmul_rn(acc[3][e], a.w);
                        }
                    }
#pragma unroll 8
                    for (int k = t * AF_BN; k < (t + 1) * AF_BN; ++k) {
                        const float4 p = *reinterpret_cast<const float4*>(&Ps[k * AFD_PS + half * 4]);
                        const float2 v = *reinterpret_cast<const float2*>(&Vs[k * KS + d]);
                        acc[0][0] = fmaf(p.x, v.x, acc[0][0]); acc[0][1] = fmaf(p.x, v.y, acc[0][1]);
                        acc[1][0] = fmaf(p.y, v.x, acc[1][0]); acc[1][1] = fmaf(p.y, v.y, acc[1][1]);
                        acc[2][0] = fmaf(p.z, v.x, acc[2][0]); acc[2][1] = fmaf(p.z, v.y, acc[2][1]);
                        acc[3][0] = fmaf(p.w, v.x, acc[3][0]); acc[3][1] = fmaf(p.w, v.y, acc[3][1]);
                    }
                }
        } else if (warp == 4 && lane < rows) {
            for (int t = 0; t < TPS; ++t) {
                if (!(seen >> t & 1)) continue;
                if (seen & ((1 << t) - 1)) l = __fmul_rn(l, alpha_s[t * AFD_RT + lane]);
#pragma unroll 16
                for (int k = t * AF_BN; k < (t + 1) * AF_BN; ++k) l = __fadd_rn(l, Ps[k * AFD_PS + lane]);
            }
            float slice_m = -INFINITY;
#pragma unroll
            for (int w = 0; w < 8; ++w) slice_m = fmaxf(slice_m, top_s[w * AFD_RT + lane]);
            if (alone) {
                ml_s[lane * 2] = slice_m;
                ml_s[lane * 2 + 1] = l;
            } else {
                g.part_ml[((int64_t)token * (n_heads * G) + u * G + row0 + lane) * g.max_slices + slice] = make_float2(slice_m, l);
            }
        }
        if (alone) __syncthreads();
        if (warp < 4 && d < D)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = half * 4 + i;
                if (row >= rows) break;
                if (alone) {
                    finish(row, ml_s[row * 2], ml_s[row * 2 + 1], acc[i][0], acc[i][1]);
                } else {
                    const int64_t at = ((int64_t)token * (n_heads * G) + u * G + row0 + row) * g.max_slices + slice;
                    *reinterpret_cast<float2*>(&g.part[at * D + d]) = make_float2(acc[i][0], acc[i][1]);
                }
            }
    }
    if (alone && first && warp < 4 && d < D)  // a request without a key
        for (int i = half * 4; i < min(half * 4 + 4, rows); ++i) finish(i, -INFINITY, 0.f, 0.f, 0.f);
}

// Joins the slices of every row: a block to a (row, output head), a thread to an element.
template <int D>
__global__ void __launch_bounds__((D + 31) / 32 * 32) attn_f32_join_kernel(const AttnF32Args g) {
    pdl_launch_dependents();
    const int d = threadIdx.x, lane = d & 31;
    const int G = g.n_q / g.n_kv, heads = g.across ? g.n_q * g.n_kv : g.n_q;
    const int64_t item = blockIdx.x;
    const int row = (int)(item / heads), h_out = (int)(item % heads);
    const HeadPair hp = head_pair(h_out / G, g.n_kv, g.across);
    const int h = hp.key * G + h_out % G;
    pdl_wait();
    // the request of the row: its own number where every request has one token, otherwise the last that starts at or before it
    int r = row, ends = 0;
    if (row >= g.n_requests || g.q_start[row] != row || (ends = g.q_start[row + 1]) != row + 1) {
        if (row >= g.q_start[g.n_requests]) return;
        int hi = g.n_requests;
        r = 0;
        while (hi - r > 1) {
            const int mid = (r + hi) >> 1;
            if (g.q_start[mid] <= row) r = mid;
            else hi = mid;
        }
        ends = g.q_start[r + 1];
    }
    const int pos = g.seq_lens[r] - (ends - row);
    float m = g.sinks ? g.sinks[h] : -INFINITY, l = g.sinks ? 1.f : 0.f, total = 0.f;
    // the slices that hold a key the row sees: those of the kept keys, then those from its lowest key on
    const int first = key_floor(pos, g.window) / AF_SLICE, last = pos < 0 ? -1 : pos / AF_SLICE;
    const int kept = g.keep > 0 ? min((g.keep - 1) / AF_SLICE + 1, first) : 0;
    const int count = last < 0 ? 0 : kept + last - first + 1;
    const int64_t at0 = item * g.max_slices;
    auto slice_at = [&](int j) { return at0 + (j < kept ? j : first + (j - kept)); };
    // 32 slices at a time, whose loads travel together: their factors side by side, a lane to each (a maximum over those
    // before is the same in any order); what is left to do in order is a product, a product and a sum a slice
    for (int j0 = 0; j0 < count; j0 += 32) {
        const int n = min(32, count - j0);
        float2 ml = make_float2(-INFINITY, 0.f);
        if (lane < n) ml = g.part_ml[slice_at(j0 + lane)];
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if (i % 8 == 0 && i >= n) break;
            v[i] = d < D && i < n ? g.part[slice_at(j0 + i) * D + d] : 0.f;
        }
        float top = ml.x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float below = __shfl_up_sync(0xffffffffu, top, o);
            if (lane >= o) top = fmaxf(top, below);
        }
        const float before = __shfl_up_sync(0xffffffffu, top, 1), all = __shfl_sync(0xffffffffu, top, 31);
        float m_lane = lane == 0 ? m : fmaxf(m, before), l_lane = 0.f;
        const float2 f = af_join(m_lane, l_lane, ml.x, ml.y);
        m = fmaxf(m, all);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if (i >= n) break;
            const float2 fi = make_float2(__shfl_sync(0xffffffffu, f.x, i), __shfl_sync(0xffffffffu, f.y, i));
            l = af_mix(l, fi, __shfl_sync(0xffffffffu, ml.y, i));
            total = af_mix(total, fi, v[i]);
        }
    }
    if (d < D)
        g.out[(int64_t)row * g.out_stride + (int64_t)h_out * D + d] =
            af_finish(total, l, g.gate ? g.gate + (int64_t)row * g.q_stride + (int64_t)h * D + d : nullptr);
}

template <int D>
int launch_attn_f32_join(const AttnF32Args& g, cudaStream_t stream) {
    const int64_t items = (int64_t)g.n_rows * (g.across ? g.n_q * g.n_kv : g.n_q);
    ss_launch(attn_f32_join_kernel<D>, dim3((unsigned)items), dim3((D + 31) / 32 * 32), 0, stream, g);
    return SS_LAUNCH_CHECK();
}

template <int D, int RT>
int launch_attn_f32_rows(const AttnF32Args& g, int n_tiles, int parts, cudaStream_t stream) {
    constexpr int smem = af_smem_bytes<D, RT>();
    static SsPerDevice opted;
    if (int rc = ss_opt_in_smem(attn_f32_kernel<D, RT>, smem, opted)) return rc;
    const int blocks = g.tile_req ? n_tiles * (64 / RT) : g.n_requests * ((g.n_q / g.n_kv + RT - 1) / RT);
    const int heads = g.across ? g.n_kv * g.n_kv : g.n_kv;
    ss_launch(attn_f32_kernel<D, RT>, dim3(blocks * heads, 1, parts), dim3(AF_THREADS), smem, stream, g);
    const int rc = SS_LAUNCH_CHECK();
    return rc || !g.part ? rc : launch_attn_f32_join<D>(g, stream);
}

template <int D, bool BOTH>
int launch_attn_f32_decode(const AttnF32Args& g, dim3 grid, cudaStream_t stream) {
    constexpr int smem = afd_smem_bytes<D, BOTH>();
    static SsPerDevice opted;
    if (int rc = ss_opt_in_smem(attn_f32_decode_kernel<D, BOTH>, smem, opted)) return rc;
    ss_launch(attn_f32_decode_kernel<D, BOTH>, grid, dim3(AFD_THREADS), smem, stream, g);
    return SS_LAUNCH_CHECK();
}

// 32 rows of a prompt portion to a block (64, with 8 warps and half the blocks: 257 us where 32 take 209, 777 tokens at the 7B sizes); a decode
// step's rows of one request in tiles of 16, where attn_f32_decode_kernel does not take them (heads of more than 128, for which it has
// no threads: 64 of them take 2 elements each of a half of the rows; and slices that pass the scratch memory's bound).
template <int D>
int launch_attn_f32(const AttnF32Args& g, int n_tiles, int parts, cudaStream_t stream) {
    if constexpr (D <= 128)
        if (g.tile_req == nullptr && (g.part != nullptr || g.max_slices == 1)) {
            const int G = g.n_q / g.n_kv, heads = g.across ? g.n_kv * g.n_kv : g.n_kv;
            const int64_t blocks = (int64_t)g.n_requests * heads * ((G + AFD_RT - 1) / AFD_RT);
            const dim3 grid((unsigned)blocks, 1, parts);
            const int rc = blocks * parts <= ss_sm_count() ? launch_attn_f32_decode<D, true>(g, grid, stream)
                                                           : launch_attn_f32_decode<D, false>(g, grid, stream);
            return rc || !g.part ? rc : launch_attn_f32_join<D>(g, stream);
        }
    if (g.tile_req == nullptr) return launch_attn_f32_rows<D, 16>(g, n_tiles, parts, stream);
    return launch_attn_f32_rows<D, 32>(g, n_tiles, parts, stream);
}
