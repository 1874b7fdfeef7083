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
// 777 tokens of two requests, one behind 300 cached ones, 28 heads of 128 on 4: 551 -> 209 us; four decoded tokens behind
// 500 on average, 12 heads of 128 on 2: 266 -> 33 us; 20 behind 800, 28 on 4: 602 -> 102 us.
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

// Joins the slices of every row: a warp to a (row, output head).
template <int D>
__global__ void __launch_bounds__(AF_THREADS) attn_f32_join_kernel(const AttnF32Args g) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int G = g.n_q / g.n_kv, heads = g.across ? g.n_q * g.n_kv : g.n_q;
    const int64_t item = (int64_t)blockIdx.x * (AF_THREADS / 32) + (threadIdx.x >> 5);
    const int row = (int)(item / heads), h_out = (int)(item % heads);
    if (row >= g.n_rows || row >= g.q_start[g.n_requests]) return;
    int lo = 0, hi = g.n_requests;  // the request of the row: the last one that starts at or before it
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (g.q_start[mid] <= row) lo = mid;
        else hi = mid;
    }
    const int r = lo, pos = g.seq_lens[r] - (g.q_start[r + 1] - row);
    const HeadPair hp = head_pair(h_out / G, g.n_kv, g.across);
    const int h = hp.key * G + h_out % G;
    constexpr int NC = (D + 127) / 128;
    float m = g.sinks ? g.sinks[h] : -INFINITY, l = g.sinks ? 1.f : 0.f;
    float tot[NC][4];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) tot[c][e] = 0.f;
    // the slices that hold a key the row sees: those of the kept keys, then those from its lowest key on
    const int first = key_floor(pos, g.window) / AF_SLICE, last = pos < 0 ? -1 : pos / AF_SLICE;
    const int kept = g.keep > 0 ? min((g.keep - 1) / AF_SLICE + 1, first) : 0;
    const int count = last < 0 ? 0 : kept + last - first + 1;
    const int64_t at0 = item * g.max_slices;
    constexpr int AHEAD = 4;
    for (int j0 = 0; j0 < count; j0 += AHEAD) {
        float2 ml[AHEAD];
        float4 v[AHEAD][NC];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
            const int j = j0 + a;
            if (j >= count) break;
            const int64_t at = at0 + (j < kept ? j : first + (j - kept));
            ml[a] = g.part_ml[at];
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if ((lane + 32 * c) * 4 < D) v[a][c] = *reinterpret_cast<const float4*>(&g.part[at * D + (lane + 32 * c) * 4]);
        }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
            if (j0 + a >= count) break;
            const float2 f = af_join(m, l, ml[a].x, ml[a].y);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if ((lane + 32 * c) * 4 >= D) break;
                tot[c][0] = af_mix(tot[c][0], f, v[a][c].x);
                tot[c][1] = af_mix(tot[c][1], f, v[a][c].y);
                tot[c][2] = af_mix(tot[c][2], f, v[a][c].z);
                tot[c][3] = af_mix(tot[c][3], f, v[a][c].w);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = (lane + 32 * c) * 4 + e;
            if (d < D)
                g.out[(int64_t)row * g.out_stride + (int64_t)h_out * D + d] =
                    af_finish(tot[c][e], l, g.gate ? g.gate + (int64_t)row * g.q_stride + (int64_t)h * D + d : nullptr);
        }
}

template <int D, int RT>
int launch_attn_f32_rows(const AttnF32Args& g, int n_tiles, int parts, cudaStream_t stream) {
    constexpr int smem = af_smem_bytes<D, RT>();
    static SsPerDevice opted;
    if (int rc = ss_opt_in_smem(attn_f32_kernel<D, RT>, smem, opted)) return rc;
    const int blocks = g.tile_req ? n_tiles * (64 / RT) : g.n_requests * ((g.n_q / g.n_kv + RT - 1) / RT);
    const int heads = g.across ? g.n_kv * g.n_kv : g.n_kv;
    ss_launch(attn_f32_kernel<D, RT>, dim3(blocks * heads, 1, parts), dim3(AF_THREADS), smem, stream, g);
    if (g.part) {
        const int64_t items = (int64_t)g.n_rows * heads * (g.n_q / g.n_kv);
        ss_launch(attn_f32_join_kernel<D>, dim3((unsigned)((items + AF_THREADS / 32 - 1) / (AF_THREADS / 32))), dim3(AF_THREADS), 0, stream, g);
    }
    return SS_LAUNCH_CHECK();
}

// 32 rows of a prompt portion to a block (64, with 8 warps and half the blocks: 257 us where 32 take 209, 777 tokens at the 7B sizes); a decode
// step's rows of one request in tiles of 16.
template <int D>
int launch_attn_f32(const AttnF32Args& g, int n_tiles, int parts, cudaStream_t stream) {
    if (g.tile_req == nullptr) return launch_attn_f32_rows<D, 16>(g, n_tiles, parts, stream);
    return launch_attn_f32_rows<D, 32>(g, n_tiles, parts, stream);
}
