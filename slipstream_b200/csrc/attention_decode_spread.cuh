// Decode attention for many requests: the tiles of all requests dealt out evenly.
//
// attn_decode_tma gives a head block of a request (a unit here) one block, or as many as the batch leaves room for; with as many
// units as two blocks an SM or more, one.  Requests differ in length, and the longest one's block is then the kernel's time while
// other SMs stand idle (48 requests of 937 to 2,813 keys, 28 heads on 4 kv heads, 128 elements: 184 MB in 50.9 us; 38.1 so, of which the second kernel is 3).  Here
// all units' tiles of 64 keys, unit after unit, are one row of tiles, which two blocks an SM share evenly: block b takes tiles cut(b) ..
// cut(b + 1) - 1, the end of one unit, whole units, the beginning of another.  Every block works the cuts out for itself from the
// lengths on the device, so a captured step needs nothing refilled when they change.  A unit inside one block is written as it is;
// of a unit that a cut divides, the blocks leave their sums in scratch memory, and a second, small kernel (a block for every cut) combines
// them: no counters and no memory that outlives the call.
//
// Inside a block everything is as in attn_decode_tma (a producer warp that brings tiles by TMA, two pairs of consumer warps, FORM 0's
// options), but the ring of tiles runs on from one unit to the next: while the consumers merge their results and fetch the next unit's
// queries, its tiles are on their way.  So the merge has memory of its own: one row per head, added to by the four warps in turn.
#pragma once

#include "attention_decode_tma.cuh"

#define DS_REQUESTS 512  // at most: their tiles' sums stand in shared memory
#define DS_SNAP 1        // a cut this close to a unit's end moves there: a piece of a tile is not worth its merge

template <int D>
constexpr int decode_spread_stages() { return D == 128 ? 3 : 5; }  // odd (see attn_decode_tma's barriers); two blocks fit on an SM
template <int D>
constexpr int decode_spread_smem_bytes() {
    // alignment slack, tiles, queries or the merge, mbarriers
    return 1024 + decode_spread_stages<D>() * 2 * MMA_BN * D * 2 + 16 * (D + 8) * 4 + 4 * decode_spread_stages<D>() * 8 + 16;
}
struct SpreadArgs {
    DecodeTmaArgs a;
    float* scratch;  // [block][its first piece, its last]: sums [16 heads][D], then maxima and denominators [16][2]
    int4* joins;     // [block]: the unit whose first part is the block's last piece (request, head block), its parts (0: none), its first's place
    int n_requests, n_blocks;
};

// The row of tiles: sums[r] tiles of one head block of the requests before r; unit w = r * per + y.
struct SpreadRow {
    const int* sums;
    int n, per, blocks, total;
    struct Unit {
        int r, y, start, tiles;
    };
    __device__ __forceinline__ Unit unit(int at) const {  // at < total
        int lo = 0, hi = n;  // sums[lo] * per <= at < sums[hi] * per
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (sums[mid] * per <= at) lo = mid;
            else hi = mid;
        }
        Unit u;
        u.r = lo;
        u.tiles = sums[lo + 1] - sums[lo];
        u.y = (at - sums[lo] * per) / u.tiles;
        u.start = sums[lo] * per + u.y * u.tiles;
        return u;
    }
    __device__ __forceinline__ int cut(int b) const {
        const uint64_t part = (uint64_t)total * (uint32_t)b;
        const int at = part >> 32 ? (int)(part / (uint32_t)blocks) : (int)((uint32_t)part / (uint32_t)blocks);
        if (at <= 0 || at >= total) return at;
        const Unit u = unit(at);
        if (at - u.start <= DS_SNAP) return u.start;
        return u.start + u.tiles - at <= DS_SNAP ? u.start + u.tiles : at;
    }
};

__device__ __forceinline__ KeyTiles spread_walk(const DecodeTmaArgs& a, int seq_len) {
    const int pos = seq_len - 1;
    return key_tiles(key_floor(pos, a.window), pos, a.keep, MMA_BN);
}

// Called by all threads of a block; sums holds DS_REQUESTS + 1.
__device__ __forceinline__ SpreadRow spread_row(const SpreadArgs& s, int* sums) {
    const int n = s.n_requests;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int len = s.a.seq_lens[i];
        sums[i + 1] = len > 0 ? spread_walk(s.a, len).count : 0;
    }
    if (threadIdx.x == 0) sums[0] = 0;
    __syncthreads();
    if (threadIdx.x < 32) {
        int before = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + threadIdx.x;
            int v = i < n ? sums[i + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += up;
            }
            if (i < n) sums[i + 1] = before + v;
            before += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    SpreadRow row;
    row.sums = sums;
    row.n = n;
    row.per = s.a.n_kv * ((s.a.n_q / s.a.n_kv + 15) / 16);
    row.blocks = s.n_blocks;
    row.total = sums[n] * row.per;
    return row;
}

template <int N>
struct SpreadQuarter {
    static constexpr int value = N;
};

template <int D>
__global__ void __launch_bounds__(DT_THREADS, 2)
attn_decode_spread(const __grid_constant__ CUtensorMap map_kv, const SpreadArgs s) {
    pdl_launch_dependents();
    constexpr int KSTR = D + 8, HALVES = D / 64, NS = decode_spread_stages<D>();
    constexpr int STAGE = 2 * MMA_BN * D;  // elements: K tile then V tile
    const DecodeTmaArgs& a = s.a;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    bf16* KV = reinterpret_cast<bf16*>(base);
    // the merge, [heads][D + 8]: of up to 8 heads beside the queries, of more in their place, when they are in registers
    float* Om = reinterpret_cast<float*>(KV + NS * STAGE);
    const bool beside = a.n_q / a.n_kv <= 8;
    bf16* Qs = reinterpret_cast<bf16*>(beside ? Om + 8 * KSTR : Om);  // [16][D + 8]
    uint64_t* full = reinterpret_cast<uint64_t*>(Om + 16 * KSTR);
    uint64_t* empty = full + 2 * NS;
    volatile int* gave_up = reinterpret_cast<volatile int*>(empty + 2 * NS);
    auto bar_of = [](int i) { return (i % NS) * 2 + (i & 1); };
    auto phase_of = [](int i) { return i / (2 * NS); };
    __shared__ int sums[DS_REQUESTS + 1];
    __shared__ float cos_s[64], sin_s[64], Mm[4][16], Lm[4][16], Mx[16], Ls[16];
    __shared__ __align__(16) bf16 newest_k[128], newest_v[128];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_q = a.n_q, n_kv = a.n_kv, page_size = a.page_size, window = a.window, keep = a.keep;
    const bool fused = a.fused != 0;
    const int G = n_q / n_kv, hblocks = (G + 15) / 16, half = a.rot_dim / 2;

    if (tid == 128) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kv) : "memory");
    if (tid == 0) {
        for (int i = 0; i < 2 * NS; ++i) { fa::mbar_init(&full[i], 1); fa::mbar_init(&empty[i], 2); }  // a pair of warps per tile
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const SpreadRow row_of_tiles = spread_row(s, sums);  // (with barriers for the whole block)
    const int my_cut = row_of_tiles.cut(blockIdx.x + (lane & 1));  // both at once
    const int begin = __shfl_sync(0xffffffffu, my_cut, 0), end = __shfl_sync(0xffffffffu, my_cut, 1);

    if (warp == 4) {
        // ---------------- producer: see attn_decode_tma; tile at of the row lies in the ring as number at - begin
        if (begin < end) {
            const int ppt = MMA_BN / page_size, p = lane / HALVES, h = lane % HALVES;
            const bool mine = p < ppt;
            const uint64_t once = fa::l2_evict_first_policy();
            bool waited = false, ok = true;
            for (int at = begin; at < end && ok;) {
                const SpreadRow::Unit u = row_of_tiles.unit(at);
                const int stop = min(end, u.start + u.tiles), pos = a.seq_lens[u.r] - 1, kvh = u.y / hblocks;
                const KeyTiles walk = spread_walk(a, pos + 1);
                const int lo = key_floor(pos, window), b_last = pos / page_size;
                const int32_t* table = a.block_tables + (int64_t)u.r * a.max_blocks;
                // the page of tile j that this lane copies; where there is none (behind the newest token, in front of
                // the window), the first that the tile does see
                auto first_of = [&](int j) {
                    const int key = walk.at(j) * MMA_BN;
                    return (key < keep ? key : max(lo, key)) / page_size;
                };
                auto page_of = [&](int j) {
                    const int blk = walk.at(j) * ppt + p, first = first_of(j);
                    return mine ? table[blk >= first && blk <= b_last ? blk : first] : 0;
                };
                int next = page_of(at - u.start);
                for (; at < stop; ++at) {
                    const int j = at - u.start, i = at - begin, st = i % NS;
                    int64_t page = next;
                    if (at + 1 < stop) next = page_of(j + 1);
                    if (i >= NS) ok = __all_sync(0xffffffffu, fa::mbar_wait(&empty[bar_of(i - NS)], phase_of(i - NS) & 1, gave_up));
                    if (!ok) break;
                    if (!fused && j == u.tiles - 1 && !waited) {
                        pdl_wait();  // the newest key and value are written by the kernel before this one
                        waited = true;
                    }
                    if (lane == 0) fa::mbar_expect_tx(&full[bar_of(i)], STAGE * 2);
                    __syncwarp();
                    if (mine) {
                        if (page < 0 || page >= a.num_pages) {
                            if (page >= a.num_pages) atomicOr(a.err, SS_ERR_PAGE_RANGE);
                            page = table[first_of(j)];
                            if (page < 0 || page >= a.num_pages) {
                                atomicOr(a.err, SS_ERR_PAGE_RANGE);
                                page = 0;
                            }
                        }
                        bf16* kd = KV + st * STAGE + h * (MMA_BN * 64) + p * page_size * 64;
                        const int z = (int)(page * 2 * n_kv + kvh);
                        fa::tma_load_3d_once(kd, &map_kv, h * 64, 0, z, &full[bar_of(i)], once);
                        fa::tma_load_3d_once(kd + MMA_BN * D, &map_kv, h * 64, 0, z + n_kv, &full[bar_of(i)], once);
                    }
                }
            }
        }
        // what the join has to do with this block's last piece
        int4 join = make_int4(0, 0, 0, 0);
        if (begin < end && end < row_of_tiles.total) {
            const SpreadRow::Unit u = row_of_tiles.unit(end);
            if (end > u.start && begin <= u.start) {
                const int stop = u.start + u.tiles;
                int c = blockIdx.x + 2;  // the first cut behind the unit's tiles
                for (;; c += 32) {
                    const uint32_t vote = __ballot_sync(0xffffffffu, c + lane >= s.n_blocks || row_of_tiles.cut(min(c + lane, s.n_blocks)) >= stop);
                    if (vote) {
                        c += __ffs(vote) - 1;
                        break;
                    }
                }
                join = make_int4(u.r, u.y, c - (int)blockIdx.x, (int)blockIdx.x * 2 + (begin == u.start ? 0 : 1));
            }
        }
        pdl_wait();  // (the scratch memory may have been another kernel's)
        if (lane == 0) s.joins[blockIdx.x] = join;
        return;
    }

    // ---------------- consumers
    pdl_wait();
    const float scale_log2 = a.scale * 1.4426950408889634f, cap_log2 = a.softcap * 1.4426950408889634f;
    const int pair = warp >> 1, key_off = (warp & 1) * 32;
    SpreadRow::Unit coming = {0, 0, 0, 0};
    int coming_row = 0, coming_len = 0;
    auto look_up = [&](int at) {
        if (at >= end) return;
        coming = row_of_tiles.unit(at);
        coming_row = a.q_start[coming.r];
        coming_len = a.seq_lens[coming.r];
    };
    look_up(begin);
    auto fetch_queries = [&]() {  // of the unit looked up
        const int c_kvh = coming.y / hblocks, c_g0 = (coming.y % hblocks) * 16, c_heads = min(16, G - c_g0);
        const bf16* from = a.q + (int64_t)coming_row * a.q_stride + (int64_t)(c_kvh * G + c_g0) * D;
        for (int c = tid; c < 16 * (D / 8); c += MMA_THREADS) {
            const int row = c / (D / 8), col = (c - row * (D / 8)) * 8;
            const bool there = row < c_heads;
            cp_async16(Qs + row * KSTR + col, from + (int64_t)(there ? row : 0) * D + col, there);
        }
        cp_async_commit();
    };
    if (begin < end) fetch_queries();
    for (int at = begin; at < end;) {
        const SpreadRow::Unit u = coming;
        const int j0 = at - u.start, j1 = min(end, u.start + u.tiles) - u.start - 1, i0 = at - begin;
        const int kvh = u.y / hblocks, g0 = (u.y % hblocks) * 16, heads_here = min(16, G - g0);
        const int row_q = coming_row, pos = coming_len - 1, lo = key_floor(pos, window);
        const KeyTiles walk = spread_walk(a, pos + 1);
        const bool last = j1 == u.tiles - 1;

        if (fused) {
            for (int i = tid; i < half; i += MMA_THREADS) {
                const float angle = __fmul_rn((float)pos, a.inv_freq[i]);
                sincosf(angle, &sin_s[i], &cos_s[i]);
            }
        }
        const int then = at + j1 - j0 + 1;
        look_up(then);
        cp_async_wait<0>();
        asm volatile("bar.sync 1, 128;" ::: "memory");  // queries, sines and cosines
        if (fused) {
            if (half % 8 == 0) {
                for (int idx = tid; idx < 16 * (half / 8); idx += MMA_THREADS) {
                    const int row = idx / (half / 8), c0 = (idx - row * (half / 8)) * 8;
                    bf16* qr = Qs + row * KSTR;
                    uint4 lo4 = *reinterpret_cast<const uint4*>(qr + c0), hi4 = *reinterpret_cast<const uint4*>(qr + c0 + half);
                    bf16* x1 = reinterpret_cast<bf16*>(&lo4);
                    bf16* x2 = reinterpret_cast<bf16*>(&hi4);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float a1 = to_float(x1[e]), a2 = to_float(x2[e]);
                        const float c = cos_s[c0 + e], sn = sin_s[c0 + e];
                        x1[e] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(a1, c), __fmul_rn(-a2, sn)));
                        x2[e] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(a2, c), __fmul_rn(a1, sn)));
                    }
                    *reinterpret_cast<uint4*>(qr + c0) = lo4;
                    *reinterpret_cast<uint4*>(qr + c0 + half) = hi4;
                }
            } else {
                for (int idx = tid; idx < 16 * half; idx += MMA_THREADS) {
                    const int row = idx / half, c0 = idx - row * half;
                    bf16* qr = Qs + row * KSTR;
                    const float x1 = to_float(qr[c0]), x2 = to_float(qr[c0 + half]);
                    const float c = cos_s[c0], sn = sin_s[c0];
                    qr[c0] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x1, c), __fmul_rn(-x2, sn)));
                    qr[c0 + half] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, sn)));
                }
            }
            if (last) {
                // rotate the newest key; keep it and the value for their tile; write both to their page
                const bf16* kn = a.q + (int64_t)row_q * a.q_stride + (int64_t)(n_q + kvh) * D;
                const bf16* vn = kn + (int64_t)n_kv * D;
                const int blk = pos / page_size, off = pos - blk * page_size;
                const int64_t page = a.block_tables[(int64_t)u.r * a.max_blocks + blk];
                const bool there = page >= 0 && page < a.num_pages, wr = g0 == 0 && there;
                if (!there && tid == 0) atomicOr(a.err, SS_ERR_PAGE_RANGE);
                bf16* kc = a.kv + (((wr ? page : 0) * 2 * n_kv + kvh) * page_size + off) * (int64_t)D;
                bf16* vc = kc + (int64_t)n_kv * page_size * D;
                const int tail = D - a.rot_dim;
                for (int idx = tid; idx < half + tail + D; idx += MMA_THREADS) {
                    if (idx < half) {
                        const float x1 = to_float(kn[idx]), x2 = to_float(kn[idx + half]);
                        const float c = cos_s[idx], sn = sin_s[idx];
                        const bf16 o1 = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x1, c), __fmul_rn(-x2, sn)));
                        const bf16 o2 = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, sn)));
                        newest_k[idx] = o1;
                        newest_k[idx + half] = o2;
                        if (wr) { kc[idx] = o1; kc[idx + half] = o2; }
                    } else if (idx < half + tail) {
                        const int d = a.rot_dim + idx - half;
                        const bf16 v = kn[d];
                        newest_k[d] = v;
                        if (wr) kc[d] = v;
                    } else {
                        const int d = idx - half - tail;
                        const bf16 v = vn[d];
                        newest_v[d] = v;
                        if (wr) vc[d] = v;
                    }
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        uint32_t qf[D / 16][4];
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
            ldmatrix_x4(qf[ks], Qs + (lane & 15) * KSTR + ks * 16 + ((lane >> 4) << 3));

        float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
        if (a.sinks && j0 == 0 && warp == 0) {  // the sink's term, one time: in the first warp of the unit's first piece
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = (lane >> 2) + h * 8;
                if (row < heads_here) {
                    m[h] = a.sinks[kvh * G + g0 + row] * 1.4426950408889634f;
                    l[h] = (lane & 3) == 0 ? 1.f : 0.f;
                }
            }
        }
        float o[D / 8][4];
#pragma unroll
        for (int d = 0; d < D / 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;

        // tile i of the ring belongs to pair i & 1; warp & 1 is its half of 32 keys.  Rows without a head (their queries are zero) are not
        // written and need no mask.
        for (int j = j0 + ((pair - i0) & 1); j <= j1; j += 2) {
            const int kt = walk.at(j), i = i0 + j - j0;
            bf16* Ks = KV + (i % NS) * STAGE;
            bf16* Vs = Ks + MMA_BN * D;
            const bool ok = fa::mbar_wait(&full[bar_of(i)], phase_of(i) & 1, gave_up);  // a wait that gives up makes every later one give up at once
            const int half_key = kt * MMA_BN + key_off, prow = pos % MMA_BN;
            if (j == u.tiles - 1 && pos >= half_key && pos < half_key + 32) {
                if (fused) {  // the newest token's row comes from the projection output, not from the page
                    for (int c = lane; c < 2 * (D / 8); c += 32) {
                        const int col = (c % (D / 8)) * 8;
                        if (c < D / 8) *reinterpret_cast<uint4*>(const_cast<bf16*>(tile_at<D, true>(Ks, prow, col))) = *reinterpret_cast<const uint4*>(newest_k + col);
                        else *reinterpret_cast<uint4*>(const_cast<bf16*>(tile_at<D, true>(Vs, prow, col))) = *reinterpret_cast<const uint4*>(newest_v + col);
                    }
                }
                if (ok) {  // values behind the newest token meet a weight of zero, and 0 x inf is not 0: cleared (see attn_decode_tma)
                    const int behind = key_off + 31 - prow;
                    for (int c = lane; c < behind * (D / 8); c += 32) {
                        const int row = prow + 1 + c / (D / 8), col = (c % (D / 8)) * 8;
                        *reinterpret_cast<uint4*>(const_cast<bf16*>(tile_at<D, true>(Vs, row, col))) = make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                __syncwarp();
            }
            if (ok && half_key <= pos) {
                if (half_key + 31 <= pos && half_key >= lo)
                    warp_tile<D, 32, false, true>(qf, Ks, Vs, key_off, kt * MMA_BN, scale_log2, pos, pos, window, m, l, o, cap_log2, keep);
                else
                    warp_tile<D, 32, true, true>(qf, Ks, Vs, key_off, kt * MMA_BN, scale_log2, pos, pos, window, m, l, o, cap_log2, keep);
            }
            __syncwarp();
            if (lane == 0) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the next copy into this stage
                fa::mbar_arrive(&empty[bar_of(i)]);
            }
        }

        // merge the four warps: each adds a quarter of its columns at a time, no two the same quarter, in a fixed order
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
            if ((lane & 3) == 0) {
                Mm[warp][(lane >> 2) + h * 8] = m[h];
                Lm[warp][(lane >> 2) + h * 8] = l[h];
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");  // (and every warp has its queries)
        if (beside && then < end) fetch_queries();  // of the next unit: they arrive meanwhile
        float factor[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = (lane >> 2) + h * 8;
            const float mm = fmaxf(fmaxf(Mm[0][row], Mm[1][row]), fmaxf(Mm[2][row], Mm[3][row]));
            factor[h] = mm != -INFINITY ? fast_exp2(m[h] - mm) : 0.f;
            if (warp == 0 && (lane & 3) == 0) {
                float ll = 0.f;
#pragma unroll
                for (int w = 0; w < 4; ++w) ll = fmaf(Lm[w][row], mm != -INFINITY ? fast_exp2(Mm[w][row] - mm) : 0.f, ll);
                Mx[row] = mm;
                Ls[row] = ll;
            }
        }
        auto add = [&](auto quarter, bool first) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = (lane >> 2) + h * 8;
                if (row < heads_here) {
#pragma unroll
                    for (int c = 0; c < D / 32; ++c) {
                        constexpr int d0 = decltype(quarter)::value * (D / 32);
                        float2* to = reinterpret_cast<float2*>(Om + row * KSTR + (d0 + c) * 8 + ((lane & 3) << 1));
                        float2 v = first ? make_float2(0.f, 0.f) : *to;
                        v.x = fmaf(o[d0 + c][2 * h], factor[h], v.x);
                        v.y = fmaf(o[d0 + c][2 * h + 1], factor[h], v.y);
                        *to = v;
                    }
                }
            }
        };
#pragma unroll 1
        for (int step = 0; step < 4; ++step) {
            switch ((warp + step) & 3) {
                case 0: add(SpreadQuarter<0>(), step == 0); break;
                case 1: add(SpreadQuarter<1>(), step == 0); break;
                case 2: add(SpreadQuarter<2>(), step == 0); break;
                default: add(SpreadQuarter<3>(), step == 0);
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        const bool whole = j0 == 0 && last;
        float* part = s.scratch + ((int64_t)blockIdx.x * 2 + (at == begin ? 0 : 1)) * 16 * (D + 2);
        const int64_t head0 = (int64_t)kvh * G + g0;
        for (int idx = tid; idx < heads_here * (D / 2); idx += MMA_THREADS) {
            const int row = idx / (D / 2), d = (idx - row * (D / 2)) * 2;
            const float ll = Ls[row];
            const float2 v = *reinterpret_cast<const float2*>(Om + row * KSTR + d);
            if (whole) {
                const float inv = ll > 0.f ? 1.f / ll : 0.f;
                float v0 = v.x * inv, v1 = v.y * inv;
                if (a.gate) {
                    const __nv_bfloat162 g2 = *reinterpret_cast<const __nv_bfloat162*>(a.gate + (int64_t)row_q * a.q_stride + (head0 + row) * D + d);
                    v0 = gated<true>(v0, __low2float(g2));
                    v1 = gated<true>(v1, __high2float(g2));
                }
                store_out2(a, (int64_t)row_q * a.out_stride + (head0 + row) * D + d, v0, v1);
            } else {
                *reinterpret_cast<float2*>(part + row * D + d) = v;
                if (d == 0) *reinterpret_cast<float2*>(part + 16 * D + row * 2) = make_float2(Mx[row], ll);
            }
        }
        at = then;
        if (!beside && at < end) {
            asm volatile("bar.sync 1, 128;" ::: "memory");  // the next unit's queries take the merge's place
            fetch_queries();
        }
    }
    if (begin >= end && tid < 16) {  // no sums, for a join that comes past: a denominator that no piece has
        *reinterpret_cast<float2*>(s.scratch + (int64_t)blockIdx.x * 2 * 16 * (D + 2) + 16 * D + tid * 2) = make_float2(-INFINITY, -1.f);
    }
    // rows of requests without a key
    for (int r = blockIdx.x; r < s.n_requests; r += gridDim.x)
        if (a.seq_lens[r] <= 0)
            for (int d = tid * 2; d < n_q * D; d += MMA_THREADS * 2) store_out2(a, (int64_t)a.q_start[r] * a.out_stride + d, 0.f, 0.f);
    if (tid == 0 && *gave_up) atomicOr(a.err, SS_ERR_WAIT_LIMIT);
}

// Behind it: block b combines the unit that begins in block b's last piece, if another block goes on with it.  It needs no shared memory, so its
// blocks already stand on the SMs, waiting, when the last of the blocks above ends; what they do then is two trips to L2 for most
// units (a part's sums, four parts at once).
#define DS_JOIN_THREADS 256
template <int D>
__global__ void __launch_bounds__(DS_JOIN_THREADS)
attn_decode_spread_join(const SpreadArgs s) {
    pdl_launch_dependents();
    const DecodeTmaArgs& a = s.a;
    pdl_wait();
    const int4 join = s.joins[blockIdx.x];
    const int parts = join.z;
    if (parts == 0) return;
    const int G = a.n_q / a.n_kv, hblocks = (G + 15) / 16, kvh = join.y / hblocks, g0 = (join.y % hblocks) * 16, heads_here = min(16, G - g0);
    const int row_q = a.q_start[join.x];
    const int64_t head0 = (int64_t)kvh * G + g0;
    for (int idx = threadIdx.x; idx < heads_here * (D / 4); idx += DS_JOIN_THREADS) {
        const int row = idx / (D / 4), d = (idx - row * (D / 4)) * 4;
        float mx = -INFINITY, den = 0.f;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = 0; k0 < parts; k0 += 4) {
            float2 ml[4];
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int part = k0 + k < parts ? k0 + k : 0;
                const float* p = s.scratch + (int64_t)(part == 0 ? join.w : ((int)blockIdx.x + part) * 2) * 16 * (D + 2);
                ml[k] = *reinterpret_cast<const float2*>(p + 16 * D + row * 2);
                v[k] = *reinterpret_cast<const float4*>(p + row * D + d);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k0 + k >= parts || ml[k].y < 0.f) continue;  // no part, or a block without a tile
                // a piece without a score above -infinity has no weight, but its sums count: those of scores that are not numbers are not either
                const float top = fmaxf(mx, ml[k].x);
                const float old = mx == -INFINITY ? 0.f : fast_exp2(mx - top), now = ml[k].x == -INFINITY ? 0.f : fast_exp2(ml[k].x - top);
                sum.x = fmaf(v[k].x, now, sum.x * old);
                sum.y = fmaf(v[k].y, now, sum.y * old);
                sum.z = fmaf(v[k].z, now, sum.z * old);
                sum.w = fmaf(v[k].w, now, sum.w * old);
                den = fmaf(ml[k].y, now, den * old);
                mx = top;
            }
        }
        const float inv = den > 0.f ? 1.f / den : 0.f;
        float o[4] = {sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv};
        if (a.gate) {
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = gated<true>(o[e], to_float(a.gate[(int64_t)row_q * a.q_stride + (head0 + row) * D + d + e]));
        }
        const int64_t at = (int64_t)row_q * a.out_stride + (head0 + row) * D + d;
        store_out2(a, at, o[0], o[1]);
        store_out2(a, at + 2, o[2], o[3]);
    }
}
