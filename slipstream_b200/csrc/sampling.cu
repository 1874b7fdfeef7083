// Token selection on the device from float32 logits: arg-max, and the reference's
// sampling chain (slipstream/engine/sampler.py:36-146): repetition penalty, then
// temperature, top-k, top-p, min-p, then a draw from the softmax of what is left.
//
// A thread-block cluster per row (up to 8 blocks, which add their histograms and compare their candidates through
// one another's shared memory); every row carries its own parameters, so greedy and sampled requests share a
// launch.  Differences from the reference, by design:
//  * the draw is a Gumbel-max race (token = argmax(x_i + g_i), g_i = -log(-log u_i))
//    over counter-based Philox4x32-10 uniforms keyed by (seed, draw index, token),
//    which has the distribution of multinomial(softmax(x)) but needs no sort, no
//    prefix sum and no host state; the same (seed, draw index) gives the same
//    token whatever else is in the batch;
//  * top-k and top-p find their threshold in a histogram over the distance from the largest value and among the few
//    values of the bin where it falls (top-p on fixed-point sums, so the result does not depend on the order of atomics);
//    rows for which that does not work out by radix selection on the value bits, among the values of the bin (too many in
//    it) or of the whole row (infinities, NaN).  Either way the threshold is a value's own bits, and tokens that tie with it are all kept;
//  * rows with temperature 0 take the arg-max of the raw logits (filters skipped,
//    as sampler.py:55-56); the lowest index wins ties.
#include "common.cuh"

#define SAMPLE_THREADS 1024  // at most: few rows have an SM to a block; many rows get blocks of half as many threads, two an SM

struct ArgMax {
    float v;
    int i;
};

__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
    // larger value wins; on equal values the lower index wins; NaN never wins
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ __forceinline__ ArgMax block_argmax(ArgMax a, ArgMax* scratch /* >= 33 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgMax b;
        b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
        b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
        a = better(a, b);
    }
    __syncthreads();
    if (lane == 0) scratch[warp] = a;
    __syncthreads();
    if (warp == 0) {
        ArgMax t = lane < nwarps ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ArgMax b;
            b.v = __shfl_xor_sync(0xffffffffu, t.v, o);
            b.i = __shfl_xor_sync(0xffffffffu, t.i, o);
            t = better(t, b);
        }
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// Arg-max in two stages so that a handful of rows still fills the GPU: ARGMAX_CHUNKS blocks per row
// each reduce a slice of the vocabulary to one packed (value, index) word; a second kernel reduces those.
// Packed word: monotone key of the value in the high half, ~index in the low half, so that the largest
// word is the largest value and, among equal values, the lowest index.  NaN never wins.
#define ARGMAX_CHUNKS 32
#define ARGMAX_THREADS 256

__device__ __forceinline__ unsigned long long pack_arg(float v, int i) {
    const uint32_t b = __float_as_uint(v);
    const uint32_t key = (v != v) ? 0u : ((b & 0x80000000u) ? ~b : (b | 0x80000000u));
    return ((unsigned long long)key << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)i);
}

__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
        v = other > v ? other : v;
    }
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned long long t = lane < nwarps ? scratch[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, t, o);
            t = other > t ? other : t;
        }
        if (lane == 0) scratch[0] = t;
    }
    __syncthreads();
    return scratch[0];
}

__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_partial_kernel(const float* __restrict__ logits, unsigned long long* __restrict__ partial, int vocab,
                      int64_t stride) {
    pdl_launch_dependents();  // the next kernel may be scheduled now; it waits for this one itself
    pdl_wait();               // nothing below runs before the kernels before this one are complete
    __shared__ unsigned long long scratch[32];
    const float* row = logits + (int64_t)blockIdx.x * stride;
    const int per = (vocab + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS;
    const int begin = blockIdx.y * per, end = min(vocab, begin + per);
    unsigned long long best = 0ull;
    // eight loads in flight per thread before the first comparison (one at a time, a block's 4,752 logits of a
    // 152,064-word vocabulary were 19 trips to L2: 7.7 us)
    constexpr int BATCH = 8;
    for (int i0 = begin + threadIdx.x; i0 < end; i0 += blockDim.x * BATCH) {
        float v[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int i = i0 + u * blockDim.x;
            v[u] = i < end ? row[i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int i = i0 + u * blockDim.x;
            if (i < end) {
                const unsigned long long w = pack_arg(v[u], i);
                best = w > best ? w : best;
            }
        }
    }
    best = block_max_u64(best, scratch);
    if (threadIdx.x == 0) partial[(int64_t)blockIdx.x * ARGMAX_CHUNKS + blockIdx.y] = best;
}

// status (optional): the device error word; its value goes to out[rows], behind the tokens, so that the one copy
// that brings the tokens to the host also says whether a kernel of the step flagged anything.
__global__ void argmax_final_kernel(const unsigned long long* __restrict__ partial, int32_t* __restrict__ out,
                                    const int* __restrict__ status) {
    pdl_launch_dependents();  // the next kernel may be scheduled now; it waits for this one itself
    pdl_wait();               // nothing below runs before the kernels before this one are complete
    unsigned long long v = partial[(int64_t)blockIdx.x * ARGMAX_CHUNKS + threadIdx.x];  // 32 threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
        v = other > v ? other : v;
    }
    if (threadIdx.x == 0) out[blockIdx.x] = v == 0ull ? 0 : (int32_t)(0xFFFFFFFFu - (uint32_t)(v & 0xFFFFFFFFull));
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) out[gridDim.x] = __ldcg(status);
}

// scratch: rows * ARGMAX_CHUNKS 64-bit words of the caller
extern "C" int ss_argmax(const float* logits, int32_t* out, int rows, int vocab, int64_t stride,
                         unsigned long long* scratch, const int* status, cudaStream_t stream) {
    if (rows <= 0) return 0;
    static_assert(ARGMAX_CHUNKS == 32, "the final kernel reduces one warp of partial results");
    ss_launch(argmax_partial_kernel, dim3(dim3(rows, ARGMAX_CHUNKS)), dim3(ARGMAX_THREADS), 0, stream, logits, scratch, vocab, stride);
    ss_launch(argmax_final_kernel, dim3(rows), dim3(32), 0, stream, scratch, out, status);
    return SS_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- Philox4x32-10

__device__ __forceinline__ void philox4x32_10(uint32_t k0, uint32_t k1, uint32_t c[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
        const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// The Gumbel noise of token i for draw number `draw` of the stream `seed` is -log(-log(u)) with u from output
// i % 4 of Philox with counter (i / 4, draw) and key seed.
__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);  // monotone: larger float, larger key
}

struct SampleShared {
    ArgMax arg[33];
    unsigned long long total[256];  // the block's histogram of one radix step
    unsigned long long word;        // a value the blocks of the cluster show one another
    uint32_t best_key;              // order_key of the best entry of the race in this block so far
    uint32_t pick_digit;
    unsigned long long pick_above;
};

// The best candidate over all blocks of the cluster (every block gets it).
__device__ __forceinline__ ArgMax cluster_argmax(ArgMax a, SampleShared& sh) {
    a = block_argmax(a, sh.arg);
    const uint32_t n = cluster_size();
    if (n == 1) return a;
    if (threadIdx.x == 0) sh.word = ((unsigned long long)__float_as_uint(a.v) << 32) | (uint32_t)a.i;
    cluster_sync_all();
    ArgMax best{-INFINITY, 0x7fffffff};
    for (uint32_t c = 0; c < n; ++c) {
        const unsigned long long w = ld_cluster_u64(&sh.word, c);
        best = better(best, ArgMax{__uint_as_float((uint32_t)(w >> 32)), (int)(uint32_t)w});
    }
    cluster_sync_all();  // sh.word may be written again
    return best;
}

// The sum of a 64-bit value over all threads of all blocks of the cluster (every thread gets it).
__device__ __forceinline__ unsigned long long cluster_sum(unsigned long long v, SampleShared& sh) {
    const int tid = threadIdx.x, warp = tid >> 5, n_warps = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((tid & 31) == 0) sh.total[warp] = v;
    __syncthreads();
    unsigned long long t = 0ull;
    for (int w = 0; w < n_warps; ++w) t += sh.total[w];
    const uint32_t n = cluster_size();
    if (n == 1) {
        __syncthreads();
        return t;
    }
    if (tid == 0) sh.word = t;
    cluster_sync_all();
    unsigned long long all = 0ull;
    for (uint32_t c = 0; c < n; ++c) all += ld_cluster_u64(&sh.word, c);
    cluster_sync_all();
    return all;
}

// value of token i after penalty and temperature
__device__ __forceinline__ float tempered(const float* row, int i, const uint32_t* seen, float penalty, float temperature) {
    float x = row[i];
    if (seen && ((seen[i >> 5] >> (i & 31)) & 1u)) x = x < 0.f ? x * penalty : x / penalty;
    return x / temperature;
}

// Histograms of a radix step.  Every warp has a histogram of its own in shared memory, and a thread adds up
// consecutive elements that fall into the same bin before it touches shared memory: logits share their top
// bits, so a single histogram with one atomic per element meant 150,000 atomics on two or three addresses
// (2 ms for one row).  All sums are integers (counts, or probabilities in fixed point), so the result does
// not depend on the order of the additions.
struct BinRun {
    int digit;
    unsigned long long sum;
};
__device__ __forceinline__ void run_add(BinRun& run, unsigned long long* warp_hist, int digit, unsigned long long w) {
    if (digit == run.digit) {
        run.sum += w;
    } else {
        if (run.sum) atomicAdd(&warp_hist[run.digit], run.sum);
        run.digit = digit;
        run.sum = w;
    }
}
__device__ __forceinline__ void run_flush(BinRun& run, unsigned long long* warp_hist) {
    if (run.sum) atomicAdd(&warp_hist[run.digit], run.sum);
    run.sum = 0ull;
}

// After the warps' histograms are complete: add them up, then find, from bin 255 downwards, the first bin d
// at which base + (sum of the bins above d) + bin d reaches `target`; bin 0 takes what never reaches it.
// Leaves d in sh.pick_digit and base + (sum of the bins above d) in sh.pick_above.  Called by all threads.
__device__ __forceinline__ void select_bin(SampleShared& sh, const unsigned long long* hists, int n_warps,
                                           unsigned long long base, unsigned long long target) {
    const int tid = threadIdx.x, lane = tid & 31;
    __syncthreads();
    if (tid < 256) {
        unsigned long long t = 0ull;
        for (int w = 0; w < n_warps; ++w) t += hists[w * 256 + tid];
        sh.total[tid] = t;
    }
    const uint32_t n_blocks = cluster_size();
    if (n_blocks > 1) {
        // every block adds up the histograms of all blocks, in block order, and so picks the same bin
        cluster_sync_all();
        unsigned long long t = 0ull;
        if (tid < 256)
            for (uint32_t c = 0; c < n_blocks; ++c) t += ld_cluster_u64(&sh.total[tid], c);
        cluster_sync_all();
        if (tid < 256) sh.total[tid] = t;
    }
    __syncthreads();
    if (tid < 32) {
        // lane l owns bins 255 - 8 l ... 248 - 8 l, highest first
        unsigned long long mine[8], lsum = 0ull;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            mine[b] = sh.total[255 - 8 * lane - b];
            lsum += mine[b];
        }
        unsigned long long incl = lsum;  // inclusive sum over lanes 0..l
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        const unsigned long long before = base + incl - lsum;
        const bool reached = before + lsum >= target;
        const uint32_t vote = __ballot_sync(0xffffffffu, reached);
        const int first = vote ? __ffs(vote) - 1 : 31;
        if (lane == first) {
            unsigned long long acc = before;
            int d = 255 - 8 * lane;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                d = 255 - 8 * lane - b;
                if (d == 0 || acc + mine[b] >= target) break;
                acc += mine[b];
            }
            sh.pick_digit = (uint32_t)d;
            sh.pick_above = acc;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------- a row in passes of four tokens a thread

struct SampleRow {
    const float* row;
    const uint32_t* seen;  // tokens under the repetition penalty, or null
    float penalty, temperature;
    int vocab, first, step;  // this thread's groups of four tokens: first, first + step, ...
    bool aligned;            // the row starts on 16 bytes
};

// Calls f(i, v) for this thread's groups: v[0..3] the values of tokens i .. i + 3 (those beyond the vocabulary do not
// exist: see `live`).  Four groups are read before the first is used.
template <typename F>
__device__ __forceinline__ void for_groups(const SampleRow& t, F f) {
    constexpr int BATCH = 4;
    const int groups = (t.vocab + 3) >> 2;
    for (int n0 = t.first; n0 < groups; n0 += t.step * BATCH) {
        float x[BATCH][4];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int i = (n0 + u * t.step) * 4;
            if (i + 3 < t.vocab && t.aligned) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(t.row + i));
                x[u][0] = q.x; x[u][1] = q.y; x[u][2] = q.z; x[u][3] = q.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[u][e] = i + e < t.vocab ? t.row[i + e] : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int i = (n0 + u * t.step) * 4;
            if (i >= t.vocab) break;
            const uint32_t marked = t.seen ? t.seen[i >> 5] >> (i & 31) : 0u;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (marked & (1u << e)) x[u][e] = x[u][e] < 0.f ? x[u][e] * t.penalty : x[u][e] / t.penalty;
                x[u][e] = x[u][e] / t.temperature;
            }
            f(i, x[u], min(4, t.vocab - i));
        }
    }
}

__device__ __forceinline__ float key_value(uint32_t key) {  // the inverse of order_key
    return __uint_as_float(key & 0x80000000u ? key & 0x7fffffffu : ~key);
}

// -log(-log u) of u = (word + 1/2) / 2^24, word a noise word's upper 24 bits.  word + 1/2 has more than a float's 24 bits from
// 2^23 on (the last word's u would be 1 and its noise infinite), so there the noise is formed from 1 - u = (z + 1/2) / 2^24 with
// z = 2^24 - 1 - word, which is exact.
__device__ __forceinline__ float gumbel(uint32_t word) {
    const uint32_t z = 0xffffffu - word;
    const float e = word < 0x800000u ? -logf(((float)word + 0.5f) * (1.0f / 16777216.0f)) : -log1pf(-((float)z + 0.5f) * (1.0f / 16777216.0f));
    return -logf(e);
}

// Token i enters the race with its value plus its Gumbel noise (noise: the four words of its group).  With z as above and n the
// zeros in front of z's 24 bits (24 for z = 0), 1 - u is at least 2^-(n + 1), and -log(-log u) is below -log(1 - u): a token whose
// value plus (n + 1) log 2 is below the best entry cannot win, and its logarithms, most of the work, are not formed.
__device__ __forceinline__ void race(ArgMax& a, float v, int i, const uint32_t* noise, SampleShared& sh) {
    const uint32_t word = noise[i & 3] >> 8;
    const float bound = v + (0.69315f * (float)(__clz(0xffffffu - word) - 7) + 0.01f);
    if (bound < key_value(*(volatile uint32_t*)&sh.best_key)) return;
    const ArgMax entry{v + gumbel(word), i};
    if (entry.v > a.v) atomicMax(&sh.best_key, order_key(entry.v));
    a = better(a, entry);
}
__device__ __forceinline__ void group_noise(uint64_t seed, uint64_t draw, int i, uint32_t (&c)[4]) {
    c[0] = (uint32_t)(i >> 2); c[1] = (uint32_t)draw; c[2] = (uint32_t)(draw >> 32); c[3] = 0x51195u;
    philox4x32_10((uint32_t)seed, (uint32_t)(seed >> 32), c);
}

#define SAMPLE_BINS 1024
#define SAMPLE_LIST 1024      // values of the threshold's bin that a block keeps
#define SAMPLE_GATHERED 4096  // ... and all blocks of a row together
#define SAMPLE_COUNTED 512    // entries that are compared with one another; more are sorted
#define SAMPLE_SHARE (1 << 18)  // values of 14 bits that a block can add up in 32

struct SampleBins {
    uint32_t parts[3][SAMPLE_BINS];         // a block's histogram: counts, or 14 bits of the mass each (see SAMPLE_SHARE)
    unsigned long long own[SAMPLE_BINS];    // the same added up
    unsigned long long sums[SAMPLE_THREADS / 32];
    unsigned long long before, inside;      // where the threshold falls: what lies in the bins in front of its bin, and in it
    int bin;
};
struct SampleGathered {
    float v[SAMPLE_GATHERED];
    int i[SAMPLE_GATHERED];
    unsigned long long mass[SAMPLE_GATHERED];
};
struct SampleFast {
    union {
        SampleBins bins;
        SampleGathered all;  // block 0 of a row
    };
    unsigned long long list[SAMPLE_LIST];  // value bits, token
    int count;
    float lo[SAMPLE_THREADS / 32], hi[SAMPLE_THREADS / 32];
    unsigned long long mass_all;
};

// Largest and smallest value over all blocks of a row.
__device__ __forceinline__ float2 cluster_range(float hi, float lo, SampleShared& sh, SampleFast& fast) {
    const int tid = threadIdx.x;
    hi = warp_max(hi);
    lo = -warp_max(-lo);
    __syncthreads();
    if ((tid & 31) == 0) { fast.hi[tid >> 5] = hi; fast.lo[tid >> 5] = lo; }
    __syncthreads();
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { hi = fmaxf(hi, fast.hi[w]); lo = fminf(lo, fast.lo[w]); }
    const uint32_t n = cluster_size();
    if (n == 1) return make_float2(hi, lo);
    if (tid == 0) sh.word = ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
    cluster_sync_all();
    for (uint32_t c = 0; c < n; ++c) {
        const unsigned long long w = ld_cluster_u64(&sh.word, c);
        hi = fmaxf(hi, __uint_as_float((uint32_t)(w >> 32)));
        lo = fminf(lo, __uint_as_float((uint32_t)w));
    }
    cluster_sync_all();
    return make_float2(hi, lo);
}

#define SAMPLE_FIX 1099511627776.0f  // 2^40: exp() in (0, 1] as fixed point

__device__ __forceinline__ int sample_bin(float v, float vmax, float scale) {
    return (int)fminf((vmax - v) * scale, (float)(SAMPLE_BINS - 1));
}

// What draw_fast found of a row before it gave it up for the length of its lists: the bin of the threshold, and how much of the
// target (a count, or a mass without top-k) lies in front of it.
struct SampleKnown {
    bool is;
    int bin;
    float scale, vmax;
    unsigned long long base, target;
};

// Decides about a long list (all of it in block 0): its values in order, the largest first, those stay that stand in front of the first of
// equal values with k or more in front of it, or with top_p of the mass, and they race.  Up to 66 steps of Batcher's bitonic network where
// comparing all with all takes 0.2 us for every thousand pairs (64 rows, top-k 2,000 and top-p 0.9: 879 us, 114 so).
__device__ __noinline__ ArgMax draw_from_sorted(SampleFast& fast, int total, int k, unsigned long long base, float tp, bool all_of_it,
                                                unsigned long long target, float vmax, float floor_val, uint64_t seed, uint64_t draw, ArgMax a,
                                                SampleShared& sh) {
    SampleGathered& g = fast.all;
    unsigned long long* entry = g.mass;  // key, token
    unsigned long long* mass = reinterpret_cast<unsigned long long*>(g.v);  // over v and i
    const int tid = threadIdx.x;
    int room = 2 * SAMPLE_COUNTED;  // the next power of two, filled up with what is below every key
    while (room < total) room *= 2;
    __syncthreads();  // the list is there
    for (int j = tid; j < room; j += blockDim.x) entry[j] = j < total ? ((unsigned long long)order_key(g.v[j]) << 32) | (uint32_t)g.i[j] : 0ull;
    for (int run = 2; run <= room; run *= 2)
        for (int apart = run / 2; apart > 0; apart /= 2) {
            __syncthreads();
            for (int p = tid; p < room / 2; p += blockDim.x) {
                const int i = 2 * p - (p & (apart - 1));
                const unsigned long long x = entry[i], y = entry[i + apart];
                if ((x < y) == ((i & run) == 0)) {
                    entry[i] = y;
                    entry[i + apart] = x;
                }
            }
        }
    if (tid == 0) fast.count = total;  // how many stay
    __syncthreads();
    auto opens = [&](int j) { return j == 0 || (uint32_t)(entry[j] >> 32) != (uint32_t)(entry[j - 1] >> 32); };
    if (k > 0) {
        for (int j = tid; j < total; j += blockDim.x)
            if (opens(j) && (unsigned long long)j + base >= (unsigned long long)k) atomicMin(&fast.count, j);
        __syncthreads();
    }
    int stay = fast.count;
    if (tp < 1.0f) {  // each thread a run of neighbours: what lies in front of them, then entry by entry
        const int share = (stay + (int)blockDim.x - 1) / (int)blockDim.x, j0 = min(stay, tid * share), j1 = min(stay, j0 + share);
        unsigned long long own = 0ull;
        for (int j = j0; j < j1; ++j) {
            mass[j] = (unsigned long long)(expf(key_value((uint32_t)(entry[j] >> 32)) - vmax) * SAMPLE_FIX);
            own += mass[j];
        }
        unsigned long long incl = own, front = 0ull, held = 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
            if ((tid & 31) >= o) incl += up;
        }
        if ((tid & 31) == 31) sh.total[tid >> 5] = incl;
        __syncthreads();
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            if (w < (tid >> 5)) front += sh.total[w];
            held += sh.total[w];
        }
        front += incl - own;
        const unsigned long long limit = all_of_it ? (unsigned long long)((double)tp * (double)held) : target - base;
        for (int j = j0; j < j1; ++j) {
            if (front >= limit && opens(j)) {
                atomicMin(&fast.count, j);
                break;
            }
            front += mass[j];
        }
        __syncthreads();
        stay = fast.count;
    }
    for (int j = tid; j < stay; j += blockDim.x) {
        const float v = key_value((uint32_t)(entry[j] >> 32));
        const int i = (int)(uint32_t)entry[j];
        if (!(v >= floor_val)) continue;
        uint32_t c[4];
        group_noise(seed, draw, i, c);
        race(a, v, i, c, sh);
    }
    return a;
}

// The draw of a row under top-k or top-p in three passes.  (1) the largest and the smallest value; (2) a histogram over
// the distance from the largest: a larger value never falls into a later bin, so the bin in which the k-th value stands, or in
// which the mass reaches top_p, holds the threshold; (3) values in front of that bin race, those in it are listed (under both
// filters all of them are listed), and block 0 decides value by value which of the list stay: a value stays while what is
// larger than it counts less than k, or holds less than top_p of the mass (`draw_from_sorted` where they are many).  Returns false
// where a step does not work out; nothing has been decided then, but `known` says where the threshold falls if it got so far.  Bound by
// issue (an exponential and up to three shared-memory additions a value) and the pass's way to L2.  64 rows of 152,064 logits, against
// radix selection with a histogram a digit (four passes for top-k, five for top-p, each forming the values anew): top-k 40 223 -> 65
// us, top-p 0.8 314 -> 98, both 377 -> 66.
__device__ __forceinline__ bool draw_fast(const SampleRow& t, int k, float tp, float mp, uint64_t seed, uint64_t draw, SampleShared& sh,
                                          SampleFast& fast, SampleKnown& known, ArgMax& best) {
    const int tid = threadIdx.x;
    const uint32_t n_blocks = cluster_size(), rank = cluster_rank();
    // (a vocabulary of more than 262,144 and a block to a row, say)
    if (k <= 0 && (int64_t)((t.vocab + 4 * t.step - 1) / (4 * t.step)) * 4 * blockDim.x > SAMPLE_SHARE) return false;
    float hi = -INFINITY, lo = INFINITY;
    for_groups(t, [&](int, const float (&v)[4], int live) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e >= live) break;
            hi = v[e] == v[e] ? fmaxf(hi, v[e]) : INFINITY;  // NaN: not here
            if (v[e] != -INFINITY) lo = fminf(lo, v[e]);
        }
    });
    const float2 range = cluster_range(hi, lo, sh, fast);
    const float vmax = range.x;
    if (!(fabsf(vmax) < INFINITY) || !(range.x - range.y < INFINITY)) return false;
    const float scale = range.x > range.y ? (float)SAMPLE_BINS / fminf(range.x - range.y, 32.f) : 1.f;
    auto bin_of = [&](float v) { return sample_bin(v, vmax, scale); };
    const bool counting = k > 0, list_all = counting && tp < 1.0f;  // top-p among the top k needs all of them

    SampleBins& b = fast.bins;
    for (int i = tid; i < 3 * SAMPLE_BINS; i += blockDim.x) (&b.parts[0][0])[i] = 0u;
    if (tid == 0) fast.count = 0;
    __syncthreads();
    for_groups(t, [&](int, const float (&v)[4], int live) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e >= live) break;
            const int at = bin_of(v[e]);
            if (counting) {
                atomicAdd(&b.parts[0][at], 1u);
            } else {
                const unsigned long long w = (unsigned long long)(expf(v[e] - vmax) * SAMPLE_FIX);
                if (w & 0x3fffu) atomicAdd(&b.parts[0][at], (uint32_t)w & 0x3fffu);
                if ((w >> 14) & 0x3fffu) atomicAdd(&b.parts[1][at], (uint32_t)(w >> 14) & 0x3fffu);
                if (w >> 28) atomicAdd(&b.parts[2][at], (uint32_t)(w >> 28));
            }
        }
    });
    __syncthreads();
    constexpr int MOST = 2;  // bins of a thread, neighbours: 1,024 or 512 threads
    const int per = SAMPLE_BINS / (int)blockDim.x;
    unsigned long long mine[MOST] = {0ull, 0ull};
#pragma unroll
    for (int u = 0; u < MOST; ++u) {
        if (u >= per) break;
        const int i = tid * per + u;
        mine[u] = (unsigned long long)b.parts[0][i] + ((unsigned long long)b.parts[1][i] << 14) + ((unsigned long long)b.parts[2][i] << 28);
        b.own[i] = mine[u];
    }
    if (n_blocks > 1) {
        cluster_sync_all();
        for (int u = 0; u < MOST; ++u) mine[u] = 0ull;
        for (uint32_t c = 0; c < n_blocks; ++c)
#pragma unroll
            for (int u = 0; u < MOST; ++u)
                if (u < per) mine[u] += ld_cluster_u64(&b.own[tid * per + u], c);
        cluster_sync_all();
    }
    // what lies in front of each bin
    unsigned long long sum = 0ull;
#pragma unroll
    for (int u = 0; u < MOST; ++u) sum += mine[u];
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += up;
    }
    if ((tid & 31) == 31) b.sums[tid >> 5] = incl;
    __syncthreads();
    unsigned long long all = 0ull, before = incl - sum;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        if (w < (tid >> 5)) before += b.sums[w];
        all += b.sums[w];
    }
    const unsigned long long target = counting ? (unsigned long long)k : (unsigned long long)((double)tp * (double)all);
    if (tid == 0) { b.bin = -1; b.before = 0ull; }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < MOST; ++u) {
        if (u >= per) break;
        if (before < target && before + mine[u] >= target) { b.bin = tid * per + u; b.before = before; b.inside = mine[u]; }
        before += mine[u];
    }
    __syncthreads();
    const int bin = b.bin;
    const unsigned long long base = b.before;
    if (bin < 0) return false;  // (the same in every block)
    known = SampleKnown{false, bin, scale, vmax, base, target};
    // (a mass does not tell of how many values it is)
    if (counting && (list_all ? base + b.inside : b.inside) > (unsigned long long)min(SAMPLE_GATHERED, (int)n_blocks * SAMPLE_LIST)) {
        known.is = true;
        return false;
    }

    const float floor_val = mp > 0.0f ? vmax + logf(mp) : -INFINITY;  // min-p: exp(x - x_max) >= min_p
    ArgMax a{-INFINITY, 0x7fffffff};
    for_groups(t, [&](int i, const float (&v)[4], int live) {
        bool races = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e >= live) break;
            const int at = bin_of(v[e]);
            if (list_all ? at <= bin : at == bin) {
                const int place = atomicAdd(&fast.count, 1);
                if (place < SAMPLE_LIST) fast.list[place] = ((unsigned long long)__float_as_uint(v[e]) << 32) | (uint32_t)(i + e);
            }
            races |= !list_all && at < bin && v[e] >= floor_val;
        }
        if (races) {
            uint32_t c[4];
            group_noise(seed, draw, i, c);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e < live && bin_of(v[e]) < bin && v[e] >= floor_val) race(a, v[e], i + e, c, sh);
        }
    });
    __syncthreads();
    // block 0 gathers the lists
    if (tid == 0) sh.word = (unsigned long long)fast.count;
    if (n_blocks > 1) cluster_sync_all();
    else __syncthreads();
    int total = 0;
    bool fits = true;
    for (uint32_t c = 0; c < n_blocks; ++c) {
        const int n = n_blocks > 1 ? (int)ld_cluster_u64(&sh.word, c) : (int)sh.word;
        fits = fits && n <= SAMPLE_LIST;
        total += n;
    }
    fits = fits && total <= SAMPLE_GATHERED;
    if (!fits) {
        if (n_blocks > 1) cluster_sync_all();  // sh.word may be written again
        __syncthreads();
        known.is = true;
        return false;
    }
    if (rank == 0) {
        SampleGathered& g = fast.all;  // (in place of the histogram, which everyone is done with)
        int at = 0;
        for (uint32_t c = 0; c < n_blocks; ++c) {
            const int n = n_blocks > 1 ? (int)ld_cluster_u64(&sh.word, c) : (int)sh.word;
            for (int j = tid; j < n; j += blockDim.x) {
                const unsigned long long w = n_blocks > 1 ? ld_cluster_u64(&fast.list[j], c) : fast.list[j];
                g.v[at + j] = __uint_as_float((uint32_t)(w >> 32));
                g.i[at + j] = (int)(uint32_t)w;
            }
            at += n;
        }
        if (total > SAMPLE_COUNTED) {
            a = draw_from_sorted(fast, total, counting ? k : 0, list_all ? 0ull : base, tp, list_all, target, vmax, floor_val, seed, draw, a, sh);
            total = 0;  // (nothing is left to do below)
        }
        if (tid == 0) fast.mass_all = 0ull;
        __syncthreads();
        // values that stay under top-k have their mass, the others none
        unsigned long long held = 0ull;
        for (int j = tid; j < total; j += blockDim.x) {
            const float v = g.v[j];
            bool stays = true;
            if (counting) {
                const uint32_t key = order_key(v);
                int larger = 0;
                for (int o = 0; o < total; ++o) larger += order_key(g.v[o]) > key;
                stays = (unsigned long long)larger + (list_all ? 0ull : base) < (unsigned long long)k;
            }
            const unsigned long long w = stays ? (unsigned long long)(expf(v - vmax) * SAMPLE_FIX) : 0ull;
            g.mass[j] = w;
            if (!stays) g.i[j] = -1;
            held += w;
        }
        unsigned long long limit = target, above = base;
        if (list_all) {
            if (held) atomicAdd(&fast.mass_all, held);
            __syncthreads();
            limit = (unsigned long long)((double)tp * (double)fast.mass_all);
            above = 0ull;
        }
        __syncthreads();
        for (int j = tid; j < total; j += blockDim.x) {
            const float v = g.v[j];
            const int i = g.i[j];
            if (i < 0 || !(v >= floor_val)) continue;
            if (tp < 1.0f) {
                const uint32_t key = order_key(v);
                unsigned long long larger = above;
                for (int o = 0; o < total; ++o) larger += order_key(g.v[o]) > key ? g.mass[o] : 0ull;
                if (larger >= limit) continue;
            }
            uint32_t c[4];
            group_noise(seed, draw, i, c);
            race(a, v, i, c, sh);
        }
    }
    if (n_blocks > 1) cluster_sync_all();  // the lists have been read
    best = a;
    return true;
}

// The keys between which a threshold lies, and the leading bytes that they share, which need no radix step.
struct KeyRange {
    uint32_t hi, lo;
};
struct RadixStart {
    uint32_t prefix, mask;
    int shift;
};
__device__ __forceinline__ RadixStart radix_start(KeyRange a) {
    const int same = a.lo == a.hi ? 4 : __clz(a.lo ^ a.hi) >> 3;
    const uint32_t mask = same == 0 ? 0u : 0xffffffffu << (32 - 8 * same);
    return RadixStart{a.lo & mask, mask, 24 - 8 * same};
}

// The largest and the smallest key over all threads of all blocks of the cluster.
__device__ __forceinline__ KeyRange cluster_key_range(KeyRange a, SampleShared& sh) {
    const int tid = threadIdx.x;
    a.hi = __reduce_max_sync(0xffffffffu, a.hi);
    a.lo = __reduce_min_sync(0xffffffffu, a.lo);
    __syncthreads();
    if ((tid & 31) == 0) sh.total[tid >> 5] = ((unsigned long long)a.hi << 32) | a.lo;
    __syncthreads();
    const uint32_t n = cluster_size();
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        a.hi = max(a.hi, (uint32_t)(sh.total[w] >> 32));
        a.lo = min(a.lo, (uint32_t)sh.total[w]);
    }
    if (n > 1) {
        if (tid == 0) sh.word = ((unsigned long long)a.hi << 32) | a.lo;
        cluster_sync_all();
        for (uint32_t c = 0; c < n; ++c) {
            const unsigned long long w = ld_cluster_u64(&sh.word, c);
            a.hi = max(a.hi, (uint32_t)(w >> 32));
            a.lo = min(a.lo, (uint32_t)w);
        }
        cluster_sync_all();
    }
    __syncthreads();
    return a;
}

// The thresholds of top-k and top-p by radix selection: the smallest key that stays, and the largest value where it is wanted.  Where `known` has
// the bin, a pass finds the keys between which its values lie (and whether top-k removes anything that can be drawn), and the
// selection goes on among them: values that share their leading bytes, or are one value, need fewer steps or none.  A
// function of its own, not in the way of the rows that do without it.
struct SampleFloor {
    uint32_t key;
    float vmax;
};
__device__ __noinline__ SampleFloor radix_floor(const SampleRow t, int k, float tp, bool wants_max, const SampleKnown known,
                                                unsigned long long* warp_hists, SampleShared& sh) {
    const float *row = t.row, pen = t.penalty, temp = t.temperature;
    const uint32_t* seen = t.seen;
    const int vocab = t.vocab, first = t.first, step = t.step, tid = threadIdx.x, n_warps = blockDim.x >> 5;
    unsigned long long* my_hist = warp_hists + (tid >> 5) * 256;
    uint32_t floor_key = 0;
    KeyRange within{0xffffffffu, 0u};
    const bool counted = k > 0;  // (what is known is a count)
    float vmax = known.vmax;
    if (known.is) {
        uint32_t hi = 0u, lo = 0xffffffffu, values = 0u;
        for_groups(t, [&](int, const float (&v)[4], int live) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (e >= live || v[e] == -INFINITY) continue;
                ++values;
                if (sample_bin(v[e], known.vmax, known.scale) != known.bin) continue;
                hi = max(hi, order_key(v[e]));
                lo = min(lo, order_key(v[e]));
            }
        });
        within = cluster_key_range(KeyRange{hi, lo}, sh);
        if (counted && cluster_sum((unsigned long long)values, sh) <= (unsigned long long)k) k = 0;
    }

    // ---- top-k: key of the k-th largest value
    if (k > 0) {
        const RadixStart from = radix_start(within);
        uint32_t prefix = from.prefix, mask = from.mask;
        unsigned long long want = (unsigned long long)k - (known.is ? known.base : 0ull);  // rank still to find inside the prefix
        for (int shift = from.shift; shift >= 0; shift -= 8) {
            for (int b = tid; b < n_warps * 256; b += blockDim.x) warp_hists[b] = 0ull;
            __syncthreads();
            BinRun run{0, 0ull};
            for (int i = first; i < vocab; i += step) {
                const uint32_t key = order_key(tempered(row, i, seen, pen, temp));
                if ((key & mask) == prefix && key >= within.lo && key <= within.hi) run_add(run, my_hist, (int)((key >> shift) & 255u), 1ull);
            }
            run_flush(run, my_hist);
            select_bin(sh, warp_hists, n_warps, 0ull, want);
            prefix |= sh.pick_digit << shift;
            mask |= 255u << shift;
            want -= sh.pick_above;
            __syncthreads();
        }
        floor_key = prefix;
    }

    // ---- maximum of what is left (needed by top-p and min-p)
    if (wants_max && !known.is) {
        ArgMax a{-INFINITY, 0x7fffffff};
        for (int i = first; i < vocab; i += step) {
            const float v = tempered(row, i, seen, pen, temp);
            if (order_key(v) >= floor_key) a = better(a, ArgMax{v, i});
        }
        vmax = cluster_argmax(a, sh).v;
    }

    // ---- top-p: keep a token iff the mass of strictly larger values is below top_p
    if (tp < 1.0f) {
        unsigned long long limit = known.target, above = known.base;  // above: mass of values whose key exceeds every key under the prefix
        if (!known.is || counted) {
            unsigned long long local = 0;  // total mass
            for (int i = first; i < vocab; i += step) {
                const float v = tempered(row, i, seen, pen, temp);
                if (order_key(v) >= floor_key) local += (unsigned long long)(expf(v - vmax) * SAMPLE_FIX);
            }
            const unsigned long long total = cluster_sum(local, sh);
            limit = (unsigned long long)((double)tp * (double)total);
            above = 0ull;
            within = KeyRange{0xffffffffu, floor_key};
        }
        __syncthreads();
        const RadixStart from = radix_start(within);
        uint32_t prefix = from.prefix, mask = from.mask;
        for (int shift = from.shift; shift >= 0; shift -= 8) {
            for (int b = tid; b < n_warps * 256; b += blockDim.x) warp_hists[b] = 0ull;
            __syncthreads();
            BinRun run{0, 0ull};
            for (int i = first; i < vocab; i += step) {
                const float v = tempered(row, i, seen, pen, temp);
                const uint32_t key = order_key(v);
                if (key >= within.lo && key <= within.hi && (key & mask) == prefix)
                    run_add(run, my_hist, (int)((key >> shift) & 255u), (unsigned long long)(expf(v - vmax) * SAMPLE_FIX));
            }
            run_flush(run, my_hist);
            // lowest digit whose bin still starts below the limit
            select_bin(sh, warp_hists, n_warps, above, limit);
            prefix |= sh.pick_digit << shift;
            mask |= 255u << shift;
            above = sh.pick_above;
            __syncthreads();
        }
        if (prefix > floor_key) floor_key = prefix;
    }
    return SampleFloor{floor_key, vmax};
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int64_t stride, int32_t* __restrict__ out,
              const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ min_p,
              const float* __restrict__ penalty, const int64_t* __restrict__ seeds,
              const int64_t* __restrict__ draws, uint32_t* __restrict__ seen_all,
              int seen_words, const int32_t* __restrict__ slots, int vocab, const int* __restrict__ status,
              int rows) {
    pdl_launch_dependents();  // the next kernel may be scheduled now; it waits for this one itself
    pdl_wait();               // nothing below runs before the kernels before this one are complete
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) out[rows] = __ldcg(status);  // as in arg-max
    __shared__ SampleShared sh;
    extern __shared__ unsigned long long warp_hists[];  // [warps][256], or SampleFast
    SampleFast& fast = *reinterpret_cast<SampleFast*>(warp_hists);
    // the blocks of a cluster share a row; block c of n takes elements (or groups of four) c * blockDim + tid, + n * blockDim, ...
    const int n_blocks = (int)cluster_size(), rank = (int)cluster_rank();
    const int r = blockIdx.x / n_blocks, tid = threadIdx.x;
    const int first = rank * blockDim.x + tid, step = n_blocks * blockDim.x;
    const float* row = logits + (int64_t)r * stride;
    const float temp = temperature[r];
    uint32_t* seen_row = (seen_all && slots && slots[r] >= 0) ? seen_all + (int64_t)slots[r] * seen_words : nullptr;

    if (tid == 0) sh.best_key = 0u;  // below every value's
    __syncthreads();

    if (temp == 0.f || top_k[r] == 1) {  // greedy: raw logits, no filters
        ArgMax a{-INFINITY, 0x7fffffff};
        const SampleRow t{row, nullptr, 1.f, 1.f, vocab, first, step, (reinterpret_cast<uintptr_t>(row) & 15) == 0};
        for_groups(t, [&](int i, const float (&v)[4], int live) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e < live) a = better(a, ArgMax{v[e], i + e});
        });
        a = cluster_argmax(a, sh);
        if (tid == 0 && rank == 0) {
            const int tok = a.i == 0x7fffffff ? 0 : a.i;
            out[r] = tok;
            if (seen_row) atomicOr(&seen_row[tok >> 5], 1u << (tok & 31));
        }
        return;
    }

    const float pen = penalty[r];
    const uint32_t* seen = (seen_row && pen != 1.0f) ? seen_row : nullptr;
    const int k = top_k[r] > 0 && top_k[r] < vocab ? top_k[r] : 0;
    const float tp = top_p[r], mp = min_p[r];
    const uint64_t seed = (uint64_t)seeds[r], draw = (uint64_t)draws[r];
    SampleKnown known{false, 0, 0.f, -INFINITY, 0ull, 0ull};
    if (k > 0 || tp < 1.0f) {
        const SampleRow t{row, seen, pen, temp, vocab, first, step, (reinterpret_cast<uintptr_t>(row) & 15) == 0};
        ArgMax a;
        if (draw_fast(t, k, tp, mp, seed, draw, sh, fast, known, a)) {
            a = cluster_argmax(a, sh);
            if (tid == 0 && rank == 0) {
                const int tok = a.i == 0x7fffffff ? 0 : a.i;
                out[r] = tok;
                if (seen_row) atomicOr(&seen_row[tok >> 5], 1u << (tok & 31));
            }
            return;
        }
        __syncthreads();
    }
    const SampleRow t{row, seen, pen, temp, vocab, first, step, (reinterpret_cast<uintptr_t>(row) & 15) == 0};
    SampleFloor least{0u, -INFINITY};  // tokens with order_key(value) < least.key are removed
    if (k > 0 || tp < 1.0f || mp > 0.0f) least = radix_floor(t, k, tp, tp < 1.0f || mp > 0.0f, known, warp_hists, sh);

    // ---- min-p: p_i / p_max = exp(x_i - x_max) >= min_p
    float floor_val = -INFINITY;
    if (mp > 0.0f) floor_val = least.vmax + logf(mp);

    // ---- Gumbel-max draw over what is left: one Philox call gives the noise of four consecutive tokens
    ArgMax a{-INFINITY, 0x7fffffff};
    for_groups(t, [&](int i, const float (&v)[4], int live) {
        bool races = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) races |= e < live && order_key(v[e]) >= least.key && v[e] >= floor_val;
        if (!races) return;
        uint32_t c[4];
        group_noise(seed, draw, i, c);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (e < live && order_key(v[e]) >= least.key && v[e] >= floor_val) race(a, v[e], i + e, c, sh);
    });
    a = cluster_argmax(a, sh);
    if (tid == 0 && rank == 0) {
        const int tok = a.i == 0x7fffffff ? 0 : a.i;
        out[r] = tok;
        if (seen_row) atomicOr(&seen_row[tok >> 5], 1u << (tok & 31));
    }
}

extern "C" int ss_sample(const float* logits, int64_t stride, int32_t* out, const float* temperature,
                         const int32_t* top_k, const float* top_p, const float* min_p,
                         const float* penalty, const int64_t* seeds, const int64_t* draws,
                         uint32_t* seen, int seen_words, const int32_t* slots, int rows, int vocab,
                         const int* status, cudaStream_t stream) {
    if (rows <= 0) return 0;
    constexpr int hists = (SAMPLE_THREADS / 32) * 256 * 8;  // a histogram per warp
    constexpr int smem = hists > (int)sizeof(SampleFast) ? hists : (int)sizeof(SampleFast);
    static SsPerDevice opted;
    if (int rc_smem = ss_opt_in_smem(sample_kernel, smem, opted)) return rc_smem;
    // blocks per row: as many as fill the GPU once (two blocks of 512 threads fit on an SM), at most 8
    int per_row = (2 * ss_sm_count()) / rows;
    const int threads = 8 * rows <= ss_sm_count() ? SAMPLE_THREADS : SAMPLE_THREADS / 2;
    per_row = per_row >= 8 ? 8 : (per_row >= 4 ? 4 : (per_row >= 2 ? 2 : 1));
    ss_launch_cluster_x(sample_kernel, dim3(rows * per_row), dim3(threads), smem, stream, per_row, logits, stride, out, temperature, top_k, top_p,
                                                       min_p, penalty, seeds, draws, seen, seen_words,
                                                       slots, vocab, status, rows);
    return SS_LAUNCH_CHECK();
}

// Set the history bits of `n` token ids in one request's row of the seen-token table.
__global__ void mark_seen_kernel(uint32_t* __restrict__ seen_row, const int32_t* __restrict__ ids, int n,
                                 int vocab) {
    pdl_launch_dependents();  // the next kernel may be scheduled now; it waits for this one itself
    pdl_wait();               // nothing below runs before the kernels before this one are complete
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = ids[i];
        if (t >= 0 && t < vocab) atomicOr(&seen_row[t >> 5], 1u << (t & 31));
    }
}

extern "C" int ss_mark_seen(uint32_t* seen_row, const int32_t* ids, int n, int vocab, cudaStream_t stream) {
    if (n <= 0) return 0;
    ss_launch(mark_seen_kernel, dim3((n + 255) / 256 > 64 ? 64 : (n + 255) / 256), dim3(256), 0, stream, seen_row, ids, n, vocab);
    return SS_LAUNCH_CHECK();
}
