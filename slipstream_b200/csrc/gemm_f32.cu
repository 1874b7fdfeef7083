// float32 matrix product on the tensor cores of sm_100a: C[M, N] = X[M, K] * W[N, K]^T (+ bias), all float32.
//
// Every operand is cut into three bfloat16 parts, a = a1 + a2 + a3 (each what the ones before left, rounded to nearest, so the
// three carry the 24 bits of a float32 exactly), on its way into shared memory, and the product is formed from the six pairs
// of parts that matter: a1 b1 in one accumulator, a1 b2 + a2 b1 + a2 b2 + a1 b3 + a3 b1 in another, because the second is
// 2^-8 of the first and its additions then round at its own size.  What is left out (a2 b3 + a3 b2 and smaller) is at most 2^-24
// of |a| |b|, 2^-27.4 in the mean square, and has no sign of its own.  (Parts cut off instead of rounded leave out up to 2^-21, always of
// the product's sign.)  The tensor core adds into an accumulator with truncation, so an accumulator collects only CHUNK = 256 elements
// of K (16 additions); the chunks' sums are added up in registers, rounded to nearest, in order.  Errors against double precision
// (2-norm), beside those of a float32 fused multiply-add chain, normal operands: K = 4 2.7e-8 / 3.9e-8, 64 7.0e-8 / 1.4e-7, 256 2.3e-7 /
// 2.9e-7, 896 2.2e-7 / 5.3e-7, 3,584 2.4e-7 / 1.1e-6.  Positive operands only, where every truncation has the same sign: K = 64 9.0e-8 /
// 1.2e-7, 128 1.8e-7 / 1.7e-7, 256 3.9e-7 / 2.5e-7, 512 3.8e-7 / 3.5e-7, 896 3.5e-7 / 4.5e-7, 3,584 3.8e-7 / 8.8e-7.
//
// An output's value is the same in every form of the kernel and for every M: the same instructions on the same 64-wide
// steps of K, the same chunks, the chunks' sums added in the same order.  So a token's logits do not depend on what else
// is in its step.  An output that comes out neither finite is formed again as the plain chain (an infinity cannot be cut
// into parts), so infinities and NaN go through as they would on CUDA cores.
//
// A block of 16 warps (17 would leave a thread 96 registers instead of 128): 8 load both operands (16 bytes a lane, 16
// lanes a row), cut them and write the three planes into a ring of stages in the
// 128-byte-swizzled K-major form; 8 add up the chunks, a quarter of the rows and half of the columns each, and the first of
// them issues tcgen05.mma (the 128 features of a weight tile are the rows, BN tokens the columns).
//   * many tokens: BN = 128 or 64, a chunk's two accumulators double-buffered in tensor memory.
//   * up to 64 tokens: BN = 16, 32 or 64; K's chunks are spread over the up to 8 blocks of a cluster, each chunk keeps
//     its own columns of tensor memory, and the blocks add all chunks of their token columns out of one another's shared
//     memory.
// Nothing is read before the wait for the kernels in front, since a weight may be a result of theirs (the first weights ahead of it
// saved 2 to 4 us of a 1.5B layer's decode step: 97.5 beside 99.5 to 101).
//
// Why tensor cores: 128 float32 lanes an SM make 74 TFLOP/s at best (the CUDA-core kernel reached 22); six bfloat16
// products at the measured 1,660 TFLOP/s make 277.  777 tokens at the 7B sizes, before and after (us): q/k/v 1,191 and
// 171, o 871 and 150, gate/up 8,663 and 1,299 (163 TFLOP/s), down 4,632 and 782.  Bound by a stage's way through shared
// memory (written as 96 KB of planes, read six times by the products): the tensor pipe is 65 % busy on an SM at work.
// Four tokens at the 1.5B sizes: gate/up 201 and 29.6 (3.7 TB/s), down 519 and 28.
#include "mma_sync.cuh"
#include "tc5.cuh"

#define F3_BM 128
#define F3_BK 64
#define F3_CHUNK 256
#define F3_LOADERS 8
#define F3_THREADS (32 * (F3_LOADERS + 8))
#define F3_TMEM 512

struct F32Args {
    const float* W;
    const float* X;
    const float* bias;
    float* C;
    int* err;
    int M, N, K;
    int64_t ldc;
};

__device__ __forceinline__ float4 f3_load(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Two floats rounded to bfloat16, packed: their next parts.  What these leave behind stays in a and b (exactly).
__device__ __forceinline__ uint32_t f3_part(float& a, float& b) {
    const uint32_t h = pack_bf16(a, b);
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    return h;
}

__device__ __forceinline__ bool f3_finite(float v) { return fabsf(v) <= 3.4028234e38f; }

// The product as one chain of fused multiply-adds, 16 elements in flight (K and the rows' starts allow four a load).  A NaN stays one, so
// a chain that has met one is done (777 rows of NaN, 4,608 features of 3,584: element by element to the end 55.6 ms, so 0.28; one such row
// 0.46 and 0.19).
__device__ __noinline__ float f3_plain(const float* __restrict__ w, const float* __restrict__ x, int K) {
    float s = 0.f;
    for (int k = 0; k < K && s == s; k += 16) {
        float4 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k + 4 * u < K) {
                a[u] = *reinterpret_cast<const float4*>(x + k + 4 * u);
                b[u] = *reinterpret_cast<const float4*>(w + k + 4 * u);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (k + 4 * u >= K) break;
            s = fmaf(a[u].x, b[u].x, s);
            s = fmaf(a[u].y, b[u].y, s);
            s = fmaf(a[u].z, b[u].z, s);
            s = fmaf(a[u].w, b[u].w, s);
        }
    }
    return s;
}

// FEW: the cluster form (see above), else the form for many tokens.
// AHEAD: steps of weights in flight, in registers (one: mostly from L2) or, with few tokens, as asynchronous copies to
// shared memory (32 KB of weights a step).
template <int BN, int STAGES, int AHEAD, bool FEW>
__global__ void __launch_bounds__(F3_THREADS, 1) gemm_f32_kernel(const F32Args g) {
    constexpr int A_PLANE = F3_BM * 128, B_PLANE = BN * 128, STAGE = 3 * (A_PLANE + B_PLANE);
    constexpr int NA = F3_BM / (2 * F3_LOADERS), NB = BN / (2 * F3_LOADERS);  // 16-byte loads of a thread per stage
    constexpr bool X_STAGED = FEW && BN <= 32;
    constexpr int ROWS = NA + (X_STAGED ? NB : 0);  // ... that pass through shared memory
    extern __shared__ unsigned char smem_raw[];
    // [barriers: 1 KB][ring of stages][FEW: copies under way].  The sums of a block's chunks, in the end, take ring and copies.
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = base + 1024;
    static_assert(!FEW || F3_TMEM / (2 * BN) * BN * F3_BM * 4 <= STAGES * STAGE + AHEAD * ROWS * F3_LOADERS * 512, "the chunks' sums fit");
    float4* staged = reinterpret_cast<float4*>(ring + STAGES * STAGE) + threadIdx.x;  // FEW: [AHEAD][ROWS][loaders' threads]
    uint64_t* full = reinterpret_cast<uint64_t*>(base);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;   // 2
    uint64_t* acc_empty = acc_full + 2;    // 2
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BN, n0 = blockIdx.y * F3_BM;
    const int k_steps = (g.K + F3_BK - 1) / F3_BK, chunks = (g.K + F3_CHUNK - 1) / F3_CHUNK;
    constexpr int STEPS = F3_CHUNK / F3_BK;  // stages of a chunk
    const int n_blocks = FEW ? (int)gridDim.z : 1, rank = FEW ? (int)blockIdx.z : 0;
    const int per = (chunks + n_blocks - 1) / n_blocks;  // chunks of a block
    const int first = min(chunks, rank * per), my_chunks = min(chunks, first + per) - first;
    const int step0 = first * STEPS, steps = max(0, min(k_steps, (first + my_chunks) * STEPS) - step0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], F3_LOADERS); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(tmem_slot)), "r"(F3_TMEM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < F3_LOADERS) {
        // ---- both operands from memory, one stage ahead in registers, into the stages' planes
        const int hi = lane >> 4, at = lane & 15;
        float4 wa[NA], xb[NB];
        // rows 16 i + 2 warp + hi of a tile, four elements of K
        const int r0 = warp * 2 + hi;
        const float* w_row = g.W + (int64_t)(n0 + r0) * g.K + at * 4;
        const float* x_row = g.X + (int64_t)(m0 + r0) * g.K + at * 4;
        auto load_w = [&](int step) {
            const int k = step * F3_BK;
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                const bool live = n0 + r0 + 16 * i < g.N && k + at * 4 < g.K;
                if constexpr (FEW) cp_async16(&staged[((step - step0) % AHEAD * ROWS + i) * 32 * F3_LOADERS], live ? w_row + (int64_t)(16 * i) * g.K + k : g.W, live);
                else wa[i] = live ? f3_load(w_row + (int64_t)(16 * i) * g.K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto load_x = [&](int step) {
            const int k = step * F3_BK;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const bool live = m0 + r0 + 16 * i < g.M && k + at * 4 < g.K;
                if constexpr (X_STAGED) cp_async16(&staged[((step - step0) % AHEAD * ROWS + NA + i) * 32 * F3_LOADERS], live ? x_row + (int64_t)(16 * i) * g.K + k : g.X, live);
                else xb[i] = live ? f3_load(x_row + (int64_t)(16 * i) * g.K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto put = [&](unsigned char* planes, int plane, int row, float4 v) {
            unsigned char* dst = planes + row * 128 + (((at >> 1) ^ (row & 7)) << 4) + (at & 1) * 8;
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint2*>(dst + p * plane) = make_uint2(f3_part(v.x, v.y), f3_part(v.z, v.w));
        };
        pdl_wait();  // (for the weights, too: a caller may have formed them a kernel ago)
        if constexpr (FEW) {  // a group of copies a step, empty ones behind the last
            for (int u = 0; u < AHEAD; ++u) {
                if (u < steps) load_w(step0 + u);
                if (X_STAGED && u < steps) load_x(step0 + u);
                cp_async_commit();
            }
        } else {
            if (steps > 0) load_w(step0);
        }
        if (!X_STAGED && steps > 0) load_x(step0);
        for (int it = 0; it < steps; ++it) {
            const int s = it % STAGES;
            if constexpr (FEW) {
                cp_async_wait<AHEAD - 1>();  // a thread reads back what it copied itself: no barrier
#pragma unroll
                for (int i = 0; i < NA; ++i) wa[i] = staged[(it % AHEAD * ROWS + i) * 32 * F3_LOADERS];
#pragma unroll
                for (int i = 0; X_STAGED && i < NB; ++i) xb[i] = staged[(it % AHEAD * ROWS + NA + i) * 32 * F3_LOADERS];
            }
            if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, gave_up))) break;
            unsigned char* stage = ring + s * STAGE;
#pragma unroll
            for (int i = 0; i < NA; ++i) put(stage, A_PLANE, r0 + 16 * i, wa[i]);
            if (it + AHEAD < steps) load_w(step0 + it + AHEAD);
#pragma unroll
            for (int i = 0; i < NB; ++i) put(stage + 3 * A_PLANE, B_PLANE, r0 + 16 * i, xb[i]);
            if (it + (X_STAGED ? AHEAD : 1) < steps) load_x(step0 + it + (X_STAGED ? AHEAD : 1));
            if (FEW) cp_async_commit();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        if (FEW) cp_async_wait<0>();
    } else {
        // ---- the chunks' sums: a thread has a feature (a lane of tensor memory) and half of the tokens
        const int quarter = warp & 3, f = n0 + quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        constexpr int COLS = FEW ? 16 : (BN / 2 + 15) / 16 * 16;
        const int col0 = ((warp - F3_LOADERS) >> 2) * COLS;
        float sum[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
        auto add_chunk = [&](int c) -> bool {
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[c & 1], (c >> 1) & 1, gave_up))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t big = lanes + (uint32_t)((c & 1) * 2 * BN + col0);
#pragma unroll
            for (int j = 0; j < COLS; j += 16) {
                if (col0 + j >= BN) break;  // an odd number of 16s: the second half is the smaller
                uint32_t b[16], s[16];
                tmem_ld16(big + j, b);
                tmem_ld16(big + BN + j, s);
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[j + e] += __uint_as_float(b[e]) + __uint_as_float(s[e]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[c & 1]);
            return true;
        };
        pdl_wait();  // (also before the waits below: the loaders stand in theirs until the kernel in front is done)
        bool ok = true;
        if (warp == F3_LOADERS) {
            // the first of them issues the products, too, and adds up a chunk once the next one's first step is issued.
            // D float32, A and B bfloat16 and K-major, N = BN, M = 128
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(F3_BM >> 4) << 24);
            for (int it = 0; it < steps && ok; ++it) {
                const int s = it % STAGES, c = it / STEPS, in_chunk = it % STEPS;
                if (!FEW && in_chunk == 0) ok = mbar_wait(&acc_empty[c & 1], ((c >> 1) & 1) ^ 1, gave_up);
                ok = __all_sync(0xffffffffu, ok && mbar_wait(&full[s], (it / STAGES) & 1, gave_up));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned char* stage = ring + s * STAGE;
                const uint64_t a1 = smem_desc(stage), a2 = smem_desc(stage + A_PLANE), a3 = smem_desc(stage + 2 * A_PLANE);
                const unsigned char* bs = stage + 3 * A_PLANE;
                const uint64_t b1 = smem_desc(bs), b2 = smem_desc(bs + B_PLANE), b3 = smem_desc(bs + 2 * B_PLANE);
                const uint32_t big = tmem + (uint32_t)((FEW ? c : (c & 1)) * 2 * BN), small = big + BN;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < F3_BK / 16; ++kk) {  // 16 elements of K = 32 bytes further along the swizzled row
                        const uint64_t o = (uint64_t)(kk * 2);
                        const uint32_t more = (in_chunk | kk) != 0;
                        umma_f16(small, a3 + o, b1 + o, idesc, more);
                        umma_f16(small, a1 + o, b3 + o, idesc, 1);
                        umma_f16(small, a2 + o, b2 + o, idesc, 1);
                        umma_f16(small, a2 + o, b1 + o, idesc, 1);
                        umma_f16(small, a1 + o, b2 + o, idesc, 1);
                        umma_f16(big, a1 + o, b1 + o, idesc, more);
                    }
                    umma_commit(&empty[s]);
                    if (FEW ? it == steps - 1 : (in_chunk == STEPS - 1 || it == steps - 1)) umma_commit(&acc_full[FEW ? 0 : (c & 1)]);
                }
                __syncwarp();
                if (!FEW && in_chunk == 0 && c > 0) ok = add_chunk(c - 1);
            }
            if (!FEW && ok && my_chunks > 0) add_chunk(my_chunks - 1);
        } else {
            for (int c = 0; c < my_chunks && !FEW && ok; ++c) ok = add_chunk(c);
        }
        if constexpr (!FEW) {
            if (f < g.N) {
                const float b = g.bias ? g.bias[f] : 0.f;
                const int live = min(COLS, min(g.M - m0, BN) - col0);
                float* out = g.C + (int64_t)(m0 + col0) * g.ldc + f;
                bool plain = false;
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    if (j < live) out[j * g.ldc] = g.bias ? sum[j] + b : sum[j];
                    plain |= j < live && !f3_finite(sum[j]);
                }
                for (int j = 0; plain && j < live; ++j) {
                    if (f3_finite(out[j * g.ldc])) continue;
                    const float v = f3_plain(g.W + (int64_t)f * g.K, g.X + (int64_t)(m0 + col0 + j) * g.K, g.K);
                    out[j * g.ldc] = g.bias ? v + b : v;
                }
            }
        } else {
            if (steps > 0) __all_sync(0xffffffffu, mbar_wait(&acc_full[0], 0, gave_up));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // every product is done: the ring carries the chunks' sums [chunk][token][128 features]
            float* sums = reinterpret_cast<float*>(ring);
            const int live = min(BN, g.M - m0);
            for (int c = 0; c < my_chunks; ++c)
#pragma unroll 1
                for (int j = ((warp - F3_LOADERS) >> 2) * 16; j < live; j += 32) {
                    uint32_t b[16], s[16];
                    tmem_ld16(lanes + (uint32_t)(c * 2 * BN + j), b);
                    tmem_ld16(lanes + (uint32_t)(c * 2 * BN + BN + j), s);
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (j + e < live) sums[(c * live + j + e) * F3_BM + quarter * 32 + lane] = __uint_as_float(b[e]) + __uint_as_float(s[e]);
                }
        }
    }
    if constexpr (FEW) {
        cluster_sync_all();
        const float* sums = reinterpret_cast<const float*>(ring);
        const int live = min(BN, g.M - m0), f = n0 + lane * 4;
        for (int j = rank + n_blocks * warp; j < live; j += n_blocks * (F3_THREADS / 32)) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c0 = 0; c0 < chunks; c0 += 8) {  // eight reads of other blocks' memory in flight
                float4 p[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (c0 + u < chunks) p[u] = ld_cluster_f32x4(sums + ((c0 + u) % per * live + j) * F3_BM + lane * 4, (uint32_t)((c0 + u) / per));
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (c0 + u < chunks) { v.x += p[u].x; v.y += p[u].y; v.z += p[u].z; v.w += p[u].w; }
            }
            const float out[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (f + e >= g.N) break;
                float o = out[e];
                if (!f3_finite(o)) o = f3_plain(g.W + (int64_t)(f + e) * g.K, g.X + (int64_t)(m0 + j) * g.K, g.K);
                g.C[(int64_t)(m0 + j) * g.ldc + f + e] = g.bias ? o + g.bias[f + e] : o;
            }
        }
    }
    if (*gave_up && threadIdx.x == 0) atomicOr(g.err, SS_ERR_WAIT_LIMIT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if constexpr (FEW) cluster_sync_before_exit();  // a block's sums are read by the others
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(F3_TMEM));
    }
}

template <int BN, int STAGES, int AHEAD, bool FEW>
struct F32Form {
    static constexpr int SMEM = STAGES * 3 * (F3_BM + BN) * 128 + 2048 + (FEW ? AHEAD * (F3_BM + (BN <= 32 ? BN : 0)) * F3_BK * 4 : 0);

    static int launch(const F32Args& g, int n_blocks, cudaStream_t stream) {
        static SsPerDevice opted;
        if (int rc = ss_opt_in_smem(gemm_f32_kernel<BN, STAGES, AHEAD, FEW>, SMEM, opted)) return rc;
        const dim3 grid((g.M + BN - 1) / BN, (g.N + F3_BM - 1) / F3_BM, n_blocks);
        if (FEW) ss_launch_cluster(gemm_f32_kernel<BN, STAGES, AHEAD, FEW>, grid, dim3(F3_THREADS), SMEM, stream, n_blocks, g);
        else ss_launch(gemm_f32_kernel<BN, STAGES, AHEAD, FEW>, grid, dim3(F3_THREADS), SMEM, stream, g);
        return SS_LAUNCH_CHECK();
    }
};

// How many clusters of n blocks, one block to an SM, run at the same time: clusters do not cross the GPU's processor
// clusters, so 36 of 4 do not fit 148 SMs (4,608 features in clusters of 4 ran as two rounds).
static int f3_resident_clusters(int n) {
    static int known[SS_MAX_DEVICES][9];  // 0: not asked yet
    const int dev = ss_current_device();
    if (dev < 0) return 1;
    if (known[dev][n] == 0) {
        using Form = F32Form<16, 2, 3, true>;
        static SsPerDevice opted;
        int count = 0;
        if (ss_opt_in_smem(gemm_f32_kernel<16, 2, 3, true>, Form::SMEM, opted) == 0)
            count = ss_resident_clusters(gemm_f32_kernel<16, 2, 3, true>, F3_THREADS, Form::SMEM, n);
        known[dev][n] = count > 0 ? count : (ss_sm_count() / n > 0 ? ss_sm_count() / n : 1);
    }
    return known[dev][n];
}

// Blocks that share the chunks of K of a tile in the form for few tokens: of 1..8, the number with the fewest rounds of
// clusters times steps of a block (and about eight steps' worth of filling and adding up), among those whose chunks fit a
// block's tensor memory (2 bn columns each); 0 where none does.
static int f3_blocks(int tiles, int K, int bn) {
    const int chunks = (K + F3_CHUNK - 1) / F3_CHUNK, room = F3_TMEM / (2 * bn);
    int best = 0;
    int64_t least = 0;
    for (int n = 1; n <= 8 && n <= chunks; ++n) {
        const int per = (chunks + n - 1) / n, fit = f3_resident_clusters(n);
        if (per > room || (n - 1) * per >= chunks) continue;  // (no block without a chunk)
        const int64_t cost = (int64_t)((tiles + fit - 1) / fit) * (per * (F3_CHUNK / F3_BK) + 8);
        if (best == 0 || cost < least) { best = n; least = cost; }
    }
    return best;
}

// K a multiple of 4 and above 0, W and X 16-byte aligned and contiguous.
extern "C" int ss_gemm_f32(const float* X, const float* W, const float* bias, float* C, int M, int N, int K, int64_t ldc,
                           int* err, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 != 0 || ((uintptr_t)X | (uintptr_t)W) % 16 != 0) return (int)cudaErrorInvalidValue;
    const F32Args g{W, X, bias, C, err, M, N, K, ldc};
    const int tiles = (N + F3_BM - 1) / F3_BM;
    if (M <= 64) {
        // the narrowest tile that holds the tokens; a narrower one, in several tiles, where K's chunks need the room
        for (int bn = M <= 16 ? 16 : (M <= 32 ? 32 : 64); bn >= 16; bn /= 2) {
            const int n = f3_blocks(tiles * ((M + bn - 1) / bn), K, bn);
            if (n == 0) continue;
            if (bn == 16) return F32Form<16, 2, 3, true>::launch(g, n, stream);
            if (bn == 32) return F32Form<32, 2, 2, true>::launch(g, n, stream);
            return F32Form<64, 2, 2, true>::launch(g, n, stream);
        }
    }
    // the width with the least rounds of blocks times a tile's time, which is nearly that of its weights alone: a round of
    // 3,584 elements of K takes 89, 85, 79, 76 and 74 us at widths of 128 to 64 (777 tokens: 3,584 features 173 us with
    // 128, 150 with 80; 4,608 features 178, 171 with 112 and 295 with 64)
    int width = 128;
    int64_t least = 0;
    for (int bn = 128; bn >= 64; bn -= 16) {
        const int64_t blocks = (int64_t)tiles * ((M + bn - 1) / bn), cost = (blocks + ss_sm_count() - 1) / ss_sm_count() * (280 + bn);
        if (bn == 128 || cost < least) { width = bn; least = cost; }
    }
    switch (width) {
        case 64: return F32Form<64, 3, 1, false>::launch(g, 1, stream);
        case 80: return F32Form<80, 2, 1, false>::launch(g, 1, stream);
        case 96: return F32Form<96, 2, 1, false>::launch(g, 1, stream);
        case 112: return F32Form<112, 2, 1, false>::launch(g, 1, stream);
        default: return F32Form<128, 2, 1, false>::launch(g, 1, stream);
    }
}
