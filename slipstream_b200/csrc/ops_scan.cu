// Two recurrences over prompt portions, a chunk of tokens at a time on the tensor cores: the state-space scan (ops_mixers.cu)
// and the matrix memory (ops_cells.cu), which those files walk token by token.  Both are, per head, with keys k and queries q
// of `dim` elements and values x of `vdim`,
//   S_t = e^(a_t) S_(t-1) + w_t k_t x_t^T,   o_t = S_t^T q_t,
// and over a chunk of C tokens from the state S_0 in front of it, with L_t = a_0 + .. + a_t, exactly
//   o_t = e^(L_t) S_0^T q_t + sum_{s <= t} e^(L_t - L_s) w_s (q_t . k_s) x_s,   S_C = e^(L_C) S_0 + sum_s e^(L_C - L_s) w_s k_s x_s^T:
// products of matrices instead of C dependent steps.
//   * state space: k = B, q = C (shared by the heads of a group), x = x, a = -exp(a_log) dt, w = dt; out = o + d_skip x.
//   * matrix memory: a = f + m_(t-1) - m_t, w = exp(i - m_t); the normaliser n is the column of a value that is always 1: its
//     part of a product is the sum of a row of weights, and q . n_0.
//
// Nothing that was 32 bits passes through 16: q, k and x are bfloat16 as they come, so q . k is a product of exact operands;
// the weighed scores, the weighed keys and S_0 are float32 and are cut into three bfloat16 parts, which hold their 24 bits, and
// each part is multiplied; L is summed in double precision and kept as two floats, so that differences of neighbours are
// exact; the tensor core truncates as it adds, so small parts have accumulators of their own, long sums two, and what a chunk adds
// to the state is summed by itself and added in float32.  Against double precision (2-norm, beside token by token): 112 heads
// of 64 x 128 over 2,045 tokens 1.2e-7 / 1.3e-7 in the outputs, 1.0e-7 / 1.1e-7 in the state; the matrix memory at 28 heads of 128
// 3.5e-7 / 3.5e-7 and 3.5e-7 / 3.5e-7.
//
// A block of 8 warps takes 8 CT value columns of a head of a request and walks its chunks of 64 tokens.  (1) Four warps form
// the scores of 16 tokens each with the keys up to the diagonal, weigh them and multiply them with the values; the other four
// multiply the same tokens' queries with the state.  The first warp, whose tokens see the fewest keys, also forms the next chunk's
// a and w.  (2) The two sums meet; every warp has 16 rows of the state, in registers as accumulators.  (3) Their parts go to
// shared memory for the next chunk.  A token with an infinity or a NaN among its values is a chunk of its own: in a product it
// would reach the tokens in front of it.
//
// Bound by the chain of a chunk's stages (copies, scores, outputs, state; 13,000 cycles a chunk of which the products take
// 3,900) with two blocks an SM to fill one another's gaps: the tensor pipe is 38 % busy, 60 % on an SM that has two blocks.  Against
// token by token (us): state space, 112 heads of 64 x 128, 8 groups, 818 + 1,227 tokens 666 -> 218, 2,048 of one request 636 ->
// 229; 24 heads of 128 x 64, 6 requests of 300 99 -> 46; matrix memory, 28 heads of 128, 760 + 1,140 tokens 357 -> 155.
#include "mma_sync.cuh"

#define SC_T 64
#define SC_THREADS 256

struct ScanArgs {
    const bf16* q;       // element 0 of the first head's (group's) queries, keys and values of row 0
    const bf16* k;
    const bf16* x;
    int64_t stride;      // of all three
    float* state;        // [slot][heads][vdim (+ 1)][dim]
    float* out;          // [rows][heads * vdim]
    const int32_t* q_start;
    const int32_t* seq_lens;
    const int32_t* slots;
    int heads, group, dim, vdim, n_slots;  // group: heads that share queries and keys
    int* err;
    // state space
    const bf16* dt;
    int64_t dt_stride;
    const float* dt_bias;
    const float* a_log;
    const float* d_skip;
    // matrix memory
    const float* gates;
    int64_t gate_stride;
    const float* bias_i;
    const float* bias_f;
    float cap, q_scale;
    const float* peak;  // in front of the step, read by all column blocks of a head: a kernel behind this one writes it
    float* nq;
    float* peaks_out;
    int sms;
};

int launch_cell_peaks(const float* peaks, float* peak, const int32_t* q_start, const int32_t* seq_lens, const int32_t* slots, int R, int H,
                      int n_slots, cudaStream_t stream);  // ops_cells.cu

namespace {

__device__ __forceinline__ float sc_log_sigmoid(float z) {  // as in ops_cells.cu
    return fminf(z, 0.f) - log1pf(expf(-fabsf(z)));
}

// The product as a function of its operands (not volatile: the compiler may move it between the loads around it).
__device__ __forceinline__ void mma_free(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Three bfloat16 parts of two floats, packed: together their 24 bits.
__device__ __forceinline__ void in_three(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16(a, b);
    a -= __uint_as_float(hi << 16);
    b -= __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(a, b);
    lo = pack_bf16(a - __uint_as_float(mid << 16), b - __uint_as_float(mid & 0xffff0000u));
}

template <int N, int CT>
struct ScanSmem {
    static constexpr int QS = N + 8, VS = CT * 8 + 8;  // strides that spread ldmatrix over all banks
    static constexpr int q = 0;                        // bf16 [SC_T][QS]
    static constexpr int k = q + SC_T * QS * 2;
    static constexpr int x = k + SC_T * QS * 2;        // bf16 [SC_T][VS]
    static constexpr int s = x + SC_T * VS * 2;        // bf16 [3][N][VS]: the state in front of the chunk, hi, mid, lo
    static constexpr int gate = s + 3 * N * VS * 2;    // float [2][4][SC_T]: L hi, L lo, w, m of this chunk and the next
    static constexpr int u = gate + 2 * 4 * SC_T * 4;  // float [SC_T]: weights of the keys in the state behind the chunk
    static constexpr int b = u + SC_T * 4;             // float [4][SC_T]: weights of the keys in front of each 16 tokens, at the first of them
    static constexpr int dot = b + 4 * SC_T * 4;       // float [SC_T]: e^(L_t) q_t . n_0
    static constexpr int n = dot + SC_T * 4;           // float [N]: the normaliser
    static constexpr int misc = n + N * 4;
    static constexpr int bytes = misc + 16;
    static constexpr int PS = CT * 8 + 8;              // float [SC_T][PS] in place of the state's parts: queries times the state
    static_assert(SC_T * PS * 4 <= 3 * N * VS * 2, "it fits");
};

// ---- requests with few tokens (decoded ones beside the prompt portions of others): token by token, with the arithmetic of
// ssm_scan_kernel and matrix_cell_kernel, which run decode steps and steps without a longer portion.  So the bits of such a request do
// not depend on what else is in its step.  A chunk of 64 tokens for one costs as much as for 64: a portion of 300 tokens
// beside 48 decoded ones, 112 heads of 64 x 128, 219 us in chunks, 184 so (all token by token 270); 500 beside 200, 821, 666 (740); 32 heads of
// 128 x 256, 500 beside 200, 1,304, 846 (831).  From two tokens on the time is about that of a chunk (48 requests of 4: 205 and 225 us, of
// 8: 203 and 299); such requests are few beside a portion.
#define SC_FEW 8

// State space: columns c0 .. c0 + cols - 1 as ssm_scan_kernel has them, four lanes a column of PER elements each.
template <int PER>
__device__ __forceinline__ void scan_few_tokens(const ScanArgs& g, int h, int q0, int q_len, float* sp, int c0, int cols) {
    const int n0 = (threadIdx.x & 3) * PER, end = min(c0 + cols, g.vdim);
    const float rate = expf(g.a_log[h]), bias = g.dt_bias[h], skip = g.d_skip[h];
    const bool vec = (reinterpret_cast<uintptr_t>(sp) & 15) == 0;
    for (int col = c0 + (threadIdx.x >> 2); col < end; col += SC_THREADS / 4) {  // whole warps: vdim comes in steps of 8
        float* st = sp + (int64_t)col * g.dim + n0;
        float S[PER];
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (n0 + i < g.dim) v = vec ? *reinterpret_cast<const float4*>(st + i) : make_float4(st[i], st[i + 1], st[i + 2], st[i + 3]);
            S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
        }
        for (int t = 0; t < q_len; ++t) {
            const int64_t row = q0 + t;
            const float z = to_float(g.dt[row * g.dt_stride + h]) + bias, dt = z > 20.f ? z : log1pf(expf(z));
            const float dec = expf(-rate * dt), xv = to_float(g.x[row * g.stride + (int64_t)h * g.vdim + col]), dx = dt * xv;
            const bf16* b = g.k + row * g.stride + (int64_t)(h / g.group) * g.dim + n0;
            const bf16* c = g.q + row * g.stride + (int64_t)(h / g.group) * g.dim + n0;
            float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
            for (int i = 0; i < PER; i += 8) {
                uint4 bw = make_uint4(0u, 0u, 0u, 0u), cw = bw;
                if (n0 + i < g.dim) {
                    bw = *reinterpret_cast<const uint4*>(b + i);
                    cw = *reinterpret_cast<const uint4*>(c + i);
                }
                const uint32_t bb[4] = {bw.x, bw.y, bw.z, bw.w}, cc[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S[i + 2 * e] = fmaf(dec, S[i + 2 * e], dx * __uint_as_float(bb[e] << 16));
                    S[i + 2 * e + 1] = fmaf(dec, S[i + 2 * e + 1], dx * __uint_as_float(bb[e] & 0xffff0000u));
                    acc0 = fmaf(S[i + 2 * e], __uint_as_float(cc[e] << 16), acc0);
                    acc1 = fmaf(S[i + 2 * e + 1], __uint_as_float(cc[e] & 0xffff0000u), acc1);
                }
            }
            float acc = acc0 + acc1;
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            if ((threadIdx.x & 3) == 0) g.out[(row * g.heads + h) * g.vdim + col] = fmaf(skip, xv, acc);
        }
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
            if (n0 + i >= g.dim) continue;
            if (vec) *reinterpret_cast<float4*>(st + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
            else { st[i] = S[i]; st[i + 1] = S[i + 1]; st[i + 2] = S[i + 2]; st[i + 3] = S[i + 3]; }
        }
    }
}

// Matrix memory: the same columns, and with the first ones the normaliser, as matrix_cell_kernel has them: eight lanes a column, lane j
// with elements 32 i + 4 j .. + 3.
template <int NI>
__device__ __forceinline__ void cell_few_tokens(const ScanArgs& g, int h, int q0, int q_len, int slot, float* sp, int c0, int cols) {
    const int j4 = (threadIdx.x & 7) * 4, own = min(c0 + cols, g.vdim) - c0, all = own + (c0 == 0);
    const float bi = g.bias_i ? g.bias_i[h] : 0.f, bf = g.bias_f ? g.bias_f[h] : 0.f;
    const bool vec = (reinterpret_cast<uintptr_t>(sp) & 15) == 0;
    for (int base = 0; base < all; base += SC_THREADS / 8) {  // (the whole warp comes along for the shuffles)
        const int place = base + (threadIdx.x >> 3), col = place < own ? c0 + place : g.vdim;
        const bool ok = place < all;
        float* st = sp + (int64_t)col * g.dim + j4;
        float S[NI * 4], m = g.peak[(int64_t)slot * g.heads + h];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* p = st + 32 * i;
            if (ok && 32 * i + j4 < g.dim) v = vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
            S[4 * i] = v.x; S[4 * i + 1] = v.y; S[4 * i + 2] = v.z; S[4 * i + 3] = v.w;
        }
        for (int t = 0; t < q_len; ++t) {
            const int64_t row = q0 + t;
            const float* gate = g.gates + row * g.gate_stride;
            const float in = g.cap * tanhf((gate[h] + bi) / g.cap), f = sc_log_sigmoid(g.cap * tanhf((gate[g.heads + h] + bf) / g.cap));
            const float now = fmaxf(f + m, in), keep = expf(f + m - now), take = expf(in - now);
            if (c0 == 0 && threadIdx.x == 0 && base == 0) g.peaks_out[row * g.heads + h] = now;
            m = now;
            const float tv = take * (col < g.vdim ? to_float(g.x[row * g.stride + (int64_t)h * g.vdim + col]) : 1.f);
            const bf16* k = g.k + row * g.stride + (int64_t)h * g.dim + j4;
            const bf16* q = g.q + row * g.stride + (int64_t)h * g.dim + j4;
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                uint2 kw = make_uint2(0u, 0u), qw = kw;
                if (32 * i + j4 < g.dim) {
                    kw = *reinterpret_cast<const uint2*>(k + 32 * i);
                    qw = *reinterpret_cast<const uint2*>(q + 32 * i);
                }
                const float kk[4] = {__uint_as_float(kw.x << 16), __uint_as_float(kw.x & 0xffff0000u), __uint_as_float(kw.y << 16), __uint_as_float(kw.y & 0xffff0000u)};
                const float qq[4] = {__uint_as_float(qw.x << 16), __uint_as_float(qw.x & 0xffff0000u), __uint_as_float(qw.y << 16), __uint_as_float(qw.y & 0xffff0000u)};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S[4 * i + e] = fmaf(keep, S[4 * i + e], kk[e] * tv);
                    acc = fmaf(S[4 * i + e], __fmul_rn(qq[e], g.q_scale), acc);
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (ok && j4 == 0) {
                if (col < g.vdim) g.out[(row * g.heads + h) * g.vdim + col] = acc;
                else g.nq[row * g.heads + h] = acc;
            }
        }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            if (!ok || 32 * i + j4 >= g.dim) continue;
            float* p = st + 32 * i;
            if (vec) *reinterpret_cast<float4*>(p) = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
            else { p[0] = S[4 * i]; p[1] = S[4 * i + 1]; p[2] = S[4 * i + 2]; p[3] = S[4 * i + 3]; }
        }
    }
}

// CELL: the matrix memory, else the state-space scan.
template <bool CELL, int N, int CT>
__global__ void __launch_bounds__(SC_THREADS, N <= 128 ? 2 : 1) scan_chunks_kernel(const ScanArgs g) {
    using M = ScanSmem<N, CT>;
    constexpr int QS = M::QS, VS = M::VS, PS = M::PS, COLS = CT * 8;
    constexpr int MPW = N >= 128 ? N / 128 : 1, TPW = N >= 128 ? CT : CT / 2;  // state: row tiles and column tiles of a warp
    static_assert(SC_THREADS / CT <= SC_T, "every thread copies values");
    static_assert(N >= 64 && N % 64 == 0 && (N / 32) % 2 == 0 && CT % 2 == 0 && TPW % 2 == 0, "tiles come in pairs");
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* Q = reinterpret_cast<bf16*>(smem + M::q);
    bf16* K = reinterpret_cast<bf16*>(smem + M::k);
    bf16* X = reinterpret_cast<bf16*>(smem + M::x);
    bf16* Sp = reinterpret_cast<bf16*>(smem + M::s);
    float* u_s = reinterpret_cast<float*>(smem + M::u);
    float* dot_s = reinterpret_cast<float*>(smem + M::dot);
    float* part_s = reinterpret_cast<float*>(smem + M::s);
    float* n_s = reinterpret_cast<float*>(smem + M::n);
    int* bad = reinterpret_cast<int*>(smem + M::misc);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (1): tokens 16 rt .. of the chunk.  The last tokens see the most keys: of two blocks of an SM they go to different quarters
    const int rt = (warp + 2 * (blockIdx.x / g.sms)) & 3;
    const bool makes_gates = warp < 4 && rt == 0;
    const int row_lo = rt * 16 + (lane >> 2), row_hi = row_lo + 8;
    const int col_blocks = (g.vdim + COLS - 1) / COLS;
    const int unit = blockIdx.x / col_blocks, c0 = (blockIdx.x % col_blocks) * COLS, r = unit / g.heads, h = unit - r * g.heads;
    const bool first_cols = CELL && c0 == 0;  // the block of a head that also has its normaliser and peaks
    pdl_launch_dependents();
    pdl_wait();
    const int q0 = g.q_start[r], q_len = g.q_start[r + 1] - q0;
    if (q_len <= 0 || g.seq_lens[r] <= 0) return;
    const int slot = g.slots[r];
    if (slot < 0 || slot >= g.n_slots) {
        if (tid == 0) atomicOr(g.err, SS_ERR_SLOT_RANGE);
        return;
    }
    if (q_len <= SC_FEW) {
        float* state = g.state + ((int64_t)slot * g.heads + h) * (g.vdim + (CELL ? 1 : 0)) * g.dim;
        if constexpr (CELL) cell_few_tokens<N / 32>(g, h, q0, q_len, slot, state, c0, COLS);
        else if (N == 64 && g.dim <= 32) scan_few_tokens<8>(g, h, q0, q_len, state, c0, COLS);
        else scan_few_tokens<N / 4>(g, h, q0, q_len, state, c0, COLS);
        return;
    }
    const bf16* q_src = g.q + (int64_t)q0 * g.stride + (int64_t)(h / g.group) * g.dim;
    const bf16* k_src = g.k + (int64_t)q0 * g.stride + (int64_t)(h / g.group) * g.dim;
    const bf16* x_src = g.x + (int64_t)q0 * g.stride + (int64_t)h * g.vdim + c0;

    // rows of a chunk into shared memory, 16 bytes a copy; zeros behind the last row, element and column
    constexpr int RUNS = N / 8, ROWS = SC_THREADS / RUNS;  // runs of 8 elements of a row; rows that all threads copy at a time
    const int f_t = tid / RUNS, f_c = (tid % RUNS) * 8;
    auto fetch_rows = [&](bf16* dst, const bf16* src, int t0) {
        const int left = f_c < g.dim ? q_len - t0 - f_t : 0;  // rows from this thread's first on
        const bf16* from = src + (int64_t)(t0 + f_t) * g.stride + f_c;
        bf16* to = dst + f_t * QS + f_c;
#pragma unroll
        for (int w = 0; w < SC_T / ROWS; ++w) cp_async16(to + w * ROWS * QS, w * ROWS < left ? from + w * ROWS * g.stride : g.q, w * ROWS < left);
    };
    constexpr int X_ROWS = SC_THREADS / CT;
    const int x_t = tid / CT, x_c = (tid % CT) * 8;
    auto fetch_values = [&](int t0) {
        const int left = c0 + x_c < g.vdim ? q_len - t0 - x_t : 0;
        const bf16* from = x_src + (int64_t)(t0 + x_t) * g.stride + x_c;
#pragma unroll
        for (int w = 0; w < SC_T / X_ROWS; ++w)
            cp_async16(X + (x_t + w * X_ROWS) * VS + x_c, w * X_ROWS < left ? from + w * X_ROWS * g.stride : g.q, w * X_ROWS < left);
    };
    fetch_rows(Q, q_src, 0);
    fetch_rows(K, k_src, 0);
    fetch_values(0);
    cp_async_commit();

    // a, w (and m) of the tokens from t0 on, summed up, by one warp: lane l has tokens 2 l and 2 l + 1
    const float rate = CELL ? 0.f : expf(g.a_log[h]), dt_bias = CELL ? 0.f : g.dt_bias[h], skip = CELL ? 0.f : g.d_skip[h];
    const float bi = CELL && g.bias_i ? g.bias_i[h] : 0.f, bf = CELL && g.bias_f ? g.bias_f[h] : 0.f;
    auto gate_row = [&](int buf, int which) { return reinterpret_cast<float*>(smem + M::gate) + (buf * 4 + which) * SC_T; };
    float raw_a[2], raw_w[2];  // what they are made of, read a chunk ahead, from token raw_at on
    int raw_at = -1;
    auto read_gates = [&](int t0) {
        raw_at = t0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = min(t0 + 2 * lane + e, q_len - 1);
            if constexpr (CELL) {
                const float* p = g.gates + (int64_t)(q0 + t) * g.gate_stride;
                raw_w[e] = p[h];
                raw_a[e] = p[g.heads + h];
            } else {
                raw_w[e] = to_float(g.dt[(int64_t)(q0 + t) * g.dt_stride + h]);
            }
        }
    };
    auto make_gates = [&](int buf, int t0, float m_prev) {
        float a[2], w[2];
        if (raw_at != t0) read_gates(t0);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            a[e] = w[e] = 0.f;
            if (t0 + 2 * lane + e >= q_len) continue;
            if constexpr (CELL) {
                w[e] = g.cap * tanhf((raw_w[e] + bi) / g.cap);
                a[e] = sc_log_sigmoid(g.cap * tanhf((raw_a[e] + bf) / g.cap));
            } else {
                const float z = raw_w[e] + dt_bias;
                w[e] = z > 20.f ? z : log1pf(expf(z));
                a[e] = -rate * w[e];
            }
        }
        if (t0 + SC_T < q_len) read_gates(t0 + SC_T);
        if constexpr (CELL) {
            float* f_s = gate_row(buf, 0);
            float* i_s = gate_row(buf, 1);
            float* m_s = gate_row(buf, 3);
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 2; ++e) { f_s[2 * lane + e] = a[e]; i_s[2 * lane + e] = w[e]; }
            __syncwarp();
            if (lane == 0) {  // the running maximum is a chain
                float m = m_prev;
                const int n = min(SC_T, q_len - t0);
                for (int t = 0; t < n; ++t) {
                    m = fmaxf(f_s[t] + m, i_s[t]);
                    m_s[t] = m;
                }
            }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 2 * lane + e;
                if (t0 + t < q_len) {
                    const float before = t ? m_s[t - 1] : m_prev, now = m_s[t];
                    a[e] = a[e] + before - now;
                    w[e] = expf(w[e] - now);
                    if (first_cols) g.peaks_out[(int64_t)(q0 + t0 + t) * g.heads + h] = now;
                }
            }
            __syncwarp();
        }
        // A decay below e^-200 is zero in 32 bits, alone or in a product: an infinite one is held there, so that the
        // differences L_t - L_s of tokens behind it are numbers.  (A NaN stays one.)
#pragma unroll
        for (int e = 0; e < 2; ++e) a[e] = a[e] < -200.f ? -200.f : a[e];
        const double a0 = (double)a[0], both = a0 + (double)a[1];
        double up_to = both;  // inclusive sum over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, up_to, o);
            if (lane >= o) up_to += up;
        }
        // the lanes in front, not `up_to` less this lane's two: a NaN of the odd token is not in front of the even one
        double before = __shfl_up_sync(0xffffffffu, up_to, 1);
        if (lane == 0) before = 0.0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const double sum = before + (e ? both : a0);
            const float hi = (float)sum;
            gate_row(buf, 0)[2 * lane + e] = hi;
            gate_row(buf, 1)[2 * lane + e] = (float)(sum - (double)hi);
            gate_row(buf, 2)[2 * lane + e] = w[e];
        }
    };
    float* sp = g.state + ((int64_t)slot * g.heads + h) * (g.vdim + (CELL ? 1 : 0)) * g.dim;
    if (tid == 0) *bad = SC_T;
    if (makes_gates) make_gates(0, 0, CELL ? g.peak[(int64_t)slot * g.heads + h] : 0.f);

    // the state as accumulators: rows (elements of the keys) s_row and 8 further of each row tile, columns of TPW tiles
    const int s_tile = N >= 128 ? 0 : (warp >> 2) * TPW;
    auto s_row = [&](int m) { return ((N >= 128 ? warp + 8 * m : (warp & 3)) * 16) + (lane >> 2); };
    float acc[MPW][TPW][4];
#pragma unroll
    for (int m = 0; m < MPW; ++m)
#pragma unroll
        for (int n = 0; n < TPW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = s_row(m) + (e >> 1) * 8, col = c0 + (s_tile + n) * 8 + (lane & 3) * 2 + (e & 1);
                acc[m][n][e] = row < g.dim && col < g.vdim ? sp[(int64_t)col * g.dim + row] : 0.f;
            }
    if (first_cols)
        for (int i = tid; i < N; i += SC_THREADS) n_s[i] = i < g.dim ? sp[(int64_t)g.vdim * g.dim + i] : 0.f;
    auto put_state = [&]() {
#pragma unroll
        for (int m = 0; m < MPW; ++m)
#pragma unroll
            for (int n = 0; n < TPW; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    bf16* at = Sp + (s_row(m) + e * 8) * VS + (s_tile + n) * 8 + (lane & 3) * 2;
                    uint32_t hi, mid, lo;
                    in_three(acc[m][n][2 * e], acc[m][n][2 * e + 1], hi, mid, lo);
                    *reinterpret_cast<uint32_t*>(at) = hi;
                    *reinterpret_cast<uint32_t*>(at + N * VS) = mid;
                    *reinterpret_cast<uint32_t*>(at + 2 * N * VS) = lo;
                }
    };
    put_state();

    int nb = 0, buf = 0;
    for (int t0 = 0; t0 < q_len; t0 += nb, buf ^= 1) {
        cp_async_wait<0>();
#pragma unroll
        for (int w = 0; w < SC_T / X_ROWS; ++w) {  // (the copies that this thread made itself)
            const uint4 v = *reinterpret_cast<const uint4*>(X + (x_t + w * X_ROWS) * VS + x_c);
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
            bool odd = false;
#pragma unroll
            for (int e = 0; e < 4; ++e) odd |= (words[e] & 0x7f80u) == 0x7f80u || (words[e] & 0x7f800000u) == 0x7f800000u;
            if (odd) atomicMin(bad, x_t + w * X_ROWS);
        }
        __syncthreads();  // the chunk's rows, its gates and the state in front of it are there
        nb = min(SC_T, q_len - t0);
        const int first_bad = *bad;
        if (first_bad < nb) {
            nb = max(first_bad, 1);
            __syncthreads();
            for (int i = tid; i < (SC_T - nb) * CT; i += SC_THREADS)
                *reinterpret_cast<uint4*>(X + (nb + i / CT) * VS + (i % CT) * 8) = make_uint4(0u, 0u, 0u, 0u);
            // (and the keys: their weights in the state are 0, which an infinite key would make a NaN)
            for (int i = tid; i < (SC_T - nb) * RUNS; i += SC_THREADS)
                *reinterpret_cast<uint4*>(K + (nb + i / RUNS) * QS + (i % RUNS) * 8) = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
        }
        const float* lh = gate_row(buf, 0);
        const float* ll = gate_row(buf, 1);
        const float* wt = gate_row(buf, 2);
        const float end_h = lh[nb - 1], end_l = ll[nb - 1];
        if (tid >= SC_THREADS - SC_T) {
            const int t = tid - (SC_THREADS - SC_T);
            u_s[t] = t < nb ? expf((end_h - lh[t]) + (end_l - ll[t])) * wt[t] : 0.f;
        }
        if (makes_gates && t0 + nb < q_len) make_gates(buf ^ 1, t0 + nb, CELL ? gate_row(buf, 3)[nb - 1] : 0.f);

        // ---- (1)
        float o[CT][4], o_low[CT][4];  // products of the upper parts, and of the others
#pragma unroll
        for (int n = 0; n < CT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n][e] = o_low[n][e] = 0.f;
        float sum_lo = 0.f, sum_hi = 0.f;  // of the weighed scores: the normaliser's part
        if (warp >= 4) {
            if (rt * 16 < nb) {
                // queries times the state: two accumulators, each with the small parts' sum or nothing in front of one half of
                // the upper parts' products (the tensor core truncates as it adds)
                constexpr int KS = N / 16;
                const bf16* q_at = Q + (rt * 16 + (lane & 15)) * QS + ((lane >> 4) << 3);
                const bf16* s_at = Sp + ((lane & 7) + (((lane >> 3) & 1) << 3)) * VS + ((lane >> 4) << 3);
                uint32_t qf[2][4], sf[2][CT / 2][4];  // a step's operands, the next one's under way
                auto load_step = [&](int i, int at) {  // steps of the lowest parts, the middle ones, the upper ones
                    const int part = 2 - i / KS, ks = i % KS;
                    ldmatrix_x4(qf[at], q_at + ks * 16);
#pragma unroll
                    for (int n = 0; n < CT / 2; ++n) ldmatrix_x4_trans(sf[at][n], s_at + (part * N + ks * 16) * VS + n * 16);
                };
                load_step(0, 0);
#pragma unroll 1
                for (int i0 = 0; i0 < 3 * KS; i0 += KS / 2) {
                    const bool last = i0 == 3 * KS - KS / 2;
#pragma unroll
                    for (int j = 0; j < KS / 2; ++j) {
                        const int at = j & 1;
                        if (!last || j + 1 < KS / 2) load_step(i0 + j + 1, at ^ 1);
                        if (last) {
#pragma unroll
                            for (int n = 0; n < CT; ++n) mma_free(o[n], qf[at], sf[at][n / 2][2 * (n & 1)], sf[at][n / 2][2 * (n & 1) + 1]);
                        } else {
#pragma unroll
                            for (int n = 0; n < CT; ++n) mma_free(o_low[n], qf[at], sf[at][n / 2][2 * (n & 1)], sf[at][n / 2][2 * (n & 1) + 1]);
                        }
                    }
                }
#pragma unroll
                for (int n = 0; n < CT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[n][e] += o_low[n][e];
                const float f_lo = expf(lh[row_lo] + ll[row_lo]), f_hi = expf(lh[row_hi] + ll[row_hi]);
#pragma unroll
                for (int n = 0; n < CT; ++n) {
                    o[n][0] *= f_lo; o[n][1] *= f_lo;
                    o[n][2] *= f_hi; o[n][3] *= f_hi;
                }
                if (first_cols) {  // q . n in front of the chunk: two lanes a token
                    const int t = rt * 16 + (lane >> 1), d0 = (lane & 1) * (N / 2);
                    float dot = 0.f;
#pragma unroll 4
                    for (int d = 0; d < N / 2; d += 2) {
                        const uint32_t qv = *reinterpret_cast<const uint32_t*>(Q + t * QS + d0 + d);
                        const float2 nv = *reinterpret_cast<const float2*>(n_s + d0 + d);
                        dot = fmaf(__uint_as_float(qv << 16), nv.x, dot);
                        dot = fmaf(__uint_as_float(qv & 0xffff0000u), nv.y, dot);
                    }
                    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                    if ((lane & 1) == 0) dot_s[t] = dot * expf(lh[t] + ll[t]);
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");  // these four warps are done with the state's parts
            if (rt * 16 < nb) {
#pragma unroll
                for (int n = 0; n < CT; ++n) {
                    const int col = n * 8 + (lane & 3) * 2;
                    *reinterpret_cast<float2*>(part_s + row_lo * PS + col) = make_float2(o[n][0], o[n][1]);
                    *reinterpret_cast<float2*>(part_s + row_hi * PS + col) = make_float2(o[n][2], o[n][3]);
                }
            }
        } else if (rt * 16 < nb) {
            // e^(L_t - L_s) w_s: for keys in front of the 16 tokens by way of the first of them (neither factor grows), within
            // them directly
            const float h_lo = lh[row_lo], l_lo = ll[row_lo], h_hi = lh[row_hi], l_hi = ll[row_hi];
            const float h_0 = lh[rt * 16], l_0 = ll[rt * 16];
            const float a_lo = expf((h_lo - h_0) + (l_lo - l_0)), a_hi = expf((h_hi - h_0) + (l_hi - l_0));
            float* b_s = reinterpret_cast<float*>(smem + M::b) + rt * SC_T;
            for (int t = lane; t < rt * 16; t += 32) b_s[t] = expf((h_0 - lh[t]) + (l_0 - ll[t])) * wt[t];
            __syncwarp();
#pragma unroll 1
            for (int kt = 0; kt <= rt; ++kt) {
                float sc[2][4], sc_b[2][4];  // (two accumulators, as above)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[n][e] = sc_b[n][e] = 0.f;
                const bf16* q_at = Q + (rt * 16 + (lane & 15)) * QS + ((lane >> 4) << 3);
                const bf16* k_at = K + (kt * 16 + (lane & 7) + ((lane >> 4) << 3)) * QS + (((lane >> 3) & 1) << 3);
                uint32_t qf[2][2][4], kf[2][2][4];  // the operands of two steps of K, those of the next two under way
                auto load_two = [&](int ks, int at) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        ldmatrix_x4(qf[at][i], q_at + (ks + i) * 16);
                        ldmatrix_x4(kf[at][i], k_at + (ks + i) * 16);
                    }
                };
                load_two(0, 0);
#pragma unroll
                for (int ks = 0; ks < N / 16; ks += 2) {
                    const int at = (ks >> 1) & 1;
                    if (ks + 2 < N / 16) load_two(ks + 2, at ^ 1);
                    mma_free(sc[0], qf[at][0], kf[at][0][0], kf[at][0][1]);
                    mma_free(sc[1], qf[at][0], kf[at][0][2], kf[at][0][3]);
                    mma_free(sc_b[0], qf[at][1], kf[at][1][0], kf[at][1][1]);
                    mma_free(sc_b[1], qf[at][1], kf[at][1][2], kf[at][1][3]);
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[n][e] += sc_b[n][e];
                uint32_t w_hi[4], w_mid[4], w_lo[4];
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const int key = kt * 16 + n * 8 + (lane & 3) * 2;
                    float v[4];
                    if (kt < rt) {
                        const float2 b = *reinterpret_cast<const float2*>(b_s + key);
                        v[0] = sc[n][0] * (a_lo * b.x);
                        v[1] = sc[n][1] * (a_lo * b.y);
                        v[2] = sc[n][2] * (a_hi * b.x);
                        v[3] = sc[n][3] * (a_hi * b.y);
                    } else {
                        const float2 kh = *reinterpret_cast<const float2*>(lh + key), kl = *reinterpret_cast<const float2*>(ll + key);
                        const float2 kw = *reinterpret_cast<const float2*>(wt + key);
                        v[0] = key <= row_lo ? sc[n][0] * (expf((h_lo - kh.x) + (l_lo - kl.x)) * kw.x) : 0.f;
                        v[1] = key + 1 <= row_lo ? sc[n][1] * (expf((h_lo - kh.y) + (l_lo - kl.y)) * kw.y) : 0.f;
                        v[2] = key <= row_hi ? sc[n][2] * (expf((h_hi - kh.x) + (l_hi - kl.x)) * kw.x) : 0.f;
                        v[3] = key + 1 <= row_hi ? sc[n][3] * (expf((h_hi - kh.y) + (l_hi - kl.y)) * kw.y) : 0.f;
                    }
                    sum_lo += v[0] + v[1];
                    sum_hi += v[2] + v[3];
                    in_three(v[0], v[1], w_hi[2 * n], w_mid[2 * n], w_lo[2 * n]);
                    in_three(v[2], v[3], w_hi[2 * n + 1], w_mid[2 * n + 1], w_lo[2 * n + 1]);
                }
                // (products of one accumulator apart from one another: one has to wait for the one before it)
                uint32_t xb[CT / 2][4];
#pragma unroll
                for (int n = 0; n < CT; n += 2)
                    ldmatrix_x4_trans(xb[n / 2], X + (kt * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * VS + n * 8 + ((lane >> 4) << 3));
#pragma unroll
                for (int n = 0; n < CT; ++n) mma_free(o_low[n], w_lo, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
#pragma unroll
                for (int n = 0; n < CT; ++n) mma_free(o_low[n], w_mid, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
#pragma unroll
                for (int n = 0; n < CT; ++n) mma_free(o[n], w_hi, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
            }
            if (first_cols) {
#pragma unroll
                for (int d = 1; d <= 2; d <<= 1) {
                    sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, d);
                    sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, d);
                }
            }
        }
        __syncthreads();  // the queries have been used, both sums and the weights u are there
        const bool more = t0 + nb < q_len;
        if (more) fetch_rows(Q, q_src, t0 + nb);
        if (tid == 0) *bad = SC_T;

        // ---- (2) the outputs
        if (warp < 4) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = e ? row_hi : row_lo;
                if (t >= nb) continue;
                float* dst = g.out + ((int64_t)(q0 + t0 + t) * g.heads + h) * g.vdim + c0 + (lane & 3) * 2;
                float2 y[CT];  // (all reads before the writes, which the compiler does not move them across)
#pragma unroll
                for (int n = 0; n < CT; ++n) {
                    const int col = n * 8 + (lane & 3) * 2;
                    const float2 p = *reinterpret_cast<const float2*>(part_s + t * PS + col);
                    y[n] = make_float2(p.x + (o[n][2 * e] + o_low[n][2 * e]), p.y + (o[n][2 * e + 1] + o_low[n][2 * e + 1]));
                    if constexpr (CELL) {
                        y[n].x *= g.q_scale;
                        y[n].y *= g.q_scale;
                    } else {
                        const uint32_t xv = *reinterpret_cast<const uint32_t*>(X + t * VS + col);
                        y[n].x = fmaf(skip, __uint_as_float(xv << 16), y[n].x);
                        y[n].y = fmaf(skip, __uint_as_float(xv & 0xffff0000u), y[n].y);
                    }
                }
#pragma unroll
                for (int n = 0; n < CT; ++n)
                    if (c0 + n * 8 < g.vdim) *reinterpret_cast<float2*>(dst + n * 8) = y[n];
                if (first_cols && (lane & 3) == 0) g.nq[(int64_t)(q0 + t0 + t) * g.heads + h] = g.q_scale * (dot_s[t] + (e ? sum_hi : sum_lo));
            }
        }

        // ---- (2) the state behind the chunk
        const float f_end = expf(end_h + end_l);
#pragma unroll
        for (int m = 0; m < MPW; ++m) {
            float d[TPW][4];
#pragma unroll
            for (int n = 0; n < TPW; ++n) d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0.f;
            const int row0 = s_row(m) - (lane >> 2);
#pragma unroll
            for (int ks = 0; ks < SC_T / 16; ++ks) {
                if (ks * 16 >= nb) break;
                uint32_t ka[4], a_hi[4], a_mid[4], a_lo[4];
                ldmatrix_x4_trans(ka, K + (ks * 16 + (lane & 7) + ((lane >> 4) << 3)) * QS + row0 + (((lane >> 3) & 1) << 3));
#pragma unroll
                for (int e = 0; e < 2; ++e) {  // registers 2 e, 2 e + 1: tokens 2 (lane % 4) + 8 e and the next of the step
                    const float2 u = *reinterpret_cast<const float2*>(u_s + ks * 16 + e * 8 + (lane & 3) * 2);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t w = ka[2 * e + i];
                        in_three(__uint_as_float(w << 16) * u.x, __uint_as_float(w & 0xffff0000u) * u.y, a_hi[2 * e + i], a_mid[2 * e + i],
                                 a_lo[2 * e + i]);
                    }
                }
                uint32_t xb[TPW / 2][4];
#pragma unroll
                for (int n = 0; n < TPW; n += 2)
                    ldmatrix_x4_trans(xb[n / 2], X + (ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * VS + (s_tile + n) * 8 + ((lane >> 4) << 3));
#pragma unroll
                for (int n = 0; n < TPW; ++n) mma_free(d[n], a_lo, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
#pragma unroll
                for (int n = 0; n < TPW; ++n) mma_free(d[n], a_mid, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
#pragma unroll
                for (int n = 0; n < TPW; ++n) mma_free(d[n], a_hi, xb[n / 2][2 * (n & 1)], xb[n / 2][2 * (n & 1) + 1]);
            }
#pragma unroll
            for (int n = 0; n < TPW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][n][e] = fmaf(f_end, acc[m][n][e], d[n][e]);
        }
        if (first_cols)
            for (int i = tid; i < N; i += SC_THREADS) {
                float add = 0.f;
#pragma unroll 8
                for (int t = 0; t < SC_T; ++t) add = fmaf(u_s[t], to_float(K[t * QS + i]), add);
                n_s[i] = fmaf(f_end, n_s[i], add);
            }
        __syncthreads();  // the keys and values have been used, the sums in place of the state's parts read
        if (more) {
            put_state();
            fetch_rows(K, k_src, t0 + nb);
            fetch_values(t0 + nb);
        }
        cp_async_commit();
    }
#pragma unroll
    for (int m = 0; m < MPW; ++m)
#pragma unroll
        for (int n = 0; n < TPW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = s_row(m) + (e >> 1) * 8, col = c0 + (s_tile + n) * 8 + (lane & 3) * 2 + (e & 1);
                if (row < g.dim && col < g.vdim) sp[(int64_t)col * g.dim + row] = acc[m][n][e];
            }
    if (first_cols)
        for (int i = tid; i < g.dim; i += SC_THREADS) sp[(int64_t)g.vdim * g.dim + i] = n_s[i];
}

template <bool CELL, int N, int CT>
static int launch_scan_as(const ScanArgs& g, int R, cudaStream_t stream) {
    constexpr int smem = ScanSmem<N, CT>::bytes;
    static SsPerDevice opted;
    if (int rc = ss_opt_in_smem(scan_chunks_kernel<CELL, N, CT>, smem, opted)) return rc;
    const int64_t blocks = (int64_t)g.heads * ((g.vdim + CT * 8 - 1) / (CT * 8)) * R;  // along x, which takes any number of requests
    if (blocks >= (1ll << 31)) return (int)cudaErrorInvalidValue;
    ss_launch(scan_chunks_kernel<CELL, N, CT>, dim3((unsigned)blocks), dim3(SC_THREADS), smem, stream, g);
    return SS_LAUNCH_CHECK();
}

// 64 columns a block; 32 beyond 128 elements of a key, for shared memory, and where 64 leave SMs without a block (twice
// the blocks form every score twice: 112 heads of 64 columns, one request of 2,048 tokens 252 -> 229 us).
template <bool CELL>
static int launch_scan(ScanArgs& g, int R, cudaStream_t stream) {
    g.sms = ss_sm_count();
    if (g.dim > 128) return launch_scan_as<CELL, 256, 4>(g, R, stream);
    const bool narrow = g.vdim <= 32 || (int64_t)g.heads * R * ((g.vdim + 63) / 64) <= ss_sm_count();
    if (g.dim > 64) return narrow ? launch_scan_as<CELL, 128, 4>(g, R, stream) : launch_scan_as<CELL, 128, 8>(g, R, stream);
    return launch_scan_as<CELL, 64, 8>(g, R, stream);
}

static bool scan_fits(const ScanArgs& g) {
    return g.dim >= 8 && g.dim <= 256 && g.dim % 8 == 0 && g.vdim >= 8 && g.vdim % 8 == 0 && g.stride % 8 == 0 &&
           (((uintptr_t)g.q | (uintptr_t)g.k | (uintptr_t)g.x | (uintptr_t)g.out) & 15) == 0;
}

}  // namespace

// bfloat16 rows; N and P in steps of 8, xbc's rows on 16-byte boundaries.  Arguments as ss_ssm_scan (ops_mixers.cu).
extern "C" int ss_ssm_scan_chunks(const void* xbc, int C, const void* dt_raw, int64_t dt_stride, const float* dt_bias, const float* a_log,
                                  const float* d_skip, float* state, float* y, const int32_t* q_start, const int32_t* seq_lens,
                                  const int32_t* slots, int R, int heads, int groups, int P, int N, int n_slots, int* err,
                                  cudaStream_t stream) {
    if (R <= 0) return 0;
    if (groups < 1 || heads < 1 || heads % groups) return (int)cudaErrorInvalidValue;
    ScanArgs g{};
    g.x = (const bf16*)xbc;
    g.k = g.x + (int64_t)heads * P;
    g.q = g.k + (int64_t)groups * N;
    g.stride = C;
    g.state = state; g.out = y; g.q_start = q_start; g.seq_lens = seq_lens; g.slots = slots;
    g.heads = heads; g.group = heads / groups; g.dim = N; g.vdim = P; g.n_slots = n_slots; g.err = err;
    g.dt = (const bf16*)dt_raw; g.dt_stride = dt_stride; g.dt_bias = dt_bias; g.a_log = a_log; g.d_skip = d_skip;
    if (!scan_fits(g)) return (int)cudaErrorInvalidValue;
    return launch_scan<false>(g, R, stream);
}

// bfloat16 rows; D and V in steps of 8, rows on 16-byte boundaries.  Arguments as ss_matrix_cell (ops_cells.cu).
extern "C" int ss_matrix_cell_chunks(const void* qkv, int64_t stride, const float* gates, int64_t gate_stride, const float* bias_i,
                                     const float* bias_f, float cap, float q_scale, float* memory, float* peak, float* num, float* nq,
                                     float* peaks_out, const int32_t* q_start, const int32_t* seq_lens, const int32_t* slots, int R, int H,
                                     int D, int V, int n_slots, int* err, cudaStream_t stream) {
    if (R <= 0) return 0;
    if (H < 1 || !(cap > 0.f)) return (int)cudaErrorInvalidValue;
    ScanArgs g{};
    g.q = (const bf16*)qkv;
    g.k = g.q + (int64_t)H * D;
    g.x = g.k + (int64_t)H * D;
    g.stride = stride;
    g.state = memory; g.out = num; g.q_start = q_start; g.seq_lens = seq_lens; g.slots = slots;
    g.heads = H; g.group = 1; g.dim = D; g.vdim = V; g.n_slots = n_slots; g.err = err;
    g.gates = gates; g.gate_stride = gate_stride; g.bias_i = bias_i; g.bias_f = bias_f; g.cap = cap; g.q_scale = q_scale;
    g.peak = peak; g.nq = nq; g.peaks_out = peaks_out;
    if (!scan_fits(g)) return (int)cudaErrorInvalidValue;
    if (int rc = launch_scan<true>(g, R, stream)) return rc;
    return launch_cell_peaks(peaks_out, peak, q_start, seq_lens, slots, R, H, n_slots, stream);
}
