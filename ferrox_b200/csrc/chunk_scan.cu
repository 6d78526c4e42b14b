// Recurrences of a matrix state per head over the tokens of a prompt, CHUNK tokens at a time instead of one by one:
//
//   mLSTM      S <- keep_t S + take_t k_t v_t^T, n likewise with k_t alone         o_t = S^T q_t / max(|n.q_t|, ..)
//   delta      S <- g_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T     o_t = S^T q_t
//   general    S <- diag(w_t) S - (a_t u_t)(u_t^T S) + k_t v_t^T                  o_t = S^T r_t
//
// (linear_state.cu, general_delta.cu, mlstm.cu state them and take steps of few tokens.)  Within a
// chunk the tokens meet through products of their keys and queries alone, so that everything but the state itself is
// worked out for all chunks at once, and what remains in the tokens' order is three small matrix products a chunk.
// With R_ts the product of the decays of tokens s+1 .. t and G_t = R_t0 that of the chunk's tokens up to t:
//
//   delta:    (I + L) U = diag(beta) V - diag(beta G) K S_0,  L_ts = beta_t R_ts k_t.k_s  (s < t)
//             U = U0 - W S_0 with [U0 | W] = (I + L)^-1 [diag(beta) V | diag(beta G) K]
//             o_t = G_t S_0^T q_t + sum_{s <= t} R_ts (q_t.k_s) u_s,   S_C = G_C S_0 + sum_s R_Cs k_s u_s^T
//   mLSTM:    the same with U = V and no product with W
//   general:  decays per key channel: rows scaled by the channels' products, u'_t = u_t G_(t-1), r'_t = r_t G_t,
//             k'_s = k_s / G_s, a'_s = a_s u_s / G_s;  y_t = u_t^T S_(t-1) solves
//             (I + A) Y = u' S_0 + B V,  A_ts = u'_t.a'_s, B_ts = u'_t.k'_s (s < t);  Y = Y0 + W S_0
//             o_t = S_0^T r'_t + sum_{s <= t} (r'_t.k'_s) v_s - (r'_t.a'_s) y_s
//             S_C = diag(G_C) S_0 + sum_s (G_C k'_s) v_s^T - (G_C a'_s) y_s^T
//             (decays above exp(-rate): over 32 tokens of a rate of 1 the products stay above 1.2e-14 and k' below 8e13 k, with
//             room to numbers' end, and every term is a ratio <= 1; stronger decays are taken token by token)
//
// Everything is 32-bit FFMA arithmetic; products of decays are taken in 64 bits and rounded once, because one of a
// chunk's is raised to the power of the chunks that a memory travels through.  State [slots, H, V, D], as before.
// Error against a 64-bit evaluation, as a multiple of that of the kernels that take the tokens one by one (read-outs and
// states; seven shapes, twelve seeds): delta 0.99 and 0.89, general 0.87 and 0.72, mLSTM's states 0.97.  It takes short chains
// in the products of a chunk's rows (in one chain of pairs a row: 1.14 for delta, 1.16 for general), a token's product with
// itself from the rows as they are, decays after a token as products of their own instead of G_C / G_t, a chunk's sum made
// before the state is added to it, and the mLSTM's maxima in 64 bits (states 1.1).
//
// Kernels: *_chunks make what a chunk needs (a block a chunk and head); walk_kernel goes through an entry's chunks in
// order (a block 16 columns of a head's state).  A walk's chunk is bound by what shared memory delivers to registers (128 bytes
// a cycle, broadcasts counted whole: 4,300 of a chunk's 5,900 cycles for heads of 128 under the delta rule, before the update's
// values were read once and doubled in registers), at 8 warps an SM; twice the warps, one half reading out while the other
// updates, took as long.  The block's tiles are as many columns as one prompt's heads leave SMs for (16 heads of 128
// columns: 128 blocks).  Where the host says which entry is how long, the longest is walked first (3,001 tokens in three
// prompts of 32 heads of 64, generalized: 297 us one block an SM in the batch's order, 246 two an SM and the longest first,
// 226 with the values read once; 2,048 of 16 heads of 128, delta: 202, 199, 186).
// The next chunk's rows travel meanwhile, a TMA box a tensor where the heads fill the tile and the
// chunk is whole, else by cp.async, whose writes take 1,500 of a chunk's cycles of shared memory (2,048 tokens of 16
// heads of 128: 239 us by cp.async where boxes took 215; by untiled bulk copies,
// one a row, 160 a chunk: twice as long).
#include <stddef.h>

#include "tc_common.cuh"
#include "api.h"

namespace {

constexpr int CHUNK = 32;
constexpr int COLS = 16;             // columns of the state a walking block owns
constexpr int WALK_THREADS = 256;
constexpr int PREP_THREADS = 256;
typedef unsigned long long u64;

__device__ __forceinline__ void fma2(u64& d, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ u64 fma2_of(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 pair(float x, float y) {
    return (u64)__float_as_uint(x) | ((u64)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float lo_of(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_of(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ float sum_of(u64 v) { return lo_of(v) + hi_of(v); }

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
    const int n = ok ? 16 : 0;       // the rest is filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp4(float* dst, const float* src, bool ok) {
    const int n = ok ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n));
}

// first row r with token_seq[r] >= b
__device__ __forceinline__ int first_row_of(const int* __restrict__ token_seq, int n_tokens, int b)
{
    int lo = 0, hi = n_tokens;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (token_seq[mid] < b) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// D rows of CHUNK tokens into shared memory, `pitch` floats apart, zeros beyond `rows` and beyond `d`.
template <int D, int THREADS>
__device__ __forceinline__ void load_rows(float* to, int pitch, const float* from, long ld, int rows, int d)
{
    constexpr int P = D / 4;
    for (int i = threadIdx.x; i < CHUNK * P; i += THREADS) {
        const int t = i / P, c = (i - t * P) * 4;
        const bool ok = t < rows && c < d;
        cp16(to + t * pitch + c, from + (ok ? (long)t * ld + c : 0), ok);
    }
}

// ------------------------------------------------------------------------------------------------ what a chunk needs
struct ChunkArgs {
    const int* tiles;                // [n][4]: first token, tokens, entry, position
    const float *q, *k, *v; long ldq, ldk, ldv;
    const float *a_pre, *low; long lda, ldl; int rank;     // general: rows [T, H * D] and [T, rank], W2 [H * D, rank] and so on
    const void *w2, *w0, *ab; int w2_dtype, w0_dtype, ab_dtype; float rate;
    float *qs, *ks, *as;             // general: r', G_C k' and -G_C a'  [T, H * D]
    const float* g;                  // decays [T, H]
    const float* gate;               // delta: beta [T, H]; mLSTM: take [T, H]
    float scale;                     // on q (mLSTM)
    int H, G, D, V;
    float *p;                        // [T, H, CHUNK or 2 CHUNK]: weights of the chunk's tokens in a token's read-out
    float *gam, *e;                  // [T, H]: G_t; R_Cs (mLSTM: times take_s).  general: gam [tiles, H, D], G_C
    float *x0, *wr;                  // [T, H, V], [T, H, D]: U0 or Y0, W
};

// Products of a chunk's decays: win[j][t] that of the 2^j tokens up to t (as many as there are), so that any run's product
// takes at most five factors.  By the first warp; tokens beyond the chunk's rows count as decays of one.
__device__ __forceinline__ void decay_windows(float g, double (*win)[CHUNK])
{
    const int t = threadIdx.x;
    double w = (double)g;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        win[j][t] = w;
        if (j == 5) break;
        const double before = __shfl_up_sync(0xffffffffu, w, 1 << j);
        if (t >= 1 << j) w *= before;
    }
}
// That of the n tokens up to t (n < 32).
__device__ __forceinline__ float decay_product(const double (*win)[CHUNK], int t, int n)
{
    double r = 1.0;
#pragma unroll
    for (int j = 0; j < 5; ++j)
        if (n >> j & 1) { r *= win[j][t]; t -= 1 << j; }
    return (float)r;
}

// One product of two rows as N chains of pairs: what a chunk's tokens are to each other enters every later sum whole.
template <int N> struct Sums {
    u64 c[N];
    __device__ __forceinline__ Sums() {
#pragma unroll
        for (int n = 0; n < N; ++n) c[n] = 0ull;
    }
    __device__ __forceinline__ void add(int n, const ulonglong2& a, const ulonglong2& b) { fma2(c[n], a.x, b.x); fma2(c[n + 1], a.y, b.y); }
    __device__ __forceinline__ float sum() const {
        float s[N];
#pragma unroll
        for (int n = 0; n < N; ++n) s[n] = sum_of(c[n]);
#pragma unroll
        for (int w = N / 2; w > 0; w >>= 1)
#pragma unroll
            for (int n = 0; n < w; ++n) s[n] += s[n + w];
        return s[0];
    }
};

// sum of l[s] x[s] over the tokens s < t (t known when compiled: x stays in registers)
__device__ __forceinline__ float before(const float* l, const float (&x)[CHUNK], int t)
{
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int s = 0; s < t; s += 4) {
        const float4 a = *reinterpret_cast<const float4*>(l + s);
        s0 = fmaf(a.x, x[s], s0);
        if (s + 1 < t) s1 = fmaf(a.y, x[s + 1], s1);
        if (s + 2 < t) s0 = fmaf(a.z, x[s + 2], s0);
        if (s + 3 < t) s1 = fmaf(a.w, x[s + 3], s1);
    }
    return s0 + s1;
}

template <int D, bool DELTA>
__global__ void __launch_bounds__(PREP_THREADS, 2) scalar_chunks(ChunkArgs a)
{
    constexpr int PITCH = D + 4, LP = CHUNK + 4, CHAINS = 4;
    extern __shared__ __align__(16) float sm[];
    float* k_s = sm;                                  // [CHUNK][PITCH]
    float* q_s = k_s + CHUNK * PITCH;
    float* l_s = q_s + CHUNK * PITCH;                 // [CHUNK][LP]
    __shared__ double win[6][CHUNK];
    __shared__ float gam[CHUNK], gate_s[CHUNK];
    fx_pdl_wait();
    const int4 tile = reinterpret_cast<const int4*>(a.tiles)[blockIdx.x];
    const int tok0 = tile.x, rows = tile.y, h = blockIdx.y, tid = threadIdx.x;
    const int kvh = h / (a.H / a.G);
    load_rows<D, PREP_THREADS>(k_s, PITCH, a.k + (long)tok0 * a.ldk + (long)kvh * a.D, a.ldk, rows, a.D);
    load_rows<D, PREP_THREADS>(q_s, PITCH, a.q + (long)tok0 * a.ldq + (long)kvh * a.D, a.ldq, rows, a.D);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // (the first column of the substitution below: its values travel while the chunk's products are made)
    float x[CHUNK];
    if (DELTA && tid < a.V) {
        const float* vp = a.v + (long)tok0 * a.ldv + (long)h * a.V + tid;
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) x[t] = t < rows ? vp[(long)t * a.ldv] : 0.f;
    }
    if (tid < CHUNK) {
        const bool ok = tid < rows;
        decay_windows(ok ? a.g[(long)(tok0 + tid) * a.H + h] : 1.f, win);
        gam[tid] = (float)win[5][tid];
        gate_s[tid] = ok ? a.gate[(long)(tok0 + tid) * a.H + h] : 0.f;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // thread (ty, tx): tokens t = ty, ty + 16 against s = tx, tx + 16
    const int ty = tid >> 4, tx = tid & 15;
    Sums<CHAINS> qk[2][2], kk[2][2];
#pragma unroll 2
    for (int d0 = 0; d0 < D; d0 += 2 * CHAINS) {
#pragma unroll
        for (int n = 0; n < CHAINS; n += 2) {
            const int d = d0 + 2 * n;
            ulonglong2 ks[2], qt[2], kt[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                ks[i] = *reinterpret_cast<const ulonglong2*>(k_s + (tx + 16 * i) * PITCH + d);
                qt[i] = *reinterpret_cast<const ulonglong2*>(q_s + (ty + 16 * i) * PITCH + d);
                if (DELTA) kt[i] = *reinterpret_cast<const ulonglong2*>(k_s + (ty + 16 * i) * PITCH + d);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    qk[i][j].add(n, qt[i], ks[j]);
                    if (DELTA) kk[i][j].add(n, kt[i], ks[j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = ty + 16 * i, s = tx + 16 * j;
            const float r = s < t ? decay_product(win, t, t - s) : 1.f;
            if (DELTA) l_s[t * LP + s] = s < t ? gate_s[t] * (r * kk[i][j].sum()) : 0.f;
            if (t < rows)
                a.p[((long)(tok0 + t) * a.H + h) * CHUNK + s] =
                    s <= t ? r * qk[i][j].sum() * (DELTA ? 1.f : a.scale * gate_s[s]) : 0.f;
        }
    if (tid < rows) {
        a.gam[(long)(tok0 + tid) * a.H + h] = gam[tid];
        a.e[(long)(tok0 + tid) * a.H + h] = decay_product(win, rows - 1, rows - 1 - tid) * (DELTA ? 1.f : gate_s[tid]);
    }
    if (!DELTA) return;
    __syncthreads();
    // forward substitution, a column a thread
    for (int c = tid; c < a.V + a.D; c += PREP_THREADS) {
        const bool val = c < a.V;
        if (val && c >= PREP_THREADS) {
            const float* vp = a.v + (long)tok0 * a.ldv + (long)h * a.V + c;
#pragma unroll
            for (int t = 0; t < CHUNK; ++t) x[t] = t < rows ? vp[(long)t * a.ldv] : 0.f;
        } else if (!val) {
#pragma unroll
            for (int t = 0; t < CHUNK; ++t) x[t] = gam[t] * k_s[t * PITCH + c - a.V];
        }
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) x[t] *= gate_s[t];
#pragma unroll
        for (int t = 1; t < CHUNK; ++t) {
            x[t] -= before(l_s + t * LP, x, t);
        }
        float* to = val ? a.x0 + ((long)tok0 * a.H + h) * a.V + c : a.wr + ((long)tok0 * a.H + h) * a.D + (c - a.V);
        const long ld = (long)a.H * (val ? a.V : a.D);
#pragma unroll
        for (int t = 0; t < CHUNK; ++t)
            if (t < rows) to[t * ld] = x[t];
    }
}

constexpr int RANK = 64;             // low-rank columns a pass

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// The decays and rates come from the projections' rows here as well (general_delta.cu states them: w = exp(-rate sigmoid(W2
// tanh(low) + w0)), a = sigmoid(a_pre + bias), u = k / sqrt(sum k^2 + 1e-6)): a block has a head's slice of W2 in shared
// memory for 32 tokens, and u, a u and w never go to memory.  (The kernel that makes them for the token-by-token form,
// eight tokens a block, took 249 us for 3,001 tokens of 32 heads of 64.)
template <int D>
__global__ void __launch_bounds__(PREP_THREADS, D <= 64 ? 2 : 1) general_chunks(ChunkArgs a)
{
    constexpr int PITCH = D + 4, LP = CHUNK + 4, RP = RANK + 4, CHAINS = D <= 64 ? 2 : 4;
    extern __shared__ __align__(16) float sm[];
    float* u_s = sm;                                  // [CHUNK][PITCH] each
    float* r_s = u_s + CHUNK * PITCH;
    float* k_s = r_s + CHUNK * PITCH;
    float* a_s = k_s + CHUNK * PITCH;
    float* g_s = a_s + CHUNK * PITCH;                 // decays, then their products up to each token
    float* A_s = g_s + CHUNK * PITCH;                 // [CHUNK][LP]
    float* B_s = A_s + CHUNK * LP;
    float* w2_s = B_s + CHUNK * LP;                   // [D][RP]
    float* th_s = w2_s + D * RP;                      // [CHUNK][RP]
    float* e_s = w2_s;                                // (when W2 has been read) products of the decays after each token
    __shared__ float len_s[CHUNK], rk_s[CHUNK], ra_s[CHUNK];
    fx_pdl_wait();
    const int4 tile = reinterpret_cast<const int4*>(a.tiles)[blockIdx.x];
    const int tok0 = tile.x, rows = tile.y, h = blockIdx.y, tid = threadIdx.x;
    const long hd = (long)a.H * a.D, at0 = (long)tok0 * hd + (long)h * a.D;
    load_rows<D, PREP_THREADS>(k_s, PITCH, a.k + (long)tok0 * a.ldk + (long)h * a.D, a.ldk, rows, a.D);
    load_rows<D, PREP_THREADS>(a_s, PITCH, a.a_pre + (long)tok0 * a.lda + (long)h * a.D, a.lda, rows, a.D);
    load_rows<D, PREP_THREADS>(r_s, PITCH, a.q + (long)tok0 * a.ldq + (long)h * a.D, a.ldq, rows, a.D);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // (the values of the first column of the substitution below travel meanwhile)
    float v[CHUNK];
    if (tid < a.V) {
        const float* vp = a.v + (long)tok0 * a.ldv + (long)h * a.V + tid;
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) v[t] = t < rows ? vp[(long)t * a.ldv] : 0.f;
    }
    // tanh(low) W2^T: thread (zy, zx) tokens zy, zy + 16, channels zx + 16 j
    const int zy = tid >> 4, zx = tid & 15;
    u64 zacc[2][D / 16];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < D / 16; ++j) zacc[i][j] = 0ull;
    for (int rc = 0; rc < a.rank; rc += RANK) {
        const int nr = min(RANK, a.rank - rc);
        __syncthreads();
        if (a.rank % 4 == 0 && (uintptr_t)a.w2 % 16 == 0) {     // four columns a load
#pragma unroll
            for (int n = 0; n < D * RANK / 4 / PREP_THREADS; ++n) {
                const int i = tid + n * PREP_THREADS, d = i / (RANK / 4), r = (i % (RANK / 4)) * 4;
                const long at = ((long)h * a.D + d) * a.rank + rc + r;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < nr && d < a.D) {
                    if (a.w2_dtype == FX_F32) {
                        x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.w2) + at);
                    } else {
                        const uint2 b = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(a.w2) + at);
                        x.x = __uint_as_float(b.x << 16); x.y = __uint_as_float(b.x & 0xffff0000u);
                        x.z = __uint_as_float(b.y << 16); x.w = __uint_as_float(b.y & 0xffff0000u);
                    }
                }
                *reinterpret_cast<float4*>(w2_s + d * RP + r) = x;
            }
        } else {
            for (int i = tid; i < D * RANK; i += PREP_THREADS) {
                const int d = i / RANK, r = i - d * RANK;
                w2_s[d * RP + r] = r < nr && d < a.D ? load_any(a.w2, a.w2_dtype, ((long)h * a.D + d) * a.rank + rc + r) : 0.f;
            }
        }
        {
            float x[CHUNK * RANK / PREP_THREADS];       // (all loads before the first tanh)
#pragma unroll
            for (int n = 0; n < CHUNK * RANK / PREP_THREADS; ++n) {
                const int i = tid + n * PREP_THREADS, t = i / RANK, r = i % RANK;
                x[n] = r < nr && t < rows ? a.low[(long)(tok0 + t) * a.ldl + rc + r] : 0.f;
            }
#pragma unroll
            for (int n = 0; n < CHUNK * RANK / PREP_THREADS; ++n) {
                const int i = tid + n * PREP_THREADS;
                th_s[i / RANK * RP + i % RANK] = tanhf(x[n]);
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int r = 0; r < RANK; r += 4) {
            ulonglong2 th[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) th[i] = *reinterpret_cast<const ulonglong2*>(th_s + (zy + 16 * i) * RP + r);
#pragma unroll
            for (int j = 0; j < D / 16; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w2_s + (zx + 16 * j) * RP + r);
#pragma unroll
                for (int i = 0; i < 2; ++i) { fma2(zacc[i][j], th[i].x, w.x); fma2(zacc[i][j], th[i].y, w.y); }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    {
        const int t = tid >> 3;                       // a token's key length, eight threads a token
        float ss = 0.f;
        for (int d = tid & 7; d < D; d += 8) ss = fmaf(k_s[t * PITCH + d], k_s[t * PITCH + d], ss);
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        if ((tid & 7) == 0) len_s[t] = sqrtf(ss + 1e-6f);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
            const int t = zy + 16 * i, d = zx + 16 * j, c = h * a.D + d;
            if (d >= a.D) { u_s[t * PITCH + d] = 0.f; g_s[t * PITCH + d] = 1.f; continue; }
            const float u = k_s[t * PITCH + d] / len_s[t];
            u_s[t * PITCH + d] = u;
            a_s[t * PITCH + d] = sigmoid_f(a_s[t * PITCH + d] + load_any(a.ab, a.ab_dtype, c)) * u;
            g_s[t * PITCH + d] = expf(-a.rate * sigmoid_f(sum_of(zacc[i][j]) + load_any(a.w0, a.w0_dtype, c)));
        }
    __syncthreads();
    {
        // what a token reads of itself, from the rows as they are: in most read-outs the largest term
        const int t = tid >> 3;
        float rk = 0.f, ra = 0.f;
        for (int d = (tid & 7) * 4; d < D; d += 32) {
            const float4 r = *reinterpret_cast<const float4*>(r_s + t * PITCH + d), k = *reinterpret_cast<const float4*>(k_s + t * PITCH + d);
            const float4 x = *reinterpret_cast<const float4*>(a_s + t * PITCH + d);
            rk = fmaf(r.x, k.x, rk); rk = fmaf(r.y, k.y, rk); rk = fmaf(r.z, k.z, rk); rk = fmaf(r.w, k.w, rk);
            ra = fmaf(r.x, x.x, ra); ra = fmaf(r.y, x.y, ra); ra = fmaf(r.z, x.z, ra); ra = fmaf(r.w, x.w, ra);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) { rk += __shfl_xor_sync(0xffffffffu, rk, o); ra += __shfl_xor_sync(0xffffffffu, ra, o); }
        if ((tid & 7) == 0) { rk_s[t] = rk; ra_s[t] = ra; }
    }
    // a channel's products of decays up to each token and after it: runs of RUN tokens a thread, then the runs on either side
    constexpr int RUNS = PREP_THREADS / D, RUN = CHUNK / RUNS;
    __shared__ double total[RUNS][D];
    {
        const int d = tid % D, run = tid / D;
        float g[RUN];
        double p = 1.0, q = 1.0;
#pragma unroll
        for (int i = 0; i < RUN; ++i) {
            const int t = run * RUN + i;
            g[i] = t < rows && d < a.D ? g_s[t * PITCH + d] : 1.f;
            p *= (double)g[i];
        }
        total[run][d] = p;
        __syncthreads();
        p = 1.0;
        for (int i = 0; i < run; ++i) p *= total[i][d];
        for (int i = run + 1; i < RUNS; ++i) q *= total[i][d];
#pragma unroll
        for (int i = 0; i < RUN; ++i) {
            p *= (double)g[i];
            g_s[(run * RUN + i) * PITCH + d] = (float)p;
            e_s[(run * RUN + RUN - 1 - i) * PITCH + d] = (float)q;
            q *= (double)g[RUN - 1 - i];
        }
        if (run == RUNS - 1 && d < a.D) a.gam[((long)blockIdx.x * a.H + h) * a.D + d] = (float)p;
    }
    __syncthreads();
    for (int i = tid; i < CHUNK * D; i += PREP_THREADS) {
        const int t = i / D, d = i - t * D, at = t * PITCH + d;
        const float g = g_s[at], e = e_s[at], k = k_s[at], x = a_s[at], rr = r_s[at] * g;
        u_s[at] *= t ? g_s[at - PITCH] : 1.f;
        k_s[at] = k / g; a_s[at] = x / g; r_s[at] = rr;
        if (t < rows && d < a.D) {
            const long to = at0 + (long)t * hd + d;
            a.qs[to] = rr; a.ks[to] = k * e; a.as[to] = -x * e;
        }
    }
    __syncthreads();
    const int ty = tid >> 4, tx = tid & 15;
    Sums<CHAINS> ua[2][2], uk[2][2], ra[2][2], rk[2][2];
#pragma unroll 2
    for (int d0 = 0; d0 < D; d0 += 2 * CHAINS) {
#pragma unroll
        for (int n = 0; n < CHAINS; n += 2) {
            const int d = d0 + 2 * n;
            ulonglong2 ks[2], as[2], ut[2], rt[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                ks[i] = *reinterpret_cast<const ulonglong2*>(k_s + (tx + 16 * i) * PITCH + d);
                as[i] = *reinterpret_cast<const ulonglong2*>(a_s + (tx + 16 * i) * PITCH + d);
                ut[i] = *reinterpret_cast<const ulonglong2*>(u_s + (ty + 16 * i) * PITCH + d);
                rt[i] = *reinterpret_cast<const ulonglong2*>(r_s + (ty + 16 * i) * PITCH + d);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    ua[i][j].add(n, ut[i], as[j]); uk[i][j].add(n, ut[i], ks[j]);
                    ra[i][j].add(n, rt[i], as[j]); rk[i][j].add(n, rt[i], ks[j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = ty + 16 * i, s = tx + 16 * j;
            A_s[t * LP + s] = s < t ? ua[i][j].sum() : 0.f;
            B_s[t * LP + s] = s < t ? uk[i][j].sum() : 0.f;
            if (t < rows) {
                float* p = a.p + ((long)(tok0 + t) * a.H + h) * (2 * CHUNK);
                p[s] = s < t ? rk[i][j].sum() : s == t ? rk_s[t] : 0.f;
                p[CHUNK + s] = s < t ? -ra[i][j].sum() : s == t ? -ra_s[t] : 0.f;
            }
        }
    __syncthreads();
    for (int c = tid; c < a.V + a.D; c += PREP_THREADS) {
        const bool val = c < a.V;
        float x[CHUNK];
        if (val) {
            x[0] = 0.f;      // (V <= PREP_THREADS: its values are here)
#pragma unroll
            for (int t = 1; t < CHUNK; ++t) {
                x[t] = before(B_s + t * LP, v, t);
            }
        } else {
#pragma unroll
            for (int t = 0; t < CHUNK; ++t) x[t] = u_s[t * PITCH + c - a.V];
        }
#pragma unroll
        for (int t = 1; t < CHUNK; ++t) {
            x[t] -= before(A_s + t * LP, x, t);
        }
        float* to = val ? a.x0 + ((long)tok0 * a.H + h) * a.V + c : a.wr + ((long)tok0 * a.H + h) * a.D + (c - a.V);
        const long ld = (long)a.H * (val ? a.V : a.D);
#pragma unroll
        for (int t = 0; t < CHUNK; ++t)
            if (t < rows) to[t * ld] = x[t];
    }
}

// The gates of an mLSTM and its running maximum of their logarithms (mlstm.cu states them): a warp an (entry, head), a lane
// a token.  m_t = max(f_t + m_(t-1), i_t) is a scan under (f, i) o (f', i') = (f + f', max(i + f', i')).  The scan's sums are of
// other numbers than the chain's, and a state (S, n, m) is off by what its maximum is off: so it runs in 64 bits up to the step's
// last token (2,048 tokens of 16 heads: 24 us in 32 bits, 31 us).
__device__ __forceinline__ float logsigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

__global__ void __launch_bounds__(32) mlstm_gates_kernel(const float* __restrict__ gates, long ldg, const void* i_bias,
                                                         const void* f_bias, int bias_dtype, float cap, float* m_state, int copies,
                                                         const float* __restrict__ norm, float* __restrict__ norm_in, int D, float* __restrict__ keep, float* __restrict__ take, float* __restrict__ floor_out,
                                                         const int* __restrict__ token_seq, const int* __restrict__ seq_slot,
                                                         int n_tokens, int H)
{
    fx_pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, lane = threadIdx.x;
    const int r0 = first_row_of(token_seq, n_tokens, b), r1 = first_row_of(token_seq, n_tokens, b + 1);
    if (r1 <= r0) return;
    float* mp = m_state + ((long)seq_slot[b] * H + h) * copies;
    // (the walk's blocks start from a copy: the first of them moves the state's own on while others may not have begun)
    for (int d = lane; d < D; d += 32) norm_in[((long)b * H + h) * D + d] = norm[((long)seq_slot[b] * H + h) * copies * D + d];
    const float bi = load_any(i_bias, bias_dtype, h), bf = load_any(f_bias, bias_dtype, h), inv_cap = 1.0f / cap;
    double m = mp[0];
    float in_i = gates[(long)min(r0 + lane, r1 - 1) * ldg + h], in_f = gates[(long)min(r0 + lane, r1 - 1) * ldg + H + h];
    for (int c0 = r0; c0 < r1; c0 += 32) {
        const int t = c0 + lane;
        const double gi = cap * tanhf((in_i + bi) * inv_cap);
        const double gf = logsigmoid_f(cap * tanhf((in_f + bf) * inv_cap));
        const float* g = gates + (long)min(t + 32, r1 - 1) * ldg;      // (the next tokens' inputs travel meanwhile)
        in_i = g[h]; in_f = g[H + h];
        double f = gf, i = gi;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double pf = __shfl_up_sync(0xffffffffu, f, o), pi = __shfl_up_sync(0xffffffffu, i, o);
            if (lane >= o) { i = fmax(pi + f, i); f = pf + f; }
        }
        double after = fmax(f + m, i);
        if (t == r1 - 1) after = (float)after;                         // as the state keeps it
        double before = __shfl_up_sync(0xffffffffu, after, 1);
        if (lane == 0) before = m;
        if (t < r1) {
            const long at = (long)t * H + h;
            keep[at] = expf((float)(gf + before - after));
            take[at] = expf((float)(gi - after));
            floor_out[at] = expf((float)-after);
        }
        m = __shfl_sync(0xffffffffu, after, min(31, r1 - 1 - c0));
    }
    for (int i = lane; i < copies; i += 32) mp[i] = (float)m;
}

// ------------------------------------------------------------------------------------------------------ the walk
struct WalkArgs {
    const float* w;                            // rows of W [T, H * D] (not mLSTM)
    const float* q; long ldq; int q_share;     // rows of q (general: r'), heads that share one
    const float* k; long ldk;                  // rows of k (general: G_C k')
    const float* a;                            // general: -G_C a'  [T, H * D]
    const float* v; long ldv;                  // general, mLSTM: values
    const float* x0;                           // delta: U0, general: Y0  [T, H * V]
    const float *p, *gam, *e;
    const float* floor_m;                      // mLSTM: exp(-m_t) [T, H], or null
    const float* norm_in;                      // mLSTM: the normaliser before the step [entries, H, D]
    float* norm; int copies;                   // and its copies in the state [slots, H, copies, D]
    float q_scale;                             // mLSTM: on q
    float* state; float* out; long ldo;
    const int *token_seq, *seq_slot;
    const int* tiles; int n_tiles;             // general: as for the chunks' kernel
    const int* walks;                          // (or null) per entry (index, first token, one past the last, first chunk), longest first
    int n_tokens, H, D, V;
    int tma;                                   // whole chunks by the boxes of WalkMaps
    int* status;                               // raised where a wait for them runs out
};
// [heads][tokens][D] of W, Q, K and (general) the third's rows, a box a chunk's rows of a head
struct WalkMaps { CUtensorMap w, q, k, a; };

enum { DELTA_RULE = 1, GENERAL = 2, MLSTM = 3 };

template <int D, int KIND> struct alignas(128) Stage {
    static constexpr bool HASW = KIND == DELTA_RULE || KIND == GENERAL;
    static constexpr int C2 = KIND == GENERAL ? 2 * CHUNK : CHUNK;      // rows that update the state
    static constexpr int PITCH = D + 4, PP = C2 + 4;
    // (eight lanes read a row's neighbouring pieces, so that rows without padding meet no bank twice)
    // (boxes land on 128-byte boundaries; without W its place is one such piece)
    float q[CHUNK * D], w[HASW ? CHUNK * D : 32], k[C2 * D], p[CHUNK * PP];
    float v[CHUNK * COLS], y[KIND == GENERAL ? CHUNK * COLS : 4];
    float gam[KIND == GENERAL ? D : CHUNK], e[CHUNK], fl[CHUNK];
};
// Partial updates of the state lie over the chunk's rows of Q (and W), which have been used by then: with the generalized rule's 120
// KB at D = 64 an SM held one block, so it holds two.
template <int D, int KIND> struct WalkSmem {
    static constexpr int PART = (WALK_THREADS / D - 1) * COLS * D;
    static constexpr bool PART_OVER_ROWS = PART <= CHUNK * D * (Stage<D, KIND>::HASW ? 2 : 1);
    Stage<D, KIND> st[2];
    float s[COLS * (D + 4)];                                     // the state's columns, along the keys
    float ut[COLS * Stage<D, KIND>::PP];                         // the update's values along the tokens,
    float un[Stage<D, KIND>::C2 * COLS];                         // and along the columns
    float part[PART_OVER_ROWS ? 4 : PART];
    float z[D], den[CHUNK];
    uint64_t bars[2];
    int abort;
};

// Partial sums of 4 tokens x 4 columns, spread over eight neighbouring lanes (kg), added up: lane kg gets column
// 2 (kg & 1) + (kg >> 1 & 1) of tokens 2 (kg >> 2) and 2 (kg >> 2) + 1.
__device__ __forceinline__ void over_lanes(const float (&x)[4][4], int kg, float (&y)[2])
{
    const bool b0 = kg & 1, b1 = kg & 2, b2 = kg & 4;
    float m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float m0 = (b0 ? x[i][2] : x[i][0]) + __shfl_xor_sync(0xffffffffu, b0 ? x[i][0] : x[i][2], 1);
        const float m1 = (b0 ? x[i][3] : x[i][1]) + __shfl_xor_sync(0xffffffffu, b0 ? x[i][1] : x[i][3], 1);
        m[i] = (b1 ? m1 : m0) + __shfl_xor_sync(0xffffffffu, b1 ? m0 : m1, 2);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) y[i] = (b2 ? m[2 + i] : m[i]) + __shfl_xor_sync(0xffffffffu, b2 ? m[i] : m[2 + i], 4);
}

// One block an SM where one prompt's heads are walked, so that what counts is a warp's chain of instructions and how many
// warps share a scheduler: two, on tiles large enough that neither the loads from shared memory (a 16-byte load of a warp
// takes four cycles of an SM) nor the moves around them outnumber the products.  Eight lanes share out the inner index of
// a tile of 4 tokens (of W and of Q) x 4 columns and add their sums by exchanges; the update's rows are shared out over
// parts of the block.  (Heads of 128 x 128, a chunk: 2 x 2 tiles with the whole inner index a thread, 4 warps: 4.1 us;
// 4 x 4 tiles, 4 warps: 3.7 us, 2,500 instructions a warp at three cycles each.)
template <int D, int KIND>
__global__ void __launch_bounds__(WALK_THREADS) walk_kernel(WalkArgs a, const __grid_constant__ WalkMaps maps)
{
    using St = Stage<D, KIND>;
    constexpr bool HASW = St::HASW;
    constexpr int C2 = St::C2, PITCH = St::PITCH, PP = St::PP;
    constexpr int DG = D / 4;                                    // a thread holds four keys of four columns of the state
    constexpr int PARTS = WALK_THREADS / D;                      // parts of the block, each with its share of the update's rows
    extern __shared__ __align__(128) unsigned char raw[];
    WalkSmem<D, KIND>& sm = *reinterpret_cast<WalkSmem<D, KIND>*>(raw);
    const int tid = threadIdx.x, h = blockIdx.y, col0 = blockIdx.x * COLS;
    fx_pdl_wait_only();
    int b = blockIdx.z, r0, r1, tile0 = 0;           // (tile0: the entry's first chunk)
    if (a.walks) {
        const int4 w = reinterpret_cast<const int4*>(a.walks)[blockIdx.z];
        b = w.x; r0 = w.y; r1 = w.z; tile0 = w.w;
    } else {
        r0 = first_row_of(a.token_seq, a.n_tokens, b);
        r1 = first_row_of(a.token_seq, a.n_tokens, b + 1);
    }
    if (r1 <= r0) return;
    const int nc = min(COLS, a.V - col0);
    const long slot = a.seq_slot[b];
    float* state = a.state + ((slot * a.H + h) * a.V + col0) * a.D;

    const long HD = (long)a.H * a.D, HV = (long)a.H * a.V;
    if (KIND == GENERAL && !a.walks) {
        int hi = a.n_tiles;
        while (tile0 < hi) {
            const int mid = (tile0 + hi) >> 1;
            if (a.tiles[mid * 4 + 2] < b) tile0 = mid + 1; else hi = mid;
        }
    }
    const uint32_t bar0 = fxtc::smem_u32(sm.bars);
    const bool tma = a.tma && fxtc::smem_u32(raw) % 128 == 0;
    if (tid == 0) {
        fxtc::mbar_init(bar0, 1);
        fxtc::mbar_init(bar0 + 8, 1);
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto fetch = [&](int c0, St& st, uint32_t bar) {
        const int rows = min(CHUNK, r1 - c0);
        if (tma && rows == CHUNK) {
            if (tid == 0) {
                constexpr uint32_t BOX = CHUNK * D * 4;
                const int kvh = h / a.q_share;
                fxtc::mbar_expect_tx(bar, BOX * (2 + (HASW ? 1 : 0) + (KIND == GENERAL ? 1 : 0)));
                fxtc::tma_load_3d(fxtc::smem_u32(st.q), &maps.q, 0, kvh, c0, bar);
                if (HASW) fxtc::tma_load_3d(fxtc::smem_u32(st.w), &maps.w, 0, h, c0, bar);
                fxtc::tma_load_3d(fxtc::smem_u32(st.k), &maps.k, 0, kvh, c0, bar);
                if (KIND == GENERAL) fxtc::tma_load_3d(fxtc::smem_u32(st.k + CHUNK * D), &maps.a, 0, h, c0, bar);
            }
        } else {
            if (HASW) load_rows<D, WALK_THREADS>(st.w, D, a.w + (long)c0 * HD + (long)h * a.D, HD, rows, a.D);
            load_rows<D, WALK_THREADS>(st.q, D, a.q + (long)c0 * a.ldq + (long)(h / a.q_share) * a.D, a.ldq, rows, a.D);
            load_rows<D, WALK_THREADS>(st.k, D, a.k + (long)c0 * a.ldk + (long)(h / a.q_share) * a.D, a.ldk, rows, a.D);
            if (KIND == GENERAL) load_rows<D, WALK_THREADS>(st.k + CHUNK * D, D, a.a + (long)c0 * HD + (long)h * a.D, HD, rows, a.D);
        }
        for (int i = tid; i < CHUNK * (C2 / 4); i += WALK_THREADS) {
            const int t = i / (C2 / 4), s = (i - t * (C2 / 4)) * 4;
            cp16(st.p + t * PP + s, a.p + (t < rows ? ((long)(c0 + t) * a.H + h) * C2 + s : 0), t < rows);
        }
        if (tid < 4 * CHUNK) {
            const int t = tid >> 2, c = (tid & 3) * 4;
            const bool ok = t < rows && c < nc;
            const long at = (long)(c0 + t) * HV + (long)h * a.V + col0 + c;
            if (KIND == DELTA_RULE) cp16(st.v + t * COLS + c, a.x0 + (ok ? at : 0), ok);
            else cp16(st.v + t * COLS + c, a.v + (ok ? (long)(c0 + t) * a.ldv + (long)h * a.V + col0 + c : 0), ok);
            if (KIND == GENERAL) cp16(st.y + t * COLS + c, a.x0 + (ok ? at : 0), ok);
        }
        if (KIND == GENERAL) {
            if (tid < DG) cp16(st.gam + tid * 4, a.gam + (tid * 4 < a.D ? ((long)(tile0 + (c0 - r0) / CHUNK) * a.H + h) * a.D + tid * 4 : 0), tid * 4 < a.D);
        } else if (tid < CHUNK) {
            const long at = tid < rows ? (long)(c0 + tid) * a.H + h : 0;
            cp4(st.gam + tid, a.gam + at, tid < rows);
            cp4(st.e + tid, a.e + at, tid < rows);
            if (KIND == MLSTM) cp4(st.fl + tid, a.floor_m + at, tid < rows);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // the state: thread (dg, cg) of part 0 holds keys 4 dg .. of columns 4 cg ..; the other parts hold updates only
    const int dg = tid % DG, cg = (tid / DG) & 3, part = tid / (DG * 4);
    u64 S[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = cg * 4 + j;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (part == 0 && c < nc && dg * 4 < a.D) x = *reinterpret_cast<const float4*>(state + (long)c * a.D + dg * 4);
        S[j][0] = pair(x.x, x.y); S[j][1] = pair(x.z, x.w);
        if (part == 0) *reinterpret_cast<float4*>(sm.s + c * PITCH + dg * 4) = x;
    }
    float z = 0.f;                                               // mLSTM: the normaliser's element tid
    if (KIND == MLSTM && tid < D) {
        z = tid < a.D ? a.norm_in[((long)b * a.H + h) * a.D + tid] : 0.f;
        sm.z[tid] = z;
    }
    __syncthreads();
    fetch(r0, sm.st[0], bar0);
    // products: tokens t0 .. t0 + 3 and columns w4 .. w4 + 3, of which this lane ends up with tokens tl, tl + 1 of column c
    const int kg = tid & 7, t0 = (tid >> 7) * 16 + ((tid >> 3) & 3) * 4, w4 = ((tid >> 5) & 3) * 4;
    const int tl = t0 + 2 * (kg >> 2), c = w4 + 2 * (kg & 1) + ((kg >> 1) & 1);
    int buf = 0;
    for (int c0 = r0, chunk = 0; c0 < r1; c0 += CHUNK, ++chunk, buf ^= 1) {
        const int rows = min(CHUNK, r1 - c0);
        St& st = sm.st[buf];
        if (tma && rows == CHUNK) fxtc::mbar_wait(bar0 + 8 * buf, (chunk >> 1) & 1, &sm.abort);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();             // this chunk's rows are there, the state is up to date, the other place is free
        if (*(volatile int*)&sm.abort) {        // (the boxes waited for are the only ones in flight: once more for them)
            if (tid == 0) {
                int again = 0;
                fxtc::mbar_wait(bar0 + 8 * buf, (chunk >> 1) & 1, &again);
                if (a.status) atomicExch(a.status, fxtc::STATUS_TC_TIMEOUT);
            }
            return;
        }
        if (c0 + CHUNK < r1) fetch(c0 + CHUNK, sm.st[buf ^ 1], bar0 + 8 * (buf ^ 1));

        // W S_0 and Q S_0
        float xq[4][4], xw[4][4];
        {
            u64 pq[4][4], pw[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { pq[i][j] = 0ull; pw[i][j] = 0ull; }
#pragma unroll 2
            for (int d = kg * 4; d < D; d += 32) {
                ulonglong2 s[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const ulonglong2*>(sm.s + (w4 + j) * PITCH + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(st.q + (t0 + i) * D + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) { fma2(pq[i][j], q.x, s[j].x); }
#pragma unroll
                    for (int j = 0; j < 4; ++j) { fma2(pq[i][j], q.y, s[j].y); }
                    if (HASW) {
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(st.w + (t0 + i) * D + d);
#pragma unroll
                        for (int j = 0; j < 4; ++j) { fma2(pw[i][j], w.x, s[j].x); }
#pragma unroll
                        for (int j = 0; j < 4; ++j) { fma2(pw[i][j], w.y, s[j].y); }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { xq[i][j] = sum_of(pq[i][j]); xw[i][j] = HASW ? sum_of(pw[i][j]) : 0.f; }
        }
        {
            float x[2], u[2], y[2];
            if (HASW) over_lanes(xw, kg, x);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = tl + i;
                u[i] = st.v[t * COLS + c];
                if (KIND == DELTA_RULE) u[i] -= x[i];
                const float ue = KIND == GENERAL ? u[i] : u[i] * st.e[t];
                sm.un[t * COLS + c] = ue;
                if (KIND == GENERAL) {
                    y[i] = st.y[t * COLS + c] + x[i];
                    sm.un[(CHUNK + t) * COLS + c] = y[i];
                }
            }
            *reinterpret_cast<float2*>(sm.ut + c * PP + tl) = make_float2(u[0], u[1]);
            if (KIND == GENERAL) *reinterpret_cast<float2*>(sm.ut + c * PP + CHUNK + tl) = make_float2(y[0], y[1]);
        }
        if (KIND == MLSTM) {
            // n_t . q_t: eight threads a token
            const int t = tid >> 3;
            float acc = 0.f;
            for (int d = kg * 4; d < D; d += 32) {
                const float4 q = *reinterpret_cast<const float4*>(st.q + t * D + d);
                const float4 n = *reinterpret_cast<const float4*>(sm.z + d);
                acc = fmaf(q.x, n.x, acc); acc = fmaf(q.y, n.y, acc); acc = fmaf(q.z, n.z, acc); acc = fmaf(q.w, n.w, acc);
            }
            acc *= st.gam[t] * a.q_scale;
            const float4 p = *reinterpret_cast<const float4*>(st.p + t * PP + kg * 4);
            acc += (p.x + p.y) + (p.z + p.w);
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (kg == 0) sm.den[t] = fmaxf(fabsf(acc), st.fl[t]) + 1e-6f;
        }
        __syncthreads();             // the update's values are there, everyone has read the state

        // the read-outs: the chunk's own tokens up to each one, on top of Q S_0 (the later tokens' values are left out, not
        // multiplied by zero: what is no number must not reach the tokens before it)
        {
            u64 o[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) o[i][j] = 0ull;
#pragma unroll
            for (int n = 0; n < C2 / 32; ++n) {
                const int s = n * 32 + kg * 4, sb = s & (CHUNK - 1);
                if (sb > t0) continue;
                const bool full = sb < t0;                       // else s .. s + 3 are the tile's own four tokens
                u64 ux[4], uy[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(sm.ut + (w4 + j) * PP + s);
                    ux[j] = u.x; uy[j] = u.y;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(st.p + (t0 + i) * PP + s);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        fma2(o[i][j], p.x, full || i > 0 ? ux[j] : ux[j] & 0xffffffffull);
                        fma2(o[i][j], p.y, full || i > 2 ? uy[j] : i > 1 ? uy[j] & 0xffffffffull : 0ull);
                    }
                }
            }
            float y[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float g = KIND == GENERAL ? 1.f : KIND == DELTA_RULE ? st.gam[t0 + i] : st.gam[t0 + i] * a.q_scale;
#pragma unroll
                for (int j = 0; j < 4; ++j) xq[i][j] = fmaf(g, xq[i][j], sum_of(o[i][j]));
            }
            over_lanes(xq, kg, y);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = tl + i;
                if (t >= rows || c >= nc) continue;
                if (KIND == MLSTM) y[i] /= sm.den[t];
                a.out[(long)(c0 + t) * a.ldo + (long)h * a.V + col0 + c] = y[i];
            }
        }

        // the state: the chunk's own sum first, then once the state before it, times the chunk's decay, on top (added to the
        // state one by one the tokens' shares would each be rounded at its size)
        u64 decay[2];
        if (KIND == GENERAL) {
            const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(st.gam + dg * 4);
            decay[0] = g.x; decay[1] = g.y;
        } else {
            const float g = st.gam[rows - 1];
            decay[0] = decay[1] = pair(g, g);
            if (KIND == MLSTM && tid < D) {
                float acc = 0.f;
#pragma unroll 8
                for (int s = 0; s < CHUNK; ++s) acc = fmaf(st.e[s], st.k[s * D + tid], acc);
                z = fmaf(g, z, acc);
            }
        }
        u64 U[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) U[j][0] = U[j][1] = 0ull;
#pragma unroll 8
        for (int i = 0; i < C2 / PARTS; ++i) {
            const int s = part * (C2 / PARTS) + i;
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(st.k + s * D + dg * 4);
            const float4 u4 = *reinterpret_cast<const float4*>(sm.un + s * COLS + cg * 4);
            const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { const u64 uu = pair(u[j], u[j]); fma2(U[j][0], k.x, uu); fma2(U[j][1], k.y, uu); }
        }
        float* const parts = WalkSmem<D, KIND>::PART_OVER_ROWS ? st.q : sm.part;       // (everyone is behind the barrier after the products with Q and W)
        if (part > 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<ulonglong2*>(parts + ((part - 1) * COLS + cg * 4 + j) * D + dg * 4) = make_ulonglong2(U[j][0], U[j][1]);
        }
        __syncthreads();
        if (part == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int i = 0; i < PARTS - 1; ++i) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(parts + (i * COLS + cg * 4 + j) * D + dg * 4);
                    U[j][0] = add2(U[j][0], x.x);
                    U[j][1] = add2(U[j][1], x.y);
                }
                S[j][0] = fma2_of(S[j][0], decay[0], U[j][0]);
                S[j][1] = fma2_of(S[j][1], decay[1], U[j][1]);
                *reinterpret_cast<ulonglong2*>(sm.s + (cg * 4 + j) * PITCH + dg * 4) = make_ulonglong2(S[j][0], S[j][1]);
            }
        }
        if (KIND == MLSTM && tid < D) sm.z[tid] = z;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // (boxes will be written where partial updates were)
    }
    fx_pdl_trigger();
    if (part == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int cc = cg * 4 + j;
            if (cc < nc && dg * 4 < a.D)
                *reinterpret_cast<float4*>(state + (long)cc * a.D + dg * 4) =
                    make_float4(lo_of(S[j][0]), hi_of(S[j][0]), lo_of(S[j][1]), hi_of(S[j][1]));
        }
    }
    if (KIND == MLSTM && blockIdx.x == 0 && tid < a.D)
        for (int i = 0; i < a.copies; ++i) a.norm[((slot * a.H + h) * a.copies + i) * a.D + tid] = z;
}

// A map of rows [tokens][heads][d], `ld` floats apart, a box a chunk's rows of a head.
bool row_map(CUtensorMap* m, const float* p, long ld, int heads, int d, int tokens)
{
    const fxtc::EncodeTiledFn fn = fxtc::encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)tokens};
    cuuint64_t strides[2] = {(cuuint64_t)d * 4, (cuuint64_t)ld * 4};
    cuuint32_t box[3] = {(cuuint32_t)d, 1, CHUNK}, steps[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static_assert(2 * (sizeof(WalkSmem<64, GENERAL>) + 1024) <= 233472, "two blocks an SM");

template <int D, int KIND> constexpr bool on_boundaries() {
    using S = Stage<D, KIND>;
    return offsetof(S, q) % 128 == 0 && offsetof(S, w) % 128 == 0 && offsetof(S, k) % 128 == 0 && sizeof(S) % 128 == 0;
}

template <int D, int KIND> int go_walk(WalkArgs a, int n_entries, cudaStream_t s)
{
    // Boxes need heads as wide as the tile (a narrower head's rows would lie closer together than the kernel reads them) and
    // as many tokens as a box has rows.  Where a map cannot be made the rows go by cp.async.
    static_assert(on_boundaries<D, KIND>(), "where boxes land");
    WalkMaps maps = {};
    a.tma = a.D == D && a.n_tokens >= CHUNK && row_map(&maps.q, a.q, a.ldq, a.H / a.q_share, D, a.n_tokens) &&
            row_map(&maps.k, a.k, a.ldk, a.H / a.q_share, D, a.n_tokens) &&
            (!Stage<D, KIND>::HASW || row_map(&maps.w, a.w, (long)a.H * D, a.H, D, a.n_tokens)) &&
            (KIND != GENERAL || row_map(&maps.a, a.a, (long)a.H * D, a.H, D, a.n_tokens));
    const int smem = (int)sizeof(WalkSmem<D, KIND>);
    // (of the current device: asked for each time)
    const cudaError_t set = cudaFuncSetAttribute(walk_kernel<D, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (set != cudaSuccess) return (int)set;
    // (not set up early: its blocks stay for the whole prompt, see fx_launch_pdl_if)
    fx_launch_pdl_if(false, walk_kernel<D, KIND>, dim3((unsigned)fx_cdiv(a.V, COLS), (unsigned)a.H, (unsigned)n_entries), WALK_THREADS,
                     (size_t)smem, s, a, maps);
    return fx_launch_status();
}

template <typename K> int go_chunks(K kernel, const ChunkArgs& a, int n_tiles, size_t smem, cudaStream_t s)
{
    const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (set != cudaSuccess) return (int)set;
    fx_launch_pdl(kernel, dim3((unsigned)n_tiles, (unsigned)a.H), PREP_THREADS, smem, s, a);
    return fx_launch_status();
}

int check(int H, int G, int D, int V, int n_entries)
{
    if (H <= 0 || H > 65535 || G <= 0 || H % G || D <= 0 || D > 128 || V <= 0 || n_entries > 65535) return FX_ERR_SIZE;
    if (D % 4 || V % 4) return FX_ERR_SIZE;
    return FX_OK;
}
bool off_grid(const void* p, long ld) { return (uintptr_t)p % 16 || ld % 4; }

}  // namespace

// The delta rule (beta [T, H]) or, with take [T, H] (a factor on k v^T), norm_in, norm and floor_m, an mLSTM's recurrence.
// q, k [T, G * D], v [T, H * V] 32-bit rows; g [T, H] the decays.  Scratch: p [T, H, CHUNK], gam and e [T, H]; delta rule: wr
// [T, H, D].  norm_in: the normaliser before the step [entries, H, D], norm its copies in the state [slots, H, copies, D],
// floor_m exp(-m_t) [T, H], as fx_mlstm_gates leaves them.  out contiguous [T, H * V] (the delta rule's U0 until a chunk's
// read-outs take its place: a block reads a chunk's share of it before it writes it).
extern "C" int fx_chunk_scan(const float* q, long ldq, const float* k, long ldk, const float* v, long ldv, const float* g,
                             const float* beta, const float* take, float q_scale, float* p, float* gam, float* e, float* wr,
                             const float* norm_in, float* norm, int copies, const float* floor_m, float* state, float* out,
                             const int* tiles, int n_tiles, const int* walks, const int* token_seq, const int* seq_slot, int n_tokens,
                             int n_entries, int H, int G, int D, int V, int* status, void* stream)
{
    if (n_tokens <= 0 || n_entries <= 0 || n_tiles <= 0) return FX_OK;
    int st = check(H, G, D, V, n_entries);
    if (st != FX_OK) return st;
    if (beta ? !wr || take || norm : !take || !norm || !norm_in || !floor_m || copies < 1) return FX_ERR_SIZE;
    if (off_grid(q, ldq) || off_grid(k, ldk) || off_grid(v, ldv) || off_grid(p, 0) || off_grid(state, 0) || off_grid(out, 0) ||
        off_grid(wr, 0) || off_grid(tiles, 0) || off_grid(walks, 0))
        return FX_ERR_ALIGN;
    cudaStream_t s = (cudaStream_t)stream;
    ChunkArgs c = {};
    c.tiles = tiles; c.q = q; c.k = k; c.v = v; c.ldq = ldq; c.ldk = ldk; c.ldv = ldv; c.g = g;
    c.gate = beta ? beta : take; c.scale = q_scale; c.H = H; c.G = G; c.D = D; c.V = V; c.p = p; c.gam = gam; c.e = e; c.x0 = out; c.wr = wr;
    const size_t small = sizeof(float) * (2 * CHUNK * (64 + 4) + CHUNK * (CHUNK + 4)), large = small + sizeof(float) * 2 * CHUNK * 64;
    if (beta) st = D <= 64 ? go_chunks(scalar_chunks<64, true>, c, n_tiles, small, s) : go_chunks(scalar_chunks<128, true>, c, n_tiles, large, s);
    else st = D <= 64 ? go_chunks(scalar_chunks<64, false>, c, n_tiles, small, s) : go_chunks(scalar_chunks<128, false>, c, n_tiles, large, s);
    if (st != FX_OK) return st;
    WalkArgs a = {};
    a.w = wr; a.q = q; a.ldq = ldq; a.q_share = H / G; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv; a.x0 = out; a.p = p; a.gam = gam; a.e = e;
    a.floor_m = floor_m; a.norm_in = norm_in; a.norm = norm; a.copies = copies; a.q_scale = q_scale; a.state = state; a.out = out;
    a.ldo = (long)H * V; a.token_seq = token_seq; a.seq_slot = seq_slot; a.n_tokens = n_tokens; a.H = H; a.D = D; a.V = V; a.walks = walks; a.status = status;
    if (beta) return D <= 64 ? go_walk<64, DELTA_RULE>(a, n_entries, s) : go_walk<128, DELTA_RULE>(a, n_entries, s);
    return D <= 64 ? go_walk<64, MLSTM>(a, n_entries, s) : go_walk<128, MLSTM>(a, n_entries, s);
}

// The generalized delta rule from its projections: r, k, v, a_pre rows [T, H * D], low rows [T, rank], w2 [H * D, rank], w0 and
// a_bias [H * D], all rows 32-bit.  Scratch: p [T, H, 2 CHUNK], gam [tiles, H, D], wr, qs, ks and as [T, H, D].  out contiguous
// [T, H * D]: it holds Y0 until a chunk's read-outs take its place.
extern "C" int fx_chunk_scan_general(const float* r, long ldr, const float* k, long ldk, const float* v, long ldv, const float* a_pre,
                                     long lda, const float* low, long ldl, const void* w2, int w2_dtype, const void* w0, int w0_dtype,
                                     const void* a_bias, int ab_dtype, float rate, int rank, float* p, float* gam, float* wr, float* qs,
                                     float* ks, float* as, float* state, float* out, const int* tiles, int n_tiles, const int* walks,
                                     const int* token_seq, const int* seq_slot, int n_tokens, int n_entries, int H, int D, int* status,
                                     void* stream)
{
    if (n_tokens <= 0 || n_entries <= 0 || n_tiles <= 0) return FX_OK;
    int st = check(H, H, D, D, n_entries);
    if (st != FX_OK) return st;
    if (rank <= 0 || !(rate >= 0.f && rate <= 1.f)) return FX_ERR_SIZE;      // (see the header)
    if (off_grid(r, ldr) || off_grid(k, ldk) || off_grid(v, ldv) || off_grid(a_pre, lda) || off_grid(p, 0) || off_grid(gam, 0) ||
        off_grid(wr, 0) || off_grid(qs, 0) || off_grid(ks, 0) || off_grid(as, 0) || off_grid(out, 0) || off_grid(state, 0) ||
        off_grid(tiles, 0) || off_grid(walks, 0))
        return FX_ERR_ALIGN;
    cudaStream_t s = (cudaStream_t)stream;
    ChunkArgs c = {};
    c.tiles = tiles; c.q = r; c.k = k; c.v = v; c.ldq = ldr; c.ldk = ldk; c.ldv = ldv; c.a_pre = a_pre; c.lda = lda; c.low = low; c.ldl = ldl;
    c.rank = rank; c.w2 = w2; c.w0 = w0; c.ab = a_bias; c.w2_dtype = w2_dtype; c.w0_dtype = w0_dtype; c.ab_dtype = ab_dtype; c.rate = rate;
    c.H = H; c.G = H; c.D = D; c.V = D; c.p = p; c.gam = gam; c.x0 = out; c.wr = wr; c.qs = qs; c.ks = ks; c.as = as;
    auto smem = [](int d) { return sizeof(float) * (5 * CHUNK * (d + 4) + 2 * CHUNK * (CHUNK + 4) + (d + CHUNK) * (RANK + 4)); };
    st = D <= 64 ? go_chunks(general_chunks<64>, c, n_tiles, smem(64), s) : go_chunks(general_chunks<128>, c, n_tiles, smem(128), s);
    if (st != FX_OK) return st;
    WalkArgs a = {};
    a.w = wr; a.q = qs; a.ldq = (long)H * D; a.q_share = 1; a.k = ks; a.ldk = (long)H * D; a.a = as; a.v = v; a.ldv = ldv; a.x0 = out;
    a.p = p; a.gam = gam; a.q_scale = 1.f; a.state = state; a.out = out; a.ldo = (long)H * D; a.token_seq = token_seq; a.seq_slot = seq_slot;
    a.n_tokens = n_tokens; a.H = H; a.D = D; a.V = D; a.tiles = tiles; a.n_tiles = n_tiles; a.walks = walks; a.status = status;
    return D <= 64 ? go_walk<64, GENERAL>(a, n_entries, s) : go_walk<128, GENERAL>(a, n_entries, s);
}

// The gates of an mLSTM for fx_chunk_scan: keep, take and floor_m [T, H] from the projected [i | f] rows; moves the running
// maximum's copies [slots, H, copies] on; norm_in [entries, H, D] gets the normaliser as it is.
extern "C" int fx_mlstm_gates(const float* gates, long ldg, const void* i_bias, const void* f_bias, int bias_dtype, float cap, float* m,
                              int copies, const float* norm, float* norm_in, int D, float* keep, float* take, float* floor_m, const int* token_seq, const int* seq_slot,
                              int n_tokens, int n_entries, int H, void* stream)
{
    if (n_tokens <= 0 || n_entries <= 0) return FX_OK;
    if (H <= 0 || H > 65535 || copies < 1 || !(cap > 0.f)) return FX_ERR_SIZE;
    fx_launch_pdl(mlstm_gates_kernel, dim3((unsigned)n_entries, (unsigned)H), 32, 0, (cudaStream_t)stream, gates, ldg, i_bias, f_bias,
                  bias_dtype, cap, m, copies, norm, norm_in, D, keep, take, floor_m, token_seq, seq_slot, n_tokens, H);
    return fx_launch_status();
}
