// Prompt attention over cache pages in 32 bits on the tensor cores: the operation of attention_f32.cu, scores and sums of
// 32-bit operands made of three bfloat16 parts each (split3.cuh), six products of parts for one of 32 bits.
//
// Two kernels.  split_kernel lays the step's queries and the keys and values that its requests see down in their parts, so that TMA
// can fetch them: planes [3][tokens][heads][dim] and [3][rows][kv heads][dim], a request's positions in rows that follow each
// other from a multiple of 64 on (`spans`), zeros where a position has no page.
// attention_kernel: a CTA 128 queries of a request and one head, against blocks of 64 keys.
//
//   S = Q K^T     tcgen05.mma 128 x 64 x dim, six for each 16 elements, the small products first, in two sums of half the elements
//                 each (the tensor core cuts where an FFMA rounds, once for each 16 elements: with parts that were cut off the result
//                 at 128 keys was 2.24e-7 off in one sum, 1.83e-7 in two; with rounded ones it is 1.47e-7, with FFMA 2.00e-7); two S in
//                 tensor memory, so that the next block's is made while this one's softmax runs
//   P = exp(..)   two threads a query: maximum and sum in 32 bits, P in its three parts into tensor memory
//   O_j = P V     tcgen05.mma 128 x dim x 64 into an accumulator of the block's own (over all keys' blocks the cuts would add
//                 up), which the query's threads add to their 32-bit registers, rescaled by the running maximum, when the next
//                 block's weights are made
//
// What cannot be had from the parts is done again from the operands as they are: a score that is no finite number, and the elements of
// a block's result that are none while the weights' sum is one (a value that is infinite or no number where the weight is 0: a key that
// the query does not see, whose value must stay out).
//
// Bound by the chain of a key block, 4 us of it: the softmax's two threads a query (a thread a query: 12 us, its registers spilled)
// and the products that wait for it, 48 of 64 columns and 24 of `dim`, 1.2 us; tiles of 128 queries of 16 heads leave SMs idle below
// 1,200 tokens.  16 heads of 128, from position 0, both kernels here against FFMA with its tiles of 32 queries: 64 tokens 12 against
// 18 us, 200: 23 against 48, 517: 42 against 145, 2000: 135 against 1299.
#include "tc_common.cuh"
#include "split3.cuh"
#include "api.h"

namespace {

using namespace fxtc;

constexpr int BQ = 128, BK = 64, NTHREADS = 320, WORKERS = 8;

// ------------------------------------------------------------------------------------------------------ parts
struct SplitArgs {
    const float* q; long ldq; int n_tokens, n_heads;
    const float *k_pages, *v_pages;
    const int* table; int table_width, page_size, n_kv_heads, dim;
    const int* spans; int n_spans;       // [n][4]: entry, first position, one past the last, first row; rows up to a multiple of 64
    const int* seq_slot;
    bf16 *qp, *kp, *vp; long rows;
};

// blockIdx.y: 0 queries, 1 keys, 2 values; 8 elements a thread.
__global__ void __launch_bounds__(256) split_kernel(SplitArgs a)
{
    fx_pdl_wait();
    const int what = blockIdx.y, heads = what ? a.n_kv_heads : a.n_heads, per = heads * a.dim / 8;
    const long rows = what ? a.rows : a.n_tokens, i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i >= rows * per) return;
    const long r = i / per;
    const int e = (int)(i - r * per) * 8;
    const float* src = nullptr;
    if (!what) {
        src = a.q + r * a.ldq + e;
    } else {
        int lo = 0, hi = a.n_spans;      // the last span that begins at or before row r
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (a.spans[mid * 4 + 3] <= r) lo = mid; else hi = mid;
        }
        const int4 s = reinterpret_cast<const int4*>(a.spans)[lo];
        const long pos = s.y + (r - s.w);
        if (pos < s.z) {
            const int page = a.table[(long)a.seq_slot[s.x] * a.table_width + pos / a.page_size];
            const int h = e / a.dim;
            if (page >= 0)
                src = (what == 1 ? a.k_pages : a.v_pages) + (((long)page * a.n_kv_heads + h) * a.page_size + pos % a.page_size) * a.dim + (e - h * a.dim);
        }
    }
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (src) { Pack<float>::load(src, v); Pack<float>::load(src + 4, v + 4); }
    uint4 p[3];
    split3_8(v, p[0], p[1], p[2]);
    bf16* to = (what == 0 ? a.qp : what == 1 ? a.kp : a.vp) + r * heads * a.dim + e;
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(to + j * rows * heads * a.dim) = p[j];
}

// ------------------------------------------------------------------------------------------------------ attention
struct Args {
    const float* q; long ldq; const float *k_pages, *v_pages;       // (as they are)
    const int* table; int table_width, page_size;
    const int* items;                    // [n][8]: first token, rows, entry, position of the first, first key block, end, row of position 0, -
    const int* seq_slot;
    float* out; long ldo;
    int n_heads, n_kv_heads, dim, window;
    float scale, softcap;
    int* status;
};

template <int D> struct Smem {           // D: the head's width rounded up to 64 or 128, zeros beyond it
    static constexpr int HALVES = D / 64;
    static constexpr int Q_PIECE = BQ * 128, K_PIECE = BK * 128;     // [rows][64 elements]
    static constexpr int Q_BYTES = 3 * HALVES * Q_PIECE, K_BYTES = 3 * HALVES * K_PIECE;
    static constexpr int K_OFF = Q_BYTES, V_OFF = K_OFF + K_BYTES, BAR_OFF = V_OFF + K_BYTES;
    static constexpr int TOTAL = BAR_OFF + 128 + 1024;
    // columns of tensor memory: two S of two sums each, the parts of P, the block's result
    static constexpr int S = 0, P = 4 * BK, O = P + 3 * BK / 2, COLS = 512;
    static_assert(O + D <= COLS, "tensor memory");
};

__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ float plain_dot(const float* x, const float* y, int n) {
    float s = 0.f;
#pragma unroll 1
    for (int i = 0; i < n && s == s; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + i), b = *reinterpret_cast<const float4*>(y + i);
        s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
    }
    return s;
}

template <int D>
__global__ void __launch_bounds__(NTHREADS, 1) attention_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                const __grid_constant__ CUtensorMap map_k,
                                                                const __grid_constant__ CUtensorMap map_v, Args a)
{
    using L = Smem<D>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int abort_flag_s;
    __shared__ uint32_t tmem_base_s;
    __shared__ float other_s[2][2][BQ];          // what a query's two threads tell each other
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int* item = a.items + (long)blockIdx.y * 8;
    const int tok0 = item[0], rows = item[1], entry = item[2], pos0 = item[3], blk0 = item[4], n_blk = item[5] - item[4], row0 = item[6];
    const int head = blockIdx.x, kvh = head / (a.n_heads / a.n_kv_heads);

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = base + L::BAR_OFF;
    const uint32_t q_full = bars, k_full = bars + 8, k_empty = bars + 16, v_full = bars + 24, v_empty = bars + 32, p_full = bars + 40,
                   o_full = bars + 48;
    auto s_full = [&](int b) { return bars + 56 + 8u * b; };
    volatile int* abort_flag = &abort_flag_s;
    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        for (uint32_t b = q_full; b <= s_full(1); b += 8) mbar_init(b, b == p_full ? WORKERS : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)L::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    fx_pdl_wait();

    if (warp == 0) {
        // ---------------- fetches ----------------
        if (lane == 0) {
            mbar_expect_tx(q_full, L::Q_BYTES);
            for (int p = 0; p < 3; ++p)
                for (int h = 0; h < L::HALVES; ++h)
                    tma_load_4d(base + (p * L::HALVES + h) * L::Q_PIECE, &map_q, h * 64, head, tok0, p, q_full);
            int nk = 0, nv = 0;
            for (int j = 0; j < n_blk; ++j) {
                const int row = row0 + (blk0 + j) * BK;
                if (!mbar_wait(k_empty, (uint32_t)(j & 1) ^ 1u, abort_flag)) break;
                mbar_expect_tx(k_full, L::K_BYTES);
                for (int p = 0; p < 3; ++p)
                    for (int h = 0; h < L::HALVES; ++h)
                        tma_load_4d(base + L::K_OFF + (p * L::HALVES + h) * L::K_PIECE, &map_k, h * 64, kvh, row, p, k_full);
                nk = j + 1;
                if (!mbar_wait(v_empty, (uint32_t)(j & 1) ^ 1u, abort_flag)) break;
                mbar_expect_tx(v_full, L::K_BYTES);
                for (int p = 0; p < 3; ++p)
                    for (int h = 0; h < L::HALVES; ++h)
                        tma_load_4d(base + L::V_OFF + (p * L::HALVES + h) * L::K_PIECE, &map_v, h * 64, kvh, row, p, v_full);
                nv = j + 1;
            }
            if (*abort_flag) {           // loads that were asked for must land before shared memory is released
                const uint32_t last[3][2] = {{q_full, 0u}, {k_full, (uint32_t)(nk - 1) & 1u}, {v_full, (uint32_t)(nv - 1) & 1u}};
                for (int i = 0; i < 3; ++i)
                    if (i == 0 || (i == 1 ? nk : nv) > 0)
                        for (uint32_t n = 0; n < WAIT_LIMIT; ++n)
                            if (mbar_try_wait(last[i][0], last[i][1])) break;
            }
        }
    } else if (warp == 1) {
        // ---------------- products ----------------
        if (lane == 0) {
            constexpr uint32_t idesc_s = instr_desc_ex(BQ, BK, 0), idesc_o = instr_desc_ex(BQ, D, 1);
            bool ok = mbar_wait(q_full, 0, abort_flag);
            auto scores = [&](int j) {
                if (!mbar_wait(k_full, (uint32_t)(j & 1), abort_flag)) return false;
                tc_fence_after();
                const uint32_t s = tmem + L::S + (j & 1) * 2 * BK;
                bool first = true;
                auto part = [&](int pq, int pk) {
#pragma unroll
                    for (int h = 0; h < L::HALVES; ++h) {
                        const uint64_t dq = smem_desc(base + (pq * L::HALVES + h) * L::Q_PIECE);
                        const uint64_t dk = smem_desc(base + L::K_OFF + (pk * L::HALVES + h) * L::K_PIECE);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int sum = (h * 4 + k) / (2 * L::HALVES);        // of the first or the second half of the elements
                            tc_mma(s + sum * BK, dq + 2u * k, dk + 2u * k, idesc_s, !first || (h * 4 + k) % (2 * L::HALVES) != 0);
                        }
                    }
                    first = false;
                };
                part(0, 2); part(2, 0); part(1, 1); part(0, 1); part(1, 0); part(0, 0);
                tc_commit(k_empty);
                tc_commit(s_full(j & 1));
                return true;
            };
            if (ok && n_blk > 0) ok = scores(0);
            for (int j = 0; j < n_blk && ok; ++j) {
                // (S of block j + 1 goes where block j - 1's was read before its P arrived)
                if (j + 1 < n_blk && !(ok = scores(j + 1))) break;
                ok = mbar_wait(p_full, (uint32_t)(j & 1), abort_flag) && mbar_wait(v_full, (uint32_t)(j & 1), abort_flag);
                if (!ok) break;
                tc_fence_after();
                bool first = true;
                auto part = [&](int pp, int pv) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint64_t dv = smem_desc_lbo_sbo(base + L::V_OFF + pv * L::HALVES * L::K_PIECE + k * 2048, L::K_PIECE, 1024);
                        tc_mma_ts(tmem + L::O, tmem + L::P + pp * (BK / 2) + 8u * k, dv, idesc_o, !first);
                        first = false;
                    }
                };
                part(0, 2); part(2, 0); part(1, 1); part(0, 1); part(1, 0); part(0, 0);
                tc_commit(v_empty);
                tc_commit(o_full);
            }
        }
    } else {
        // ---------------- softmax: two threads a query, half of a block's keys and half of the result's elements each ----------------
        constexpr int HK = BK / 2, HD = D / 2;
        const int quad = warp & 3, half = (warp - 2) >> 2, r = quad * 32 + lane, pos = pos0 + r, lo = fx_first_key(pos, a.window, 0);
        const int d0 = half * HD;
        const bool idle = quad * 32 >= rows;         // none of the warp's rows exists
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const int* table = a.table + (long)a.seq_slot[entry] * a.table_width;
        const float* qr = a.q + (long)(tok0 + min(r, rows - 1)) * a.ldq + (long)head * a.dim;
        const int last_lo = fx_first_key(pos0 + rows - 1, a.window, 0);
        // m, alpha: of the newest block; m_of, alpha_of: of the block whose result is added next; l: the sum of this thread's keys
        float o[HD], m = -INFINITY, l = 0.f, alpha = 0.f, m_of = 0.f, alpha_of = 0.f;
#pragma unroll
        for (int d = 0; d < HD; ++d) o[d] = 0.f;
        auto page_of = [&](int kb) { return table[kb / a.page_size]; };      // (a block of keys lies in one page)
        auto row_of = [&](const float* pages, int kb, int j) {
            return pages + (((long)page_of(kb) * a.n_kv_heads + kvh) * a.page_size + kb % a.page_size + j) * a.dim;
        };
        auto scaled = [&](float s) {
            float x = s * a.scale;
            if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
            return x;
        };
        constexpr uint32_t INF_BITS = 0x7f800000u;
        // block j's result: o <- o alpha + O_j
        auto add_up = [&](int j) {
            if (!__all_sync(0xffffffffu, mbar_wait(o_full, (uint32_t)(j & 1), abort_flag))) return false;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < HD; c += 32) {
                uint32_t b[32], most = 0;
                tc_ld32(lanes + L::O + d0 + c, b);
                tc_ld_wait_for(b);
#pragma unroll
                for (int d = 0; d < 32; ++d) most = max(most, b[d] & 0x7fffffffu);
                uint32_t odd = 0;
                if (most >= INF_BITS && r < rows) {
                    // elements that are no finite numbers, from the operands as they are
#pragma unroll
                    for (int d = 0; d < 32; ++d)
                        if ((b[d] & 0x7fffffffu) >= INF_BITS) { odd |= 1u << d; b[d] = 0; }
                }
#pragma unroll
                for (int d = 0; d < 32; ++d) o[c + d] = fmaf(o[c + d], alpha_of, __uint_as_float(b[d]));
                if (odd == 0) continue;
                const int kb = (blk0 + j) * BK;
                const bool edge = kb + BK - 1 > pos0 || kb < last_lo;
#pragma unroll 1
                for (int i = 0; i < BK; ++i) {
                    const int key = kb + i;
                    if (key > pos || key < lo || page_of(kb) < 0) continue;
                    const float p = expf(scaled(plain_dot(qr, row_of(a.k_pages, kb, i), a.dim)) - m_of);
                    if (edge && p == 0.f) continue;
                    const float* v = row_of(a.v_pages, kb, i) + d0 + c;
#pragma unroll
                    for (int d = 0; d < 32; ++d)
                        if ((odd >> d & 1) && d0 + c + d < a.dim) o[c + d] = fmaf(p, v[d], o[c + d]);
                }
            }
            return true;
        };
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < n_blk; ++j) {
            ok = __all_sync(0xffffffffu, mbar_wait(s_full(j & 1), (uint32_t)((j >> 1) & 1), abort_flag) && !*abort_flag);
            if (idle) {              // (waits for the results as well, or it would arrive for two blocks at once)
                if (j > 0) ok = ok && __all_sync(0xffffffffu, mbar_wait(o_full, (uint32_t)((j - 1) & 1), abort_flag));
                if (!ok) break;
                if (lane == 0) mbar_arrive(p_full);
                continue;
            }
            if (!ok) break;
            tc_fence_after();
            const int kb = (blk0 + j) * BK, k0 = kb + half * HK;
            const bool mapped = page_of(kb) >= 0;
            const bool inside = mapped && kb + BK - 1 <= pos0 && kb >= last_lo;      // every key visible to every row
            uint32_t x[HK], most = 0;
            {
                uint32_t y[HK];
                tc_ld32(lanes + L::S + (j & 1) * 2 * BK + half * HK, x);
                tc_ld32(lanes + L::S + (j & 1) * 2 * BK + BK + half * HK, y);
                tc_ld_wait_for(x);
                tc_ld_wait_for(y);
#pragma unroll
                for (int i = 0; i < HK; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) + __uint_as_float(y[i]));
            }
#pragma unroll
            for (int i = 0; i < HK; ++i) most = max(most, x[i] & 0x7fffffffu);
            if (most >= INF_BITS && mapped && r < rows) {
                uint32_t odd = 0;
#pragma unroll
                for (int i = 0; i < HK; ++i) odd |= (x[i] & 0x7fffffffu) < INF_BITS ? 0u : 1u << i;
#pragma unroll 1
                for (; odd; odd &= odd - 1) {
                    const int i = __ffs(odd) - 1;
                    if (k0 + i > pos || k0 + i < lo) continue;
                    const float s = plain_dot(qr, row_of(a.k_pages, kb, half * HK + i), a.dim);
#pragma unroll
                    for (int n = 0; n < HK; ++n)
                        if (n == i) x[n] = __float_as_uint(s);
                }
            }
            if (a.softcap > 0.f) {
#pragma unroll
                for (int i = 0; i < HK; ++i) x[i] = __float_as_uint(scaled(__uint_as_float(x[i])));
            } else {
#pragma unroll
                for (int i = 0; i < HK; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * a.scale);
            }
            if (!inside) {
#pragma unroll
                for (int i = 0; i < HK; ++i)
                    if (!mapped || k0 + i > pos || k0 + i < lo) x[i] = 0xff800000u;      // -inf
            }
            float top0 = -INFINITY, top1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < HK; i += 2) { top0 = fmaxf(top0, __uint_as_float(x[i])); top1 = fmaxf(top1, __uint_as_float(x[i + 1])); }
            other_s[j & 1][half][r] = fmaxf(top0, top1);
            asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");           // the two warps of these rows
            const float mn = fmaxf(m, fmaxf(fmaxf(top0, top1), other_s[j & 1][half ^ 1][r]));
            // (nothing seen yet: whatever the reference, every weight is 0)
            const float ref = mn == -INFINITY ? 0.f : mn;
            alpha = m == -INFINITY ? 0.f : expf(m - mn);
            m = mn;
            float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
            for (int i = 0; i < HK; i += 2) {
                const float p0 = expf(__uint_as_float(x[i]) - ref), p1 = expf(__uint_as_float(x[i + 1]) - ref);
                sum0 += p0; sum1 += p1;
                x[i] = __float_as_uint(p0); x[i + 1] = __float_as_uint(p1);
            }
            l = l * alpha + (sum0 + sum1);
            // The block before this one, whose product ran meanwhile: with its result there, its weights' place is free.
            if (j > 0 && !(ok = add_up(j - 1))) break;
            alpha_of = alpha; m_of = m;
#pragma unroll
            for (int c = 0; c < HK; c += 16) {
                uint32_t w[3][8];
#pragma unroll
                for (int i = 0; i < 16; i += 2)
                    split3(__uint_as_float(x[c + i]), __uint_as_float(x[c + i + 1]), w[0][i / 2], w[1][i / 2], w[2][i / 2]);
#pragma unroll
                for (int p = 0; p < 3; ++p) tc_st8(lanes + L::P + p * (BK / 2) + (half * HK + c) / 2, w[p]);
            }
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        if (ok && n_blk > 0 && !idle) ok = add_up(n_blk - 1);
        // (a warp that gave up lets its partner past the meeting that it can be at; behind that the partner sees that it gave up)
        if (!ok && !idle) asm volatile("bar.arrive %0, 64;" :: "r"(1 + quad) : "memory");
        if (ok && !idle && n_blk > 0) {
            other_s[n_blk & 1][half][r] = l;
            asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
            const float all = other_s[n_blk & 1][0][r] + other_s[n_blk & 1][1][r];
            const float inv = all > 0.f ? 1.0f / all : all == 0.f ? 0.f : all;      // (no number stays none)
            float* to = a.out + (long)(tok0 + r) * a.ldo + (long)head * a.dim + d0;
            if (r < rows) {
#pragma unroll
                for (int d = 0; d < HD; d += 4)
                    if (d0 + d < a.dim) *reinterpret_cast<float4*>(to + d) = make_float4(o[d] * inv, o[d + 1] * inv, o[d + 2] * inv, o[d + 3] * inv);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)L::COLS) : "memory");
    }
    if (threadIdx.x == 0 && abort_flag_s && a.status) atomicExch(a.status, STATUS_TC_TIMEOUT);
}

// planes [3][rows][heads][dim] of bfloat16, a box `box` rows of 64 elements of a head
bool plane_map(CUtensorMap* m, const bf16* p, int dim, int heads, long rows, uint32_t box)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[4] = {(cuuint64_t)dim, (cuuint64_t)heads, (cuuint64_t)rows, 3};
    cuuint64_t strides[3] = {(cuuint64_t)dim * 2, (cuuint64_t)heads * dim * 2, (cuuint64_t)rows * heads * dim * 2};
    cuuint32_t boxes[4] = {64, 1, box, 1}, steps[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(p), dims, strides, boxes, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D> int go(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const Args& a, int n_items, cudaStream_t s)
{
    // (of the current device: asked for each time)
    if (const cudaError_t e = cudaFuncSetAttribute(attention_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D>::TOTAL)) return (int)e;
    fx_launch_pdl(attention_kernel<D>, dim3((unsigned)a.n_heads, (unsigned)n_items), NTHREADS, Smem<D>::TOTAL, s, mq, mk, mv, a);
    return fx_launch_status();
}

}  // namespace

// q rows [n_tokens, ldq] beginning with the query heads; pages [page][kv head][position][dim], page_size a multiple of 64; head_dim a
// multiple of 8, 128 at most.  items: int32 [n_items, 8] = (first token, rows <= 128, entry, position of the first, first key block of 64
// positions, end of the key blocks, the plane row of the entry's position 0, -); spans: int32 [n_spans, 4] = (entry, first position, a
// multiple of 64, one past the last, first row, a multiple of 64), in the order of their rows, `rows` of them all (a multiple of 64).
// work, 16-byte aligned: 6 (n_tokens n_heads + 2 rows n_kv_heads) head_dim bytes.
extern "C" int fx_prefill_attention_f32_tc(const void* q, long ldq, int n_tokens, const void* k_pages, const void* v_pages,
                                           const int* block_table, int table_width, int page_size, const int* items, int n_items,
                                           const int* spans, int n_spans, long rows, const int* seq_slot, void* out, long ldo, int n_heads,
                                           int n_kv_heads, int head_dim, int window, float scale, float softcap, void* work, long work_bytes,
                                           int* status, void* stream)
{
    if (n_items <= 0 || n_tokens <= 0) return FX_OK;
    if (head_dim <= 0 || head_dim % 8 || head_dim > 128 || n_kv_heads <= 0 || n_heads % n_kv_heads || n_heads > 65535 || n_items > 65535 ||
        page_size <= 0 || page_size % 64 || rows <= 0 || rows % 64 || n_spans <= 0 || rows > 0x7fffffffL)
        return FX_ERR_SIZE;
    const long q_size = (long)n_tokens * n_heads * head_dim, kv_size = rows * n_kv_heads * head_dim;
    if (work_bytes < 6 * (q_size + 2 * kv_size)) return FX_ERR_SIZE;
    if (ldq % 4 || ldo % 4 || (uintptr_t)q % 16 || (uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16 || (uintptr_t)out % 16 ||
        (uintptr_t)work % 16 || (uintptr_t)spans % 16)
        return FX_ERR_ALIGN;
    SplitArgs sp = {(const float*)q, ldq, n_tokens, n_heads, (const float*)k_pages, (const float*)v_pages, block_table, table_width, page_size,
                    n_kv_heads, head_dim, spans, n_spans, seq_slot, (bf16*)work, (bf16*)work + 3 * q_size, (bf16*)work + 3 * (q_size + kv_size), rows};
    CUtensorMap mq, mk, mv;
    if (!plane_map(&mq, sp.qp, head_dim, n_heads, n_tokens, BQ) || !plane_map(&mk, sp.kp, head_dim, n_kv_heads, rows, BK) ||
        !plane_map(&mv, sp.vp, head_dim, n_kv_heads, rows, BK))
        return FX_ERR_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    const long most = q_size > kv_size ? q_size : kv_size;
    fx_launch_pdl(split_kernel, dim3((unsigned)fx_cdiv(most / 8, 256), 3), 256, 0, s, sp);
    if (const int e = fx_launch_status()) return e;
    Args a = {(const float*)q, ldq, (const float*)k_pages, (const float*)v_pages, block_table, table_width, page_size, items, seq_slot,
              (float*)out, ldo, n_heads, n_kv_heads, head_dim, window, scale, softcap, status};
    return head_dim <= 64 ? go<64>(mq, mk, mv, a, n_items, s) : go<128>(mq, mk, mv, a, n_items, s);
}
