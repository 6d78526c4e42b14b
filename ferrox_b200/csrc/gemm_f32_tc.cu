// C[M,N] (+)= A[M,K] . W[N,K]^T (+ bias) of 32-bit operands on the tensor cores.
//
// A 32-bit value is the sum of three bfloat16 (split3.cuh).  Of the nine products of two such sums six are made: hi.hi,
// hi.mid, mid.hi, mid.mid, hi.lo, lo.hi; what is left out is up to 2^-24 of a product, 2^-27 on average.  Products of two
// bfloat16 are exact in 32 bits.  The tensor
// core adds them up by cutting instead of rounding, which over K = 2,048 would cost 1e-5; so its accumulator holds only 32
// elements of K (the small products first, then two instructions of large ones), and each thread adds these sums to
// 32-bit registers of its own, rounding as an FFMA does.  What cannot be had from the parts is done again by a
// plain loop: an element whose sum is no finite number (an operand that is infinite or no number, or an overflow).
//
// How far it is from 64-bit sums (relative 2-norm; the FFMA kernels of gemm_f32.cu in brackets, K of 1,024 to 7,808, 12 to 2,000 rows):
// operands of both signs 0.9e-7 to 1.7e-7 (1.9e-7 to 5.7e-7), or with magnitudes over four decades 1.0e-7 to 1.6e-7 (2.1e-7 to 4.0e-7).
// Not nearer everywhere: of one sign, where the cuts all have that sign, 0.7e-7 to 1.0e-7 (0.7e-7 to 2.5e-7), up to 1.3 times as far
// where FFMA's K is cut into many runs; results of a single product 4.6e-8 (2.5e-8: half a unit in the last place), at most 1.5e-7.
//
// What bounds it: six bfloat16 products where an FFMA kernel does one, so a sixth of 1,680 TFLOP/s = 280 against 64.
// A tile is 128 rows of W in the accumulator's lanes and NT <= 208 rows of A in its columns (M = 517: three tiles of 176, 2
// % of padding, where 128-row tiles of A would have 24 %).  Warp 0 fetches W as it is and the parts of A (made beforehand by
// split_kernel: they are used by every tile) by TMA; eight warps take W apart, each thread 16 elements of a row, on its way
// from shared memory to tensor memory, where the products have it as their first operand (from shared memory it would take
// a third of what that can deliver), and add up the accumulators; warp 1 issues the products.  While the products of
// stage g run, the workers take stage g + 1 of W apart and add up stage g - 1.
// Measured (weights from memory, replayed graphs; before: the FFMA tiles): 517 x 15616 x 2048 805 -> 172 us (192 TFLOP/s), 517 x
// 2048 x 7808 397 -> 92, 2,000 x 15616 x 2048 2,746 -> 581 (220), 64 x 15616 x 2048 102 -> 54; the three kernels take 14 us however
// little there is to do.
// Every CTA gets the same number of stages: whole tiles as far as they go round, then the rest cut along K into equal
// shares (`sk_tiles` tiles over `sk_ctas` CTAs), whose sums go to `part`; sum_kernel adds a tile's up in the order of K.
#include "tc_common.cuh"
#include "split3.cuh"
#include "api.h"

namespace {

using namespace fxtc;

constexpr int BW = 128;              // rows of W a tile = lanes of tensor memory
constexpr int KS = 32;               // elements of K a stage
constexpr int NW = 8;                // worker warps
constexpr int NTHREADS = 32 * (2 + NW);
constexpr int RAW_BYTES = BW * KS * 4;
constexpr int W_PLANE = KS / 2, W_COLS = 3 * W_PLANE;      // columns of tensor memory: of a part of W's stage, of its three

template <int NT> struct Cfg {
    static constexpr int XP_PLANE = NT * KS * 2, XP_BYTES = 3 * XP_PLANE;
    static constexpr int RAW = 6;                                     // places of W as it comes
    static constexpr int XS = NT <= 128 ? 5 : 3;                      // places of A's parts
    static constexpr int SMEM = RAW * RAW_BYTES + XS * XP_BYTES + 1024 /* alignment */ + 256 /* barriers */;
    static constexpr int TMEM = NT <= 16 ? 128 : NT <= 80 ? 256 : 512;   // 2 (NT + W_COLS) columns, a power of two
    static_assert(2 * (NT + W_COLS) <= TMEM, "accumulators and parts of W");
    static_assert(SMEM <= 232448, "shared memory of a block");
};

struct Args {
    const float* X; long ldx;
    const float* W; long ldw;
    const void* bias; int bias_dtype;
    float* C; long ldc; int accumulate;
    int M, N, K;
    int t_tiles, tiles, stages;      // tiles of rows of A; all tiles; stages of a whole tile
    int sk_tiles, sk_ctas;           // the first tiles, cut along K into equal shares of so many CTAs
    float* part;
    int* status;
};

// The CTA whose share of `all` stages, cut into n nearly equal ones, holds stage i.
__device__ __forceinline__ int share_of(long i, long all, int n) {
    int c = (int)(i * n / all);
    while ((c + 1) * all / n <= i) ++c;
    return c;
}

// The pieces of work of a CTA, in order: its share of the tiles that are cut (parts of one or two), then whole tiles.
struct Piece { int tile, s0, s1, slot; };    // slot < 0: a whole tile

struct Pieces {
    long at, end;                    // stages of the cut tiles that are left
    int which, next;
    __device__ __forceinline__ Pieces(const Args& a) {
        const long all = (long)a.sk_tiles * a.stages;
        const bool in = (int)blockIdx.x < a.sk_ctas;
        at = in ? blockIdx.x * all / a.sk_ctas : 0;
        end = in ? (blockIdx.x + 1L) * all / a.sk_ctas : 0;
        which = 0;
        next = a.sk_tiles + blockIdx.x;
    }
    __device__ __forceinline__ bool take(const Args& a, Piece& p) {
        if (at < end) {
            p.tile = (int)(at / a.stages);
            p.s0 = (int)(at - (long)p.tile * a.stages);
            p.s1 = (int)min((long)a.stages, end - (long)p.tile * a.stages);
            p.slot = p.s0 == 0 && p.s1 == a.stages ? -1 : 2 * (int)blockIdx.x + which;
            at += p.s1 - p.s0;
            ++which;
            return true;
        }
        if (next >= a.tiles) return false;
        p.tile = next; p.s0 = 0; p.s1 = a.stages; p.slot = -1;
        next += gridDim.x;
        return true;
    }
};

__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Rows of 64 bytes along K in the 64-byte swizzle, groups of eight rows 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld_wait8(uint32_t* r) {     // (as tc_ld_wait_for)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]) :: "memory");
}
__device__ __forceinline__ void tc_ld_wait16(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}

__device__ __forceinline__ void tc_st8(uint32_t taddr, uint4 a, uint4 b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}

// A's rows in their three parts: planes [3][M][Kp] of bfloat16, Kp = K rounded up to 8; 8 elements a thread.
__global__ void __launch_bounds__(256) split_kernel(const float* X, long ldx, int M, int K, int Kp, bf16* planes)
{
    fx_pdl_wait();
    const int per_row = Kp / 8;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long)M * per_row) return;
    const long r = i / per_row;
    const int k = (int)(i - r * per_row) * 8;
    float v[8];
    Pack<float>::load(X + r * ldx + k, v);
    if (k + 8 <= K) Pack<float>::load(X + r * ldx + k + 4, v + 4);
    else v[4] = v[5] = v[6] = v[7] = 0.f;
    uint4 p[3];
    split3_8(v, p[0], p[1], p[2]);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(planes + ((long)j * M + r) * Kp + k) = p[j];
}

// sum over [k0, k1) as a plain kernel makes it, for elements that the parts cannot give (see the top)
__device__ __forceinline__ float plain_dot(const float* x, const float* w, int k0, int k1) {
    float s = 0.f;
#pragma unroll 1
    for (int k = k0; k < k1 && s == s; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
    }
    return s;
}

template <int NT>
__global__ void __launch_bounds__(NTHREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                  const __grid_constant__ CUtensorMap map_x, Args a)
{
    using C = Cfg<NT>;
    constexpr int HALF = NT / 2;                 // columns of the accumulator a worker warp adds up
    extern __shared__ uint8_t smem_raw[];
    __shared__ int abort_flag_s;
    __shared__ uint32_t tmem_base_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t xp_base = base + C::RAW * RAW_BYTES;
    const uint32_t bars = xp_base + C::XS * C::XP_BYTES;
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_empty = [&](int s) { return bars + 8u * (C::RAW + s); };
    auto x_full = [&](int s) { return bars + 8u * (2 * C::RAW + s); };
    auto x_empty = [&](int s) { return bars + 8u * (2 * C::RAW + C::XS + s); };
    auto wp_full = [&](int b) { return bars + 8u * (2 * C::RAW + 2 * C::XS + b); };
    auto acc_full = [&](int b) { return bars + 8u * (2 * C::RAW + 2 * C::XS + 2 + b); };
    volatile int* abort_flag = &abort_flag_s;

    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        for (int s = 0; s < C::RAW; ++s) { mbar_init(raw_full(s), 1); mbar_init(raw_empty(s), NW); }
        for (int s = 0; s < C::XS; ++s) { mbar_init(x_full(s), 1); mbar_init(x_empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(wp_full(b), NW); mbar_init(acc_full(b), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    if (warp == 0) {
        // ---------------- fetches ----------------
        if (lane == 0) {
            // W is not the kernel's before this one (that is split_kernel, which has waited for all before it); its first
            // stages travel while A is taken apart
            Pieces todo(a), ahead_todo(a);
            Piece p{}, q{};
            int g = 0, w_issued = 0;
            bool ok = true, waited = false;
            bool more_w = ahead_todo.take(a, q);
            int ws = q.s0;
            auto fetch_w = [&](bool may_wait) {          // the next stage of W, if its place is free
                const int s = w_issued % C::RAW;
                const uint32_t parity = (uint32_t)((w_issued / C::RAW) & 1) ^ 1u;
                if (!may_wait && !mbar_try_wait(raw_empty(s), parity)) return false;
                if (may_wait && !mbar_wait(raw_empty(s), parity, abort_flag)) { ok = false; return false; }
                mbar_expect_tx(raw_full(s), RAW_BYTES);
                tma_load_2d(base + s * RAW_BYTES, &map_w, ws * KS, q.tile / a.t_tiles * BW, raw_full(s));
                ++w_issued;
                if (++ws == q.s1) { more_w = ahead_todo.take(a, q); ws = q.s0; }
                return true;
            };
            for (int i = 0; i < C::RAW && more_w; ++i) fetch_w(true);
            while (ok && todo.take(a, p)) {
                for (int s = p.s0; s < p.s1 && ok; ++s, ++g) {
                    if (!waited) { fx_pdl_wait(); waited = true; }
                    while (ok && more_w && w_issued <= g) fetch_w(true);     // this stage's own, whatever happens
                    if (!ok) break;
                    const int xs = g % C::XS;
                    if (!mbar_wait(x_empty(xs), (uint32_t)((g / C::XS) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(x_full(xs), C::XP_BYTES);
                    tma_load_3d(xp_base + xs * C::XP_BYTES, &map_x, s * KS, p.tile % a.t_tiles * NT, 0, x_full(xs));
                    while (ok && more_w && w_issued < g + 1 + C::RAW && fetch_w(false)) {}
                }
            }
            if (!waited) fx_pdl_wait();
            if (*abort_flag) {
                // loads that were asked for must land before the CTA's shared memory is released
                for (int i = max(0, w_issued - C::RAW); i < w_issued; ++i)
                    for (uint32_t n = 0; n < WAIT_LIMIT; ++n)
                        if (mbar_try_wait(raw_full(i % C::RAW), (uint32_t)((i / C::RAW) & 1))) break;
                for (int i = max(0, g - C::XS); i < g; ++i)
                    for (uint32_t n = 0; n < WAIT_LIMIT; ++n)
                        if (mbar_try_wait(x_full(i % C::XS), (uint32_t)((i / C::XS) & 1))) break;
            }
        }
    } else if (warp == 1) {
        // ---------------- products ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc(BW, NT);
            Pieces todo(a);
            Piece p{};
            int g = 0;
            bool ok = true;
            while (ok && todo.take(a, p)) {
                for (int s = p.s0; s < p.s1; ++s, ++g) {
                    const int b = g & 1, xs = g % C::XS;
                    // the workers arrive with stage g of W when they have added up stage g - 2: the accumulator is free too
                    ok = mbar_wait(wp_full(b), (uint32_t)((g >> 1) & 1), abort_flag) &&
                         mbar_wait(x_full(xs), (uint32_t)((g / C::XS) & 1), abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t acc = tmem_base + (uint32_t)(b * NT);
                    const uint32_t w0 = tmem_base + (uint32_t)(2 * NT + b * W_COLS), w1 = w0 + W_PLANE, w2 = w1 + W_PLANE;
                    const uint64_t x0 = smem_desc64(xp_base + xs * C::XP_BYTES), x1 = smem_desc64(xp_base + xs * C::XP_BYTES + C::XP_PLANE),
                                   x2 = smem_desc64(xp_base + xs * C::XP_BYTES + 2 * C::XP_PLANE);
                    // small products first; 16 elements of K are 8 columns of W and 32 bytes of A (2 in the descriptors' units)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        tc_mma_ts(acc, w0 + 8u * k, x2 + 2u * k, idesc, k != 0);
                        tc_mma_ts(acc, w2 + 8u * k, x0 + 2u * k, idesc, 1);
                        tc_mma_ts(acc, w1 + 8u * k, x1 + 2u * k, idesc, 1);
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        tc_mma_ts(acc, w0 + 8u * k, x1 + 2u * k, idesc, 1);
                        tc_mma_ts(acc, w1 + 8u * k, x0 + 2u * k, idesc, 1);
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) tc_mma_ts(acc, w0 + 8u * k, x0 + 2u * k, idesc, 1);
                    tc_commit(x_empty(xs));
                    tc_commit(acc_full(b));
                }
            }
        }
    } else {
        // ---------------- workers ----------------
        const int wk = warp - 2, quad = warp & 3, half = wk >> 2;
        const int row = quad * 32 + lane;                 // of W, and of tensor memory
        const uint32_t my_lanes = tmem_base + ((uint32_t)(quad * 32) << 16);
        float acc[HALF];
#pragma unroll
        for (int j = 0; j < HALF; ++j) acc[j] = 0.f;

        auto take_apart = [&](int g) {
            const int s = g % C::RAW;
            if (!__all_sync(0xffffffffu, mbar_wait(raw_full(s), (uint32_t)((g / C::RAW) & 1), abort_flag))) return false;
            const uint32_t src = base + s * RAW_BYTES + row * 128;       // this thread: elements 16 half .. 16 half + 15 of its row
            float v[2][8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t at = src + ((uint32_t)(4 * half + c) ^ (uint32_t)(row & 7)) * 16;
                float* d = v[c >> 1] + 4 * (c & 1);
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(at) : "memory");
            }
            uint4 part[2][3];
#pragma unroll
            for (int u = 0; u < 2; ++u) split3_8(v[u], part[u][0], part[u][1], part[u][2]);
            const uint32_t dst = my_lanes + (uint32_t)(2 * NT + (g & 1) * W_COLS + 8 * half);
#pragma unroll
            for (int i = 0; i < 3; ++i) tc_st8(dst + i * W_PLANE, part[0][i], part[1][i]);
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            // The place of W as it comes is given back only here, where what was read has been used: an arrival right behind
            // the loads overtook them when the tensor cores held shared memory busy, and the next rows were there before.
            if (lane == 0) { mbar_arrive(wp_full(g & 1)); mbar_arrive(raw_empty(s)); }
            return true;
        };

        auto add_up = [&](int g) {
            const int b = g & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(acc_full(b), (uint32_t)((g >> 1) & 1), abort_flag))) return false;
            tc_fence_after();
            const uint32_t at = my_lanes + (uint32_t)(b * NT + half * HALF);
            constexpr int N16 = HALF / 16;
            if constexpr (HALF % 16 == 8) {
                uint32_t r[8];
                tc_ld8(at + N16 * 16, r);
                tc_ld_wait8(r);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[N16 * 16 + j] += __uint_as_float(r[j]);
            }
            if constexpr (N16 > 0) {
                uint32_t r[2][16];
                tc_ld16(at, r[0]);
#pragma unroll
                for (int c = 0; c < N16; ++c) {
                    tc_ld_wait16(r[c & 1]);
                    if (c + 1 < N16) tc_ld16(at + (c + 1) * 16, r[(c + 1) & 1]);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c * 16 + j] += __uint_as_float(r[c & 1][j]);
                }
            }
            return true;
        };

        auto finish = [&](const Piece& p) {              // a piece's sums are complete
            fx_pdl_wait_only();
            const int n = p.tile / a.t_tiles * BW + quad * 32 + lane, t0 = p.tile % a.t_tiles * NT + half * HALF;
            const int cols = n < a.N ? min(HALF, a.M - t0) : 0;         // this lane's columns that exist (it may be none)
            // what is no finite number is made once more
            uint32_t odd[(HALF + 31) / 32];
#pragma unroll
            for (int i = 0; i < (HALF + 31) / 32; ++i) odd[i] = 0;
#pragma unroll
            for (int j = 0; j < HALF; ++j)
                if (j < cols && !(fabsf(acc[j]) <= 3.402823466e38f)) odd[j / 32] |= 1u << (j % 32);
            const float bias = a.bias && n < a.N ? load_any(a.bias, a.bias_dtype, n) : 0.f;
            if (p.slot >= 0) {
                float* mine = a.part + ((long)p.slot * NW + wk) * HALF * 32 + lane;
#pragma unroll
                for (int j = 0; j < HALF; ++j) mine[j * 32] = acc[j];
            } else {
                float* c8 = a.C + (long)t0 * a.ldc + n;
#pragma unroll
                for (int j0 = 0; j0 < HALF; j0 += 8) {
                    float old[8];
                    float* c = c8;
#pragma unroll
                    for (int j = 0; j < 8; ++j, c += a.ldc) old[j] = a.accumulate && j0 + j < cols ? *c : 0.f;
                    c = c8;
                    asm volatile("" : "+l"(c) :: "memory");          // (or the compiler keeps every column's address,
#pragma unroll
                    for (int j = 0; j < 8; ++j, c += a.ldc) {
                        const float v = acc[j0 + j] + bias;
                        if (j0 + j < cols && !(odd[j0 / 32] >> ((j0 + j) % 32) & 1)) *c = a.accumulate ? old[j] + v : v;
                    }
                    c8 = c;
                    asm volatile("" : "+l"(c8) :: "memory");         // of these eight and of the tile)
                }
            }
#pragma unroll
            for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
            // (a warp whose sums are all finite goes past this)
#pragma unroll
            for (int i = 0; i < (HALF + 31) / 32; ++i)
#pragma unroll 1
                for (; odd[i]; odd[i] &= odd[i] - 1) {
                    const int j = i * 32 + __ffs(odd[i]) - 1;
                    const float v = plain_dot(a.X + (long)(t0 + j) * a.ldx, a.W + (long)n * a.ldw, p.s0 * KS, min(a.K, p.s1 * KS));
                    float* c = a.C + (long)(t0 + j) * a.ldc + n;
                    if (p.slot >= 0) a.part[(((long)p.slot * NW + wk) * HALF + j) * 32 + lane] = v;
                    else *c = a.accumulate ? *c + (v + bias) : v + bias;
                }
        };

        Pieces todo(a);
        Piece p{}, before{};
        bool have = todo.take(a, p);
        int s = p.s0;
#pragma unroll 1
        for (int g = 0;; ++g) {
            if (have && !take_apart(g)) break;
            if (g > 0) {
                if (!add_up(g - 1)) break;
                if (!have || s == p.s0) finish(before);      // stage g - 1 was the last of the piece before
            }
            if (!have) break;
            if (++s == p.s1) { before = p; have = todo.take(a, p); s = p.s0; }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::TMEM) : "memory");
    }
    if (threadIdx.x == 0 && abort_flag_s && a.status) atomicExch(a.status, STATUS_TC_TIMEOUT);
}

// The tiles that were cut: their shares, added in the order of K.  A thread has four neighbouring features of a row of A.
__global__ void __launch_bounds__(256) sum_kernel(Args a, int nt)
{
    fx_pdl_wait();
    const int half = nt / 2, quarter = threadIdx.x & 7;
    const long i = (long)blockIdx.x * 32 + (threadIdx.x >> 3);       // (tile, worker warp, column)
    if (i >= (long)a.sk_tiles * NW * half) return;
    const int j = (int)(i % half), wk = (int)(i / half % NW), tile = (int)(i / half / NW);
    const int quad = (wk + 2) & 3;                                    // (the workers are warps 2 .. 9)
    const int n = tile / a.t_tiles * BW + quad * 32 + quarter * 4, t = tile % a.t_tiles * nt + (wk >> 2) * half + j;
    if (t >= a.M || n >= a.N) return;
    const long all = (long)a.sk_tiles * a.stages, b0 = (long)tile * a.stages;
    const int first = share_of(b0, all, a.sk_ctas), last = share_of(b0 + a.stages - 1, all, a.sk_ctas);
    if (first == last) return;                                        // (a share that is the whole tile has been stored)
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int c = first; c <= last; ++c) {
        const int slot = 2 * c + (c * all / a.sk_ctas < b0 ? 1 : 0);  // a CTA's share begins in this tile or in the one before it
        const float4 p = *reinterpret_cast<const float4*>(a.part + (((long)slot * NW + wk) * half + j) * 32 + quarter * 4);
        v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    float* c = a.C + (long)t * a.ldc + n;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (n + e < a.N) {
            if (a.bias) v[e] += load_any(a.bias, a.bias_dtype, n + e);
            c[e] = a.accumulate ? c[e] + v[e] : v[e];
        }
}

template <int NT> int go(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, int grid, cudaStream_t s)
{
    auto kern = gemm_f32_tc_kernel<NT>;
    // of the current device: asked for each time
    if (const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<NT>::SMEM)) return (int)e;
    fx_launch_pdl(kern, dim3((unsigned)grid), NTHREADS, Cfg<NT>::SMEM, s, mw, mx, a);
    return fx_launch_status();
}

template <int NT> int pick(int n_tile, const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, int grid, cudaStream_t s)
{
    if (n_tile == NT) return go<NT>(mw, mx, a, grid, s);
    if constexpr (NT > 16) return pick<NT - 16>(n_tile, mw, mx, a, grid, s);
    return FX_ERR_SIZE;
}

constexpr int MIN_SHARE = 4;         // stages a CTA is worth waking for

}  // namespace

// n_tile: rows of A a tile, 16 .. 208 in steps of 16.  `work`, 16-byte aligned: the planes of A (6 M Kp bytes, Kp = K rounded up
// to 8), then the shares of the tiles that are cut (n_tile x 1,024 bytes for each SM).
extern "C" int fx_gemm_f32_tc(const void* X, long ldx, const void* W, long ldw, const void* bias, int bias_dtype, void* C, long ldc,
                              int accumulate, int M, int N, int K, int n_tile, void* work, long work_bytes, int* status,
                              void* stream)
{
    if (M <= 0 || N <= 0) return FX_OK;
    if (K <= 0 || n_tile < 16 || n_tile > 208 || n_tile % 16) return FX_ERR_SIZE;
    if (K % 4 || ldx % 4 || ldw % 4 || (uintptr_t)X % 16 || (uintptr_t)W % 16 || (uintptr_t)work % 16) return FX_ERR_ALIGN;
    const long Kp = fx_cdiv(K, 8) * 8, sms = fx_sm_count();
    const long planes = 6L * M * Kp, parts = sms * 2 * BW * n_tile * 4;
    if (work_bytes < planes + parts) return FX_ERR_SIZE;
    const long t_tiles = fx_cdiv(M, n_tile), tiles = t_tiles * fx_cdiv(N, BW);
    if (tiles > 0x7fffffffL / 2 || fx_cdiv((long)M * (Kp / 8), 256) > 0x7fffffffL) return FX_ERR_SIZE;
    Args a;
    a.X = (const float*)X; a.ldx = ldx; a.W = (const float*)W; a.ldw = ldw; a.bias = bias; a.bias_dtype = bias_dtype;
    a.C = (float*)C; a.ldc = ldc; a.accumulate = accumulate; a.M = M; a.N = N; a.K = K;
    a.t_tiles = (int)t_tiles; a.tiles = (int)tiles; a.stages = (int)fx_cdiv(K, KS);
    a.part = (float*)((char*)work + planes); a.status = status;
    // whole tiles as far as they go round; the rest in equal shares
    a.sk_tiles = (int)(tiles % sms);
    const long stages = (long)a.sk_tiles * a.stages;
    const long shares = stages / MIN_SHARE > a.sk_tiles ? stages / MIN_SHARE : a.sk_tiles;
    a.sk_ctas = (int)(shares < sms ? shares : sms);
    const int grid = (int)(tiles < sms ? a.sk_ctas : sms);

    EncodeTiledFn fn = encode_fn();
    if (!fn) return FX_ERR_SIZE;
    CUtensorMap mw, mx;
    {
        cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)ldw * 4};
        cuuint32_t box[2] = {KS, BW}, es[2] = {1, 1};
        if (fn(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(W), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return FX_ERR_SIZE;
    }
    {
        cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3}, strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)M * Kp * 2};
        cuuint32_t box[3] = {KS, (cuuint32_t)n_tile, 3}, es[3] = {1, 1, 1};
        if (fn(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, work, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return FX_ERR_SIZE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    fx_launch_pdl(split_kernel, dim3((unsigned)fx_cdiv((long)M * (Kp / 8), 256)), 256, 0, s, (const float*)X, ldx, M, K, (int)Kp,
                  (bf16*)work);
    if (const int e = fx_launch_status()) return e;
    if (const int e = pick<208>(n_tile, mw, mx, a, grid, s)) return e;
    if (a.sk_tiles) {
        fx_launch_pdl(sum_kernel, dim3((unsigned)fx_cdiv((long)a.sk_tiles * NW * (n_tile / 2), 32)), 256, 0, s, a, n_tile);
        return fx_launch_status();
    }
    return FX_OK;
}
