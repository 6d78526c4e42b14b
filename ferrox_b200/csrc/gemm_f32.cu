// C[M,N] (+)= A[M,K] . W[N,K]^T (+ bias) in true 32-bit arithmetic (FFMA, no tensor core): the products of the 32-bit
// engine that gemm_f32_tc.cu does not take.  Two kernels; kernels/ops.py: gemm_f32_plan chooses.
//
//  * `stream`: few rows, or few rows a group.  The time is the time to stream W once, so a block takes R rows of W, its
//    eight warps share out K in chunks of 128 (a lane four elements, 16-byte loads that bypass L1), the loads of the next
//    tile are asked for before this one is reduced, and each lane keeps R x MT partial sums.  They are added over the
//    lanes by halving exchanges and over the warps in warp order: a row's result depends on nothing but K.  Measured
//    (replayed graphs, weights from memory): 1 x 11264 x 2048 in 14.0 us (6.6 TB/s; 64-row tiles with 16-element stages
//    took 165 us and more for any such step), 4 rows 18.7 us, 8 rows 29.9 us; 32 rows on 60 experts of 2816 x 2048 93 us
//    (6.2 TB/s).
//  * `tile`: BM x 128 tiles, a thread 8 x 8 outputs.  Rows of A and W lie in shared memory as they lie in memory (16
//    elements of K a stage, four places filled by cp.async), and a thread's products run along K in pairs, one
//    fma.rn.f32x2 for elements (k, k + 1) of one output: no transposing on the way in, and half the instructions (plain
//    FFMA with this much register traffic stops at 39 TFLOP/s, the pairs at 64).  The even and the odd elements of K are
//    thus summed apart and added at the end.  The next operands are read from shared memory while the products of this
//    step run.  517 x 6144 x 2048: 516 us with a 4 x 4 tile a thread, 314 us now (41 TFLOP/s); 1184 x 32768 x 2048: 48
//    TFLOP/s.  BM = 128, 64 or 32 by how evenly the tiles fill the SMs; where they are too few, K is cut into runs whose
//    partial sums a second kernel adds in order.  A thread's 8 x 4 outputs on twice the warps were 8 % slower.
//
// Error against 64-bit sums at K = 2048: 1.0e-7 (stream), 5.7e-7 (tile); one thread summing K in order: 8.1e-7.
// Grouped mode (`group_offsets`): rows [off[g], off[g+1]) use matrix g of W; `a_rows` gathers rows of A.  The host knows
// how many rows there are, not how they lie: tiles_better().
// The element-at-a-time kernel of gemm_generic.cu takes what is refused here (K or strides no multiple of 4, operands
// off the 16-byte grid, mixed element types).
#include "common.cuh"
#include "api.h"

namespace {

constexpr int MAX_ACTIVE = 1024;     // groups the stream kernel lists in shared memory

struct Args {
    const float* A; long lda; const int* a_rows;
    const float* W; long ldw; long w_gs;
    const void* bias; int bias_dtype;
    float* C; long ldc; int accumulate;
    int M, N, K;
    const int* offsets; int G;
    float* part; int splits; int split_len;
};

// For groups where tiles_better() decides, for so many rows a pass.  (A struct of its own: with these in Args the compiler made tiles
// of 64 and 32 rows that took 3 % longer.)
struct PickArgs : Args {
    int pass, sms, tiles_y;          // (rows of tiles)
    int* picked;                     // the tiles' kernel, which runs first, leaves its answer here
};

// Groups whose rows are few on average may hide some that have most of them: the stream kernel takes `pass` rows of a group
// at a time, and the blocks that hold a large group's rows of W go through its passes one after the other.  In microseconds
// on a B200: 3.3 a pass of 4 rows (2.2 of 2) of a block's 8 rows of W and 2,048 elements of K, two blocks an SM, but no less
// than the largest group's passes; 0.0555 an element of K a round of 32-row tiles, three in flight on two SMs, and 3.  Both
// kernels are launched and one of the two has nothing to do.  60 experts of 2816 x 2048: 240 rows spread evenly 276 us
// streamed (527 in tiles), a quarter of them on each of four 130 in tiles (262 streamed), 360 rows on one 227 (574).
__device__ __forceinline__ bool tiles_better(const PickArgs& a, int lane)
{
    int passes = 0, most = 0, tiles = 0;
    for (int g = lane; g < a.G; g += 32) {
        const int rows = a.offsets[g + 1] - a.offsets[g], n = (rows + a.pass - 1) / a.pass;
        passes += n;
        most = max(most, n);
        tiles += (rows + 31) / 32;
    }
    passes = __reduce_add_sync(0xffffffffu, passes);
    most = __reduce_max_sync(0xffffffffu, most);
    tiles = __reduce_add_sync(0xffffffffu, tiles);
    const long blocks = (a.N + 7) / 8, slots = 2 * a.sms;
    const long turns = max((passes * blocks + slots - 1) / slots, most * ((blocks + slots - 1) / slots));
    const long rounds = (2L * tiles * ((a.N + 127) / 128) + 3 * a.sms - 1) / (3 * a.sms);
    return turns * ((a.K + 2047) / 2048) * (a.pass <= 2 ? 22000 : 33000) > rounds * a.K * 555 + 30000;
}

__device__ __forceinline__ float4 ld_stream(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// ------------------------------------------------------------------------------------------------------ stream
constexpr int SW = 8;                // warps of a block
constexpr int CHUNK = 128;           // elements of K a warp takes at a time

// R: rows of W a block holds; two chunks of each are in flight.  Eight rows, and four where eight tokens' sums leave no
// registers for more: two blocks an SM are worth more than rows (8 tokens x 6144 x 2048: R = 8 with one block an SM 24.0
// us, R = 4 with two 16.9 us).
template <int MT, int R, typename A>
__global__ void __launch_bounds__(SW * 32, 2) stream_kernel(A a)
{
    constexpr int U = 2;
    __shared__ float red[SW][MT * R];
    __shared__ int act[MAX_ACTIVE];
    __shared__ int n_act;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_chunks = (a.K + CHUNK - 1) / CHUNK;
    const int tiles_n = (a.N + R - 1) / R;
    float4 w[U][R];

    auto load_pass = [&](const float* W, int n0, int i0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (warp + SW * (i0 + u)) * CHUNK + lane * 4;
#pragma unroll
            for (int r = 0; r < R; ++r)
                w[u][r] = k < a.K ? ld_stream(W + (long)min(n0 + r, a.N - 1) * a.ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };

    // a plain product's weights do not depend on the kernel before this one
    bool have_first = false;
    if (!a.offsets && (int)blockIdx.x < tiles_n) { load_pass(a.W, blockIdx.x * R, 0); have_first = true; }
    fx_pdl_wait();
    int total = tiles_n;
    if (a.offsets) {
        // the groups that have rows, in order
        if (warp == 0) {
            int n = 0;
            for (int g0 = 0; g0 < a.G; g0 += 32) {
                const int g = g0 + lane;
                const bool has = g < a.G && a.offsets[g + 1] > a.offsets[g];
                const unsigned m = __ballot_sync(0xffffffffu, has);
                if (has) act[n + __popc(m & ((1u << lane) - 1))] = g;
                n += __popc(m);
            }
            if constexpr (sizeof(A) != sizeof(Args)) n = *a.picked ? 0 : n;
            if (lane == 0) n_act = n;
        }
        __syncthreads();
        total = tiles_n * n_act;
    }

    for (int idx = blockIdx.x; idx < total; idx += gridDim.x) {
        const int slot = idx / tiles_n, n0 = (idx - slot * tiles_n) * R;
        const int g = a.offsets ? act[slot] : 0;
        const float* W = a.W + (long)g * a.w_gs;
        const int row_begin = a.offsets ? a.offsets[g] : 0, row_end = a.offsets ? a.offsets[g + 1] : a.M;
        if (!have_first) { load_pass(W, n0, 0); have_first = true; }
        for (int tok0 = row_begin; tok0 < row_end; tok0 += MT) {
            const float* x[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int r = tok0 + m;
                x[m] = r < row_end ? a.A + (long)(a.a_rows ? a.a_rows[r] : r) * a.lda + lane * 4 : nullptr;
            }
            float v[MT * R];
#pragma unroll
            for (int i = 0; i < MT * R; ++i) v[i] = 0.f;
            for (int i0 = 0; warp + SW * i0 < n_chunks; i0 += U) {
                if (!(have_first && i0 == 0)) load_pass(W, n0, i0);
                have_first = false;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = (warp + SW * (i0 + u)) * CHUNK;
                    if (c + lane * 4 >= a.K) break;
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        if (!x[m]) continue;
                        const float4 xv = *reinterpret_cast<const float4*>(x[m] + c);
#pragma unroll
                        for (int r = 0; r < R; ++r) v[m * R + r] = fmaf(w[u][r].x, xv.x, v[m * R + r]);
#pragma unroll
                        for (int r = 0; r < R; ++r) v[m * R + r] = fmaf(w[u][r].y, xv.y, v[m * R + r]);
#pragma unroll
                        for (int r = 0; r < R; ++r) v[m * R + r] = fmaf(w[u][r].z, xv.z, v[m * R + r]);
#pragma unroll
                        for (int r = 0; r < R; ++r) v[m * R + r] = fmaf(w[u][r].w, xv.w, v[m * R + r]);
                    }
                }
            }
            have_first = false;
            if (tok0 + MT >= row_end && idx + (int)gridDim.x < total) {
                // the next tile's weights travel while this one is reduced
                const int nidx = idx + gridDim.x, nslot = nidx / tiles_n;
                load_pass(a.W + (long)(a.offsets ? act[nslot] : 0) * a.w_gs, (nidx - nslot * tiles_n) * R, 0);
                have_first = true;
            }
            // over the lanes: every exchange halves the values a lane holds, until it has one or two complete ones
            int n = MT * R, at = 0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                if (n > 1) {
                    n >>= 1;
                    const bool up = lane & off;
#pragma unroll
                    for (int i = 0; i < MT * R / 2; ++i) {
                        if (i >= n) break;
                        const float lo = v[i], hi = v[i + n];
                        v[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, off);
                    }
                    if (up) at += n;
                } else {
                    v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
                }
            }
            __syncthreads();     // the sums before these have been read
#pragma unroll
            for (int i = 0; i < (MT * R > 32 ? MT * R / 32 : 1); ++i) red[warp][at + i] = v[i];
            __syncthreads();
            for (int o = threadIdx.x; o < MT * R; o += SW * 32) {
                const int r = tok0 + o / R, col = n0 + o % R;
                if (r >= row_end || col >= a.N) continue;
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < SW; ++i) s += red[i][o];
                if (a.bias) s += load_any(a.bias, a.bias_dtype, col);
                float* c = a.C + (long)r * a.ldc + col;
                *c = a.accumulate ? *c + s : s;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------ tile
constexpr int BN = 128, BK = 16, STAGES = 4;
constexpr int PITCH = BK + 4;        // floats a row in shared memory: eight neighbouring rows' 16-byte pieces lie in
                                     // different banks

typedef unsigned long long u64;

__device__ __forceinline__ void fma2(u64& d, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool valid) {
    const int n = valid ? 16 : 0;    // the rest is filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(n));
}

// With PickArgs it may have nothing to do, and takes no more blocks than go at once (1,500 that ask and leave take 7 us).
template <int BM, typename A>
__global__ void __launch_bounds__(BM * 2) tile_kernel(A a)
{
    constexpr bool PICK = sizeof(A) != sizeof(Args);
    constexpr int NT = BM * 2;                       // threads
    constexpr int CA = BM * (BK / 4) / NT, CB = BN * (BK / 4) / NT;   // 16-byte copies of a thread a stage
    constexpr int STAGE = (BM + BN) * PITCH;         // floats
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    fx_pdl_wait();
    if constexpr (PICK) {
        const bool mine = tiles_better(a, lane);      // (the same answer in every warp)
        if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) *a.picked = mine;
        if (!mine) return;
    }
    int y = blockIdx.y;
    do {
        int row0 = y * BM, row_end = a.M;
        const float* W = a.W;
        if (a.offsets) {
            // block row y is the y-th tile of rows of the groups laid one after the other (every warp finds it for itself)
            int left = y, found = -1;
            for (int g0 = 0; g0 < a.G && found < 0; g0 += 32) {
                const int g = g0 + lane;
                const int rows = g < a.G ? a.offsets[g + 1] - a.offsets[g] : 0;
                const int t = (rows + BM - 1) / BM;
                int sum = t;                              // tiles of the groups up to this lane's
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += v;
                }
                const unsigned m = __ballot_sync(0xffffffffu, sum > left);
                if (m) {
                    const int l = __ffs(m) - 1;
                    found = g0 + l;
                    left -= __shfl_sync(0xffffffffu, sum - t, l);
                } else {
                    left -= __shfl_sync(0xffffffffu, sum, 31);
                }
            }
            if (found < 0) return;
            row0 = a.offsets[found] + left * BM;
            row_end = a.offsets[found + 1];
            W += (long)found * a.w_gs;
        }
        const int n0 = blockIdx.x * BN;
        const int k_begin = blockIdx.z * a.split_len, k_end = min(a.K, k_begin + a.split_len);
        const int n_stages = (k_end - k_begin + BK - 1) / BK;

        // what this thread copies of every stage: piece `kc` of rows lr, lr + NT / 4, ...
        const int lr = tid >> 2, kc = (tid & 3) * 4;
        const float* a_src[CA];
        bool a_ok[CA];
#pragma unroll
        for (int i = 0; i < CA; ++i) {
            const int r = row0 + lr + i * (NT / 4);
            a_ok[i] = r < row_end;
            a_src[i] = a.A + (a_ok[i] ? (long)(a.a_rows ? a.a_rows[r] : r) * a.lda : 0) + kc;
        }
        const uint32_t smem = (uint32_t)__cvta_generic_to_shared(sm);
        const uint32_t dst = smem + (uint32_t)(lr * PITCH + kc) * 4;
        auto fetch = [&](int s) {
            if (s < n_stages) {
                const int k = k_begin + s * BK;
                const bool in_k = k + kc < k_end;
                const uint32_t d = dst + (uint32_t)((s % STAGES) * STAGE) * 4;
#pragma unroll
                for (int i = 0; i < CA; ++i)
                    cp16(d + i * (NT / 4) * PITCH * 4, a_src[i] + (in_k ? k : 0), a_ok[i] && in_k);
#pragma unroll
                for (int i = 0; i < CB; ++i) {
                    const int n = n0 + lr + i * (NT / 4);
                    const bool ok = n < a.N && in_k;
                    cp16(d + (BM + i * (NT / 4)) * PITCH * 4, W + (ok ? (long)n * a.ldw + k + kc : 0), ok);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };

        // a warp owns 32 x 64 outputs, a lane rows ty + 4 i and columns tx + 8 j of them
        const int wm = warp >> 1, wn = warp & 1;
        const int ty = lane >> 3, tx = lane & 7;
        const uint32_t a_at = smem + (uint32_t)((wm * 32 + ty) * PITCH) * 4;
        const uint32_t b_at = smem + (uint32_t)((BM + wn * 64 + tx) * PITCH) * 4;
        u64 acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;

        // Four elements of K a step.  The next step's rows of A and the next column's of W are read while this one's
        // products run; the last step of a stage reads the next stage's, after the block has met.  By then everyone is done
        // with the stage before this one, and its place is filled again.
        u64 av[2][8][2], bv[2][2];
        auto lds = [](u64* v, uint32_t at) {
            asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(at));
        };
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) fetch(s);
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) lds(av[0][i], a_at + i * 4 * PITCH * 4);
        lds(bv[0], b_at);
        uint32_t base = 0;                                // this stage's place
        for (int s = 0; s < n_stages; ++s) {
            const uint32_t next = s % STAGES == STAGES - 1 ? 0 : base + STAGE * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q == 3) {
                    asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 3) : "memory");
                    __syncthreads();
                    fetch(s + STAGES - 1);
                }
                const uint32_t off = q == 3 ? next : base + (q + 1) * 16;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    lds(bv[(j + 1) & 1], j == 7 ? b_at + off : b_at + base + (j + 1) * 8 * PITCH * 4 + q * 16);
                    lds(av[(q + 1) & 1][j], a_at + off + j * 4 * PITCH * 4);
#pragma unroll
                    for (int i = 0; i < 8; ++i) fma2(acc[i][j], av[q & 1][i][0], bv[j & 1][0]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) fma2(acc[i][j], av[q & 1][i][1], bv[j & 1][1]);
                }
            }
            base = next;
        }

#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = row0 + wm * 32 + ty + 4 * i;
            if (r >= row_end) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + wn * 64 + tx + 8 * j;
                if (n >= a.N) continue;
                float v = __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
                if (a.part) {
                    a.part[((long)blockIdx.z * a.M + r) * a.N + n] = v;
                    continue;
                }
                if (a.bias) v += load_any(a.bias, a.bias_dtype, n);
                float* c = a.C + (long)r * a.ldc + n;
                *c = a.accumulate ? *c + v : v;
            }
        }
        if constexpr (PICK) {
            __syncthreads();             // (everyone is done with the places in shared memory)
            y += gridDim.y;
            if (y < a.tiles_y) continue;
        }
        break;
    } while (true);
}

// The runs' partial sums, added in order; V neighbouring outputs of a row a thread.
template <int V>
__global__ void __launch_bounds__(128) add_runs_kernel(Args a)
{
    fx_pdl_wait();
    const long i = ((long)blockIdx.x * 128 + threadIdx.x) * V, all = (long)a.M * a.N;
    if (i >= all) return;
    const int r = (int)(i / a.N), n = (int)(i - (long)r * a.N);
    float v[V];
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = 0.f;
#pragma unroll 8
    for (int s = 0; s < a.splits; ++s) {
        if (V == 4) {
            const float4 p = *reinterpret_cast<const float4*>(a.part + (long)s * all + i);
            v[0] += p.x; v[1] += p.y; v[2] += p.z; v[V - 1] += p.w;
        } else {
            v[0] += a.part[(long)s * all + i];
        }
    }
    float* c = a.C + (long)r * a.ldc + n;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        if (a.bias) v[j] += load_any(a.bias, a.bias_dtype, n + j);
        c[j] = a.accumulate ? c[j] + v[j] : v[j];
    }
}

template <int MT, int R, typename A> int go_stream(const A& a, bool early, cudaStream_t s)
{
    const long tiles = fx_cdiv(a.N, R) * (long)(a.offsets ? a.G : 1), resident = 2L * fx_sm_count();
    fx_launch_pdl_if(early, stream_kernel<MT, R, A>, dim3((unsigned)(tiles < resident ? tiles : resident)), SW * 32, 0, s, a);
    return fx_launch_status();
}

template <typename K> int allow_smem(K kernel, size_t bytes)       // of the current device: asked for each time
{
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
constexpr size_t tile_smem(int bm) { return sizeof(float) * STAGES * (bm + BN) * PITCH; }

template <int BM> int go_tile(const Args& a, cudaStream_t s)
{
    const long rows = fx_cdiv(a.M, BM) + (a.offsets ? a.G : 0);
    if (rows > 65535) return FX_ERR_SIZE;
    if (const int e = allow_smem(tile_kernel<BM, Args>, tile_smem(BM))) return e;
    fx_launch_pdl(tile_kernel<BM, Args>, dim3((unsigned)fx_cdiv(a.N, BN), (unsigned)rows, (unsigned)a.splits), BM * 2, tile_smem(BM), s, a);
    if (a.splits > 1) {
        const int st = fx_launch_status();
        if (st != FX_OK) return st;
        if (a.N % 4 == 0 && (uintptr_t)a.part % 16 == 0)
            fx_launch_pdl(add_runs_kernel<4>, dim3((unsigned)fx_cdiv((long)a.M * a.N, 512)), 128, 0, s, a);
        else
            fx_launch_pdl(add_runs_kernel<1>, dim3((unsigned)fx_cdiv((long)a.M * a.N, 128)), 128, 0, s, a);
    }
    return fx_launch_status();
}

// The stream kernel, and where the groups' sizes are to decide the tiles before it: neither set up early beside the other, whose
// registers and L1 it would sit on while it has nothing to do (281 us became 400).
template <int MT, int R> int go_few(const Args& a, int* picked, cudaStream_t s)
{
    if (!picked) return go_stream<MT, R>(a, true, s);
    constexpr int BM = 32;
    PickArgs p;
    static_cast<Args&>(p) = a;
    p.pass = MT; p.sms = fx_sm_count(); p.tiles_y = (int)(fx_cdiv(a.M, BM) + a.G); p.picked = picked;
    const long cols = fx_cdiv(a.N, BN), at_once = fx_cdiv(4L * p.sms, cols), y = at_once < p.tiles_y ? at_once : p.tiles_y;
    if (const int e = allow_smem(tile_kernel<BM, PickArgs>, tile_smem(BM))) return e;
    fx_launch_pdl_if(false, tile_kernel<BM, PickArgs>, dim3((unsigned)cols, (unsigned)y), BM * 2, tile_smem(BM), s, p);
    if (const int e = fx_launch_status()) return e;
    return go_stream<MT, R>(p, false, s);
}

}  // namespace

// `form` > 0: the tile kernel with that many rows a tile (128, 64, 32) and K cut into `splits` runs (partial sums in
// `part`, splits * M * N floats; not with groups).  `form` < 0: the stream kernel with -form rows a pass (1, 2, 4, 8); with
// groups and `splits` 2 that or tiles of 32 rows, as the groups' sizes say (two launches; `part` holds an int).
extern "C" int fx_gemm_f32(const void* A, long lda, const int* a_rows, const void* W, long ldw, const void* bias,
                           int bias_dtype, void* C, long ldc, int accumulate, int M, int N, int K,
                           const int* group_offsets, int n_groups, long w_group_stride, int form, int splits, void* part,
                           void* stream)
{
    if (M <= 0 || N <= 0) return FX_OK;
    if (K <= 0 || splits < 1 || (splits > 1 && (!part || (group_offsets ? form >= 0 || splits > 2 : form < 0)))) return FX_ERR_SIZE;
    if (K % 4 || lda % 4 || ldw % 4 || w_group_stride % 4 || (uintptr_t)A % 16 || (uintptr_t)W % 16) return FX_ERR_ALIGN;
    if (form < 0 && group_offsets && n_groups > MAX_ACTIVE) return FX_ERR_SIZE;
    Args a;
    a.A = (const float*)A; a.lda = lda; a.a_rows = a_rows; a.W = (const float*)W; a.ldw = ldw; a.w_gs = w_group_stride;
    a.bias = bias; a.bias_dtype = bias_dtype; a.C = (float*)C; a.ldc = ldc; a.accumulate = accumulate;
    a.M = M; a.N = N; a.K = K; a.offsets = group_offsets; a.G = n_groups; a.part = splits > 1 && !group_offsets ? (float*)part : nullptr;
    int* picked = group_offsets && splits > 1 ? (int*)part : nullptr;
    if (picked) splits = 1;
    a.split_len = (int)(fx_cdiv(fx_cdiv(K, splits), BK) * BK);
    a.splits = splits;
    cudaStream_t s = (cudaStream_t)stream;
    switch (form) {
        case 128: return go_tile<128>(a, s);
        case 64: return go_tile<64>(a, s);
        case 32: return go_tile<32>(a, s);
        case -1: return go_few<1, 8>(a, picked, s);
        case -2: return go_few<2, 8>(a, picked, s);
        case -4: return go_few<4, 8>(a, picked, s);
        case -8: return go_few<8, 4>(a, picked, s);
    }
    return FX_ERR_SIZE;
}
