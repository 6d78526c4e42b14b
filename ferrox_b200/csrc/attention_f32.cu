// Prompt attention over cache pages in true 32-bit arithmetic: tiles of 32 queries of one request and one head against
// blocks of 64 keys, running maximum and sum, FFMA products.  What a query sees is the function of absolute positions that
// attention_generic.cu states (causal, a window, capped scores); the sums run over blocks of 64 keys from the first
// visible block of the tile on.
//
// A block of 128 threads: thread (ty, tx) of 8 x 16 owns rows ty + 8 i, keys tx + 16 j of the scores, elements 4 tx .. of
// the result.  Scores run along the head in pairs, results along two neighbouring elements (fma.rn.f32x2).  Keys of the
// next block travel (cp.async) while the softmax and the result of this one are worked out, values while the next scores
// are.  Shared memory (91 KB at 128 elements) holds two blocks an SM, so that one's barriers hide behind the other's
// products.  517 tokens, 16 heads of 128: the warp-per-(token, head) kernel, whose lanes walk one key row each, took 1.30
// ms a layer, bound by its uncoalesced loads.  Entries that see 64 keys or more (128 with heads of 64) go to attention_f32_tc.cu
// where it takes their heads and pages: 42 against 145 us there.
#include "common.cuh"
#include "api.h"

namespace {

constexpr int BQ = 32, BK = 64, NT = 128;
typedef unsigned long long u64;

__device__ __forceinline__ void fma2(u64& d, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ u64 pair(float x, float y) {
    return (u64)__float_as_uint(x) | ((u64)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float lo_of(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_of(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }

struct AttArgs {
    const float* q; long ldq; const float* k_pages; const float* v_pages;
    const int* table; int table_width; int page_size;
    const int* tiles;            // [n][4]: first token, rows, entry, position of the first row
    const int* seq_slot;
    float* out; long ldo;
    int n_heads, n_kv_heads, dim, window;
    float scale, softcap;
};

template <int D> struct Smem {   // D: the head's width rounded up to 64 or 128, zeros beyond it
    static constexpr int PITCH = D + 4, PP = BK + 4;
    float q[BQ * PITCH], k[BK * PITCH], v[BK * D], p[BQ * PP];
    int mapped[BK];              // whether the key's position has a page
};

template <int D>
__global__ void __launch_bounds__(NT, 2) attention_f32_kernel(AttArgs a)
{
    constexpr int PITCH = Smem<D>::PITCH, PP = Smem<D>::PP, PIECES = D / 4, C = D / 64;
    extern __shared__ __align__(16) unsigned char raw[];
    Smem<D>& sm = *reinterpret_cast<Smem<D>*>(raw);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    fx_pdl_wait();
    const int4 tile = reinterpret_cast<const int4*>(a.tiles)[blockIdx.x];
    const int tok0 = tile.x, rows = tile.y, pos0 = tile.w;
    const int h = blockIdx.y, kvh = h / (a.n_heads / a.n_kv_heads);
    const int* table = a.table + (long)a.seq_slot[tile.z] * a.table_width;
    const int last = pos0 + rows - 1;
    const int first = fx_first_key(pos0, a.window, 0) / BK * BK;

    const bool one_page = a.page_size % BK == 0;     // a block of keys lies in one page: one look at the table
    auto fetch = [&](const float* pages, float* to, int pitch, int kb, bool note) {
        int page0 = 0, at0 = 0;
        if (one_page) { page0 = table[kb / a.page_size]; at0 = kb % a.page_size; }
        for (int i = tid; i < BK * PIECES; i += NT) {
            const int r = i / PIECES, d = (i - r * PIECES) * 4, key = kb + r;
            int page = -1, at = at0 + r;
            if (key <= last) {
                page = page0;
                if (!one_page) { page = table[key / a.page_size]; at = key % a.page_size; }
            }
            const bool ok = page >= 0 && d < a.dim;
            const float* src = ok ? pages + (((long)page * a.n_kv_heads + kvh) * a.page_size + at) * a.dim + d : pages;
            const int n = ok ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         :: "r"((uint32_t)__cvta_generic_to_shared(to + r * pitch + d)), "l"(src), "r"(n));
            if (note && d == 0) sm.mapped[r] = page >= 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = tid; i < BQ * PIECES; i += NT) {
        const int r = i / PIECES, d = (i - r * PIECES) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows && d < a.dim) x = *reinterpret_cast<const float4*>(a.q + (long)(tok0 + r) * a.ldq + (long)h * a.dim + d);
        *reinterpret_cast<float4*>(sm.q + r * PITCH + d) = x;
    }
    fetch(a.k_pages, sm.k, PITCH, first, true);
    fetch(a.v_pages, sm.v, D, first, false);

    float m[4], l[4];
    u64 o[4][2 * C];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * C; ++c) o[i][c] = 0ull;
    }
    const int n_rows = (rows + 7) / 8;           // of a thread's four rows, those that exist in the tile
    for (int kb = first; kb <= last; kb += BK) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                         // this block's keys are there
        u64 s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0ull;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            ulonglong2 kv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const ulonglong2*>(sm.k + (tx + 16 * j) * PITCH + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i >= n_rows) break;
                const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(sm.q + (ty + 8 * i) * PITCH + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) { fma2(s[i][j], qv.x, kv[j].x); fma2(s[i][j], qv.y, kv[j].y); }
            }
        }
        bool mapped[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) mapped[j] = sm.mapped[tx + 16 * j];
        __syncthreads();                         // everyone has read the keys
        if (kb + BK <= last) fetch(a.k_pages, sm.k, PITCH, kb + BK, true);
        else asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= n_rows) break;
            const int pos = pos0 + ty + 8 * i, lo = fx_first_key(pos, a.window, 0);
            float x[4], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = kb + tx + 16 * j;
                x[j] = (lo_of(s[i][j]) + hi_of(s[i][j])) * a.scale;
                if (a.softcap > 0.f) x[j] = a.softcap * tanhf(x[j] / a.softcap);
                if (key < lo || key > pos || !mapped[j]) x[j] = -INFINITY;
                top = fmaxf(top, x[j]);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float mn = fmaxf(m[i], top);
            const float alpha = m[i] == -INFINITY ? 0.f : expf(m[i] - mn);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = x[j] == -INFINITY ? 0.f : expf(x[j] - mn);
                sm.p[(ty + 8 * i) * PP + tx + 16 * j] = p;
                sum += p;
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l[i] = l[i] * alpha + sum;
            m[i] = mn;
#pragma unroll
            for (int c = 0; c < 2 * C; ++c) o[i][c] = pair(lo_of(o[i][c]) * alpha, hi_of(o[i][c]) * alpha);
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                         // this block's values and everyone's weights are there
        // where some rows do not see some keys, those keys' values stay out of their sums (0 times an infinity is none)
        const bool edge = kb + BK - 1 > pos0 || (a.window > 0 && kb < fx_first_key(last, a.window, 0));
#pragma unroll 4
        for (int j = 0; j < BK; j += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i >= n_rows) break;
                w[i] = *reinterpret_cast<const float4*>(sm.p + (ty + 8 * i) * PP + j);
            }
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                ulonglong2 vv[C];
#pragma unroll
                for (int c = 0; c < C; ++c) vv[c] = *reinterpret_cast<const ulonglong2*>(sm.v + (j + jj) * D + tx * 4 + 64 * c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= n_rows) break;
                    const float p = jj == 0 ? w[i].x : jj == 1 ? w[i].y : jj == 2 ? w[i].z : w[i].w;
                    if (edge && p == 0.f) continue;
                    const u64 pp = pair(p, p);
#pragma unroll
                    for (int c = 0; c < C; ++c) { fma2(o[i][2 * c], pp, vv[c].x); fma2(o[i][2 * c + 1], pp, vv[c].y); }
                }
            }
        }
        __syncthreads();                         // everyone has read the values and the weights
        if (kb + BK <= last) fetch(a.v_pages, sm.v, D, kb + BK, false);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + 8 * i;
        if (r >= rows) break;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        float* to = a.out + (long)(tok0 + r) * a.ldo + (long)h * a.dim;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int d = tx * 4 + 64 * c;
            if (d < a.dim)
                *reinterpret_cast<float4*>(to + d) = make_float4(lo_of(o[i][2 * c]) * inv, hi_of(o[i][2 * c]) * inv,
                                                                 lo_of(o[i][2 * c + 1]) * inv, hi_of(o[i][2 * c + 1]) * inv);
        }
    }
}

template <int D> int go(const AttArgs& a, int n_tiles, cudaStream_t s)
{
    const cudaError_t set = cudaFuncSetAttribute(attention_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)sizeof(Smem<D>));      // (of the current device: asked for each time)
    if (set != cudaSuccess) return (int)set;
    fx_launch_pdl(attention_f32_kernel<D>, dim3((unsigned)n_tiles, (unsigned)a.n_heads), NT, sizeof(Smem<D>), s, a);
    return fx_launch_status();
}

}  // namespace

// Rows of 32 queries at most a tile; head widths that are a multiple of 4 and at most 128; 16-byte rows.
extern "C" int fx_prefill_attention_f32(const void* q, long ldq, const void* k_pages, const void* v_pages,
                                        const int* block_table, int table_width, int page_size, const int* tiles, int n_tiles,
                                        const int* seq_slot, void* out, long ldo, int n_heads, int n_kv_heads, int head_dim,
                                        int window, float scale, float softcap, void* stream)
{
    if (n_tiles <= 0) return FX_OK;
    if (head_dim <= 0 || head_dim % 4 || head_dim > 128 || n_kv_heads <= 0 || n_heads % n_kv_heads || n_heads > 65535 ||
        page_size <= 0)
        return FX_ERR_SIZE;
    if (ldq % 4 || ldo % 4 || (uintptr_t)q % 16 || (uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16 || (uintptr_t)out % 16 ||
        (uintptr_t)tiles % 16)
        return FX_ERR_ALIGN;
    AttArgs a = {(const float*)q, ldq, (const float*)k_pages, (const float*)v_pages, block_table, table_width, page_size,
                 tiles, seq_slot, (float*)out, ldo, n_heads, n_kv_heads, head_dim, window, scale, softcap};
    return head_dim <= 64 ? go<64>(a, n_tiles, (cudaStream_t)stream) : go<128>(a, n_tiles, (cudaStream_t)stream);
}
