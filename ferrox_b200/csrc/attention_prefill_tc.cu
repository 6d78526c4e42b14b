// Attention for prompt portions on the 5th-generation tensor cores (bfloat16, keys of up to 192 and values of up to
// 128 elements a head in steps of 8, pages of 64 positions or a multiple).  Key and value widths may differ; in shared
// and tensor memory both are rounded up to 64, 128 or 192 (D and V below), the rest filled with zeros by the TMA.
//
// One CTA takes up to 256 query tokens of one request and one head, as two sub-tiles of 128 rows, and
// walks that request's keys in blocks of 128 positions (earlier steps' keys and the portion's own alike,
// found through the block table).  For each sub-tile t and key block j:
//
//   S_t = Q_t K_j^T    tcgen05.mma 128 x 128 x head_dim; Q and K tiles in shared memory (TMA, 128-byte
//                      swizzle), S_t in tensor memory (32-bit)
//   P_t = exp2(...)    each of the sub-tile's 128 softmax threads owns one query row: tcgen05.ld of its
//                      row of S, mask by absolute position (query p sees keys max(0, p - W + 1) .. p),
//                      running max and sum in 32 bits; P rounded to bfloat16 and written back over the
//                      first columns of S_t (tcgen05.st), where the next product reads it as its A operand
//   O_t += P_t V_j     tcgen05.mma 128 x head_dim x 128, A from tensor memory, V as an N-major B operand,
//                      exactly as TMA lays the [key][head_dim] rows down; O_t stays in tensor memory
//
// The running maximum of a row is only raised when it grows by more than 2^8 (the weights then stay
// below 2^8 and the final division by the row sum makes the result the same); when it is raised, the
// row's thread scales its row of O_t in tensor memory.  This takes the accumulator out of the softmax
// threads' registers and off their critical path.
//
// Warp 0 issues the TMA loads (K and V blocks double-buffered), warp 1 issues the tensor-core
// instructions and owns the tensor-memory allocation (512 columns: S_0, S_1, O_0, O_1), warps 2-5 are
// sub-tile 0's softmax threads and warps 6-9 sub-tile 1's, warp 10 clears what nobody sees.  The products are issued in the order
// PV_0(j), S_0(j+1), PV_1(j), S_1(j+1): while one sub-tile's threads work on their block the tensor
// cores work for the other.  Every wait is bounded (status code 3 on time-out, then the roles leave,
// tensor memory is freed and the kernel returns).  Keys that are masked are still multiplied, with weight 0, and 0 times a
// value that is infinite or no number is none.  So what lies in a block's place in shared memory for a position that no query of
// the item sees is zero: where there is no page the TMA fills it in (a page number behind the last), and in the blocks at the
// edges (behind the last query, before the first one's window) warp 10 clears the rows of V before their product.
// What one query sees and another of its sub-tile does not stays: elements of a result that are no finite number while the
// weights' sum is one are made again from the operands as they are (remake), so that such a value reaches only the queries that see
// it.  (Looking for them and the call take 0.2 us of a prompt of 53 tokens, 0.3 to 1.1 us of 55 to 110.)
//
// A work item is a tile of queries, a head and a run of key blocks [kb_begin, kb_end).  The host cuts the
// key blocks of long tiles into runs (the last 256 queries of a long prompt see many times the keys the
// first see, and a portion behind a long cached prefix is a single tile with all of them), so that the
// items are of similar length and there are enough of them for every SM; the heavy ones come first in the
// table.  An item that holds all of its tile's key blocks writes the tile's output.  Any other writes what
// it has (the unnormalised sums in 32 bits, and each row's reference maximum and sum of weights) into
// scratch memory, and a second kernel (prefill_merge_kernel) adds a tile's runs up in their order.
//
// Queries, keys and values are reached through strides of their own (rows that hold all heads side by side, or pages);
// `value_share` consecutive key heads may read one value head.
//
// Options: `keep_first` (with a window: the request's first positions stay visible; the key blocks that hold them and lie
// before a tile's own are walked first, by its first run), `softcap` (scores pass through c tanh(s / c); the row's maximum
// is taken before, tanh keeps the order), `chunk` (a query sees the keys of its own chunk of that many positions only, counted from the request's
// start), `sinks` (one number per head: exp(sink_h) joins the softmax's denominator once, at the end or in the merge),
// `gate` (token rows of n_heads * value_dim: the result is multiplied by sigmoid(gate) before it is rounded), `turn`
// ([tokens][value_dim / 2] (cos, sin): pair (2m, 2m + 1) of the result is turned by minus that angle before the gate).
//
// What bounds it: the softmax threads' instructions a score (4.5 plain, 12 capped) beside the two products; an item costs 13 us
// before its first key block.  The general forms against the mma.sync kernels that took them before (16 heads of 128, 2,048
// tokens in a window of 1,024): with kept first keys 111 -> 61 us, capped 127 -> 83; 16 heads of 192 and 128, 2,048 tokens: 220
// -> 76; 32 maps of 64 on values of 128, capped, 1,531 tokens: 130 -> 100.  A warp none of whose rows exists leaves its block to
// the others (300 tokens beside 15 single ones, capped: 176 -> 124).
//
// Reference: crates/ferrox-core/src/attention.rs:531-563 (query t over keys 0..=t), :146-175 (online
// softmax), :484-524 (window), :572-610 (pages), :432-449 (grouped heads).  The mma.sync kernel of
// attention_prefill.cu remains for other head sizes and page sizes.
#include "tc_common.cuh"
#include "api.h"

namespace {

using namespace fxtc;

constexpr int BQ = 128, BKEY = 128, NTHREADS = 352, TMEM_COLS = 512;
constexpr float RAISE_MAX_BY = 8.f;   // in powers of two

__device__ __forceinline__ float fast_exp2(float x) {   // 2^x, approximate; -inf gives 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// How a score becomes a weight: the plain kernel's exponential is the hardware's (weights below 2^-126 are 0), the general
// forms' is exp2f, and their denominators add up the weights as the second product has them (rounded to bfloat16: a row with
// one large weight then has none of its rounding).
// What rescales a row, its sink and the merge of its runs is done the same way: weights below 2^-126 reach a result whose values
// are large enough.
enum { FAST = 0, GENERAL = 1, CAPPED = 2 };
template <int MODE> __device__ __forceinline__ float exp2_of(float x) { return MODE == FAST ? fast_exp2(x) : exp2f(x); }

// A capped score in powers of two, c log2(e) tanh(k s) with k = scale / c.  Up to k s = 1/2, tanh(x) = x + x z p(z), z = x^2, p
// fitted (weighted least squares towards the smallest largest error, 1.5e-8 of tanh(x); in 32 bits 7.5e-8): a cubic in s^2
// whose coefficients hold k and the unit, two scores an instruction, no special function.  Beyond, tanhf.  The caps taken here (up
// to CAP_MAX) keep every weight above 2^-126, where exp2f is the hardware's exponential.
constexpr float CAP_MAX = 40.f, CAP_SMALL = 0.5f;
struct Cap {
    float k, unit, cap, c[4];        // c: of s^3, s^5, s^7, s^9
};

__device__ __forceinline__ uint64_t pair_of(float x, float y) { return (uint64_t)__float_as_uint(x) | ((uint64_t)__float_as_uint(y) << 32); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// 32 scores <- capped, less ref
__device__ __forceinline__ void cap_small(const Cap& cap, uint32_t* s, float ref) {
    const uint64_t c0 = pair_of(cap.c[0], cap.c[0]), c1 = pair_of(cap.c[1], cap.c[1]), c2 = pair_of(cap.c[2], cap.c[2]),
                   c3 = pair_of(cap.c[3], cap.c[3]), u = pair_of(cap.unit, cap.unit), r = pair_of(-ref, -ref);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const uint64_t x = (uint64_t)s[i] | ((uint64_t)s[i + 1] << 32), x2 = mul2(x, x);
        const uint64_t q = fma2(fma2(fma2(c3, x2, c2), x2, c1), x2, c0);
        const uint64_t y = fma2(mul2(x, x2), q, fma2(x, u, r));
        s[i] = (uint32_t)y; s[i + 1] = (uint32_t)(y >> 32);
    }
}
__device__ __forceinline__ void cap_any(const Cap& cap, uint32_t* s, float ref) {
#pragma unroll
    for (int i = 0; i < 32; ++i) s[i] = __float_as_uint(fmaf(cap.cap, tanhf(cap.k * __uint_as_float(s[i])), -ref));
}

constexpr int ITEM_INTS = 8;   // a work item: first flat token, rows, entry, first position, kb_begin, kb_end, part, kept blocks

struct AttnArgs {
    const int* block_table; int table_width; int page_size, n_pages;
    const int* tiles; const int* seq_slot;
    const bf16 *q, *k, *v; long ldq, ldqh, kv_at[6];      // the operands, for remake; strides of a page, a head, a position: keys, values
    int head_dim;
    bf16* out; long ldo;
    float* part_o; float* part_ml;   // partial results of items that hold a run of their tile's key blocks only
    int n_heads, n_kv_heads, window, chunk;
    int keep_first, value_share;
    Cap cap;                         // CAPPED
    int value_dim;                   // elements of a value head (V: rounded up)
    const float* sinks;              // (optional) one per head
    const bf16* gate; long ldg;      // (optional) token rows of n_heads * value_dim
    const float* turn;               // (optional) [tokens][value_dim / 2] (cos, sin)
    float scale_log2e;
    int* status;
};

// What a row's sums are multiplied with at the end: 1 / (l + the head's sink), l being relative to 2^ref.
template <int MODE> __device__ __forceinline__ float inverse_sum(float l, float ref, const float* sinks, int head) {
    if (!(l > 0.f)) return 0.f;
    if (!sinks) return 1.f / l;
    const float sk = sinks[head] * 1.4426950408889634f, mm = fmaxf(ref, sk), f = exp2_of<MODE>(ref - mm);
    return f / (l * f + exp2_of<MODE>(sk - mm));
}

// Row `row` of this block's item: the elements of its result (in `out`, or the 32-bit sums of an item that holds a run) that are no finite
// numbers, made again from the operands as they are, over the keys that the query sees, weights rounded as for the product, against the
// reference `ref`; `inv`: one over the weights' sum.  Rare, and out of line: it reads anew what it needs to know, so that the kernel keeps no registers for it.
template <int MODE, int V>
__device__ __noinline__ void remake(const AttnArgs& a, int row, float ref, float inv)
{
    const int* item = a.tiles + (long)blockIdx.y * ITEM_INTS;
    const int* table = a.block_table + (long)a.seq_slot[item[2]] * a.table_width;
    const int head = blockIdx.x, kvh = head / (a.n_heads / a.n_kv_heads), pos = item[3] + row, lo = fx_first_key(pos, a.window, a.chunk);
    const int first_blk = item[4], end_blk = item[5], part = item[6], n_kept = item[7];
    const long token = item[0] + row;
    const bf16 *q = a.q + token * a.ldq + head * a.ldqh, *k_head = a.k + kvh * a.kv_at[1], *v_head = a.v + kvh / a.value_share * a.kv_at[4];
    float* sums = part >= 0 ? a.part_o + (((long)part * a.n_heads + head) * (2 * BQ) + row) * V : nullptr;
    bf16* dst = a.out + token * a.ldo + (long)head * a.value_dim;
    const bf16* gate = a.gate ? a.gate + token * a.ldg + (long)head * a.value_dim : nullptr;
    const float* turn = a.turn ? a.turn + token * a.value_dim : nullptr;
    for (int c = 0; c < a.value_dim; c += 8) {
        float o[8];
        uint32_t odd = 0;
        for (int d = 0; d < 8; ++d) {
            const float x = sums ? sums[c + d] : __bfloat162float(dst[c + d]);
            if (!(fabsf(x) < INFINITY)) odd |= turn && !sums ? 3u << (d & ~1) : 1u << d;       // (a pair that was turned: both)
            o[d] = 0.f;
        }
        uint32_t left = odd;                      // what no key yet made no number
        for (int j = n_kept > 0 ? 0 : first_blk; j < end_blk && left; j = j + 1 == n_kept ? first_blk : j + 1)
            for (int key = j * BKEY; key < (j + 1) * BKEY && key <= pos && left; ++key) {
                if (key < lo && key >= a.keep_first) continue;
                const int page = table[key / a.page_size], at = key % a.page_size;
                if (page < 0) continue;
                const bf16* k = k_head + page * a.kv_at[0] + at * a.kv_at[2];
                float s = 0.f;
                for (int d = 0; d < a.head_dim; d += 8) {
                    float x[8], y[8];
                    Pack<bf16>::load(q + d, x);
                    Pack<bf16>::load(k + d, y);
                    for (int i = 0; i < 8; ++i) s = fmaf(x[i], y[i], s);
                }
                const float x = MODE == CAPPED ? fmaf(a.cap.cap, tanhf(a.cap.k * s), -ref) : fmaf(s, a.scale_log2e, -ref);
                const float w = __bfloat162float(__float2bfloat16_rn(exp2_of<MODE>(x)));
                float v[8];
                Pack<bf16>::load(v_head + page * a.kv_at[3] + at * a.kv_at[5] + c, v);
                left = 0;
                for (int d = 0; d < 8; ++d) {
                    o[d] = fmaf(w, v[d], o[d]);
                    if ((odd >> d & 1) && o[d] == o[d]) left |= 1u << d;
                }
            }
        if (turn && !sums)
            for (int d = 0; d < 8; d += 2) {
                o[d] *= inv; o[d + 1] *= inv;
                fx_turn_back(o[d], o[d + 1], *reinterpret_cast<const float2*>(turn + c + d));
            }
        for (int d = 0; d < 8; ++d) {
            if (!(odd >> d & 1)) continue;
            if (sums) { sums[c + d] = o[d]; continue; }
            if (!turn) o[d] *= inv;
            if (gate) o[d] *= fx_sigmoid_fast(__bfloat162float(gate[c + d]));
            dst[c + d] = __float2bfloat16_rn(o[d]);
        }
    }
}

template <int D, int V>
struct Smem {
    static constexpr int HALVES = D / 64, V_HALVES = V / 64;   // 64-element (128-byte) slices of a key's, a value's row
    static constexpr int SUB = 128 * 128;                  // bytes of a [128 rows x 128 bytes] piece
    static constexpr int Q_BYTES = HALVES * SUB, K_BYTES = HALVES * SUB, V_BYTES = V_HALVES * SUB;
    static constexpr int V_PLACES = D > 128 ? 1 : 2;       // (wider keys leave room for one block of values)
    static constexpr int Q_OFF = 0, K_OFF = 2 * Q_BYTES, V_OFF = K_OFF + 2 * K_BYTES;
    static constexpr int BAR_OFF = V_OFF + V_PLACES * V_BYTES;
    static constexpr int TOTAL = BAR_OFF + 128 + 1024;     // barriers, alignment slack
    static_assert(TOTAL <= 232448 - 64, "shared memory of a block");
};

template <int D, int V, int MODE>
__global__ void __launch_bounds__(NTHREADS, 1) prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                           const __grid_constant__ CUtensorMap map_k,
                                                                           const __grid_constant__ CUtensorMap map_v,
                                                                           const __grid_constant__ AttnArgs a)
{
    using L = Smem<D, V>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int abort_flag_s;
    __shared__ uint32_t tmem_base_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // The host lists heavy items first, and blocks are handed out with blockIdx.x running fastest: every head's
    // heaviest item, then every head's next one, so that the light items fill the gaps at the end.
    const int* item = a.tiles + (long)blockIdx.y * ITEM_INTS;
    const int tok0 = item[0], rows = item[1], entry = item[2], pos0 = item[3];
    const int kb_begin = item[4], kb_end = item[5], part = item[6], n_kept = item[7];
    const int head = blockIdx.x;
    const int kvh = head / (a.n_heads / a.n_kv_heads);
    const int last_pos = pos0 + rows - 1;
    // sub-tile t: rows_of(t) rows from position pos0 + 128 t; it needs the key blocks blk_lo(t) .. blk_hi(t)
    const int nt = rows > BQ ? 2 : 1;
    auto rows_of = [&](int t) { return min(BQ, rows - t * BQ); };
    auto blk_lo = [&](int t) {
        return fx_first_key(pos0 + t * BQ, a.window, a.chunk) / BKEY;
    };
    auto blk_hi = [&](int t) { return (pos0 + t * BQ + rows_of(t) - 1) / BKEY; };
    // the key blocks of sub-tile t inside this item's run: lo_t[t] .. hi_t[t] (none if lo > hi)
    const int lo0 = max(blk_lo(0), kb_begin), hi0 = min(blk_hi(0), kb_end - 1);
    const int lo1 = nt > 1 ? max(blk_lo(1), kb_begin) : 1, hi1 = nt > 1 ? min(blk_hi(1), kb_end - 1) : 0;
    auto lo_of = [&](int t) { return t ? lo1 : lo0; };
    auto hi_of = [&](int t) { return t ? hi1 : hi0; };
    const bool act0 = lo0 <= hi0, act1 = lo1 <= hi1;
    const int first_blk = act0 && act1 ? min(lo0, lo1) : act0 ? lo0 : lo1;
    const int last_blk = act0 && act1 ? max(hi0, hi1) : act0 ? hi0 : hi1;
    // what the item walks: the kept blocks 0 .. n_kept - 1, then first_blk .. last_blk
    const int n_walk = n_kept + max(0, last_blk - first_blk + 1), kept_end = (a.keep_first + BKEY - 1) / BKEY;
    auto block_of = [&](int i) { return i < n_kept ? i : first_blk + i - n_kept; };
    auto active = [&](int t, int i) {
        if (t >= nt || i >= n_walk) return false;
        const int j = block_of(i);
        return (j >= lo_of(t) && j <= hi_of(t)) || (j < kept_end && j < blk_lo(t));
    };
    // walked blocks with positions that no query of the item sees: the last kept one, the window's first, the last
    const int lo_item = fx_first_key(pos0, a.window, a.chunk);
    auto is_edge = [&](int i) {
        const int kb = block_of(i) * BKEY;
        return i >= 0 && i < n_walk && (kb + BKEY - 1 > last_pos || (kb < lo_item && kb + BKEY > a.keep_first)) && (active(0, i) || active(1, i));
    };
    const int edge0 = is_edge(n_kept - 1) ? n_kept - 1 : -1, edge1 = is_edge(n_kept) ? n_kept : -1, edge2 = is_edge(n_walk - 1) ? n_walk - 1 : -1;
    auto at_edge = [&](int i) { return i == edge0 || i == edge1 || i == edge2; };
    auto last_of = [&](int t) {                            // the last walked block that sub-tile t needs (none: -1)
        int i = n_walk - 1;
        while (i >= 0 && !active(t, i)) --i;
        return i;
    };

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar0 = base + L::BAR_OFF;
    const uint32_t q_full = bar0;
    auto s_full = [&](int t) { return bar0 + 8 + 8u * t; };
    auto p_full = [&](int t) { return bar0 + 24 + 8u * t; };
    auto o_done = [&](int t) { return bar0 + 40 + 8u * t; };
    auto k_full = [&](int b) { return bar0 + 56 + 8u * b; };
    auto v_full = [&](int b) { return bar0 + 72 + 8u * b; };
    auto kv_empty = [&](int b) { return bar0 + 88 + 8u * b; };
    // where the loads of a block at an edge arrive: its k_full and v_full are raised when what nobody sees has been cleared
    auto v_edge = [&](int b) { return bar0 + 104 + 8u * b; };
    volatile int* abort_flag = &abort_flag_s;

    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        mbar_init(q_full, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(s_full(b), 1); mbar_init(p_full(b), 4); mbar_init(o_done(b), 1);
            mbar_init(k_full(b), 1); mbar_init(v_full(b), 1); mbar_init(kv_empty(b), 1);
            mbar_init(v_edge(b), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    fx_pdl_wait();   // set up while the kernel before this one drains; its results (q, the pages) from here on
    auto tmem_s = [&](int t) { return tmem_base + 128u * t; };        // S_t, and P_t over its first 64 columns
    auto tmem_o = [&](int t) { return tmem_base + 256u + 128u * t; };

    if (warp == 0) {
        // ---------------- producer: Q once, then K and V blocks ----------------
        if (lane == 0) {
            mbar_expect_tx(q_full, nt * L::Q_BYTES);
            for (int t = 0; t < nt; ++t)
                for (int h = 0; h < L::HALVES; ++h)
                    tma_load_3d(base + L::Q_OFF + t * L::Q_BYTES + h * L::SUB, &map_q, h * 64, head, tok0 + t * BQ, q_full);
            const int* table = a.block_table + (long)a.seq_slot[entry] * a.table_width;
            int issued = 0, v_issued = 0;
            uint32_t v_edges = 0;           // loads at edges so far, odd or even, a bit a place
            for (int i = 0; i < n_walk; ++i) {
                const int j = block_of(i), b = i & 1, vb = L::V_PLACES == 2 ? b : 0;
                if (!mbar_wait(kv_empty(b), (uint32_t)((i >> 1) & 1) ^ 1u, abort_flag)) break;
                int page[2], off[2];
                for (int hk = 0; hk < 2; ++hk) {   // the two runs of 64 keys of the block
                    const int key = j * BKEY + hk * 64;
                    const int p = key <= last_pos ? table[key / a.page_size] : -1;
                    page[hk] = p >= 0 ? p : a.n_pages;      // no page (beyond the request, or before its window): zeros
                    off[hk] = p >= 0 ? key % a.page_size : 0;
                }
                const bool edge = at_edge(i);
                const uint32_t v_bar = edge ? v_edge(vb) : v_full(vb);
                mbar_expect_tx(k_full(b), L::K_BYTES);
                for (int h = 0; h < L::HALVES; ++h)
                    for (int hk = 0; hk < 2; ++hk)
                        tma_load_4d(base + L::K_OFF + b * L::K_BYTES + h * L::SUB + hk * 8192, &map_k, h * 64, off[hk], kvh,
                                    page[hk], k_full(b));
                issued = i + 1;
                // (one place of values: free when the block before this one has been multiplied)
                if (L::V_PLACES == 1 && i > 0 && !mbar_wait(kv_empty((i - 1) & 1), (uint32_t)(((i - 1) >> 1) & 1), abort_flag)) break;
                mbar_expect_tx(v_bar, L::V_BYTES);
                for (int h = 0; h < L::V_HALVES; ++h)
                    for (int hk = 0; hk < 2; ++hk)
                        tma_load_4d(base + L::V_OFF + vb * L::V_BYTES + h * L::SUB + hk * 8192, &map_v, h * 64, off[hk],
                                    kvh / a.value_share, page[hk], v_bar);
                v_issued = i + 1;
                if (edge) v_edges ^= 1u << vb;
            }
            if (*abort_flag) {   // loads already issued must land before the shared memory is released
                // (each the last of its place, so that an edge's phase is the one before the next)
                for (int i = max(0, issued - 2); i < issued; ++i)
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(k_full(i & 1), (uint32_t)((i >> 1) & 1))) break;
                for (int i = max(0, v_issued - L::V_PLACES); i < v_issued; ++i) {
                    const bool edge = at_edge(i);
                    const int vb = i % L::V_PLACES;
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(edge ? v_edge(vb) : v_full(vb), edge ? (v_edges >> vb & 1u) ^ 1u : (uint32_t)((i / L::V_PLACES) & 1))) break;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- tensor-core issue ----------------
        if (lane == 0) {
            constexpr uint32_t idesc_s = instr_desc_ex(BQ, BKEY, 0);   // S: B = K tile, K-major
            constexpr uint32_t idesc_o = instr_desc_ex(BQ, V, 1);      // O: B = V tile, N-major
            int k_ready = -1;              // the last walked block whose K is known to have landed
            const int last0 = last_of(0), last1 = last_of(1);
            bool ok = mbar_wait(q_full, 0, abort_flag);
            auto issue_s = [&](int t, int i) {
                const int b = i & 1;
                if (k_ready < i) {
                    if (!mbar_wait(k_full(b), (uint32_t)((i >> 1) & 1), abort_flag)) return false;
                    k_ready = i;
                    tc_fence_after();
                }
#pragma unroll
                for (int h = 0; h < L::HALVES; ++h) {
                    const uint64_t dq = smem_desc(base + L::Q_OFF + t * L::Q_BYTES + h * L::SUB);
                    const uint64_t dk = smem_desc(base + L::K_OFF + b * L::K_BYTES + h * L::SUB);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc_mma(tmem_s(t), dq + 2u * k, dk + 2u * k, idesc_s, (h | k) != 0);
                }
                tc_commit(s_full(t));
                return true;
            };
            for (int t = 0; t < nt && ok; ++t)
                if (active(t, 0)) ok = issue_s(t, 0);
            int n_p[2] = {0, 0};   // blocks of each sub-tile whose P has been taken
            for (int i = 0; i < n_walk && ok; ++i) {
                const int b = i & 1, vb = L::V_PLACES == 2 ? b : 0;
                bool v_ready = false;
                for (int t = 0; t < nt && ok; ++t) {
                    if (active(t, i)) {
                        ok = mbar_wait(p_full(t), (uint32_t)(n_p[t] & 1), abort_flag);
                        if (ok && !v_ready) { ok = mbar_wait(v_full(vb), (uint32_t)((i / L::V_PLACES) & 1), abort_flag); v_ready = true; }
                        if (!ok) break;
                        tc_fence_after();
                        // O_t += P V: 8 steps of 16 keys.  A = P from tensor memory, 8 columns a step.  B = V,
                        // N-major: a step covers two 8-key groups (1024 bytes each, the stride operand); the two
                        // 64-element slices of the head dimension lie SUB bytes apart (the leading operand).
#pragma unroll
                        for (int ks = 0; ks < BKEY / 16; ++ks) {
                            const uint64_t dv = smem_desc_lbo_sbo(base + L::V_OFF + vb * L::V_BYTES + ks * 2048, L::SUB, 1024);
                            tc_mma_ts(tmem_o(t), tmem_s(t) + 8u * ks, dv, idesc_o, (n_p[t] | ks) != 0);
                        }
                        ++n_p[t];
                        if (i == (t ? last1 : last0)) tc_commit(o_done(t));
                    }
                    if (t == nt - 1) tc_commit(kv_empty(b));   // every product that reads this stage has been issued
                    if (active(t, i + 1)) ok = issue_s(t, i + 1);
                }
            }
        }
    } else if (warp < 10) {
        // ---------------- softmax: one query row per thread ----------------
        const int t = (warp - 2) >> 2;
        const int quad = warp & 3;                       // the lanes of tensor memory this warp may touch
        const int r = quad * 32 + lane;
        if (t < nt) {
            const int rows_t = rows_of(t);
            const int pos0_t = pos0 + t * BQ;
            const int p_r = pos0_t + r;                  // absolute position of this row
            const int lo_r = fx_first_key(p_r, a.window, a.chunk);
            const int lo_last = fx_first_key(pos0_t + BQ - 1, a.window, a.chunk);     // the largest of the sub-tile's rows
            const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
            const uint32_t ts = tmem_s(t) + lane_off, to = tmem_o(t) + lane_off;
            const float sl2 = MODE == CAPPED ? 1.f : a.scale_log2e;   // (a capped score is one of 2's powers already)
            float m = -INFINITY, l = 0.f;
            bool ok = true;
            int cnt = 0;
            for (int i = 0; i < n_walk; ++i) {
                if (!active(t, i)) continue;
                const int j = block_of(i);
                ok = __all_sync(0xffffffffu, mbar_wait(s_full(t), (uint32_t)(cnt & 1), abort_flag));
                if (!ok) break;
                tc_fence_after();
                if (quad * 32 >= rows_t) {           // none of the warp's rows exists: what its rows of P hold reaches no others
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(p_full(t));
                    ++cnt;
                    continue;
                }
                const int kb = j * BKEY;
                // every key of the block visible to every row of the sub-tile: no masking (most blocks)
                const bool interior = kb + BKEY - 1 <= pos0_t && (kb >= lo_last || kb + BKEY <= a.keep_first);
                // The row of S is read in chunks of 32 columns into two register buffers in turn: the load of the
                // next chunk is in flight while the current one is worked on.
                uint32_t ca[32], cb[32], pk[32];
                auto mask = [&](uint32_t* c, int chunk, uint32_t with) {
                    if (interior) return;
#pragma unroll
                    for (int k = 0; k < 32; ++k) {
                        const int key = kb + chunk * 32 + k;
                        if (key > p_r || (key < lo_r && key >= a.keep_first)) c[k] = with;
                    }
                };
                constexpr uint32_t MINUS_INF = 0xff800000u, NO_NUMBER = 0x7fffffffu;
                // first pass: the row's maximum
                float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY, size0 = 0.f, size1 = 0.f;
                auto take_max = [&](uint32_t* c, int chunk) {
                    mask(c, chunk, NO_NUMBER);           // (what fmaxf passes over, also where sizes are taken)
                    if (MODE == CAPPED) {
#pragma unroll
                        for (int k = 0; k < 32; k += 2) {
                            size0 = fmaxf(size0, fabsf(__uint_as_float(c[k]))); size1 = fmaxf(size1, fabsf(__uint_as_float(c[k + 1])));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 32; k += 4) {
                        mx0 = fmaxf(mx0, __uint_as_float(c[k])); mx1 = fmaxf(mx1, __uint_as_float(c[k + 1]));
                        mx2 = fmaxf(mx2, __uint_as_float(c[k + 2])); mx3 = fmaxf(mx3, __uint_as_float(c[k + 3]));
                    }
                };
                tc_ld32(ts, ca);
                tc_ld_wait_for(ca);
                tc_ld32(ts + 32, cb); take_max(ca, 0); tc_ld_wait_for(cb);
                tc_ld32(ts + 64, ca); take_max(cb, 1); tc_ld_wait_for(ca);
                tc_ld32(ts + 96, cb); take_max(ca, 2); tc_ld_wait_for(cb);
                tc_ld32(ts, ca);      take_max(cb, 3);   // chunk 0 again, for the second pass
                float top = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
                const bool all_small = MODE == CAPPED && __all_sync(0xffffffffu, r >= rows_t || fmaxf(size0, size1) * a.cap.k <= CAP_SMALL);
                if (MODE == CAPPED && top != -INFINITY) {
                    // (as its weight will be worked out, but for the last place)
                    const float x2 = top * top, q = fmaf(fmaf(fmaf(a.cap.c[3], x2, a.cap.c[2]), x2, a.cap.c[1]), x2, a.cap.c[0]);
                    top = all_small ? fmaf(top * x2, q, top * a.cap.unit) : a.cap.cap * tanhf(a.cap.k * top);
                }
                const float mn = fmaxf(m, top);
                // (rows that do not exist, another request's queries, have no say in the others' references)
                const bool raise = r < rows_t && mn > m && (m == -INFINITY || (mn - m) * sl2 > RAISE_MAX_BY);
                if (__any_sync(0xffffffffu, raise)) {
                    const float alpha = m == -INFINITY ? 0.f : exp2_of<MODE>((m - mn) * sl2);
                    l *= alpha;
                    m = mn;
                    if (cnt > 0) {   // the sums so far of this row, in tensor memory, take the new reference too
#pragma unroll
                        for (int c = 0; c < V / 32; ++c) {
                            tc_ld32(to + c * 32, cb);
                            tc_ld_wait_for(cb);
#pragma unroll
                            for (int k = 0; k < 32; ++k) cb[k] = __float_as_uint(__uint_as_float(cb[k]) * alpha);
                            tc_st32(to + c * 32, cb);
                        }
                    }
                }
                // second pass: P = exp2(S * scale - reference), as bfloat16 pairs over the first 64 columns of S
                // (columns 0-31 are written after columns 0-63 were read, columns 32-63 after all were)
                const float ref = m == -INFINITY ? 0.f : m * sl2;
                float sum0 = 0.f, sum1 = 0.f;
                auto weight = [&](uint32_t c) {
                    if (MODE == CAPPED) return fast_exp2(__uint_as_float(c));
                    const float x = fmaf(__uint_as_float(c), sl2, -ref);
                    return MODE == FAST ? fast_exp2(x) : exp2f(x);
                };
                auto take_exp = [&](uint32_t* c, int chunk, uint32_t* out) {
                    if (MODE == CAPPED) {
                        if (all_small) cap_small(a.cap, c, ref); else cap_any(a.cap, c, ref);
                    }
                    mask(c, chunk, MINUS_INF);
#pragma unroll
                    for (int k = 0; k < 32; k += 2) {
                        float e0 = weight(c[k]), e1 = weight(c[k + 1]);
                        __nv_bfloat162 pr = __floats2bfloat162_rn(e0, e1);
                        if (MODE != FAST) {
                            const uint32_t w = *reinterpret_cast<uint32_t*>(&pr);
                            e0 = __uint_as_float(w << 16); e1 = __uint_as_float(w & 0xffff0000u);
                        }
                        sum0 += e0; sum1 += e1;
                        out[k >> 1] = *reinterpret_cast<uint32_t*>(&pr);
                    }
                };
                tc_ld_wait_for(ca);
                tc_ld32(ts + 32, cb); take_exp(ca, 0, pk);      tc_ld_wait_for(cb);
                tc_ld32(ts + 64, ca); take_exp(cb, 1, pk + 16); tc_ld_wait_for(ca);
                tc_ld32(ts + 96, cb);
                tc_st32(ts, pk);                                 // the loads of columns 0-63 have completed
                take_exp(ca, 2, pk);
                tc_ld_wait_for(cb);
                take_exp(cb, 3, pk + 16);
                tc_st32(ts + 32, pk);
                l += sum0 + sum1;
                tc_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full(t));
                ++cnt;
            }
            const bool has_blocks = last_of(t) >= 0;
            float again_inv = 1.f;
            __nv_bfloat162 zero[4] = {};
            float none[4] = {0.f, 0.f, 0.f, 0.f};        // no number where an element of this row's result is no finite number
            if (ok && has_blocks) ok = __all_sync(0xffffffffu, mbar_wait(o_done(t), 0, abort_flag));
            if (ok && part >= 0) {
                // a run of the tile's key blocks: the sums as they are, each row's reference and sum of weights
                tc_fence_after();
                const long slot = ((long)part * a.n_heads + head) * (2 * BQ) + t * BQ + r;
                if (r < rows_t) { a.part_ml[slot * 2] = has_blocks ? m : -INFINITY; a.part_ml[slot * 2 + 1] = has_blocks ? l : 0.f; }
                if (has_blocks) {
                    float* dst = a.part_o + slot * V;
#pragma unroll
                    for (int c = 0; c < V / 32; ++c) {
                        uint32_t ob[32];
                        tc_ld32(to + c * 32, ob);
                        tc_ld_wait();
                        if (r < rows_t) {
#pragma unroll
                            for (int k = 0; k < 32; ++k) none[k & 3] = fmaf(__uint_as_float(ob[k]), 0.f, none[k & 3]);
#pragma unroll
                            for (int k = 0; k < 32; k += 4)
                                *reinterpret_cast<uint4*>(dst + c * 32 + k) = make_uint4(ob[k], ob[k + 1], ob[k + 2], ob[k + 3]);
                        }
                    }
                }
            } else if (ok && has_blocks) {
                tc_fence_after();
                const float inv = inverse_sum<MODE>(l, m * sl2, a.sinks, head);
                bf16* dst = a.out + (long)(tok0 + t * BQ + r) * a.ldo + (long)head * a.value_dim;
                const bf16* gate = a.gate ? a.gate + (long)(tok0 + t * BQ + r) * a.ldg + (long)head * a.value_dim : nullptr;
                const float* turn = a.turn ? a.turn + (long)(tok0 + t * BQ + r) * a.value_dim : nullptr;
#pragma unroll
                for (int c = 0; c < V / 32; ++c) {
                    uint32_t ob[32];
                    tc_ld32(to + c * 32, ob);
                    tc_ld_wait();
                    if (r < rows_t) {
#pragma unroll
                        for (int k = 0; k < 32; k += 8) {
                            if (c * 32 + k >= a.value_dim) continue;      // (zeros beyond the value's width)
                            float x[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(ob[k + e]) * inv;
                            if (turn) {
                                const float4 c0 = *reinterpret_cast<const float4*>(turn + c * 32 + k);
                                const float4 c1 = *reinterpret_cast<const float4*>(turn + c * 32 + k + 4);
                                fx_turn_back(x[0], x[1], make_float2(c0.x, c0.y)); fx_turn_back(x[2], x[3], make_float2(c0.z, c0.w));
                                fx_turn_back(x[4], x[5], make_float2(c1.x, c1.y)); fx_turn_back(x[6], x[7], make_float2(c1.z, c1.w));
                            }
                            if (gate) {
                                float g[8];
                                Pack<bf16>::load(gate + c * 32 + k, g);
#pragma unroll
                                for (int e = 0; e < 8; ++e) x[e] *= fx_sigmoid_fast(g[e]);
                            }
                            __nv_bfloat162 y[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                y[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
                                zero[e] = __hfma2(y[e], __nv_bfloat162(0.f, 0.f), zero[e]);
                            }
                            *reinterpret_cast<uint4*>(dst + c * 32 + k) = *reinterpret_cast<const uint4*>(y);
                        }
                    }
                }
                again_inv = inv;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) none[e] += __low2float(zero[e]) + __high2float(zero[e]);
            const float sum = (none[0] + none[1]) + (none[2] + none[3]);
            if (sum != sum && l > 0.f && l < INFINITY) remake<MODE, V>(a, t * BQ + r, m * sl2, again_inv);
        }
    } else {
        // ---------------- zeros where nobody sees a position ----------------
        // (A warp of its own: among the softmax threads' lines these cost 3 us of 55 in items without an edge.  Its code comes last: before
        // theirs it cost the plain form 1 to 2 per cent.)
        auto clear_rows = [&](uint32_t at, int slices, int from, int to) {
            for (int h = 0; h < slices; ++h)
#pragma unroll 4
                for (int c = from * 128 + lane * 16; c < to * 128; c += 512)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at + h * L::SUB + c), "r"(0) : "memory");
        };
        auto clear = [&](uint32_t at, int slices, int kb) {
            clear_rows(at, slices, max(0, a.keep_first - kb), min(BKEY, lo_item - kb));
            clear_rows(at, slices, max(0, last_pos + 1 - kb), BKEY);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
        };
        uint32_t v_phases = 0;             // a bit a place
        for (int i = 0; i < n_walk; ++i) {
            if (!at_edge(i)) continue;
            const int vb = L::V_PLACES == 2 ? i & 1 : 0, kb = block_of(i) * BKEY;
            if (!__all_sync(0xffffffffu, mbar_wait(v_edge(vb), v_phases >> vb & 1u, abort_flag))) break;
            v_phases ^= 1u << vb;
            clear(base + L::V_OFF + vb * L::V_BYTES, L::V_HALVES, kb);
            if (lane == 0) mbar_arrive(v_full(vb));
        }
    }

    // ---- teardown ---------------------------------------------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0 && abort_flag_s && a.status) atomicExch(a.status, STATUS_TC_TIMEOUT);
}

// Adds up the runs of key blocks of the tiles that were cut: row r of a tile has, from run c, the sums o_c (32-bit,
// relative to the reference m_c) and the sum of weights l_c; with M = max m_c the result is
// sum_c o_c 2^((m_c - M) s) / sum_c l_c 2^((m_c - M) s), the runs taken in their order.  A run without visible keys
// for the row has m_c = -inf and is skipped.  merges: int32 [n, 4] = (first flat token, rows, first part, runs).
template <int V, int MODE>
__global__ void __launch_bounds__(128) prefill_merge_kernel(const int* __restrict__ merges, const float* __restrict__ part_o,
                                                            const float* __restrict__ part_ml, bf16* __restrict__ out, long ldo,
                                                            int n_heads, float scale_log2e, int value_dim,
                                                            const float* __restrict__ sinks,
                                                            const bf16* __restrict__ gate, long ldg,
                                                            const float* __restrict__ turn)
{
    fx_pdl_wait();
    const int* mg = merges + (long)blockIdx.x * 4;
    const int tok0 = mg[0], rows = mg[1], part0 = mg[2], runs = mg[3];
    const int head = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int PER = V / 32;   // elements of a row per lane
    const int r = blockIdx.z * 4 + warp;   // a warp a row: all of a row's loads are on their way together
    if (r >= rows) return;
    const long slot0 = ((long)part0 * n_heads + head) * (2 * BQ) + r;
    const long run_stride = (long)n_heads * (2 * BQ);          // slots from one run to the next
    // lane c holds run c's reference and sum (runs <= 32)
    float m_c = -INFINITY, l_c = 0.f;
    if (lane < runs) {
        const float2 ml = *reinterpret_cast<const float2*>(part_ml + (slot0 + lane * run_stride) * 2);
        m_c = ml.x; l_c = ml.y;
    }
    const float mx = warp_max(m_c);
    const float w_c = m_c == -INFINITY ? -1.f : exp2_of<MODE>((m_c - mx) * scale_log2e);      // (-1: no visible keys)
    float acc[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] = 0.f;
    float l = 0.f;
#pragma unroll 4
    for (int c = 0; c < runs; ++c) {
        const float w = __shfl_sync(0xffffffffu, w_c, c);
        const float l_of = __shfl_sync(0xffffffffu, l_c, c);
        if (w == -1.f) continue;   // a run without visible keys for this row wrote no sums
        l = fmaf(l_of, w, l);
        const float* src = part_o + (slot0 + c * run_stride) * V + lane * PER;
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(src[i], w, acc[i]);
    }
    if (lane * PER >= value_dim) return;
    const float inv = inverse_sum<MODE>(l, mx * scale_log2e, sinks, head);
    bf16* dst = out + (long)(tok0 + r) * ldo + (long)head * value_dim + lane * PER;
    const bf16* g = gate ? gate + (long)(tok0 + r) * ldg + (long)head * value_dim + lane * PER : nullptr;
    static_assert(PER % 2 == 0, "a lane holds whole pairs");
    if (turn) {
#pragma unroll
        for (int i = 0; i < PER; i += 2)
            fx_turn_back(acc[i], acc[i + 1], *reinterpret_cast<const float2*>(turn + (long)(tok0 + r) * value_dim + lane * PER + i));
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        float x = acc[i] * inv;
        if (g) x *= fx_sigmoid_fast(__bfloat162float(g[i]));
        dst[i] = __float2bfloat16_rn(x);
    }
}

bool encode(CUtensorMap* map, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D, int V, int MODE>
int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const AttnArgs& a, dim3 grid, const int* merges,
           int n_merges, cudaStream_t s)
{
    auto kern = prefill_attention_tc_kernel<D, V, MODE>;
    // of the current device: asked for each time
    if (const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D, V>::TOTAL)) return (int)e;
    fx_launch_pdl(kern, grid, NTHREADS, Smem<D, V>::TOTAL, s, mq, mk, mv, a);
    const float unit = MODE == CAPPED ? 1.f : a.scale_log2e;
    if (n_merges > 0)
        fx_launch_pdl(prefill_merge_kernel<V, MODE>, dim3(n_merges, a.n_heads, 2 * BQ / 4), 128, 0, s, merges, (const float*)a.part_o,
                      (const float*)a.part_ml, a.out, a.ldo, a.n_heads, unit, a.value_dim, a.sinks, a.gate, a.ldg, a.turn);
    return fx_launch_status();
}

template <int MODE>
int pick(int head_dim, int value_dim, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const AttnArgs& a, dim3 grid,
         const int* merges, int n_merges, cudaStream_t s)
{
    const bool narrow = value_dim <= 64;
    if (head_dim <= 64) return narrow ? launch<64, 64, MODE>(mq, mk, mv, a, grid, merges, n_merges, s) : launch<64, 128, MODE>(mq, mk, mv, a, grid, merges, n_merges, s);
    if (head_dim <= 128) return narrow ? launch<128, 64, MODE>(mq, mk, mv, a, grid, merges, n_merges, s) : launch<128, 128, MODE>(mq, mk, mv, a, grid, merges, n_merges, s);
    if constexpr (MODE == GENERAL)
        return narrow ? launch<192, 64, MODE>(mq, mk, mv, a, grid, merges, n_merges, s) : launch<192, 128, MODE>(mq, mk, mv, a, grid, merges, n_merges, s);
    return FX_ERR_SIZE;
}

}  // namespace

// items: int32 [n_items, 8] = (first flat token, rows <= 256, entry index, absolute position of the first row, first
// key block of 128 positions, end of the key blocks, part or -1, kept blocks: blocks 0 .. that - 1 before the first, for keep_first), the heavy ones first.  An item with part -1
// holds every key block its tile sees and writes the tile's output; the items of a tile that was cut write their
// partial results to part_o [parts, n_heads, 256, value_dim rounded up to 64 or 128] and part_ml [parts, n_heads, 256, 2] (32-bit), and
// merges: int32 [n_merges, 4] = (first flat token, rows, first part, runs) tells the second kernel which to add up
// (a tile's runs have consecutive parts, in the order of their keys).
// q: rows `ldq` elements apart, heads `ldqh`; n_tokens its number of rows.  kv_strides (elements; null: pages [page][kv head]
// [position][width]): of a page, a head and a position of the keys, then of the values.  general: exp2f for the weights, as every
// softcap, keep_first, value_share or key width above 128 has it (those refuse 0).
// Refuses (FX_ERR_SIZE / FX_ERR_ALIGN) what it does not take; the caller then uses the mma.sync kernel.
extern "C" int fx_prefill_attention_tc(const void* q, long ldq, long ldqh, int n_tokens, const void* k_pages, const void* v_pages,
                                       int n_pages, const int* block_table, int table_width, int page_size,
                                       const int* tiles, int n_tiles, const int* seq_slot, void* out, long ldo,
                                       int n_heads, int n_kv_heads, int head_dim, int value_dim, int window, int chunk,
                                       float scale, const float* sinks, const void* gate, long ldg, const float* turn,
                                       const long* kv_strides, int keep_first, float softcap, int value_share, int general, int* status,
                                       float* part_o, float* part_ml, const int* merges, int n_merges, void* stream)
{
    if (n_tiles <= 0) return FX_OK;
    if (n_merges > 0 && (!part_o || !part_ml || !merges || (uintptr_t)part_o % 16)) return FX_ERR_ALIGN;
    if (keep_first < 0 || value_share < 1 || n_kv_heads % value_share || !(softcap >= 0.f) || softcap > CAP_MAX) return FX_ERR_SIZE;
    if (softcap > 0.f && !(scale / softcap >= 1e-4f && scale / softcap <= 1e4f)) return FX_ERR_SIZE;      // (the coefficients' range)
    if (!general && (softcap > 0.f || keep_first || value_share > 1 || head_dim > 128)) return FX_ERR_SIZE;
    if (head_dim <= 0 || head_dim > (softcap > 0.f ? 128 : 192) || head_dim % 8 || value_dim <= 0 || value_dim > 128 || value_dim % 8 ||
        page_size < 64 || page_size % 64 || n_kv_heads <= 0 || n_heads % n_kv_heads || chunk < 0 || !(scale > 0.f))
        return FX_ERR_SIZE;
    if (ldqh % 8 || ldq % 8 || ldo % 8 || (uintptr_t)q % 16 || (uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16 || (uintptr_t)out % 16)
        return FX_ERR_ALIGN;
    if ((gate && (ldg % 8 || (uintptr_t)gate % 16)) || (uintptr_t)turn % 16) return FX_ERR_ALIGN;
    if (n_tiles > 65535) return FX_ERR_SIZE;
    CUtensorMap mq, mk, mv;
    AttnArgs a;
    {
        cuuint64_t dims[3] = {(cuuint64_t)head_dim, (cuuint64_t)n_heads, (cuuint64_t)n_tokens};
        cuuint64_t strides[2] = {(cuuint64_t)ldqh * 2, (cuuint64_t)ldq * 2};
        cuuint32_t box[3] = {64, 1, 128};
        if (!encode(&mq, q, 3, dims, strides, box)) return FX_ERR_SIZE;
    }
    for (int v = 0; v < 2; ++v) {
        const int width = v ? value_dim : head_dim;
        const int heads = v ? n_kv_heads / value_share : n_kv_heads;
        long at[3] = {(long)heads * page_size * width, (long)page_size * width, width};      // of a page, a head, a position
        for (int i = 0; i < 3; ++i) {
            if (kv_strides) at[i] = kv_strides[3 * v + i];
            if (at[i] % 8) return FX_ERR_ALIGN;
            a.kv_at[3 * v + i] = at[i];
        }
        cuuint64_t dims[4] = {(cuuint64_t)width, (cuuint64_t)page_size, (cuuint64_t)heads, (cuuint64_t)n_pages};
        cuuint64_t strides[3] = {(cuuint64_t)at[2] * 2, (cuuint64_t)at[1] * 2, (cuuint64_t)at[0] * 2};
        cuuint32_t box[4] = {64, 64, 1, 1};
        if (!encode(v ? &mv : &mk, v ? v_pages : k_pages, 4, dims, strides, box)) return FX_ERR_SIZE;
    }
    a.block_table = block_table; a.table_width = table_width; a.page_size = page_size; a.n_pages = n_pages;
    a.q = (const bf16*)q; a.k = (const bf16*)k_pages; a.v = (const bf16*)v_pages; a.ldq = ldq; a.ldqh = ldqh; a.head_dim = head_dim;
    a.tiles = tiles; a.seq_slot = seq_slot; a.out = (bf16*)out; a.ldo = ldo;
    a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.window = window; a.chunk = chunk; a.value_dim = value_dim;
    a.sinks = sinks; a.gate = (const bf16*)gate; a.ldg = ldg; a.turn = turn;
    a.scale_log2e = scale * 1.4426950408889634f; a.status = status;
    a.part_o = part_o; a.part_ml = part_ml; a.keep_first = window > 0 ? keep_first : 0; a.value_share = value_share;
    if (softcap > 0.f) {
        const double k = (double)scale / softcap, u = (double)scale * 1.4426950408889634, p[4] = {-0.33333140612, 0.13325783610, -0.05303649604, 0.01721787080};
        double kk = k * k;
        for (int i = 0; i < 4; ++i, kk *= k * k) a.cap.c[i] = (float)(u * kk * p[i]);
        a.cap.k = (float)k; a.cap.unit = (float)u; a.cap.cap = softcap * 1.4426950408889634f;
    }
    dim3 grid(n_heads, n_tiles);
    cudaStream_t s = (cudaStream_t)stream;
    if (softcap > 0.f) return pick<CAPPED>(head_dim, value_dim, mq, mk, mv, a, grid, merges, n_merges, s);
    if (general) return pick<GENERAL>(head_dim, value_dim, mq, mk, mv, a, grid, merges, n_merges, s);
    return pick<FAST>(head_dim, value_dim, mq, mk, mv, a, grid, merges, n_merges, s);
}
