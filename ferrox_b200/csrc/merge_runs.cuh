// The sum over the runs of keys that separate blocks took for one (token, head), for the attention kernels that leave partial
// results to a second kernel: run s has the largest score m_s, the weights' sum l_s and the values' sum o_s [dim], and either has no
// keys (nothing was written) or counts for exp(m_s - m).  The order of the sums is that of the runs.
//
// Bound by latency: the few runs of a head are a few KB.  A thread that walks them waits for each maximum, and then for each sum and
// value, in turn; here a thread takes a run's maximum and weight, and the values of eight runs are under way at once.
// B200, what the merge adds to a step: 16 tokens, 16 heads of 256 in 9 runs 30 -> 10 us; 4 tokens, 16 heads of 128 in 11 runs 8.9 -> 6.3.
#pragma once
#include "common.cuh"

constexpr int FX_MERGE_MAX_THREADS = 256;

// Threads of a block: one for each element, whole warps.
inline int fx_merge_threads(int dim) { return dim >= FX_MERGE_MAX_THREADS ? FX_MERGE_MAX_THREADS : (dim + 31) / 32 * 32; }

struct RunsOfHead {
    const float *o, *ml;         // [n][dim], [n][2]
    int n, dim;
};

// The largest score of the runs; -inf: none has keys.  All threads of the block call it together.
template <typename HasKeys> __device__ __forceinline__ float fx_runs_max(const RunsOfHead& r, HasKeys has_keys)
{
    __shared__ float of_warp[FX_MERGE_MAX_THREADS / 32];
    float m = -INFINITY;
    for (int s = threadIdx.x; s < r.n; s += blockDim.x)
        if (has_keys(s)) m = fmaxf(m, r.ml[2 * s]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x % 32 == 0) of_warp[threadIdx.x / 32] = m;
    __syncthreads();
    for (int w = 0; w < (int)blockDim.x / 32; ++w) m = fmaxf(m, of_warp[w]);
    return m;
}

// (values' sum of element e, weights' sum), beginning with (0, l).  All threads call it together; `in`: e is an element.
template <typename HasKeys, typename Weight>
__device__ __forceinline__ float2 fx_runs_sum(const RunsOfHead& r, int e, bool in, float m, float l, HasKeys has_keys, Weight weight)
{
    __shared__ float w_s[FX_MERGE_MAX_THREADS], l_s[FX_MERGE_MAX_THREADS];
    float a = 0.f;
    for (int s0 = 0; s0 < r.n; s0 += blockDim.x) {
        const int s = s0 + threadIdx.x, here = min(r.n - s0, (int)blockDim.x);
        float w = -1.f, ls = 0.f;                // (-1: no keys)
        if (s < r.n && has_keys(s)) {
            const float ms = r.ml[2 * s];
            ls = r.ml[2 * s + 1];
            if (ms != -INFINITY) w = weight(ms - m);
        }
        __syncthreads();                         // (everyone is done with the runs before these)
        w_s[threadIdx.x] = w;
        l_s[threadIdx.x] = ls;
        __syncthreads();
        for (int i0 = 0; in && i0 < here; i0 += 8) {
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = i0 + i < here && w_s[i0 + i] != -1.f ? r.o[(long)(s0 + i0 + i) * r.dim + e] : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i0 + i >= here || w_s[i0 + i] == -1.f) continue;
                l += l_s[i0 + i] * w_s[i0 + i];
                a += o[i] * w_s[i0 + i];
            }
        }
    }
    return make_float2(a, l);
}
