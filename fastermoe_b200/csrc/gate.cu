// Gate top-k: the k largest logits of every token and their expert indices, and the
// backward of that selection.  Replaces the torch.topk call of the reference's gates
// (fmoe/gates/naive_gate.py:31-34, gshard_gate.py / switch_gate.py through NaiveGate)
// and the scatter its autograd runs in the backward pass.
//
// One warp per token.  Each lane keeps the best k of the logits it strides over in
// registers (descending value, ascending expert index among equal values; NaN ranks
// above every number, as in torch.topk), then k rounds of a warp arg-max pick the
// winners in order.  Values are copied, never rounded.
#include "common.cuh"
#include <algorithm>
#include <climits>
#include <cmath>

namespace fmoe {
namespace {

constexpr int kTopKMax = 8;

// (a, ia) ranks before (b, ib)
__device__ __forceinline__ bool ranks_before(float a, int ia, float b, int ib) {
    const bool na = a != a, nb = b != b;
    if (na != nb) return na;
    if (!na && a != b) return a > b;
    return ia < ib;
}

// Softmax over the k selected logits (best[0] is the largest; NaN ranks first), as values of T.
template <typename T>
__device__ __forceinline__ void store_softmax(const float (&best)[kTopKMax], int k, T* __restrict__ values) {
    float p[kTopKMax], sum = 0.f;
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j)
        if (j < k) { p[j] = expf(best[j] - best[0]); sum += p[j]; }
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j)
        if (j < k) values[j] = from_float<T>(p[j] / sum);
}

// SOFTMAX: the values are the softmax over the selected logits.  As an operator of its own that softmax cost a launch
// in each direction (1.4-2 us of device time, 10 us of host time) for k values per token.
template <typename T, bool SOFTMAX>
__global__ void __launch_bounds__(256)
topk_forward_kernel(const T* __restrict__ logits, int64_t n_tokens, int n_expert, int k, T* __restrict__ values,
                    int64_t* __restrict__ indices) {
    const int lane = threadIdx.x & 31;
    const int64_t tok = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tok >= n_tokens) return;
    const T* row = logits + tok * n_expert;
    float best[kTopKMax];
    int best_i[kTopKMax];
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j) { best[j] = -INFINITY; best_i[j] = INT_MAX; }
    for (int e = lane; e < n_expert; e += 32) {
        float v = to_float(row[e]);
        int vi = e;
        // insertion into the lane's sorted list (entries past k are never read)
#pragma unroll
        for (int j = 0; j < kTopKMax; ++j) {
            if (j < k && ranks_before(v, vi, best[j], best_i[j])) {
                const float tv = best[j]; const int ti = best_i[j];
                best[j] = v; best_i[j] = vi;
                v = tv; vi = ti;
            }
        }
    }
    float won[kTopKMax];
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j) {
        if (j >= k) break;
        float v = best[0];
        int vi = best_i[0];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int oi = __shfl_xor_sync(0xffffffffu, vi, off);
            if (ranks_before(ov, oi, v, vi)) { v = ov; vi = oi; }
        }
        if (best_i[0] == vi) {  // this lane owned the winner: drop it
#pragma unroll
            for (int q = 0; q + 1 < kTopKMax; ++q) { best[q] = best[q + 1]; best_i[q] = best_i[q + 1]; }
            best[kTopKMax - 1] = -INFINITY; best_i[kTopKMax - 1] = INT_MAX;
        }
        won[j] = v;
        if (lane == 0) {
            if (!SOFTMAX) values[tok * k + j] = row[vi];
            indices[tok * k + j] = vi;
        }
    }
    if (SOFTMAX) {          // all lanes know the winners: each stores one probability (131072 x 256, k = 8: 252 us by one lane, 241)
        float mine = 0.f, sum = 0.f;
#pragma unroll
        for (int j = 0; j < kTopKMax; ++j)
            if (j < k) {
                const float p = expf(won[j] - won[0]);
                sum += p;
                if (j == lane) mine = p;
            }
        if (lane < k) values[tok * k + lane] = from_float<T>(mine / sum);
    }
}

// Few experts (<= 32): one THREAD per token; a warp then reads 32 consecutive rows, i.e. one
// contiguous stretch of the logits, and no lane idles.  Same order as the warp kernel.
template <typename T, bool SOFTMAX>
__global__ void __launch_bounds__(256)
topk_forward_small_kernel(const T* __restrict__ logits, int64_t n_tokens, int n_expert, int k, T* __restrict__ values,
                          int64_t* __restrict__ indices) {
    const int64_t tok = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tok >= n_tokens) return;
    const T* row = logits + tok * n_expert;
    float best[kTopKMax];
    int best_i[kTopKMax];
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j) { best[j] = -INFINITY; best_i[j] = INT_MAX; }
    for (int e = 0; e < n_expert; ++e) {
        float v = to_float(row[e]);
        int vi = e;
#pragma unroll
        for (int j = 0; j < kTopKMax; ++j) {
            if (j < k && ranks_before(v, vi, best[j], best_i[j])) {
                const float tv = best[j]; const int ti = best_i[j];
                best[j] = v; best_i[j] = vi;
                v = tv; vi = ti;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kTopKMax; ++j) {
        if (j < k) {
            if (!SOFTMAX) values[tok * k + j] = row[best_i[j]];
            indices[tok * k + j] = best_i[j];
        }
    }
    if (SOFTMAX) store_softmax<T>(best, k, values + tok * k);
}

template <typename T, bool SOFTMAX>
__global__ void __launch_bounds__(256)
topk_backward_kernel(const T* __restrict__ grad_values, const T* __restrict__ probs, const int64_t* __restrict__ indices, int64_t n_tokens,
                     int n_expert, int k, T* __restrict__ grad_logits) {
    const int64_t total = n_tokens * n_expert;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tok = i / n_expert;
        const int e = (int)(i - tok * n_expert);
        float g = 0.f, p = 0.f, dot = 0.f;
        for (int j = 0; j < k; ++j) {
            const float gj = to_float(grad_values[tok * k + j]);
            const float pj = SOFTMAX ? to_float(probs[tok * k + j]) : 1.f;
            if (SOFTMAX) dot = fmaf(pj, gj, dot);
            if (indices[tok * k + j] == e) { g += pj * gj; p += pj; }
        }
        grad_logits[i] = from_float<T>(SOFTMAX && p != 0.f ? g - p * dot : g);
    }
}

}  // namespace
}  // namespace fmoe

using namespace fmoe;

namespace {

template <typename T, bool SOFTMAX>
void launch_topk(const void* logits, int64_t n_tokens, int n_expert, int k, void* values, int64_t* indices, cudaStream_t st) {
    if (n_expert <= 32)
        topk_forward_small_kernel<T, SOFTMAX><<<(unsigned)ceil_div(n_tokens, 256), 256, 0, st>>>((const T*)logits, n_tokens, n_expert, k, (T*)values, indices);
    else
        topk_forward_kernel<T, SOFTMAX><<<(unsigned)ceil_div(n_tokens, 8), 256, 0, st>>>((const T*)logits, n_tokens, n_expert, k, (T*)values, indices);
}

template <bool SOFTMAX>
int topk(const void* logits, int64_t n_tokens, int32_t n_expert_total, int32_t k, int32_t dtype, void* values, int64_t* indices,
         cudaStream_t st) {
    FMOE_REQUIRE(n_tokens >= 0 && n_expert_total > 0, "gate_topk: n_tokens=%lld n_expert_total=%d", (long long)n_tokens,
                 n_expert_total);
    FMOE_REQUIRE(k >= 1 && k <= kTopKMax && k <= n_expert_total, "gate_topk: k=%d (1..%d, <= n_expert_total)", k, kTopKMax);
    FMOE_REQUIRE(dtype_size(dtype) > 0, "gate_topk: unknown dtype %d", dtype);
    if (n_tokens == 0) return 0;
    FMOE_REQUIRE(logits && values && indices, "gate_topk: null pointer");
    switch (dtype) {
        case FMOE_F32: launch_topk<float, SOFTMAX>(logits, n_tokens, n_expert_total, k, values, indices, st); break;
        case FMOE_F16: launch_topk<__half, SOFTMAX>(logits, n_tokens, n_expert_total, k, values, indices, st); break;
        default: launch_topk<__nv_bfloat16, SOFTMAX>(logits, n_tokens, n_expert_total, k, values, indices, st); break;
    }
    FMOE_CHECK_LAUNCH();
    return 0;
}

template <bool SOFTMAX>
int topk_backward(const void* grad, const void* probs, const int64_t* indices, int64_t n_tokens, int32_t n_expert_total, int32_t k,
                  int32_t dtype, void* grad_logits, cudaStream_t st) {
    FMOE_REQUIRE(n_tokens >= 0 && n_expert_total > 0 && k >= 1 && k <= kTopKMax, "gate_topk_backward: bad sizes");
    FMOE_REQUIRE(dtype_size(dtype) > 0, "gate_topk_backward: unknown dtype %d", dtype);
    if (n_tokens == 0) return 0;
    FMOE_REQUIRE(grad && indices && grad_logits && (!SOFTMAX || probs), "gate_topk_backward: null pointer");
    const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(n_tokens * n_expert_total, 256), 148 * 16);
    switch (dtype) {
        case FMOE_F32: topk_backward_kernel<float, SOFTMAX><<<blocks, 256, 0, st>>>((const float*)grad, (const float*)probs, indices, n_tokens, n_expert_total, k, (float*)grad_logits); break;
        case FMOE_F16: topk_backward_kernel<__half, SOFTMAX><<<blocks, 256, 0, st>>>((const __half*)grad, (const __half*)probs, indices, n_tokens, n_expert_total, k, (__half*)grad_logits); break;
        default: topk_backward_kernel<__nv_bfloat16, SOFTMAX><<<blocks, 256, 0, st>>>((const __nv_bfloat16*)grad, (const __nv_bfloat16*)probs, indices, n_tokens, n_expert_total, k, (__nv_bfloat16*)grad_logits); break;
    }
    FMOE_CHECK_LAUNCH();
    return 0;
}

}  // namespace

extern "C" int fmoe_gate_topk(const void* logits, int64_t n_tokens, int32_t n_expert_total, int32_t k, int32_t dtype,
                              void* values, int64_t* indices, fmoe_stream_t stream) {
    return topk<false>(logits, n_tokens, n_expert_total, k, dtype, values, indices, (cudaStream_t)stream);
}

extern "C" int fmoe_gate_topk_softmax(const void* logits, int64_t n_tokens, int32_t n_expert_total, int32_t k, int32_t dtype,
                                      void* probs, int64_t* indices, fmoe_stream_t stream) {
    return topk<true>(logits, n_tokens, n_expert_total, k, dtype, probs, indices, (cudaStream_t)stream);
}

extern "C" int fmoe_gate_topk_backward(const void* grad_values, const int64_t* indices, int64_t n_tokens,
                                       int32_t n_expert_total, int32_t k, int32_t dtype, void* grad_logits,
                                       fmoe_stream_t stream) {
    return topk_backward<false>(grad_values, nullptr, indices, n_tokens, n_expert_total, k, dtype, grad_logits, (cudaStream_t)stream);
}

extern "C" int fmoe_gate_topk_softmax_backward(const void* grad_probs, const void* probs, const int64_t* indices,
                                               int64_t n_tokens, int32_t n_expert_total, int32_t k, int32_t dtype,
                                               void* grad_logits, fmoe_stream_t stream) {
    return topk_backward<true>(grad_probs, probs, indices, n_tokens, n_expert_total, k, dtype, grad_logits, (cudaStream_t)stream);
}

// ---- balance loss of the capacity gates ------------------------------------------------------------------------
// Seventeen small torch operators (nine forward, eight backward) on [T, E] values were bound by their launches; two
// kernels forward and one backward here (step of 8192 tokens with a capacity gate, 1024 x 4096, 16 experts: 1054 us
// with the operators, 1014 with the kernels).  One warp per token: lane l holds the experts l, l + 32, ...
namespace fmoe {
namespace {

constexpr int kBalMax = 256, kBalRegs = kBalMax / 32, kBalWarps = 8;

// Threads of the finishing block per expert: what is left of kBalMax when the experts are rounded up to a power of two.
__host__ __device__ constexpr int balance_parts(int n_expert) {
    int w = 1;
    while (w < n_expert) w *= 2;
    return kBalMax / w;
}
// Blocks of the summing kernel: a block per eight tokens, as many as the finishing threads add in 128 steps each, at most 512
// (131072 tokens, 16 experts, loss and gradient: 158 us with 128 blocks and one finishing thread per expert, 86 here).
int balance_blocks(int64_t n_tokens, int n_expert) {
    return (int)std::min<int64_t>(ceil_div(n_tokens, kBalWarps), 128 * std::min(balance_parts(n_expert), 4));
}

// softmax of one row; the lanes' shares of it (zero past n_expert)
template <typename T>
__device__ __forceinline__ void warp_softmax(const T* __restrict__ row, int n_expert, int lane, float (&p)[kBalRegs]) {
    float top = -INFINITY;
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i) {
        const int e = i * 32 + lane;
        p[i] = e < n_expert ? to_float<T>(row[e]) : -INFINITY;
        top = fmaxf(top, p[i]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i) {
        p[i] = i * 32 + lane < n_expert ? expf(p[i] - top) : 0.f;     // (a row with NaN, or of -inf alone, becomes NaN)
        sum += p[i];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float r = 1.f / sum;
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i)
        if (i * 32 + lane < n_expert) p[i] *= r;
}

// partial[block][e]: sum of the probabilities of the block's tokens; counts[block][e]: first choices
template <typename T>
__global__ void __launch_bounds__(kBalWarps * 32)
balance_sums_kernel(const T* __restrict__ logits, const int64_t* __restrict__ first, int64_t stride, int64_t n_tokens,
                    int n_expert, float* __restrict__ partial, int* __restrict__ counts) {
    __shared__ float sums[kBalWarps][kBalMax];
    __shared__ int hist[kBalMax];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) hist[e] = 0;
    __syncthreads();
    float acc[kBalRegs] = {};
    for (int64_t t = (int64_t)blockIdx.x * kBalWarps + warp; t < n_tokens; t += (int64_t)gridDim.x * kBalWarps) {
        float p[kBalRegs];
        warp_softmax<T>(logits + t * n_expert, n_expert, lane, p);
#pragma unroll
        for (int i = 0; i < kBalRegs; ++i) acc[i] += p[i];
        if (lane == 0) {
            const int64_t e = first[t * stride];
            if (e >= 0 && e < n_expert) atomicAdd(hist + (int)e, 1);
        }
    }
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i) sums[warp][i * 32 + lane] = acc[i];
    __syncthreads();
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kBalWarps; ++w) s += sums[w][e];
        partial[(size_t)blockIdx.x * n_expert + e] = s;
        counts[(size_t)blockIdx.x * n_expert + e] = hist[e];
    }
}

__global__ void __launch_bounds__(kBalMax)
balance_finish_kernel(const float* __restrict__ partial, const int* __restrict__ counts, int blocks, int64_t n_tokens,
                      int n_expert, float scale, float* __restrict__ loss, float* __restrict__ share) {
    __shared__ float terms[kBalMax], sums[kBalMax];
    __shared__ int hits[kBalMax];
    const int parts = balance_parts(n_expert), width = kBalMax / parts, e = threadIdx.x % width, part = threadIdx.x / width;
    float s = 0.f;
    int c = 0;
    if (e < n_expert) {
#pragma unroll 8
        for (int b = part; b < blocks; b += parts) {
            s += partial[(size_t)b * n_expert + e];
            c += counts[(size_t)b * n_expert + e];
        }
    }
    sums[threadIdx.x] = s;
    hits[threadIdx.x] = c;
    __syncthreads();
    float term = 0.f;
    if (part == 0 && e < n_expert) {
        for (int q = 1; q < parts; ++q) { s += sums[q * width + e]; c += hits[q * width + e]; }
        const float f = (float)c / (float)n_tokens;
        share[e] = f;
        term = f * (s / (float)n_tokens);
    }
    terms[threadIdx.x] = term;       // (zero for the parts after the first)
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < n_expert; ++i) t += terms[i];
        *loss = t * scale;
    }
}

template <typename T>
__global__ void __launch_bounds__(kBalWarps * 32)
balance_backward_kernel(const T* __restrict__ logits, const float* __restrict__ share, const float* __restrict__ grad_loss,
                        int64_t n_tokens, int n_expert, float scale, T* __restrict__ grad) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * kBalWarps + warp;
    if (t >= n_tokens) return;
    const float g = *grad_loss * scale / (float)n_tokens;
    float p[kBalRegs], w[kBalRegs], dot = 0.f;
    warp_softmax<T>(logits + t * n_expert, n_expert, lane, p);
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i) {
        const int e = i * 32 + lane;
        w[i] = e < n_expert ? g * share[e] : 0.f;
        dot = fmaf(p[i], w[i], dot);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
#pragma unroll
    for (int i = 0; i < kBalRegs; ++i) {
        const int e = i * 32 + lane;
        if (e < n_expert) grad[t * n_expert + e] = from_float<T>(p[i] * (w[i] - dot));
    }
}

int check_balance(const void* logits, int64_t n_tokens, int32_t n_expert, int32_t dtype) {
    FMOE_REQUIRE(n_tokens > 0 && n_expert > 0 && n_expert <= kBalMax, "balance_loss: n_tokens=%lld n_expert=%d (1..%d)",
                 (long long)n_tokens, n_expert, kBalMax);
    FMOE_REQUIRE(dtype_size(dtype) > 0, "balance_loss: unknown dtype %d", dtype);
    FMOE_REQUIRE(logits, "balance_loss: null pointer");
    return 0;
}

}  // namespace
}  // namespace fmoe

extern "C" size_t fmoe_balance_loss_scratch_bytes(int64_t n_tokens, int32_t n_expert) {
    return n_tokens > 0 && n_expert > 0 ? (size_t)balance_blocks(n_tokens, n_expert) * (size_t)n_expert * 8 : 0;
}

extern "C" int fmoe_balance_loss(const void* logits, const int64_t* first_choice, int64_t choice_stride, int64_t n_tokens,
                                 int32_t n_expert, int32_t dtype, float scale, float* loss, float* share, void* scratch,
                                 fmoe_stream_t stream) {
    if (int rc = check_balance(logits, n_tokens, n_expert, dtype)) return rc;
    FMOE_REQUIRE(first_choice && loss && share && scratch, "balance_loss: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = balance_blocks(n_tokens, n_expert);
    float* partial = (float*)scratch;
    int* counts = (int*)scratch + (size_t)blocks * n_expert;
    switch (dtype) {
        case FMOE_F32: balance_sums_kernel<float><<<blocks, kBalWarps * 32, 0, st>>>((const float*)logits, first_choice, choice_stride, n_tokens, n_expert, partial, counts); break;
        case FMOE_F16: balance_sums_kernel<__half><<<blocks, kBalWarps * 32, 0, st>>>((const __half*)logits, first_choice, choice_stride, n_tokens, n_expert, partial, counts); break;
        default: balance_sums_kernel<__nv_bfloat16><<<blocks, kBalWarps * 32, 0, st>>>((const __nv_bfloat16*)logits, first_choice, choice_stride, n_tokens, n_expert, partial, counts); break;
    }
    FMOE_CHECK_LAUNCH();
    balance_finish_kernel<<<1, kBalMax, 0, st>>>(partial, counts, blocks, n_tokens, n_expert, scale, loss, share);
    FMOE_CHECK_LAUNCH();
    return 0;
}

extern "C" int fmoe_balance_loss_backward(const void* logits, const float* share, const float* grad_loss, int64_t n_tokens,
                                          int32_t n_expert, int32_t dtype, float scale, void* grad_logits, fmoe_stream_t stream) {
    if (int rc = check_balance(logits, n_tokens, n_expert, dtype)) return rc;
    FMOE_REQUIRE(share && grad_loss && grad_logits, "balance_loss_backward: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)ceil_div(n_tokens, kBalWarps);
    switch (dtype) {
        case FMOE_F32: balance_backward_kernel<float><<<blocks, kBalWarps * 32, 0, st>>>((const float*)logits, share, grad_loss, n_tokens, n_expert, scale, (float*)grad_logits); break;
        case FMOE_F16: balance_backward_kernel<__half><<<blocks, kBalWarps * 32, 0, st>>>((const __half*)logits, share, grad_loss, n_tokens, n_expert, scale, (__half*)grad_logits); break;
        default: balance_backward_kernel<__nv_bfloat16><<<blocks, kBalWarps * 32, 0, st>>>((const __nv_bfloat16*)logits, share, grad_loss, n_tokens, n_expert, scale, (__nv_bfloat16*)grad_logits); break;
    }
    FMOE_CHECK_LAUNCH();
    return 0;
}
