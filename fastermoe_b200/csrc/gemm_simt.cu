// Grouped expert GEMM on the FFMA pipe (fp32 accumulate, fixed summation order).
//
// This is the path for fp32 tensors, whose parity bound (rtol 1e-5 against an
// fp32 reference) rules out TF32 tensor-core math, and for bf16/fp16 shapes the
// tcgen05 kernels do not take (feature sizes that are not multiples of their
// tiles).  It computes the three products of the reference's fmoe_linear
// (cuda/parallel_linear.cuh:55-161) for all experts in one launch each, reading
// the segment boundaries from device memory.
#include "common.cuh"
#include "gemm.h"
#include <initializer_list>
#include <type_traits>

namespace fmoe {
namespace {

// Tile BM x 128 x 16, 2 * BM threads (BM = 128 or 64), an 8 x 8 micro-tile per thread.  What bounds the kernel
// is issue on the FMA pipe: a 4 x 4 micro-tile reads one shared-memory word per two multiply-adds, so the
// pipe waits for shared memory (19 TFLOP/s); 8 x 8 reads one per four, with 16-byte loads, and the
// multiply-adds go out two columns at a time (fma.rn.f32x2), which leaves issue slots for those loads.  Each
// output is still one fused multiply-add chain in ascending order of the contraction index.  Global loads of
// the next 16 contraction steps are in registers while the current ones are multiplied; two shared-memory
// buffers, one barrier per step.  Measured (4096 rows, 512 x 2048, fp32): 425 us with 4 x 4 micro-tiles, 203 now
// (42 TFLOP/s; the FMA pipe is busy 69 % of the active cycles, the rest is the last wave and the latency of the
// operand loads).  Steps of 8 instead of 16 were slower (230 us): the loads then have too little time to arrive.
constexpr int BN = 128, BK = 16;
constexpr int SEG_CHUNK = 128;      // segment offsets looked at per round by find_tile

// Four consecutive elements as they lie in memory, the ones past `valid` zero: one vector (VEC: 4 divides the extent, so
// a vector is either inside or outside) or element by element.
template <typename T, bool VEC>
struct Raw4 {
    using Word = typename std::conditional<sizeof(T) == 4, float, unsigned short>::type;
    using Vec = typename std::conditional<sizeof(T) == 4, float4, uint2>::type;
    typename std::conditional<VEC, Vec, Word[4]>::type q;
    __device__ __forceinline__ void load(const T* __restrict__ src, int valid) {
        if constexpr (VEC) {
            q = valid > 0 ? __ldg(reinterpret_cast<const Vec*>(src)) : Vec{};
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = i < valid ? __ldg(reinterpret_cast<const Word*>(src) + i) : Word(0);
        }
    }
    __device__ __forceinline__ void get(float* out) const {
        const T* v = reinterpret_cast<const T*>(&q);
#pragma unroll
        for (int i = 0; i < 4; ++i) out[i] = to_float<T>(v[i]);
    }
};

template <typename T, bool VEC>
__device__ __forceinline__ void load4(const T* __restrict__ src, int valid, float* out) {
    Raw4<T, VEC> r;
    r.load(src, valid);
    r.get(out);
}

template <typename T, bool VEC>
__device__ __forceinline__ void store4(T* __restrict__ dst, int valid, const float* v) {
    if (VEC) {
        if (valid <= 0) return;
        if (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            uint2 q;
            T* h = reinterpret_cast<T*>(&q);
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = from_float<T>(v[i]);
            *reinterpret_cast<uint2*>(dst) = q;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < valid) dst[i] = from_float<T>(v[i]);
    }
}

// One operand tile, R rows x BK contraction steps, staged in registers as it lies in memory and then stored in fp32 as
// sm[k][r].  (Converting 16-bit elements when they are staged would wait for the loads before the multiply-adds that
// should cover them.)
// KC: the contraction index is contiguous in memory (element (r, k) at r * ld + k); otherwise the row index is
// (element at k * ld + r).  rows / steps bound the tile: elements outside are zero.
template <typename T, int R, int TH, bool KC, bool VEC>
struct Operand {
    static constexpr int NV = R * BK / 4 / TH;      // vectors of four per thread
    static constexpr int LD = R + 4;
    Raw4<T, VEC> stage[NV];
    __device__ __forceinline__ void load(const T* __restrict__ src, int64_t ld, int rows, int steps) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = threadIdx.x + i * TH;
            if (KC) {
                const int r = v / (BK / 4), k = (v % (BK / 4)) * 4;
                stage[i].load(src + (int64_t)r * ld + k, r < rows ? steps - k : 0);
            } else {
                const int k = v / (R / 4), r = (v % (R / 4)) * 4;
                stage[i].load(src + (int64_t)k * ld + r, k < steps ? rows - r : 0);
            }
        }
    }
    __device__ __forceinline__ void put(float (*sm)[LD]) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = threadIdx.x + i * TH;
            float f[4];
            stage[i].get(f);
            if (KC) {
                const int r = v / (BK / 4), k = (v % (BK / 4)) * 4;
#pragma unroll
                for (int j = 0; j < 4; ++j) sm[k + j][r] = f[j];
            } else {
                const int k = v / (R / 4), r = (v % (R / 4)) * 4;
                *reinterpret_cast<float4*>(&sm[k][r]) = make_float4(f[0], f[1], f[2], f[3]);
            }
        }
    }
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 fma_pair(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// The block's product: acc[i][j] = sum_k A(row_i, k) B(col_2j.., k), rows ty*4 + {0..3} and BM/2 + ty*4 + {0..3},
// columns tx*4 + {0..3} and 64 + tx*4 + {0..3}.  A warp covers 4 x 8 threads of the 2D arrangement.
template <typename T, int BM, bool A_KC, bool B_KC, bool VEC>
struct Block {
    static constexpr int TH = 2 * BM;
    using OpA = Operand<T, BM, TH, A_KC, VEC>;
    using OpB = Operand<T, BN, TH, B_KC, VEC>;
    struct Smem {
        float a[2][BK][OpA::LD];
        float b[2][BK][OpB::LD];
    };
    __device__ static int ty() { return (threadIdx.x >> 6) * 4 + ((threadIdx.x & 31) >> 3); }
    __device__ static int tx() { return ((threadIdx.x >> 5) & 1) * 8 + (threadIdx.x & 7); }

    __device__ __forceinline__ static void run(Smem& sm, const T* a, int64_t lda, int rows, const T* b, int64_t ldb, int cols,
                                               int64_t kdim, f32x2 (&acc)[8][4]) {
        OpA oa;
        OpB ob;
        const int r0 = ty() * 4, c0 = tx() * 4;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        if (kdim <= 0) return;
        const int64_t step_a = A_KC ? BK : BK * lda, step_b = B_KC ? BK : BK * ldb;
        int steps = (int)min((int64_t)BK, kdim);
        oa.load(a, lda, rows, steps);
        ob.load(b, ldb, cols, steps);
        oa.put(sm.a[0]);
        ob.put(sm.b[0]);
        __syncthreads();
        int buf = 0;
        for (int64_t k0 = 0; k0 < kdim; k0 += BK) {
            const bool more = k0 + BK < kdim;
            if (more) {
                a += step_a;
                b += step_b;
                steps = (int)min((int64_t)BK, kdim - k0 - BK);
                oa.load(a, lda, rows, steps);
                ob.load(b, ldb, cols, steps);
            }
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(&sm.a[buf][k][r0]);
                const float4 a1 = *reinterpret_cast<const float4*>(&sm.a[buf][k][r0 + BM / 2]);
                const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&sm.b[buf][k][c0]);
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&sm.b[buf][k][c0 + BN / 2]);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f32x2 ai = pair(av[i], av[i]);
                    acc[i][0] = fma_pair(ai, b0.x, acc[i][0]);
                    acc[i][1] = fma_pair(ai, b0.y, acc[i][1]);
                    acc[i][2] = fma_pair(ai, b1.x, acc[i][2]);
                    acc[i][3] = fma_pair(ai, b1.y, acc[i][3]);
                }
            }
            if (more) {
                oa.put(sm.a[buf ^ 1]);
                ob.put(sm.b[buf ^ 1]);
            }
            __syncthreads();
            buf ^= 1;
        }
    }
};

struct TileMap {
    int expert;
    int64_t row0;  // first row of the tile (absolute)
    int rows;      // valid rows in the tile
};

// Maps a linear m-tile index to (expert, rows) by walking the segment table (ranges are clamped
// to the buffer's n_rows rows and to run forwards, see safe_seg_range).  The block fetches the offsets together:
// one thread after another walking them in global memory costs a memory latency per expert.
__device__ __forceinline__ bool find_tile(const int64_t* __restrict__ off, const HostSegs& hs, int n_expert, int bm,
                                          int64_t n_rows, int64_t tile, int64_t (*seg)[2], TileMap& tm) {
    int64_t acc = 0, prev_hi = 0;
    for (int e0 = 0; e0 < n_expert; e0 += SEG_CHUNK) {
        const int n = min(SEG_CHUNK, n_expert - e0);
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            seg[i][0] = hs.n ? (int64_t)hs.lo[e0 + i] : off[e0 + i];
            seg[i][1] = hs.n ? (int64_t)hs.hi[e0 + i] : off[e0 + i + 1];
        }
        __syncthreads();
        for (int i = 0; i < n; ++i) {
            const int64_t lo = min(max(seg[i][0], prev_hi), n_rows), hi = min(max(seg[i][1], lo), n_rows);
            prev_hi = hi;
            const int64_t nt = (hi - lo + bm - 1) / bm;
            if (tile < acc + nt) {
                const int64_t r0 = lo + (tile - acc) * bm;
                tm.expert = e0 + i;
                tm.row0 = r0;
                tm.rows = (int)min((int64_t)bm, hi - r0);
                return true;
            }
            acc += nt;
        }
    }
    return false;
}

__device__ __forceinline__ void unpair(const f32x2 (&acc)[4], float* v) {
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2 * j]), "=f"(v[2 * j + 1]) : "l"(acc[j]));
}

// MODE 0: Y[m,n]  = sum_k X[m,k] W[e][n,k] (+bias, activation)      rows ragged
// MODE 1: dX[m,k] = sum_n dY[m,n] W[e][n,k] (* saved activation derivative)  rows ragged
template <typename T, int MODE, int BM, bool VEC>
__global__ void __launch_bounds__(2 * BM, 256 / BM)
rows_gemm_kernel(const T* __restrict__ a, const T* __restrict__ w, const T* __restrict__ bias,
                 const int64_t* __restrict__ off, const __grid_constant__ HostSegs hs, T* __restrict__ c,
                 T* __restrict__ pre_out, const T* __restrict__ act_pre, int n_expert, int64_t n_rows, int64_t in_feat,
                 int64_t out_feat, int act) {
    using B = Block<T, BM, true, MODE == 0, VEC>;
    __shared__ __align__(16) typename B::Smem sm;
    static_assert(sizeof(sm) >= SEG_CHUNK * 2 * sizeof(int64_t), "the segment table is read through the operand buffers");
    TileMap tm;
    if (!find_tile(off, hs, n_expert, BM, n_rows, blockIdx.x, reinterpret_cast<int64_t(*)[2]>(&sm), tm)) return;
    __syncthreads();
    const int64_t kdim = MODE == 0 ? in_feat : out_feat;  // contraction length
    const int64_t ndim = MODE == 0 ? out_feat : in_feat;  // output columns
    const int64_t n0 = (int64_t)blockIdx.y * BN;
    const int n_valid = (int)min((int64_t)BN, ndim - n0);
    const T* wp = w + (int64_t)tm.expert * in_feat * out_feat;
    f32x2 acc[8][4];
    // B(k, n): MODE 0 -> W[n0+n, k] (k contiguous); MODE 1 -> W[k, n0+n] (n contiguous); rows of in_feat elements either way
    B::run(sm, a + tm.row0 * kdim, kdim, tm.rows, MODE == 0 ? wp + n0 * in_feat : wp + n0, in_feat, n_valid, kdim, acc);
    // One copy of the epilogue for the eight rows of a thread, which take their turn in acc[0].  (Unrolled, 64 copies of
    // erff and of the derivative's expf are fetched by a block that runs each once: 128 rows of two experts, 64 x 256,
    // fp32 took 45 us, 18 here; 4096 rows of four, 512 x 2048: 239 and 221.)
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
        const int r = (i >> 2) * (BM / 2) + B::ty() * 4 + (i & 3);
        const int64_t row = (tm.row0 + r) * ndim;
        float v[8];
        unpair(acc[0], v);
#pragma unroll
        for (int u = 0; u < 7; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[u][j] = acc[u + 1][j];
        if (r >= tm.rows) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int cidx = h * (BN / 2) + B::tx() * 4, valid = n_valid - cidx;
            if (valid <= 0) continue;
            const int64_t col = n0 + cidx;
            float* q = v + 4 * h;
            if (MODE == 0) {
                if (bias) {
                    float bv[4];
                    load4<T, VEC>(bias + (int64_t)tm.expert * out_feat + col, valid, bv);
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[j] += bv[j];
                }
                if (pre_out && saves_derivative(act)) {
                    float g[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) g[j] = act_grad(q[j], act);
                    store4<T, VEC>(pre_out + row + col, valid, g);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = apply_act(q[j], act);
            } else if (act_pre) {
                float s[4];
                load4<T, VEC>(act_pre + row + col, valid, s);
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] *= saved_act_grad(s[j], act);
            }
            store4<T, VEC>(c + row + col, valid, q);
        }
    }
}

// dW[e][n,k] = sum_{m in seg e} dY[m,n] X[m,k]     grid (n tiles, k tiles, E)
template <typename T, int BM, bool VEC>
__global__ void __launch_bounds__(2 * BM, 256 / BM)
wgrad_kernel(const T* __restrict__ dy, const T* __restrict__ x, const int64_t* __restrict__ off,
             const __grid_constant__ HostSegs hs, T* __restrict__ dw, int64_t n_rows, int64_t in_feat, int64_t out_feat,
             int accumulate) {
    using B = Block<T, BM, false, false, VEC>;
    __shared__ __align__(16) typename B::Smem sm;
    const int e = blockIdx.z;
    int64_t lo, hi;
    safe_seg_range(off, hs, e, n_rows, lo, hi);
    const int64_t n0 = (int64_t)blockIdx.x * BM, k0 = (int64_t)blockIdx.y * BN;
    const int nv = (int)min((int64_t)BM, out_feat - n0), kv = (int)min((int64_t)BN, in_feat - k0);
    f32x2 acc[8][4];
    B::run(sm, dy + lo * out_feat + n0, out_feat, nv, x + lo * in_feat + k0, in_feat, kv, hi - lo, acc);
    T* out = dw + (int64_t)e * in_feat * out_feat;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = (i >> 2) * (BM / 2) + B::ty() * 4 + (i & 3);
        if (r >= nv) continue;
        float v[8];
        unpair(acc[i], v);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int cidx = h * (BN / 2) + B::tx() * 4, valid = kv - cidx;
            if (valid <= 0) continue;
            T* o = out + (n0 + r) * in_feat + k0 + cidx;
            float* q = v + 4 * h;
            if (accumulate) {
                float old[4];
                load4<T, VEC>(o, valid, old);
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] += old[j];
            }
            store4<T, VEC>(o, valid, q);
        }
    }
}

// out[e][n] = sum_{m in seg e} rows[m,n] (bias gradients).  Block: 32 columns x 8 row lanes, eight rows in flight per lane.
template <typename T>
__global__ void __launch_bounds__(256)
colsum_kernel(const T* __restrict__ rows, const int64_t* __restrict__ off, const __grid_constant__ HostSegs hs,
              T* __restrict__ out, int64_t n_rows, int64_t n_cols, int accumulate) {
    __shared__ float red[8][33];
    const int e = blockIdx.y;
    const int cx = threadIdx.x % 32, ry = threadIdx.x / 32;
    const int64_t col = (int64_t)blockIdx.x * 32 + cx;
    int64_t lo, hi;
    safe_seg_range(off, hs, e, n_rows, lo, hi);
    float s = 0.f;
    if (col < n_cols) {
        int64_t m = lo + ry;
        for (; m + 56 < hi; m += 64) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = to_float<T>(rows[(m + 8 * u) * n_cols + col]);
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        for (; m < hi; m += 8) s += to_float<T>(rows[m * n_cols + col]);
    }
    red[ry][cx] = s;
    __syncthreads();
    if (ry == 0 && col < n_cols) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += red[i][cx];
        const int64_t o = (int64_t)e * n_cols + col;
        if (accumulate) t += to_float<T>(out[o]);
        out[o] = from_float<T>(t);
    }
}

const HostSegs kNoSegs = {};

// Vectors of four elements: both widths and every operand on such a boundary.
template <typename T>
bool vec4_ok(int64_t in_feat, int64_t out_feat, std::initializer_list<const void*> ptrs) {
    if (in_feat % 4 || out_feat % 4) return false;
    for (const void* p : ptrs)
        if ((uintptr_t)p & (4 * sizeof(T) - 1)) return false;
    return true;
}

// 128-row tiles (two blocks per SM) when they fill the chip, 64-row tiles (four per SM) below that: with 136 tall
// tiles (4096 rows of four experts, 512 columns, contraction 2048) the 64-row form took 220 us, the tall one 278.
bool tall_tiles(int64_t tiles128) { return tiles128 >= 2 * (int64_t)sm_count(); }

template <typename T, int MODE>
int rows_gemm(const void* x, const void* w, const void* bias, const int64_t* seg, const HostSegs& hs, void* y, void* pre,
              const void* act_pre, int n_expert, int64_t n_rows, int64_t in_feat, int64_t out_feat, int act, cudaStream_t st) {
    const int64_t n_tiles = ceil_div(MODE == 0 ? out_feat : in_feat, BN);
    const bool tall = tall_tiles(ceil_div(n_rows, 128) * n_tiles);
    const bool vec = vec4_ok<T>(in_feat, out_feat, {x, w, bias, y, pre, act_pre});
    auto kern = tall ? (vec ? rows_gemm_kernel<T, MODE, 128, true> : rows_gemm_kernel<T, MODE, 128, false>)
                     : (vec ? rows_gemm_kernel<T, MODE, 64, true> : rows_gemm_kernel<T, MODE, 64, false>);
    const int bm = tall ? 128 : 64;
    dim3 grid((unsigned)(ceil_div(n_rows, bm) + n_expert), (unsigned)n_tiles);
    kern<<<grid, 2 * bm, 0, st>>>((const T*)x, (const T*)w, (const T*)bias, seg, hs, (T*)y, (T*)pre, (const T*)act_pre,
                                  n_expert, n_rows, in_feat, out_feat, act);
    FMOE_CHECK_LAUNCH();
    return 0;
}

template <typename T>
int forward_t(const LinearArgs& a, cudaStream_t st) {
    return rows_gemm<T, 0>(a.x, a.weight, a.bias, a.seg_offsets, a.host_segs ? *a.host_segs : kNoSegs, a.y, a.pre_act, nullptr,
                           a.n_expert, a.n_rows, a.in_feat, a.out_feat, a.activation, st);
}

template <typename T>
int colsum(const void* rows, const LinearBwdArgs& a, const HostSegs& hs, void* out, int64_t n_cols, int accumulate, cudaStream_t st) {
    dim3 grid((unsigned)ceil_div(n_cols, 32), (unsigned)a.n_expert);
    colsum_kernel<T><<<grid, 256, 0, st>>>((const T*)rows, a.seg_offsets, hs, (T*)out, a.n_rows, n_cols, accumulate);
    FMOE_CHECK_LAUNCH();
    return 0;
}

template <typename T>
int backward_t(const LinearBwdArgs& a, cudaStream_t st) {
    const HostSegs& hs = a.host_segs ? *a.host_segs : kNoSegs;
    if (a.grad_x && a.n_rows > 0) {
        if (int rc = rows_gemm<T, 1>(a.grad_y, a.weight, nullptr, a.seg_offsets, hs, a.grad_x, nullptr, a.act_pre, a.n_expert,
                                     a.n_rows, a.in_feat, a.out_feat, a.activation, st)) return rc;
    }
    if (a.grad_w) {
        const int64_t k_tiles = ceil_div(a.in_feat, BN);
        const bool tall = tall_tiles(ceil_div(a.out_feat, 128) * k_tiles * a.n_expert);
        const bool vec = vec4_ok<T>(a.in_feat, a.out_feat, {a.grad_y, a.x, a.grad_w});
        auto kern = tall ? (vec ? wgrad_kernel<T, 128, true> : wgrad_kernel<T, 128, false>)
                         : (vec ? wgrad_kernel<T, 64, true> : wgrad_kernel<T, 64, false>);
        const int bm = tall ? 128 : 64;
        dim3 grid((unsigned)ceil_div(a.out_feat, bm), (unsigned)k_tiles, (unsigned)a.n_expert);
        kern<<<grid, 2 * bm, 0, st>>>((const T*)a.grad_y, (const T*)a.x, a.seg_offsets, hs, (T*)a.grad_w, a.n_rows, a.in_feat,
                                      a.out_feat, a.accumulate);
        FMOE_CHECK_LAUNCH();
    }
    if (a.grad_b) {
        if (int rc = colsum<T>(a.grad_y, a, hs, a.grad_b, a.out_feat, a.accumulate, st)) return rc;
    }
    if (a.grad_x_colsum) return colsum<T>(a.grad_x, a, hs, a.grad_x_colsum, a.in_feat, 0, st);
    return 0;
}

}  // namespace

int simt_linear_forward(const LinearArgs& a, cudaStream_t st) {
    if (a.n_rows == 0) return 0;
    switch (a.dtype) {
        case FMOE_F32: return forward_t<float>(a, st);
        case FMOE_F16: return forward_t<__half>(a, st);
        default: return forward_t<__nv_bfloat16>(a, st);
    }
}

int simt_linear_backward(const LinearBwdArgs& a, cudaStream_t st) {
    switch (a.dtype) {
        case FMOE_F32: return backward_t<float>(a, st);
        case FMOE_F16: return backward_t<__half>(a, st);
        default: return backward_t<__nv_bfloat16>(a, st);
    }
}

}  // namespace fmoe
