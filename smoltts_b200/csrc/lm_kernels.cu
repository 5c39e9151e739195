// Hybrid language-model engine (sm_100a): ragged-batch step over a paged key/value pool and per-sequence recurrent
// state slots.  See include/smoltts_b200_lm.h for what every entry point takes and returns.
//
// Precision: the residual stream, all norms, attention scores / softmax weights and the whole recurrence run in fp32.
// T (bf16 or float) is the element type of matrices, of the inputs of the matrix products and of the key/value pool;
// every matrix product accumulates in fp32 and writes fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <string>
#include <vector>

#include "../../include/smoltts_b200_lm.h"
#include "common.cuh"
#include "f32_tile.cuh"
#include "sampler.cuh"
#include "tmap_host.h"
#include "umma.cuh"

#define SMOL_OK 0
#define SMOL_ERR_INVALID (-1)
#define SMOL_ERR_UNBOUND (-2)
#define SMOL_ERR_CUDA (-3)
#define SMOL_ERR_UNSUPPORTED (-4)
#define SMOL_ERR_CAPACITY (-5)

namespace smol {
namespace lm {

template <class T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <class T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

// Sum over the block; every thread gets the result.  `red` holds 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        float t = l < nw ? red[l] : 0.0f;
        t = warp_sum(t);
        if (l == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

// A row in registers as 16-byte pieces, V per thread.  LONE: the row has a block of its own, a piece per thread, and the warps' sums meet behind one barrier;
// otherwise the row has one warp and needs none.  Both add in the same order -- the sums of 32 pieces side by side, one after the other --, so a row's bits do not
// depend on how many rows a step has.
template <int V, bool LONE>
struct RowPieces {
    __device__ static __forceinline__ int row() { return LONE ? (int)blockIdx.x : (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); }
    __device__ static __forceinline__ int column(int i) { return 4 * (LONE ? (int)threadIdx.x : (int)(threadIdx.x & 31) + 32 * i); }
    // `red`: 16 floats that no other sum of the kernel uses
    __device__ static __forceinline__ float sum(float (&v)[V], float* red) {
#pragma unroll
        for (int x = 16; x > 0; x >>= 1)
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], x);
        if (!LONE) {
#pragma unroll
            for (int i = 1; i < V; ++i) v[0] += v[i];
            return v[0];
        }
        const int nw = (int)blockDim.x >> 5;
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v[0];
        __syncthreads();
        float t = red[0];
        for (int i = 1; i < nw; ++i) t += red[i];
        return t;
    }
};
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y));
}
__device__ __forceinline__ float squares(const float4 v) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))); }
template <class T> __device__ __forceinline__ void store4(T* p, float a, float b, float c, float d);
template <> __device__ __forceinline__ void store4<float>(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
template <> __device__ __forceinline__ void store4<bf16>(bf16* p, float a, float b, float c, float d) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
// v * r * (off + w)
template <class T>
__device__ __forceinline__ void store_normed(T* p, const float4 v, float r, float off, const float4 w) {
    store4<T>(p, v.x * r * (off + w.x), v.y * r * (off + w.y), v.z * r * (off + w.z), v.w * r * (off + w.w));
}

// ---------------------------------------------------------------------------------------------------------------------
// Embedding: x[t] = embed[token[t]] * scale, then the first layer's norm -> hn.  The norms of the sandwich block multiply
// by woff + w: woff = 1 for one-plus weight vectors, 0 for plain ones.
template <class T>
__global__ void embed_norm_kernel(const int32_t* __restrict__ tokens, const T* __restrict__ embed, float scale, int D, int vocab,
                                  const float* __restrict__ wn, float eps, float* __restrict__ x, T* __restrict__ hn, const float woff) {
    dep_wait();
    dep_go();
    __shared__ float red[33];
    const int t = blockIdx.x;
    int tok = tokens[t];
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    const T* e = embed + (size_t)tok * D;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        const float v = to_f<T>(e[c]) * scale;
        x[(size_t)t * D + c] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float r = 1.0f / sqrtf(ss / (float)D + eps);
    for (int c = threadIdx.x; c < D; c += blockDim.x) hn[(size_t)t * D + c] = from_f<T>(x[(size_t)t * D + c] * r * (woff + wn[c]));
}

// The same with the row in registers (D a multiple of 4, aligned rows): see add_norm_vec_kernel.  (2048 rows of 768: 6 us as against 11.)
template <class T, int V, bool LONE>
__global__ void __launch_bounds__(LONE ? 512 : 128) embed_norm_vec_kernel(const int32_t* __restrict__ tokens, const T* __restrict__ embed, float scale, int D, int vocab,
                                                                          const float* __restrict__ wn, float eps, float* __restrict__ x, T* __restrict__ hn, const float woff, int rows) {
    dep_wait();
    dep_go();
    using R = RowPieces<V, LONE>;
    __shared__ float red[16];
    const int t = R::row();
    if (t >= rows) return;
    int tok = tokens[t];
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    const T* e = embed + (size_t)tok * D;
    const size_t o = (size_t)t * D;
    float4 v[V];
    float ss[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = R::column(i) < D ? load4(e + R::column(i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        v[i] = make_float4(v[i].x * scale, v[i].y * scale, v[i].z * scale, v[i].w * scale);
        if (R::column(i) < D) *reinterpret_cast<float4*>(x + o + R::column(i)) = v[i];
        ss[i] = squares(v[i]);
    }
    const float r = 1.0f / sqrtf(R::sum(ss, red) / (float)D + eps);
#pragma unroll
    for (int i = 0; i < V; ++i)
        if (R::column(i) < D) store_normed<T>(hn + o + R::column(i), v[i], r, woff, load4(wn + R::column(i)));
}

// RMS norm of selected rows -> T.  rows == nullptr: row r of the output is row r of the input.
template <class T>
__global__ void norm_rows_kernel(const float* __restrict__ x, const int32_t* __restrict__ rows, const float* __restrict__ w, float eps,
                                 int D, T* __restrict__ out, const float woff) {
    dep_wait();
    dep_go();
    __shared__ float red[33];
    const int r = blockIdx.x;
    const float* xr = x + (size_t)(rows ? rows[r] : r) * D;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < D; c += blockDim.x) ss += xr[c] * xr[c];
    ss = block_sum(ss, red);
    const float s = 1.0f / sqrtf(ss / (float)D + eps);
    for (int c = threadIdx.x; c < D; c += blockDim.x) out[(size_t)r * D + c] = from_f<T>(xr[c] * s * (woff + w[c]));
}

template <class T, int V, bool LONE>
__global__ void __launch_bounds__(LONE ? 512 : 128) norm_rows_vec_kernel(const float* __restrict__ x, const int32_t* __restrict__ rows, const float* __restrict__ w, float eps,
                                                                         int D, T* __restrict__ out, const float woff, int n_rows) {
    dep_wait();
    dep_go();
    using R = RowPieces<V, LONE>;
    __shared__ float red[16];
    const int r = R::row();
    if (r >= n_rows) return;
    const float* xr = x + (size_t)(rows ? rows[r] : r) * D;
    float4 v[V];
    float ss[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = R::column(i) < D ? load4(xr + R::column(i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < V; ++i) ss[i] = squares(v[i]);
    const float f = 1.0f / sqrtf(R::sum(ss, red) / (float)D + eps);
#pragma unroll
    for (int i = 0; i < V; ++i)
        if (R::column(i) < D) store_normed<T>(out + (size_t)r * D + R::column(i), v[i], f, woff, load4(w + R::column(i)));
}

// End of a sublayer fused with the start of the next one:
//   x <- x + ls * (y / rms(y) * (woff + wb));   hn <- x / rms(x) * (woff + wn)     (wn == nullptr: no next norm)
// yb != nullptr: a bias [D] joins y first (the output projection's).  rs.yp != nullptr: y is instead the routed experts'
// weighted sum, taken here (hin: the sublayer's input, which identity outputs hand on).  One block per row; the new row
// is kept in shared memory between the two passes.
constexpr int kRowRegs = 8;   // add_norm keeps a row in registers when it has at most 8 elements per thread

// The sublayer's output of a routed feed-forward, summed on the fly by the norm kernel that follows it: for the `top`
// choices k of a token (ascending), weight[k] * (row slot_of[k] of the experts' outputs, or the token's input itself where
// slot_of[k] < 0: an identity output).  sel_w == nullptr: every weight is 1 (the weights went into the experts' inputs).
struct RoutedSum {
    const float* yp;              // nullptr: the sublayer's output is y
    const int32_t* slot_of;
    const float* sel_w;
    int top;
};

template <class T>
__global__ void add_norm_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ wb,
                                const float* __restrict__ ls, const float* __restrict__ wn, float eps, int D, T* __restrict__ hn,
                                const float woff, const float* __restrict__ yb, const RoutedSum rs, const T* hin) {
    dep_wait();
    dep_go();
    extern __shared__ float row[];
    __shared__ float red[33];
    const size_t o = (size_t)blockIdx.x * D;
    auto y_at = [&](int c) -> float {
        if (!rs.yp) return y[o + c] + (yb ? yb[c] : 0.0f);
        float acc = 0.0f;
        for (int k = 0; k < rs.top; ++k) {
            const int slot = rs.slot_of[(size_t)blockIdx.x * rs.top + k];
            const float v = slot >= 0 ? rs.yp[(size_t)slot * D + c] : to_f<T>(hin[o + c]);
            acc = fmaf(rs.sel_w ? rs.sel_w[(size_t)blockIdx.x * rs.top + k] : 1.0f, v, acc);
        }
        return acc;
    };
    if (D <= (int)blockDim.x * kRowRegs) {
        // every operand is loaded before the first reduction: the kernel waits for global memory once
        float yv[kRowRegs], xv[kRowRegs], lv[kRowRegs], bv[kRowRegs], nv[kRowRegs];
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < kRowRegs; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            const bool in = c < D;
            yv[i] = in ? y_at(c) : 0.0f;
            xv[i] = in ? x[o + c] : 0.0f;
            lv[i] = in ? ls[c] : 0.0f;
            bv[i] = in ? wb[c] : 0.0f;
            nv[i] = (in && wn) ? wn[c] : 0.0f;
            ss += yv[i] * yv[i];
        }
        ss = block_sum(ss, red);
        const float r = 1.0f / sqrtf(ss / (float)D + eps);
        float s2 = 0.0f;
#pragma unroll
        for (int i = 0; i < kRowRegs; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            const float v = xv[i] + lv[i] * (yv[i] * r * (woff + bv[i]));
            xv[i] = v;
            if (c < D) {
                x[o + c] = v;
                s2 += v * v;
            }
        }
        if (!wn) return;
        s2 = block_sum(s2, red);
        const float r2 = 1.0f / sqrtf(s2 / (float)D + eps);
#pragma unroll
        for (int i = 0; i < kRowRegs; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            if (c < D) hn[o + c] = from_f<T>(xv[i] * r2 * (woff + nv[i]));
        }
        return;
    }
    float ss = 0.0f;
    float* ysum = row;            // the sublayer's output of this row, then the new row
    for (int c = threadIdx.x; c < D; c += blockDim.x) { const float v = y_at(c); ysum[c] = v; ss += v * v; }
    ss = block_sum(ss, red);
    const float r = 1.0f / sqrtf(ss / (float)D + eps);
    float s2 = 0.0f;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        const float v = x[o + c] + ls[c] * (ysum[c] * r * (woff + wb[c]));
        x[o + c] = v;
        row[c] = v;
        s2 += v * v;
    }
    if (!wn) return;
    s2 = block_sum(s2, red);
    const float r2 = 1.0f / sqrtf(s2 / (float)D + eps);
    for (int c = threadIdx.x; c < D; c += blockDim.x) hn[o + c] = from_f<T>(row[c] * r2 * (woff + wn[c]));
}

// The same with the rows as 16-byte pieces in registers (D a multiple of 4 up to 2048, aligned rows).  What bounds it is waiting: for the rows (one round of loads),
// then for the two sums.  Many rows: a warp per row, so that a row's sums are shuffles and an SM's rows are all in flight at once (2048 rows of 768: 7 us as against
// 13 for a block of 128 threads per row, 4-byte loads and six barriers).  Few rows: a block per row, a piece per thread, one barrier per sum, and the weights -- no
// kernel of a step writes them, and the step's first kernel has waited for what did -- loaded before the wait for the kernel in front (one row: 1.7 as against 4.5).
template <class T, int V, bool LONE>
__global__ void __launch_bounds__(LONE ? 512 : 128) add_norm_vec_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ wb, const float* __restrict__ ls,
                                                                        const float* __restrict__ wn, float eps, int D, T* __restrict__ hn, const float woff,
                                                                        const float* __restrict__ yb, const RoutedSum rs, const T* hin, int rows) {
    using R = RowPieces<V, LONE>;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 early[4] = {none, none, none, none};
    if (LONE && R::column(0) < D) {
        early[0] = load4(ls + R::column(0));
        early[1] = load4(wb + R::column(0));
        if (wn) early[2] = load4(wn + R::column(0));
        if (yb) early[3] = load4(yb + R::column(0));
    }
    dep_wait();
    dep_go();
    __shared__ float red[2][16];
    const int t = R::row();
    if (t >= rows) return;
    const size_t o = (size_t)t * D;
    float4 xv[V], yv[V];
    float ss[V], s2[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int c = R::column(i);
        const bool in = c < D;
        xv[i] = in ? load4(x + o + c) : none;
        yv[i] = none;
        if (!in) continue;
        if (!rs.yp) yv[i] = load4(y + o + c);
    }
    if (rs.yp) {
        for (int k = 0; k < rs.top; ++k) {
            const int slot = rs.slot_of[(size_t)t * rs.top + k];
            const float w = rs.sel_w ? rs.sel_w[(size_t)t * rs.top + k] : 1.0f;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const int c = R::column(i);
                if (c >= D) continue;
                const float4 v = slot >= 0 ? load4(rs.yp + (size_t)slot * D + c) : load4(hin + o + c);
                yv[i] = make_float4(fmaf(w, v.x, yv[i].x), fmaf(w, v.y, yv[i].y), fmaf(w, v.z, yv[i].z), fmaf(w, v.w, yv[i].w));
            }
        }
    } else if (yb) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const float4 v = LONE ? early[3] : R::column(i) < D ? load4(yb + R::column(i)) : none;
            yv[i] = make_float4(yv[i].x + v.x, yv[i].y + v.y, yv[i].z + v.z, yv[i].w + v.w);
        }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) ss[i] = squares(yv[i]);
    const float r = 1.0f / sqrtf(R::sum(ss, red[0]) / (float)D + eps);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int c = R::column(i);
        s2[i] = 0.0f;
        if (c >= D) continue;
        const float4 l = LONE ? early[0] : load4(ls + c), b = LONE ? early[1] : load4(wb + c), u = yv[i];
        float4& v = xv[i];
        v.x += l.x * (u.x * r * (woff + b.x));
        v.y += l.y * (u.y * r * (woff + b.y));
        v.z += l.z * (u.z * r * (woff + b.z));
        v.w += l.w * (u.w * r * (woff + b.w));
        *reinterpret_cast<float4*>(x + o + c) = v;
        s2[i] = squares(v);
    }
    if (!wn) return;
    const float r2 = 1.0f / sqrtf(R::sum(s2, red[1]) / (float)D + eps);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int c = R::column(i);
        if (c < D) store_normed<T>(hn + o + c, xv[i], r2, woff, LONE ? early[2] : load4(wn + c));
    }
}
constexpr int kRowPiecesMax = 2048;      // widths up to which rows stay in registers
constexpr int kWarpRows = 512;           // rows from which a warp has a row of its own

// Three sums over the block at once; every thread gets the results.  `red` holds 3 x 33 floats.
__device__ __forceinline__ void block_sum3(float& a, float& b, float& c, float (*red)[33]) {
    a = warp_sum(a);
    b = warp_sum(b);
    c = warp_sum(c);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    if (l == 0) { red[0][w] = a; red[1][w] = b; red[2][w] = c; }
    __syncthreads();
    if (w < 3) {
        float t = l < nw ? red[w][l] : 0.0f;
        t = warp_sum(t);
        if (l == 0) red[w][32] = t;
    }
    __syncthreads();
    a = red[0][32];
    b = red[1][32];
    c = red[2][32];
}

// PolyNorm: out = a z/rms(z) + b z^2/rms(z^2) + c z^3/rms(z^3) + e over a token's feed-forward vector.  The three sums
// are taken in one pass and reduced together; rows whose length is a multiple of 4 move as 16-byte pieces.
constexpr int kPolynormThreads = 256;
template <class T>
__global__ void polynorm_kernel(const float* __restrict__ z, const float* __restrict__ coef, float eps, int F, T* __restrict__ out) {
    dep_wait();
    dep_go();
    __shared__ float red[3][33];
    const size_t o = (size_t)blockIdx.x * F;
    const bool vec = F % 4 == 0;
    float s2 = 0.0f, s4 = 0.0f, s6 = 0.0f;
    auto add = [&](float v) {
        const float v2 = v * v;
        s2 += v2;
        s4 += v2 * v2;
        s6 += v2 * v2 * v2;
    };
    if (vec) {
        for (int c = threadIdx.x * 4; c < F; c += blockDim.x * 4) {
            const float4 v = *reinterpret_cast<const float4*>(z + o + c);
            add(v.x); add(v.y); add(v.z); add(v.w);
        }
    } else {
        for (int c = threadIdx.x; c < F; c += blockDim.x) add(z[o + c]);
    }
    block_sum3(s2, s4, s6, red);
    const float a = coef[0] / sqrtf(s2 / (float)F + eps), b = coef[1] / sqrtf(s4 / (float)F + eps),
                cc = coef[2] / sqrtf(s6 / (float)F + eps), e = coef[3];
    auto f = [&](float v) { return a * v + b * v * v + cc * v * v * v + e; };
    if (vec) {
        for (int c = threadIdx.x * 4; c < F; c += blockDim.x * 4) {
            const float4 v = *reinterpret_cast<const float4*>(z + o + c);
            store4<T>(out + o + c, f(v.x), f(v.y), f(v.z), f(v.w));
        }
    } else {
        for (int c = threadIdx.x; c < F; c += blockDim.x) out[o + c] = from_f<T>(f(z[o + c]));
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Where the operands of a matrix product live beyond the plain case (a [M, K], w [N, K], y [M, N], all contiguous).
//  - lda / ldy: row strides of a and y; blockIdx.z is a batch index with the strides sa / sw / sy (one product per head).
//  - grouped rows (tile_group != nullptr): the rows are sorted by group (expert), group g owning rows seg[g] .. seg[g+1]-1
//    and the weight matrix w + g * sw; blockIdx.y walks a tile table built on the device (tiles beyond *n_tiles leave at
//    once), and row r of the sorted order reads a's row gather[r] / gather_div (gather == nullptr: row r itself).
//  - bf16 products only: a_f32 -- a holds fp32 and is rounded to bf16 as it is staged; y_bf16 -- y holds bf16 (a result that
//    feeds the next product directly).
struct GemmIo {
    int lda, ldy;
    long long sa, sw, sy;
    const int32_t *tile_group, *tile_row0, *seg, *n_tiles, *gather;
    int gather_div;
    int a_f32, y_bf16;
};
constexpr int kGroupTile = 32;     // rows per tile of a grouped product (the tile table is built for this height)
static GemmIo plain_io(int K, int N) {
    GemmIo io;
    io.lda = K; io.ldy = N; io.sa = io.sw = io.sy = 0;
    io.tile_group = io.tile_row0 = io.seg = io.n_tiles = io.gather = nullptr;
    io.gather_div = 1;
    io.a_f32 = io.y_bf16 = 0;
    return io;
}

// Matrix product, fp32, operands whose rows are whole 16-byte pieces: y[M, N] = a[M, K] . w[N, K]^T on a tile of f32_tile.cuh (tensor cores; FMAs for the shortest
// sums), K shared by a cluster of CTAs along grid.x where the output has too few tiles to fill the GPU.
// 300 rows, 768 to 4608 columns and k: 57 us a product against 331 on the form below, which stages element by element and is bound by
// instruction issue.
template <int BM, int BN, class T>
__global__ void __launch_bounds__(T::NT) gemm_f32_tile_kernel(const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, const GemmIo io) {
    dep_wait();      // (and no early dep_go: the next kernel's blocks would take room from the CTAs that are still to come)
    extern __shared__ __align__(16) float f32_sm[];
    __shared__ long long arow[BM];
    int m0 = blockIdx.y * BM;
    const int n0 = (int)(blockIdx.x / f32t::cluster_size()) * BN;
    a += blockIdx.z * io.sa;
    w += blockIdx.z * io.sw;
    y += blockIdx.z * io.sy;
    if (io.tile_group) {
        if ((int)blockIdx.y >= *io.n_tiles) return;          // every rank of the cluster
        const int g = io.tile_group[blockIdx.y];
        m0 = io.tile_row0[blockIdx.y];
        M = io.seg[g + 1];
        w += (long long)g * io.sw;
    }
    for (int r = threadIdx.x; r < BM; r += T::NT) {
        const int m = m0 + r;
        arow[r] = m < M ? (long long)(io.gather ? io.gather[m] / io.gather_div : m) * io.lda : -1;
    }
    __syncthreads();
    int k_lo, k_hi;
    f32t::rank_range(K, k_lo, k_hi);
    typename T::Out out;
    T::product(f32_sm, k_lo, k_hi, [&](int r) { return arow[r] >= 0 ? a + arow[r] : nullptr; }, [](int k) -> long long { return k; },
                           [&](int r) { return n0 + r < N ? w + (size_t)(n0 + r) * K : nullptr; }, [] {}, out);
    const bool whole = io.ldy % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
    T::finish(f32_sm, out, [&](int r, int c, float4 v) {
        if (m0 + r >= M) return;
        float* to = y + (size_t)(m0 + r) * io.ldy + n0 + c;
        if (whole && n0 + c + 4 <= N) { *reinterpret_cast<float4*>(to) = v; return; }
        if (n0 + c < N) to[0] = v.x;
        if (n0 + c + 1 < N) to[1] = v.y;
        if (n0 + c + 2 < N) to[2] = v.z;
        if (n0 + c + 3 < N) to[3] = v.w;
    });
}

// The same for any sizes and alignment: plain FMAs, k ascending (the result of a row does not depend on M).
template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w,
                                                                        float* __restrict__ y, int M, int N, int K, const GemmIo io) {
    dep_wait();
    dep_go();
    constexpr int NT = (BM / TM) * (BN / TN);
    __shared__ float As[BK][BM + 1];
    __shared__ float Ws[BK][BN + 1];
    __shared__ long long arow[BM];
    int m0 = blockIdx.y * BM;
    const int n0 = blockIdx.x * BN;
    a += blockIdx.z * io.sa;
    w += blockIdx.z * io.sw;
    y += blockIdx.z * io.sy;
    if (io.tile_group) {
        if ((int)blockIdx.y >= *io.n_tiles) return;
        const int g = io.tile_group[blockIdx.y];
        m0 = io.tile_row0[blockIdx.y];
        M = io.seg[g + 1];
        w += (long long)g * io.sw;
    }
    for (int r = threadIdx.x; r < BM; r += NT) {
        const int m = m0 + r;
        arow[r] = m < M ? (long long)(io.gather ? io.gather[m] / io.gather_div : m) * io.lda : -1;
    }
    __syncthreads();
    const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int i = threadIdx.x; i < BM * BK; i += NT) {
            const int r = i / BK, c = i % BK;
            As[c][r] = (arow[r] >= 0 && k0 + c < K) ? a[arow[r] + k0 + c] : 0.0f;
        }
        for (int i = threadIdx.x; i < BN * BK; i += NT) {
            const int r = i / BK, c = i % BK;
            Ws[c][r] = (n0 + r < N && k0 + c < K) ? w[(size_t)(n0 + r) * K + k0 + c] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float av[TM], wv[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) wv[j] = Ws[k][tx + j * (BN / TN)];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int m = m0 + ty * TM + i, n = n0 + tx + j * (BN / TN);
            if (m < M && n < N) y[(size_t)m * io.ldy + n] = acc[i][j];
        }
}

// Matrix product, bf16 inputs on the tensor cores (mma.sync m16n8k16, fp32 accumulation): 4 warps, tile (WR*MT*16) x (WC*NT*8),
// K in steps of 32 through shared memory, the next step's global loads in flight during the MMAs.
constexpr int kGemmBK = 32;
constexpr int kGemmLd = kGemmBK + 8;   // 80-byte rows: fragment loads hit 32 distinct banks

// off[i]: element offset of the i-th row this thread fetches (negative: a row outside the matrix, read as zeros)
template <int ROWS>
__device__ __forceinline__ void gemm_fetch(const bf16* __restrict__ src, const long long (&off)[ROWS * 4 / 128], int K, int k0, bool vec,
                                           uint4 (&reg)[ROWS * 4 / 128], bool f32 = false) {
#pragma unroll
    for (int i = 0; i < ROWS * 4 / 128; ++i) {
        const int c = (threadIdx.x & 3) * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (off[i] >= 0 && f32) {
            const float* p = reinterpret_cast<const float*>(src) + off[i] + k0 + c;
            float e[8];
            if (vec && k0 + c + 8 <= K) {
                const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
                e[0] = lo.x; e[1] = lo.y; e[2] = lo.z; e[3] = lo.w; e[4] = hi.x; e[5] = hi.y; e[6] = hi.z; e[7] = hi.w;
            } else {
#pragma unroll
                for (int x = 0; x < 8; ++x) e[x] = (k0 + c + x < K) ? p[x] : 0.0f;
            }
            v = make_uint4(pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]), pack_bf16(e[4], e[5]), pack_bf16(e[6], e[7]));
        } else if (off[i] >= 0) {
            const bf16* p = src + off[i] + k0 + c;
            if (vec && k0 + c + 8 <= K) {
                v = *reinterpret_cast<const uint4*>(p);
            } else {
                uint16_t h[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) h[e] = (k0 + c + e < K) ? reinterpret_cast<const uint16_t*>(p)[e] : (uint16_t)0;
                v.x = h[0] | ((uint32_t)h[1] << 16); v.y = h[2] | ((uint32_t)h[3] << 16);
                v.z = h[4] | ((uint32_t)h[5] << 16); v.w = h[6] | ((uint32_t)h[7] << 16);
            }
        }
        reg[i] = v;
    }
}
template <int ROWS>
__device__ __forceinline__ void gemm_stash(bf16* dst, const uint4 (&reg)[ROWS * 4 / 128]) {
#pragma unroll
    for (int i = 0; i < ROWS * 4 / 128; ++i) {
        const int id = threadIdx.x + i * 128, r = id >> 2, c = (id & 3) * 8;
        *reinterpret_cast<uint4*>(dst + r * kGemmLd + c) = reg[i];
    }
}

// `vec`: every row of a and w starts on a 16-byte boundary and K is a multiple of 8 (whole 16-byte pieces).
template <int WR, int WC, int MT, int NT>
__global__ void __launch_bounds__(128) gemm_bf16_kernel(const bf16* __restrict__ a, const bf16* __restrict__ w, float* __restrict__ y,
                                                        int M, int N, int K, const GemmIo io, const bool vec) {
    dep_wait();
    dep_go();
    static_assert(WR * WC == 4, "four warps");
    constexpr int BM = WR * MT * 16, BN = WC * NT * 8;
    static_assert(BM % 32 == 0 && BN % 32 == 0, "tile rows are fetched 32 at a time");
    __shared__ __align__(16) bf16 As[2][BM * kGemmLd];
    __shared__ __align__(16) bf16 Ws[2][BN * kGemmLd];
    int m0 = blockIdx.y * BM;
    const int n0 = blockIdx.x * BN;
    const bool af = io.a_f32 != 0;
    a = af ? reinterpret_cast<const bf16*>(reinterpret_cast<const float*>(a) + blockIdx.z * io.sa) : a + blockIdx.z * io.sa;
    w += blockIdx.z * io.sw;
    const size_t y_base = (size_t)blockIdx.z * io.sy;
    if (io.tile_group) {
        if ((int)blockIdx.y >= *io.n_tiles) return;
        const int g = io.tile_group[blockIdx.y];
        m0 = io.tile_row0[blockIdx.y];
        M = io.seg[g + 1];
        w += (long long)g * io.sw;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int wm = (warp / WC) * MT * 16, wn = (warp % WC) * NT * 8;
    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
    uint4 ra[BM * 4 / 128], rw[BN * 4 / 128];
    long long oa[BM * 4 / 128], ow[BN * 4 / 128];
#pragma unroll
    for (int i = 0; i < BM * 4 / 128; ++i) {
        const int m = m0 + ((threadIdx.x + i * 128) >> 2);
        oa[i] = m < M ? (long long)(io.gather ? io.gather[m] / io.gather_div : m) * io.lda : -1;
    }
#pragma unroll
    for (int i = 0; i < BN * 4 / 128; ++i) {
        const int n = n0 + ((threadIdx.x + i * 128) >> 2);
        ow[i] = n < N ? (long long)n * K : -1;
    }
    gemm_fetch<BM>(a, oa, K, 0, vec, ra, af);
    gemm_fetch<BN>(w, ow, K, 0, vec, rw);
    gemm_stash<BM>(As[0], ra);
    gemm_stash<BN>(Ws[0], rw);
    __syncthreads();
    const int steps = (K + kGemmBK - 1) / kGemmBK;
    for (int s = 0; s < steps; ++s) {
        const int cur = s & 1;
        if (s + 1 < steps) {
            gemm_fetch<BM>(a, oa, K, (s + 1) * kGemmBK, vec, ra, af);
            gemm_fetch<BN>(w, ow, K, (s + 1) * kGemmBK, vec, rw);
        }
#pragma unroll
        for (int kk = 0; kk < kGemmBK; kk += 16) {
            uint32_t af[MT][4], bfr[NT][2];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const bf16* p = As[cur] + (wm + i * 16 + g) * kGemmLd + kk + tq * 2;
                af[i][0] = *reinterpret_cast<const uint32_t*>(p);
                af[i][1] = *reinterpret_cast<const uint32_t*>(p + 8 * kGemmLd);
                af[i][2] = *reinterpret_cast<const uint32_t*>(p + 8);
                af[i][3] = *reinterpret_cast<const uint32_t*>(p + 8 * kGemmLd + 8);
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const bf16* p = Ws[cur] + (wn + j * 8 + g) * kGemmLd + kk + tq * 2;
                bfr[j][0] = *reinterpret_cast<const uint32_t*>(p);
                bfr[j][1] = *reinterpret_cast<const uint32_t*>(p + 8);
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) mma_bf16_16816(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bfr[j][0], bfr[j][1]);
        }
        if (s + 1 < steps) {
            gemm_stash<BM>(As[cur ^ 1], ra);
            gemm_stash<BN>(Ws[cur ^ 1], rw);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int m = m0 + wm + i * 16 + g, n = n0 + wn + j * 8 + tq * 2;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int mm = m + (e >> 1) * 8, nn = n + (e & 1);
                if (mm < M && nn < N) {
                    const size_t at = y_base + (size_t)mm * io.ldy + nn;
                    if (io.y_bf16) reinterpret_cast<bf16*>(y)[at] = __float2bfloat16_rn(acc[i][j][e]);
                    else y[at] = acc[i][j][e];
                }
            }
        }
}

// Matrix product for few rows (decoding): bound by reading the weights once.  A block owns NR weight rows, its warps share K in
// interleaved steps of 32: a lane reads whole 16-byte pieces -- 8 neighbouring k of a weight row and of an activation row -- and hands
// them to m16n8k16 MMAs.  Both operands use the same assignment of k to fragment places, so the sum over k is the plain one in
// another order; the warps' shares are added in warp order.
// NR 16: the weights are the 16-row operand, a tile of activations its 8 columns.  NR 8 (narrow products, whose blocks of 16 would not
// reach every SM): the weights are the 8 columns, a tile of activations the 16 rows.
// On the CUDA cores (one warp per column) five rows cost 40 conversions and multiply-adds per 16 bytes of weights: 18.9 us per product
// over a decode step of width 1536 (17 MB each, 0.9 TB/s) against 6.8 us here; one row of 768 x 4608 takes 8.2 us with NR 16 and 6.4
// with NR 8.
// WARPS follows from K, NR from N.  Needs K % 8 == 0 and 16-byte aligned operands.
// An MMA drops what of its products lies below the last place of the sum it adds to, and a chain of them collects these losses: every MMA starts
// from zero, its sums are added in rounded fp32, the warps' shares in fp64 with one rounding.  Error against 64 bits at K =
// 768 / 4608: 5.5e-8 / 7.4e-8 (one warp per column with FMAs 6.5e-8 / 8.6e-8; a chain of MMAs per warp 1.1e-7 / 2.7e-7, a twentieth faster: 5 x
// 1536 x 4096 5.6 us against 6.0).
template <int NR, int MT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) gemm_few_kernel(const bf16* __restrict__ a, const bf16* __restrict__ w, float* __restrict__ y,
                                                              int M, int N, int K) {
    constexpr int WT = NR / 8, AT = NR == 16 ? MT : 2 * MT;      // 8-row pieces of weights and of activations per step
    constexpr int U = WT + AT <= 3 ? 4 : 2;                      // steps of 32 whose loads are in flight together
    constexpr int OUT = NR * (NR == 16 ? 8 : 16) * MT;           // outputs of the block
    __shared__ float part[WARPS][OUT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int n0 = blockIdx.x * NR;
    const bf16* wr[WT];
#pragma unroll
    for (int i = 0; i < WT; ++i) wr[i] = w + (size_t)min(n0 + i * 8 + g, N - 1) * K + tq * 8;
    float acc[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.0f;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 p[U][WT];
    auto load_weights = [&](int k0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * 32;
#pragma unroll
            for (int i = 0; i < WT; ++i) p[u][i] = k + tq * 8 < K ? ldg_stream(wr[i] + k) : zero;
        }
    };
    load_weights(warp * 32);             // no kernel of a step writes weights: the first ones are on their way before the wait (smol_lm_linear launches plainly)
    dep_wait();
    dep_go();
    for (int k0 = warp * 32; k0 < K; k0 += WARPS * 32 * U) {
        uint4 x[U][AT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * 32 + tq * 8;
#pragma unroll
            for (int i = 0; i < AT; ++i) {
                const int m = i * 8 + g;
                x[u][i] = (m < M && k < K) ? ldg_v4(a + (size_t)m * K + k) : zero;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                float lo[4] = {0.0f, 0.0f, 0.0f, 0.0f}, hi[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if constexpr (NR == 16) {
                    mma_bf16_16816(lo, p[u][0].x, p[u][1].x, p[u][0].y, p[u][1].y, x[u][i].x, x[u][i].y);
                    mma_bf16_16816(hi, p[u][0].z, p[u][1].z, p[u][0].w, p[u][1].w, x[u][i].z, x[u][i].w);
                } else {
                    mma_bf16_16816(lo, x[u][2 * i].x, x[u][2 * i + 1].x, x[u][2 * i].y, x[u][2 * i + 1].y, p[u][0].x, p[u][0].y);
                    mma_bf16_16816(hi, x[u][2 * i].z, x[u][2 * i + 1].z, x[u][2 * i].w, x[u][2 * i + 1].w, p[u][0].z, p[u][0].w);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][e] += lo[e] + hi[e];
            }
        load_weights(k0 + WARPS * 32 * U);
    }
    // part[warp][m * NR + n]: neighbouring outputs of a row side by side.  acc[.][e]: tile row g + (e / 2) * 8, tile column 2 tq + e % 2
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = g + (e >> 1) * 8, c = tq * 2 + (e & 1);
            part[warp][NR == 16 ? (i * 8 + c) * NR + r : (i * 16 + r) * NR + c] = acc[i][e];
        }
    __syncthreads();
    for (int o = threadIdx.x; o < OUT; o += WARPS * 32) {
        const int m = o / NR, n = n0 + o % NR;
        double t = part[0][o];
#pragma unroll
        for (int x = 1; x < WARPS; ++x) t += part[x][o];
        if (m < M && n < N) y[(size_t)m * N + n] = (float)t;
    }
}
constexpr int kFewRows = 32;             // most rows of gemm_few_kernel
constexpr int kFewLongK = 2048;          // from this K on 16 warps share it
constexpr int kFewWideN = 16 * 148;      // from this N on blocks of 16 weight rows give every SM one

}  // namespace lm
}  // namespace smol

#include "lm_gemm_tc.cuh"

namespace smol {
namespace lm {

// ---------------------------------------------------------------------------------------------------------------------
// Softmax attention over the paged pool.  A cached position holds, per key/value head, a key row of d elements (row
// stride k_ld) and a value row of dv elements (row stride v_ld); with v_in_k the value is the first dv elements of the key
// row (a latent that serves as both).  Optional per head: a distance penalty r1 ln(1 + r2 (i - j)) taken off the score
// (r1 == nullptr: none) and a key-less sink logit in the softmax denominator (sink == nullptr: none).  The output is
// multiplied by sigmoid(proj[t][gate_off + h * gate_ld + c * gate_step]): a gate per channel or (gate_step 0) per head.
// Sink attention's proj row layout: q [H*d] | k [G*d] | v [G*dv] | gate [H*dv] (no gate rows with has_gate == 0).
// Further options, each off at its zero value: `bias` added to the projection's rows as they are read; `window` > 0 limits
// a query at position i to the keys 0 <= i - j < window; `softcap` > 0 bends the scaled score to softcap * tanh(score /
// softcap) before the penalties; `slope` takes slope_h * (i - j) off.  The result is multiplied by out_scale and written
// with the row stride out_ld (two mixers side by side share one buffer).
// Differential attention (maps 2): every head has two softmax maps over the same values -- query rows [H][maps][d], key rows
// [G][maps][d], a cached position holding G * maps key rows and G value rows; with a and b the maps' results a head's output is
// o = a - diff_lambda * b, divided by its root mean square over dv, times diff_scale, before the gate.
struct AttnArgs {
    const float* proj;
    int n_in;
    const int32_t *tok_seq, *tok_pos, *block_table;
    int max_pages, page_size, n_pages;
    size_t page_elems, k_off, v_off;   // element offsets of this run's keys / values inside a page
    int k_ld, v_ld, v_in_k;
    size_t gate_off;
    int gate_ld, gate_step;
    int H, G, d, dv;
    float scale, eps;
    const float *q_norm, *k_norm, *r1, *r2, *sink;
    int n_tokens;
    int32_t* err;
    const int32_t* seq_start;
    int split_len, n_splits, short_rows;   // few-token path: key range per block, ranges per row, rows = sequences x kShortSeq
    float* part;                           // [short_rows][H][n_splits][dv + 2]: running maximum, denominator, unnormalised output
    const float *bias, *slope;
    int window, has_gate, out_ld;
    float softcap, two_over_cap, out_scale;      // two_over_cap = 2 / softcap (0 without a cap)
    float temp_coef = 0.0f, temp_every = 0.0f;   // query temperature (temp_every 0: none), see attn_temperature
    int maps = 1;                                // softmax maps per head
    float diff_lambda = 0.0f, diff_scale = 1.0f;
    int own_kv = 1;                              // 0: the cached keys and values are another layer's, the projection holds none
    int rot_pairs = 0, rot_half = 0;             // rotated pairs of q and k (whole-projection norms only): i with i + rot_pairs, or 2i with 2i + 1
    float rot_mult = 1.0f;                       // multiplies cosine and sine
    const float* freq = nullptr;                 // [rot_pairs]
};

// what a query at `pos` is multiplied by: 1 + coef * ln(floor((pos + 1) / every) + 1)
__device__ __forceinline__ float attn_temperature(const AttnArgs& A, int pos) {
    return A.temp_every > 0.0f ? 1.0f + A.temp_coef * logf(floorf((float)(pos + 1) / A.temp_every) + 1.0f) : 1.0f;
}

// first key a query at `pos` sees
__device__ __forceinline__ int attn_first_key(const AttnArgs& A, int pos) { return A.window > 0 ? max(0, pos - A.window + 1) : 0; }

// what follows the dot product: scale, soft cap, distance penalties.  FAST: hardware exponential / logarithm (bf16 engine).
template <bool FAST>
__device__ __forceinline__ float attn_score(const AttnArgs& A, float dot, int dist, float r1, float r2, float slope) {
    float s = dot * A.scale;
    if (A.softcap > 0.0f) {
        // FAST: tanh z = 1 - 2 / (e^{2z} + 1) with the hardware exponential and division (an overflowing e^{2z} gives 1)
        if (FAST) s = A.softcap * (1.0f - __fdividef(2.0f, __expf(s * A.two_over_cap) + 1.0f));
        else s = A.softcap * tanhf(s / A.softcap);
    }
    if (A.r1) s -= r1 * (FAST ? __logf(1.0f + r2 * (float)dist) : log1pf(r2 * (float)dist));
    if (A.slope) s -= slope * (float)dist;
    return s;
}

// One warp per (token, slot): the first H * maps slots norm a query row into qbuf (times the query temperature), the next
// G * maps norm a key row into the pool, the last G copy a value head into the pool (own_kv 0: query rows only).
// q_norm / k_norm == nullptr: no norm.
template <class T>
__global__ void attn_prep_kernel(const AttnArgs A, T* __restrict__ qbuf, T* __restrict__ pool) {
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int HQ = A.H * A.maps, GK = A.G * A.maps, slots = HQ + (A.own_kv ? GK + A.G : 0);
    if (unit >= A.n_tokens * slots) { dep_wait(); return; }
    const int t = unit / slots, s = unit % slots, pos = A.tok_pos[t];
    const int pg = pos / A.page_size, in_pg = pos % A.page_size;
    const int page = s >= HQ && pg < A.max_pages ? A.block_table[(size_t)A.tok_seq[t] * A.max_pages + pg] : -1;
    dep_wait();
    dep_go();
    const float* row = A.proj + (size_t)t * A.n_in;
    if (s < HQ) {
        const float* q = row + s * A.d;
        const float* qb = A.bias ? A.bias + s * A.d : nullptr;
        float ss = 0.0f;
        for (int c = lane; c < A.d; c += 32) { const float v = q[c] + (qb ? qb[c] : 0.0f); ss += v * v; }
        ss = warp_sum(ss);
        const float r = (A.q_norm ? 1.0f / sqrtf(ss / (float)A.d + A.eps) : 1.0f) * attn_temperature(A, pos);
        for (int c = lane; c < A.d; c += 32)
            qbuf[((size_t)t * HQ + s) * A.d + c] = from_f<T>((q[c] + (qb ? qb[c] : 0.0f)) * r * (A.q_norm ? A.q_norm[c] : 1.0f));
        return;
    }
    if (page < 0 || page >= A.n_pages) {
        if (lane == 0) atomicExch(A.err, 1);
        return;
    }
    T* base = pool + (size_t)page * A.page_elems;
    if (s < HQ + GK) {
        const int gk = s - HQ;
        const float* k = row + HQ * A.d + gk * A.d;
        const float* kb = A.bias ? A.bias + HQ * A.d + gk * A.d : nullptr;
        float ss = 0.0f;
        for (int c = lane; c < A.d; c += 32) { const float v = k[c] + (kb ? kb[c] : 0.0f); ss += v * v; }
        ss = warp_sum(ss);
        const float r = A.k_norm ? 1.0f / sqrtf(ss / (float)A.d + A.eps) : 1.0f;
        T* dst = base + A.k_off + ((size_t)gk * A.page_size + in_pg) * A.d;
        for (int c = lane; c < A.d; c += 32) dst[c] = from_f<T>((k[c] + (kb ? kb[c] : 0.0f)) * r * (A.k_norm ? A.k_norm[c] : 1.0f));
    } else {
        const int gv = s - HQ - GK;
        const float* v = row + (HQ + GK) * A.d + gv * A.dv;
        const float* vb = A.bias ? A.bias + (HQ + GK) * A.d + gv * A.dv : nullptr;
        T* dst = base + A.v_off + ((size_t)gv * A.page_size + in_pg) * A.dv;
        for (int c = lane; c < A.dv; c += 32) dst[c] = from_f<T>(v[c] + (vb ? vb[c] : 0.0f));
    }
}

// The same for heads of up to 4 L elements whose rows are whole 16-byte pieces: a piece per lane, L lanes per unit.  Nearly all of it is waiting for loads: 2048 tokens of 20
// heads of 64 6.9 us as against 13.8 with 4-byte loads and a warp per unit (24 with four units per warp).
template <class T, int L>
__global__ void __launch_bounds__(128) attn_prep_vec_kernel(const AttnArgs A, T* __restrict__ qbuf, T* __restrict__ pool) {
    const int unit = (int)(blockIdx.x * blockDim.x + threadIdx.x) / L, c = 4 * (threadIdx.x % L);
    const int HQ = A.H * A.maps, GK = A.G * A.maps, slots = HQ + (A.own_kv ? GK + A.G : 0);
    const bool live = unit < A.n_tokens * slots;
    const int t = live ? unit / slots : 0, s = unit - t * slots, pos = A.tok_pos[t];
    const int pg = pos / A.page_size, in_pg = pos - pg * A.page_size;
    const int page = s >= HQ && pg < A.max_pages ? A.block_table[(size_t)A.tok_seq[t] * A.max_pages + pg] : -1;
    const bool key = s >= HQ && s < HQ + GK, in = live && c < (s < HQ + GK ? A.d : A.dv);
    const int at = (s < HQ + GK ? s * A.d : (HQ + GK) * A.d + (s - HQ - GK) * A.dv) + c;
    const float* norm = s < HQ ? A.q_norm : key ? A.k_norm : nullptr;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f), w = in && norm ? load4(norm + c) : make_float4(1.0f, 1.0f, 1.0f, 1.0f), b = in && A.bias ? load4(A.bias + at) : none;
    dep_wait();
    dep_go();
    float4 v = in ? load4(A.proj + (size_t)t * A.n_in + at) : none;
    v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
    float ss = squares(v);
#pragma unroll
    for (int x = L / 2; x > 0; x >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, x);
    float r = norm ? 1.0f / sqrtf(ss / (float)A.d + A.eps) : 1.0f;
    T* to;
    if (s < HQ) {
        r *= attn_temperature(A, pos);
        to = qbuf + ((size_t)t * HQ + s) * A.d + c;
    } else {
        if (live && (page < 0 || page >= A.n_pages)) {
            if (c == 0) atomicExch(A.err, 1);
            return;
        }
        to = pool + (size_t)page * A.page_elems + (key ? A.k_off + ((size_t)(s - HQ) * A.page_size + in_pg) * A.d : A.v_off + ((size_t)(s - HQ - GK) * A.page_size + in_pg) * A.dv) + c;
    }
    if (in) store4<T>(to, v.x * r * w.x, v.y * r * w.y, v.z * r * w.z, v.w * r * w.w);
}

// The same preparation with query and key norms over the WHOLE projection: one root mean square for all query heads of a
// token (weights q_norm [H*d]) and one for all key heads (k_norm [G*d]).  One block per token.  Loads go out kPrepBatch
// at a time before their first use: a lone token (decoding) waits for memory a few times, not once per element.
// ROT: queries and keys are rotated after the norm, the token's cosines and sines taken once for all heads.
constexpr int kPrepBatch = 4;
constexpr int kMaxRotPairs = 256;

template <class T, bool ROT>
__global__ void __launch_bounds__(256) attn_prep_whole_kernel(const AttnArgs A, T* __restrict__ qbuf, T* __restrict__ pool) {
    __shared__ float red[2][33];
    __shared__ float turn[2][ROT ? kMaxRotPairs : 1];
    const int t = blockIdx.x, nq = A.H * A.d, nk = A.G * A.d, nv = A.G * A.dv;
    const float* row = A.proj + (size_t)t * A.n_in;
    const int pos = A.tok_pos[t];
    const int pg = pos / A.page_size, in_pg = pos % A.page_size;
    const int page = pg < A.max_pages ? A.block_table[(size_t)A.tok_seq[t] * A.max_pages + pg] : -1;
    // sum of squares of row[lo .. lo + n) + bias
    auto sum_sq = [&](int lo, int n) {
        float ss = 0.0f;
        for (int c0 = threadIdx.x; c0 < n; c0 += blockDim.x * kPrepBatch) {
            float v[kPrepBatch], bv[kPrepBatch];
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) {
                const int c = c0 + u * blockDim.x;
                v[u] = c < n ? row[lo + c] : 0.0f;
                bv[u] = (c < n && A.bias) ? A.bias[lo + c] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) ss = fmaf(v[u] + bv[u], v[u] + bv[u], ss);
        }
        return ss;
    };
    if (ROT)
        for (int i = threadIdx.x; i < A.rot_pairs; i += blockDim.x) {
            float sn, cs;
            sincosf((float)pos * A.freq[i], &sn, &cs);
            turn[0][i] = cs * A.rot_mult;
            turn[1][i] = sn * A.rot_mult;
        }
    dep_wait();
    dep_go();
    float sq = sum_sq(0, nq), sk = sum_sq(nq, nk);
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    if (l == 0) { red[0][w] = sq; red[1][w] = sk; }
    __syncthreads();
    sq = 0.0f;
    sk = 0.0f;
    for (int i = 0; i < nw; ++i) { sq += red[0][i]; sk += red[1][i]; }      // the same order in every thread
    const float rq = 1.0f / sqrtf(sq / (float)nq + A.eps), rk = 1.0f / sqrtf(sk / (float)nk + A.eps);
    // element c of row[lo ..) + bias, times mul, times weight[c] (nullptr: 1) -> store(c, value)
    auto emit = [&](int lo, int n, float mul, const float* weight, auto store) {
        for (int c0 = threadIdx.x; c0 < n; c0 += blockDim.x * kPrepBatch) {
            float v[kPrepBatch], wv[kPrepBatch];
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) {
                const int c = c0 + u * blockDim.x;
                v[u] = c < n ? row[lo + c] + (A.bias ? A.bias[lo + c] : 0.0f) : 0.0f;
                wv[u] = (c < n && weight) ? weight[c] : 1.0f;
            }
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) {
                const int c = c0 + u * blockDim.x;
                if (c < n) store(c, v[u] * mul * wv[u]);
            }
        }
    };
    // the same with the rotation: a rotated element also reads its pair's other one
    auto emit_rotated = [&](int lo, int n, float mul, const float* weight, auto store) {
        for (int c0 = threadIdx.x; c0 < n; c0 += blockDim.x * kPrepBatch) {
            float v[kPrepBatch], o[kPrepBatch], cs[kPrepBatch], sn[kPrepBatch];
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) {
                const int c = c0 + u * blockDim.x, i = c % A.d;
                int p = 0, other = -1;
                bool first = true;
                if (c < n && i < 2 * A.rot_pairs) {
                    first = A.rot_half ? i < A.rot_pairs : i % 2 == 0;
                    p = A.rot_half ? (first ? i : i - A.rot_pairs) : i / 2;
                    const int step = A.rot_half ? A.rot_pairs : 1;
                    other = first ? c + step : c - step;
                }
                v[u] = c < n ? (row[lo + c] + (A.bias ? A.bias[lo + c] : 0.0f)) * (weight ? weight[c] : 1.0f) : 0.0f;
                o[u] = other >= 0 ? (row[lo + other] + (A.bias ? A.bias[lo + other] : 0.0f)) * (weight ? weight[other] : 1.0f) : 0.0f;
                cs[u] = other >= 0 ? turn[0][p] : 1.0f;
                sn[u] = other >= 0 ? (first ? -turn[1][p] : turn[1][p]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kPrepBatch; ++u) {
                const int c = c0 + u * blockDim.x;
                if (c < n) store(c, (v[u] * mul) * cs[u] + (o[u] * mul) * sn[u]);
            }
        }
    };
    auto emit_qk = [&](int lo, int n, float mul, const float* weight, auto store) {
        if constexpr (ROT) emit_rotated(lo, n, mul, weight, store);
        else emit(lo, n, mul, weight, store);
    };
    emit_qk(0, nq, rq * attn_temperature(A, pos), A.q_norm, [&](int c, float v) { qbuf[(size_t)t * nq + c] = from_f<T>(v); });
    if (page < 0 || page >= A.n_pages) {
        if (threadIdx.x == 0) atomicExch(A.err, 1);
        return;
    }
    T* base = pool + (size_t)page * A.page_elems;
    emit_qk(nq, nk, rk, A.k_norm, [&](int c, float v) {
        const int g = c / A.d, i = c - g * A.d;
        base[A.k_off + ((size_t)g * A.page_size + in_pg) * A.d + i] = from_f<T>(v);
    });
    emit(nq + nk, nv, 1.0f, nullptr, [&](int c, float v) {
        const int g = c / A.dv, i = c - g * A.dv;
        base[A.v_off + ((size_t)g * A.page_size + in_pg) * A.dv + i] = from_f<T>(v);
    });
}

// One warp per (token, query head), 32 keys per round: lane j scores key j (full dot product, the query in shared
// memory), the round's softmax weights are shared by shuffles and every lane accumulates dv / 32 output columns.
// The sink enters as the initial state of the running softmax: maximum = sink, denominator = 1, no value.
constexpr int kAttnWarps = 4;
constexpr int kAttnMaxV = 16;  // value size up to 512; the kernels are built for 8 (up to 256) and 16 lanes' worth of columns

__device__ __forceinline__ float attn_gate(const AttnArgs& A, size_t t, int h, int c) {
    if (!A.has_gate) return A.out_scale;
    return A.out_scale * sigmoidf_(A.proj[t * A.n_in + A.gate_off + (size_t)h * A.gate_ld + (size_t)c * A.gate_step]);
}

// A head's finished result from the columns a warp holds (column lane + 32 e in o[e], the maps already joined): the
// differential form's division by the root mean square, then the gate.
template <class T, int MAXV, int MAPS>
__device__ __forceinline__ void attn_finish(const AttnArgs& A, size_t t, int h, int lane, float (&o)[MAXV], T* __restrict__ out) {
    float r = 1.0f;
    if (MAPS == 2) {
        float ss = 0.0f;
#pragma unroll
        for (int e = 0; e < MAXV; ++e) ss = fmaf(o[e], o[e], ss);      // columns beyond dv hold zeros
        r = A.diff_scale / sqrtf(warp_sum(ss) / (float)A.dv + A.eps);
    }
#pragma unroll
    for (int e = 0; e < MAXV; ++e) {
        const int c = lane + e * 32;
        if (c < A.dv) out[t * A.out_ld + h * A.dv + c] = from_f<T>((MAPS == 2 ? o[e] * r : o[e]) * attn_gate(A, t, h, c));
    }
}

template <class T, int MAXV, int MAPS>
__global__ void __launch_bounds__(kAttnWarps * 32) attn_kernel(const AttnArgs A, const T* __restrict__ qbuf, const T* __restrict__ pool,
                                                               T* __restrict__ out) {
    dep_wait();
    dep_go();
    extern __shared__ float qs_all[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x * kAttnWarps + warp;
    if (unit >= A.n_tokens * A.H) return;
    const int t = unit / A.H, h = unit % A.H;
    const int g = h / (A.H / A.G);
    float* qs = qs_all + warp * A.d;
    const int pos = A.tok_pos[t];
    const int32_t* bt = A.block_table + (size_t)A.tok_seq[t] * A.max_pages;
    const float r1 = A.r1 ? A.r1[h] : 0.0f, r2 = A.r1 ? A.r2[h] : 0.0f, slope = A.slope ? A.slope[h] : 0.0f;
    float sum[MAXV];                    // the maps' joined result
#pragma unroll
    for (int map = 0; map < MAPS; ++map) {
        __syncwarp();
        for (int c = lane; c < A.d; c += 32) qs[c] = to_f<T>(qbuf[(((size_t)t * A.H + h) * MAPS + map) * A.d + c]);
        __syncwarp();
        float m = A.sink ? A.sink[h] : -INFINITY, l = A.sink ? 1.0f : 0.0f;
        float o[MAXV];
#pragma unroll
        for (int e = 0; e < MAXV; ++e) o[e] = 0.0f;
        for (int j0 = attn_first_key(A, pos); j0 <= pos; j0 += 32) {
            const int j = j0 + lane;
            float s = -INFINITY;
            const T* vrow = nullptr;
            if (j <= pos) {
                const int page = bt[j / A.page_size], in_pg = j % A.page_size;
                const T* base = pool + (size_t)page * A.page_elems;
                const T* k = base + A.k_off + ((size_t)(g * MAPS + map) * A.page_size + in_pg) * A.k_ld;
                vrow = base + A.v_off + ((size_t)g * A.page_size + in_pg) * A.v_ld;
                float dot = 0.0f;
                for (int c = 0; c < A.d; ++c) dot = fmaf(qs[c], to_f<T>(k[c]), dot);
                s = attn_score<false>(A, dot, pos - j, r1, r2, slope);
            }
            const float mn = fmaxf(m, warp_max(s));          // finite: lane 0 of every round holds a visible key
            const float p = (j <= pos) ? expf(s - mn) : 0.0f;
            const float corr = expf(m - mn);
            l = l * corr + warp_sum(p);
            m = mn;
#pragma unroll
            for (int e = 0; e < MAXV; ++e) o[e] *= corr;
            const int cnt = min(32, pos - j0 + 1);
            for (int jj = 0; jj < cnt; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, p, jj);
                const T* vr = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(vrow), jj));
#pragma unroll
                for (int e = 0; e < MAXV; ++e) {
                    const int c = lane + e * 32;
                    if (c < A.dv) o[e] = fmaf(pj, to_f<T>(vr[c]), o[e]);
                }
            }
        }
        const float inv = 1.0f / l;
#pragma unroll
        for (int e = 0; e < MAXV; ++e) sum[e] = map == 0 ? o[e] * inv : fmaf(-A.diff_lambda, o[e] * inv, sum[e]);
    }
    attn_finish<T, MAXV, MAPS>(A, t, h, lane, sum, out);
}

// ---------------------------------------------------------------------------------------------------------------------
// Attention for sequences that bring few tokens (decoding, short portions): the keys of a row are cut into fixed
// ranges of A.split_len positions, one block per (row, key/value head, range), whose warps take the query heads of
// that key/value head; a second kernel merges the ranges with the sink and applies the gate.  The ranges are absolute
// positions, so a row's result does not depend on what else is in the step.
constexpr int kGraphMaxTokens = 64;   // steps of at most this many tokens are replayed from a captured graph
constexpr int kShortSeq = 8;          // a sequence with at most this many tokens in a step takes this path

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// q (fp32, shared memory) . k (one cached key row), 16-byte loads where both rows allow them
template <class T> __device__ __forceinline__ float key_dot(const float* qs, const T* k, int d);
template <> __device__ __forceinline__ float key_dot<float>(const float* qs, const float* k, int d) {
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
    if (d % 4 == 0 && (reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(qs)) % 16 == 0) {
#pragma unroll 4
        for (int c = 0; c < d; c += 4) {
            const float4 v = *reinterpret_cast<const float4*>(k + c), x = *reinterpret_cast<const float4*>(qs + c);
            a0 = fmaf(x.x, v.x, a0); a1 = fmaf(x.y, v.y, a1); a2 = fmaf(x.z, v.z, a2); a3 = fmaf(x.w, v.w, a3);
        }
    } else {
        for (int c = 0; c < d; ++c) a0 = fmaf(qs[c], k[c], a0);
    }
    return (a0 + a1) + (a2 + a3);
}
template <> __device__ __forceinline__ float key_dot<bf16>(const float* qs, const bf16* k, int d) {
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
    if (d % 8 == 0 && (reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(qs)) % 16 == 0) {
#pragma unroll 4
        for (int c = 0; c < d; c += 8) {
            const uint4 v = *reinterpret_cast<const uint4*>(k + c);
            const float4 x = *reinterpret_cast<const float4*>(qs + c), y = *reinterpret_cast<const float4*>(qs + c + 4);
            a0 = fmaf(x.x, bf_lo(v.x), a0); a1 = fmaf(x.y, bf_hi(v.x), a1);
            a2 = fmaf(x.z, bf_lo(v.y), a2); a3 = fmaf(x.w, bf_hi(v.y), a3);
            a0 = fmaf(y.x, bf_lo(v.z), a0); a1 = fmaf(y.y, bf_hi(v.z), a1);
            a2 = fmaf(y.z, bf_lo(v.w), a2); a3 = fmaf(y.w, bf_hi(v.w), a3);
        }
    } else {
        for (int c = 0; c < d; ++c) a0 = fmaf(qs[c], __bfloat162float(k[c]), a0);
    }
    return (a0 + a1) + (a2 + a3);
}

// two neighbouring elements (the address is a multiple of their size)
__device__ __forceinline__ float2 load_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_pair(const bf16* p) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p);
    return make_float2(bf_lo(v), bf_hi(v));
}
// row stride of the staged values: an even number of elements
template <class T> __host__ __device__ constexpr int split_value_ld(int dv) { return (dv + 16 / (int)sizeof(T) + 1) / 2 * 2; }

// Prompts without a tensor-core form (float32; bf16 heads above 128): a block takes 4 R neighbouring rows of a sequence and one head, a warp R of them, 32 keys and
// values at a time in shared memory.  A lane scores one key for the warp's R rows, so a key's 16-byte loads and a value's are shared by R rows; a row's sums are
// those of a warp of its own: it takes nothing from a key or value that it does not see.
// What bounds it is shared memory: a 16-byte load of a key and one of each query for 4 R multiply-adds.  300 rows of 12 heads of 64, float32: 60 us
// (1100: 332) against 230 (2237) for a warp per row that reads its keys from global memory, a row per lane (attn_kernel, which stays for rows that leave no room
// for the tiles and for some that are no whole pieces); 9 rows 5.7 against 8.8, 7 x 170 76 against 249; two maps of 64 and values of 128, 300 rows 91 against 330; a latent of 160, 79 against 431.
constexpr int kRowsKeys = 32, kRowsWarps = 4, kRowsSmemMax = 100 * 1024;
template <class T> __host__ __device__ constexpr int rows_ld(int d) { return (d * (int)sizeof(T) + 15) / 16 * 16 / (int)sizeof(T) + 16 / (int)sizeof(T); }      // 16-byte rows, an odd number of them
template <class T> static constexpr size_t rows_smem(int R, int d, int dv, bool v_in_k) {
    return (size_t)kRowsWarps * R * ((d + 3) / 4 * 4 + kRowsKeys) * 4 + (size_t)kRowsKeys * (rows_ld<T>(d) + (v_in_k ? 0 : rows_ld<T>(dv))) * sizeof(T);
}
template <class T, int MAXV, int MAPS, int R>
__global__ void __launch_bounds__(kRowsWarps * 32) attn_rows_kernel(const AttnArgs A, const T* __restrict__ qbuf, const T* __restrict__ pool, T* __restrict__ out) {
    dep_wait();
    dep_go();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    constexpr int kPad = 16 / (int)sizeof(T), KEYS = kRowsKeys, RB = kRowsWarps * R;
    const int h = blockIdx.y, s = blockIdx.z, t0 = A.seq_start[s], n = A.seq_start[s + 1] - t0, r0 = blockIdx.x * RB;
    if (r0 >= n) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = h / (A.H / A.G), rows = min(RB, n - r0);
    const int pos0 = A.tok_pos[t0 + r0], mine = min(R, max(0, rows - warp * R)), my_pos = pos0 + warp * R;      // (a sequence's tokens of a step are neighbours)
    const int qd = (A.d + 3) / 4 * 4, ldk = rows_ld<T>(A.d), ldv = A.v_in_k ? ldk : rows_ld<T>(A.dv);
    float* qs = reinterpret_cast<float*>(sm_raw) + warp * R * qd;
    float* ps = reinterpret_cast<float*>(sm_raw) + RB * qd + warp * R * KEYS;      // [KEYS][R]
    T* Ks = reinterpret_cast<T*>(sm_raw + (size_t)RB * (qd + KEYS) * 4);
    T* Vs = A.v_in_k ? Ks : Ks + KEYS * ldk;
    const int32_t* bt = A.block_table + (size_t)s * A.max_pages;
    const float r1 = A.r1 ? A.r1[h] : 0.0f, r2 = A.r1 ? A.r2[h] : 0.0f, slope = A.slope ? A.slope[h] : 0.0f;
    const bool kvec = (A.d * sizeof(T)) % 16 == 0 && (A.k_ld * sizeof(T)) % 16 == 0 && (A.k_off * sizeof(T)) % 16 == 0;
    const bool vvec = (A.dv * sizeof(T)) % 16 == 0 && (A.v_ld * sizeof(T)) % 16 == 0 && (A.v_off * sizeof(T)) % 16 == 0;
    const int kchunks = kvec ? A.d / kPad : A.d, vchunks = A.v_in_k ? 0 : vvec ? A.dv / kPad : A.dv;
    const int j_first = attn_first_key(A, pos0), j_last = pos0 + rows - 1;      // keys that some row of the block sees
    float sum[R][MAXV];                    // the maps' joined results
#pragma unroll
    for (int map = 0; map < MAPS; ++map) {
        __syncwarp();
        for (int i = 0; i < mine; ++i)
            for (int c = lane; c < qd; c += 32) qs[i * qd + c] = c < A.d ? to_f<T>(qbuf[(((size_t)(t0 + r0 + warp * R + i) * A.H + h) * MAPS + map) * A.d + c]) : 0.0f;
        float m[R], l[R], o[R][MAXV];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            m[i] = A.sink ? A.sink[h] : -INFINITY;
            l[i] = A.sink ? 1.0f : 0.0f;
#pragma unroll
            for (int e = 0; e < MAXV; ++e) o[i][e] = 0.0f;
        }
        // Tiles begin at multiples of KEYS: a row's sums depend neither on its place in the block nor on what the block's first row sees of a window.
        for (int j0 = j_first / KEYS * KEYS; j0 <= j_last; j0 += KEYS) {
            const int skip = max(0, j_first - j0), cnt = min(KEYS, j_last - j0 + 1);
            __syncthreads();
            {
                const int jr = min(max(j0 + lane, j_first), j_last), page = bt[jr / A.page_size], place = jr % A.page_size;      // (pages in front of the window may be gone)
                for (int c = lane; c - lane < kchunks + vchunks; c += 32) {
                    const bool key = c < kchunks, live = c < kchunks + vchunks;
                    const int piece = key ? c : c - kchunks, step = (key ? kvec : vvec) ? kPad : 1, ld = key ? A.k_ld : A.v_ld, dst_ld = key ? ldk : ldv;
                    const T* src0 = pool + (key ? A.k_off + (size_t)(g * MAPS + map) * A.page_size * ld : A.v_off + (size_t)g * A.page_size * ld) + piece * step;
                    T* dst0 = (key ? Ks : Vs) + piece * step;
#pragma unroll 4
                    for (int r = skip + warp; r < cnt; r += kRowsWarps) {
                        const int pg = __shfl_sync(0xffffffffu, page, r), at = __shfl_sync(0xffffffffu, place, r);
                        const T* src = src0 + (size_t)pg * A.page_elems + (size_t)at * ld;
                        T* dst = dst0 + r * dst_ld;
                        if (!live) continue;
                        if (step == kPad) cp_async16(dst, src);
                        else *dst = *src;
                    }
                }
                cp_async_commit_group();
                cp_async_wait_group<0>();
            }
            __syncthreads();
            if (mine == 0 || j0 > my_pos + mine - 1) continue;
            float dot[R];
#pragma unroll
            for (int i = 0; i < R; ++i) dot[i] = 0.0f;
            const T* kr = Ks + lane * ldk;
            int c = 0;
            if (sizeof(T) == 4) {
#pragma unroll 4
                for (; c + 4 <= A.d; c += 4) {
                    const float4 k = *reinterpret_cast<const float4*>(kr + c);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const float4 q = *reinterpret_cast<const float4*>(qs + i * qd + c);
                        dot[i] = fmaf(q.x, k.x, fmaf(q.y, k.y, fmaf(q.z, k.z, fmaf(q.w, k.w, dot[i]))));
                    }
                }
            }
            for (; c < A.d; ++c) {
                const float k = to_f<T>(kr[c]);
#pragma unroll
                for (int i = 0; i < R; ++i) dot[i] = fmaf(qs[i * qd + c], k, dot[i]);
            }
            const int j = j0 + lane;
            int lo[R], hi[R], all_lo = 0, all_hi = KEYS - 1;      // the tile's keys that a row sees; that every row sees
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int pos = my_pos + i;
                lo[i] = max(0, attn_first_key(A, pos) - j0);
                hi[i] = i < mine ? min(cnt - 1, pos - j0) : -1;
                all_lo = max(all_lo, lo[i]);
                all_hi = min(all_hi, hi[i]);
                const bool seen = lane >= lo[i] && lane <= hi[i];
                const float sc = seen ? attn_score<false>(A, dot[i], pos - j, r1, r2, slope) : -INFINITY;
                const float mn = fmaxf(m[i], warp_max(sc));
                const float p = seen ? expf(sc - mn) : 0.0f, corr = mn == -INFINITY ? 1.0f : expf(m[i] - mn);
                l[i] = l[i] * corr + warp_sum(p);
                m[i] = mn;
                ps[lane * R + i] = p;
#pragma unroll
                for (int e = 0; e < MAXV; ++e) o[i][e] *= corr;
            }
            __syncwarp();
            auto add = [&](int jj, bool every) {
                float p[R];
#pragma unroll
                for (int i = 0; i < R; ++i) p[i] = ps[jj * R + i];
#pragma unroll
                for (int e = 0; e < MAXV; ++e) {
                    const int c2 = lane + 32 * e;
                    if (c2 >= A.dv) continue;
                    const float v = to_f<T>(Vs[jj * ldv + c2]);
#pragma unroll
                    for (int i = 0; i < R; ++i)
                        if (every || (jj >= lo[i] && jj <= hi[i])) o[i][e] = fmaf(p[i], v, o[i][e]);
                }
            };
            for (int jj = skip; jj < min(all_lo, cnt); ++jj) add(jj, false);
#pragma unroll 4
            for (int jj = all_lo; jj <= all_hi; ++jj) add(jj, true);
            for (int jj = max(all_lo, all_hi + 1); jj < cnt; ++jj) add(jj, false);
            __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float inv = 1.0f / l[i];
#pragma unroll
            for (int e = 0; e < MAXV; ++e) sum[i][e] = map == 0 ? o[i][e] * inv : fmaf(-A.diff_lambda, o[i][e] * inv, sum[i][e]);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (i < mine) attn_finish<T, MAXV, MAPS>(A, t0 + r0 + warp * R + i, h, lane, sum[i], out);
}

// KPL 2: a round's 64 keys are two halves, and all first halves of the range make one softmax state, all second halves another; the two are joined at the end.
// PARTS 2: a query row has two warps, a half each.  PARTS 1: one warp takes both, side by side.  The arithmetic is the same: which of the two forms a step takes
// does not show in the result.  A warp's own chain of shared-memory loads and sums bounds the kernel where every block has an SM to itself: one row at 2048
// positions of 12 heads of 64 8.2 us with two warps, 9.5 with one; with more blocks than SMs the smaller ones win (5 rows at 700, two maps of 6 heads: 16.2 against 12.4).
template <class T, int MAXV, int KPL, int PARTS>
__global__ void __launch_bounds__(256 * PARTS) attn_split_kernel(const AttnArgs A, const T* __restrict__ qbuf, const T* pool) {
    // One block per (row, key/value head x group of up to 8 of its query rows, key range); PARTS warps per query row (a query
    // head, or one of its maps: the block then stages every map's keys beside the values they share).
    // 32 * KPL keys and values at a time (KPL keys per lane) are staged in shared memory (rows padded by 16 bytes: conflict-free
    // row-per-lane reads), so that no global load sits inside the softmax / value loops.
    extern __shared__ __align__(16) unsigned char sm_raw[];
    static_assert(KPL % PARTS == 0 && KPL <= 2, "one or two states per query row");
    constexpr int kPad = 16 / (int)sizeof(T), KEYS = 32 * KPL, HV = KPL / PARTS, OWN = 32 * HV;      // keys of a round; halves, keys of a warp
    const int s = blockIdx.x / kShortSeq, r = blockIdx.x % kShortSeq;
    const int t0 = A.seq_start[s], n = A.seq_start[s + 1] - t0;
    if (n > kShortSeq || r >= n) { dep_wait(); return; }
    const int t = t0 + r, pos = A.tok_pos[t];
    // with a window the ranges are counted from the one that holds the row's first visible key
    const int j_first = attn_first_key(A, pos);
    const int range = j_first / A.split_len + blockIdx.z;
    if (range * A.split_len > pos) { dep_wait(); return; }
    const int j_lo = max(range * A.split_len, j_first);
    const int j_hi = min(pos, (range + 1) * A.split_len - 1);
    const int Gq = A.H / A.G * A.maps, nwarp = blockDim.x >> 5, nrow = nwarp / PARTS;
    const int groups = (Gq + nrow - 1) / nrow;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, own = warp % nrow, key0 = warp / nrow * OWN;
    const int g = blockIdx.y / groups, hq = (blockIdx.y % groups) * nrow + own;
    const bool active = hq < Gq;
    const int h = g * Gq + (active ? hq : 0), map = h % A.maps, head = h / A.maps;      // h: query row
    const int ldk = A.v_in_k ? (A.d + kPad + 1) / 2 * 2 : A.d + kPad, ldv = A.v_in_k ? ldk : split_value_ld<T>(A.dv);
    float* qs = reinterpret_cast<float*>(sm_raw) + warp * A.d;
    float* ps = reinterpret_cast<float*>(sm_raw) + nwarp * A.d + warp * OWN;
    T* Ks = reinterpret_cast<T*>(sm_raw + (((size_t)nwarp * (A.d + OWN) * 4 + 15) / 16) * 16);
    T* Vs = A.v_in_k ? Ks : Ks + KEYS * ldk * A.maps;
    const int32_t* bt = A.block_table + (size_t)s * A.max_pages;
    const float r1 = A.r1 ? A.r1[head] : 0.0f, r2 = A.r1 ? A.r2[head] : 0.0f, slope = A.slope ? A.slope[head] : 0.0f;
    float m[HV], l[HV];
    float o[HV][MAXV];                   // columns 2 lane + 64 (e / 2) + e % 2
#pragma unroll
    for (int x = 0; x < HV; ++x) {
        m[x] = -INFINITY;
        l[x] = 0.0f;
#pragma unroll
        for (int e = 0; e < MAXV; ++e) o[x][e] = 0.0f;
    }
    // whole 16-byte pieces when every cached row starts on a 16-byte boundary (pages are 16-byte aligned)
    const bool kvec = (A.d * sizeof(T)) % 16 == 0 && (A.k_ld * sizeof(T)) % 16 == 0 && (A.k_off * sizeof(T)) % 16 == 0;
    const bool vvec = (A.dv * sizeof(T)) % 16 == 0 && (A.v_ld * sizeof(T)) % 16 == 0 && (A.v_off * sizeof(T)) % 16 == 0;
    const int kchunk1 = kvec ? A.d / kPad : A.d, kchunks = kchunk1 * A.maps, vchunks = A.v_in_k ? 0 : (vvec ? A.dv / kPad : A.dv);
    // rows [from, to) of the round that starts at j0, on their way
    auto stage = [&](int j0, int from, int to) {
        // Where the round's rows are cached: lane r looks rows r, r + 32 up.  Then a warp per row, its lanes side by side over the
        // row's pieces (a lane keeps its piece over the rows, so that nothing is divided inside the loop).
        int page[KPL], place[KPL];
#pragma unroll
        for (int x = 0; x < KPL; ++x) {
            const int jr = min(j0 + lane + 32 * x, j_hi), pg = jr / A.page_size;
            place[x] = jr - pg * A.page_size;
            page[x] = bt[pg];
        }
        for (int c = lane; c - lane < kchunks + vchunks; c += 32) {
            const bool key = c < kchunks, mine = c < kchunks + vchunks;
            const int km = key && A.maps > 1 ? c / kchunk1 : 0, piece = key ? c - km * kchunk1 : c - kchunks;
            const int step = (key ? kvec : vvec) ? kPad : 1, ld = key ? A.k_ld : A.v_ld;
            const T* src0 = pool + (key ? A.k_off + (size_t)(g * A.maps + km) * A.page_size * ld : A.v_off + (size_t)g * A.page_size * ld) + piece * step;
            T* dst0 = (key ? Ks + km * KEYS * ldk : Vs) + piece * step;
            const int dst_ld = key ? ldk : ldv;
#pragma unroll
            for (int x = 0; x < KPL; ++x)
#pragma unroll 4
                for (int r = warp + (max(0, from - 32 * x) + nwarp - 1 - warp) / nwarp * nwarp; r < min(32, to - 32 * x); r += nwarp) {
                    const int pg = __shfl_sync(0xffffffffu, page[x], r), in_pg = __shfl_sync(0xffffffffu, place[x], r);
                    const T* src = src0 + (size_t)pg * A.page_elems + (size_t)in_pg * ld;
                    T* dst = dst0 + (r + 32 * x) * dst_ld;
                    if (!mine) continue;
                    if (step == kPad) cp_async16(dst, src);
                    else *dst = *src;
                }
        }
    };
    // The first round's rows of earlier steps do not wait for the kernel in front, which caches this step's.
    const int old = min(max(A.tok_pos[t0] - j_lo, 0), min(KEYS, j_hi - j_lo + 1));
    stage(j_lo, 0, old);
    dep_wait();
    dep_go();
    for (int c = lane; c < A.d; c += 32) qs[c] = to_f<T>(qbuf[((size_t)t * A.H * A.maps + h) * A.d + c]);
    for (int j0 = j_lo; j0 <= j_hi; j0 += KEYS) {
        const int cnt = min(KEYS, j_hi - j0 + 1);
        if (j0 > j_lo) __syncthreads();
        if (j0 > j_lo || old < cnt) stage(j0, j0 > j_lo ? 0 : old, cnt);
        cp_async_commit_group();
        cp_async_wait_group<0>();
        __syncthreads();
        if (!active) continue;
        if (key0 >= cnt) continue;
#pragma unroll
        for (int x = 0; x < HV; ++x) {
            const int row = key0 + lane + 32 * x;
            const float sc = row < cnt ? attn_score<false>(A, key_dot<T>(qs, Ks + (map * KEYS + row) * ldk, A.d), pos - (j0 + row), r1, r2, slope) : -INFINITY;
            const float mn = fmaxf(m[x], warp_max(sc)), base = mn == -INFINITY ? 0.0f : mn;      // (a half with no key yet: weights of 0)
            const float p = row < cnt ? expf(sc - base) : 0.0f, corr = expf(m[x] - base);
            ps[lane + 32 * x] = p;
            l[x] = fmaf(l[x], corr, warp_sum(p));
            m[x] = mn;
#pragma unroll
            for (int e = 0; e < MAXV; ++e) o[x][e] *= corr;
        }
        __syncwarp();
        auto add_value = [&](int x, int jj) {
            const float pj = ps[32 * x + jj];
            const T* row = Vs + (key0 + 32 * x + jj) * ldv + 2 * lane;
#pragma unroll
            for (int e = 0; e < MAXV; e += 2)
                if (2 * lane + e * 32 < A.dv) {      // an odd last column's neighbour is padding and is not stored
                    const float2 v = load_pair(row + e * 32);
                    o[x][e] = fmaf(pj, v.x, o[x][e]);
                    o[x][e + 1] = fmaf(pj, v.y, o[x][e + 1]);
                }
        };
        // keys that all of the warp's halves have, then those of the first alone; the next keys' loads go out under the current products
        const int every = min(32, max(0, cnt - key0 - 32 * (HV - 1))), first = min(32, cnt - key0);
        int jj = 0;
        for (; jj + 8 / HV <= every; jj += 8 / HV) {
#pragma unroll
            for (int u = 0; u < 8 / HV; ++u)
#pragma unroll
                for (int x = 0; x < HV; ++x) add_value(x, jj + u);
        }
        for (; jj < every; ++jj)
#pragma unroll
            for (int x = 0; x < HV; ++x) add_value(x, jj);
        if (HV > 1) {
            for (; jj + 8 <= first; jj += 8) {
#pragma unroll
                for (int u = 0; u < 8; ++u) add_value(0, jj + u);
            }
            for (; jj < first; ++jj) add_value(0, jj);
        }
        __syncwarp();
    }
    if (KPL == 2) {
        float m2 = m[HV - 1], l2 = l[HV - 1], o2[MAXV];
#pragma unroll
        for (int e = 0; e < MAXV; ++e) o2[e] = o[HV - 1][e];
        if (PARTS == 2) {
            float* other = reinterpret_cast<float*>(sm_raw) + nwarp * (A.d + OWN) + own * (MAXV * 32 + 2);      // over the staged keys
            __syncthreads();
            if (key0 > 0) {
                if (lane == 0) { other[0] = m2; other[1] = l2; }
#pragma unroll
                for (int e = 0; e < MAXV; ++e) other[2 + e * 32 + lane] = o2[e];
            }
            __syncthreads();
            if (key0 > 0) return;
            m2 = other[0];
            l2 = other[1];
#pragma unroll
            for (int e = 0; e < MAXV; ++e) o2[e] = other[2 + e * 32 + lane];
        }
        // the range has keys for its second halves: not to be read off their largest score, which passes over what is not a number
        if (j_hi - j_lo >= 32) {
            const float mn = fmaxf(m[0], m2), base = mn == -INFINITY ? 0.0f : mn, w1 = expf(m[0] - base), w2 = expf(m2 - base);
            l[0] = fmaf(l2, w2, l[0] * w1);
            m[0] = mn;
#pragma unroll
            for (int e = 0; e < MAXV; ++e) o[0][e] = fmaf(o2[e], w2, o[0][e] * w1);
        }
    }
    if (!active) return;
    float* dst = A.part + (((size_t)blockIdx.x * A.H * A.maps + h) * A.n_splits + blockIdx.z) * (A.dv + 2);
    if (lane == 0) { dst[0] = m[0]; dst[1] = l[0]; }
#pragma unroll
    for (int e = 0; e < MAXV; ++e) {
        const int c = 2 * lane + e / 2 * 64 + e % 2;
        if (c < A.dv) dst[2 + c] = o[0][e];
    }
}

// One block per (row, query head): merges the ranges of every map and joins the maps; the sink enters here, once, with no value.
// The ranges are dealt out to the block's warps (those of a map in turn), so that a row with many of them waits for global memory a
// few times only; the warps' shares are added in warp order.
constexpr int kMergeWarps = 8;      // per map
template <class T, int MAXV, int MAPS>
__global__ void __launch_bounds__(kMergeWarps * MAPS * 32) attn_merge_kernel(const AttnArgs A, T* __restrict__ out) {
    constexpr int PER = kMergeWarps, ALL = PER * MAPS;   // warps per map, of the block
    extern __shared__ float share[];                    // [ALL][dv], then [ALL] denominators
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x = blockIdx.x / A.H, h = blockIdx.x % A.H;
    const int s = x / kShortSeq, r = x % kShortSeq;
    const int t0 = A.seq_start[s], n = A.seq_start[s + 1] - t0;
    if (n > kShortSeq || r >= n) { dep_wait(); return; }
    const int t = t0 + r, pos = A.tok_pos[t];
    const int ns = pos / A.split_len - attn_first_key(A, pos) / A.split_len + 1;
    const int map = warp / PER, w0 = warp % PER;
    const float* src = A.part + (((size_t)x * A.H + h) * MAPS + map) * A.n_splits * (A.dv + 2);
    const float sink = A.sink ? A.sink[h] : -INFINITY;
    dep_wait();
    dep_go();
    float M = sink;
    for (int z = lane; z < ns; z += 32) M = fmaxf(M, src[(size_t)z * (A.dv + 2)]);
    M = warp_max(M);
    float l = 0.0f;
    float o[MAXV];
#pragma unroll
    for (int e = 0; e < MAXV; ++e) o[e] = 0.0f;
    // lane i holds the weight of this warp's range number i
    for (int z0 = w0; z0 < ns; z0 += 32 * PER) {
        const int z = z0 + lane * PER, cnt = min(32, (ns - z0 + PER - 1) / PER);
        float wz = 0.0f;
        if (z < ns) {
            const float* p = src + (size_t)z * (A.dv + 2);
            wz = expf(p[0] - M);
            l = fmaf(p[1], wz, l);
        }
#pragma unroll 4
        for (int i = 0; i < cnt; ++i) {
            const float w = __shfl_sync(0xffffffffu, wz, i);
            const float* p = src + (size_t)(z0 + i * PER) * (A.dv + 2) + 2;
#pragma unroll
            for (int e = 0; e < MAXV; ++e) {
                const int c = lane + e * 32;
                if (c < A.dv) o[e] = fmaf(p[c], w, o[e]);
            }
        }
    }
    l = warp_sum(l);
    if (lane == 0) share[ALL * A.dv + warp] = l + (w0 == 0 ? expf(sink - M) : 0.0f);
#pragma unroll
    for (int e = 0; e < MAXV; ++e) {
        const int c = lane + e * 32;
        if (c < A.dv) share[warp * A.dv + c] = o[e];
    }
    // from here on a thread per column
    constexpr int COLS = MAXV * 32 / (ALL * 32) > 1 ? MAXV * 32 / (ALL * 32) : 1;
    float gate[COLS], sum[COLS];
#pragma unroll
    for (int e = 0; e < COLS; ++e) {
        const int c = threadIdx.x + e * ALL * 32;
        gate[e] = c < A.dv ? attn_gate(A, t, h, c) : 0.0f;
    }
    __syncthreads();
    float inv[MAPS], ss = 0.0f;
#pragma unroll
    for (int mp = 0; mp < MAPS; ++mp) {
        float den = 0.0f;
#pragma unroll
        for (int w = 0; w < PER; ++w) den += share[ALL * A.dv + mp * PER + w];
        inv[mp] = (mp == 0 ? 1.0f : -A.diff_lambda) / den;
    }
#pragma unroll
    for (int e = 0; e < COLS; ++e) {
        const int c = threadIdx.x + e * ALL * 32;
        sum[e] = 0.0f;
        if (c < A.dv) {
#pragma unroll
            for (int mp = 0; mp < MAPS; ++mp) {
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < PER; ++w) v += share[(mp * PER + w) * A.dv + c];
                sum[e] = fmaf(v, inv[mp], sum[e]);
            }
        }
        ss = fmaf(sum[e], sum[e], ss);
    }
    float scale = 1.0f;
    if (MAPS == 2) {
        __shared__ float red[33];
        scale = A.diff_scale / sqrtf(block_sum(ss, red) / (float)A.dv + A.eps);
    }
#pragma unroll
    for (int e = 0; e < COLS; ++e) {
        const int c = threadIdx.x + e * ALL * 32;
        if (c < A.dv) out[(size_t)t * A.out_ld + h * A.dv + c] = from_f<T>((MAPS == 2 ? sum[e] * scale : sum[e]) * gate[e]);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Attention for prompt portions, bf16, on mma.sync m16n8k16 (fp32 accumulation): the forms that attn_flash_tc_kernel does not serve (see
// launch_flash_tc).  One block per
// (64-row tile of a sequence's rows in this step, sequence, query head); each of the four warps owns 16 rows.  Keys and
// values are staged 64 positions at a time from the paged pool into shared memory (head sizes padded with zeros to DP).
// Scores, the distance penalty, the running maximum and the softmax weights are fp32; for the weights x values product a
// weight is split into a bf16 head and a bf16 remainder (two MMAs), which keeps 16 mantissa bits of it.  The sink is
// the initial state of the running softmax: maximum = sink, denominator = 1.
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t& r0, uint32_t& r1, const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a));
}
// four 8 x 8 blocks at once (lane l gives the address of row l % 8 of block l / 8)
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// 2^x by the hardware instruction (relative error about 2^-22)
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 64 rows of `cols` bf16 into a [64][DP + 8] tile; src(row) is the row's address or nullptr (zero row).  ASYNC: whole
// 16-byte pieces of aligned rows go by cp.async (the caller commits and waits); everything else is stored directly.
template <int DP, bool ASYNC, int NTHR, class RowPtr>
__device__ __forceinline__ void stage_rows(bf16* dst, int cols, RowPtr src) {
    constexpr int LD = DP + 8;
    const bool vec = (cols % 8) == 0;
    for (int idx = threadIdx.x; idx < 64 * (DP / 8); idx += NTHR) {
        const int row = idx / (DP / 8), c = (idx % (DP / 8)) * 8;
        const bf16* p = src(row);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (p && c < cols) {
            if (vec && (reinterpret_cast<uintptr_t>(p) % 16) == 0) {
                if (ASYNC) {
                    cp_async16(dst + row * LD + c, p + c);
                    continue;
                }
                v = *reinterpret_cast<const uint4*>(p + c);
            } else {
                uint16_t hh[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) hh[e] = (c + e < cols) ? reinterpret_cast<const uint16_t*>(p)[c + e] : (uint16_t)0;
                v.x = hh[0] | ((uint32_t)hh[1] << 16); v.y = hh[2] | ((uint32_t)hh[3] << 16);
                v.z = hh[4] | ((uint32_t)hh[5] << 16); v.w = hh[6] | ((uint32_t)hh[7] << 16);
            }
        }
        *reinterpret_cast<uint4*>(dst + row * LD + c) = v;
    }
}

// The exponentials and the penalty's logarithm use the hardware approximations (relative error about 2^-22): this form
// serves bf16 only, whose products carry 2^-9.
// DK / DV: key and value sizes padded to multiples of 16.  VK: the values are the first columns of the key rows (a cached
// latent that serves as both), so only key tiles are staged and DV <= DK.
// MAPS 2 (differential attention): four warps per map, both over the one staged value tile; at the end the second map's rows
// pass through shared memory to the first map's warps, which join and finish them.
template <int DK, int DV, bool VK, int MAPS>
__global__ void __launch_bounds__(128 * MAPS) attn_flash_kernel(const AttnArgs A, const bf16* __restrict__ qbuf, const bf16* __restrict__ pool,
                                                         bf16* __restrict__ out) {
    dep_wait();
    dep_go();
    constexpr int LD = DK + 8, kTile = 64 * LD, LDV = VK ? LD : DV + 8, kTileV = 64 * LDV;
    static_assert(!VK || (DV <= DK && MAPS == 1), "values inside the key rows");
    constexpr int NTHR = 128 * MAPS;
    extern __shared__ __align__(16) unsigned char flash_smem[];      // keys [2][MAPS][64][LD], values [2][64][LDV]: two tiles in turn
    bf16* Ks = reinterpret_cast<bf16*>(flash_smem);
    bf16* Vs = VK ? Ks : Ks + 2 * MAPS * kTile;
    const int s = blockIdx.y;
    const int t0 = A.seq_start[s], n = A.seq_start[s + 1] - t0;
    const int tile = gridDim.z - 1 - blockIdx.z;      // the tiles with the most keys start first, those of every head together
    if (n <= kShortSeq || tile * 64 >= n) return;
    const int h = blockIdx.x, g = h / (A.H / A.G);
    const int map = MAPS == 1 ? 0 : threadIdx.x / 128, warp = (threadIdx.x >> 5) % 4, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const int pos0 = A.tok_pos[t0];
    const int32_t* bt = A.block_table + (size_t)s * A.max_pages;
    // queries of the tile -> A fragments
#pragma unroll
    for (int mp = 0; mp < MAPS; ++mp)
        stage_rows<DK, false, NTHR>(Ks + mp * kTile, A.d, [&](int row) -> const bf16* {
            return tile * 64 + row < n ? qbuf + (((size_t)(t0 + tile * 64 + row) * A.H + h) * MAPS + mp) * A.d : nullptr;
        });
    __syncthreads();
    uint32_t qf[DK / 16][4];
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk) {
        const bf16* p = Ks + map * kTile + (warp * 16 + gq) * LD + kk * 16 + tq * 2;
        qf[kk][0] = *reinterpret_cast<const uint32_t*>(p);
        qf[kk][1] = *reinterpret_cast<const uint32_t*>(p + 8 * LD);
        qf[kk][2] = *reinterpret_cast<const uint32_t*>(p + 8);
        qf[kk][3] = *reinterpret_cast<const uint32_t*>(p + 8 * LD + 8);
    }
    __syncthreads();
    const int row_a = tile * 64 + warp * 16 + gq, row_b = row_a + 8;
    const int i_a = pos0 + row_a, i_b = pos0 + row_b;
    const int last_pos = pos0 + min(n, tile * 64 + 64) - 1;
    const bool penalty = A.r1 != nullptr;
    const float r1 = penalty ? A.r1[h] : 0.0f, r2 = penalty ? A.r2[h] : 0.0f, sink = A.sink ? A.sink[h] : -INFINITY;
    const float slope = A.slope ? A.slope[h] : 0.0f;
    const int win = A.window > 0 ? A.window : 0x3fffffff;
    // the first key tile any row of this block sees (tiles are 64 absolute positions)
    const int j_start = attn_first_key(A, pos0 + tile * 64) / 64 * 64;
    float m_a = sink, m_b = sink, l_a = (tq == 0 && A.sink) ? 1.0f : 0.0f, l_b = l_a;
    float o[DV / 8][4];
#pragma unroll
    for (int nt = 0; nt < DV / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[nt][e] = 0.0f;
    const bool one_page = A.page_size % 64 == 0;
    // the score is the scaled product alone
    const bool plain = !penalty && !A.slope && A.softcap == 0.0f && A.window == 0 && A.scale > 0.0f;
    // the next tile of keys and values is on its way (cp.async) while the current one is multiplied
    auto stage_tile = [&](int j0, int buf) {
        // a tile within one page is looked up once, else every row for itself
        const int pg0 = j0 / A.page_size;
        const bf16* base0 = pool + (size_t)bt[pg0] * A.page_elems;
        const int in0 = j0 - pg0 * A.page_size;
        auto row_of = [&](int row, size_t off, int width, int in_head) -> const bf16* {
            const int j = j0 + row;
            if (j > last_pos) return nullptr;
            if (one_page) return base0 + off + ((size_t)in_head * A.page_size + in0 + row) * width;
            return pool + (size_t)bt[j / A.page_size] * A.page_elems + off + ((size_t)in_head * A.page_size + j % A.page_size) * width;
        };
#pragma unroll
        for (int mp = 0; mp < MAPS; ++mp)
            stage_rows<DK, true, NTHR>(Ks + (buf * MAPS + mp) * kTile, A.d, [&](int row) { return row_of(row, A.k_off, A.k_ld, g * MAPS + mp); });
        if (!VK) stage_rows<DV, true, NTHR>(Vs + buf * kTileV, A.dv, [&](int row) { return row_of(row, A.v_off, A.v_ld, g); });
        cp_async_commit_group();
    };
    stage_tile(j_start, 0);
    int buf = 0;
    for (int j0 = j_start; j0 <= last_pos; j0 += 64, buf ^= 1) {
        if (j0 + 64 <= last_pos) {
            stage_tile(j0 + 64, buf ^ 1);
            cp_async_wait_group<1>();
        } else {
            cp_async_wait_group<0>();
        }
        __syncthreads();
        const bf16* Kt = Ks + (buf * MAPS + map) * kTile;
        const bf16* Vt = Vs + buf * kTileV;
        if (j0 <= pos0 + tile * 64 + warp * 16 + 15 && j0 + 63 > pos0 + tile * 64 + warp * 16 - win) {      // this warp's rows see a key of the tile
            float S[8][4];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[nt][e] = 0.0f;
#pragma unroll
            for (int kk = 0; kk < DK / 16; ++kk)
#pragma unroll
                for (int nt = 0; nt < 8; nt += 4) {
                    uint32_t k0[4], k1[4];          // two 8-key blocks each, their 16 coordinates in two halves
                    const bf16* p = Kt + (nt * 8 + (lane & 7) + (lane >> 4) * 8) * LD + kk * 16 + ((lane >> 3) & 1) * 8;
                    ldmatrix_x4(k0, p);
                    ldmatrix_x4(k1, p + 16 * LD);
                    mma_bf16_16816(S[nt], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], k0[0], k0[1]);
                    mma_bf16_16816(S[nt + 1], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], k0[2], k0[3]);
                    mma_bf16_16816(S[nt + 2], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], k1[0], k1[1]);
                    mma_bf16_16816(S[nt + 3], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], k1[2], k1[3]);
                }
            // scores: scaled, capped, penalised and masked -- or, in a tile that every row of the warp sees whole and where the score
            // is the scaled product alone, left as they are with the scale inside the exponent
            const bool direct = plain && j0 + 63 <= pos0 + tile * 64 + warp * 16;
            float mx_a = -INFINITY, mx_b = -INFINITY;
            if (!direct) {
#pragma unroll
                for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = j0 + nt * 8 + tq * 2 + (e & 1);
                        const int i = e < 2 ? i_a : i_b;
                        S[nt][e] = (j <= i && i - j < win) ? attn_score<true>(A, S[nt][e], i - j, r1, r2, slope) : -INFINITY;
                    }
            }
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                mx_a = fmaxf(mx_a, fmaxf(S[nt][0], S[nt][1]));
                mx_b = fmaxf(mx_b, fmaxf(S[nt][2], S[nt][3]));
            }
            mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
            mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
            mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
            mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
            const float mul = direct ? A.scale : 1.0f;
            // without a sink a row of the tile's padding (beyond the sequence's rows) sees no key at all: keep its maximum finite
            const float mn_a = fmaxf(fmaxf(m_a, mx_a * mul), -1e30f), mn_b = fmaxf(fmaxf(m_b, mx_b * mul), -1e30f);
            constexpr float kLog2e = 1.4426950408889634f;
            const float ca = exp2_fast((m_a - mn_a) * kLog2e), cb = exp2_fast((m_b - mn_b) * kLog2e);
            m_a = mn_a; m_b = mn_b;
            l_a *= ca; l_b *= cb;
#pragma unroll
            for (int nt = 0; nt < DV / 8; ++nt) { o[nt][0] *= ca; o[nt][1] *= ca; o[nt][2] *= cb; o[nt][3] *= cb; }
            const float mul2 = mul * kLog2e, na = -mn_a * kLog2e, nb = -mn_b * kLog2e;
            uint32_t hi[8][2], lo[8][2];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float p0 = exp2_fast(fmaf(S[nt][0], mul2, na)), p1 = exp2_fast(fmaf(S[nt][1], mul2, na));
                const float p2 = exp2_fast(fmaf(S[nt][2], mul2, nb)), p3 = exp2_fast(fmaf(S[nt][3], mul2, nb));
                l_a += p0 + p1;
                l_b += p2 + p3;
                hi[nt][0] = pack_bf16(p0, p1);
                hi[nt][1] = pack_bf16(p2, p3);
                lo[nt][0] = pack_bf16(p0 - bf_lo(hi[nt][0]), p1 - bf_hi(hi[nt][0]));
                lo[nt][1] = pack_bf16(p2 - bf_lo(hi[nt][1]), p3 - bf_hi(hi[nt][1]));
            }
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2)
#pragma unroll
                for (int nt = 0; nt < DV / 8; nt += 4) {
                    uint32_t v0[4], v1[4];          // two 8-column blocks each; all heads of the weights first, then all remainders
                    const bf16* p = Vt + (k2 * 16 + (lane & 15)) * LDV + nt * 8 + (lane >> 4) * 8;
                    ldmatrix_x4_trans(v0, p);
                    ldmatrix_x4_trans(v1, p + 16);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const uint32_t(&w)[8][2] = x == 0 ? hi : lo;
                        mma_bf16_16816(o[nt], w[2 * k2][0], w[2 * k2][1], w[2 * k2 + 1][0], w[2 * k2 + 1][1], v0[0], v0[1]);
                        mma_bf16_16816(o[nt + 1], w[2 * k2][0], w[2 * k2][1], w[2 * k2 + 1][0], w[2 * k2 + 1][1], v0[2], v0[3]);
                        mma_bf16_16816(o[nt + 2], w[2 * k2][0], w[2 * k2][1], w[2 * k2 + 1][0], w[2 * k2 + 1][1], v1[0], v1[1]);
                        mma_bf16_16816(o[nt + 3], w[2 * k2][0], w[2 * k2][1], w[2 * k2 + 1][0], w[2 * k2 + 1][1], v1[2], v1[3]);
                    }
                }
        }
        __syncthreads();
    }
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
    float inv_a = 1.0f / l_a, inv_b = 1.0f / l_b;
    if (MAPS == 2) {
        // (the loop's last barrier has passed: the key and value tiles are free)
        constexpr int LDX = DV + 2;
        float* other = reinterpret_cast<float*>(flash_smem);       // [64][LDX]
        const int ra = warp * 16 + gq;
        if (map == 1) {
#pragma unroll
            for (int nt = 0; nt < DV / 8; ++nt) {
                *reinterpret_cast<float2*>(other + ra * LDX + nt * 8 + tq * 2) = make_float2(o[nt][0] * inv_a, o[nt][1] * inv_a);
                *reinterpret_cast<float2*>(other + (ra + 8) * LDX + nt * 8 + tq * 2) = make_float2(o[nt][2] * inv_b, o[nt][3] * inv_b);
            }
        }
        __syncthreads();
        if (map == 1) return;
        float sa = 0.0f, sb = 0.0f;
#pragma unroll
        for (int nt = 0; nt < DV / 8; ++nt) {
            const float2 xa = *reinterpret_cast<const float2*>(other + ra * LDX + nt * 8 + tq * 2);
            const float2 xb = *reinterpret_cast<const float2*>(other + (ra + 8) * LDX + nt * 8 + tq * 2);
            o[nt][0] = fmaf(-A.diff_lambda, xa.x, o[nt][0] * inv_a); o[nt][1] = fmaf(-A.diff_lambda, xa.y, o[nt][1] * inv_a);
            o[nt][2] = fmaf(-A.diff_lambda, xb.x, o[nt][2] * inv_b); o[nt][3] = fmaf(-A.diff_lambda, xb.y, o[nt][3] * inv_b);
            sa = fmaf(o[nt][0], o[nt][0], fmaf(o[nt][1], o[nt][1], sa));
            sb = fmaf(o[nt][2], o[nt][2], fmaf(o[nt][3], o[nt][3], sb));
        }
        sa += __shfl_xor_sync(0xffffffffu, sa, 1);
        sa += __shfl_xor_sync(0xffffffffu, sa, 2);
        sb += __shfl_xor_sync(0xffffffffu, sb, 1);
        sb += __shfl_xor_sync(0xffffffffu, sb, 2);
        inv_a = A.diff_scale / sqrtf(sa / (float)A.dv + A.eps);     // columns beyond dv hold zeros
        inv_b = A.diff_scale / sqrtf(sb / (float)A.dv + A.eps);
    }
#pragma unroll
    for (int nt = 0; nt < DV / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = e < 2 ? row_a : row_b, c = nt * 8 + tq * 2 + (e & 1);
            if (row < n && c < A.dv) {
                const size_t t = t0 + row;
                out[t * A.out_ld + h * A.dv + c] = __float2bfloat16_rn(o[nt][e] * (e < 2 ? inv_a : inv_b) * attn_gate(A, t, h, c));
            }
        }
}

// ---------------------------------------------------------------------------------------------------------------------
// Generalized delta rule.  proj row layout: r | k | v | gate | rate (each H*d), then the decay's inner vector [rank].
struct DeltaArgs {
    const float* proj;
    int n_in, H, d, rank, n_tokens;
    float decay_coef, unit_eps, eps;
    const float *rate_bias, *decay_w2, *decay_bias, *out_norm;
    const int32_t *seq_start, *seq_pos0, *seq_slot;
    size_t slot_floats, state_off;
    int n_slots;
    int32_t* err;
};

// Per token and channel: decay w = exp(-coef * sigmoid(w2 tanh(inner) + bias)), unit key u, removal vector a * u.
// ukey nullptr: the decay alone (the four-token scan takes the rest from the projection).
// A block takes TT tokens and blockDim.x channels: the second decay matrix (rank x HD fp32, from L2) is read once per TT tokens.
// One token per block made 2048 tokens of 12 x 64 channels and rank 64 read 400 MB of it: 84 us; eight: 27 us.
template <int TT>
__global__ void __launch_bounds__(128) delta_prep_kernel(const DeltaArgs A, float* __restrict__ decay, float* __restrict__ ukey, float* __restrict__ aukey) {
    // a lone token's share of W2 comes while the kernel in front ends: its products would wait for it eight rows at a time (6 us, 3.7 now)
    constexpr int EARLY = TT == 1 ? 64 : 1;
    float early[EARLY], early_bias = 0.0f;
    if (TT == 1) {
        const int HD = A.H * A.d, c = blockIdx.y * blockDim.x + threadIdx.x;
        if (c < HD) early_bias = A.decay_bias[c];
#pragma unroll
        for (int r = 0; r < EARLY; ++r) early[r] = r < A.rank && c < HD ? A.decay_w2[(size_t)r * HD + c] : 0.0f;
    }
    dep_wait();
    dep_go();
    extern __shared__ float th[];   // tanh(inner) [rank][TT], then 1/|k| [TT][H]
    const int t0 = blockIdx.x * TT, nt = min(TT, A.n_tokens - t0), HD = A.H * A.d;      // blockIdx.y: a slice of blockDim.x channels
    float* inv = th + A.rank * TT;
    for (int i = threadIdx.x; i < A.rank * TT; i += blockDim.x) {
        const int tt = i / A.rank, r = i - tt * A.rank;
        th[r * TT + tt] = tt < nt ? tanhf(A.proj[(size_t)(t0 + tt) * A.n_in + 5 * HD + r]) : 0.0f;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int c_lo = blockIdx.y * blockDim.x, c_hi = min(HD, c_lo + blockDim.x);      // this block's channels (gridDim.y slices cover HD)
    if (c_lo >= c_hi) return;
    const int h_lo = c_lo / A.d, nh = (c_hi - 1) / A.d - h_lo + 1;
    for (int x = warp; ukey && x < nh * nt; x += nw) {
        const int tt = x / nh, h = h_lo + x - tt * nh;
        const float* k = A.proj + (size_t)(t0 + tt) * A.n_in + HD + h * A.d;
        float ss = 0.0f;
        for (int c = lane; c < A.d; c += 32) ss += k[c] * k[c];
        ss = warp_sum(ss);
        if (lane == 0) inv[tt * A.H + h] = 1.0f / sqrtf(ss + A.unit_eps);
    }
    __syncthreads();
    const int c = c_lo + threadIdx.x;
    if (c >= c_hi) return;
    float lo[TT];
    const float bias = TT == 1 ? early_bias : A.decay_bias[c];
#pragma unroll
    for (int tt = 0; tt < TT; ++tt) lo[tt] = bias;
    if (TT == 1) {
#pragma unroll
        for (int r = 0; r < EARLY; ++r)
            if (r < A.rank) lo[0] = fmaf(early[r], th[r], lo[0]);
    }
#pragma unroll 8
    for (int r = TT == 1 ? EARLY : 0; r < A.rank; ++r) {
        const float wv = A.decay_w2[(size_t)r * HD + c];
#pragma unroll
        for (int tt = 0; tt < TT; ++tt) lo[tt] = fmaf(wv, th[r * TT + tt], lo[tt]);
    }
    const float rb = A.rate_bias[c];
#pragma unroll
    for (int tt = 0; tt < TT; ++tt)
        if (tt < nt) {
            const float* row = A.proj + (size_t)(t0 + tt) * A.n_in;
            const size_t at = (size_t)(t0 + tt) * HD + c;
            decay[at] = expf(-A.decay_coef * sigmoidf_(lo[tt]));
            if (!ukey) continue;
            const float u = row[HD + c] * inv[tt * A.H + c / A.d];
            ukey[at] = u;
            aukey[at] = sigmoidf_(row[4 * HD + c] + rb) * u;
        }
}
constexpr int kDecayTokens = 8;          // tokens per block of the decay kernels
constexpr int kDecayMinTokens = 128;     // fewer: a token per block (more blocks than the reuse is worth)

// The recurrence.  The value columns of a head's state never mix: column j follows
//   seen = sum_i u_i S_ij;   S_ij <- w_i S_ij - (a u)_i seen + k_i v_j;   o_j = sum_i S_ij r_i
// on its own.  So a head is cut into groups of CB columns, one block per (sequence, head, group), which puts a head on
// several SMs.  L adjacent lanes share a column: lane q keeps the rows 4*(e*L + q) .. +3 (e = 0 .. R/4-1, R = DK / L,
// DK >= d key channels; channels beyond d are padded with zero keys) in registers, so that the L lanes read consecutive
// 16-byte pieces of a key-channel vector, and the two sums over key channels end with log2(L) shuffles.
// Everything a token needs (r, k, u, a u, w over the key channels; v over the block's columns) is brought into shared
// memory kDeltaChunk tokens at a time with cp.async, the next chunk while the current one is computed; inside a chunk
// the next token's vectors are read into registers before the current token is computed, so the token loop waits for
// neither global nor shared memory.  The raw o goes to global memory; the kernels of lm_mechanisms.cuh that end a recurrence finish it.
constexpr int kDeltaChunk = 16;

__host__ __device__ constexpr int delta_lanes(int DK) { return DK >= 256 ? 16 : DK >= 64 ? 8 : 4; }
__host__ __device__ constexpr int delta_block_cols(int DK) { return DK * delta_lanes(DK) <= 128 ? DK : 128 / delta_lanes(DK); }
__host__ __device__ constexpr int delta_buf_floats(int DK) { return kDeltaChunk * (5 * DK + delta_block_cols(DK)); }

template <int VEC> __device__ __forceinline__ void cp_async_f(float* smem, const float* gmem);
template <> __device__ __forceinline__ void cp_async_f<1>(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(gmem));
}
template <> __device__ __forceinline__ void cp_async_f<4>(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Tokens c0 .. c0+n-1 of head h into one buffer: r | k | u | a u | w as [chunk][DK], then v of columns j0 .. j0+nc-1 as [chunk][CB].
// VEC = 4 needs d, n_in and nc to be multiples of 4 (16-byte copies).
template <int DK, int VEC>
__device__ __forceinline__ void delta_stage(const DeltaArgs& A, float* buf, int c0, int n, int h, int j0, int nc, const float* decay,
                                            const float* ukey, const float* aukey) {
    constexpr int CB = delta_block_cols(DK), PL = kDeltaChunk * DK;
    const int d = A.d, HD = A.H * d, dq = d / VEC, ncq = nc / VEC;
    for (int idx = threadIdx.x; idx < n * dq; idx += blockDim.x) {
        const int tt = idx / dq, i = (idx - tt * dq) * VEC;
        const float* prow = A.proj + (size_t)(c0 + tt) * A.n_in + h * d + i;
        const size_t vrow = (size_t)(c0 + tt) * HD + h * d + i;
        float* dst = buf + tt * DK + i;
        cp_async_f<VEC>(dst, prow);                         // r
        cp_async_f<VEC>(dst + PL, prow + HD);               // k
        cp_async_f<VEC>(dst + 2 * PL, ukey + vrow);
        cp_async_f<VEC>(dst + 3 * PL, aukey + vrow);
        cp_async_f<VEC>(dst + 4 * PL, decay + vrow);
    }
    for (int idx = threadIdx.x; idx < n * ncq; idx += blockDim.x) {
        const int tt = idx / ncq, j = (idx - tt * ncq) * VEC;
        cp_async_f<VEC>(buf + 5 * PL + tt * CB + j, A.proj + (size_t)(c0 + tt) * A.n_in + 2 * HD + h * d + j0 + j);
    }
}

// One token's vectors as a lane holds them: RV 16-byte pieces of r, k, u, a u, w and the column's v.
template <int RV>
struct DeltaToken {
    float4 r[RV], k[RV], u[RV], a[RV], w[RV];
    float v;
    __device__ __forceinline__ void load(const float4* s4, const float* s_v, int row, int row_pieces, int lanes, int plane, int cb) {
        v = s_v[row * cb];
#pragma unroll
        for (int e = 0; e < RV; ++e) {
            const float4* p = s4 + row * row_pieces + e * lanes;
            r[e] = p[0];
            k[e] = p[plane];
            u[e] = p[2 * plane];
            a[e] = p[3 * plane];
            w[e] = p[4 * plane];
        }
    }
};

template <int DK>
__global__ void __launch_bounds__(delta_block_cols(DK) * delta_lanes(DK)) delta_scan_kernel(const DeltaArgs A, const float* __restrict__ decay,
                                                                                           const float* __restrict__ ukey,
                                                                                           const float* __restrict__ aukey,
                                                                                           float* __restrict__ state_pool, float* __restrict__ o_raw) {
    constexpr int L = delta_lanes(DK), CB = delta_block_cols(DK), NS = DK / CB, RV = DK / L / 4, PL = kDeltaChunk * DK;
    constexpr int kBuf = delta_buf_floats(DK);
    static_assert(DK % (4 * L) == 0, "every lane owns whole 16-byte pieces");
    extern __shared__ __align__(16) float sh[];
    const int d = A.d, HD = A.H * d;
    const int group = blockIdx.x % NS, sh_id = blockIdx.x / NS;
    const int seq = sh_id / A.H, h = sh_id % A.H;
    const int j0 = group * CB;
    if (j0 >= d) { dep_wait(); return; }          // a group of padded columns only
    const int nc = min(CB, d - j0);
    const int col = threadIdx.x / L, q = threadIdx.x % L, j = j0 + col;
    const int t0 = A.seq_start[seq], t1 = A.seq_start[seq + 1];
    const int slot = A.seq_slot[seq];
    if (slot < 0 || slot >= A.n_slots) {
        if (threadIdx.x == 0) atomicExch(A.err, 2);
        dep_wait();
        return;
    }
    const bool vec = (d % 4 == 0) && (A.n_in % 4 == 0);
    if (d < DK || nc < CB) {                      // padded channels and columns stay zero for good
        for (int i = threadIdx.x; i < 2 * kBuf; i += blockDim.x) sh[i] = 0.0f;
        __syncthreads();
    }
    float* st = state_pool + (size_t)slot * A.slot_floats + A.state_off + (size_t)h * d * d;
    float S[RV][4];
    const bool fresh = A.seq_pos0[seq] == 0;
#pragma unroll
    for (int e = 0; e < RV; ++e)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * (e * L + q) + x;
            S[e][x] = (!fresh && i < d && j < d) ? st[(size_t)i * d + j] : 0.0f;
        }
    dep_wait();
    dep_go();
    if (vec) delta_stage<DK, 4>(A, sh, t0, min(kDeltaChunk, t1 - t0), h, j0, nc, decay, ukey, aukey);
    else delta_stage<DK, 1>(A, sh, t0, min(kDeltaChunk, t1 - t0), h, j0, nc, decay, ukey, aukey);
    cp_async_commit();
    float po = 0.0f;                              // this lane's share of the previous token's o
    int cur = 0;
    for (int c0 = t0; c0 < t1; c0 += kDeltaChunk, cur ^= 1) {
        const int n = min(kDeltaChunk, t1 - c0);
        cp_async_wait<0>();
        __syncthreads();                          // this chunk has landed; every thread is done with the other buffer
        if (c0 + kDeltaChunk < t1) {
            const int nn = min(kDeltaChunk, t1 - c0 - kDeltaChunk);
            if (vec) delta_stage<DK, 4>(A, sh + (cur ^ 1) * kBuf, c0 + kDeltaChunk, nn, h, j0, nc, decay, ukey, aukey);
            else delta_stage<DK, 1>(A, sh + (cur ^ 1) * kBuf, c0 + kDeltaChunk, nn, h, j0, nc, decay, ukey, aukey);
            cp_async_commit();
        }
        const float* b = sh + cur * kBuf;
        const float4* s4 = reinterpret_cast<const float4*>(b) + q;      // piece e of a vector of token tt: s4[(tt*DK)/4 + e*L]
        const float* s_v = b + 5 * PL + col;
        // two register sets take turns: while one token is computed from one set, the next token's vectors land in the other
        DeltaToken<RV> ta, tb;
        ta.load(s4, s_v, 0, DK / 4, L, PL / 4, CB);
        auto step = [&](const DeltaToken<RV>& c, int tt) {
            float sa = 0.0f, sb = 0.0f;
#pragma unroll
            for (int e = 0; e < RV; ++e) {
                sa = fmaf(c.u[e].x, S[e][0], sa);
                sb = fmaf(c.u[e].y, S[e][1], sb);
                sa = fmaf(c.u[e].z, S[e][2], sa);
                sb = fmaf(c.u[e].w, S[e][3], sb);
            }
            float seen = sa + sb;
            // this token's `seen` and the previous token's o go through the shuffle stages side by side
#pragma unroll
            for (int s = 1; s < L; s <<= 1) {
                const float x = __shfl_xor_sync(0xffffffffu, seen, s), y = __shfl_xor_sync(0xffffffffu, po, s);
                seen += x;
                po += y;
            }
            if (q == 0 && j < d && c0 + tt > t0) o_raw[(size_t)(c0 + tt - 1) * HD + h * d + j] = po;
            const float ns = -seen;
            sa = 0.0f;
            sb = 0.0f;
#pragma unroll
            for (int e = 0; e < RV; ++e) {
                S[e][0] = fmaf(c.a[e].x, ns, fmaf(c.w[e].x, S[e][0], c.k[e].x * c.v));
                S[e][1] = fmaf(c.a[e].y, ns, fmaf(c.w[e].y, S[e][1], c.k[e].y * c.v));
                S[e][2] = fmaf(c.a[e].z, ns, fmaf(c.w[e].z, S[e][2], c.k[e].z * c.v));
                S[e][3] = fmaf(c.a[e].w, ns, fmaf(c.w[e].w, S[e][3], c.k[e].w * c.v));
                sa = fmaf(S[e][0], c.r[e].x, sa);
                sb = fmaf(S[e][1], c.r[e].y, sb);
                sa = fmaf(S[e][2], c.r[e].z, sa);
                sb = fmaf(S[e][3], c.r[e].w, sb);
            }
            po = sa + sb;
        };
        for (int tt = 0; tt < n; tt += 2) {
            tb.load(s4, s_v, min(tt + 1, kDeltaChunk - 1), DK / 4, L, PL / 4, CB);      // a row after the last is read and dropped
            step(ta, tt);
            if (tt + 1 < n) {
                ta.load(s4, s_v, min(tt + 2, kDeltaChunk - 1), DK / 4, L, PL / 4, CB);
                step(tb, tt + 1);
            }
        }
    }
#pragma unroll
    for (int s = 1; s < L; s <<= 1) po += __shfl_xor_sync(0xffffffffu, po, s);
    if (q == 0 && j < d && t1 > t0) o_raw[(size_t)(t1 - 1) * HD + h * d + j] = po;
#pragma unroll
    for (int e = 0; e < RV; ++e)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * (e * L + q) + x;
            if (i < d && j < d) st[(size_t)i * d + j] = S[e][x];
        }
}

// ---------------------------------------------------------------------------------------------------------------------
// Sampling: the library's integer-weight sampler, one block per row.
template <int PER>
__global__ void __launch_bounds__(kThreads) lm_sample_kernel(const float* __restrict__ logits, int n, int rows, float temp, int top_k,
                                                             float top_p, float min_p, unsigned long long seed,
                                                             const int32_t* __restrict__ seq_id, const int32_t* __restrict__ step,
                                                             int32_t* __restrict__ out) {
    dep_wait();
    dep_go();
    extern __shared__ __align__(16) float lg[];
    __shared__ SampleScratch sc;
    for (int b = blockIdx.x; b < rows; b += gridDim.x) {
        for (int i = threadIdx.x; i < n; i += kThreads) lg[i] = logits[(size_t)b * n + i];
        __syncthreads();
        const int tok = sample_row<kThreads, PER>(lg, n, temp, top_k, top_p, min_p, seed, step ? (uint32_t)step[b] : 0u,
                                                  seq_id ? (uint32_t)seq_id[b] : (uint32_t)b, 0u, sc);
        if (threadIdx.x == 0) out[b] = tok;
        __syncthreads();
    }
}

}  // namespace lm
}  // namespace smol

#include "lm_flash_tc.cuh"
#include "lm_mechanisms.cuh"
#include "lm_sigmoid_linear.cuh"
#include "lm_delta_mlstm.cuh"
#include "lm_quad_scan.cuh"
#include "lm_chunk_scan.cuh"

// =====================================================================================================================
// Host side
using namespace smol::lm;
using smol::bf16;

static thread_local std::string g_err;
static int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}
#define CU(expr)                                                                                  \
    do {                                                                                          \
        cudaError_t e_ = (expr);                                                                  \
        if (e_ != cudaSuccess) return fail(SMOL_ERR_CUDA, std::string(#expr ": ") + cudaGetErrorString(e_)); \
    } while (0)

struct RunInfo {
    int layer;
    size_t k_off = 0, v_off = 0;   // attention: element offsets inside a page
    size_t state_off = 0;          // recurrent: float offset inside a slot
    size_t freq_off = 0;           // latent attention: float offset of the run's rotation frequencies in the table
    size_t conv_off = 0;           // state-space, gated delta: float offset of the convolution's last inputs inside a slot
    size_t unit_off = 0, m_off = 0;   // mLSTM: float offsets of the key sums and the running maxima inside a slot
    int flags = 0;                 // SMOL_LM_RUN_*
};

struct SmolLm {
    SmolLmConfig cfg;
    std::vector<SmolLmLayer> layers;
    std::vector<SmolLmLayer> sides;       // sides[i]: the mixer beside layer i's (layers[i].side points here, or is null)
    std::vector<RunInfo> runs;
    std::vector<RunInfo> side_runs;       // the cache / state placement of a run's side mixer
    size_t o_conv = 0, o_head = 0;        // state-space: convolved channels [T][channels], per-head decay and step [2][T][heads]
    int max_conv = 0, max_ssd_heads = 0;
    size_t o_rec = 0, max_rec = 0, max_quad = 0;      // prompts' scans: records of a chunk, of a group over all heads [floats]
    size_t o_pairs = 0;                   // four-token scan: products between a group's queries and keys
    int max_pair_heads = 0;
    SmolLmGlobals g{};
    size_t page_elems = 0, slot_floats = 0, esize = 2;
    int max_in = 0, max_mix = 0, max_ff = 0, max_hd = 0, max_q = 0;
    bool any_restart = false, any_own_proj = false, any_merge = false;
    // workspace carving (byte offsets)
    size_t o_x, o_hn, o_proj, o_mix, o_y, o_z, o_act, o_dec, o_u, o_au, o_oraw, o_q, o_hw, o_err, o_part, total;
    // post-norm block: every layer result of the step; latent attention: query latent (T), full query (fp32 and T), query in
    // latent space (fp32), rotation frequencies; routed feed-forward: choices, sorted order, tile table, per-pair buffers
    size_t o_hist = 0, o_cq = 0, o_qf = 0, o_freq = 0;
    size_t o_x0 = 0, o_mix2 = 0, o_y2 = 0, o_spart = 0, o_cat = 0;
    int max_sig_cols = 0;                     // sigmoid attention: widest heads * vdim (partial sums of the tiled kernel's key ranges)    // pre-norm block: the embedding output; mixers with their own output projections: the second result
    size_t o_rlogits = 0, o_rdone = 0, o_ap = 0, o_sel_id = 0, o_sel_w = 0, o_perm = 0, o_slot_of = 0, o_seg = 0, o_tile_g = 0, o_tile_r = 0, o_ntiles = 0, o_zp = 0, o_actp = 0, o_yp = 0;
    int max_routed = 0, max_cq = 0, max_qf = 0, max_top = 0, max_experts = 0, max_pair_ff = 0;
    std::vector<float> freq_table;
    int split_len = 256, max_splits = 1, max_heads = 1, max_vdim = 1;
    char* ws = nullptr;
    void* pages = nullptr;
    float* slots = nullptr;
    int n_pages = 0, n_slots = 0;
    bool bound = false;
    bool tc_ready = false;      // the tcgen05 matrix product may be launched (attribute set, driver entry point found)
    int n_sms = 1;
    int64_t launches = 0;
    // small steps (decoding) are captured once per shape into a CUDA graph and replayed
    struct Captured { SmolLmStep key; cudaGraphExec_t exec; int64_t launches; };
    std::vector<Captured> graphs;
    cudaStream_t cap_stream = nullptr;
    // parallel block: the feed-forward runs on its own stream beside the mixer, between these two events; output-norm block: a side
    // mixer beside the layer's own
    cudaStream_t ff_stream = nullptr;
    cudaEvent_t ff_start = nullptr, ff_done = nullptr;
    ~SmolLm() {
        if (ff_start) cudaEventDestroy(ff_start);
        if (ff_done) cudaEventDestroy(ff_done);
        if (ff_stream) cudaStreamDestroy(ff_stream);
        for (auto& g : graphs) cudaGraphExecDestroy(g.exec);
        if (cap_stream) cudaStreamDestroy(cap_stream);
    }
};

constexpr int kAttnSplitSmemMax = 200 * 1024;      // shared memory the few-token attention may ask for
constexpr int kAttnSplitWideSmem = 64 * 1024;      // ... and up to which it takes 64 keys at a time instead of 32

static size_t al256(size_t v) { return (v + 255) / 256 * 256; }

// softmax attention: score maps per head, and the rows of q, k and v in the input projection
static int maps_of(const SmolLmLayer& L) { return L.n_maps > 1 ? L.n_maps : 1; }
static int attn_qkv_rows(const SmolLmLayer& L) {
    return L.heads * maps_of(L) * L.dim + (L.kv_from > 0 ? 0 : L.kv_heads * (maps_of(L) * L.dim + L.vdim));
}
static int n_in_of(const SmolLmLayer& L) {
    if (L.mixer == SMOL_LM_MIX_SINK_ATTENTION) return attn_qkv_rows(L) + (L.no_gate ? 0 : L.heads * L.vdim);
    if (L.mixer == SMOL_LM_MIX_GATED_DELTA) return 2 * L.kv_heads * L.dim + 2 * L.heads * L.vdim + 2 * L.heads;
    if (L.mixer == SMOL_LM_MIX_MLSTM) return 2 * L.heads * L.dim + 2 * L.heads * L.vdim + 2 * L.heads;
    if (L.mixer == SMOL_LM_MIX_STATE_SPACE) return 2 * L.heads * L.vdim + 2 * L.bc_groups * L.n_state + L.heads;
    if (L.mixer == SMOL_LM_MIX_LATENT_ATTENTION) return L.q_rank + L.kv_rank + L.rot_dim + L.heads;
    if (L.mixer == SMOL_LM_MIX_GATED_LINEAR) return 2 * L.heads * L.dim + 2 * L.heads * L.vdim + L.rank;
    if (L.mixer == SMOL_LM_MIX_SIGMOID_ATTENTION) return L.heads * L.dim + L.kv_heads * L.dim + L.heads;
    if (L.mixer == SMOL_LM_MIX_LIGHTNING || L.mixer == SMOL_LM_MIX_RETENTION) return 2 * L.heads * L.dim + 2 * L.heads * L.vdim;
    if (L.mixer == SMOL_LM_MIX_HGRN2) return 2 * L.heads * L.dim + L.heads * L.vdim;
    return 5 * L.heads * L.dim + L.rank;
}

// columns a mixer hands to the output projection
static int mix_cols_of(const SmolLmLayer& L) { return L.mixer == SMOL_LM_MIX_GENERAL_DELTA ? L.heads * L.dim : L.heads * L.vdim; }
static bool pairable(const SmolLmLayer& L) {
    return L.mixer == SMOL_LM_MIX_SINK_ATTENTION || L.mixer == SMOL_LM_MIX_STATE_SPACE || L.mixer == SMOL_LM_MIX_SIGMOID_ATTENTION ||
           L.mixer == SMOL_LM_MIX_LIGHTNING || L.mixer == SMOL_LM_MIX_RETENTION || L.mixer == SMOL_LM_MIX_GATED_DELTA || L.mixer == SMOL_LM_MIX_MLSTM;
}
// Parallel block: the rows of the fused input projection that serve the feed-forward (shared expert's gate and up, router, shared
// gate), and the projection's whole height (a multiple of 8).
static int ff_rows_of(const SmolLmLayer& L) {
    return L.mlp == SMOL_LM_MLP_EXPERTS ? (L.ff_plain ? 1 : 2) * L.shared_ff + L.n_experts + L.n_identity + (L.shared_gate ? 1 : 0) : 0;
}
static int parallel_n_in_of(const SmolLmLayer& L) { return (n_in_of(L) + ff_rows_of(L) + 7) / 8 * 8; }
// Height of a layer's fused input projection.
static int full_n_in_of(const SmolLmLayer& L, int block) {
    if (block == SMOL_LM_BLOCK_PARALLEL) return parallel_n_in_of(L);
    const int n = n_in_of(L) + (L.side ? n_in_of(*L.side) : 0);
    return block == SMOL_LM_BLOCK_OUTNORM ? (n + 7) / 8 * 8 : n;
}
// base^(-2i/dims) for the dims/2 rotated pairs of a rotating mixer, stretched band by band when L.rot_stretch is set,
// interpolated along a ramp when L.rot_yarn is (see the header)
static void push_frequencies(std::vector<float>& table, const SmolLmLayer& L, bool stretch) {
    const double two_pi = 6.283185307179586476925286766559;
    for (int i = 0; i < L.rot_dims / 2; ++i) {
        double f = pow((double)L.rot_base, -2.0 * i / (double)L.rot_dims);
        if (stretch && L.rot_stretch != 0.0f) {
            const double wl = two_pi / f, orig = L.rot_original;
            if (wl > orig / L.rot_low) {
                f = f / L.rot_stretch;
            } else if (wl >= orig / L.rot_high) {
                const double b = (orig / wl - L.rot_low) / ((double)L.rot_high - L.rot_low);
                f = (1.0 - b) * f / L.rot_stretch + b * f;
            }
        }
        if (L.rot_yarn > 0.0f) {
            auto dim_of = [&](double turns) { return L.rot_dims * log(L.rot_original / (two_pi * turns)) / (2.0 * log((double)L.rot_base)); };
            const double lo = std::max(floor(dim_of(L.rot_fast)), 0.0), hi = std::min(ceil(dim_of(L.rot_slow)), L.rot_dims - 1.0);
            const double ramp = std::min(std::max((i - lo) / std::max(hi - lo, 0.001), 0.0), 1.0);
            f = f / L.rot_yarn * ramp + f * (1.0 - ramp);
        }
        table.push_back((float)f);
    }
}

extern "C" int smol_lm_abi_version(void) { return SMOL_LM_ABI_VERSION; }
extern "C" size_t smol_lm_struct_bytes(int which) {
    return which == 0 ? sizeof(SmolLmLayer) : which == 1 ? sizeof(SmolLmConfig) : which == 2 ? sizeof(SmolLmGlobals) : which == 3 ? sizeof(SmolLmStep) : 0;
}
extern "C" const char* smol_lm_last_error(void) { return g_err.c_str(); }

// The four-token scan over a step in which some sequence brings at least kQuadMinTokens tokens, kQuadMeanTokens in the mean (fewer: its two
// launches and the records of single tokens cost more than the chain they shorten).  One layer of 12 x 64 x 64 as a whole, generalized delta rule,
// 16 / 24 / 40 / 300 / 1200 tokens: 61 / 68 / 166 / 142 / 275 us against 56 / 65 / 165 / 166 / 370; the two scans alone, 17 tokens
// beside 15 / 63 single ones: 28 / 67 us against 11 / 20.
static bool quad_pays(int n_seqs, int n_tokens, int max_n) { return max_n >= kQuadMinTokens && n_tokens >= kQuadMeanTokens * n_seqs; }
// The scan by chunks, or one of those that go four tokens at a time.  By chunks a sequence must be long enough to pay for its records, and a step's blocks of eight
// columns must not be many more than the SMs run at once: then either form fills them, and the one with less to do wins -- the more so the fewer channels a head has,
// since chunks pad to 32; just above what runs at once a nearly empty second wave costs most.  Time by chunks over the other form's, records included, from 1 to 128
// heads, 1 to 16 sequences, 144 to 1000 tokens (blocks per SM in brackets):
//   generalized delta rule: 0.45 to 0.79 with 64 channels; 16 [1.5] 0.82, [1.7] 1.03; 128, 144 / 160 tokens [0.9] 1.04 / 0.95, otherwise 0.60 to 0.83
//   one decay per head: 64 [2.0] 0.92, [2.6] 1.06, [3] and more 0.66 to 0.98; 48 x 24 [1.9] 0.92, [2.4] 1.19; 32 x 32 [5.2] 0.97, [13.8] 1.14; 16 [1.5] 0.88, [1.6] 1.04; above 64, 144 tokens 0.64 to 1.00
//   decays per channel: 64 [1.9] 0.95, [2.6] 1.13, [4] 1.10, 64 x 128 [5] and more 0.80 to 1.00; 48 x 24 [1.5] 1.00, [1.9] 1.10; 32 x 32 [1.5] 0.96, [2.0] 1.05, 32 x 128 0.79 to 0.99; 16 [1.0] 0.99,
//     [1.3] 1.08; 128, 144 / 176 / 208 tokens [0.9] 1.18 / 1.10 / 0.99, otherwise 0.75 to 1.01
//   gated delta rule: 64 [3.5] 0.95, [5.2] 1.07; 48 x 24 [1.9] 0.87, [2.6] 1.13; 32 [2.6] 0.94, [3.2] 1.11; 16 [1.0] 0.92, [1.3] 1.08; 128, 176 / 208 tokens 1.06 / 0.99; 256, 256 / 320
//     tokens 1.03 / 0.96, but [2.6], where blocks of two leave a third of them for a second wave, 1.20 / 1.14
//   mLSTM: 64 0.40 to 0.95; 48 x 24 [4.1] 0.79, [5.2] 1.06; 32 [8.3] 0.99; 16 [1.9] 0.92, [2.6] 1.08
static bool chunks_pay(int kind, bool unit, int n_seqs, int heads, int n_tokens, int max_n, int d, int columns, int n_sms) {
    if (n_tokens < kQuadMeanTokens * n_seqs) return false;
    const double blocks = (double)n_seqs * heads * chunk_blocks(columns) / n_sms;      // per SM
    const bool wave = blocks <= 2.0 || blocks > 3.0;                                   // (64 channels: an SM runs two)
    if (kind == kScanGeneralDelta) {
        const int min_n = d <= 64 ? 256 : blocks > 0.8 && blocks <= 0.9 ? 160 : 144;
        return max_n >= min_n && (d > 16 || blocks <= 1.5);
    }
    if (kind == kScanGatedDelta) {
        if (max_n < (d <= 64 ? 256 : d <= 128 ? 208 : 320)) return false;
        return d > 128 ? blocks <= 2.0 || blocks >= 5.0 : d > 64 || blocks <= (d <= 16 ? 1.0 : d < 64 ? 2.0 : 3.5);
    }
    if (unit) return max_n >= (d <= 64 ? 256 : 208) && (d >= 64 || blocks <= (d <= 16 ? 2.0 : 4.0));
    if (kind == kScanHeadDecay) return max_n >= (d <= 64 ? 256 : 144) && (d > 64 || (d == 64 ? wave : blocks <= (d <= 16 ? 1.5 : d <= 32 ? 5.0 : 2.0)));
    if (d > 64) return max_n >= (blocks > 0.75 && blocks <= 1.2 ? 208 : 144);
    if (max_n < 256) return false;
    if (d > 16 && columns >= 2 * d) return d <= 32 || wave;
    return blocks <= (d <= 16 ? 1.0 : d < 64 ? 1.5 : 2.0);
}

extern "C" int smol_lm_create(const SmolLmConfig* cfg, const SmolLmLayer* layers, const int32_t* run_layer, SmolLm** out) {
    if (!cfg || !layers || !run_layer || !out) return fail(SMOL_ERR_INVALID, "smol_lm_create: null argument");
    if (cfg->dtype != SMOL_LM_BF16 && cfg->dtype != SMOL_LM_F32) return fail(SMOL_ERR_INVALID, "dtype must be 0 (bf16) or 1 (f32)");
    if (cfg->vocab < 1 || cfg->width < 1 || cfg->n_layers < 1 || cfg->n_runs < 1 || cfg->page_size < 1 || cfg->max_step_tokens < 1 ||
        cfg->max_step_seqs < 1 || cfg->max_want < 1 || cfg->max_context < 1)
        return fail(SMOL_ERR_INVALID, "smol_lm_create: sizes must be positive");
    SmolLm* m = new SmolLm();
    m->cfg = *cfg;
    m->cfg.run_flags = nullptr;      // the caller's array is read below and not kept
    m->esize = cfg->dtype == SMOL_LM_F32 ? 4 : 2;
    m->layers.assign(layers, layers + cfg->n_layers);
    m->sides.resize(cfg->n_layers);
    for (int i = 0; i < cfg->n_layers; ++i)
        if (m->layers[i].side) {
            m->sides[i] = *m->layers[i].side;
            m->sides[i].side = nullptr;
            m->layers[i].side = &m->sides[i];
        }
    // places one mixer's cache or state in the pools and widens the workspace for it; returns 0 or an error code
    auto place = [&](const SmolLmLayer& L, RunInfo& r) -> int {
        if (L.heads < 1 || (L.dim < 1 && L.mixer != SMOL_LM_MIX_STATE_SPACE)) return fail(SMOL_ERR_INVALID, "a layer needs heads >= 1 and dim >= 1");
        if (L.in_bias && !pairable(L)) return fail(SMOL_ERR_UNSUPPORTED, "in_bias: softmax attention and the state-space recurrence only");
        if (L.mixer == SMOL_LM_MIX_SINK_ATTENTION) {
            if (L.kv_heads < 1 || L.heads % L.kv_heads != 0 || L.vdim < 1) return fail(SMOL_ERR_INVALID, "attention: heads must be a multiple of kv_heads");
            if (L.vdim > 32 * kAttnMaxV) return fail(SMOL_ERR_UNSUPPORTED, "attention: value size above 512");
            if (L.window < 0 || L.softcap < 0.0f || L.q_temp_every < 0.0f) return fail(SMOL_ERR_INVALID, "attention: window, softcap and q_temp_every must not be negative");
            if (!L.q_norm != !L.k_norm || (L.norm_whole && !L.q_norm)) return fail(SMOL_ERR_INVALID, "attention: q_norm and k_norm come together, norm_whole needs them");
            const int maps = maps_of(L);
            if (maps > 2 || (maps == 2 && (L.norm_whole || L.sink))) return fail(SMOL_ERR_UNSUPPORTED, "attention: at most two maps, norms per map and no sink with two");
            if (L.rot_dims < 0 || L.rot_dims > L.dim || L.rot_dims % 2) return fail(SMOL_ERR_INVALID, "attention: rot_dims even and at most dim");
            if (L.rot_dims > 0 && (!L.norm_whole || L.rot_dims > 2 * kMaxRotPairs)) return fail(SMOL_ERR_UNSUPPORTED, "attention: rotation needs norm_whole and at most 512 coordinates");
            const size_t split_smem = ((size_t)std::min(L.heads / L.kv_heads * maps, 8) * (L.dim + 32) * 4 + 15) / 16 * 16 +
                                      (size_t)32 * (maps * (L.dim + 16 / m->esize + 1) + L.vdim + 16 / m->esize + 1) * m->esize;
            if (split_smem > (size_t)kAttnSplitSmemMax) return fail(SMOL_ERR_UNSUPPORTED, "attention: key and value sizes need more shared memory than an SM has");
            if (L.kv_from > 0) {
                // another layer's cache, as its latest run leaves it
                const RunInfo* lender = nullptr;
                for (const RunInfo& o : m->runs)
                    if (o.layer == L.kv_from - 1) lender = &o;
                if (!lender) return fail(SMOL_ERR_INVALID, "attention: kv_from must name an earlier layer");
                const SmolLmLayer& O = m->layers[lender->layer];
                if (O.mixer != L.mixer || O.kv_from > 0 || O.kv_heads != L.kv_heads || O.dim != L.dim || O.vdim != L.vdim || maps_of(O) != maps || L.norm_whole)
                    return fail(SMOL_ERR_INVALID, "attention: kv_from must name an attention layer with own keys and values and the same sizes");
                r.k_off = lender->k_off;
                r.v_off = lender->v_off;
            } else {
                r.k_off = m->page_elems;
                r.v_off = r.k_off + (size_t)L.kv_heads * maps * cfg->page_size * L.dim;
                m->page_elems = r.v_off + (size_t)L.kv_heads * cfg->page_size * L.vdim;
            }
            r.freq_off = m->freq_table.size();
            push_frequencies(m->freq_table, L, true);
            m->max_q = std::max(m->max_q, L.heads * maps * L.dim);
            m->max_heads = std::max(m->max_heads, L.heads * maps);
            m->max_vdim = std::max(m->max_vdim, L.vdim);
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
        } else if (L.mixer == SMOL_LM_MIX_GATED_DELTA) {
            if (L.dim > 256 || L.conv_taps > kMaxTaps) return fail(SMOL_ERR_UNSUPPORTED, "gated delta rule: key size above 256 or more than 16 taps");
            if (L.vdim < 1 || L.kv_heads < 1 || L.heads % L.kv_heads != 0 || L.conv_taps < 1 || !L.conv_w || !L.a_log || !L.dt_bias || !L.out_norm)
                return fail(SMOL_ERR_INVALID, "gated delta rule: heads must be a multiple of kv_heads, vdim and taps positive, conv_w, a_log, dt_bias and out_norm set");
            const int ch = 2 * L.kv_heads * L.dim + L.heads * L.vdim;
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.vdim;
            r.conv_off = m->slot_floats;
            m->slot_floats += (size_t)(L.conv_taps - 1) * ch;
            m->slot_floats = (m->slot_floats + 3) / 4 * 4;
            m->max_hd = std::max(m->max_hd, L.heads * L.vdim);
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
            m->max_conv = std::max(m->max_conv, ch);
            m->max_ssd_heads = std::max(m->max_ssd_heads, L.heads);        // decay and step
            m->max_pair_heads = std::max(m->max_pair_heads, L.kv_heads);
        } else if (L.mixer == SMOL_LM_MIX_MLSTM) {
            if (L.dim > 256) return fail(SMOL_ERR_UNSUPPORTED, "recurrent mixer: key size above 256");
            if (L.vdim < 1 || !(L.gate_cap > 0.0f) || !L.rate_bias || !L.decay_bias || !L.out_norm)
                return fail(SMOL_ERR_INVALID, "mLSTM: vdim and gate_cap must be positive, rate_bias, decay_bias and out_norm set");
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.vdim;
            r.unit_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim;
            r.m_off = m->slot_floats;
            m->slot_floats += L.heads;
            m->slot_floats = (m->slot_floats + 3) / 4 * 4;
            m->max_hd = std::max(m->max_hd, L.heads * L.vdim);
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
            m->max_conv = std::max(m->max_conv, 1);
            m->max_ssd_heads = std::max(m->max_ssd_heads, 2 * L.heads);        // decay and write weight, floor, key sum . query
            m->max_pair_heads = std::max(m->max_pair_heads, L.heads);
        } else if (L.mixer == SMOL_LM_MIX_STATE_SPACE) {
            if (L.vdim < 1 || L.n_state < 1 || L.bc_groups < 1 || L.heads % L.bc_groups != 0 || L.conv_taps < 1 || L.norm_parts < 1 ||
                (L.heads * L.vdim) % L.norm_parts != 0)
                return fail(SMOL_ERR_INVALID, "state-space: heads must be a multiple of bc_groups, heads * vdim of norm_parts");
            if (L.n_state > 256 || L.conv_taps > kMaxTaps) return fail(SMOL_ERR_UNSUPPORTED, "state-space: state size above 256 or more than 16 taps");
            const int ch = L.heads * L.vdim + 2 * L.bc_groups * L.n_state;
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.n_state * L.vdim;
            r.conv_off = m->slot_floats;
            m->slot_floats += (size_t)(L.conv_taps - 1) * ch;
            m->slot_floats = (m->slot_floats + 3) / 4 * 4;          // the next state starts on a 16-byte boundary
            m->max_hd = std::max(m->max_hd, L.heads * L.vdim);
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
            m->max_conv = std::max(m->max_conv, ch);
            m->max_ssd_heads = std::max(m->max_ssd_heads, L.heads);
        } else if (L.mixer == SMOL_LM_MIX_GENERAL_DELTA) {
            if (L.dim > 256) return fail(SMOL_ERR_UNSUPPORTED, "recurrent mixer: key size above 256");
            if (L.rank < 1) return fail(SMOL_ERR_INVALID, "recurrent mixer: rank must be positive");
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.dim;
            m->max_hd = std::max(m->max_hd, L.heads * L.dim);
            m->max_mix = std::max(m->max_mix, L.heads * L.dim);
        } else if (L.mixer == SMOL_LM_MIX_LATENT_ATTENTION) {
            if (L.vdim < 1 || L.q_rank < 1 || L.kv_rank < 1 || L.rot_dim < 0 || L.rot_dims < 0 || L.rot_dims > L.rot_dim || L.rot_dims % 2)
                return fail(SMOL_ERR_INVALID, "latent attention: vdim, q_rank, kv_rank must be positive, rot_dims even and at most rot_dim");
            if (L.kv_rank > 32 * kAttnMaxV) return fail(SMOL_ERR_UNSUPPORTED, "latent attention: latent size above 512");
            // a cached position: the latent, then the shared rotated key part; keys and values are the same row
            r.k_off = r.v_off = m->page_elems;
            m->page_elems += (size_t)cfg->page_size * (L.kv_rank + L.rot_dim);
            r.freq_off = m->freq_table.size();
            push_frequencies(m->freq_table, L, true);
            m->max_q = std::max(m->max_q, L.heads * (L.kv_rank + L.rot_dim));
            m->max_heads = std::max(m->max_heads, L.heads);
            m->max_vdim = std::max(m->max_vdim, L.kv_rank);
            m->max_mix = std::max(m->max_mix, L.heads * std::max(L.kv_rank, L.vdim));
            m->max_hd = std::max(m->max_hd, L.heads * L.vdim);
            m->max_cq = std::max(m->max_cq, L.q_rank);
            m->max_qf = std::max(m->max_qf, L.heads * (L.dim + L.rot_dim));
        } else if (L.mixer == SMOL_LM_MIX_SIGMOID_ATTENTION) {
            if (L.kv_heads < 1 || L.heads % L.kv_heads != 0 || L.vdim != L.dim) return fail(SMOL_ERR_INVALID, "sigmoid attention: heads must be a multiple of kv_heads and vdim equal to dim");
            if (L.heads > kSigmoidMaxHeads || L.vdim > 32 * kAttnMaxV) return fail(SMOL_ERR_UNSUPPORTED, "sigmoid attention: more than 32 heads or a head size above 512");
            if (L.chunk < 0 || L.rot_dims < 0 || L.rot_dims > L.dim || L.rot_dims % 2 || !L.head_bias || !L.talk)
                return fail(SMOL_ERR_INVALID, "sigmoid attention: chunk must not be negative, rot_dims even and at most dim, head_bias and talk set");
            r.k_off = m->page_elems;
            r.v_off = r.k_off + (size_t)L.kv_heads * cfg->page_size * L.dim;
            m->page_elems = r.v_off + (size_t)L.kv_heads * cfg->page_size * L.vdim;
            r.freq_off = m->freq_table.size();
            push_frequencies(m->freq_table, L, true);
            m->max_sig_cols = std::max(m->max_sig_cols, L.heads * L.vdim);
            m->max_q = std::max(m->max_q, L.heads * L.dim);
            m->max_heads = std::max(m->max_heads, L.heads);
            m->max_vdim = std::max(m->max_vdim, L.vdim);
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
        } else if (L.mixer == SMOL_LM_MIX_RETENTION) {
            if (L.dim > 256) return fail(SMOL_ERR_UNSUPPORTED, "recurrent mixer: key size above 256");
            if (L.vdim < 1 || !L.head_decay || L.rot_dims < 0 || L.rot_dims > L.dim || L.rot_dims % 2)
                return fail(SMOL_ERR_INVALID, "retention: vdim must be positive, head_decay set, rot_dims even and at most dim");
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.vdim;
            m->slot_floats = (m->slot_floats + 3) / 4 * 4;
            r.freq_off = m->freq_table.size();
            push_frequencies(m->freq_table, L, true);
            m->max_hd = std::max(m->max_hd, L.heads * std::max(L.dim, L.vdim));
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
            m->max_conv = std::max(m->max_conv, 2 * L.heads * L.dim);
        } else if (L.mixer == SMOL_LM_MIX_LIGHTNING || L.mixer == SMOL_LM_MIX_HGRN2) {
            if (L.dim > 256) return fail(SMOL_ERR_UNSUPPORTED, "recurrent mixer: key size above 256");
            if (L.vdim < 1 || !L.out_norm) return fail(SMOL_ERR_INVALID, "linear attention: vdim must be positive and out_norm set");
            if (L.mixer == SMOL_LM_MIX_LIGHTNING && !L.head_decay) return fail(SMOL_ERR_INVALID, "lightning attention: head_decay");
            if (L.mixer == SMOL_LM_MIX_HGRN2 && (!L.forget_lower || !L.rate_bias)) return fail(SMOL_ERR_INVALID, "HGRN2: forget_lower and rate_bias");
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.vdim;
            m->slot_floats = (m->slot_floats + 3) / 4 * 4;
            m->max_hd = std::max(m->max_hd, L.heads * std::max(L.dim, L.vdim));
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
            if (L.mixer == SMOL_LM_MIX_LIGHTNING) {
                m->max_conv = std::max(m->max_conv, 2 * L.heads * L.dim + L.heads * L.vdim);
                m->max_ssd_heads = std::max(m->max_ssd_heads, L.heads);
            }
        } else if (L.mixer == SMOL_LM_MIX_GATED_LINEAR) {
            if (L.dim > 256) return fail(SMOL_ERR_UNSUPPORTED, "recurrent mixer: key size above 256");
            if (L.rank < 1 || L.vdim < 1 || !(L.decay_tau > 0.0f)) return fail(SMOL_ERR_INVALID, "gated linear: rank, vdim, tau must be positive");
            r.state_off = m->slot_floats;
            m->slot_floats += (size_t)L.heads * L.dim * L.vdim;
            m->max_hd = std::max(m->max_hd, L.heads * std::max(L.dim, L.vdim));
            m->max_mix = std::max(m->max_mix, L.heads * L.vdim);
        } else {
            return fail(SMOL_ERR_UNSUPPORTED, "unknown mixer kind");
        }
        return SMOL_OK;
    };
    for (int n = 0; n < cfg->n_runs; ++n) {
        const int li = run_layer[n];
        if (li < 0 || li >= cfg->n_layers) { delete m; return fail(SMOL_ERR_INVALID, "run_layer entry outside the layer array"); }
        const SmolLmLayer& L = m->layers[li];
        RunInfo r, rs;
        r.layer = rs.layer = li;
        r.flags = cfg->run_flags ? cfg->run_flags[n] : 0;
        if (r.flags & SMOL_LM_RUN_ADD_EMBED) m->any_restart = true;
        if (r.flags & SMOL_LM_RUN_MERGE_EMBED) m->any_merge = true;
        int rc = place(L, r);
        const bool prenorm = cfg->block == SMOL_LM_BLOCK_PRENORM, parallel = cfg->block == SMOL_LM_BLOCK_PARALLEL, outnorm = cfg->block == SMOL_LM_BLOCK_OUTNORM;
        if (rc == SMOL_OK && outnorm) {
            if (!L.norm1 || (L.mlp != SMOL_LM_MLP_NONE && !L.norm2)) rc = fail(SMOL_ERR_INVALID, "output-norm block: norm weights");
            else if ((L.mlp != SMOL_LM_MLP_NONE && L.mlp != SMOL_LM_MLP_GATED) || !pairable(L))
                rc = fail(SMOL_ERR_UNSUPPORTED, "output-norm block: dense gated feed-forwards or none; no HGRN2, latent attention, gated linear or generalized delta mixers");
        }
        if (rc == SMOL_OK && L.side) {
            if (!pairable(L) || !pairable(*L.side)) rc = fail(SMOL_ERR_UNSUPPORTED, "mixers side by side: softmax or sigmoid attention, the state-space recurrence, lightning attention");
            else if (cfg->block == SMOL_LM_BLOCK_POSTNORM || parallel) rc = fail(SMOL_ERR_UNSUPPORTED, "mixers side by side need the sandwich or the pre-norm block");
            else if (L.proj_norm && (!prenorm || !L.side->proj_norm || !L.side->w_out)) rc = fail(SMOL_ERR_INVALID, "proj_norm: the pre-norm block, and set on both mixers with their own w_out");
            else rc = place(*L.side, rs);
            if (rc == SMOL_OK) m->max_mix = std::max(m->max_mix, mix_cols_of(L) + mix_cols_of(*L.side));
            if (rc == SMOL_OK && L.proj_norm) m->any_own_proj = true;
        }
        const bool norm2 = prenorm && L.mlp != SMOL_LM_MLP_NONE;
        if (rc == SMOL_OK && (prenorm || parallel)) {
            if (cfg->norm_kind < SMOL_LM_NORM_RMS || cfg->norm_kind > SMOL_LM_NORM_LAYER) rc = fail(SMOL_ERR_INVALID, "unknown norm kind");
            else if (!L.norm1 || (norm2 && !L.norm2)) rc = fail(SMOL_ERR_INVALID, "pre-norm and parallel block: norm weights");
            else if (cfg->norm_kind == SMOL_LM_NORM_DYT && (!L.norm1_alpha || (norm2 && !L.norm2_alpha))) rc = fail(SMOL_ERR_INVALID, "the Dynamic-Tanh norms need alphas");
            else if (cfg->norm_kind != SMOL_LM_NORM_RMS && (!L.norm1_shift || (norm2 && !L.norm2_shift))) rc = fail(SMOL_ERR_INVALID, "Dynamic-Tanh and layer norms need shifts");
            else if (parallel && ((L.mlp != SMOL_LM_MLP_NONE && L.mlp != SMOL_LM_MLP_EXPERTS) || !pairable(L) || L.in_bias))
                rc = fail(SMOL_ERR_UNSUPPORTED, "parallel block: routed feed-forwards or none, softmax / sigmoid attention, state-space, lightning or retention mixers without biases");
            else if (L.mlp == SMOL_LM_MLP_POLYNORM || L.route_input || L.out_bias || L.n_identity > 0)
                rc = fail(SMOL_ERR_UNSUPPORTED, "pre-norm and parallel block: PolyNorm feed-forwards, input-weighted routing, identity outputs and out_bias are not built");
        }
        if (rc == SMOL_OK && ((r.flags & SMOL_LM_RUN_ADD_EMBED) && !prenorm)) rc = fail(SMOL_ERR_UNSUPPORTED, "runs that add the embedding output need the pre-norm block");
        if (rc == SMOL_OK && ((r.flags & SMOL_LM_RUN_MERGE_EMBED) || L.shared_gate) && !parallel) rc = fail(SMOL_ERR_UNSUPPORTED, "merging runs and gated shared experts need the parallel block");
        if (rc == SMOL_OK && !prenorm && !parallel && !outnorm && (L.shared_ff > 0 || L.proj_norm || L.mixer >= SMOL_LM_MIX_SIGMOID_ATTENTION ||
                                         (L.side && L.side->mixer >= SMOL_LM_MIX_SIGMOID_ATTENTION)))
            rc = fail(SMOL_ERR_UNSUPPORTED, "shared experts, proj_norm, sigmoid / lightning attention, HGRN2 and retention need the pre-norm or the parallel block");
        if (rc == SMOL_OK && L.shared_ff > 0 && (L.mlp != SMOL_LM_MLP_EXPERTS || (!parallel && (!L.w_shared_in || !L.w_shared_out)))) rc = fail(SMOL_ERR_INVALID, "shared expert: routed feed-forwards only, with both matrices");
        if (rc == SMOL_OK && cfg->block == SMOL_LM_BLOCK_POSTNORM && (L.out_bias || L.route_input))
            rc = fail(SMOL_ERR_UNSUPPORTED, "out_bias and route_input need the sandwich block");
        if (rc != SMOL_OK) { delete m; return rc; }
        if (L.mlp < SMOL_LM_MLP_NONE || L.mlp > SMOL_LM_MLP_EXPERTS) { delete m; return fail(SMOL_ERR_UNSUPPORTED, "unknown feed-forward kind"); }
        if (L.mlp == SMOL_LM_MLP_POLYNORM) m->max_ff = std::max(m->max_ff, L.ff);
        if (L.mlp == SMOL_LM_MLP_GATED || L.mlp == SMOL_LM_MLP_EXPERTS) {
            if (L.ff < 1 || L.mlp_act < SMOL_LM_ACT_GELU_TANH || L.mlp_act > SMOL_LM_ACT_RELU_SQUARED) { delete m; return fail(SMOL_ERR_INVALID, "gated feed-forward: ff and activation"); }
        }
        if (L.mlp == SMOL_LM_MLP_GATED) m->max_ff = std::max(m->max_ff, 2 * L.ff);
        if (L.mlp == SMOL_LM_MLP_EXPERTS) {
            const int E = L.n_experts + L.n_identity;
            if (L.n_experts < 0 || L.n_identity < 0 || E < 1 || E > kMaxRouted || L.top_k < 1 || L.top_k > kMaxTop || L.n_groups < 1 ||
                E % L.n_groups != 0 || L.keep_groups < 1 || L.keep_groups > L.n_groups || L.top_k > L.keep_groups * (E / L.n_groups)) {
                delete m;
                return fail(SMOL_ERR_INVALID, "routed feed-forward: experts, groups and top do not fit each other");
            }
            m->max_top = std::max(m->max_top, L.top_k);
            m->max_routed = std::max(m->max_routed, E);
            m->max_experts = std::max(m->max_experts, L.n_experts);
            m->max_pair_ff = std::max(m->max_pair_ff, L.top_k * L.ff);
            if (L.shared_ff > 0 && !parallel) m->max_ff = std::max(m->max_ff, (L.ff_plain ? 1 : 2) * L.shared_ff);
            if (parallel) m->max_mix = std::max(m->max_mix, mix_cols_of(L) + L.shared_ff);
        }
        m->max_in = std::max(m->max_in, full_n_in_of(L, cfg->block));
        m->runs.push_back(r);
        m->side_runs.push_back(rs);
    }
    // pages hold 16-byte aligned rows whatever the sizes
    m->page_elems = (m->page_elems + 7) / 8 * 8;
    const size_t T = cfg->max_step_tokens, D = cfg->width, E = m->esize;
    size_t o = 0;
    auto carve = [&](size_t bytes) { size_t at = o; o += al256(bytes); return at; };
    m->o_x = carve(T * D * 4);
    m->o_hn = carve(T * D * E);
    m->o_proj = carve(T * (size_t)m->max_in * 4);
    m->o_mix = carve(T * (size_t)std::max(m->max_mix, 1) * E);
    m->o_y = carve(T * D * 4);
    m->o_z = carve(T * (size_t)std::max(m->max_ff, 1) * 4);
    m->o_act = carve(T * (size_t)std::max(m->max_ff, 1) * E);
    m->o_dec = carve(T * (size_t)std::max(m->max_hd, 1) * 4);
    m->o_u = carve(T * (size_t)std::max(m->max_hd, 1) * 4);
    m->o_au = carve(T * (size_t)std::max(m->max_hd, 1) * 4);
    m->o_oraw = carve(T * (size_t)std::max(m->max_hd, 1) * 4);
    m->o_q = carve(T * (size_t)std::max(m->max_q, 1) * E);
    m->o_hw = carve((size_t)cfg->max_want * D * E);
    m->o_err = carve(256);
    // few-token attention: key ranges of split_len positions (64 while the context stays below 16 384: a decoding row
    // then spreads over context / 64 blocks per key/value head), at most 256 of them per row; ranges are launched four at a time
    const int ctx = std::max(cfg->max_context, 1);
    m->split_len = std::max(64, ((ctx + 255) / 256 + 63) / 64 * 64);
    m->max_splits = ((ctx + m->split_len - 1) / m->split_len + 3) / 4 * 4;
    m->o_part = carve((size_t)cfg->max_step_seqs * kShortSeq * m->max_heads * m->max_splits * (m->max_vdim + 2) * 4);
    if (cfg->block == SMOL_LM_BLOCK_POSTNORM) m->o_hist = carve((size_t)(cfg->n_runs + 1) * T * D * 4);
    if (m->max_cq > 0) {
        m->o_cq = carve(T * (size_t)m->max_cq * E);
        m->o_qf = carve(T * (size_t)m->max_qf * 4);
    }
    if (!m->freq_table.empty()) m->o_freq = carve(m->freq_table.size() * 4 + 4);
    if (m->any_restart) m->o_x0 = carve(T * D * 4);
    if (m->any_merge) m->o_cat = carve(2 * T * D * E);
    if (m->max_sig_cols > 0 && cfg->dtype == SMOL_LM_BF16) m->o_spart = carve((size_t)kSigmoidRanges * T * m->max_sig_cols * 4);
    if (m->any_own_proj) {
        m->o_mix2 = carve(T * (size_t)std::max(m->max_mix, 1) * E);
        m->o_y2 = carve(T * D * 4);
    }
    if (m->max_conv > 0) {
        m->o_conv = carve(T * (size_t)m->max_conv * 4);
        m->o_head = carve(2 * T * (size_t)m->max_ssd_heads * 4);
    }
    for (const RunInfo& r : m->runs)
        for (const SmolLmLayer* L : {(const SmolLmLayer*)&m->layers[r.layer], m->layers[r.layer].side}) {
            if (!L) continue;
            const bool ssd = L->mixer == SMOL_LM_MIX_STATE_SPACE, general = L->mixer == SMOL_LM_MIX_GENERAL_DELTA, unit = L->mixer == SMOL_LM_MIX_MLSTM;
            const bool gated = L->mixer == SMOL_LM_MIX_GATED_DELTA, channel = L->mixer == SMOL_LM_MIX_GATED_LINEAR || L->mixer == SMOL_LM_MIX_HGRN2;
            if (!general && !gated && !unit && !channel && !ssd && L->mixer != SMOL_LM_MIX_LIGHTNING && L->mixer != SMOL_LM_MIX_RETENTION) continue;
            // records of the forms that a step of this engine can take, on however many SMs
            const int kind = general ? kScanGeneralDelta : gated ? kScanGatedDelta : channel ? kScanChannelDecay : kScanHeadDecay;
            const int d = ssd ? L->n_state : L->dim, columns = general ? L->dim : L->vdim + (unit ? 1 : 0), n = cfg->max_step_tokens;
            if (chunks_pay(kind, unit, 1, L->heads, n, n, d, columns, 1 << 20))
                m->max_rec = std::max(m->max_rec, (size_t)L->heads * chunk_record(scan_removes(kind), chunk_pad(d), columns));
            if (!gated && !unit && quad_pays(1, n, n)) m->max_quad = std::max(m->max_quad, (size_t)L->heads * quad_record(general ? kFormGeneral : kFormAdd, quad_pad(d)));
        }
    if (m->max_rec + m->max_quad > 0)
        m->o_rec = carve(std::max((T / kChunk + cfg->max_step_seqs + 1) * m->max_rec, (T / kQuad + cfg->max_step_seqs + 1) * m->max_quad) * 4);
    if (m->max_pair_heads > 0) m->o_pairs = carve(T * (size_t)m->max_pair_heads * kPairFloats * 4);
    if (m->max_top > 0) {
        const size_t pairs = T * (size_t)m->max_top;
        m->o_sel_id = carve(pairs * 4);
        m->o_sel_w = carve(pairs * 4);
        m->o_perm = carve(pairs * 4);
        m->o_slot_of = carve(pairs * 4);
        m->o_seg = carve(((size_t)m->max_experts + 1) * 4);
        m->o_tile_g = carve((pairs / kGroupTile + m->max_experts + 1) * 4);
        m->o_tile_r = carve((pairs / kGroupTile + m->max_experts + 1) * 4);
        m->o_ntiles = carve(4);
        m->o_zp = carve(T * (size_t)m->max_pair_ff * 2 * 4);
        m->o_actp = carve(T * (size_t)m->max_pair_ff * E);
        m->o_yp = carve(pairs * D * 4);
        m->o_ap = carve(pairs * D * E);
        m->o_rlogits = carve(T * (size_t)m->max_routed * 4);
        m->o_rdone = carve(T * 4);          // counters: zero between steps (the caller's workspace starts zeroed; the kernel resets them)
    }
    m->total = o;
    *out = m;
    return SMOL_OK;
}

extern "C" void smol_lm_destroy(SmolLm* m) { delete m; }
extern "C" size_t smol_lm_page_bytes(const SmolLm* m) { return m ? std::max<size_t>(m->page_elems, 8) * m->esize : 0; }
extern "C" size_t smol_lm_slot_bytes(const SmolLm* m) { return m ? std::max<size_t>(m->slot_floats, 4) * 4 : 0; }
extern "C" size_t smol_lm_workspace_bytes(const SmolLm* m) { return m ? m->total : 0; }
extern "C" int64_t smol_lm_launch_count(const SmolLm* m) { return m ? m->launches : 0; }
extern "C" int32_t* smol_lm_error_word(SmolLm* m) { return (m && m->bound) ? reinterpret_cast<int32_t*>(m->ws + m->o_err) : nullptr; }

// Shared memory the scan asks for when another kernel runs beside it: at most two of its blocks then share an SM (left to
// itself the hardware packs them onto the few SMs that happen to have room, and a scan is bound by its slowest block), and
// one still fits beside a tcgen05 product's block.
constexpr int kScanSpread = 76 * 1024;

template <int DK>
static cudaError_t scan_attribute() {
    cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * delta_buf_floats(DK) * sizeof(float)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gla_scan_kernel<DK, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)(2 * gla_buf_floats(DK) * sizeof(float))));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(group_scan_kernel<DK, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)(2 * group_scan_buf_floats(DK) * sizeof(float))));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(group_scan_kernel<DK, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)(2 * group_scan_buf_floats(DK) * sizeof(float))));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gla_scan_kernel<DK, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)(2 * gla_buf_floats(DK) * sizeof(float))));
    return e;
}
template <int DK>
static cudaError_t quad_attribute() {
    cudaError_t e = cudaFuncSetAttribute(quad_scan_kernel<DK, kFormAdd>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)quad_smem(kFormAdd, DK)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(quad_scan_kernel<DK, kFormGeneral>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(kScanSpread, (int)quad_smem(kFormGeneral, DK)));
    return e;
}
template <int DK>
static cudaError_t chunk_attributes() {
    const auto allow = [](auto kernel, size_t bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); };
    cudaError_t e = allow(chunk_scan_kernel<DK, true, 1>, std::max((size_t)kScanSpread, chunk_smem(true, DK, 1)));
    if (e == cudaSuccess) e = allow(chunk_scan_kernel<DK, false, 1>, std::max((size_t)kScanSpread, chunk_smem(false, DK, 1)));
    if constexpr (DK > 64) {
        if (e == cudaSuccess) e = allow(chunk_scan_kernel<DK, true, 2>, chunk_smem(true, DK, 2));
        if (e == cudaSuccess) e = allow(chunk_scan_kernel<DK, false, 2>, chunk_smem(false, DK, 2));
    }
    if (e == cudaSuccess) e = allow(chunk_prep_kernel<kScanGeneralDelta, DK>, chunk_prep_floats(kScanGeneralDelta, DK) * sizeof(float));
    if (e == cudaSuccess) e = allow(chunk_prep_kernel<kScanChannelDecay, DK>, chunk_prep_floats(kScanChannelDecay, DK) * sizeof(float));
    if (e == cudaSuccess) e = allow(chunk_prep_head_kernel<kScanGatedDelta, DK>, chunk_prep_floats(kScanGatedDelta, DK) * sizeof(float));
    if (e == cudaSuccess) e = allow(chunk_prep_head_kernel<kScanHeadDecay, DK>, chunk_prep_floats(kScanHeadDecay, DK) * sizeof(float));
    return e;
}
static constexpr int flash_smem_bytes(int DK, int DV, bool vk, int maps = 1) { return 2 * 64 * (maps * (DK + 8) + (vk ? 0 : DV + 8)) * (int)sizeof(bf16); }

template <int DK, int HPW>
static cudaError_t sigmoid_flash_attributes() {
    cudaError_t e = cudaFuncSetAttribute(sigmoid_flash_kernel<DK, HPW, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sigmoid_flash_kernel<DK, HPW, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    return e;
}

template <class T>
static cudaError_t set_kernel_attributes() {
    cudaError_t e = scan_attribute<16>();
    if (e == cudaSuccess) e = scan_attribute<32>();
    if (e == cudaSuccess) e = scan_attribute<64>();
    if (e == cudaSuccess) e = scan_attribute<128>();
    if (e == cudaSuccess) e = scan_attribute<256>();
    if (e == cudaSuccess) e = quad_attribute<32>();
    if (e == cudaSuccess) e = chunk_attributes<32>();
    if (e == cudaSuccess) e = quad_attribute<64>();
    if (e == cudaSuccess) e = chunk_attributes<64>();
    if (e == cudaSuccess) e = quad_attribute<128>();
    if (e == cudaSuccess) e = chunk_attributes<128>();
    if (e == cudaSuccess) e = quad_attribute<256>();
    if (e == cudaSuccess) e = chunk_attributes<256>();
    const auto rows = [&](auto kernel) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmemMax);
    };
    rows(attn_rows_kernel<T, 8, 1, 1>); rows(attn_rows_kernel<T, 8, 2, 1>); rows(attn_rows_kernel<T, 16, 1, 1>); rows(attn_rows_kernel<T, 16, 2, 1>);
    rows(attn_rows_kernel<T, 8, 1, 4>); rows(attn_rows_kernel<T, 8, 2, 4>); rows(attn_rows_kernel<T, 16, 1, 4>); rows(attn_rows_kernel<T, 16, 2, 4>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_split_kernel<T, 8, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSplitSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_split_kernel<T, 8, 2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSplitWideSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_split_kernel<T, 8, 2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSplitWideSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_split_kernel<T, 16, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSplitSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sigmoid_attn_kernel<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sigmoid_attn_kernel<T, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sigmoid_split_kernel<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSigmoidSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sigmoid_split_kernel<T, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSigmoidSmemMax);
    if (e == cudaSuccess) e = sigmoid_flash_attributes<32, 1>();
    if (e == cudaSuccess) e = sigmoid_flash_attributes<64, 1>();
    if (e == cudaSuccess) e = sigmoid_flash_attributes<96, 1>();
    if (e == cudaSuccess) e = sigmoid_flash_attributes<128, 1>();
    if (e == cudaSuccess) e = sigmoid_flash_attributes<32, 2>();
    if (e == cudaSuccess) e = sigmoid_flash_attributes<64, 2>();
#define SMOL_FLASH_ATTR(DK, DV, VK, MAPS)                                                                                        \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_flash_kernel<DK, DV, VK, MAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                   flash_smem_bytes(DK, DV, VK, MAPS))
    SMOL_FLASH_ATTR(128, 128, false, 1);
    SMOL_FLASH_ATTR(64, 128, false, 1);
    SMOL_FLASH_ATTR(192, 128, true, 1);
    SMOL_FLASH_ATTR(192, 192, true, 1);
    SMOL_FLASH_ATTR(64, 64, false, 2);
    SMOL_FLASH_ATTR(64, 128, false, 2);
    SMOL_FLASH_ATTR(128, 128, false, 2);
#undef SMOL_FLASH_ATTR
#define SMOL_FLASH_TC_ATTR(DK, DV, VK, MAPS) \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_flash_tc_kernel<DK, DV, VK, MAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, ft_smem(DK, DV, VK, MAPS))
    SMOL_FLASH_TC_ATTR(64, 64, false, 1);
    SMOL_FLASH_TC_ATTR(64, 128, false, 1);
    SMOL_FLASH_TC_ATTR(128, 128, false, 1);
    SMOL_FLASH_TC_ATTR(64, 64, true, 1);
    SMOL_FLASH_TC_ATTR(128, 128, true, 1);
    SMOL_FLASH_TC_ATTR(192, 128, true, 1);
    SMOL_FLASH_TC_ATTR(64, 64, false, 2);
    SMOL_FLASH_TC_ATTR(64, 128, false, 2);
#undef SMOL_FLASH_TC_ATTR
    return e;
}

template <int BN>
static cudaError_t gemm_tc_prepare_sized() { return cudaFuncSetAttribute(gemm_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_tc_smem<BN>()); }
static cudaError_t gemm_tc_prepare() {
    for (cudaError_t e : {gemm_tc_prepare_sized<64>(), gemm_tc_prepare_sized<96>(), gemm_tc_prepare_sized<128>(), gemm_tc_prepare_sized<192>(), gemm_tc_prepare_sized<256>()})
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

extern "C" int smol_lm_bind(SmolLm* m, const SmolLmGlobals* g, void* d_workspace, size_t workspace_bytes, void* d_pages, int32_t n_pages,
                            void* d_slots, int32_t n_slots) {
    if (!m || !g || !d_workspace || !d_pages || !d_slots) return fail(SMOL_ERR_INVALID, "smol_lm_bind: null argument");
    if (workspace_bytes < m->total) return fail(SMOL_ERR_CAPACITY, "smol_lm_bind: workspace too small");
    if (reinterpret_cast<uintptr_t>(d_workspace) % 256 || reinterpret_cast<uintptr_t>(d_pages) % 16)
        return fail(SMOL_ERR_INVALID, "smol_lm_bind: workspace must be 256-byte aligned, pages 16-byte aligned");
    if (n_pages < 1 || n_slots < 1) return fail(SMOL_ERR_INVALID, "smol_lm_bind: need at least one page and one slot");
    if (!g->embed || !g->head || !g->final_norm) return fail(SMOL_ERR_INVALID, "smol_lm_bind: missing global weights");
    CU(set_kernel_attributes<float>());
    CU(set_kernel_attributes<bf16>());
    int dev = 0;
    CU(cudaGetDevice(&dev));
    CU(cudaDeviceGetAttribute(&m->n_sms, cudaDevAttrMultiProcessorCount, dev));
    CU(gemm_tc_prepare());
    m->tc_ready = smol::tensor_map_encoder() != nullptr && m->n_sms > 0;
    m->g = *g;
    m->ws = static_cast<char*>(d_workspace);
    m->pages = d_pages;
    m->slots = static_cast<float*>(d_slots);
    m->n_pages = n_pages;
    m->n_slots = n_slots;
    if (m->cfg.block == SMOL_LM_BLOCK_POSTNORM && (size_t)m->cfg.width * 8 > 48 * 1024) {
        // the post-norm kernel keeps two fp32 copies of a row in shared memory
        if ((size_t)m->cfg.width * 8 > 200 * 1024) return fail(SMOL_ERR_UNSUPPORTED, "smol_lm_bind: width above 25600 with the post-norm block");
        CU(cudaFuncSetAttribute(post_norm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 8));
        CU(cudaFuncSetAttribute(post_norm_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 8));
    }
    if (m->max_top > 0) CU(cudaMemset(m->ws + m->o_rdone, 0, (size_t)m->cfg.max_step_tokens * 4));      // the router's per-token counters
    if (!m->freq_table.empty())
        CU(cudaMemcpy(m->ws + m->o_freq, m->freq_table.data(), m->freq_table.size() * sizeof(float), cudaMemcpyHostToDevice));
    if (m->cfg.block == SMOL_LM_BLOCK_POSTNORM && !g->embed_norm) return fail(SMOL_ERR_INVALID, "smol_lm_bind: the post-norm block needs embed_norm");
    if (m->cfg.block == SMOL_LM_BLOCK_PRENORM && m->cfg.norm_kind == SMOL_LM_NORM_DYT && (!g->final_norm_shift || !g->final_norm_alpha))
        return fail(SMOL_ERR_INVALID, "smol_lm_bind: the Dynamic-Tanh final norm needs its shift and alpha");
    if ((m->cfg.block == SMOL_LM_BLOCK_PRENORM || m->cfg.block == SMOL_LM_BLOCK_PARALLEL) && m->cfg.norm_kind == SMOL_LM_NORM_LAYER && !g->final_norm_shift)
        return fail(SMOL_ERR_INVALID, "smol_lm_bind: the final layer norm needs its shift");
    if (m->any_merge && !g->w_merge) return fail(SMOL_ERR_INVALID, "smol_lm_bind: merging runs need w_merge");
    if ((m->cfg.block == SMOL_LM_BLOCK_PARALLEL || m->cfg.block == SMOL_LM_BLOCK_OUTNORM) && !m->ff_stream) {
        CU(cudaStreamCreateWithFlags(&m->ff_stream, cudaStreamNonBlocking));
        CU(cudaEventCreateWithFlags(&m->ff_start, cudaEventDisableTiming));
        CU(cudaEventCreateWithFlags(&m->ff_done, cudaEventDisableTiming));
    }
    if ((size_t)m->cfg.width * 4 > 48 * 1024) {
        CU((cudaFuncSetAttribute(residual_norm_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 4)));
        CU((cudaFuncSetAttribute(residual_norm_kernel<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 4)));
        CU((cudaFuncSetAttribute(residual_norm_kernel<bf16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 4)));
        CU((cudaFuncSetAttribute(residual_norm_kernel<bf16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, m->cfg.width * 4)));
    }
    m->bound = true;
    return SMOL_OK;
}

namespace smol {
namespace lm {
// gemm_few_kernel of one row that a prologue makes (a form of its own: shared with the plain one it cost that 1.4 % in decoding).
// begin(): the prologue; row(k): 8 elements of the row; part: [WARPS][few_out(NR)], in the place of the row.
constexpr int few_out(int nr) { return nr * (nr == 16 ? 8 : 16); }     // outputs of a block (those of one activation row count)
template <int NR, int WARPS, class Begin, class Row>
__device__ __forceinline__ void few_product(const bf16* __restrict__ w, float* __restrict__ y, int N, int K, float* part, Begin begin, Row row) {
    constexpr int WT = NR / 8, AT = NR == 16 ? 1 : 2;            // 8-row pieces of weights and of activations per step
    constexpr int U = WT + AT <= 3 ? 4 : 2;                      // steps of 32 whose loads are in flight together
    constexpr int OUT = few_out(NR);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int n0 = blockIdx.x * NR;
    const bf16* wr[WT];
#pragma unroll
    for (int i = 0; i < WT; ++i) wr[i] = w + (size_t)min(n0 + i * 8 + g, N - 1) * K + tq * 8;
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = 0.0f;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 p[U][WT];
    auto load_weights = [&](int k0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * 32;
#pragma unroll
            for (int i = 0; i < WT; ++i) p[u][i] = k + tq * 8 < K ? ldg_stream(wr[i] + k) : zero;
        }
    };
    load_weights(warp * 32);             // no kernel of a step writes weights: the first ones are on their way before the wait (smol_lm_linear launches plainly)
    begin();
    for (int k0 = warp * 32; k0 < K; k0 += WARPS * 32 * U) {
        uint4 x[U][AT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * 32 + tq * 8;
#pragma unroll
            for (int i = 0; i < AT; ++i) {
                const int m = i * 8 + g;
                x[u][i] = (m < 1 && k < K) ? row(k) : zero;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float lo[4] = {0.0f, 0.0f, 0.0f, 0.0f}, hi[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if constexpr (NR == 16) {
                mma_bf16_16816(lo, p[u][0].x, p[u][1].x, p[u][0].y, p[u][1].y, x[u][0].x, x[u][0].y);
                mma_bf16_16816(hi, p[u][0].z, p[u][1].z, p[u][0].w, p[u][1].w, x[u][0].z, x[u][0].w);
            } else {
                mma_bf16_16816(lo, x[u][0].x, x[u][1].x, x[u][0].y, x[u][1].y, p[u][0].x, p[u][0].y);
                mma_bf16_16816(hi, x[u][0].z, x[u][1].z, x[u][0].w, x[u][1].w, p[u][0].z, p[u][0].w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] += lo[e] + hi[e];
        }
        load_weights(k0 + WARPS * 32 * U);
    }
    __syncthreads();
    // part[warp][m * NR + n]: neighbouring outputs of a row side by side.  acc[e]: tile row g + (e / 2) * 8, tile column 2 tq + e % 2
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int r = g + (e >> 1) * 8, c = tq * 2 + (e & 1);
        part[warp * OUT + (NR == 16 ? c * NR + r : r * NR + c)] = acc[e];
    }
    __syncthreads();
    for (int o = threadIdx.x; o < OUT; o += WARPS * 32) {
        const int m = o / NR, n = n0 + o % NR;
        double t = part[o];
#pragma unroll
        for (int x = 1; x < WARPS; ++x) t += part[x * OUT + o];
        if (m < 1 && n < N) y[n] = (float)t;
    }
}
// Down-projection of one row with PolyNorm in its prologue: every block takes the row's activation into shared memory, behind its first
// weights.  As a kernel of its own it is one more link of the step's chain, whatever it computes: one token through 10 layers of width 768,
// 4 steps 1622 us -> 1589.  Two and more rows stay with two kernels: what the
// blocks repeat costs more than the launch (2 rows 992 | 999, 4: 1042 | 1104, 8: 1097 | 1117 through 6 layers), as do gated units, whose input is twice as
// long (5 rows of width 1536 990 | 1063).
constexpr size_t kFewActSmem = 48 * 1024 - 512;
template <int NR, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) gemm_polynorm_kernel(const float* __restrict__ z, const float* __restrict__ coef, float eps,
                                                                   const bf16* __restrict__ w, float* __restrict__ y, int N, int K) {
    extern __shared__ uint4 few_smem[];
    __shared__ float red[3][33];
    bf16* xs = reinterpret_cast<bf16*>(few_smem);
    few_product<NR, WARPS>(w, y, N, K, reinterpret_cast<float*>(few_smem), [&] {
        dep_wait();
        dep_go();
        float s2 = 0.0f, s4 = 0.0f, s6 = 0.0f;
        // the sums by polynorm_kernel's threads, each with the elements it has there: a row's bits do not depend on which form takes it
        if (threadIdx.x < kPolynormThreads) {
#pragma unroll 4
            for (int c = threadIdx.x * 4; c < K; c += kPolynormThreads * 4) {
                const float4 v = *reinterpret_cast<const float4*>(z + c);
                const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float v2 = e[j] * e[j];
                    s2 += v2;
                    s4 += v2 * v2;
                    s6 += v2 * v2 * v2;
                }
            }
        }
        block_sum3(s2, s4, s6, red);
        const float a = coef[0] / sqrtf(s2 / (float)K + eps), b = coef[1] / sqrtf(s4 / (float)K + eps), cc = coef[2] / sqrtf(s6 / (float)K + eps), e = coef[3];
        auto f = [&](float v) { return a * v + b * v * v + cc * v * v * v + e; };
#pragma unroll 4
        for (int c = threadIdx.x * 4; c < K; c += WARPS * 128) {
            const float4 v = *reinterpret_cast<const float4*>(z + c);
            store4<bf16>(xs + c, f(v.x), f(v.y), f(v.z), f(v.w));
        }
        __syncthreads();
    }, [&](int k) { return *reinterpret_cast<const uint4*>(xs + k); });
}
}  // namespace lm
}  // namespace smol

// The kernels of a step are launched with programmatic stream serialization and begin with dep_wait(): a kernel's blocks are set up while
// the kernel before it drains, instead of after.  What bounds a decoding step is its chain of some hundred dependent kernels of two to ten
// microseconds: 10 layers of width 768, one token against 2048 cached ones, 4 steps 1780 us -> 1615; 5 sequences of 700 through 4 layers of
// width 1536, 1024 -> 940.  A launch right after a wait for another stream's event goes out plainly.
// What no kernel of the step writes -- weights, the step's index arrays, cached rows of earlier steps, slots' states that only the kernel itself writes -- is read before
// dep_wait(): a kernel's blocks start when every block of the one in front has passed its own dep_wait(), so all before that one has completed and is visible.  (The
// step's first kernel reads nothing before it: in front of it may be anything.  And no block leaves without it: a kernel of blocks that all left at once would be
// complete before the one in front of it.)
static thread_local bool t_plain_next = false;
static cudaError_t wait_event(cudaStream_t st, cudaEvent_t e) {
    t_plain_next = true;
    return cudaStreamWaitEvent(st, e, 0);
}
template <class... P, class... X>
static cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, X&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = t_plain_next ? 0 : 1;
    t_plain_next = false;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<X>(args))...);
}

// Kernels whose few long blocks need the SMs to themselves: set up early, they crowd onto those SMs that the kernel before leaves first,
// two or three to one, and the rest stay idle.  Scans, attention and fp32 products of prompts are launched this way; with all of them early,
// 2048 tokens through two layers of width 768 took 786 us instead of 665 (706 with every launch plain), 300 in fp32 917 instead of 830.
// The tcgen05 products keep the SM to themselves by their shared memory and gain by the early start (1138 us instead of 1164).
template <class... P, class... X>
static cudaError_t plain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, X&&... args) {
    t_plain_next = true;
    return pdl_launch(kernel, grid, block, smem, st, std::forward<X>(args)...);
}

// Launches the form of a row kernel for `rows` rows of D: go(V, LONE, blocks, threads).  False: the rows are not whole 16-byte pieces, or too wide.
template <class Go>
static bool row_pieces(int rows, int D, uintptr_t addresses, Go go) {
    if (D % 4 != 0 || D > kRowPiecesMax || addresses % 16 != 0) return false;
    using std::integral_constant;
    if (rows < kWarpRows) go(integral_constant<int, 1>{}, TrueType{}, rows, (D / 4 + 31) / 32 * 32);
    else if (D <= 768) go(integral_constant<int, 6>{}, FalseType{}, (rows + 3) / 4, 128);
    else if (D <= 1536) go(integral_constant<int, 12>{}, FalseType{}, (rows + 3) / 4, 128);
    else go(integral_constant<int, 16>{}, FalseType{}, (rows + 3) / 4, 128);
    return true;
}
template <class... P>
static uintptr_t addresses_of(const P*... p) { return (reinterpret_cast<uintptr_t>(p) | ...); }

// y fp32 [M, N] = a [M, K] . w [N, K]^T
template <class T>
static cudaError_t linear(SmolLm* m, const T* a, const T* w, float* y, int M, int N, int K, cudaStream_t st);

// The general form: `io` places the operands (strides, a batch of `batch` products, or rows grouped by expert, in which
// case M is the largest number of rows and `tiles` the size of the tile table's grid; tile_rows is the table's tile height).
template <class T>
static cudaError_t linear_ex(SmolLm* m, const T* a, const T* w, float* y, int M, int N, int K, const GemmIo& io, int batch, int tiles,
                             cudaStream_t st);

// Sums of fewer k stay on FMAs: what an operand's two parts leave out then weighs more than the roundings of the longer chain (error against 64 bits, parts | FMAs, K
// 16: 0.97e-7 | 0.61e-7, 64: 1.06 | 1.05, 100: 1.15 | 1.30, 256: 1.22 | 1.49).  The times are alike, some 10 us with the launch.
constexpr int kPartsMinK = 72;
template <int BM, int BN, class T>
static cudaError_t launch_f32_tile(const float* a, const float* w, float* y, int M, int N, int K, const GemmIo& io, int batch, int row_tiles, cudaStream_t st) {
    const int cols = (N + BN - 1) / BN;
    // CTAs per tile: as many as bring the grid of a single row of tiles to about four per SM, each with at least 128 k.  From N, K and the
    // batch alone: a row's sums must not depend on how many rows the step holds.  (K shared by 1 / 2 / 4: 300 rows of 4608 x 768 60 / 50 / 54 us, 1024 rows 137 / 139 /
    // 150; of 768 x 4608 by 2 / 4 / 8: 76 / 66 / 59 and 166 / 158 / 154.)
    int S = 1;
    while (S < 8 && (long long)cols * batch * S < 4 * 148 && K / (2 * S) >= 128) S *= 2;
    static_assert(T::kSmemBytes <= 48 * 1024, "no attribute needed");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cols * S, row_tiles, batch);
    cfg.blockDim = dim3(T::NT);
    cfg.dynamicSmemBytes = T::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    t_plain_next = false;      // launched plainly, as plain_launch does
    return cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<BM, BN, T>, a, w, y, M, N, K, io);
}

template <>
cudaError_t linear_ex<float>(SmolLm* m, const float* a, const float* w, float* y, int M, int N, int K, const GemmIo& io, int batch, int tiles,
                             cudaStream_t st) {
    m->launches++;
    // whole 16-byte pieces in every row of both operands
    if (K % 4 == 0 && io.lda % 4 == 0 && io.sa % 4 == 0 && io.sw % 4 == 0 && (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) % 16 == 0) {
        using namespace smol::f32t;
        const auto on = [&](auto group, auto few, auto many) {
            if (io.tile_group) return launch_f32_tile<kGroupTile, 64, decltype(group)>(a, w, y, M, N, K, io, 1, tiles, st);
            if (M <= 16) return launch_f32_tile<16, 64, decltype(few)>(a, w, y, M, N, K, io, batch, (M + 15) / 16, st);
            return launch_f32_tile<64, 64, decltype(many)>(a, w, y, M, N, K, io, batch, (M + 63) / 64, st);
        };
        if (K < kPartsMinK) return on(Tile<kGroupTile, 64, 8, 8, 0>{}, Tile<16, 64, 4, 4, 0>{}, Tile<64, 64, 8, 8, 0>{});
        return on(MmaTile<kGroupTile, 64, 16, 32>{}, MmaTile<16, 64, 16, 16>{}, MmaTile<64, 64, 32, 32>{});
    }
    if (io.tile_group) {
        dim3 grid((N + 63) / 64, tiles, 1);
        pdl_launch(gemm_f32_kernel<32, 64, 16, 2, 4>, grid, 256, 0, st, a, w, y, M, N, K, io);
    } else if (M <= 16) {
        dim3 grid((N + 63) / 64, (M + 15) / 16, batch);
        pdl_launch(gemm_f32_kernel<16, 64, 16, 1, 4>, grid, 256, 0, st, a, w, y, M, N, K, io);
    } else {
        dim3 grid((N + 63) / 64, (M + 63) / 64, batch);
        pdl_launch(gemm_f32_kernel<64, 64, 16, 4, 4>, grid, 256, 0, st, a, w, y, M, N, K, io);
    }
    return cudaGetLastError();
}

template <>
cudaError_t linear<float>(SmolLm* m, const float* a, const float* w, float* y, int M, int N, int K, cudaStream_t st) {
    return linear_ex<float>(m, a, w, y, M, N, K, plain_io(K, N), 1, 0, st);
}

static bool io_vec(const void* a, const void* w, int K, const GemmIo& io) {
    const int ea = io.a_f32 ? 4 : 8;       // elements of a in 16 bytes
    return K % 8 == 0 && io.lda % ea == 0 && io.sa % ea == 0 && io.sw % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
}

template <>
cudaError_t linear_ex<bf16>(SmolLm* m, const bf16* a, const bf16* w, float* y, int M, int N, int K, const GemmIo& io, int batch, int tiles,
                            cudaStream_t st) {
    const bool vec = io_vec(a, w, K, io);
    if (io.tile_group) {
        dim3 grid((N + 31) / 32, tiles, 1);
        pdl_launch(gemm_bf16_kernel<1, 4, 2, 1>, grid, 128, 0, st, a, w, y, M, N, K, io, vec);       // 32 x 32
    } else if (M <= 32) {
        dim3 grid((N + 31) / 32, (M + 31) / 32, batch);
        pdl_launch(gemm_bf16_kernel<1, 4, 2, 1>, grid, 128, 0, st, a, w, y, M, N, K, io, vec);       // 32 x 32
    } else if (M <= 256 || ((N + 63) / 64) * ((M + 127) / 128) * batch < 2 * m->n_sms) {      // 128-row tiles only when they still fill the GPU twice
        dim3 grid((N + 63) / 64, (M + 63) / 64, batch);
        pdl_launch(gemm_bf16_kernel<2, 2, 2, 4>, grid, 128, 0, st, a, w, y, M, N, K, io, vec);       // 64 x 64
    } else {
        dim3 grid((N + 63) / 64, (M + 127) / 128, batch);
        pdl_launch(gemm_bf16_kernel<2, 2, 4, 4>, grid, 128, 0, st, a, w, y, M, N, K, io, vec);       // 128 x 64
    }
    m->launches++;
    return cudaGetLastError();
}

// Width of the tcgen05 tiles: the one whose waves over the SMs take the fewest clocks.  A stage of a tile costs its bytes through the
// SM's 64 bytes per clock from L2 (more than its MMAs cost at every width); the last epilogue follows the width.
static int gemm_tc_pick(int row_tiles, int N, int K, int n_sms) {
    static const int widths[] = {256, 192, 128, 96, 64};
    const int nk = (K + smol::umma::kBK - 1) / smol::umma::kBK;
    int best = 128;
    double least = 1e30;
    for (int bn : widths) {
        const long long tiles = (long long)row_tiles * ((N + bn - 1) / bn), waves = (tiles + n_sms - 1) / n_sms;
        const double clocks = (double)waves * nk * 2 * (smol::umma::kM + bn) + 6.0 * bn;
        if (clocks < least) { least = clocks; best = bn; }
    }
    return best;
}
template <int BN>
static bool launch_gemm_tc_sized(const bf16* a, const bf16* w, float* y, int M, int N, int row_tiles, int groups, int K, const GemmIo& io, int n_sms,
                                 cudaStream_t st) {
    CUtensorMap ta, tw;
    if (!smol::make_tensor_map_2d(&ta, a, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)smol::umma::kM) ||
        !smol::make_tensor_map_2d(&tw, w, (uint64_t)groups * N, (uint64_t)K, (uint64_t)K, (uint32_t)BN))
        return false;
    const long long tiles = (long long)row_tiles * ((N + BN - 1) / BN);
    const int grid = io.tile_group ? n_sms : (int)std::min<long long>(tiles, n_sms);
    pdl_launch(gemm_tc_kernel<BN>, grid, kTcThreads, gemm_tc_smem<BN>(), st, ta, tw, y, M, N, K, io);
    return true;
}
// false: the driver refused a tensor map (the caller takes another form)
static bool launch_gemm_tc(const bf16* a, const bf16* w, float* y, int M, int N, int row_tiles, int groups, int K, const GemmIo& io, int n_sms, cudaStream_t st) {
    switch (gemm_tc_pick(row_tiles, N, K, n_sms)) {
        case 256: return launch_gemm_tc_sized<256>(a, w, y, M, N, row_tiles, groups, K, io, n_sms, st);
        case 192: return launch_gemm_tc_sized<192>(a, w, y, M, N, row_tiles, groups, K, io, n_sms, st);
        case 128: return launch_gemm_tc_sized<128>(a, w, y, M, N, row_tiles, groups, K, io, n_sms, st);
        case 96: return launch_gemm_tc_sized<96>(a, w, y, M, N, row_tiles, groups, K, io, n_sms, st);
        default: return launch_gemm_tc_sized<64>(a, w, y, M, N, row_tiles, groups, K, io, n_sms, st);
    }
}

template <>
cudaError_t linear<bf16>(SmolLm* m, const bf16* a, const bf16* w, float* y, int M, int N, int K, cudaStream_t st) {
    const bool aligned = K % 8 == 0 && (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
    if (M >= kTcMinRows && N >= kTcMinCols && K >= smol::umma::kBK && aligned && m->tc_ready &&
        launch_gemm_tc(a, w, y, M, N, (M + smol::umma::kM - 1) / smol::umma::kM, 1, K, plain_io(K, N), m->n_sms, st)) {
        m->launches++;
        return cudaGetLastError();
    }
    if (M <= kFewRows && aligned) {
        // the block's shape by N and K alone: a row's result must not depend on what else the step holds beyond its number of rows
#define SMOL_FEW(NR, MT)                                                                                          \
        do {                                                                                                      \
            if (K >= kFewLongK) pdl_launch(gemm_few_kernel<NR, MT, 16>, (N + NR - 1) / NR, 512, 0, st, a, w, y, M, N, K); \
            else pdl_launch(gemm_few_kernel<NR, MT, 8>, (N + NR - 1) / NR, 256, 0, st, a, w, y, M, N, K);                 \
        } while (0)
        if (N < kFewWideN) {
            if (M <= 16) SMOL_FEW(8, 1);
            else SMOL_FEW(8, 2);
        } else if (M <= 8) SMOL_FEW(16, 1);
        else if (M <= 16) SMOL_FEW(16, 2);
        else SMOL_FEW(16, 4);
#undef SMOL_FEW
    } else {
        return linear_ex<bf16>(m, a, w, y, M, N, K, plain_io(K, N), 1, 0, st);
    }
    m->launches++;
    return cudaGetLastError();
}

// y [N] = polynorm(z [K]) . w^T in one kernel (gemm_polynorm_kernel); false: the row does not fit its shared memory or is not whole pieces.
static bool linear_polynorm_row(SmolLm* m, const float* z, const float* coef, const bf16* w, float* y, int N, int K, cudaStream_t st) {
    if (K % 8 != 0 || reinterpret_cast<uintptr_t>(w) % 16 != 0 || (size_t)K * 2 > kFewActSmem) return false;
#define SMOL_FEW_POLY(NR, WARPS)                                                                                                           \
    pdl_launch(gemm_polynorm_kernel<NR, WARPS>, (N + NR - 1) / NR, WARPS * 32, std::max((size_t)K * 2, (size_t)WARPS * few_out(NR) * 4), st, \
               z, coef, m->cfg.norm_eps, w, y, N, K)
    if (N < kFewWideN) {
        if (K >= kFewLongK) SMOL_FEW_POLY(8, 16);
        else SMOL_FEW_POLY(8, 8);
    } else if (K >= kFewLongK) SMOL_FEW_POLY(16, 16);
    else SMOL_FEW_POLY(16, 8);
#undef SMOL_FEW_POLY
    m->launches++;
    return true;
}

// Grouped product on the tcgen05 tile: a [rows, K] sorted by group, w [groups * N, K], the table cut into 128-row tiles.
// Returns false if this form does not apply (then the caller takes the mma.sync form with its own table).
static bool linear_grouped_tc(SmolLm* m, const bf16* a, const bf16* w, float* y, int rows, int groups, int N, int K, const GemmIo& io,
                              cudaStream_t st) {
    const bool aligned = K % 8 == 0 && (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
    if (!(N >= kTcMinCols && K >= smol::umma::kBK && aligned && m->tc_ready)) return false;
    if (!launch_gemm_tc(a, w, y, rows, N, rows / smol::umma::kM + groups / 2 + 1, groups, K, io, m->n_sms, st)) return false;
    m->launches++;
    return true;
}

template <int DK>
static cudaError_t launch_scan(const DeltaArgs& A, int n_seqs, const float* dec, const float* u, const float* au, float* pool, float* o_raw,
                               cudaStream_t st) {
    constexpr int threads = delta_block_cols(DK) * delta_lanes(DK), groups = DK / delta_block_cols(DK);
    pdl_launch(delta_scan_kernel<DK>, n_seqs * A.H * groups, threads, 2 * delta_buf_floats(DK) * sizeof(float), st, A, dec, u, au, pool, o_raw);
    return cudaGetLastError();
}

template <int KIND, int DK>
static cudaError_t launch_quad_sized(SmolLm* m, QuadSource Q, QuadArgs A, int n_seqs, int max_n, float* o_raw, cudaStream_t st, size_t min_smem) {
    constexpr int FORM = quad_form(KIND);
    float* rec = reinterpret_cast<float*>(m->ws + m->o_rec);
    Q.cap = A.cap = m->cfg.max_step_tokens / kQuad + m->cfg.max_step_seqs + 1;
    pdl_launch(quad_prep_kernel<KIND, DK>, dim3((max_n + kQuad - 1) / kQuad, n_seqs, (Q.H + 3) / 4), 128, 0, st, Q, rec);
    A.rec = rec;
    const int parts = (A.dv + kQuadCols - 1) / kQuadCols;
    plain_launch(quad_scan_kernel<DK, FORM>, n_seqs * A.H * parts, kQuadThreads, std::max(quad_smem(FORM, DK), min_smem), st, A, m->slots, o_raw);
    m->launches += 1;
    return cudaGetLastError();
}
template <int KIND>
static cudaError_t launch_quad(SmolLm* m, const QuadSource& Q, const QuadArgs& A, int n_seqs, int max_n, float* o_raw, cudaStream_t st, size_t min_smem = 0) {
    switch (quad_pad(A.d)) {
        case 32: return launch_quad_sized<KIND, 32>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        case 64: return launch_quad_sized<KIND, 64>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        case 128: return launch_quad_sized<KIND, 128>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        default: return launch_quad_sized<KIND, 256>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
    }
}

template <int KIND, int DK>
static cudaError_t launch_chunks_sized(SmolLm* m, ChunkSource Q, ChunkArgs A, int n_seqs, int max_n, float* o_raw, cudaStream_t st, size_t min_smem) {
    constexpr bool REM = scan_removes(KIND);
    float* rec = reinterpret_cast<float*>(m->ws + m->o_rec);
    Q.cap = A.cap = m->cfg.max_step_tokens / kChunk + m->cfg.max_step_seqs + 1;
    const dim3 grid((max_n + kChunk - 1) / kChunk, n_seqs, Q.H);
    constexpr size_t prep_smem = chunk_prep_floats(KIND, DK) * sizeof(float);
    if constexpr (KIND == kScanGeneralDelta || KIND == kScanChannelDecay) pdl_launch(chunk_prep_kernel<KIND, DK>, grid, 128, prep_smem, st, Q, rec);
    else pdl_launch(chunk_prep_head_kernel<KIND, DK>, grid, 128, prep_smem, st, Q, rec);
    A.rec = rec;
    // Above 64 channels a block has an SM to itself.  Where single blocks of columns would not all run at once, it takes two, whose products share the
    // records' fragments (measured with operands in two parts: 12 heads of 128, 1801 tokens 140 us for 96 blocks of two, 144 for 192 single ones with half the ring, two
    // to an SM; 3 x 12 heads of 64, 1000 tokens 57 in twos, 46 single).
    const int parts = chunk_blocks(Q.columns), threads = chunk_warps(DK) * 64 + 32;
    if constexpr (DK > 64) {
        if (n_seqs * A.H * parts > m->n_sms) {
            plain_launch(chunk_scan_kernel<DK, REM, 2>, n_seqs * A.H * ((parts + 1) / 2), threads, std::max(chunk_smem(REM, DK, 2), min_smem), st, A, m->slots, o_raw);
            m->launches += 1;
            return cudaGetLastError();
        }
    }
    plain_launch(chunk_scan_kernel<DK, REM, 1>, n_seqs * A.H * parts, threads, std::max(chunk_smem(REM, DK, 1), min_smem), st, A, m->slots, o_raw);
    m->launches += 1;
    return cudaGetLastError();
}
template <int KIND>
static cudaError_t launch_chunks(SmolLm* m, const ChunkSource& Q, const ChunkArgs& A, int n_seqs, int max_n, float* o_raw, cudaStream_t st, size_t min_smem = 0) {
    switch (chunk_pad(A.d)) {
        case 32: return launch_chunks_sized<KIND, 32>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        case 64: return launch_chunks_sized<KIND, 64>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        case 128: return launch_chunks_sized<KIND, 128>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
        default: return launch_chunks_sized<KIND, 256>(m, Q, A, n_seqs, max_n, o_raw, st, min_smem);
    }
}

template <int DK>
static cudaError_t launch_gla_scan(const GlaArgs& A, int n_seqs, const float* dec, float* pool, float* o_raw, cudaStream_t st, size_t min_smem) {
    constexpr int CB = gla_block_cols(DK), threads = CB * gla_lanes(DK);
    const int groups = (A.dv + CB - 1) / CB;
    const size_t smem = std::max(2 * gla_buf_floats(DK) * sizeof(float), min_smem);
    if (A.head_decay) pdl_launch(gla_scan_kernel<DK, true>, n_seqs * A.H * groups, threads, smem, st, A, dec, pool, o_raw);
    else pdl_launch(gla_scan_kernel<DK, false>, n_seqs * A.H * groups, threads, smem, st, A, dec, pool, o_raw);
    return cudaGetLastError();
}
// the scan over key sizes up to 256: the smallest built size that holds A.d
static cudaError_t launch_gla_scan_any(SmolLm* m, const GlaArgs& A, int n_seqs, int n_tokens, int max_n, const float* dec, float* pool, float* o_raw, cudaStream_t st,
                                        size_t min_smem = 0) {
    if (chunks_pay(A.head_decay ? kScanHeadDecay : kScanChannelDecay, false, n_seqs, A.H, n_tokens, max_n, A.d, A.dv, m->n_sms)) {
        const ChunkSource Q{A.H, A.qk_share, A.d, A.dv, A.dv, A.q_src, A.k_src, A.q_ld, A.k_ld, A.v_src, A.v_ld, dec, A.head_decay, A.head_step, A.head_ld, 1,
                            nullptr, nullptr, 0.0f, A.seq_start, 0};
        const ChunkArgs S{A.H, A.d, A.dv, nullptr, 0, A.q_scale, A.seq_start, A.seq_pos0, A.seq_slot, A.slot_floats, A.state_off, A.n_slots, A.err, nullptr, 0, ConvIo{}};
        if (A.head_decay) return launch_chunks<kScanHeadDecay>(m, Q, S, n_seqs, max_n, o_raw, st, min_smem);
        return launch_chunks<kScanChannelDecay>(m, Q, S, n_seqs, max_n, o_raw, st, min_smem);
    }
    if (quad_pays(n_seqs, n_tokens, max_n)) {
        QuadSource Q{A.H, A.qk_share, A.d, A.q_src, A.k_src, A.q_ld, A.k_ld, dec, A.head_decay, A.head_step, A.head_ld, 1, nullptr, nullptr, 0.0f, A.seq_start, 0};
        QuadArgs S{A.H, A.d, A.dv, nullptr, 0, A.v_src, A.v_ld, A.q_scale, A.seq_start, A.seq_pos0, A.seq_slot, A.slot_floats, A.state_off, A.n_slots, A.err};
        if (A.head_decay) return launch_quad<kQuadHeadDecay>(m, Q, S, n_seqs, max_n, o_raw, st, min_smem);
        return launch_quad<kQuadChannelDecay>(m, Q, S, n_seqs, max_n, o_raw, st, min_smem);
    }
    if (A.d <= 16) return launch_gla_scan<16>(A, n_seqs, dec, pool, o_raw, st, min_smem);
    if (A.d <= 32) return launch_gla_scan<32>(A, n_seqs, dec, pool, o_raw, st, min_smem);
    if (A.d <= 64) return launch_gla_scan<64>(A, n_seqs, dec, pool, o_raw, st, min_smem);
    if (A.d <= 128) return launch_gla_scan<128>(A, n_seqs, dec, pool, o_raw, st, min_smem);
    return launch_gla_scan<256>(A, n_seqs, dec, pool, o_raw, st, min_smem);
}

template <int DK, bool DELTA>
static cudaError_t launch_group_scan(const GroupScanArgs& A, int n_seqs, float* pool, float* o_raw, cudaStream_t st, size_t min_smem) {
    constexpr int CB = gla_block_cols(DK), threads = CB * gla_lanes(DK);
    const int parts = (A.dv + (A.unit_out ? 1 : 0) + CB - 1) / CB;
    plain_launch(group_scan_kernel<DK, DELTA>, n_seqs * A.H * parts, threads, std::max(2 * group_scan_buf_floats(DK) * sizeof(float), min_smem), st, A, pool, o_raw);
    return cudaGetLastError();
}
// The gated delta rule's and the mLSTM's scan: by chunks, or four tokens at a time -- the group's products (not needed where every sequence brings one
// token), then the recurrence itself.
template <bool DELTA>
static cudaError_t launch_group_scan_any(SmolLm* m, const GroupScanArgs& A, float* pairs, int n_seqs, int n_tokens, int max_n, float* pool, float* o_raw, cudaStream_t st,
                                         size_t min_smem = 0) {
    if (chunks_pay(DELTA ? kScanGatedDelta : kScanHeadDecay, A.unit_out != nullptr, n_seqs, A.H, n_tokens, max_n, A.d, A.dv + (A.unit_out ? 1 : 0), m->n_sms)) {
        const ChunkSource Q{A.H, A.H / A.G, A.d, A.dv, A.dv + (A.unit_out ? 1 : 0), A.q_src, A.k_src, A.q_ld, A.k_ld, A.v_src, A.v_ld, nullptr, A.head, A.head + 1, 2 * A.H, 2,
                            nullptr, nullptr, 0.0f, A.seq_start, 0};
        const ChunkArgs S{A.H, A.d, A.dv, nullptr, 0, A.q_scale, A.seq_start, A.seq_pos0, A.seq_slot, A.slot_floats, A.state_off, A.n_slots, A.err, A.unit_out, A.unit_off, A.conv};
        m->launches += 1;
        return launch_chunks<DELTA ? kScanGatedDelta : kScanHeadDecay>(m, Q, S, n_seqs, max_n, o_raw, st, min_smem);
    }
    if (max_n > 1) {
        pdl_launch(scan_pairs_kernel<DELTA>, dim3((max_n + kScanGroup - 1) / kScanGroup, n_seqs, (A.G + 3) / 4), 128, 0, st, A, pairs);
        m->launches++;
    }
    m->launches++;
    if (A.d <= 16) return launch_group_scan<16, DELTA>(A, n_seqs, pool, o_raw, st, min_smem);
    if (A.d <= 32) return launch_group_scan<32, DELTA>(A, n_seqs, pool, o_raw, st, min_smem);
    if (A.d <= 64) return launch_group_scan<64, DELTA>(A, n_seqs, pool, o_raw, st, min_smem);
    if (A.d <= 128) return launch_group_scan<128, DELTA>(A, n_seqs, pool, o_raw, st, min_smem);
    return launch_group_scan<256, DELTA>(A, n_seqs, pool, o_raw, st, min_smem);
}

// attn_flash_tc_kernel where every row it copies is made of whole 16-byte pieces.  False: not launched (unaligned rows, sizes it is not built
// for, or attn_flash_kernel is the faster one).  A block takes an SM to itself, pads to 128 rows and spends 10 us or so before and after its keys,
// so it loses where there are more blocks than SMs and little to do in each: 12 heads of 64, 16 x 12 tokens 22 us against 17, 32 x 64 31
// against 21, 64 x 20 behind 100 others 70 against 47; but 16 x 16 behind 512 43 against 56, 8 x 300 33 against 42, one sequence of 9 11
// against 16.  A narrow latent (40 + 8), whose rows are keys and values in one: 16 x 16 behind 512 37 against 29.  Wider rows (128): 16 x 12
// 31 against 30, 32 x 64 56 against 65.  Heads of 16, one sequence of 9: 11 against 8.  Two maps: faster everywhere (12 heads of 64 / 128, 9 / 100 / 512 / 1536
// tokens 18 / 31 / 51 / 96 us against 27 / 33 / 55 / 144).  `keys`: positions in whole groups of ranges, as the captured steps know them.
template <int MAPS>
static bool launch_flash_tc(const AttnArgs& A, int n_seqs, int max_n, int keys, int n_sms, const bf16* qbuf, const bf16* pool, bf16* out, cudaStream_t st) {
    constexpr int kFewKeys = 256;
    const size_t rows = A.d | A.dv | A.out_ld | A.page_elems | A.k_off | A.k_ld | (A.v_in_k ? 0 : A.v_off | A.v_ld);
    if (rows % 8 != 0 || (reinterpret_cast<uintptr_t>(qbuf) | reinterpret_cast<uintptr_t>(pool) | reinterpret_cast<uintptr_t>(out)) % 16 != 0) return false;
    if (A.dv > 128 || A.d > (MAPS == 2 ? 64 : A.v_in_k ? 192 : 128)) return false;
    if (MAPS == 1) {
        const bool narrow = A.d <= 64 && A.dv <= 64, crowded = (long long)A.H * n_seqs > n_sms;
        if (crowded && max_n <= (narrow ? 64 : 16) && (keys <= kFewKeys || (narrow && A.v_in_k))) return false;
        if (!A.v_in_k && A.d <= 32 && A.dv <= 32 && max_n <= 16 && keys <= kFewKeys) return false;
    }
    const dim3 grid(A.H, n_seqs, (max_n + kFtRows - 1) / kFtRows);
#define SMOL_FLASH_TC(DK, DV, VK) plain_launch(attn_flash_tc_kernel<DK, DV, VK, MAPS>, grid, ft_threads(DV, MAPS), ft_smem(DK, DV, VK, MAPS), st, A, qbuf, pool, out)
    if constexpr (MAPS == 1) {
        if (A.v_in_k) {
            if (A.d <= 64) SMOL_FLASH_TC(64, 64, true);
            else if (A.d <= 128) SMOL_FLASH_TC(128, 128, true);
            else SMOL_FLASH_TC(192, 128, true);
            return true;
        }
        if (A.d > 64) {
            SMOL_FLASH_TC(128, 128, false);
            return true;
        }
    }
    if (A.dv <= 64) SMOL_FLASH_TC(64, 64, false);
    else SMOL_FLASH_TC(64, 128, false);
#undef SMOL_FLASH_TC
    return true;
}

// The attention kernels over the rows of a step: prompt portions on the tensor-core form (bf16, `flash`) or the
// warp-per-row form, sequences of few tokens on the split-range form.  `A` is complete except for the fields set here.
template <class T, int MAXV, int MAPS>
static void launch_attention(SmolLm* m, const SmolLmStep* s, AttnArgs& A, bool flash, const T* qbuf, const T* pool, T* mix, cudaStream_t st) {
    const SmolLmConfig& c = m->cfg;
    const int Tn = s->n_tokens;
    A.seq_start = s->seq_start;
    A.split_len = m->split_len;
    A.short_rows = s->n_seqs * kShortSeq;
    A.part = reinterpret_cast<float*>(m->ws + m->o_part);
    const int min_n = s->min_seq_tokens > 0 ? s->min_seq_tokens : 1;
    const int max_n = s->max_seq_tokens > 0 ? s->max_seq_tokens : Tn;
    const int max_pos = s->max_pos > 0 ? std::min(s->max_pos, c.max_context - 1) : c.max_context - 1;
    A.n_splits = std::min(m->max_splits, (max_pos / m->split_len + 4) / 4 * 4);
    const int keys = A.n_splits * m->split_len;
    if (A.window > 0) A.n_splits = std::min(A.n_splits, ((A.window - 1) / m->split_len + 2 + 3) / 4 * 4);      // ranges a window can touch
    if (max_n > kShortSeq) {
        if (flash) {
            dim3 grid(A.H, s->n_seqs, (max_n + 63) / 64);
            const int hp = std::max(A.d, A.dv);
            const bf16* qb = reinterpret_cast<const bf16*>(qbuf);
            const bf16* pl = reinterpret_cast<const bf16*>(pool);
            bf16* mx = reinterpret_cast<bf16*>(mix);
#define SMOL_FLASH(DK, DV, VK) plain_launch(attn_flash_kernel<DK, DV, VK, MAPS>, grid, 128 * MAPS, flash_smem_bytes(DK, DV, VK, MAPS), st, A, qb, pl, mx)
            bool done = launch_flash_tc<MAPS>(A, s->n_seqs, max_n, keys, m->n_sms, qb, pl, mx, st);
            if constexpr (MAPS == 1) {
                if (done || !A.v_in_k) {
                } else if (A.d <= 64) SMOL_FLASH(64, 64, true);
                else if (A.d <= 128) SMOL_FLASH(128, 128, true);
                else if (A.dv <= 128) SMOL_FLASH(192, 128, true);
                else SMOL_FLASH(192, 192, true);
                done = done || A.v_in_k;
            }
            if (done) {
            } else if (hp <= 32) SMOL_FLASH(32, 32, false);
            else if (hp <= 64) SMOL_FLASH(64, 64, false);
            else if (A.d <= 64) SMOL_FLASH(64, 128, false);
            else SMOL_FLASH(128, 128, false);
#undef SMOL_FLASH
        } else {
            // every row, also those of short sequences
            const int au = Tn * A.H;
            // Rows that are not whole 16-byte pieces are staged an element at a time, which a block of four rows a warp pays for once per sixteen rows.  A layer of 8 heads as a
            // whole against one that reads keys and values where they lie (attn_kernel): bf16, keys or values of whole pieces 0.44 to 0.88; neither, heads of 130: 1 x 300 tokens (152
            // blocks of 16 rows) 1.10, 1 x 64 (32) 1.07, 1 x 150 (80) 0.92, 1 x 1100 (552) 0.70; keys of 20 and values of 140, 7 x 170 1.40, 4 x 40 (96) 0.81, of 300 1.51 and 0.86.  float32, heads of 33 0.63
            // to 0.89, of 130 1 x 300 1.14, 7 x 170 (616) 0.99, 1 x 1100 0.85.  Whole pieces: 0.2 to 0.8.
            const int e = 16 / (int)sizeof(T), blocks = s->n_seqs * A.H * ((max_n + 15) / 16);
            const bool k_pieces = A.d % e == 0 && A.k_ld % e == 0 && A.k_off % e == 0, v_pieces = A.v_in_k ? k_pieces : A.dv % e == 0 && A.v_ld % e == 0 && A.v_off % e == 0;
            const bool many = blocks >= 3 * m->n_sms, wave = blocks < m->n_sms && blocks * 5 >= 2 * m->n_sms;      // (wave: of blocks of four rows)
            const bool rows = (k_pieces && v_pieces) || (sizeof(T) == 4 ? std::max(A.d, A.dv) <= 64 || many
                              : wave || (A.dv <= 256 && (k_pieces || v_pieces || (A.d >= 64 && many))));
            const int R = blocks >= m->n_sms ? 4 : 1;      // four rows of a warp where that still fills the SMs
            const size_t smem = rows_smem<T>(R, A.d, A.dv, A.v_in_k);
            if (smem > (size_t)kRowsSmemMax || !rows)
                plain_launch(attn_kernel<T, MAXV, MAPS>, (au + kAttnWarps - 1) / kAttnWarps, kAttnWarps * 32, kAttnWarps * A.d * sizeof(float), st, A, qbuf, pool, mix);
            else if (R == 4) plain_launch(attn_rows_kernel<T, MAXV, MAPS, 4>, dim3((max_n + 15) / 16, A.H, s->n_seqs), kRowsWarps * 32, smem, st, A, qbuf, pool, mix);
            else plain_launch(attn_rows_kernel<T, MAXV, MAPS, 1>, dim3((max_n + 3) / 4, A.H, s->n_seqs), kRowsWarps * 32, smem, st, A, qbuf, pool, mix);
        }
        m->launches += 1;
    }
    if (min_n <= kShortSeq && (flash || max_n <= kShortSeq)) {
        const int Gq = A.H / A.G * MAPS, nwarp = std::min(Gq, 8), groups = (Gq + nwarp - 1) / nwarp;
        const int pad = 16 / (int)sizeof(T);
        // queries and weights of every warp, then the staged keys and values or, afterwards, the states to be joined
        auto smem_of = [&](int keys, int parts) {
            const size_t staged = (size_t)keys * (MAPS * (A.d + pad + 1) + (A.v_in_k ? 0 : split_value_ld<T>(A.dv))) * sizeof(T), joined = parts == 2 ? (size_t)nwarp * (MAXV * 32 + 2) * 4 : 0;
            return ((size_t)nwarp * (parts * A.d + keys) * 4 + 15) / 16 * 16 + std::max(staged, joined);
        };
        dim3 grid(A.short_rows, A.G * groups, A.n_splits);
        const bool alone = (long long)std::min(Tn, A.short_rows) * A.G * groups * A.n_splits <= m->n_sms;
        bool wide = false;
        if constexpr (MAXV == 8) {
            wide = smem_of(64, 2) <= (size_t)kAttnSplitWideSmem;
            if (wide && alone) pdl_launch(attn_split_kernel<T, MAXV, 2, 2>, grid, nwarp * 64, smem_of(64, 2), st, A, qbuf, pool);
            else if (wide) pdl_launch(attn_split_kernel<T, MAXV, 2, 1>, grid, nwarp * 32, smem_of(64, 1), st, A, qbuf, pool);
        }
        if (!wide) pdl_launch(attn_split_kernel<T, MAXV, 1, 1>, grid, nwarp * 32, smem_of(32, 1), st, A, qbuf, pool);
        pdl_launch(attn_merge_kernel<T, MAXV, MAPS>, A.short_rows * A.H, kMergeWarps * MAPS * 32, kMergeWarps * MAPS * (A.dv + 1) * sizeof(float), st, A, mix);
        m->launches += 2;
    }
}

// The tiled sigmoid attention over the sequences that bring more than kShortSeq tokens.  Returns false where this form does
// not apply (fp32 engine, sizes it is not built for, unaligned cached rows, more shared memory than an SM has): the caller
// then runs the warp-per-head kernel over every row.
static size_t sigmoid_flash_smem(int H, int G, int DK, int KT) {
    return (size_t)2 * G * KT * (DK + 8) * sizeof(bf16) + ((size_t)H * 16 * (KT + 8) + (size_t)H * H) * sizeof(float);
}
template <int DK, int HPW>
static bool launch_sigmoid_flash_sized(const SigmoidArgs& S, dim3 grid, int threads, const bf16* qbuf, const bf16* pool, bf16* out, cudaStream_t st) {
    const AttnArgs& A = S.a;
    if (sigmoid_flash_smem(A.H, A.G, DK, 64) <= (size_t)kSigmoidSmemMax) {
        pdl_launch(sigmoid_flash_kernel<DK, HPW, 64>, grid, threads, sigmoid_flash_smem(A.H, A.G, DK, 64), st, S, qbuf, pool, out);
        return true;
    }
    if (sigmoid_flash_smem(A.H, A.G, DK, 32) <= (size_t)kSigmoidSmemMax) {
        pdl_launch(sigmoid_flash_kernel<DK, HPW, 32>, grid, threads, sigmoid_flash_smem(A.H, A.G, DK, 32), st, S, qbuf, pool, out);
        return true;
    }
    return false;
}
static bool launch_sigmoid_flash(SmolLm* m, const SmolLmStep* s, SigmoidArgs& S, int max_n, const bf16* qbuf, const bf16* pool, bf16* out,
                                 bool is_bf16, cudaStream_t st) {
    const AttnArgs& A = S.a;
    if (!is_bf16 || A.d % 8 != 0 || A.d > 128 || A.k_off % 8 != 0 || A.v_off % 8 != 0) return false;
    // Key ranges: a quarter of the positions a row tile can see (at least 256, whole 64-key tiles), more only where that
    // would cut a tile into more than kSigmoidRanges ranges.  The ranges depend on the mask and the pool's size alone.
    const int span = S.chunk > 0 ? std::min(S.chunk + 15, m->cfg.max_context) : m->cfg.max_context;
    auto ranges_of = [&](int len) { return S.chunk > 0 ? (span + len - 1) / len + 1 : (span + len - 1) / len; };
    int len = std::max(256, ((span + 3) / 4 + 63) / 64 * 64);
    while (ranges_of(len) > kSigmoidRanges) len += 64;
    S.range_len = len;
    S.n_ranges = ranges_of(len);
    if (span <= 512) {                       // few keys per row: one range, the result written directly
        S.range_len = 1 << 30;
        S.n_ranges = 1;
    }
    S.partial = reinterpret_cast<float*>(m->ws + m->o_spart);
    const dim3 grid((max_n + 15) / 16, s->n_seqs, S.n_ranges);
    bool done;
    if (A.H <= 16) {
        const int threads = A.H * 32;
        if (A.d <= 32) done = launch_sigmoid_flash_sized<32, 1>(S, grid, threads, qbuf, pool, out, st);
        else if (A.d <= 64) done = launch_sigmoid_flash_sized<64, 1>(S, grid, threads, qbuf, pool, out, st);
        else if (A.d <= 96) done = launch_sigmoid_flash_sized<96, 1>(S, grid, threads, qbuf, pool, out, st);
        else done = launch_sigmoid_flash_sized<128, 1>(S, grid, threads, qbuf, pool, out, st);
    } else {
        const int threads = (A.H + 1) / 2 * 32;
        if (A.d <= 32) done = launch_sigmoid_flash_sized<32, 2>(S, grid, threads, qbuf, pool, out, st);
        else if (A.d <= 64) done = launch_sigmoid_flash_sized<64, 2>(S, grid, threads, qbuf, pool, out, st);
        else done = false;
    }
    if (done && S.n_ranges > 1) {
        pdl_launch(sigmoid_merge_kernel, A.n_tokens, 128, 0, st, S, out);
        m->launches += 1;
    }
    if (done) m->launches += 1;
    return done;
}

template <class T>
static void launch_residual_norm(const ResidualArgs& A, int rows, int threads, T* hn, cudaStream_t st) {
    uintptr_t at = 0;
    for (const void* p : {(const void*)A.x, (const void*)A.y, (const void*)A.y2, (const void*)A.y_w, (const void*)A.y2_w, (const void*)A.rs.yp, (const void*)A.trace,
                          (const void*)A.x0, (const void*)A.cat, (const void*)A.y_b, (const void*)A.next.w, (const void*)A.next.shift, (const void*)hn})
        at |= reinterpret_cast<uintptr_t>(p);
    if (A.D % 4 == 0 && at % 16 == 0) pdl_launch(residual_norm_kernel<T, true>, rows, threads, A.D * sizeof(float), st, A, hn);
    else pdl_launch(residual_norm_kernel<T, false>, rows, threads, A.D * sizeof(float), st, A, hn);
}

template <class T>
static void launch_gla_out(const GlaArgs& A, const float* o_raw, T* out, cudaStream_t st) {
    const int units = A.n_tokens * A.H;
    const size_t gate_at = A.gate_off >= 0 ? (size_t)A.gate_off : (size_t)2 * A.H * A.d + (size_t)A.H * A.dv;
    // whole 16-byte pieces of every row
    const bool vec = A.dv % 4 == 0 && A.n_in % 4 == 0 && gate_at % 4 == 0 && A.out_ld % 4 == 0 && addresses_of(A.proj, A.out_norm, o_raw) % 16 == 0 && addresses_of(out) % 8 == 0;
    if (vec && A.dv == 64) pdl_launch(gla_out_vec_kernel<T, 16>, (units + 7) / 8, 128, 0, st, A, o_raw, out);
    else if (vec && A.dv == 128) pdl_launch(gla_out_vec_kernel<T, 32>, (units + 3) / 4, 128, 0, st, A, o_raw, out);
    else pdl_launch(gla_out_kernel<T>, (units + 3) / 4, 128, 0, st, A, o_raw, out);
}

template <class T>
static int step_impl(SmolLm* m, const SmolLmStep* s, cudaStream_t st) {
    const SmolLmConfig& c = m->cfg;
    const int Tn = s->n_tokens, D = c.width;
    float* x = reinterpret_cast<float*>(m->ws + m->o_x);
    T* hn = reinterpret_cast<T*>(m->ws + m->o_hn);
    float* proj = reinterpret_cast<float*>(m->ws + m->o_proj);
    T* mix = reinterpret_cast<T*>(m->ws + m->o_mix);
    float* y = reinterpret_cast<float*>(m->ws + m->o_y);
    float* z = reinterpret_cast<float*>(m->ws + m->o_z);
    T* act = reinterpret_cast<T*>(m->ws + m->o_act);
    float* dec = reinterpret_cast<float*>(m->ws + m->o_dec);
    float* uk = reinterpret_cast<float*>(m->ws + m->o_u);
    float* auk = reinterpret_cast<float*>(m->ws + m->o_au);
    float* oraw = reinterpret_cast<float*>(m->ws + m->o_oraw);
    T* qbuf = reinterpret_cast<T*>(m->ws + m->o_q);
    T* hw = reinterpret_cast<T*>(m->ws + m->o_hw);
    int32_t* err = reinterpret_cast<int32_t*>(m->ws + m->o_err);
    float* hist = reinterpret_cast<float*>(m->ws + m->o_hist);
    T* pool = static_cast<T*>(m->pages);
    const int nthr = D >= 1024 ? 256 : 128;
    const bool postnorm = c.block == SMOL_LM_BLOCK_POSTNORM, parallel = c.block == SMOL_LM_BLOCK_PARALLEL;
    const bool prenorm = c.block == SMOL_LM_BLOCK_PRENORM, outnorm = c.block == SMOL_LM_BLOCK_OUTNORM;
    float* x0 = m->any_restart ? reinterpret_cast<float*>(m->ws + m->o_x0) : nullptr;
    T* cat = m->any_merge ? reinterpret_cast<T*>(m->ws + m->o_cat) : nullptr;
    T* mix2 = reinterpret_cast<T*>(m->ws + m->o_mix2);
    float* y2 = reinterpret_cast<float*>(m->ws + m->o_y2);
    auto norm_of = [&](const float* w, const float* shift, const float* alpha) { return NormSpec{c.norm_kind, w, shift, alpha, c.norm_eps}; };
    const NormSpec no_norm{c.norm_kind, nullptr, nullptr, nullptr, c.norm_eps}, copy_row{kNormCopy, nullptr, nullptr, nullptr, c.norm_eps};
    const size_t hist_stride = (size_t)Tn * D;
    const int max_n = s->max_seq_tokens > 0 ? s->max_seq_tokens : Tn;      // most tokens a sequence brings
    constexpr bool kIsF32 = sizeof(T) == 4;
    const float woff = c.norm_plain ? 0.0f : 1.0f;
    float* conv = reinterpret_cast<float*>(m->ws + m->o_conv);
    float* head = reinterpret_cast<float*>(m->ws + m->o_head);
    auto cast_grid = [](size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 8); };

    if (postnorm) {
        pdl_launch(embed_gain_norm_kernel<T>, Tn, nthr, 0, st, s->tokens, static_cast<const T*>(m->g.embed), D, c.vocab, m->g.embed_norm, c.norm_eps, x, hist, hn);
    } else if (outnorm) {
        pdl_launch(embed_prenorm_kernel<T>, Tn, nthr, 0, st, s->tokens, static_cast<const T*>(m->g.embed), c.embed_scale, D, c.vocab, copy_row, x, nullptr, hn, nullptr);
    } else if (prenorm || parallel) {
        const SmolLmLayer& L0 = m->layers[m->runs[0].layer];
        const bool merge = m->runs[0].flags & SMOL_LM_RUN_MERGE_EMBED;
        pdl_launch(embed_prenorm_kernel<T>, Tn, nthr, 0, st, s->tokens, static_cast<const T*>(m->g.embed), c.embed_scale, D, c.vocab,
                                                     merge ? no_norm : norm_of(L0.norm1, L0.norm1_shift, L0.norm1_alpha), x, x0, hn, cat);
    } else {
        const T* table = static_cast<const T*>(m->g.embed);
        const float* w = m->layers[m->runs[0].layer].norm1;
        if (!row_pieces(Tn, D, addresses_of(table, w, x, hn), [&](auto v, auto lone, int blocks, int threads) {
                pdl_launch(embed_norm_vec_kernel<T, decltype(v)::value, decltype(lone)::value>, blocks, threads, 0, st, s->tokens, table, c.embed_scale, D, c.vocab, w, c.norm_eps, x, hn, woff, Tn);
            }))
            pdl_launch(embed_norm_kernel<T>, Tn, nthr, 0, st, s->tokens, table, c.embed_scale, D, c.vocab, w, c.norm_eps, x, hn, woff);
    }
    m->launches++;
    auto add_norm = [&](const float* wb, const float* ls, const float* wn, const float* yb, const RoutedSum& rs) {
        if (!row_pieces(Tn, D, addresses_of(x, y, wb, ls, wn, yb, hn, rs.yp), [&](auto v, auto lone, int blocks, int threads) {
                pdl_launch(add_norm_vec_kernel<T, decltype(v)::value, decltype(lone)::value>, blocks, threads, 0, st, x, y, wb, ls, wn, c.norm_eps, D, hn, woff, yb, rs, hn, Tn);
            }))
            pdl_launch(add_norm_kernel<T>, Tn, nthr, D * sizeof(float), st, x, y, wb, ls, wn, c.norm_eps, D, hn, woff, yb, rs, hn);
    };
    for (size_t n = 0; n < m->runs.size(); ++n) {
        const RunInfo& R = m->runs[n];
        const SmolLmLayer& L = m->layers[R.layer];
        const int n_in_main = n_in_of(L), n_in = full_n_in_of(L, c.block);
        if (R.flags & SMOL_LM_RUN_MERGE_EMBED) {
            // the stream starts anew from the merged rows, which the previous run's last kernel (or the embedding) has left in cat
            CU(linear<T>(m, cat, static_cast<const T*>(m->g.w_merge), x, Tn, D, 2 * D, st));
            pdl_launch(prenorm_rows_kernel<T>, Tn, nthr, 0, st, x, nullptr, norm_of(L.norm1, L.norm1_shift, L.norm1_alpha), D, hn);
            m->launches++;
        }
        CU(linear<T>(m, hn, static_cast<const T*>(L.w_in), proj, Tn, n_in, D, st));
        // row stride of the mixers' shared result (parallel block: the shared expert's unit stands behind the mixer's columns)
        const int mix_ld = mix_cols_of(L) + (L.side ? mix_cols_of(*L.side) : 0) + (parallel && L.mlp == SMOL_LM_MLP_EXPERTS ? L.shared_ff : 0);
        int mix_cols;
        int out_ld_now = mix_ld;        // row stride of the buffer the current mixer writes
        const T* mix_in = mix;          // what the output projection reads
        cudaStream_t ms = st;           // the stream the current mixer runs on
        // Softmax attention over keys and values in the paged pool.  pj / bias: this mixer's rows of the fused projection.
        auto attention = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, const float* bias, T* mix_at) -> int {
            AttnArgs A;
            A.proj = pj; A.n_in = n_in; A.bias = bias;
            A.tok_seq = s->tok_seq; A.tok_pos = s->tok_pos; A.block_table = s->block_table;
            A.max_pages = s->max_pages; A.page_size = c.page_size; A.n_pages = m->n_pages;
            A.page_elems = m->page_elems; A.k_off = Ri.k_off; A.v_off = Ri.v_off;
            A.H = M.heads; A.scale = M.score_scale; A.eps = c.norm_eps;
            A.n_tokens = Tn; A.err = err;
            A.G = M.kv_heads; A.d = M.dim; A.dv = M.vdim;
            A.k_ld = M.dim; A.v_ld = M.vdim; A.v_in_k = 0;
            A.gate_off = (size_t)attn_qkv_rows(M); A.gate_ld = M.vdim; A.gate_step = 1;
            A.has_gate = M.no_gate ? 0 : 1;
            A.q_norm = M.q_norm; A.k_norm = M.k_norm; A.r1 = M.dist_r1; A.r2 = M.dist_r2; A.sink = M.sink;
            A.slope = M.dist_slope; A.window = M.window; A.softcap = M.softcap; A.two_over_cap = M.softcap > 0.0f ? 2.0f / M.softcap : 0.0f;
            A.out_ld = out_ld_now; A.out_scale = M.mix_scale;
            A.temp_coef = M.q_temp_coef; A.temp_every = M.q_temp_every;
            A.maps = maps_of(M); A.diff_lambda = M.diff_lambda; A.diff_scale = M.diff_scale; A.own_kv = M.kv_from == 0;
            if (M.norm_whole) {
                const int threads = Tn > 64 ? 128 : 256;      // few tokens: more loads in flight per token
                A.rot_pairs = M.rot_dims / 2; A.rot_half = M.rot_half; A.rot_mult = M.rot_mult != 0.0f ? M.rot_mult : 1.0f;
                A.freq = reinterpret_cast<const float*>(m->ws + m->o_freq) + Ri.freq_off;
                if (A.rot_pairs > 0) pdl_launch(attn_prep_whole_kernel<T, true>, Tn, threads, 0, ms, A, qbuf, pool);
                else pdl_launch(attn_prep_whole_kernel<T, false>, Tn, threads, 0, ms, A, qbuf, pool);
            } else {
                const int units = Tn * (M.heads * A.maps + (A.own_kv ? M.kv_heads * (A.maps + 1) : 0));
                // whole 16-byte pieces of every row read, 4-element pieces of every row written
                const bool vec = M.dim % 4 == 0 && M.vdim % 4 == 0 && n_in % 4 == 0 && Ri.k_off % 4 == 0 && Ri.v_off % 4 == 0 && m->page_elems % 4 == 0 &&
                                 addresses_of(pj, bias, M.q_norm, M.k_norm, qbuf, pool) % 16 == 0;
                if (vec && std::max(M.dim, M.vdim) <= 64) pdl_launch(attn_prep_vec_kernel<T, 16>, (units + 7) / 8, 128, 0, ms, A, qbuf, pool);
                else if (vec && std::max(M.dim, M.vdim) <= 128) pdl_launch(attn_prep_vec_kernel<T, 32>, (units + 3) / 4, 128, 0, ms, A, qbuf, pool);
                else pdl_launch(attn_prep_kernel<T>, (units + 3) / 4, 128, 0, ms, A, qbuf, pool);
            }
            m->launches += 1;
            const bool flash = sizeof(T) == 2 && std::max(M.dim, M.vdim) <= 128;
            if (A.maps == 2) {
                if (M.vdim <= 256) launch_attention<T, 8, 2>(m, s, A, flash, qbuf, pool, mix_at, ms);
                else launch_attention<T, 16, 2>(m, s, A, flash, qbuf, pool, mix_at, ms);
            } else if (M.vdim <= 256) launch_attention<T, 8, 1>(m, s, A, flash, qbuf, pool, mix_at, ms);
            else launch_attention<T, 16, 1>(m, s, A, flash, qbuf, pool, mix_at, ms);
            return SMOL_OK;
        };
        // State-space recurrence: convolution and per-head step / decay, the scan over the slot's state, then skip, gate and the
        // grouped norm (whose kernel also leaves the slot's new convolution inputs).
        auto state_space = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, const float* bias, T* mix_at) -> int {
            const int inner = M.heads * M.vdim, gn = M.bc_groups * M.n_state, ch = inner + 2 * gn;
            SsdArgs P;
            P.proj = pj; P.bias = bias; P.n_in = n_in; P.H = M.heads; P.dv = M.vdim; P.N = M.n_state; P.G = M.bc_groups;
            P.taps = M.conv_taps; P.parts = M.norm_parts; P.n_tokens = Tn; P.n_seqs = s->n_seqs; P.eps = c.norm_eps;
            P.conv_w = M.conv_w; P.conv_b = M.conv_b; P.dt_bias = M.dt_bias; P.a_log = M.a_log; P.skip = M.skip; P.out_norm = M.out_norm;
            P.seq_start = s->seq_start; P.seq_pos0 = s->seq_pos0; P.seq_slot = s->seq_slot; P.tok_seq = s->tok_seq;
            P.slot_floats = m->slot_floats; P.conv_off = Ri.conv_off; P.n_slots = m->n_slots; P.err = err;
            P.out_ld = out_ld_now; P.out_scale = M.mix_scale;
            const dim3 cgrid(Tn, (ch + 127) / 128);
            pdl_launch(ssd_conv_kernel, cgrid, 128, 0, ms, P, m->slots, conv, head);
            GlaArgs A;
            A.proj = pj; A.n_in = n_in; A.H = M.heads; A.d = M.n_state; A.dv = M.vdim; A.rank = 0; A.n_tokens = Tn;
            A.q_scale = 1.0f; A.tau = 1.0f; A.eps = c.norm_eps;
            A.decay_w2 = A.decay_bias = A.out_norm = nullptr;
            A.seq_start = s->seq_start; A.seq_pos0 = s->seq_pos0; A.seq_slot = s->seq_slot;
            A.slot_floats = m->slot_floats; A.state_off = Ri.state_off; A.n_slots = m->n_slots; A.err = err;
            A.q_src = conv + inner + gn; A.k_src = conv + inner; A.v_src = conv;
            A.q_ld = A.k_ld = A.v_ld = ch;
            A.qk_share = M.heads / M.bc_groups;
            A.head_decay = head; A.head_step = head + (size_t)Tn * M.heads; A.head_ld = M.heads;
            A.out_ld = out_ld_now; A.out_scale = 1.0f;
            CU(launch_gla_scan_any(m, A, s->n_seqs, Tn, max_n, nullptr, m->slots, oraw, ms));
            pdl_launch(ssd_out_kernel<T>, dim3(Tn, M.norm_parts), 256, 0, ms, P, oraw, conv, mix_at, m->slots);
            m->launches += 3;
            return SMOL_OK;
        };
        // Mixers side by side that own their output projections keep their results apart: row stride = own columns.
        const bool own_proj = L.side && L.proj_norm;
        // Sigmoid attention over keys and values in the paged pool.
        auto sigmoid_attention = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, const float* bias, T* mix_at, int ld) -> int {
            SigmoidArgs S;
            AttnArgs& A = S.a;
            A.proj = pj; A.n_in = n_in; A.bias = bias;
            A.tok_seq = s->tok_seq; A.tok_pos = s->tok_pos; A.block_table = s->block_table;
            A.max_pages = s->max_pages; A.page_size = c.page_size; A.n_pages = m->n_pages;
            A.page_elems = m->page_elems; A.k_off = Ri.k_off; A.v_off = Ri.v_off;
            A.H = M.heads; A.G = M.kv_heads; A.d = M.dim; A.dv = M.vdim; A.scale = M.score_scale; A.eps = c.norm_eps;
            A.n_tokens = Tn; A.err = err; A.seq_start = s->seq_start;
            A.k_ld = M.dim; A.v_ld = M.vdim; A.v_in_k = 0;
            A.gate_off = (size_t)(M.heads + M.kv_heads) * M.dim; A.gate_ld = 1; A.gate_step = 0; A.has_gate = 1;
            A.q_norm = A.k_norm = A.r1 = A.r2 = A.sink = A.slope = nullptr;
            A.window = 0; A.softcap = A.two_over_cap = 0.0f;
            A.split_len = A.n_splits = A.short_rows = 0; A.part = nullptr;
            A.out_ld = ld; A.out_scale = 1.0f;
            S.chunk = M.chunk; S.rot_pairs = M.rot_dims / 2; S.head_bias = M.head_bias; S.talk = M.talk; S.only = 0;
            S.range_len = 1 << 30; S.n_ranges = 1; S.partial = nullptr;
            S.freq = reinterpret_cast<const float*>(m->ws + m->o_freq) + Ri.freq_off;
            const int units = Tn * (M.heads + M.kv_heads);
            pdl_launch(sigmoid_prep_kernel<T>, (units + 3) / 4, 128, 0, ms, S, qbuf, pool);
            m->launches += 1;
            const int min_n = s->min_seq_tokens > 0 ? s->min_seq_tokens : 1;
            // sequences that bring more than a few tokens take the tiled tensor-core form (bf16), the others a warp per head
            const bool tiled = max_n > kShortSeq && launch_sigmoid_flash(m, s, S, max_n, reinterpret_cast<const bf16*>(qbuf), reinterpret_cast<const bf16*>(pool),
                                                                         reinterpret_cast<bf16*>(mix_at), sizeof(T) == 2, ms);
            // sequences of few tokens (decoding): key ranges over separate blocks, merged afterwards
            const size_t split_smem = sigmoid_split_smem<T>(M.heads, M.kv_heads, M.dim, M.vdim);
            const bool split = min_n <= kShortSeq && split_smem <= (size_t)kSigmoidSmemMax;
            if (split) {
                const int max_pos = s->max_pos > 0 ? std::min(s->max_pos, c.max_context - 1) : c.max_context - 1;
                A.split_len = m->split_len;
                A.short_rows = s->n_seqs * kShortSeq;
                A.part = reinterpret_cast<float*>(m->ws + m->o_part);
                A.n_splits = std::min(m->max_splits, (max_pos / m->split_len + 4) / 4 * 4);
                if (M.chunk > 0) A.n_splits = std::min(A.n_splits, ((M.chunk - 1) / m->split_len + 2 + 3) / 4 * 4);      // ranges a chunk can touch
                const dim3 grid(A.short_rows, A.n_splits);
                if (M.vdim <= 256) pdl_launch(sigmoid_split_kernel<T, 8>, grid, M.heads * 32, split_smem, ms, S, qbuf, pool);
                else pdl_launch(sigmoid_split_kernel<T, 16>, grid, M.heads * 32, split_smem, ms, S, qbuf, pool);
                pdl_launch(sigmoid_short_merge_kernel<T>, A.short_rows, 128, 0, ms, S, mix_at);
                m->launches += 2;
            }
            const bool long_left = max_n > kShortSeq && !tiled, short_left = min_n <= kShortSeq && !split;
            if (long_left || short_left) {
                // the warp-per-head form: every row, or only the rows the other two forms left
                S.only = (long_left && short_left) ? 0 : long_left ? 1 : 2;
                const size_t smem = ((size_t)M.heads * (M.dim + 32) + (size_t)M.heads * M.heads) * sizeof(float);
                if (M.vdim <= 256) pdl_launch(sigmoid_attn_kernel<T, 8>, Tn, M.heads * 32, smem, ms, S, qbuf, pool, mix_at);
                else pdl_launch(sigmoid_attn_kernel<T, 16>, Tn, M.heads * 32, smem, ms, S, qbuf, pool, mix_at);
                m->launches += 1;
            }
            return SMOL_OK;
        };
        // The scan's arguments for a linear attention with state [dim, vdim] per head in the slot.
        auto scan_args = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj) {
            GlaArgs A;
            A.proj = pj; A.n_in = n_in; A.H = M.heads; A.d = M.dim; A.dv = M.vdim; A.rank = 0; A.n_tokens = Tn;
            A.q_scale = 1.0f; A.tau = 1.0f; A.eps = c.norm_eps;
            A.decay_w2 = A.decay_bias = A.out_norm = nullptr;
            A.seq_start = s->seq_start; A.seq_pos0 = s->seq_pos0; A.seq_slot = s->seq_slot;
            A.slot_floats = m->slot_floats; A.state_off = Ri.state_off; A.n_slots = m->n_slots; A.err = err;
            A.qk_share = 1; A.head_decay = A.head_step = nullptr; A.head_ld = M.heads;
            A.out_ld = M.heads * M.vdim; A.out_scale = 1.0f;
            return A;
        };
        // Lightning attention: silu on q, k, v; the scan in its one-decay-per-head form; norm over all heads, sigmoid gate.
        auto lightning = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, T* mix_at, int ld) -> int {
            const int hd = M.heads * M.dim, hv = M.heads * M.vdim, na = 2 * hd + hv;
            LinPrepArgs P{pj, n_in, M.heads, M.dim, M.vdim, Tn, M.head_decay, nullptr, nullptr};
            pdl_launch(lightning_prep_kernel, dim3(Tn, (na + 1023) / 1024), 256, 0, ms, P, conv, head);
            GlaArgs A = scan_args(M, Ri, pj);
            A.q_src = conv; A.k_src = conv + hd; A.v_src = conv + 2 * hd;
            A.q_ld = A.k_ld = A.v_ld = na;
            A.head_decay = head; A.head_step = head + (size_t)Tn * M.heads;
            CU(launch_gla_scan_any(m, A, s->n_seqs, Tn, max_n, nullptr, m->slots, oraw, ms));
            LinOutArgs O{pj, n_in, hv, hv, hv, 1, ld, (size_t)2 * hd + hv, c.norm_eps, 1.0f, M.out_norm};
            pdl_launch(lin_attn_out_kernel<T>, dim3(Tn, 1), 256, 0, ms, O, oraw, mix_at);
            m->launches += 3;
            return SMOL_OK;
        };
        // Retention: rotated q and k, the scan with one constant decay per head, RMS division per head and silu gate.
        auto retention = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, T* mix_at, int ld) -> int {
            const int hd = M.heads * M.dim, pairs = M.rot_dims / 2, per = M.heads * (M.dim - pairs);
            RetentionArgs P{pj, n_in, M.heads, M.dim, pairs, M.rot_half, M.score_scale, reinterpret_cast<const float*>(m->ws + m->o_freq) + Ri.freq_off, s->tok_pos};
            pdl_launch(retention_prep_kernel, dim3(Tn, (per + 511) / 512), 128, 0, ms, P, conv);
            GlaArgs A = scan_args(M, Ri, pj);
            A.q_src = conv; A.k_src = conv + hd; A.v_src = pj + 2 * hd;
            A.q_ld = A.k_ld = 2 * hd; A.v_ld = n_in;
            A.head_decay = M.head_decay; A.head_ld = 0;
            CU(launch_gla_scan_any(m, A, s->n_seqs, Tn, max_n, nullptr, m->slots, oraw, ms, parallel && Tn > kGraphMaxTokens ? kScanSpread : 0));
            A.out_ld = ld; A.out_scale = M.mix_scale;
            launch_gla_out<T>(A, oraw, mix_at, ms);
            m->launches += 3;
            return SMOL_OK;
        };
        // The four-token scan's arguments for a state [dim, vdim] per head in the slot.
        float* pairs = reinterpret_cast<float*>(m->ws + m->o_pairs);
        auto group_args = [&](const SmolLmLayer& M, const RunInfo& Ri, int G) {
            GroupScanArgs A;
            A.H = M.heads; A.G = G; A.d = M.dim; A.dv = M.vdim; A.q_scale = 1.0f;
            A.head = head; A.pairs = pairs;
            A.seq_start = s->seq_start; A.seq_pos0 = s->seq_pos0; A.seq_slot = s->seq_slot;
            A.slot_floats = m->slot_floats; A.state_off = Ri.state_off; A.n_slots = m->n_slots; A.err = err;
            A.unit_out = nullptr; A.unit_off = 0;
            A.conv = ConvIo{};
            return A;
        };
        // Gated delta rule: convolutions, unit vectors, decay and step; the scan over the slot's state; norm per head, silu gate.
        auto gated_delta = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, T* mix_at, int ld) -> int {
            const int hv = M.heads * M.vdim, gd = M.kv_heads * M.dim, ch = 2 * gd + hv;
            GatedDeltaArgs P;
            P.proj = pj; P.n_in = n_in; P.H = M.heads; P.G = M.kv_heads; P.d = M.dim; P.dv = M.vdim;
            P.q_scale = M.score_scale; P.unit_eps = M.unit_eps; P.a_log = M.a_log; P.dt_bias = M.dt_bias;
            P.tok_seq = s->tok_seq; P.err = err;
            P.conv = ConvIo{pj, nullptr, n_in, ch, M.conv_taps, M.conv_w, nullptr, s->seq_start, s->seq_pos0, s->seq_slot, m->slot_floats, Ri.conv_off, m->n_slots};
            const int warps = M.kv_heads + (hv + kGatedDeltaCols - 1) / kGatedDeltaCols;
            if (Tn <= kGraphMaxTokens) pdl_launch(gated_delta_prep_kernel<true>, dim3(Tn, (warps + 3) / 4), 128, 0, ms, P, m->slots, conv, head, pairs);
            else pdl_launch(gated_delta_prep_kernel<false>, dim3(Tn, (warps + 3) / 4), 128, 0, ms, P, m->slots, conv, head, pairs);
            GroupScanArgs S = group_args(M, Ri, M.kv_heads);
            S.q_src = conv; S.k_src = conv + gd; S.v_src = conv + 2 * gd;
            S.q_ld = S.k_ld = S.v_ld = ch;
            S.conv = P.conv;
            CU(launch_group_scan_any<true>(m, S, pairs, s->n_seqs, Tn, max_n, m->slots, oraw, ms));
            GlaArgs A = scan_args(M, Ri, pj);
            A.out_norm = M.out_norm; A.gate_off = ch; A.out_ld = ld; A.out_scale = M.mix_scale;
            launch_gla_out<T>(A, oraw, mix_at, ms);
            m->launches += 2;
            return SMOL_OK;
        };
        // mLSTM: gates and running maximum, the scan with the unit column (the key sum's product with the query), then the
        // denominator, norm per head and sigmoid gate.
        auto mlstm = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, T* mix_at, int ld) -> int {
            const int hd = M.heads * M.dim, hv = M.heads * M.vdim;
            const size_t TH = (size_t)Tn * M.heads;
            float *floor_at = head + 2 * TH, *den = head + 3 * TH;
            MlstmArgs P;
            P.proj = pj; P.n_in = n_in; P.H = M.heads; P.d = M.dim; P.gate_off = (size_t)2 * hd + 2 * hv; P.cap = M.gate_cap;
            P.i_bias = M.rate_bias; P.f_bias = M.decay_bias;
            P.seq_start = s->seq_start; P.seq_pos0 = s->seq_pos0; P.seq_slot = s->seq_slot;
            P.slot_floats = m->slot_floats; P.m_off = Ri.m_off; P.n_slots = m->n_slots; P.err = err;
            pdl_launch(mlstm_gate_kernel, s->n_seqs * M.heads, std::min(kMlstmTile, (max_n + 31) / 32 * 32), 0, ms, P, m->slots, head, floor_at, pairs);
            GroupScanArgs S = group_args(M, Ri, M.heads);
            S.q_src = pj; S.k_src = pj + hd; S.v_src = pj + 2 * hd;
            S.q_ld = S.k_ld = S.v_ld = n_in;
            S.q_scale = M.score_scale;
            S.unit_out = den; S.unit_off = Ri.unit_off;
            CU(launch_group_scan_any<false>(m, S, pairs, s->n_seqs, Tn, max_n, m->slots, oraw, ms, ms != st && Tn > kGraphMaxTokens ? kScanSpread : 0));
            GlaArgs A = scan_args(M, Ri, pj);
            A.den = den; A.den_floor = floor_at; A.den_eps = M.den_eps;
            A.out_norm = M.out_norm; A.norm_own = 1; A.gate_sigmoid = 1; A.out_ld = ld; A.out_scale = M.mix_scale;
            launch_gla_out<T>(A, oraw, mix_at, ms);
            m->launches += 2;
            return SMOL_OK;
        };
        auto run_mixer = [&](const SmolLmLayer& M, const RunInfo& Ri, const float* pj, const float* bias, T* mix_at, int ld) -> int {
            out_ld_now = ld;
            if (M.mixer == SMOL_LM_MIX_SINK_ATTENTION) return attention(M, Ri, pj, bias, mix_at);
            if (M.mixer == SMOL_LM_MIX_STATE_SPACE) return state_space(M, Ri, pj, bias, mix_at);
            if (M.mixer == SMOL_LM_MIX_SIGMOID_ATTENTION) return sigmoid_attention(M, Ri, pj, bias, mix_at, ld);
            if (M.mixer == SMOL_LM_MIX_RETENTION) return retention(M, Ri, pj, mix_at, ld);
            if (M.mixer == SMOL_LM_MIX_GATED_DELTA) return gated_delta(M, Ri, pj, mix_at, ld);
            if (M.mixer == SMOL_LM_MIX_MLSTM) return mlstm(M, Ri, pj, mix_at, ld);
            return lightning(M, Ri, pj, mix_at, ld);
        };
        // the feed-forward reads hn and leaves its output in y, routed experts theirs in `routed` for the kernel that follows
        RoutedSum routed;
        routed.yp = nullptr; routed.slot_of = nullptr; routed.sel_w = nullptr; routed.top = 0;
        const RoutedSum no_sum = routed;
        auto actp_of = [](const SmolLmLayer& M) { return ActParams{M.mlp_act, M.act_limit, M.act_alpha, 0}; };
        // the experts (and a shared expert) of a routed feed-forward may lack gate rows
        auto expert_actp = [](const SmolLmLayer& M) { return ActParams{M.mlp_act, M.act_limit, M.act_alpha, M.ff_plain ? 1 : 0}; };
        auto feed_forward = [&](cudaStream_t st) -> int {
            if (L.mlp == SMOL_LM_MLP_POLYNORM) {
                CU(linear<T>(m, hn, static_cast<const T*>(L.w_up), z, Tn, L.ff, D, st));
                if (kIsF32 || Tn != 1 || !linear_polynorm_row(m, z, L.act, static_cast<const bf16*>(L.w_down), y, D, L.ff, st)) {
                    pdl_launch(polynorm_kernel<T>, Tn, kPolynormThreads, 0, st, z, L.act, c.norm_eps, L.ff, act);
                    CU(linear<T>(m, act, static_cast<const T*>(L.w_down), y, Tn, D, L.ff, st));
                    m->launches += 1;
                }
            } else if (L.mlp == SMOL_LM_MLP_GATED) {
                CU(linear<T>(m, hn, static_cast<const T*>(L.w_up), z, Tn, 2 * L.ff, D, st));
                pdl_launch(gated_act_kernel<T>, cast_grid((size_t)Tn * L.ff / 4), 256, 0, st, z, L.ff, actp_of(L), (size_t)Tn, act);
                CU(linear<T>(m, act, static_cast<const T*>(L.w_down), y, Tn, D, L.ff, st));
                m->launches += 1;
            } else if (L.mlp == SMOL_LM_MLP_EXPERTS) {
                int32_t* sel_id = reinterpret_cast<int32_t*>(m->ws + m->o_sel_id);
                float* sel_w = reinterpret_cast<float*>(m->ws + m->o_sel_w);
                int32_t* perm = reinterpret_cast<int32_t*>(m->ws + m->o_perm);
                int32_t* slot_of = reinterpret_cast<int32_t*>(m->ws + m->o_slot_of);
                int32_t* seg = reinterpret_cast<int32_t*>(m->ws + m->o_seg);
                int32_t* tile_g = reinterpret_cast<int32_t*>(m->ws + m->o_tile_g);
                int32_t* tile_r = reinterpret_cast<int32_t*>(m->ws + m->o_tile_r);
                int32_t* n_tiles = reinterpret_cast<int32_t*>(m->ws + m->o_ntiles);
                float* zp = reinterpret_cast<float*>(m->ws + m->o_zp);
                T* actp = reinterpret_cast<T*>(m->ws + m->o_actp);
                float* yp = reinterpret_cast<float*>(m->ws + m->o_yp);
                RouteArgs Rt;
                Rt.w_router = L.w_router; Rt.bias = L.route_bias; Rt.D = D; Rt.E = L.n_experts + L.n_identity; Rt.E_real = L.n_experts;
                Rt.top = L.top_k; Rt.n_groups = L.n_groups; Rt.keep = L.keep_groups; Rt.scale = L.router_scale; Rt.n_tokens = Tn;
                Rt.score = L.router_score; Rt.plain = L.router_plain; Rt.group_top = L.group_rank_top; Rt.logit_bias = L.router_bias;
                Rt.given = nullptr; Rt.given_ld = n_in; Rt.perm = Rt.slot_of = Rt.n_sorted = nullptr;
                Rt.unit_in = Rt.unit_gate = nullptr; Rt.unit_out = nullptr; Rt.unit_ff = Rt.unit_ld = 0; Rt.unit_act = expert_actp(L);
                const int pairs = Tn * L.top_k;
                const bool few = !kIsF32 && L.n_experts > 0 && pairs <= kMoeGemvPairs && D % 8 == 0 && L.ff % 8 == 0 && L.ff <= 16384;
                const bool direct = few && L.n_identity == 0;      // the pairs stay in their order: nothing to sort
                if (direct) { Rt.perm = perm; Rt.slot_of = slot_of; Rt.n_sorted = seg + L.n_experts; }
                // the router reads the sublayer's input in fp32 where the block keeps it (post-norm), else its T form
                float* r_logits = reinterpret_cast<float*>(m->ws + m->o_rlogits);
                int32_t* r_done = reinterpret_cast<int32_t*>(m->ws + m->o_rdone);
                if (parallel) {
                    // the fused input product has left the shared expert's gate and up, the router's logits and the shared gate
                    // behind the mixer's columns
                    const int SF = (L.ff_plain ? 1 : 2) * L.shared_ff;
                    Rt.given = proj + n_in_main + SF;
                    Rt.unit_in = proj + n_in_main; Rt.unit_gate = L.shared_gate ? Rt.given + Rt.E : nullptr;
                    Rt.unit_out = mix + mix_cols_of(L); Rt.unit_ff = L.shared_ff; Rt.unit_ld = mix_ld;
                }
                const dim3 rgrid(Tn, parallel ? 1 : (Rt.E + 3) / 4);
                if (postnorm) pdl_launch(moe_route_kernel<float>, rgrid, 128, 0, st, Rt, x, r_logits, r_done, sel_id, sel_w);
                else pdl_launch(moe_route_kernel<T>, rgrid, 128, 0, st, Rt, hn, r_logits, r_done, sel_id, sel_w);
                m->launches += 1;
                if (L.n_experts > 0) {
                    // three forms of the two grouped products, by how many rows an expert gets: a warp per output column for
                    // a handful of pairs (decoding), 32-row mma.sync tiles, 128-row tcgen05 tiles over rows copied into sorted order
                    const int NF = L.ff_plain ? L.ff : 2 * L.ff;          // rows of an expert's first matrix
                    const bool big = !kIsF32 && !few && m->tc_ready && pairs / L.n_experts >= 64 && D % 8 == 0 && L.ff % 8 == 0 &&
                                     NF >= kTcMinCols && D >= kTcMinCols && D >= smol::umma::kBK && L.ff >= smol::umma::kBK;
                    const int tile_rows = big ? smol::umma::kM : kGroupTile;
                    if (!direct) {
                        pdl_launch(moe_index_kernel, 1, 256, 0, st, sel_id, pairs, L.n_experts, tile_rows, seg, perm, slot_of, tile_g, tile_r, n_tiles);
                        m->launches++;
                    }
                    const int tiles = pairs / kGroupTile + L.n_experts;
                    GemmIo io = plain_io(D, NF);
                    io.sw = (long long)NF * D;
                    io.tile_group = tile_g; io.tile_row0 = tile_r; io.seg = seg; io.n_tiles = n_tiles;
                    GemmIo io2 = plain_io(L.ff, D);
                    io2.sw = (long long)D * L.ff;
                    io2.tile_group = tile_g; io2.tile_row0 = tile_r; io2.seg = seg; io2.n_tiles = n_tiles;
                    const size_t act_n = (size_t)pairs * L.ff;
                    // a router whose weight multiplies the expert's input: the rows are copied into sorted order, each times
                    // its weight, and the products read that copy
                    T* ap = reinterpret_cast<T*>(m->ws + m->o_ap);
                    if (L.route_input) {
                        pdl_launch(moe_gather_scaled_kernel<T>, pairs, 128, 0, st, hn, perm, L.top_k, sel_w, seg + L.n_experts, D, ap);
                        m->launches++;
                    }
                    if (few) {
                        pdl_launch(moe_gemv_kernel<false>, dim3((NF + 7) / 8, pairs), 256, 0, st, L.route_input ? ap : hn, perm, L.route_input ? 0 : L.top_k, sel_id,
                                                                                         seg + L.n_experts, reinterpret_cast<const bf16*>(L.w_experts_in), io.sw,
                                                                                         zp, NF, D, expert_actp(L));
                        // the second product applies the activation as it reads the first one's result
                        pdl_launch(moe_gemv_kernel<true>, dim3((D + 7) / 8, pairs), 256, L.ff * sizeof(bf16), st, zp, perm, 0, sel_id, seg + L.n_experts,
                                                                                        reinterpret_cast<const bf16*>(L.w_experts_out), io2.sw, yp, D, L.ff, expert_actp(L));
                        m->launches += 1;
                    } else {
                        bool done = false;
                        if (big) {
                            if (!L.route_input) {
                                pdl_launch(moe_gather_kernel, pairs, 128, 0, st, reinterpret_cast<const bf16*>(hn), perm, L.top_k, seg + L.n_experts, D,
                                                                         reinterpret_cast<bf16*>(ap));
                                m->launches++;
                            }
                            done = linear_grouped_tc(m, reinterpret_cast<const bf16*>(ap), reinterpret_cast<const bf16*>(L.w_experts_in), zp, pairs, L.n_experts,
                                                     NF, D, io, st);
                        }
                        if (!done) {
                            if (!L.route_input) { io.gather = perm; io.gather_div = L.top_k; }
                            CU(linear_ex<T>(m, L.route_input ? ap : hn, static_cast<const T*>(L.w_experts_in), zp, pairs, NF, D, io, 1, tiles, st));
                        }
                        pdl_launch(gated_act_kernel<T>, cast_grid(act_n / 4), 256, 0, st, zp, L.ff, expert_actp(L), (size_t)pairs, actp);
                        if (!(big && linear_grouped_tc(m, reinterpret_cast<const bf16*>(actp), reinterpret_cast<const bf16*>(L.w_experts_out), yp, pairs,
                                                       L.n_experts, D, L.ff, io2, st)))
                            CU(linear_ex<T>(m, actp, static_cast<const T*>(L.w_experts_out), yp, pairs, D, L.ff, io2, 1, tiles, st));
                    }
                    m->launches += 1;
                } else {
                    CU(cudaMemsetAsync(slot_of, 0xff, (size_t)pairs * 4, st));
                }
                if (L.shared_ff > 0 && !parallel) {
                    // the expert every token uses: its result lands in y and joins the routed sum in the kernel that follows
                    const int SF = L.ff_plain ? L.shared_ff : 2 * L.shared_ff;
                    CU(linear<T>(m, hn, static_cast<const T*>(L.w_shared_in), z, Tn, SF, D, st));
                    pdl_launch(gated_act_kernel<T>, cast_grid((size_t)Tn * L.shared_ff / 4), 256, 0, st, z, L.shared_ff, expert_actp(L), (size_t)Tn, act);
                    CU(linear<T>(m, act, static_cast<const T*>(L.w_shared_out), y, Tn, D, L.shared_ff, st));
                    m->launches += 1;
                }
                // summed by the norm that follows
                routed.yp = yp; routed.slot_of = slot_of; routed.sel_w = L.route_input ? nullptr : sel_w; routed.top = L.top_k;
            }
            return SMOL_OK;
        };
        // Parallel block: both sublayers read the same projection, so the feed-forward runs on its own stream beside the mixer.
        const bool beside = parallel && L.mlp != SMOL_LM_MLP_NONE;
        if (parallel && L.mlp != SMOL_LM_MLP_NONE) {
            if (beside) {
                CU(cudaEventRecord(m->ff_start, st));
                CU(wait_event(m->ff_stream, m->ff_start));
            }
            const int rc = feed_forward(beside ? m->ff_stream : st);
            if (rc != SMOL_OK) return rc;
            if (beside) CU(cudaEventRecord(m->ff_done, m->ff_stream));
        }
        if (pairable(L)) {
            // The pair of the output-norm block shares no buffer but the result, of which each writes its own columns: the side
            // mixer runs on its own stream beside the layer's.
            const bool fork = outnorm && L.side;
            int rc = SMOL_OK;
            auto run_side = [&]() -> int {
                const SmolLmLayer& S = *L.side;
                const float* sb = L.in_bias ? L.in_bias + n_in_main : nullptr;
                return run_mixer(S, m->side_runs[n], proj + n_in_main, sb, own_proj ? mix2 : mix + mix_cols_of(L), own_proj ? mix_cols_of(S) : mix_ld);
            };
            if (fork) {
                CU(cudaEventRecord(m->ff_start, st));
                CU(wait_event(m->ff_stream, m->ff_start));
                ms = m->ff_stream;
                rc = run_side();
                CU(cudaEventRecord(m->ff_done, m->ff_stream));
                ms = st;
            }
            if (rc == SMOL_OK) rc = run_mixer(L, R, proj, L.in_bias, mix, own_proj ? mix_cols_of(L) : mix_ld);
            if (rc == SMOL_OK && L.side && !fork) rc = run_side();
            if (rc == SMOL_OK && fork) CU(wait_event(st, m->ff_done));
            if (rc != SMOL_OK) return rc;
            mix_cols = own_proj ? mix_cols_of(L) : mix_ld;
        } else if (L.mixer == SMOL_LM_MIX_HGRN2) {
            // q = silu(.), decay = the bounded forget gate, key = 1 - decay; norm per head, no gate
            const int hd = L.heads * L.dim, hv = L.heads * L.vdim;
            LinPrepArgs P{proj, n_in, L.heads, L.dim, L.vdim, Tn, nullptr, L.rate_bias, L.forget_lower};
            pdl_launch(hgrn2_prep_kernel, dim3(Tn, (hd + 1023) / 1024), 256, 0, st, P, uk, auk, dec);
            GlaArgs A = scan_args(L, R, proj);
            A.q_src = uk; A.k_src = auk; A.v_src = proj + 2 * hd;
            A.q_ld = A.k_ld = hd; A.v_ld = n_in;
            CU(launch_gla_scan_any(m, A, s->n_seqs, Tn, max_n, dec, m->slots, oraw, st));
            LinOutArgs O{proj, n_in, hv, L.vdim, L.vdim, 0, hv, 0, c.norm_eps, 1.0f, L.out_norm};
            pdl_launch(lin_attn_out_kernel<T>, dim3(Tn, L.heads), 128, 0, st, O, oraw, mix);
            m->launches += 3;
            mix_cols = hv;
        } else if (L.mixer == SMOL_LM_MIX_LATENT_ATTENTION) {
            AttnArgs A;
            A.proj = proj; A.n_in = n_in; A.bias = nullptr;
            A.tok_seq = s->tok_seq; A.tok_pos = s->tok_pos; A.block_table = s->block_table;
            A.max_pages = s->max_pages; A.page_size = c.page_size; A.n_pages = m->n_pages;
            A.page_elems = m->page_elems; A.k_off = R.k_off; A.v_off = R.v_off;
            A.H = L.heads; A.scale = L.score_scale; A.eps = c.norm_eps;
            A.n_tokens = Tn; A.err = err;
            A.slope = nullptr; A.window = 0; A.softcap = A.two_over_cap = 0.0f; A.has_gate = 1; A.out_scale = 1.0f; A.out_ld = L.heads * L.kv_rank;
            {
                const int dk = L.kv_rank + L.rot_dim, qw = L.dim + L.rot_dim;
                T* cq = reinterpret_cast<T*>(m->ws + m->o_cq);
                float* qf = reinterpret_cast<float*>(m->ws + m->o_qf);
                LatentArgs P;
                P.proj = proj; P.n_in = n_in; P.q_rank = L.q_rank; P.kv_rank = L.kv_rank; P.rot = L.rot_dim; P.rot_pairs = L.rot_dims / 2; P.H = L.heads; P.d = L.dim;
                P.eps = c.norm_eps; P.q_lat_norm = L.q_lat_norm; P.kv_lat_norm = L.kv_lat_norm;
                P.freq = reinterpret_cast<const float*>(m->ws + m->o_freq) + R.freq_off;
                P.tok_seq = s->tok_seq; P.tok_pos = s->tok_pos; P.block_table = s->block_table;
                P.max_pages = s->max_pages; P.page_size = c.page_size; P.n_pages = m->n_pages; P.n_tokens = Tn;
                P.page_elems = m->page_elems; P.k_off = R.k_off; P.err = err;
                pdl_launch(latent_prep_kernel<T>, Tn, 128, 0, st, P, cq, pool);
                CU(linear<T>(m, cq, static_cast<const T*>(L.w_q_up), qf, Tn, L.heads * qw, L.q_rank, st));
                // per head: the unrotated query [Tn, dim] times the transposed key expansion [kv_rank, dim]^T, written where
                // the attention reads its queries (bf16 engine: read from the fp32 q, written in bf16)
                GemmIo io = plain_io(L.dim, L.kv_rank);
                io.lda = L.heads * qw; io.ldy = L.heads * dk;
                io.sa = qw; io.sw = (long long)L.kv_rank * L.dim; io.sy = dk;
                io.a_f32 = io.y_bf16 = kIsF32 ? 0 : 1;
                CU(linear_ex<T>(m, reinterpret_cast<const T*>(qf), static_cast<const T*>(L.w_k_up_t), reinterpret_cast<float*>(qbuf), Tn, L.kv_rank,
                                L.dim, io, L.heads, 0, st));
                pdl_launch(latent_query_kernel<T>, (Tn * L.heads + 3) / 4, 128, 0, st, P, qf, qbuf);
                m->launches += 2;
                A.G = 1; A.d = dk; A.dv = L.kv_rank;
                A.k_ld = dk; A.v_ld = dk; A.v_in_k = 1;
                A.gate_off = (size_t)L.q_rank + dk; A.gate_ld = 1; A.gate_step = 0;
                A.q_norm = A.k_norm = A.r1 = A.r2 = A.sink = nullptr;
                const bool flash = sizeof(T) == 2 && dk <= 192;          // larger latents take the warp-per-row form for prompt portions
                if (L.kv_rank <= 256) launch_attention<T, 8, 1>(m, s, A, flash, qbuf, pool, mix, st);
                else launch_attention<T, 16, 1>(m, s, A, flash, qbuf, pool, mix, st);
                // per head: the attended latent [Tn, kv_rank] times the value expansion [vdim, kv_rank]^T
                GemmIo iv = plain_io(L.kv_rank, L.vdim);
                iv.lda = L.heads * L.kv_rank; iv.ldy = L.heads * L.vdim;
                iv.sa = L.kv_rank; iv.sw = (long long)L.vdim * L.kv_rank; iv.sy = L.vdim;
                iv.y_bf16 = kIsF32 ? 0 : 1;
                T* expanded = reinterpret_cast<T*>(oraw);          // [Tn, heads * vdim] in T
                CU(linear_ex<T>(m, mix, static_cast<const T*>(L.w_v_up), reinterpret_cast<float*>(expanded), Tn, L.vdim, L.kv_rank, iv, L.heads, 0, st));
                mix_cols = L.heads * L.vdim;
                mix_in = expanded;
            }
        } else if (L.mixer == SMOL_LM_MIX_GATED_LINEAR) {
            GlaArgs A;
            A.proj = proj; A.n_in = n_in; A.H = L.heads; A.d = L.dim; A.dv = L.vdim; A.rank = L.rank; A.n_tokens = Tn;
            A.q_scale = L.score_scale; A.tau = L.decay_tau; A.eps = c.norm_eps;
            A.decay_w2 = L.decay_w2; A.decay_bias = L.decay_bias; A.out_norm = L.out_norm;
            A.seq_start = s->seq_start; A.seq_pos0 = s->seq_pos0; A.seq_slot = s->seq_slot;
            A.slot_floats = m->slot_floats; A.state_off = R.state_off; A.n_slots = m->n_slots; A.err = err;
            gla_sources_from_proj(A);
            const int slices = (L.heads * L.dim + 127) / 128;
            if (Tn >= kDecayMinTokens && kDecayTokens * L.rank * sizeof(float) <= 48 * 1024)
                pdl_launch(gla_prep_kernel<kDecayTokens>, dim3((Tn + kDecayTokens - 1) / kDecayTokens, slices), 128, kDecayTokens * L.rank * sizeof(float), st, A, dec);
            else pdl_launch(gla_prep_kernel<1>, dim3(Tn, slices), 128, L.rank * sizeof(float), st, A, dec);
            CU(launch_gla_scan_any(m, A, s->n_seqs, Tn, max_n, dec, m->slots, oraw, st));
            launch_gla_out<T>(A, oraw, mix, st);
            m->launches += 3;
            mix_cols = L.heads * L.vdim;
        } else {
            DeltaArgs A;
            A.proj = proj; A.n_in = n_in; A.H = L.heads; A.d = L.dim; A.rank = L.rank; A.n_tokens = Tn;
            A.decay_coef = L.decay_coef; A.unit_eps = L.unit_eps; A.eps = c.norm_eps;
            A.rate_bias = L.rate_bias; A.decay_w2 = L.decay_w2; A.decay_bias = L.decay_bias; A.out_norm = L.out_norm;
            A.seq_start = s->seq_start; A.seq_pos0 = s->seq_pos0; A.seq_slot = s->seq_slot;
            A.slot_floats = m->slot_floats; A.state_off = R.state_off; A.n_slots = m->n_slots; A.err = err;
            const bool chunks = chunks_pay(kScanGeneralDelta, false, s->n_seqs, L.heads, Tn, max_n, L.dim, L.dim, m->n_sms), quad = !chunks && quad_pays(s->n_seqs, Tn, max_n);
            float *u_to = chunks || quad ? nullptr : uk, *au_to = chunks || quad ? nullptr : auk;
            const size_t prep_smem = (size_t)(L.rank + L.heads) * sizeof(float);
            const int slices = (L.heads * L.dim + 127) / 128;
            if (Tn >= kDecayMinTokens && kDecayTokens * prep_smem <= 48 * 1024)
                pdl_launch(delta_prep_kernel<kDecayTokens>, dim3((Tn + kDecayTokens - 1) / kDecayTokens, slices), 128, kDecayTokens * prep_smem, st, A, dec, u_to, au_to);
            else pdl_launch(delta_prep_kernel<1>, dim3(Tn, slices), 128, prep_smem, st, A, dec, u_to, au_to);
            cudaError_t e;
            if (chunks) {
                const int HD = L.heads * L.dim;
                const ChunkSource Q{L.heads, 1, L.dim, L.dim, L.dim, proj, proj + HD, n_in, n_in, proj + 2 * HD, n_in, dec, nullptr, nullptr, 0, 0,
                                    proj + 4 * HD, L.rate_bias, L.unit_eps, s->seq_start, 0};
                const ChunkArgs S{L.heads, L.dim, L.dim, nullptr, 0, 1.0f, s->seq_start, s->seq_pos0, s->seq_slot, m->slot_floats, R.state_off, m->n_slots, err, nullptr, 0, ConvIo{}};
                e = launch_chunks<kScanGeneralDelta>(m, Q, S, s->n_seqs, max_n, oraw, st);
            } else if (quad) {
                const int HD = L.heads * L.dim;
                QuadSource Q{L.heads, 1, L.dim, proj, proj + HD, n_in, n_in, dec, nullptr, nullptr, 0, 0, proj + 4 * HD, L.rate_bias, L.unit_eps, s->seq_start, 0};
                QuadArgs S{L.heads, L.dim, L.dim, nullptr, 0, proj + 2 * HD, n_in, 1.0f, s->seq_start, s->seq_pos0, s->seq_slot, m->slot_floats, R.state_off, m->n_slots, err};
                e = launch_quad<kQuadGeneralDelta>(m, Q, S, s->n_seqs, max_n, oraw, st);
            } else if (L.dim <= 16) e = launch_scan<16>(A, s->n_seqs, dec, uk, auk, m->slots, oraw, st);
            else if (L.dim <= 32) e = launch_scan<32>(A, s->n_seqs, dec, uk, auk, m->slots, oraw, st);
            else if (L.dim <= 64) e = launch_scan<64>(A, s->n_seqs, dec, uk, auk, m->slots, oraw, st);
            else if (L.dim <= 128) e = launch_scan<128>(A, s->n_seqs, dec, uk, auk, m->slots, oraw, st);
            else e = launch_scan<256>(A, s->n_seqs, dec, uk, auk, m->slots, oraw, st);
            CU(e);
            GlaArgs O = scan_args(L, R, proj);
            O.dv = L.dim; O.out_norm = L.out_norm; O.norm_own = 1; O.gate_off = 3LL * L.heads * L.dim; O.gate_sigmoid = 1; O.out_ld = L.heads * L.dim;
            launch_gla_out<T>(O, oraw, mix, st);
            m->launches += 3;
            mix_cols = L.heads * L.dim;
        }
        if (beside) CU(wait_event(st, m->ff_done));      // also: w_out covers the shared expert's unit
        CU(linear<T>(m, mix_in, static_cast<const T*>(L.w_out), y, Tn, D, mix_cols, st));
        if (own_proj) CU(linear<T>(m, mix2, static_cast<const T*>(L.side->w_out), y2, Tn, D, mix_cols_of(*L.side), st));
        const bool last = n + 1 == m->runs.size();
        const float* next_norm1 = last ? nullptr : m->layers[m->runs[n + 1].layer].norm1;
        if (parallel) {
            // x += m * (mixer and shared expert, one output product; routed experts' sum); the traced row, then either the next
            // run's norm or the row of a merging run
            const SmolLmLayer* Ln = last ? nullptr : &m->layers[m->runs[n + 1].layer];
            const bool merge = !last && (m->runs[n + 1].flags & SMOL_LM_RUN_MERGE_EMBED);
            ResidualArgs Ra;
            Ra.x = x; Ra.D = D; Ra.eps = c.norm_eps;
            Ra.y = y; Ra.y_w = Ra.y2 = Ra.y2_w = nullptr; Ra.sy = c.residual_mult; Ra.sy2 = 0.0f;
            Ra.rs = routed; Ra.s_routed = c.residual_mult;
            Ra.trace = s->trace ? s->trace + n * (size_t)Tn * D : nullptr; Ra.x0 = nullptr; Ra.cat = merge ? cat : nullptr;
            Ra.next = (Ln && !merge) ? norm_of(Ln->norm1, Ln->norm1_shift, Ln->norm1_alpha) : no_norm;
            launch_residual_norm<T>(Ra, Tn, nthr, hn, st);
            m->launches += 1;
        } else if (outnorm) {
            // x += r(mixer + bias) * norm1, x += r(feed-forward) * norm2; each kernel leaves the new stream in T for the next sublayer
            const bool has_ff = L.mlp != SMOL_LM_MLP_NONE;
            float* tr_row = s->trace ? s->trace + n * (size_t)Tn * D : nullptr;
            ResidualArgs Ra;
            Ra.x = x; Ra.D = D; Ra.eps = c.norm_eps;
            Ra.y = y; Ra.y_w = L.norm1; Ra.y_b = L.out_bias; Ra.sy = 1.0f;
            Ra.y2 = Ra.y2_w = nullptr; Ra.sy2 = 0.0f;
            Ra.rs = no_sum; Ra.s_routed = 1.0f; Ra.x0 = nullptr; Ra.cat = nullptr;
            Ra.trace = has_ff ? nullptr : tr_row;
            Ra.next = has_ff || !last ? copy_row : no_norm;
            launch_residual_norm<T>(Ra, Tn, nthr, hn, st);
            m->launches += 1;
            if (has_ff) {
                const int rc = feed_forward(st);
                if (rc != SMOL_OK) return rc;
                Ra.y_w = L.norm2; Ra.y_b = nullptr; Ra.trace = tr_row;
                Ra.next = last ? no_norm : copy_row;
                launch_residual_norm<T>(Ra, Tn, nthr, hn, st);
                m->launches += 1;
            }
        } else if (prenorm) {
            // x += mixer (mixers with their own projections: each normed over the width first); x += feed-forward.  The kernel
            // that ends the layer also leaves the traced row, restarts the stream where the next run asks for it and applies
            // the next layer's first norm.
            const bool has_ff = L.mlp != SMOL_LM_MLP_NONE;
            const SmolLmLayer* Ln = last ? nullptr : &m->layers[m->runs[n + 1].layer];
            const NormSpec after = Ln ? norm_of(Ln->norm1, Ln->norm1_shift, Ln->norm1_alpha) : no_norm;
            const float* restart = (!last && (m->runs[n + 1].flags & SMOL_LM_RUN_ADD_EMBED)) ? x0 : nullptr;
            float* tr_row = s->trace ? s->trace + n * (size_t)Tn * D : nullptr;
            ResidualArgs Ra;
            Ra.x = x; Ra.D = D; Ra.eps = c.norm_eps;
            Ra.y = y; Ra.y_w = own_proj ? L.proj_norm : nullptr; Ra.sy = own_proj ? L.mix_scale : 1.0f;
            Ra.y2 = own_proj ? y2 : nullptr; Ra.y2_w = own_proj ? L.side->proj_norm : nullptr; Ra.sy2 = own_proj ? L.side->mix_scale : 0.0f;
            Ra.rs = no_sum; Ra.s_routed = 1.0f; Ra.cat = nullptr;
            Ra.trace = has_ff ? nullptr : tr_row; Ra.x0 = has_ff ? nullptr : restart;
            Ra.next = has_ff ? norm_of(L.norm2, L.norm2_shift, L.norm2_alpha) : after;
            launch_residual_norm<T>(Ra, Tn, nthr, hn, st);
            m->launches += 1;
            if (has_ff) {
                const int rc = feed_forward(st);
                if (rc != SMOL_OK) return rc;
                const bool summed = routed.yp != nullptr;
                Ra.y = (!summed || L.shared_ff > 0) ? y : nullptr; Ra.y_w = nullptr; Ra.sy = 1.0f;
                Ra.y2 = nullptr; Ra.y2_w = nullptr; Ra.sy2 = 0.0f;
                Ra.rs = routed;
                Ra.trace = tr_row; Ra.x0 = restart; Ra.next = after;
                launch_residual_norm<T>(Ra, Tn, nthr, hn, st);
                m->launches += 1;
            }
        } else if (postnorm) {
            // x <- g1 * rms_divide(alpha x + mixer); x <- g2 * rms_divide(alpha x + ff); the layer's result joins the history
            // and the stream becomes the weighted sum of the history
            const bool has_ff = L.mlp != SMOL_LM_MLP_NONE;
            pdl_launch(post_norm_kernel<T>, Tn, nthr, 2 * D * sizeof(float), st, x, y, c.residual_alpha, L.norm1, c.norm_eps, D, has_ff ? nullptr : hist,
                                                                      hist_stride, (int)n + 2, L.depth_mix, nullptr, hn, no_sum);
            m->launches += 1;
            if (has_ff) {
                const int rc = feed_forward(st);
                if (rc != SMOL_OK) return rc;
                pdl_launch(post_norm_kernel<T>, Tn, nthr, 2 * D * sizeof(float), st, x, y, c.residual_alpha, L.norm2, c.norm_eps, D, hist, hist_stride,
                                                                          (int)n + 2, L.depth_mix, nullptr, hn, routed);
                m->launches += 1;
            }
        } else if (L.mlp != SMOL_LM_MLP_NONE) {
            add_norm(L.norm1b, L.ls1, L.norm2, L.out_bias, no_sum);
            const int rc = feed_forward(st);
            if (rc != SMOL_OK) return rc;
            add_norm(L.norm2b, L.ls2, next_norm1, nullptr, routed);
            m->launches += 2;
        } else {
            add_norm(L.norm1b, L.ls1, next_norm1, L.out_bias, no_sum);
            m->launches += 1;
        }
        if (s->trace && !prenorm && !parallel && !outnorm) CU(cudaMemcpyAsync(s->trace + n * (size_t)Tn * D, x, (size_t)Tn * D * 4, cudaMemcpyDeviceToDevice, st));
    }
    if (s->n_want > 0) {
        if (postnorm) pdl_launch(post_norm_kernel<T>, s->n_want, nthr, 2 * D * sizeof(float), st, x, nullptr, c.logit_scale, m->g.final_norm, c.norm_eps, D, nullptr, 0, 0,
                                                                                      nullptr, s->want_rows, hw, RoutedSum{nullptr, nullptr, nullptr, 0});
        else if (prenorm || parallel || outnorm) pdl_launch(prenorm_rows_kernel<T>, s->n_want, nthr, 0, st, x, s->want_rows, norm_of(m->g.final_norm, m->g.final_norm_shift, m->g.final_norm_alpha), D, hw);
        else if (!row_pieces(s->n_want, D, addresses_of(x, m->g.final_norm, hw), [&](auto v, auto lone, int blocks, int threads) {
                     pdl_launch(norm_rows_vec_kernel<T, decltype(v)::value, decltype(lone)::value>, blocks, threads, 0, st, x, s->want_rows, m->g.final_norm, c.norm_eps, D, hw, woff, s->n_want);
                 }))
            pdl_launch(norm_rows_kernel<T>, s->n_want, nthr, 0, st, x, s->want_rows, m->g.final_norm, c.norm_eps, D, hw, woff);
        m->launches++;
        CU(linear<T>(m, hw, static_cast<const T*>(m->g.head), s->logits, s->n_want, c.vocab, D, st));
        const float lscale = postnorm ? 1.0f : c.logit_scale;      // the post-norm block scales inside the final norm
        if (lscale != 1.0f || c.logit_softcap > 0.0f) {
            pdl_launch(logit_finish_kernel, cast_grid((size_t)s->n_want * c.vocab), 256, 0, st, s->logits, lscale, c.logit_softcap, (size_t)s->n_want * c.vocab);
            m->launches++;
        }
    }
    CU(cudaGetLastError());
    return SMOL_OK;
}

extern "C" int smol_lm_step(SmolLm* m, const SmolLmStep* s, void* stream) {
    if (!m || !s) return fail(SMOL_ERR_INVALID, "smol_lm_step: null argument");
    if (!m->bound) return fail(SMOL_ERR_UNBOUND, "smol_lm_step: bind weights and pools first");
    if (s->n_tokens < 1 || s->n_seqs < 1 || s->n_want < 0 || s->max_pages < 1) return fail(SMOL_ERR_INVALID, "smol_lm_step: empty step");
    if (s->n_tokens > m->cfg.max_step_tokens || s->n_seqs > m->cfg.max_step_seqs || s->n_want > m->cfg.max_want)
        return fail(SMOL_ERR_CAPACITY, "smol_lm_step: step larger than the workspace was made for");
    if (!s->tokens || !s->tok_seq || !s->tok_pos || !s->seq_start || !s->seq_pos0 || !s->seq_slot || !s->block_table ||
        (s->n_want > 0 && (!s->want_rows || !s->logits)))
        return fail(SMOL_ERR_INVALID, "smol_lm_step: null array");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!m->cfg.use_graph || s->trace || s->n_tokens > kGraphMaxTokens)
        return m->cfg.dtype == SMOL_LM_F32 ? step_impl<float>(m, s, st) : step_impl<bf16>(m, s, st);
    // The launches of a step depend on the struct's scalars and pointers only (the arrays' contents are read on the device),
    // except that max_pos matters through the number of key ranges alone.
    SmolLmStep key = *s;
    const int max_pos = s->max_pos > 0 ? std::min(s->max_pos, m->cfg.max_context - 1) : m->cfg.max_context - 1;
    key.max_pos = std::min(m->cfg.max_context - 1, (max_pos / m->split_len + 4) / 4 * 4 * m->split_len - 1);
    for (auto& g : m->graphs)
        if (memcmp(&g.key, &key, sizeof(key)) == 0) {
            CU(cudaGraphLaunch(g.exec, st));
            m->launches += g.launches;
            return SMOL_OK;
        }
    if (!m->cap_stream) CU(cudaStreamCreateWithFlags(&m->cap_stream, cudaStreamNonBlocking));
    const int64_t before = m->launches;
    CU(cudaStreamBeginCapture(m->cap_stream, cudaStreamCaptureModeThreadLocal));
    const int rc = m->cfg.dtype == SMOL_LM_F32 ? step_impl<float>(m, &key, m->cap_stream) : step_impl<bf16>(m, &key, m->cap_stream);
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(m->cap_stream, &graph);
    if (rc != SMOL_OK) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    if (ce != cudaSuccess) return fail(SMOL_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(ce));
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return fail(SMOL_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ie));
    if (m->graphs.size() >= 64) {
        cudaGraphExecDestroy(m->graphs.front().exec);
        m->graphs.erase(m->graphs.begin());
    }
    m->graphs.push_back({key, exec, m->launches - before});
    CU(cudaGraphLaunch(exec, st));
    return SMOL_OK;
}

extern "C" int smol_lm_linear(SmolLm* m, const void* d_a, const void* d_w, float* d_y, int32_t M, int32_t N, int32_t K, void* stream) {
    if (!m || !d_a || !d_w || !d_y || M < 1 || N < 1 || K < 1) return fail(SMOL_ERR_INVALID, "smol_lm_linear: bad argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // w is the caller's: the kernel in front may have made it, and the products read w before they wait for that kernel
    t_plain_next = true;
    if (m->cfg.dtype == SMOL_LM_F32) CU(linear<float>(m, static_cast<const float*>(d_a), static_cast<const float*>(d_w), d_y, M, N, K, st));
    else CU(linear<bf16>(m, static_cast<const bf16*>(d_a), static_cast<const bf16*>(d_w), d_y, M, N, K, st));
    return SMOL_OK;
}

extern "C" int smol_lm_sample(SmolLm* m, const float* d_logits, int32_t rows, int32_t n, float temp, int32_t top_k, float top_p,
                              float min_p, uint64_t seed, const int32_t* d_seq_id, const int32_t* d_step, int32_t* d_out, void* stream) {
    if (!m || !d_logits || !d_out || rows < 1) return fail(SMOL_ERR_INVALID, "smol_lm_sample: bad argument");
    if (n < 1 || n > smol::kThreads * 64) return fail(SMOL_ERR_UNSUPPORTED, "smol_lm_sample: n outside [1, 32768]");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = (size_t)n * sizeof(float);
    const int grid = rows < 1024 ? rows : 1024;
    if (n <= smol::kThreads * 8) {
        CU(cudaFuncSetAttribute(lm_sample_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
        pdl_launch(lm_sample_kernel<8>, grid, smol::kThreads, smem, st, d_logits, n, rows, temp, top_k, top_p, min_p, seed, d_seq_id, d_step, d_out);
    } else {
        CU(cudaFuncSetAttribute(lm_sample_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
        pdl_launch(lm_sample_kernel<64>, grid, smol::kThreads, smem, st, d_logits, n, rows, temp, top_k, top_p, min_p, seed, d_seq_id, d_step, d_out);
    }
    CU(cudaGetLastError());
    m->launches++;
    return SMOL_OK;
}
