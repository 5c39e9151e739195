// fp32 matrix-product tile on packed FMAs (sm_100a), shared by the codec and the language-model engine.
//
// out[BM rows][BN columns] = A . W^T over a range of k, both operands k-contiguous.  cp.async brings BK = 16 k at a time into a ring
// of row-major stages (rows of 20 floats: eight neighbouring rows start in eight different 16-byte bank groups), a thread owns
// TM x TN outputs and multiplies k-pairs with fma.rn.f32x2: each accumulator is a pair (sum over even k, sum over odd k), so the
// pairs come straight from 16-byte shared-memory loads, with nothing to duplicate or transpose, and one instruction does two
// multiply-adds: (TM + TN) loads feed 2 TM TN of them.  Plain FMAs at 4 x 4 outputs, the form before, were bound by instruction issue.
//
// A cluster of S CTAs along grid.x shares one output tile, each taking a contiguous range of k; the partial tiles meet through
// distributed shared memory and are added in rank order.  The arithmetic of an output -- which k a rank takes, the two chains, the
// order of ranks -- follows from K and S alone, never from the tile's shape or from what else is in the launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace smol {
namespace f32t {

constexpr int kBK = 16, kLD = kBK + 4, kStages = 3;

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float pair_sum(unsigned long long v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
// 16 bytes, or zeros without touching memory (`src` is any valid address then)
__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(in ? 16 : 0));
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::); }
template <int N> __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ float ld_rank(const float* p, uint32_t rank) {
    float v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
                 : "=f"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return v;
}

// Threads are laid out as THM x THN (a warp is 4 x 8 of them, or 2 x 16 where THN is 16 times more than needed); a thread's rows are
// ty + i * THM and its columns tx + j * THN.
template <int BM, int BN, int TM, int TN>
struct Tile {
    static constexpr int THM = BM / TM, THN = BN / TN, NT = THM * THN;
    static_assert(THM % 4 == 0 && THN % 8 == 0, "warps of 4 x 8 threads");
    static constexpr int PA = (BM * 4 + NT - 1) / NT, PW = (BN * 4 + NT - 1) / NT;      // 16-byte pieces of a stage a thread copies
    static constexpr int kStageFloats = (BM + BN) * kLD;
    static constexpr int kSmemFloats = kStages * kStageFloats > BM * (BN + 1) ? kStages * kStageFloats : BM * (BN + 1);
    static constexpr size_t kSmemBytes = (size_t)kSmemFloats * 4;

    __device__ static __forceinline__ int ty() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w / (THN / 8)) * 4 + (l >> 3); }
    __device__ static __forceinline__ int tx() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w % (THN / 8)) * 8 + (l & 7); }

    // k in [k_lo, k_hi) (multiples of 4).  a_src(row, k) / w_src(row, k): address of 4 floats, nullptr for zeros; shape(v, row, k): what
    // becomes of 4 floats of A before they are multiplied (called once per piece by the thread that copied it).  before(): called
    // after the first copies of W are on their way and before anything of A is read.
    template <bool SHAPE, class ASrc, class WSrc, class Shape, class Before>
    __device__ static __forceinline__ void product(float* sm, int k_lo, int k_hi, ASrc a_src, WSrc w_src, Shape shape, Before before, float (&out)[TM][TN]) {
        const int tid = threadIdx.x, row_y = ty(), row_x = tx();
        unsigned long long acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
        const int steps = (k_hi - k_lo + kBK - 1) / kBK;
        auto copy_w = [&](int s) {
            float* Ws = sm + (s % kStages) * kStageFloats + BM * kLD;
            const int k0 = k_lo + s * kBK;
#pragma unroll
            for (int x = 0; x < PW; ++x) {
                const int id = tid + x * NT, r = id >> 2, k = k0 + (id & 3) * 4;
                if (BN * 4 % NT != 0 && r >= BN) break;
                const float* p = k < k_hi ? w_src(r, k) : nullptr;
                copy16(Ws + r * kLD + (id & 3) * 4, p ? p : w_src(0, k_lo), p != nullptr);
            }
        };
        auto copy_a = [&](int s) {
            float* As = sm + (s % kStages) * kStageFloats;
            const int k0 = k_lo + s * kBK;
#pragma unroll
            for (int x = 0; x < PA; ++x) {
                const int id = tid + x * NT, r = id >> 2, k = k0 + (id & 3) * 4;
                if (BM * 4 % NT != 0 && r >= BM) break;
                const float* p = k < k_hi ? a_src(r, k) : nullptr;
                copy16(As + r * kLD + (id & 3) * 4, p ? p : w_src(0, k_lo), p != nullptr);
            }
        };
        // group s of the copies: stage s (W of the first stages goes out ahead of `before`, in the first groups all the same)
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s)
            if (s < steps) copy_w(s);
        before();
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s) {
            if (s < steps) copy_a(s);
            commit();
        }
        for (int s = 0; s < steps; ++s) {
            float* As = sm + (s % kStages) * kStageFloats;
            const float* Ws = As + BM * kLD;
            wait<kStages - 2>();
            if (SHAPE) {
#pragma unroll
                for (int x = 0; x < PA; ++x) {
                    const int id = tid + x * NT, r = id >> 2, k = k_lo + s * kBK + (id & 3) * 4;
                    if (BM * 4 % NT != 0 && r >= BM) break;
                    float4* p = reinterpret_cast<float4*>(As + r * kLD + (id & 3) * 4);
                    if (k < k_hi) *p = shape(*p, r, k);
                }
            }
            __syncthreads();
            if (s + kStages - 1 < steps) { copy_w(s + kStages - 1); copy_a(s + kStages - 1); }
            commit();
#pragma unroll
            for (int q = 0; q < kBK; q += 4) {
                ulonglong2 a[TM], w[TN];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(As + (row_y + i * THM) * kLD + q);
#pragma unroll
                for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(Ws + (row_x + j * THN) * kLD + q);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a[i].y, w[j].y, acc[i][j]);
            }
        }
        wait<0>();
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) out[i][j] = pair_sum(acc[i][j]);
    }

    // Hands every output of the tile to done(row, column, value): straight from the registers, or -- a cluster -- each rank its share of
    // the rows after the partial tiles are added in rank order.  Every thread of every rank calls it.
    template <class Done>
    __device__ static __forceinline__ void finish(float* sm, const float (&out)[TM][TN], Done done) {
        const uint32_t S = cluster_size();
        if (S == 1) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) done(ty() + i * THM, tx() + j * THN, out[i][j]);
            return;
        }
        __syncthreads();                     // the stages are read by now
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) sm[(ty() + i * THM) * (BN + 1) + tx() + j * THN] = out[i][j];
        cluster_sync();
        const int per = (BM + (int)S - 1) / (int)S, lo = (int)cluster_rank() * per, hi = min(BM, lo + per);
        for (int o = lo * BN + threadIdx.x; o < hi * BN; o += NT) {
            const int r = o / BN, c = o - r * BN;
            float v = ld_rank(sm + r * (BN + 1) + c, 0);
            for (uint32_t x = 1; x < S; ++x) v += ld_rank(sm + r * (BN + 1) + c, x);
            done(r, c, v);
        }
        cluster_sync();                      // nobody leaves while its tile is being read
    }
    // this rank's range of k: whole steps, contiguous
    __device__ static __forceinline__ void range(int K, int& lo, int& hi) {
        const int S = (int)cluster_size(), per = ((K + kBK - 1) / kBK + S - 1) / S * kBK;
        lo = min(K, (int)cluster_rank() * per);
        hi = min(K, lo + per);
    }
};

}  // namespace f32t
}  // namespace smol
