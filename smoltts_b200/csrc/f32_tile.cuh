// fp32 matrix-product tile on packed FMAs (sm_100a), shared by the codec and the language-model engine.
//
// out[BM rows][BN columns] = A . W^T over a range of k, both operands k-contiguous.  cp.async brings BK = 16 k at a time into a ring
// of row-major stages (rows of 20 floats: eight neighbouring rows start in eight different 16-byte bank groups), a thread owns
// TM x TN outputs and multiplies k-pairs with fma.rn.f32x2: each accumulator is a pair (sum over even k, sum over odd k), so the
// pairs come straight from 16-byte shared-memory loads, with nothing to duplicate or transpose, and one instruction does two
// multiply-adds (at the rate of two: measured 72 TFLOP/s either way, but half the issue slots).  What bounds it is shared memory: a
// warp's 16-byte load takes four clocks of the SM, however many lanes share an address, so 8 x 8 outputs per thread just balance the FMAs
// (64 per 16 floats loaded); 8 x 4 are at two thirds.  Small tiles therefore have few threads, not small thread tiles.
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
__device__ __forceinline__ float4 ld_rank(const float* p, uint32_t rank) {
    float4 v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return v;
}

// Threads are laid out as THM x THN, a warp 4 x 8 of them.  A thread's rows are ty + i * THM.  Its columns come in runs of four
// (column(tx, j)), so that results move as 16-byte pieces; the columns of W lie in shared memory in the order j * THN + tx, so that
// neighbouring threads read neighbouring rows all the same.
template <int BM, int BN, int TM, int TN>
struct Tile {
    static constexpr int THM = BM / TM, THN = BN / TN, NT = THM * THN;
    static_assert(THM % 4 == 0 && THN % 8 == 0, "warps of 4 x 8 threads");
    static_assert(TN % 4 == 0, "runs of four columns");
    static_assert(NT % 4 == 0, "a thread's pieces have one place in a step");
    static constexpr int PA = (BM * 4 + NT - 1) / NT, PW = (BN * 4 + NT - 1) / NT;      // 16-byte pieces of a stage a thread copies
    static constexpr int kStageFloats = (BM + BN) * kLD;
    static constexpr int kOutLd = BN + 4;          // floats between the rows of a partial tile
    static constexpr int kSmemFloats = kStages * kStageFloats > BM * kOutLd ? kStages * kStageFloats : BM * kOutLd;
    static constexpr size_t kSmemBytes = (size_t)kSmemFloats * 4;

    __device__ static __forceinline__ int ty() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w / (THN / 8)) * 4 + (l >> 3); }
    __device__ static __forceinline__ int tx() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w % (THN / 8)) * 8 + (l & 7); }

    // column of a thread's j-th output, and the other way round: the column that lies at place p of W's stage
    __device__ static __forceinline__ int column(int x, int j) { return (j / 4) * (4 * THN) + x * 4 + j % 4; }
    __device__ static __forceinline__ int column_at(int p) { return column(p % THN, p / THN); }

    // k in [k_lo, k_hi) (multiples of 4).  a_row(r) / w_row(r): a row's address, nullptr for zeros; a_at(k): where in its row k lies.
    // before(): called after the first copies of W are on their way and before anything of A is read.
    // RUN > 0: the two chains of an output are added up and begin anew every RUN steps.
    template <int RUN, class ARow, class AAt, class WRow, class Before>
    __device__ static __forceinline__ void product(float* sm, int k_lo, int k_hi, ARow a_row, AAt a_at, WRow w_row, Before before, float (&out)[TM][TN]) {
        const int tid = threadIdx.x, row_y = ty(), row_x = tx(), kp = (tid & 3) * 4;      // kp: this thread's place in a step
        unsigned long long acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) { acc[i][j] = 0ull; out[i][j] = 0.0f; }
        const int steps = (k_hi - k_lo + kBK - 1) / kBK;
        const float *ap[PA], *wp[PW], *any = w_row(0);      // (column 0 is always there)
#pragma unroll
        for (int x = 0; x < PA; ++x) ap[x] = (tid + x * NT) >> 2 < BM ? a_row((tid + x * NT) >> 2) : nullptr;
#pragma unroll
        for (int x = 0; x < PW; ++x) wp[x] = (tid + x * NT) >> 2 < BN ? w_row(column_at((tid + x * NT) >> 2)) : nullptr;
        auto copy_w = [&](int s) {
            float* Ws = sm + (s % kStages) * kStageFloats + BM * kLD + kp;
            const int k = k_lo + s * kBK + kp;
#pragma unroll
            for (int x = 0; x < PW; ++x) {
                const int r = (tid + x * NT) >> 2;
                if (BN * 4 % NT != 0 && r >= BN) break;
                const bool in = k < k_hi && wp[x];
                copy16(Ws + r * kLD, in ? wp[x] + k : any, in);
            }
        };
        auto copy_a = [&](int s) {
            float* As = sm + (s % kStages) * kStageFloats + kp;
            const int k = k_lo + s * kBK + kp;
            const long long at = a_at(k);
#pragma unroll
            for (int x = 0; x < PA; ++x) {
                const int r = (tid + x * NT) >> 2;
                if (BM * 4 % NT != 0 && r >= BM) break;
                const bool in = k < k_hi && ap[x];
                copy16(As + r * kLD, in ? ap[x] + at : any, in);
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
            const float *As = sm + (s % kStages) * kStageFloats, *Ws = As + BM * kLD;
            wait<kStages - 2>();
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
            if (RUN > 0 && s % RUN == RUN - 1) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) { out[i][j] += pair_sum(acc[i][j]); acc[i][j] = 0ull; }
            }
        }
        wait<0>();
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) out[i][j] += pair_sum(acc[i][j]);
    }

    // Hands the outputs of the tile to done(row, column, four values) -- four columns from a multiple of 4 on: straight from the
    // registers, or -- a cluster -- each rank its share of the rows after the partial tiles are added in rank order.  Every thread of
    // every rank calls it.
    template <class Done>
    __device__ static __forceinline__ void finish(float* sm, const float (&out)[TM][TN], Done done) {
        const uint32_t S = cluster_size();
        if (S == 1) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; j += 4) done(ty() + i * THM, column(tx(), j), make_float4(out[i][j], out[i][j + 1], out[i][j + 2], out[i][j + 3]));
            return;
        }
        __syncthreads();                     // the stages are read by now
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<float4*>(sm + (ty() + i * THM) * kOutLd + column(tx(), j)) = make_float4(out[i][j], out[i][j + 1], out[i][j + 2], out[i][j + 3]);
        cluster_sync();
        const int per = (BM + (int)S - 1) / (int)S, lo = (int)cluster_rank() * per, hi = min(BM, lo + per);
        for (int o = lo * (BN / 4) + threadIdx.x; o < hi * (BN / 4); o += NT) {
            const int r = o / (BN / 4), c = (o - r * (BN / 4)) * 4;
            float4 v = ld_rank(sm + r * kOutLd + c, 0);
            for (uint32_t x = 1; x < S; ++x) {
                const float4 u = ld_rank(sm + r * kOutLd + c, x);
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
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
