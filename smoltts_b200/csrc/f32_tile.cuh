// fp32 matrix-product tiles (sm_100a), shared by the codec and the language-model engine: MmaTile on the tensor cores, Tile on packed FMAs.
//
// out[BM rows][BN columns] = A . W^T over a range of k, both operands k-contiguous.  cp.async brings BK = 16 k at a time into a ring
// of row-major stages (rows of 20 floats: eight neighbouring rows start in eight different 16-byte bank groups).
//
// MmaTile (the language models' float32 engine, sums of 72 k and more): a warp takes WM x WN outputs and multiplies with mma.sync m16n8k8 on tf32 parts: every fp32 operand is hi + lo,
// 11 bits each and the sign of lo, made from the fragments that ldmatrix brings, and a product is lo hi + hi lo + hi hi.  (Left out: lo lo, at most 2^-22 of the product,
// and the last bit, 2^-23, of an operand whose lo needs twelve; the errors below have both in them.)  The
// tensor core drops what its sum has below the last place, so a sum runs over 8 k, smallest parts first, and is added in fp32.
// Parts cannot hold everything that fp32 holds: the lo of an infinity is no number, an operand in the last half step of tf32 below the largest float has an infinite
// hi, and operands below 2^-115 have a denormal lo.  So an output that comes out not finite, or below 2^-80 and not zero, is made once more from the operands
// themselves, on FMAs: whatever is wrong with the parts of a finite product's operands shows in one of the two, except where an operand below 2^-115 meets one
// above 2^35, or its product vanishes beside larger ones.
// What bounds it is the MMAs, 170 multiply-adds per clock and SM after the three parts, and the instructions that split operands and add sums beside them:
// 300 x 4608 x 768 56 us (38 TFLOP/s), 1024 x 4608 x 768 137 (53); Tile, which reads 16 bytes of shared memory (four clocks of the SM) for every 16 multiply-adds, 77
// and 201.  Without splitting and adding 3072 x 1536 x 1024 takes 142 us instead of 181.  Warps of 64 x 32 in tiles of 64 x 64 or 128 x 64: 174 there, but 20 to 40 %
// slower on a few hundred rows; sums over 16 k 174 as well, but further from 64 bits where all products have one sign (8.0e-8 against 6.7e-8).
// Errors against 64 bits (rows x columns x K, MmaTile | Tile; shorter sums than 72 k go to Tile, see lm_kernels.cu): 300 x 4608 x 768 1.37e-7 | 1.83e-7, 300 x 768 x 4608 1.89e-7 | 3.10e-7, 64 x 64 x 8192 2.4e-7 | 4.2e-7;
// values in [0, 1): 6.7e-8 | 6.7e-8, 7.7e-8 | 8.1e-8, 8.0e-8 | 9.1e-8.
//
// Tile (the codec, and the engine's shorter sums): a thread owns TM x TN outputs and multiplies k-pairs with fma.rn.f32x2: each accumulator is a pair (sum over even k, sum over odd k), so the
// pairs come straight from 16-byte shared-memory loads, with nothing to duplicate or transpose, and one instruction does two
// multiply-adds (at the rate of two: measured 72 TFLOP/s either way, but half the issue slots).  What bounds it is shared memory: a
// warp's 16-byte load takes four clocks of the SM, however many lanes share an address, so 8 x 8 outputs per thread just balance the FMAs
// (64 per 16 floats loaded); 8 x 4 are at two thirds.  Small tiles therefore have few threads, not small thread tiles.  (On MmaTile 48 streams of four frames
// take 2.54 ms instead of 3.59 and are closer to 64 bits, 6.7e-7 against 8.7e-7; few streams, whose sums of 16 k round to nearest, would be further off, 5.7e-7 against
// 4.6e-7, and would no longer be as far ahead of many as they have to be.)
//
// A cluster of S CTAs along grid.x shares one output tile, each taking a contiguous range of k; the partial tiles meet through
// distributed shared memory and are added in rank order.  The arithmetic of an output -- which k a rank takes, the order of its sums, the
// order of ranks -- follows from K, S and the kind of tile alone, never from the tile's shape or from what else is in the launch.
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

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const float* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// hi = x to 11 bits, lo the rest (the MMA ignores what lo has behind its own 11)
__device__ __forceinline__ void tf32_parts(uint32_t x, uint32_t& hi, uint32_t& lo) {
    hi = (x + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(__uint_as_float(x) - __uint_as_float(hi));
}


// One thread's share of bringing the stages: NT threads, 16-byte pieces; a_row(r) / w_row(column): a row's address, nullptr for zeros; a_at(k): where in its row k
// lies; column_at(p): the column at place p of W's stage.  k in [k_lo, k_hi), multiples of 4.
template <int BM, int BN, int NT, class AAt>
struct Feed {
    static_assert(NT % 4 == 0, "a thread's pieces have one place in a step");
    static constexpr int PA = (BM * 4 + NT - 1) / NT, PW = (BN * 4 + NT - 1) / NT;      // pieces of a stage a thread copies
    static constexpr int kStageFloats = (BM + BN) * kLD;
    const float *ap[PA], *wp[PW], *any;
    float* sm;
    AAt a_at;
    int k_lo, k_hi, steps;

    template <class ARow, class WRow, class ColumnAt>
    __device__ __forceinline__ Feed(float* sm_, int lo, int hi, ARow a_row, AAt at, WRow w_row, ColumnAt column_at)
        : any(w_row(0)) /* (column 0 is always there) */, sm(sm_ + (threadIdx.x & 3) * 4), a_at(at), k_lo(lo + (threadIdx.x & 3) * 4), k_hi(hi), steps((hi - lo + kBK - 1) / kBK) {
#pragma unroll
        for (int x = 0; x < PA; ++x) ap[x] = row(x) < BM ? a_row(row(x)) : nullptr;
#pragma unroll
        for (int x = 0; x < PW; ++x) wp[x] = row(x) < BN ? w_row(column_at(row(x))) : nullptr;
    }
    __device__ static __forceinline__ int row(int x) { return (int)(threadIdx.x + x * NT) >> 2; }
    __device__ __forceinline__ void copy_w(int s) const {
        float* Ws = sm + (s % kStages) * kStageFloats + BM * kLD;
        const int k = k_lo + s * kBK;
#pragma unroll
        for (int x = 0; x < PW; ++x) {
            if (BN * 4 % NT != 0 && row(x) >= BN) break;
            const bool in = k < k_hi && wp[x];
            copy16(Ws + row(x) * kLD, in ? wp[x] + k : any, in);
        }
    }
    __device__ __forceinline__ void copy_a(int s) const {
        float* As = sm + (s % kStages) * kStageFloats;
        const int k = k_lo + s * kBK;
        const long long at = a_at(k);
#pragma unroll
        for (int x = 0; x < PA; ++x) {
            if (BM * 4 % NT != 0 && row(x) >= BM) break;
            const bool in = k < k_hi && ap[x];
            copy16(As + row(x) * kLD, in ? ap[x] + at : any, in);
        }
    }
    // group s of the copies: stage s.  before(): called when the first copies of W are on their way and before anything of A is read.
    template <class Before>
    __device__ __forceinline__ void start(Before before) const {
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s)
            if (s < steps) copy_w(s);
        before();
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s) {
            if (s < steps) copy_a(s);
            commit();
        }
    }
    // stage s has landed, and the one that was read before it is on its way anew
    __device__ __forceinline__ void next(int s) const {
        wait<kStages - 2>();
        __syncthreads();
        if (s + kStages - 1 < steps) { copy_w(s + kStages - 1); copy_a(s + kStages - 1); }
        commit();
    }
};

// this rank's range of k: whole steps, contiguous
__device__ __forceinline__ void rank_range(int K, int& lo, int& hi) {
    const int S = (int)cluster_size(), per = ((K + kBK - 1) / kBK + S - 1) / S * kBK;
    lo = min(K, (int)cluster_rank() * per);
    hi = min(K, lo + per);
}
// Hands the outputs of a tile to done(row, column, four values) -- four columns from a multiple of 4 on: straight from the registers (each(take): take(row, column,
// four values) for all of a thread's), or -- a cluster -- each rank its share of the rows after the partial tiles are added in rank order.  Every thread of every
// rank calls it.
template <int BM, int BN, int NT, class Each, class Done>
__device__ __forceinline__ void finish_tile(float* sm, Each each, Done done) {
    constexpr int kOutLd = BN + 4;           // floats between the rows of a partial tile
    const uint32_t S = cluster_size();
    if (S == 1) {
        each(done);
        return;
    }
    __syncthreads();                         // the stages are read by now
    each([&](int r, int c, float4 v) { *reinterpret_cast<float4*>(sm + r * kOutLd + c) = v; });
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
    cluster_sync();                          // nobody leaves while its tile is being read
}
template <int BM, int BN>
constexpr size_t tile_smem_bytes() {
    constexpr int stages = kStages * (BM + BN) * kLD, partial = BM * (BN + 4);
    return (size_t)(stages > partial ? stages : partial) * 4;
}

// A warp has MF x NF fragments of 16 x 8.  The columns of W lie in shared memory so that the two columns a lane has of fragments 2 j and 2 j + 1 are four
// neighbours: results move as 16-byte pieces.
template <int BM, int BN, int WM, int WN>
struct MmaTile {
    static constexpr int WARPS_N = BN / WN, NT = BM / WM * WARPS_N * 32, MF = WM / 16, NF = WN / 8, kStageFloats = (BM + BN) * kLD;
    static_assert(WM % 16 == 0 && WN % 16 == 0 && BM % WM == 0 && BN % WN == 0, "whole pairs of fragments");
    static constexpr size_t kSmemBytes = tile_smem_bytes<BM, BN>();
    typedef float Out[MF][NF][4];

    // the column that lies at place p of W's stage
    __device__ static __forceinline__ int column_at(int p) { return (p & ~15) + ((p >> 1) & 3) * 4 + ((p >> 3) & 1) * 2 + (p & 1); }

    template <class ARow, class AAt, class WRow, class Before>
    __device__ static __forceinline__ void product(float* sm, int k_lo, int k_hi, ARow a_row, AAt a_at, WRow w_row, Before before, Out& out) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int m = 0; m < MF; ++m)
#pragma unroll
            for (int n = 0; n < NF; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) out[m][n][e] = 0.0f;
        // where this lane's rows of the fragments start in a stage
        const int a_off = (warp / WARPS_N * WM + (lane & 15)) * kLD + (lane >> 4) * 4, w_off = (BM + warp % WARPS_N * WN + (lane & 7)) * kLD + (lane >> 3) * 4;
        const Feed<BM, BN, NT, AAt> feed(sm, k_lo, k_hi, a_row, a_at, w_row, column_at);
        feed.start(before);
        for (int s = 0; s < feed.steps; ++s) {
            const float* stage = sm + (s % kStages) * kStageFloats;
            feed.next(s);
            uint32_t w[NF][4];
#pragma unroll
            for (int n = 0; n < NF; ++n) ldmatrix4(w[n], stage + w_off + n * 8 * kLD);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t whi[NF][2], wlo[NF][2];
#pragma unroll
                for (int n = 0; n < NF; ++n)
#pragma unroll
                    for (int x = 0; x < 2; ++x) tf32_parts(w[n][2 * k + x], whi[n][x], wlo[n][x]);
#pragma unroll
                for (int m = 0; m < MF; ++m) {
                    uint32_t a[4], hi[4], lo[4];
                    ldmatrix4(a, stage + a_off + m * 16 * kLD + k * 8);
#pragma unroll
                    for (int x = 0; x < 4; ++x) tf32_parts(a[x], hi[x], lo[x]);
                    float sum[NF][4];
#pragma unroll
                    for (int n = 0; n < NF; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) sum[n][e] = 0.0f;
                    // the small products first: what the tensor core drops is below the last place of what it has so far
#pragma unroll
                    for (int n = 0; n < NF; ++n) mma_tf32(sum[n], lo, whi[n][0], whi[n][1]);
#pragma unroll
                    for (int n = 0; n < NF; ++n) mma_tf32(sum[n], hi, wlo[n][0], wlo[n][1]);
#pragma unroll
                    for (int n = 0; n < NF; ++n) mma_tf32(sum[n], hi, whi[n][0], whi[n][1]);
#pragma unroll
                    for (int n = 0; n < NF; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) out[m][n][e] += sum[n][e];
                }
            }
        }
        wait<0>();
        // outputs that parts cannot make
        static_assert(MF * NF * 4 <= 32, "a bit per output");
        uint32_t again = 0;
#pragma unroll
        for (int i = 0; i < MF * NF * 4; ++i) {
            const float x = fabsf(out[i / (NF * 4)][i / 4 % NF][i % 4]);
            if (!(x >= 0x1p-80f && x <= 0x1.fffffep127f) && x != 0.0f) again |= 1u << i;
        }
        while (again) {
            const int i = __ffs((int)again) - 1, n = i / 4 % NF, e = i % 4;
            again &= again - 1;
            const float* ar = a_row(warp / WARPS_N * WM + i / (NF * 4) * 16 + lane / 4 + 8 * (e >> 1));
            const float* wr = w_row(column_at(warp % WARPS_N * WN + n * 8 + 2 * (lane & 3) + (e & 1)));
            float sum = 0.0f;
            if (ar && wr)
                for (int k = k_lo; k < k_hi; k += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(ar + a_at(k)), y = *reinterpret_cast<const float4*>(wr + k);
                    sum = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, sum))));
                }
#pragma unroll
            for (int z = 0; z < MF * NF * 4; ++z)
                if (z == i) out[z / (NF * 4)][z / 4 % NF][z % 4] = sum;
        }
    }

    template <class Done>
    __device__ static __forceinline__ void finish(float* sm, const Out& out, Done done) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = warp / WARPS_N * WM + lane / 4, c0 = warp % WARPS_N * WN + (lane & 3) * 4;
        finish_tile<BM, BN, NT>(sm, [&](auto&& take) {
#pragma unroll
            for (int m = 0; m < MF; ++m)
#pragma unroll
                for (int j = 0; j < NF / 2; ++j)
#pragma unroll
                    for (int x = 0; x < 2; ++x)
                        take(r0 + m * 16 + 8 * x, c0 + j * 16, make_float4(out[m][2 * j][2 * x], out[m][2 * j][2 * x + 1], out[m][2 * j + 1][2 * x], out[m][2 * j + 1][2 * x + 1]));
        }, done);
    }
};

// Threads are laid out as THM x THN, a warp 4 x 8 of them.  A thread's rows are ty + i * THM.  Its columns come in runs of four
// (column(tx, j)), so that results move as 16-byte pieces; the columns of W lie in shared memory in the order j * THN + tx, so that
// neighbouring threads read neighbouring rows all the same.  RUN > 0: the two chains of an output are added up and begin anew every RUN steps.
template <int BM, int BN, int TM, int TN, int RUN>
struct Tile {
    static constexpr int THM = BM / TM, THN = BN / TN, NT = THM * THN, kStageFloats = (BM + BN) * kLD;
    static_assert(THM % 4 == 0 && THN % 8 == 0, "warps of 4 x 8 threads");
    static_assert(TN % 4 == 0, "runs of four columns");
    static constexpr size_t kSmemBytes = tile_smem_bytes<BM, BN>();
    typedef float Out[TM][TN];

    __device__ static __forceinline__ int ty() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w / (THN / 8)) * 4 + (l >> 3); }
    __device__ static __forceinline__ int tx() { const int w = threadIdx.x >> 5, l = threadIdx.x & 31; return (w % (THN / 8)) * 8 + (l & 7); }

    // column of a thread's j-th output, and the other way round: the column that lies at place p of W's stage
    __device__ static __forceinline__ int column(int x, int j) { return (j / 4) * (4 * THN) + x * 4 + j % 4; }
    __device__ static __forceinline__ int column_at(int p) { return column(p % THN, p / THN); }

    template <class ARow, class AAt, class WRow, class Before>
    __device__ static __forceinline__ void product(float* sm, int k_lo, int k_hi, ARow a_row, AAt a_at, WRow w_row, Before before, Out& out) {
        const int row_y = ty(), row_x = tx();
        unsigned long long acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) { acc[i][j] = 0ull; out[i][j] = 0.0f; }
        const Feed<BM, BN, NT, AAt> feed(sm, k_lo, k_hi, a_row, a_at, w_row, column_at);
        feed.start(before);
        for (int s = 0; s < feed.steps; ++s) {
            const float *As = sm + (s % kStages) * kStageFloats, *Ws = As + BM * kLD;
            feed.next(s);
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
            if (RUN > 0 && s % (RUN > 0 ? RUN : 1) == RUN - 1) {
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

    template <class Done>
    __device__ static __forceinline__ void finish(float* sm, const Out& out, Done done) {
        finish_tile<BM, BN, NT>(sm, [&](auto&& take) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; j += 4) take(ty() + i * THM, column(tx(), j), make_float4(out[i][j], out[i][j + 1], out[i][j + 2], out[i][j + 3]));
        }, done);
    }
};

}  // namespace f32t
}  // namespace smol
