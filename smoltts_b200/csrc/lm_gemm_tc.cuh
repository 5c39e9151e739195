// Matrix product for many rows (prompt portions), bf16 on the 5th-generation tensor cores (sm_100a).  Included by lm_kernels.cu.
//
// y[M, N] = a[M, K] . w[N, K]^T in tiles of 128 rows x BN columns, one persistent CTA per SM walking them; row tiles that share a weight
// tile run on neighbouring CTAs.  The roles of a CTA overlap instead of taking turns: two threads keep TMA loads of 64-element K stages
// going through a ring, a warp issues tcgen05.mma into one of two accumulators in tensor memory, and eight warps drain the other
// accumulator meanwhile.
//
// An accumulator drops what lies below its last place with every MMA, so K is summed in four parts, each in an accumulator begun anew, which
// the draining warps add in fp32 registers: error against 64 bits 1.8e-7 at K = 768, 1.1e-6 at 4608 (one accumulator over all of K: 7.3e-7 and
// 5.0e-6; values in [0, 1): 2.4e-7 and 2.2e-6 against 1.3e-6 and 1.5e-5).  It costs no time as the MMAs are issued now: the whole warp walks, one
// elected lane issues, and the operands stay in uniform registers (2048 x 768 x 4608 27 us, 1801 x 1536 x 6144 36; one accumulator and a
// single thread walking 29 and 39, four parts and a single thread 47 and 63).
//
// What bounds it: a stage brings (128 + BN) x 128 bytes through the SM's 64 bytes per clock from L2 and takes 2 BN clocks of the tensor
// pipe, so up to BN = 128 the loads take twice as long as the MMAs and at 256 half again; wide tiles win as long as they still fill the
// SMs, which gemm_tc_pick weighs.  The accumulators leave through a warp's own padded rows in shared memory, so that global stores are
// whole 128-byte lines.  2048 rows of the width-768 Pamasun layers: 17.5 us a product against 28 with 96-column tiles whose loads, MMAs
// and epilogue took turns; 1801 rows of width 1536: 33 us against 60.
// Rows and columns outside the matrices are zero-filled by TMA (a partial last K stage adds zeros); rows past M of the activation
// buffer hold stale values whose accumulator lanes are never stored.
#pragma once

namespace smol {
namespace lm {

constexpr int kTcEpilogueWarps = 8;
constexpr int kTcThreads = 128 + kTcEpilogueWarps * 32;      // warps 0 and 2: loads of activations and weights, 1: MMAs, 4 to 11: epilogue
constexpr int kTcParts = 4;              // partial sums of a tile: a quarter of K each
constexpr int kTcMinRows = 257;          // below this the mma.sync tiles fill the GPU better than 128-row tiles
constexpr int kTcMinCols = 96;
constexpr int kTcStageLd = 36;           // floats between the staged rows of a 16 x 32 piece: conflict-free for 16-byte accesses

template <int BN> constexpr int gemm_tc_stages() { return BN >= 256 ? 4 : BN >= 192 ? 5 : 6; }
template <int BN> constexpr int gemm_tc_stage_bytes() { return (umma::kM + BN) * umma::kBK * 2; }
template <int BN> constexpr int gemm_tc_smem() { return gemm_tc_stages<BN>() * gemm_tc_stage_bytes<BN>() + kTcEpilogueWarps * 16 * kTcStageLd * 4 + 1024; }

struct GemmTcBars {
    uint64_t full[8], empty[8];      // ring stages: bytes landed / consumed by the MMAs
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem;
};

__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::s2u(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

// One MMA / one commit by the warp's elected lane, every lane calling: the operands stay in uniform registers.  `more` 0: the accumulator begins anew.
__device__ __forceinline__ void mma_bf16_one(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.u32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
__device__ __forceinline__ void commit_one(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(umma::s2u(bar)) : "memory");
}

// Grouped rows (io.tile_group != nullptr): the row tiles come from the device-built table (128 rows each, group g's rows end
// at seg[g + 1]; rows of the tile beyond that belong to the next group and are computed but not stored), and group g's
// weights are rows g * N .. of the weight map.
template <int BN>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                                                                float* __restrict__ y, const int M, const int N, const int K, const GemmIo io) {
    constexpr int ST = gemm_tc_stages<BN>(), SB = gemm_tc_stage_bytes<BN>(), kA = umma::kM * umma::kBK * 2, kSteps = umma::kBK / 16;
    static_assert(BN % 32 == 0 && BN <= 256 && ST <= 8, "tile width");
    extern __shared__ unsigned char tc_smem[];
    __shared__ GemmTcBars bars;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { umma::bar_init(&bars.full[s], 2); umma::bar_init(&bars.empty[s], 1); }
        for (int i = 0; i < 2; ++i) { umma::bar_init(&bars.acc_full[i], 1); umma::bar_init(&bars.acc_empty[i], kTcEpilogueWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) umma::tmem_alloc(&bars.tmem);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = bars.tmem;
    if (warp != 2 || io.tile_group) dep_wait();      // a plain product's weights need not wait for the kernel before (smol_lm_linear, whose w that may have made, launches plainly)
    dep_go();
    const int m_tiles = io.tile_group ? *io.n_tiles : (M + umma::kM - 1) / umma::kM, n_tiles = (N + BN - 1) / BN;
    const int tiles = m_tiles * n_tiles, nk = (K + umma::kBK - 1) / umma::kBK;
    // where tile u lies: first row of a, end of the rows that are stored, first row of w
    auto place = [&](int u, int& m0, int& m_end, int& w_row) {
        m0 = (u % m_tiles) * umma::kM;
        m_end = M;
        w_row = (u / m_tiles) * BN;
        if (io.tile_group) {
            const int g = io.tile_group[u % m_tiles];
            m0 = io.tile_row0[u % m_tiles];
            m_end = io.seg[g + 1];
            w_row += g * N;
        }
    };
    if ((warp == 0 || warp == 2) && lane == 0) {
        // ---- loads: warp 0 the activation box of every stage, warp 2 the weight box ----
        uint32_t c = 0;
        for (int u = blockIdx.x; u < tiles; u += gridDim.x) {
            int m0, m_end, w_row;
            place(u, m0, m_end, w_row);
            for (int kc = 0; kc < nk; ++kc, ++c) {
                const uint32_t s = c % ST;
                if (c >= ST) umma::bar_wait(&bars.empty[s], (c / ST - 1u) & 1u);
                const uint32_t at = umma::s2u(ring + (size_t)s * SB);
                if (warp == 0) {
                    umma::bar_expect_tx(&bars.full[s], kA);
                    umma::tma_load_2d(at, &tm_a, kc * umma::kBK, m0, &bars.full[s]);
                } else {
                    umma::bar_expect_tx(&bars.full[s], SB - kA);
                    umma::tma_load_2d(at + kA, &tm_w, kc * umma::kBK, w_row, &bars.full[s]);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMAs: nk of the tile's 4 nk into one accumulator, the next nk into the other (the whole warp walks, one lane issues) ----
        const uint32_t idesc = umma::instr_desc(BN);
        uint32_t c = 0, p = 0;      // stages, parts so far
        for (int u = blockIdx.x; u < tiles; u += gridDim.x) {
            int n = 0;              // MMAs of the part so far
            for (int kc = 0; kc < nk; ++kc, ++c) {
                const uint32_t s = c % ST;
                umma::bar_wait(&bars.full[s], (c / ST) & 1u);
                if (n == 0 && p >= 2) umma::bar_wait(&bars.acc_empty[p & 1u], (p / 2 - 1u) & 1u);
                umma::fence_after_sync();
                const uint64_t da = umma::smem_desc_sw128(umma::s2u(ring + (size_t)s * SB)), dw = umma::smem_desc_sw128(umma::s2u(ring + (size_t)s * SB) + kA);
                if (n + kSteps <= nk) {
#pragma unroll
                    for (int q = 0; q < kSteps; ++q) mma_bf16_one(tmem + (p & 1u) * BN, da + q * 2, dw + q * 2, idesc, (uint32_t)(n + q));
                    n += kSteps;
                } else {
#pragma unroll 1
                    for (int q = 0; q < kSteps; ++q) {
                        if (n == nk) {
                            commit_one(&bars.acc_full[p++ & 1u]);
                            n = 0;
                            if (p >= 2) umma::bar_wait(&bars.acc_empty[p & 1u], (p / 2 - 1u) & 1u);
                            umma::fence_after_sync();
                        }
                        mma_bf16_one(tmem + (p & 1u) * BN, da + q * 2, dw + q * 2, idesc, (uint32_t)n);
                        ++n;
                    }
                }
                commit_one(&bars.empty[s]);
                if (n == nk) {                                   // after `empty`: nothing of the block's is in flight once its last part is read
                    commit_one(&bars.acc_full[p++ & 1u]);
                    n = 0;
                }
            }
        }
    } else if (warp >= 4) {
        // ---- epilogue: rows 32 (w % 4) .. + 31, half of the columns ----
        constexpr int HC = (BN / 2 + 31) / 32 * 32;      // columns of the first half
        const int quad = warp & 3, half = (warp - 4) >> 2, cols = half ? BN - HC : HC;
        float* stage = reinterpret_cast<float*>(ring + (size_t)ST * SB) + (warp - 4) * 16 * kTcStageLd;
        const bool vec = N % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
        uint32_t p = 0;
        for (int u = blockIdx.x; u < tiles; u += gridDim.x) {
            int m0, m_end, w_row;
            place(u, m0, m_end, w_row);
            const int n0 = (u / m_tiles) * BN + half * HC, r0 = m0 + quad * 32, here = min(cols, N - n0);
            float sum[HC];
#pragma unroll
            for (int i = 0; i < HC; ++i) sum[i] = 0.0f;
#pragma unroll 1
            for (int x = 0; x < kTcParts; ++x, ++p) {
                const uint32_t b = p & 1u, d = tmem + b * BN + half * HC + ((uint32_t)(quad * 32) << 16);
                umma::bar_wait(&bars.acc_full[b], (p / 2) & 1u);
                __syncwarp();
                umma::fence_after_sync();
#pragma unroll
                for (int c0 = 0; c0 < HC; c0 += 16) {
                    if (c0 >= here) break;
                    uint32_t v[16];
                    tmem_ld16_issue(d + c0, v);
                    umma::tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) sum[c0 + e] += __uint_as_float(v[e]);
                }
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) bar_arrive(&bars.acc_empty[b]);
            }
            if (r0 >= m_end) continue;
#pragma unroll
            for (int c0 = 0; c0 < HC; c0 += 32) {
                if (c0 >= here) break;
                const int col = n0 + c0 + (lane & 7) * 4;
#pragma unroll
                for (int h = 0; h < 2; ++h) {            // 16 rows at a time
                    __syncwarp();
                    if (lane >> 4 == h) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            *reinterpret_cast<float4*>(stage + (lane & 15) * kTcStageLd + i * 4) = make_float4(sum[c0 + 4 * i], sum[c0 + 4 * i + 1], sum[c0 + 4 * i + 2], sum[c0 + 4 * i + 3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int r = i * 4 + (lane >> 3), m = r0 + h * 16 + r;
                        const float4 o = *reinterpret_cast<const float4*>(stage + r * kTcStageLd + (lane & 7) * 4);
                        if (m >= m_end) continue;
                        float* to = y + (size_t)m * N + col;
                        if (vec) {
                            if (col < N) *reinterpret_cast<float4*>(to) = o;
                        } else {
                            if (col < N) to[0] = o.x;
                            if (col + 1 < N) to[1] = o.y;
                            if (col + 2 < N) to[2] = o.z;
                            if (col + 3 < N) to[3] = o.w;
                        }
                    }
                }
            }
        }
    }
    __syncwarp();
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 1) umma::tmem_free(tmem);
}

}  // namespace lm
}  // namespace smol
