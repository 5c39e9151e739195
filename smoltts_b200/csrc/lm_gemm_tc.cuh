// Matrix product for many rows (prompt portions), bf16 on the 5th-generation tensor cores (sm_100a).  Included by lm_kernels.cu.
//
// y[M, N] = a[M, K] . w[N, K]^T in tiles of 128 rows x BN columns, one persistent CTA per SM walking them; row tiles that share a weight
// tile run on neighbouring CTAs.  The roles of a CTA overlap instead of taking turns: two threads keep TMA loads of 64-element K stages
// going through a ring, one thread issues tcgen05.mma into one of two accumulators in tensor memory, and four warps drain the other
// accumulator while the next tile is multiplied.
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

constexpr int kTcThreads = 256;          // warps 0 and 2: loads of activations and weights, 1: MMAs, 4 to 7: epilogue
constexpr int kTcMinRows = 257;          // below this the mma.sync tiles fill the GPU better than 128-row tiles
constexpr int kTcMinCols = 96;
constexpr int kTcStageLd = 36;           // floats between the staged rows of a 32 x 32 piece: conflict-free for 16-byte accesses

template <int BN> constexpr int gemm_tc_stages() { return BN >= 256 ? 4 : BN >= 192 ? 5 : 6; }
template <int BN> constexpr int gemm_tc_stage_bytes() { return (umma::kM + BN) * umma::kBK * 2; }
template <int BN> constexpr int gemm_tc_smem() { return gemm_tc_stages<BN>() * gemm_tc_stage_bytes<BN>() + 4 * 32 * kTcStageLd * 4 + 1024; }

struct GemmTcBars {
    uint64_t full[8], empty[8];      // ring stages: bytes landed / consumed by the MMAs
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem;
};

__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::s2u(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr) : "memory");
}

// Grouped rows (io.tile_group != nullptr): the row tiles come from the device-built table (128 rows each, group g's rows end
// at seg[g + 1]; rows of the tile beyond that belong to the next group and are computed but not stored), and group g's
// weights are rows g * N .. of the weight map.
template <int BN>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                                                                float* __restrict__ y, const int M, const int N, const int K, const GemmIo io) {
    constexpr int ST = gemm_tc_stages<BN>(), SB = gemm_tc_stage_bytes<BN>(), kA = umma::kM * umma::kBK * 2;
    static_assert(BN % 32 == 0 && BN <= 256 && ST <= 8, "tile width");
    extern __shared__ unsigned char tc_smem[];
    __shared__ GemmTcBars bars;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { umma::bar_init(&bars.full[s], 2); umma::bar_init(&bars.empty[s], 1); }
        for (int i = 0; i < 2; ++i) { umma::bar_init(&bars.acc_full[i], 1); umma::bar_init(&bars.acc_empty[i], 4); }
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
    } else if (warp == 1 && lane == 0) {
        // ---- MMAs ----
        const uint32_t idesc = umma::instr_desc(BN);
        uint32_t c = 0, t = 0;
        for (int u = blockIdx.x; u < tiles; u += gridDim.x, ++t) {
            const uint32_t b = t & 1u, d = tmem + b * BN;
            if (t >= 2) umma::bar_wait(&bars.acc_empty[b], (t / 2 - 1u) & 1u);
            umma::fence_after_sync();
            for (int kc = 0; kc < nk; ++kc, ++c) {
                const uint32_t s = c % ST;
                umma::bar_wait(&bars.full[s], (c / ST) & 1u);
                umma::fence_after_sync();
                const uint32_t at = umma::s2u(ring + (size_t)s * SB);
#pragma unroll
                for (int q = 0; q < umma::kBK / 16; ++q)
                    umma::mma_bf16(d, umma::smem_desc_sw128(at + q * 32), umma::smem_desc_sw128(at + kA + q * 32), idesc, (kc > 0 || q > 0) ? 1u : 0u);
                umma::commit(&bars.empty[s]);
            }
            umma::commit(&bars.acc_full[b]);
        }
    } else if (warp >= 4) {
        // ---- epilogue: warp w drains the accumulator rows 32 (w - 4) .. + 31, 32 columns at a time ----
        float* stage = reinterpret_cast<float*>(ring + (size_t)ST * SB) + (warp - 4) * 32 * kTcStageLd;
        const bool vec = N % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
        uint32_t t = 0;
        for (int u = blockIdx.x; u < tiles; u += gridDim.x, ++t) {
            int m0, m_end, w_row;
            place(u, m0, m_end, w_row);
            const int n0 = (u / m_tiles) * BN, r0 = m0 + (warp - 4) * 32;
            const uint32_t b = t & 1u;
            umma::bar_wait(&bars.acc_full[b], (t / 2) & 1u);
            umma::fence_after_sync();
            const uint32_t d = tmem + b * BN + ((uint32_t)((warp - 4) * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < BN && n0 + c0 < N; c0 += 32) {
                uint32_t v[32];
                tmem_ld32_issue(d + c0, v);
                umma::tmem_ld_wait();
                if (r0 >= m_end) continue;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(stage + lane * kTcStageLd + i * 4) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                __syncwarp();
                const int col = n0 + c0 + (lane & 7) * 4;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + (lane >> 3), m = r0 + r;
                    const float4 o = *reinterpret_cast<const float4*>(stage + r * kTcStageLd + (lane & 7) * 4);
                    if (m >= m_end) continue;
                    float* p = y + (size_t)m * N + col;
                    if (vec) {
                        if (col < N) *reinterpret_cast<float4*>(p) = o;
                    } else {
                        if (col < N) p[0] = o.x;
                        if (col + 1 < N) p[1] = o.y;
                        if (col + 2 < N) p[2] = o.z;
                        if (col + 3 < N) p[3] = o.w;
                    }
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars.acc_empty[b]);
        }
    }
    __syncwarp();
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 1) umma::tmem_free(tmem);
}

}  // namespace lm
}  // namespace smol
