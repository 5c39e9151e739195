// Softmax attention of prompt portions on the 5th-generation tensor cores, bf16 (sm_100a).  Included by lm_kernels.cu.
//
// One block per (128 rows of a sequence in this step, sequence, query head).  Keys and values come 64 positions at a time from the paged
// pool.  The roles run side by side: loader warps keep a ring of three or four stages filled (one each, so that as many loads are in flight; 128-byte-swizzled rows of 64 columns, which serve the product with the queries k-contiguous and the one with the weights
// n-contiguous, so nothing is transposed), one thread issues the tcgen05 products, sixteen warps take the scores out of tensor memory -- four threads per row, 16 columns each -- and keep the running softmax.  The scores of the next 64
// positions are multiplied while the current ones are worked on, the product with the values while the next ones are.  That product is
// read back from tensor memory and joins the fp32 running sums, which stay in registers.
//
// As in attn_flash_kernel scores, penalties, maximum, denominator and sums are fp32, a softmax weight enters as a bf16 head and a bf16
// remainder (two MMAs), the sink is the initial state of the running softmax, and a row takes nothing from 64 positions it does not see.
// Differential attention (MAPS 2) walks the keys once per map; the first map's result waits in shared memory, each thread's own part.
//
// What bounds it: the instructions of a step, the loaders' as much as the softmax's 64 x 128 scores with one exponential (and, with a distance
// penalty, one logarithm) each -- hence four threads per row, whose latencies cover one another, a warp per stage, and addresses that advance
// by constants.  Two threads per row and three stages: 84 / 98 / 48 / 99 us instead of the following; a look at the page, the limit and the
// swizzle for every row copied: 64 / 82 / 42 / 97.
// 2048 tokens, 12 heads of 64 with a distance penalty: 57 us, attn_flash_kernel 165; 1801 tokens, 12 heads of 128: 74 against 219; 1024
// tokens, 12 heads over a latent of 160: 40 against 101; 3 x 1000 tokens, 6 heads of two maps: 72 against 116.
#pragma once

#include <type_traits>

namespace smol {
namespace lm {

constexpr int kFtRows = 128, kFtKeys = 64;
constexpr int kFtParts = 4, kFtCols = kFtKeys / kFtParts;                   // threads per row, score columns of each
constexpr int kFtSoftWarps = 4 * kFtParts, kFtMaxStages = 4;
constexpr int kFtPBytes = kFtRows * kFtKeys * 2;                              // heads or remainders of a step's weights
// VK: the values are the first columns of the key rows
__host__ __device__ constexpr int ft_stage_bytes(int DK, int DV, bool VK) { return kFtKeys * 2 * (DK + (VK ? 0 : DV)); }
// three stages where a fourth does not fit
__host__ __device__ constexpr int ft_stages(int DV, int MAPS) { return MAPS == 2 && DV == 128 ? 3 : kFtMaxStages; }
__host__ __device__ constexpr int ft_threads(int DV, int MAPS) { return (kFtSoftWarps + 1 + ft_stages(DV, MAPS)) * 32; }
__host__ __device__ constexpr int ft_smem(int DK, int DV, bool VK, int MAPS) {
    return 1024 + MAPS * kFtRows * DK * 2 + ft_stages(DV, MAPS) * ft_stage_bytes(DK, DV, VK) + 2 * kFtPBytes + (MAPS - 1) * kFtRows * DV * 4;
}

struct FlashTcBars {
    uint64_t full[kFtMaxStages], empty[kFtMaxStages];          // stages of keys and values
    uint64_t s_full[2], s_empty[2];      // scores in tensor memory
    uint64_t p_full, o_full;             // weights in shared memory (their product's last result has been read); weights x values in tensor memory
    uint32_t tmem;
};

// byte of 16-byte piece c of row r in a tile of 128-byte rows with the 128-byte swizzle
__device__ __forceinline__ int sw128_at(int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); }
__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::s2u(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// The instruction and shared-memory descriptors of an operand B that lies n-contiguous: rows of 64 columns per k, 8 rows of k 1024 bytes
// apart, the next 64 columns kFtKeys rows further.
__device__ __forceinline__ uint32_t instr_desc_bn(int n) { return umma::instr_desc(n) | (1u << 16); }
__device__ __forceinline__ uint64_t smem_desc_bn(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kFtKeys * 128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ float log2_fast(float x) {      // hardware instruction, x >= 1
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max_of(const float (&S)[kFtCols]) {
    float part[4] = {S[0], S[1], S[2], S[3]};
#pragma unroll
    for (int e = 4; e < kFtCols; ++e) part[e % 4] = fmaxf(part[e % 4], S[e]);
    return fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
}
// The scores of a thread's columns in units of log2 (multiplied by log2 e), dist = the row's position - the first column's; MASK: columns the
// row does not see are -inf.  The distance penalty r1 ln(1 + r2 d) is r1 log2(1 + r2 d) in these units.
template <bool GENERAL, bool PENALTY, bool MASK>
__device__ __forceinline__ void ft_scores(const AttnArgs& A, float (&S)[kFtCols], int dist, int win, float r1, float r2, float slope) {
    constexpr float kLog2e = 1.4426950408889634f;
    const float d0 = (float)dist, x0 = fmaf(r2, d0, 1.0f), scale = A.scale * kLog2e;
#pragma unroll
    for (int e = 0; e < kFtCols; ++e) {
        float v;
        if (GENERAL) {
            v = S[e] * A.scale;
            if (A.softcap > 0.0f) v = A.softcap * (1.0f - __fdividef(2.0f, __expf(v * A.two_over_cap) + 1.0f));
            v = (v - slope * (d0 - (float)e)) * kLog2e;
            if (PENALTY) v = fmaf(-r1, log2_fast(fmaf(-(float)e, r2, x0)), v);
        } else if (PENALTY) {
            v = fmaf(S[e], scale, -r1 * log2_fast(fmaf(-(float)e, r2, x0)));
        } else {
            v = S[e] * scale;
        }
        S[e] = !MASK || (dist - e >= 0 && dist - e < win) ? v : -INFINITY;
    }
}
template <bool MASK>
__device__ __forceinline__ void ft_scores_any(const AttnArgs& A, float (&S)[kFtCols], int dist, int win, float r1, float r2, float slope) {
    if (A.softcap > 0.0f || A.slope) {
        if (A.r1) ft_scores<true, true, MASK>(A, S, dist, win, r1, r2, slope);
        else ft_scores<true, false, MASK>(A, S, dist, win, r1, r2, slope);
    } else if (A.r1) ft_scores<false, true, MASK>(A, S, dist, win, r1, r2, slope);
    else ft_scores<false, false, MASK>(A, S, dist, win, r1, r2, slope);
}

// DK / DV: key and value sizes padded to multiples of 64 (zeros).  d, dv and every row stride and offset are multiples of 8 elements.
template <int DK, int DV, bool VK, int MAPS>
__global__ void __launch_bounds__(ft_threads(DV, MAPS), 1) attn_flash_tc_kernel(const AttnArgs A, const bf16* __restrict__ qbuf, const bf16* __restrict__ pool,
                                                                      bf16* __restrict__ out) {
    constexpr int NB = ft_stages(DV, MAPS), SB = ft_stage_bytes(DK, DV, VK), OC = DV / kFtParts;
    static_assert(DK % 64 == 0 && DV % 64 == 0 && DV <= 128 && (!VK || (DV <= DK && MAPS == 1)), "tile sizes");
    extern __shared__ unsigned char ft_smem_raw[];
    __shared__ FlashTcBars bars;
    __shared__ float s_max[2][kFtParts][kFtRows], s_sum[2][kFtParts][kFtRows];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *Qs = base, *KV = Qs + MAPS * kFtRows * DK * 2, *Ps = KV + NB * SB;          // Ps: heads, then remainders
    float* first_map = reinterpret_cast<float*>(Ps + 2 * kFtPBytes);                           // MAPS 2: [OC][threads of the softmax]
    dep_wait();
    const int s = blockIdx.y, t0 = A.seq_start[s], n = A.seq_start[s + 1] - t0;
    const int tile = gridDim.z - 1 - blockIdx.z;                                               // the tiles with the most keys start first
    if (n <= kShortSeq || tile * kFtRows >= n) return;
    const int h = blockIdx.x, g = h / (A.H / A.G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos0 = A.tok_pos[t0], row0 = tile * kFtRows, last_pos = pos0 + min(n, row0 + kFtRows) - 1;
    const int j_start = attn_first_key(A, pos0 + row0) / kFtKeys * kFtKeys, tiles = (last_pos - j_start) / kFtKeys + 1, steps = MAPS * tiles;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) { umma::bar_init(&bars.full[i], 32); umma::bar_init(&bars.empty[i], 1); }
        for (int i = 0; i < 2; ++i) { umma::bar_init(&bars.s_full[i], 1); umma::bar_init(&bars.s_empty[i], kFtSoftWarps); }
        umma::bar_init(&bars.p_full, kFtSoftWarps);
        umma::bar_init(&bars.o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kFtSoftWarps) umma::tmem_alloc(&bars.tmem);
    // queries of the tile: rows beyond the sequence and columns beyond d are zeros
    for (int i = threadIdx.x; i < MAPS * kFtRows * (DK / 8); i += ft_threads(DV, MAPS)) {
        const int mp = i / (kFtRows * (DK / 8)), r = i / (DK / 8) % kFtRows, c = i % (DK / 8);
        const bool in = row0 + r < n && c * 8 < A.d;
        cp_async16_or_zero(Qs + mp * (kFtRows * DK * 2) + (c / 8) * (kFtRows * 128) + sw128_at(r, c % 8),
                           in ? qbuf + (((size_t)(t0 + row0 + r) * A.H + h) * MAPS + mp) * A.d + c * 8 : qbuf, in);
    }
    cp_async_commit_group();
    cp_async_wait_group<0>();
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    dep_go();      // behind the allocation: a kernel set up early that wants tensor memory too must not get it first
    umma::fence_after_sync();
    const uint32_t tmem = bars.tmem, tm_o = tmem + 2 * kFtKeys;                                 // scores at columns 0 and 64, products from 128 on
    if (warp > kFtSoftWarps) {
        // ---- loaders: a warp per stage ----
        const int st = warp - kFtSoftWarps - 1;
        const int32_t* bt = A.block_table + (size_t)s * A.max_pages;
        const bool one_page = A.page_size % kFtKeys == 0;
        for (int i = st; i < steps; i += NB) {
            const int map = MAPS == 1 ? 0 : i / tiles, j0 = j_start + (i - map * tiles) * kFtKeys;
            unsigned char* Kt = KV + st * SB;
            // the page and the position in it of keys lane and lane + 32 (within one page: of the first key)
            const bf16* page[2];
            int in_page[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int j = one_page ? j0 : min(j0 + 32 * x + lane, last_pos), pg = j / A.page_size;
                page[x] = pool + (size_t)bt[pg] * A.page_elems;
                in_page[x] = j - pg * A.page_size;
            }
            if (i >= NB) umma::bar_wait(&bars.empty[st], (i / NB - 1) & 1);
            __syncwarp();
            // 64 rows of a head into blocks of 64 columns, eight lanes per row, four rows at a time; zeros beyond `width` and last_pos
            auto copy = [&](unsigned char* to, auto blocks_of, size_t off, int head, int ld, int width) {
                constexpr int blocks = decltype(blocks_of)::value;
                if (one_page && j0 + kFtKeys - 1 <= last_pos) {
                    // whole rows of one page: addresses advance by constants (rows y 4 .. + 3: the swizzle alternates with y)
                    const bf16* p = page[0] + off + ((size_t)head * A.page_size + in_page[0] + (lane >> 3)) * ld;
                    const uint32_t d = umma::s2u(to) + (lane >> 3) * 128;
                    const uint32_t d01[2] = {d + (((lane & 7) ^ (lane >> 3)) << 4), d + (((lane & 7) ^ (4 + (lane >> 3))) << 4)};
                    uint32_t bytes[blocks];
                    int col[blocks];
#pragma unroll
                    for (int cb = 0; cb < blocks; ++cb) {
                        const int c = cb * 64 + (lane & 7) * 8;
                        bytes[cb] = c < width ? 16 : 0;
                        col[cb] = c < width ? c : 0;
                    }
#pragma unroll
                    for (int y = 0; y < 16; ++y, p += 4 * (size_t)ld)
#pragma unroll
                        for (int cb = 0; cb < blocks; ++cb)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d01[y & 1] + y * 512 + cb * (kFtKeys * 128)), "l"(p + col[cb]), "r"(bytes[cb]) : "memory");
                    return;
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const bf16* at = page[x] + off + ((size_t)head * A.page_size + in_page[x]) * ld;
#pragma unroll 2
                    for (int y = 0; y < 8; ++y) {
                        const int r = y * 4 + (lane >> 3), row = 32 * x + r;
                        const bf16* src = one_page ? at + (size_t)row * ld : reinterpret_cast<const bf16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(at), r));
#pragma unroll
                        for (int cb = 0; cb < blocks; ++cb) {
                            const int c = cb * 64 + (lane & 7) * 8;
                            const bool in = c < width && j0 + row <= last_pos;
                            cp_async16_or_zero(to + cb * (kFtKeys * 128) + sw128_at(row, lane & 7), in ? src + c : pool, in);
                        }
                    }
                }
            };
            copy(Kt, std::integral_constant<int, DK / 64>{}, A.k_off, g * MAPS + map, A.k_ld, A.d);
            if (!VK) copy(Kt + kFtKeys * DK * 2, std::integral_constant<int, DV / 64>{}, A.v_off, g, A.v_ld, A.dv);
            cp_async_commit_group();
            cp_async_wait_group<0>();
            umma::fence_async_smem();
            bar_arrive(&bars.full[st]);
        }
    } else if (warp == kFtSoftWarps) {
        if (lane == 0) {
            // ---- products ----
            const uint32_t p0 = umma::s2u(Ps), id_s = umma::instr_desc(kFtKeys), id_o = instr_desc_bn(DV);
            auto values = [&](int i) {
                const int st = i % NB;
                umma::bar_wait(&bars.p_full, i & 1);
                umma::fence_after_sync();
                const uint32_t v = umma::s2u(KV + st * SB + (VK ? 0 : kFtKeys * DK * 2));
#pragma unroll
                for (int x = 0; x < 2; ++x)                  // all heads, then all remainders
#pragma unroll
                    for (int k = 0; k < kFtKeys / 16; ++k)
                        umma::mma_bf16(tm_o, umma::smem_desc_sw128(p0 + x * kFtPBytes + k * 32), smem_desc_bn(v + k * 16 * 128), id_o, (x > 0 || k > 0) ? 1u : 0u);
                umma::commit(&bars.empty[st]);
                umma::commit(&bars.o_full);                  // last: nothing of the block's is in flight once its final product is read
            };
            for (int i = 0; i < steps; ++i) {
                const int b = i & 1, st = i % NB;
                umma::bar_wait(&bars.full[st], (i / NB) & 1);
                if (i >= 2) umma::bar_wait(&bars.s_empty[b], ((i >> 1) - 1) & 1);
                umma::fence_after_sync();
                const uint32_t k0 = umma::s2u(KV + st * SB), q0 = umma::s2u(Qs) + (MAPS == 2 && i >= tiles ? kFtRows * DK * 2 : 0);
#pragma unroll
                for (int k = 0; k < DK / 16; ++k)
                    umma::mma_bf16(tmem + b * kFtKeys, umma::smem_desc_sw128(q0 + (k / 4) * (kFtRows * 128) + (k % 4) * 32),
                                   umma::smem_desc_sw128(k0 + (k / 4) * (kFtKeys * 128) + (k % 4) * 32), id_s, k > 0 ? 1u : 0u);
                umma::commit(&bars.s_full[b]);
                if (i > 0) values(i - 1);
            }
            values(steps - 1);
        }
    } else {
        // ---- softmax: warps q, q + 4, q + 8, q + 12 share rows 32 q .. + 31; part p has columns 16 p .. + 15 of the scores, a quarter of the values' ----
        const int quad = warp & 3, part = warp >> 2, row = quad * 32 + lane, i_pos = pos0 + row0 + row, first_pos = i_pos - lane;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        constexpr float kLog2e = 1.4426950408889634f;
        const float r1 = A.r1 ? A.r1[h] : 0.0f, r2 = A.r1 ? A.r2[h] : 0.0f, sink = A.sink ? A.sink[h] * kLog2e : -INFINITY, slope = A.slope ? A.slope[h] : 0.0f;
        const int win = A.window > 0 ? A.window : 0x3fffffff;
        // the score is the scaled product alone
        const bool plain = !A.r1 && !A.slope && A.softcap == 0.0f && A.window == 0 && A.scale > 0.0f;
        float m = sink, l = (part == 0 && A.sink) ? 1.0f : 0.0f;      // m in units of log2
        float o[OC];
#pragma unroll
        for (int c = 0; c < OC; ++c) o[c] = 0.0f;
        auto row_barrier = [&] { asm volatile("bar.sync %0, %1;" ::"r"(quad + 1), "n"(kFtParts * 32) : "memory"); };
        auto over_parts = [&](const float (&x)[kFtParts][kFtRows]) { return (x[0][row] + x[1][row]) + (x[2][row] + x[3][row]); };
        // o += weights x values of step i, whose keys begin at j0
        auto take_product = [&](int i, int j0) {
            umma::bar_wait(&bars.o_full, i & 1);
            __syncwarp();
            umma::fence_after_sync();
            const bool sees = j0 <= i_pos && j0 + kFtKeys - 1 > i_pos - win;
            uint32_t v[OC / 8][8];
#pragma unroll
            for (int x = 0; x < OC / 8; ++x) umma::tmem_ld8_issue(tm_o + part * OC + 8 * x + lanes, v[x]);
            umma::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < OC; ++e) o[e] += sees ? __uint_as_float(v[e / 8][e % 8]) : 0.0f;
            umma::fence_before_sync();
        };
        float inv = 0.0f;
        for (int i = 0; i < steps; ++i) {
            const int b = i & 1, map = MAPS == 2 && i >= tiles, jt = j_start + (i - map * tiles) * kFtKeys, j0 = jt + part * kFtCols;
            const bool fresh = i == 0 || (MAPS == 2 && i == tiles);
            umma::bar_wait(&bars.s_full[b], (i >> 1) & 1);
            __syncwarp();
            umma::fence_after_sync();
            float S[kFtCols];
            {
                uint32_t v[kFtCols / 8][8];
#pragma unroll
                for (int x = 0; x < kFtCols / 8; ++x) umma::tmem_ld8_issue(tmem + b * kFtKeys + part * kFtCols + 8 * x + lanes, v[x]);
                umma::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < kFtCols; ++e) S[e] = __uint_as_float(v[e / 8][e % 8]);
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars.s_empty[b]);
            if (MAPS == 2 && i == tiles) {
                // the first map is complete
                take_product(i - 1, j_start + (tiles - 1) * kFtKeys);
                s_sum[0][part][row] = l;
                row_barrier();
                inv = 1.0f / over_parts(s_sum[0]);
#pragma unroll
                for (int c = 0; c < OC; ++c) { first_map[c * (kFtSoftWarps * 32) + threadIdx.x] = o[c] * inv; o[c] = 0.0f; }
                m = sink;
                l = (part == 0 && A.sink) ? 1.0f : 0.0f;
            }
            const bool seen = j0 + kFtCols - 1 <= first_pos && A.window == 0, direct = plain && seen;       // every row of the warp sees every column
            if (!seen) ft_scores_any<true>(A, S, i_pos - j0, win, r1, r2, slope);
            else if (!direct) ft_scores_any<false>(A, S, i_pos - j0, win, r1, r2, slope);
            const float mul = direct ? A.scale * kLog2e : 1.0f;
            s_max[b][part][row] = max_of(S) * mul;
            row_barrier();
            const float mx = fmaxf(fmaxf(s_max[b][0][row], s_max[b][1][row]), fmaxf(s_max[b][2][row], s_max[b][3][row]));
            // without a sink a row of the tile's padding (or outside a window) may have seen no key yet: keep its maximum finite
            const float mn = fmaxf(fmaxf(m, mx), -1e30f), corr = exp2_fast(m - mn);
            m = mn;
            l *= corr;
            uint32_t hi[kFtCols / 2], lo[kFtCols / 2];
            float sums[2] = {0.0f, 0.0f};
#pragma unroll
            for (int e = 0; e < kFtCols / 2; ++e) {
                const float w0 = exp2_fast(fmaf(S[2 * e], mul, -mn)), w1 = exp2_fast(fmaf(S[2 * e + 1], mul, -mn));
                sums[e % 2] += w0 + w1;
                hi[e] = pack_bf16(w0, w1);
                lo[e] = pack_bf16(w0 - bf_lo(hi[e]), w1 - bf_hi(hi[e]));
            }
            l += sums[0] + sums[1];
            if (!fresh) {
                take_product(i - 1, jt - kFtKeys);
#pragma unroll
                for (int c = 0; c < OC; ++c) o[c] *= corr;
            }
            // (the product of the step before is complete: its weights are no longer read)
#pragma unroll
            for (int c = 0; c < kFtCols / 8; ++c) {
                unsigned char* to = Ps + sw128_at(row, part * (kFtCols / 8) + c);
                *reinterpret_cast<uint4*>(to) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                *reinterpret_cast<uint4*>(to + kFtPBytes) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
            }
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars.p_full);
        }
        take_product(steps - 1, j_start + (tiles - 1) * kFtKeys);
        s_sum[1][part][row] = l;
        row_barrier();
        inv = 1.0f / over_parts(s_sum[1]);
        float scale = inv;
        if (MAPS == 2) {
            float ss = 0.0f;
#pragma unroll
            for (int c = 0; c < OC; ++c) {
                o[c] = fmaf(-A.diff_lambda, o[c] * inv, first_map[c * (kFtSoftWarps * 32) + threadIdx.x]);
                ss = fmaf(o[c], o[c], ss);                                      // columns beyond dv hold zeros
            }
            s_max[0][part][row] = ss;
            row_barrier();
            scale = A.diff_scale / sqrtf(over_parts(s_max[0]) / (float)A.dv + A.eps);
        }
        if (row0 + row < n) {
            const size_t t = t0 + row0 + row;
#pragma unroll
            for (int c = 0; c < OC; c += 8) {
                const int col = part * OC + c;
                if (col < A.dv) {
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = o[c + e] * scale * attn_gate(A, t, h, col + e);
                    *reinterpret_cast<uint4*>(out + t * A.out_ld + h * A.dv + col) =
                        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                }
            }
        }
    }
    __syncwarp();
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kFtSoftWarps) umma::tmem_free(tmem);
}

}  // namespace lm
}  // namespace smol
