// The prompt of one sequence: the slow transformer over its positions as one persistent kernel with the same phases and grid barrier as
// decode_kernel.cu.  Included by decode_kernel.cu after rows_phases.cuh and tile_phases.cuh (whose batch attention, split barrier and row
// steps it uses).
//
// A weight phase Y[rows][n_out] = X[rows][K] * W[n_out][K]^T is cut into units (128-row tile, block of `blk` weight rows; wo and
// w2 also into K slices, so that a unit's chain is K = 768 long and the SMs are full); blk is the smallest multiple of 16 that
// gives every CTA at most one unit.  A unit streams its 128 x K activations and blk x K weights through a ring of 64-element
// stages: one thread loads activation boxes, one weight boxes, a warp issues the MMAs and twelve warps read the accumulators.
// Weight boxes of a phase's first stages are issued before the barrier in front of it; everything else about a phase waits.
// K step q of every stage goes to accumulator q, the four are added in fp32: a tensor-memory accumulator drops what lies
// below its last place with every MMA, so chains are kept at 12.
//
// What needs whole rows happens in steps between: the sum of the K slices, the residual add and the next RMSNorm (five rows
// per CTA and pass).  Measured (150m, prompt -> logits, us): 40 positions 623, 212: 706, 800: 1467; one thread that issued
// loads and MMAs, no weights before the barrier, and a slow step behind it for the last position took 917, 1219 and 2017.
#pragma once

namespace smol {

constexpr int kPrStages = 7;                                   // 28 KB each: 128 activation rows + 96 weight rows
constexpr int kPrRing = kPrStages * umma::kStageBytes;
constexpr int kPrEpilogueWarp = 4;                             // first of the warps that read accumulators
constexpr int kPrData = kPrRing > kWarps * kAttnStage ? kPrRing : kWarps * kAttnStage;
// behind the ring: copies of the kernel's arguments.  The last position's products, the attentions and the row steps are functions of their own
// (the weight phases are not: calls, and arguments through a stack that the L1 beside the ring does not hold, cost 5 % of a prompt of 212
// positions, 844 us against 801), and reading an argument through a reference there is a load from the parameter space: several hundred clocks.
constexpr int kPrModel = (sizeof(DevModel) + 127) / 128 * 128, kPrArgs = (sizeof(CallArgs) + 127) / 128 * 128;
constexpr int kPrSmem = kPrData + kPrModel + kPrArgs;
static_assert(kPrSmem <= 226 * 1024, "ring and arguments");

// K slices of wo and w2; their partial sums meet in prompt_finish.
__device__ __forceinline__ int prompt_slices(int K) { return K % (4 * umma::kBK) == 0 ? 4 : K % (2 * umma::kBK) == 0 ? 2 : 1; }

struct PromptBars {
    uint64_t full[kPrStages], empty[kPrStages];   // bytes landed / consumed by the MMAs
    uint64_t acc_full, acc_empty;
    uint32_t tmem_base;
};
__shared__ __align__(8) PromptBars g_pr;

// One MMA / one commit by the warp's elected lane, every lane calling: the operands stay in uniform registers (a single thread's
// loop needs 360 ns for the four MMAs of a stage).
__device__ __forceinline__ void mma_elected(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.u32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
__device__ __forceinline__ void commit_elected(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(umma::s2u(bar)) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::s2u(bar)) : "memory");
}

__device__ __noinline__ void prompt_finish(const DevModel& M, const CallArgs& A, const Ctx& c, const uint16_t* res, uint16_t* dst, int D, int slices, const uint16_t* norm_w, int last_row) {
    tile_finish(M, A, c, res, dst, D, slices, norm_w, last_row);
}

// The last position of a prompt whose logits are wanted, row `row` of the tile: its dot products in the order of the one-row
// kernel (phase_gemv: lane-strided chunks of 8, two chains, a butterfly; slices of 1024 in order), so that the logits of a
// prompt are to the bit those of its last position decoded alone.  The epilogue warps do it while the MMAs run: 5 to 41 weight
// rows per CTA, which the tiles bring into L2 as well.
// Weights of up to two rows of up to 1024 elements (w2: of one row of 3072) wait in registers: they are loaded before the
// barrier in front of the phase.
template <int CH>
__device__ __forceinline__ float row_dot(const uint4 (&wv)[CH], const uint4 (&xv)[CH], int K, int lane) {
    float tot = 0.f;
#pragma unroll
    for (int c0 = 0; c0 < CH; c0 += 4) {      // slices of 1024
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int i = c0; i < CH && i < c0 + 4; ++i) {
            if ((lane + 32 * i) * 8 < K) {
                float wf[8], xf[8];
                unpack8(wv[i], wf); unpack8(xv[i], xf);
#pragma unroll
                for (int e = 0; e < 4; ++e) { a0 = fmaf(wf[e], xf[e], a0); a1 = fmaf(wf[4 + e], xf[4 + e], a1); }
            }
        }
        if (c0 * 256 < K) tot = __fadd_rn(tot, warp_sum(a0 + a1));
    }
    return tot;
}
constexpr int kRowCh = 3, kRowChWide = 12;   // 768 / 256, 3072 / 256
__device__ __forceinline__ void row_fill(const uint16_t* w, int K, int lane, uint4 (&v)[kRowCh]) {
#pragma unroll
    for (int i = 0; i < kRowCh; ++i) v[i] = (lane + 32 * i) * 8 < K ? __ldg(reinterpret_cast<const uint4*>(w) + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ void row_read(const uint16_t* x, int K, int lane, uint4 (&v)[kRowCh]) {
#pragma unroll
    for (int i = 0; i < kRowCh; ++i) v[i] = (lane + 32 * i) * 8 < K ? ldcg_v4(reinterpret_cast<const uint4*>(x) + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
}

// Units of a phase: pairs of wqkv rows, a row of w1 and of w3, a row.
__device__ __forceinline__ int row_units(const DevModel& M, int kind) {
    return kind == PH_QKV ? (M.n_head + 2 * M.n_kv) * kHeadDim / 2 : kind == PH_W13 ? M.inter : kind == PH_HEAD ? M.vocab : M.dim;
}
__device__ __forceinline__ void row_fetch(const DevModel& M, int kind, int layer, int u, int lane, uint4 (&a)[kRowCh], uint4 (&b)[kRowCh]) {
    const DevLayer& L = M.layers[layer];
    const int D = M.dim;
    if (kind == PH_QKV) { row_fill(L.wqkv + (size_t)(2 * u) * D, D, lane, a); row_fill(L.wqkv + (size_t)(2 * u + 1) * D, D, lane, b); }
    else if (kind == PH_W13) { row_fill(L.w1 + (size_t)u * D, D, lane, a); row_fill(L.w3 + (size_t)u * D, D, lane, b); }
    else {
        row_fill((kind == PH_HEAD ? M.head : L.wo) + (size_t)u * D, D, lane, a);
#pragma unroll
        for (int i = 0; i < kRowCh; ++i) b[i] = a[i];
    }
}
__device__ __forceinline__ void row_finish(const DevModel& M, const CallArgs& A, int kind, int layer, int row, int u, int lane, const uint4 (&a)[kRowCh],
                                           const uint4 (&b)[kRowCh], const uint4 (&x)[kRowCh], int pos, int page, uint32_t cs) {
    const int D = M.dim;
    const float va = row_dot<kRowCh>(a, x, D, lane);
    if (kind == PH_HEAD) {
        if (lane == 0) M.token_logits[u] = bf16_round(va);
        return;
    }
    if (kind == PH_WO) {      // the first K slice's partial sum (prompt_finish)
        if (lane == 0) M.kpart[(size_t)row * D + u] = va;
        return;
    }
    const float vb = row_dot<kRowCh>(b, x, D, lane);
    if (lane != 0) return;
    if (kind == PH_W13) {
        const float g = bf16_round(va);
        M.act[(size_t)row * M.inter + u] = f_to_bf(__fmul_rn(bf16_round(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g)))), bf16_round(vb)));
        return;
    }
    const int Hkv = M.n_kv, q_rows = M.n_head * kHeadDim, k_end = q_rows + Hkv * kHeadDim, n0 = 2 * u;
    float v0 = bf16_round(va), v1 = bf16_round(vb);
    if (n0 < k_end) {
        const float co = bf_lo(cs), si = bf_hi(cs);
        const float r0 = bf16_round(__fsub_rn(__fmul_rn(v0, co), __fmul_rn(v1, si)));
        const float r1 = bf16_round(__fadd_rn(__fmul_rn(v1, co), __fmul_rn(v0, si)));
        v0 = r0; v1 = r1;
    }
    if (n0 < q_rows) { *reinterpret_cast<uint32_t*>(M.q + (size_t)row * q_rows + n0) = pack_bf16(v0, v1); return; }
    const int is_v = n0 >= k_end ? 1 : 0, n1 = n0 - (is_v ? k_end : q_rows), ps = M.page_size;
    if (page < 0) return;
    *reinterpret_cast<uint32_t*>(M.kv_pool + ((((size_t)page * M.n_layer + layer) * 2 + is_v) * Hkv + n1 / kHeadDim) * ((size_t)ps * kHeadDim)
                                 + (size_t)(pos % ps) * kHeadDim + (n1 & (kHeadDim - 1))) = pack_bf16(v0, v1);
}

__device__ __forceinline__ void row_prefetch(const DevModel& M, int kind, int layer, int u, int lane) {
    const DevLayer& L = M.layers[layer];
    const int K = kind == PH_W2 ? M.inter : M.dim;
    const uint16_t* p = kind == PH_QKV ? L.wqkv + (size_t)(2 * u) * K : kind == PH_W13 ? L.w1 + (size_t)u * K : (kind == PH_WO ? L.wo : L.w2) + (size_t)u * K;
    const uint16_t* q = kind == PH_QKV ? p + K : kind == PH_W13 ? L.w3 + (size_t)u * K : p;
    for (int e = lane * 64; e < K; e += 32 * 64) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + e));
        if (q != p) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + e));
    }
}
__device__ __noinline__ void row_narrow(const DevModel& M, const CallArgs& A, int kind, int layer, int row, int u, int step, int end, int lane) {
    uint4 x[kRowCh], a[2][kRowCh], b[2][kRowCh];
    row_fetch(M, kind, layer, u, lane, a[0], b[0]);
    row_read((kind == PH_WO ? M.attn : M.xn) + (size_t)row * M.dim, M.dim, lane, x);
    if (u + step < end) row_fetch(M, kind, layer, u + step, lane, a[1], b[1]);      // (a unit's weights are on their way while another is summed)
    int pos = 0, page = -1;
    if (kind == PH_QKV) {
        const int bs = row_seq(A, row);
        pos = ldcg_i32(A.b.seq_len + bs) + row_off(A, row);
        if (pos < A.b.max_pages * M.page_size) page = ldcg_i32(A.b.block_table + (size_t)bs * A.b.max_pages + pos / M.page_size);
    }
    const uint16_t* rope = M.rope + (size_t)min(pos, M.max_seq_len - 1) * kHeadDim;
    for (; u < end; u += 2 * step) {
        uint32_t cs = 0u;
        if (kind == PH_QKV) cs = __ldg(reinterpret_cast<const uint32_t*>(rope + ((2 * u) & (kHeadDim - 1))));
        row_finish(M, A, kind, layer, row, u, lane, a[0], b[0], x, pos, page, cs);
        if (u + step >= end) return;
        if (u + 2 * step < end) row_fetch(M, kind, layer, u + 2 * step, lane, a[0], b[0]);
        if (kind == PH_QKV) cs = __ldg(reinterpret_cast<const uint32_t*>(rope + ((2 * (u + step)) & (kHeadDim - 1))));
        row_finish(M, A, kind, layer, row, u + step, lane, a[1], b[1], x, pos, page, cs);
        if (u + 3 * step < end) row_fetch(M, kind, layer, u + 3 * step, lane, a[1], b[1]);
    }
}
__device__ __noinline__ void row_wide(const DevModel& M, int row, int layer, int u, int step, int end, int lane) {
    const int F = M.inter;
    const uint4* xp = reinterpret_cast<const uint4*>(M.act + (size_t)row * F);
    for (; u < end; u += step) {
        uint4 x[kRowChWide], w[kRowChWide];
        const uint4* wp = reinterpret_cast<const uint4*>(M.layers[layer].w2 + (size_t)u * F);
#pragma unroll
        for (int i = 0; i < kRowChWide; ++i) {
            const bool in = (lane + 32 * i) * 8 < F;
            w[i] = in ? __ldg(wp + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
            x[i] = in ? ldcg_v4(xp + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
        }
        const float v = row_dot<kRowChWide>(w, x, F, lane);
        if (lane == 0) M.kpart[(size_t)row * M.dim + u] = v;
    }
}

// One weight phase; on return the CTA has finished its units, the barrier behind it is the caller's.
template <bool kTimed>
__device__ __forceinline__ void prompt_gemm(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, RowsSync& sy, uint32_t& chunk, uint32_t& tile, const int last_row) {
    const int kind = ph.kind;
    const int D = M.dim, F = M.inter, Hq = M.n_head, Hkv = M.n_kv;
    const int q_rows = Hq * kHeadDim, k_end = (Hq + Hkv) * kHeadDim;
    const int K = kind == PH_W2 ? F : D;
    const int n_out = kind == PH_QKV ? (Hq + 2 * Hkv) * kHeadDim : kind == PH_W13 ? F : D;
    const int rows = A.batch;
    unsigned char* ring = reinterpret_cast<unsigned char*>(c.xs);
    const int warp = c.warp, lane = c.lane;

    const unsigned char* tm = M.tmaps;
    const int box_idx = rows <= 32 ? 2 : rows <= 64 ? 1 : 0;   // activation box of 32 / 64 / 128 rows: the rest of a stage holds stale rows whose accumulator lanes nobody reads
    const int a_bytes = (umma::kM >> box_idx) * umma::kBK * 2;
    const void* tm_a = tm + (size_t)kTensorMapBytes * (box_idx * TM_ACT_MAPS + (kind == PH_WO ? TM_ATTN : kind == PH_W2 ? TM_ACT : TM_XN));
    const int which = kind == PH_QKV ? 0 : kind == PH_WO ? 1 : kind == PH_W13 ? 2 : 4;
    const int w0 = tm_weight_index(ph.layer, which), w1 = tm_weight_index(ph.layer, 3);
    const bool paired = kind == PH_W13;
    const int n_split = kind != PH_WO && kind != PH_W2 ? 1 : prompt_slices(K);
    const int nk = K / n_split / umma::kBK;
    const int m_tiles = (rows + umma::kM - 1) / umma::kM, cap = paired ? umma::kMaxN / 2 : umma::kMaxN;
    int blk = 16;
    while (blk < cap && m_tiles * ((n_out + blk - 1) / blk) * n_split > c.n_ctas) blk += 16;
    const int n_units = m_tiles * ((n_out + blk - 1) / blk) * n_split, n_blk = paired ? 2 * blk : blk;
    const int my_units = n_units > c.cta ? (n_units - 1 - c.cta) / c.n_ctas + 1 : 0;
    // unit u: row tile (those that share a weight block run on neighbouring CTAs), K slice, weight block
    auto place = [&](int u, int& m0, int& ks, int& n0) {
        m0 = (u % m_tiles) * umma::kM;
        const int r = u / m_tiles;
        ks = r % n_split;
        n0 = (r / n_split) * blk;
    };
    auto load_w = [&](uint32_t g, int n0, int k0) {
        const uint32_t s = g % kPrStages, b = umma::s2u(ring + (size_t)s * umma::kStageBytes) + umma::kStageA;
        umma::bar_expect_tx(&g_pr.full[s], (uint32_t)(n_blk * umma::kBK * 2));
        umma::tma_load_2d(b, tm + (size_t)kTensorMapBytes * tm_weight_slot(w0, blk), k0, n0, &g_pr.full[s]);
        if (paired) umma::tma_load_2d(b + blk * umma::kBK * 2, tm + (size_t)kTensorMapBytes * tm_weight_slot(w1, blk), k0, n0, &g_pr.full[s]);
    };
    // the first stages' weights do not wait for the phase before (the ring is empty: that phase's accumulators have been read)
    const int early = my_units ? min(nk, kPrStages) : 0;
    if (warp == 2 && lane == 0 && early) {
        int m0, ks, n0;
        place(c.cta, m0, ks, n0);
        for (int kc = 0; kc < early; ++kc) load_w(chunk + kc, n0, (ks * nk + kc) * umma::kBK);
    }
    // (the last row's weights neither: into L2)
    const bool dots = last_row >= 0 && warp >= kPrEpilogueWarp;
    const int u_first = dots ? (warp - kPrEpilogueWarp) * c.n_ctas + c.cta : 0, u_step = (kWarps - kPrEpilogueWarp) * c.n_ctas, u_end = dots ? row_units(M, kind) : 0;
    for (int u = u_first; u < u_end; u += u_step) row_prefetch(M, kind, ph.layer, u, lane);
    rows_sync_in<kTimed>(M, sy);
    if (warp == 0 && lane == 0) {
        fence_proxy_async_global();      // rows written by st.global in other CTAs
        uint32_t g = chunk;
        for (int u = c.cta; u < n_units; u += c.n_ctas) {
            int m0, ks, n0;
            place(u, m0, ks, n0);
            for (int kc = 0; kc < nk; ++kc, ++g) {
                const uint32_t s = g % kPrStages;
                if (g >= (uint32_t)kPrStages) umma::bar_wait(&g_pr.empty[s], (g / kPrStages - 1u) & 1u);
                umma::bar_expect_tx(&g_pr.full[s], (uint32_t)a_bytes);
                umma::tma_load_2d(umma::s2u(ring + (size_t)s * umma::kStageBytes), tm_a, (ks * nk + kc) * umma::kBK, m0, &g_pr.full[s]);
            }
        }
    } else if (warp == 2 && lane == 0) {
        uint32_t g = chunk;
        for (int u = c.cta; u < n_units; u += c.n_ctas) {
            int m0, ks, n0;
            place(u, m0, ks, n0);
            for (int kc = 0; kc < nk; ++kc, ++g) {
                if (u == c.cta && kc < early) continue;
                if (g >= (uint32_t)kPrStages) umma::bar_wait(&g_pr.empty[g % kPrStages], (g / kPrStages - 1u) & 1u);
                load_w(g, n0, (ks * nk + kc) * umma::kBK);
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma::instr_desc(n_blk), tmem = g_pr.tmem_base;
        uint32_t g = chunk, t = tile;
        for (int i = 0; i < my_units; ++i, ++t) {
            if (t > 0) umma::bar_wait(&g_pr.acc_empty, (t - 1u) & 1u);
            umma::fence_after_sync();
            for (int kc = 0; kc < nk; ++kc, ++g) {
                const uint32_t s = g % kPrStages;
                umma::bar_wait(&g_pr.full[s], (g / kPrStages) & 1u);
                umma::fence_after_sync();
                const uint32_t a = umma::s2u(ring + (size_t)s * umma::kStageBytes);
                const uint64_t da = umma::smem_desc_sw128(a), db = umma::smem_desc_sw128(a + umma::kStageA);
#pragma unroll
                for (int q = 0; q < umma::kAcc; ++q) mma_elected(tmem + (uint32_t)(q * n_blk), da + q * 2, db + q * 2, idesc, (uint32_t)kc);
                commit_elected(&g_pr.empty[s]);
            }
            commit_elected(&g_pr.acc_full);
        }
    } else if (warp >= kPrEpilogueWarp) {
        const int quad = warp & 3, part = (warp >> 2) - 1;
        constexpr int kParts = kWarps / 4 - 1;
        const uint32_t base = g_pr.tmem_base + ((uint32_t)(quad * 32) << 16);
        uint32_t t = tile;
        const bool prof = kTimed && c.cta == 0 && c.tid == kPrEpilogueWarp * 32;   // segments: last position | copies and MMAs | accumulators
        unsigned long long stamp = 0ull;
        if (prof) stamp = globaltimer_ns();
        if (u_first < u_end) {
            if (kind == PH_W2) row_wide(M, last_row, ph.layer, u_first, u_step, u_end, lane);
            else row_narrow(M, A, kind, ph.layer, last_row, u_first, u_step, u_end, lane);
        }
        __syncwarp();
        if (prof) rows_stamp(M, kind, ph.fast, 1, stamp);
        for (int u = c.cta; u < n_units; u += c.n_ctas, ++t) {
            int m0, ks, n0;
            place(u, m0, ks, n0);
            const int bg = m0 + quad * 32 + lane;
            const bool live = bg < rows && bg != last_row;
            int pos = 0, page = -1;
            if (kind == PH_QKV && live) {      // cache slot of the row (-1: nothing is appended)
                const int bs = row_seq(A, bg);
                pos = ldcg_i32(A.b.seq_len + bs) + row_off(A, bg);
                if (seq_active(M, A, c, bg) && pos < A.b.max_pages * M.page_size) page = ldcg_i32(A.b.block_table + (size_t)bs * A.b.max_pages + pos / M.page_size);
            }
            umma::bar_wait(&g_pr.acc_full, t & 1u);
            __syncwarp();
            umma::fence_after_sync();
            if (prof) rows_stamp(M, kind, ph.fast, 2, stamp);
            for (int cg = part; cg * 8 < blk; cg += kParts) {
                float acc[8], up[8];
                __syncwarp();
                if (paired) umma::tmem_ld8_sum2(base + (uint32_t)(cg * 8), base + (uint32_t)(blk + cg * 8), n_blk, acc, up);
                else umma::tmem_ld8_sum(base + (uint32_t)(cg * 8), n_blk, acc);
                const int u0 = n0 + cg * 8;
                if (!live || u0 >= n_out) continue;
                if (paired) {
                    float o[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {   // F.silu in fp32, bf16 out: the exactly rounded result from the table over all bf16 arguments
                        const float sg = bf_to_f(__ldg(M.silu_lut + f_to_bf(acc[e])));
                        o[e] = __fmul_rn(sg, bf16_round(up[e]));
                    }
                    *reinterpret_cast<uint4*>(M.act + (size_t)bg * F + u0) = pack8(o);
                    continue;
                }
                if (kind != PH_QKV) {
                    float* pp = M.kpart + ((size_t)ks * M.ws_rows + bg) * D + u0;
                    *reinterpret_cast<float4*>(pp) = make_float4(acc[0], acc[1], acc[2], acc[3]);
                    *reinterpret_cast<float4*>(pp + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
                    continue;
                }
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = bf16_round(acc[e]);
                if (u0 < k_end) {  // q and k rows: interleaved-pair RoPE with the bf16 table (P:616-640); never past the table (host checks bound pos)
                    const uint4 cs = __ldg(reinterpret_cast<const uint4*>(M.rope + (size_t)min(pos, M.max_seq_len - 1) * kHeadDim + (u0 & (kHeadDim - 1))));
                    const uint32_t cw[4] = {cs.x, cs.y, cs.z, cs.w};
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const float co = bf_lo(cw[e >> 1]), si = bf_hi(cw[e >> 1]);
                        const float r0 = bf16_round(__fsub_rn(__fmul_rn(v[e], co), __fmul_rn(v[e + 1], si)));
                        const float r1 = bf16_round(__fadd_rn(__fmul_rn(v[e + 1], co), __fmul_rn(v[e], si)));
                        v[e] = r0; v[e + 1] = r1;
                    }
                }
                if (u0 < q_rows) { *reinterpret_cast<uint4*>(M.q + (size_t)bg * q_rows + u0) = pack8(v); continue; }
                const int is_v = u0 >= k_end ? 1 : 0, n1 = u0 - (is_v ? k_end : q_rows), ps = M.page_size;
                if (page < 0) continue;
                *reinterpret_cast<uint4*>(M.kv_pool + ((((size_t)page * M.n_layer + ph.layer) * 2 + is_v) * Hkv + n1 / kHeadDim) * ((size_t)ps * kHeadDim)
                                          + (size_t)(pos % ps) * kHeadDim + (n1 & (kHeadDim - 1))) = pack8(v);
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&g_pr.acc_empty);
            if (prof) rows_stamp(M, kind, ph.fast, 3, stamp);
        }
    }
    __syncwarp();
    __syncthreads();
    chunk += (uint32_t)(my_units * nk);
    tile += (uint32_t)my_units;
}

template <bool kTimed>
__device__ __noinline__ void prompt_attn_rows(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, RowsSync& sy, const void* kv_map, int last_row) { phase_attn_batch<true, kTimed>(M, A, c, ph, sy, kv_map, last_row); }
__device__ __noinline__ void prompt_attn_alone(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, int splits, int row) { phase_attn_g(M, A, c, ph, splits, row, 1); }
template <bool kTimed>
__device__ __forceinline__ void prompt_attn(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, RowsSync& sy, const void* kv_map, int last_row) {
    if (last_row < 0) {
        prompt_attn_rows<kTimed>(M, A, c, ph, sy, kv_map, -1);
        return;
    }
    // the last row as decoded alone, on a few CTAs of its own
    const int ns = min((ldcg_i32(A.b.seq_len + row_seq(A, last_row)) + row_off(A, last_row)) / kSplitMin + 1, kMaxSplits);
    const int n_alone = min(min(M.n_kv * ns, 20), c.n_ctas / 4);
    Ctx cs = c;
    cs.n_ctas = c.n_ctas - n_alone;
    if (c.cta < cs.n_ctas) prompt_attn_rows<kTimed>(M, A, cs, ph, sy, kv_map, last_row);
    if (c.cta >= cs.n_ctas || n_alone == 0) {
        cs.cta = c.cta - (n_alone ? cs.n_ctas : 0);
        cs.n_ctas = n_alone ? n_alone : c.n_ctas;
        __syncthreads();
        prompt_attn_alone(M, A, cs, ph, ns, last_row);
    }
}

// What the kernel begins with: the arguments' copies, barriers, tensor memory.
__device__ __forceinline__ void prompt_setup(const DevModel& Mp, const CallArgs& Ap, unsigned char* smem_dyn, Ctx& c, RowsSync& sy) {
    for (int i = threadIdx.x; i < (int)(sizeof(DevModel) / 4); i += kThreads) reinterpret_cast<uint32_t*>(smem_dyn + kPrData)[i] = reinterpret_cast<const uint32_t*>(&Mp)[i];
    for (int i = threadIdx.x; i < (int)(sizeof(CallArgs) / 4); i += kThreads) reinterpret_cast<uint32_t*>(smem_dyn + kPrData + kPrModel)[i] = reinterpret_cast<const uint32_t*>(&Ap)[i];
    c.cta = blockIdx.x; c.n_ctas = gridDim.x; c.tid = threadIdx.x;
    c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31;
    c.xs = reinterpret_cast<float*>(smem_dyn);
    c.stage = smem_dyn;
    c.iter = 0;
    if (c.tid == 0) {
        for (int s = 0; s < kPrStages; ++s) { mbar_init(&g_pr.full[s], 2u); mbar_init(&g_pr.empty[s], 1u); }
        mbar_init(&g_pr.acc_full, 1u);
        mbar_init(&g_pr.acc_empty, (uint32_t)(kWarps - kPrEpilogueWarp));
        for (int i = 0; i < 2 * kWarps; ++i) { mbar_init(&g_kvbar[i], 1u); g_kvpar[i] = 0u; }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        g_gave_up = 0u;
    }
    if (c.warp == 0) umma::tmem_alloc(&g_pr.tmem_base);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    sy.target = ldcg_u32(Mp.barrier + 1); sy.par_w = 0; sy.par_x = 0; sy.pending = false; sy.failed = false; sy.phase = 0; sy.next = -1; sy.waits_for = 0;
}

// The phase recorder (thread 0 of CTA 0, profiling builds): a phase's time without its waits (rows_sync_in takes them off), the
// arrival behind it, and the row steps around its tiles as segment 0.
template <bool kTimed>
struct PhaseTimer {
    bool on;
    unsigned long long t0, t1, ts;
    __device__ __forceinline__ explicit PhaseTimer(const Ctx& c) : on(kTimed && c.cta == 0 && c.tid == 0) { if (on) t0 = globaltimer_ns(); }
    __device__ __forceinline__ void rest() { if (on) ts = globaltimer_ns(); }
    __device__ __forceinline__ void step(const DevModel& M, const Phase& ph) { if (on) rows_stamp(M, ph.kind, ph.fast, 0, ts); }
    __device__ __forceinline__ void end(const DevModel& M, int p) { if (on) { t1 = globaltimer_ns(); M.prof[2 * p] += t1 - t0; } }
    __device__ __forceinline__ void arrived(const DevModel& M, int p) { if (on) { t0 = globaltimer_ns(); M.prof[2 * p + 1] += t0 - t1; } }
};

template <bool kTimed>
__global__ void __launch_bounds__(kThreads, 1)
smol_prompt_kernel(const __grid_constant__ DevModel Mp, const __grid_constant__ CallArgs Ap) {
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    const DevModel& M = *reinterpret_cast<const DevModel*>(smem_dyn + kPrData);
    const CallArgs& A = *reinterpret_cast<const CallArgs*>(smem_dyn + kPrData + kPrModel);
    Ctx c;
    RowsSync sy;
    prompt_setup(Mp, Ap, smem_dyn, c, sy);
    uint32_t chunk = 0, tile = 0;
    if (A.wait_probe && c.cta == 0 && c.tid == 0) rows_wait(M, &g_kvbar[2 * kWarps - 1], 0u);   // (nothing completes it)
    for (int it = 0; it < A.n_iter && !sy.failed; ++it) {
        c.iter = it;
        const bool last_iter = it == A.n_iter - 1;
        const int last_row = last_iter && A.whole_prompt > 0 ? A.head_row : -1;
        if (kTimed) sy.phase = 0;
        PhaseTimer<kTimed> timer(c);
        rows_sync_in<kTimed>(M, sy);
        timer.rest();
        tile_row_step(M, A, c, M.dim, M.x, M.layers[0].attention_norm, [&](int bg, int ch, float (&x)[8]) { embed_chunk(M, A, c, bg, ch, x); });
        timer.step(M, unpack_phase(M.prog[0]));
        rows_arrive<kTimed>(M, c, sy);
        for (int p = 0; p < phases_per_prefill_step(M.n_layer) && !sy.failed; ++p) {
            const Phase ph = unpack_phase(M.prog[p]);
            if (kTimed) sy.phase = p;
            if (ph.kind == PH_ATTN) {
                rows_sync_in<kTimed>(M, sy);
                prompt_attn<kTimed>(M, A, c, ph, sy, Ap.kv_map, last_row);
            } else {
                prompt_gemm<kTimed>(M, A, c, ph, sy, chunk, tile, last_row);
                if (ph.kind == PH_WO || ph.kind == PH_W2) {   // h = stream + wo(attn) (P:499); stream = h + w2(act) (P:500); and the norm of the phase that reads it
                    rows_arrive<kTimed>(M, c, sy);
                    rows_sync_in<kTimed>(M, sy);
                    timer.rest();
                    const bool wo = ph.kind == PH_WO;
                    const uint16_t* norm = wo ? M.layers[ph.layer].ffn_norm : ph.layer + 1 < M.n_layer ? M.layers[ph.layer + 1].attention_norm : M.norm;
                    prompt_finish(M, A, c, wo ? M.x : M.h, wo ? M.h : M.x, M.dim, prompt_slices(wo ? M.dim : M.inter), norm, last_row);
                    timer.step(M, ph);
                }
            }
            if (p == phases_per_prefill_step(M.n_layer) - 1 && c.cta == 0) {
                // every sequence advances by the positions of this tile that lie inside its prompt
                const int T = A.tile_t > 1 ? A.tile_t : 1;
                for (int b = c.tid; b < A.real_batch; b += kThreads) {
                    int n_act = prompt_positions(A, b) - (A.iter_base + it * T);
                    n_act = n_act < 0 ? 0 : (n_act > T ? T : n_act);
                    if (n_act) A.b.seq_len[b] = ldcg_i32(A.b.seq_len + b) + n_act;
                }
            }
            timer.end(M, p);
            if (!sy.failed && !(last_iter && A.whole_prompt == 0 && p == phases_per_prefill_step(M.n_layer) - 1)) rows_arrive<kTimed>(M, c, sy);
            timer.arrived(M, p);
        }
    }
    if (A.whole_prompt > 0 && !sy.failed) {
        if (kTimed) sy.phase = 5 * M.n_layer;        // the LM head's
        PhaseTimer<kTimed> timer(c);
        rows_sync_in<kTimed>(M, sy);
        if (c.cta == 0 && A.head_row > 0)      // the last position's hidden state (pre-norm) -> row 0
            for (int i = c.tid; i < M.dim / 8; i += kThreads) *reinterpret_cast<uint4*>(M.x + i * 8) = ldcg_v4(M.x + (size_t)A.head_row * M.dim + i * 8);
        uint4 x[kRowCh], w[kRowCh];
        row_read(M.xn + (size_t)A.head_row * M.dim, M.dim, c.lane, x);
        for (int u = c.warp * c.n_ctas + c.cta; u < M.vocab; u += kWarps * c.n_ctas) {
            row_fetch(M, PH_HEAD, 0, u, c.lane, w, w);
            row_finish(M, A, PH_HEAD, 0, A.head_row, u, c.lane, w, w, x, 0, -1, 0u);
        }
        timer.end(M, 5 * M.n_layer);
    }
    if (c.cta == 0 && !sy.failed) {
        // leave the last prompt column as the pending input of the first decode frame (G:66-73)
        for (int i = c.tid; i < A.real_batch * M.n_rows; i += kThreads) {
            const int b = i / M.n_rows, r = i - b * M.n_rows;
            A.b.tokens[i] = ldcg_i32(A.prompt + ((size_t)b * M.n_rows + r) * A.s_max + prompt_last(A, b));
        }
        if (c.tid == 0) M.barrier[1] = sy.target;
    }
    umma::fence_before_sync();
    __syncthreads();
    if (c.warp == 0) umma::tmem_free(g_pr.tmem_base);
}

}  // namespace smol
