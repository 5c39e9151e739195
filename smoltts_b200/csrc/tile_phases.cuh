// The batched engine on 128-row tiles: the weight phases of decode_kernel.cu as tcgen05 tiles (umma.cuh) for frames of more sequences than
// rows_phases.cuh takes, and for prompts of many sequences or few positions, plus the batch forms of the two attentions.
// Included by decode_kernel.cu (uses its Ctx, grid barrier, embedding and row bookkeeping helpers).
//
// A weight phase Y[rows][n_out] = f(X)[rows][K] * W[n_out][K]^T is cut into units (128-row tile, block of `blk` weight rows; wo and w2 also
// into K slices); blk is the smallest multiple of 16 that gives every CTA at most one unit.  A unit streams its 128 x K activation
// tile and blk x K weight rows through a ring of TMA copies in 64-element stages; what needs whole rows (embedding, RMSNorm, depth
// attention, sums of K slices) happens in row steps between grid barriers, the epilogues (RoPE + KV append, silu * up, logits) read the fp32
// accumulator from TMEM.  Same rounding points as the GEMV kernels (bf16 after every Linear / norm stage / RoPE / silu / product /
// residual add); the sums are in rows_phases.cuh's order and round alike, so a row's bits are the same in both.
// A frame is bound by its 380 barriers and row steps, hardly by its rows: 160 / 256 sequences (150m, caches of <= 100 positions) take 2361 /
// 2435 us.  The same tiles with rows_phases.cuh's split barrier and attention, and the phases as functions: 2631 / 2686 (calls that save
// registers to stacks which the L1 beside 227 KB of shared memory does not hold, and four warps per attention unit of one split).
#pragma once

namespace smol {

__device__ void phase_sample(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, bool feed = false);

// Row steps of the tensor-core variant (pre-step of a normed phase, post-step of a split-K phase).  Three warps per row
// (one 16-byte chunk per lane: every load of a row is in flight at once), five rows per CTA and pass, rows spread over
// the grid.  load(bg, ch, x) produces chunk ch of row bg; the row goes to `raw` (if any) as it is and, if norm_w is given,
// through RMSNorm (P:601-613: fp32 normalise, round to bf16, multiply by the bf16 weight, round again) to M.xn.
constexpr int kRowWarps = 3;
constexpr int kRowsPerPass = kWarps / kRowWarps;

template <class Load>
__device__ __forceinline__ void tile_row_step(const DevModel& M, const CallArgs& A, const Ctx& c, int D, uint16_t* raw,
                                            const uint16_t* norm_w, Load load) {
    const int nch = D >> 3;
    const int slot = c.warp / kRowWarps, wi = c.warp - slot * kRowWarps;
    const int ch = wi * 32 + c.lane;
    for (int row0 = c.cta * kRowsPerPass; row0 < A.batch; row0 += c.n_ctas * kRowsPerPass) {
        const int bg = row0 + slot;
        const bool act = slot < kRowsPerPass && bg < A.batch && ch < nch;
        float x[8];
        float ss = 0.f;
        uint4 wv = make_uint4(0u, 0u, 0u, 0u);
        if (act) {
            if (norm_w != nullptr) wv = __ldg(reinterpret_cast<const uint4*>(norm_w + ch * 8));
            load(bg, ch, x);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss = fmaf(x[e], x[e], ss);
        }
        ss = warp_sum(ss);
        if (c.lane == 0) g_part[c.warp] = ss;
        __syncthreads();
        if (act) {
            if (raw != nullptr) *reinterpret_cast<uint4*>(raw + (size_t)bg * D + ch * 8) = pack8(x);
            if (norm_w != nullptr) {
                float t = 0.f;
                for (int i = 0; i < kRowWarps; ++i) t += g_part[slot * kRowWarps + i];
                const float mean = __fdiv_rn(t, (float)D);
                const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, M.eps)));
                float wf[8], o[8];
                unpack8(wv, wf);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(bf16_round(__fmul_rn(x[e], r)), wf[e]);
                *reinterpret_cast<uint4*>(M.xn + (size_t)bg * D + ch * 8) = pack8(o);
            }
        }
        __syncthreads();
    }
}

// Input pre-step of a normed weight phase: gather the row (token embedding P:205-221, the slow hidden state or the
// previous depth code's embedding G:136-140, or a residual stream), keep the raw row as the residual stream where the
// phase starts one (`spill`), and write RMSNorm(row) to M.xn, which the phase's tiles read through TMA.
// src_kind: 0 token embedding, 1 slow hidden state, 2 embedding of the previous depth code, 3 `base` rows.
__device__ void tile_norm_rows(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, int src_kind,
                             const uint16_t* base, uint16_t* spill, const uint16_t* norm_w, int D) {
    tile_row_step(M, A, c, D, spill, norm_w, [&](int bg, int ch, float (&x)[8]) {
        if (src_kind == 0) { embed_chunk(M, A, c, bg, ch, x); return; }
        const uint16_t* src = base + (size_t)bg * D;
        if (src_kind == 1) {
            src = M.x + (size_t)bg * D;
        } else if (src_kind == 2) {
            const int code = ldcg_i32(M.frame_tokens + (size_t)bg * M.n_rows + ph.depth_pos);
            const int off = M.depthwise_wte ? (M.dup0 ? ph.depth_pos - 1 : ph.depth_pos) * M.codebook_size : 0;
            src = M.fast_embeddings + (size_t)(code + off) * D;
        }
        unpack8(ldcg_v4(src + ch * 8), x);
    });
}

// Post-step of the phases whose K is cut (wo, w2): dst = res + bf16(sum of the K slices' partial sums, in slice order): the Linear's bf16 output plus the residual (P:499-500)
// -- and, when the next phase of the launch is the normed phase that reads dst (w13 after wo; the next layer's QKV or the head after w2), its
// RMSNorm into M.xn.  Row last_row (a prompt's last position, whose dot products are not cut) has one partial sum.
__device__ __forceinline__ void tile_finish(const DevModel& M, const CallArgs& A, const Ctx& c, const uint16_t* res, uint16_t* dst, int D, int slices, const uint16_t* norm_w,
                                            const int last_row = -1) {
    tile_row_step(M, A, c, D, dst, norm_w, [&](int bg, int ch, float (&x)[8]) {
        const int n_split = bg == last_row ? 1 : slices;
        const uint4 rv = ldcg_v4(res + (size_t)bg * D + ch * 8);
        float4 pa[kTcKSplit], pb[kTcKSplit];
#pragma unroll
        for (int sp = 0; sp < kTcKSplit; ++sp) {
            const float* pp = M.kpart + ((size_t)min(sp, n_split - 1) * M.ws_rows + bg) * D + ch * 8;
            pa[sp] = __ldcg(reinterpret_cast<const float4*>(pp));
            pb[sp] = __ldcg(reinterpret_cast<const float4*>(pp + 4));
        }
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int sp = 0; sp < kTcKSplit; ++sp) {
            if (sp < n_split) {
                acc[0] = __fadd_rn(acc[0], pa[sp].x); acc[1] = __fadd_rn(acc[1], pa[sp].y);
                acc[2] = __fadd_rn(acc[2], pa[sp].z); acc[3] = __fadd_rn(acc[3], pa[sp].w);
                acc[4] = __fadd_rn(acc[4], pb[sp].x); acc[5] = __fadd_rn(acc[5], pb[sp].y);
                acc[6] = __fadd_rn(acc[6], pb[sp].z); acc[7] = __fadd_rn(acc[7], pb[sp].w);
            }
        }
        float rf[8];
        unpack8(rv, rf);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = bf16_round(__fadd_rn(rf[e], bf16_round(acc[e])));
    });
}

// Attention of the depth transformer for every (row, head) of the batch, one warp per pair, spread over the grid; the result goes to M.attn
// (the wo tiles read it after a grid barrier).
__device__ __forceinline__ void tile_depth_attention(const DevModel& M, const CallArgs& A, const Ctx& c, int layer, int depth_pos) {
    const int Hq = M.fn_head, Hkv = M.fn_kv, G = Hq / Hkv, D = M.fdim, kvw = Hkv * kHeadDim;
    for (int pair = c.cta * kWarps + c.warp; pair < A.batch * Hq; pair += c.n_ctas * kWarps) {
        const int bg = pair / Hq, hq = pair - bg * Hq, kvh = hq / G;
        const uint16_t* qp = M.q + (size_t)bg * Hq * kHeadDim + hq * kHeadDim + (c.lane & 3) * 16;
        const uint16_t* kp = M.fkv + ((size_t)(bg * M.n_flayer + layer) * 2) * M.depth * kvw + kvh * kHeadDim;
        uint32_t* dst = reinterpret_cast<uint32_t*>(M.attn + (size_t)bg * D + hq * kHeadDim + 2 * c.lane);
        const uint4 q[2] = {ldcg_v4(qp), ldcg_v4(qp + 8)};    // every load of the pair is issued before the first use
        if (depth_pos < 8) {
            uint4 k[1][2];
            uint32_t v[8];
            depth_load<false>(kp, kvw, M.depth, depth_pos, c.lane, k, v);
            *dst = depth_head<false>(q, k, v, depth_pos, c.lane);
        } else {
            uint4 k[2][2];
            uint32_t v[16];
            depth_load<true>(kp, kvw, M.depth, depth_pos, c.lane, k, v);
            *dst = depth_head<true>(q, k, v, depth_pos, c.lane);
        }
    }
}

// Decode / prefill attention over the paged cache for a batch.  Unit = one WARP per (query group, kv head, split); a
// query group is one decode row, or up to 16/G consecutive prompt positions of one sequence.  Per 16 cached positions:
// S = Q K^T (2 n-tiles x 4 k-steps), online softmax in base 2 with P rounded to bf16 for the PV product as the reference's
// SDPA does (P:559-566; the denominator sums the unrounded fp32 values), O += P V (8 n-tiles).  K, V and Q fragments are
// loaded straight from global memory with 16-byte loads: the k index of the QK product and the n index of the PV product
// are permuted so that every thread's fragment words are contiguous in memory (a dot product does not care about the
// order of its dims as long as both operands use the same one).
// Splits of a long row meet through M.partial / M.split_count; the last arriver combines them in split order.
__device__ __forceinline__ void tile_attn(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph) {
    const int Hq = M.n_head, Hkv = M.n_kv, ps = M.page_size, G = Hq / Hkv;
    const int cap = A.b.max_pages * ps;
    const int T = A.tile_t > 1 ? A.tile_t : 1;
    const int P = T > 1 ? 16 / G : 1;              // query positions per unit
    const int gps = (T + P - 1) / P;               // units (groups) per sequence
    const int n_groups = (A.batch / T) * gps;
    const int gq = c.lane >> 2, tq = c.lane & 3;   // fragment coordinates of this lane
    // splits to enumerate: enough for the longest row of the batch (one pass over seq_len; rows with fewer splits skip)
    if (c.tid == 0) g_flag = 1;
    __syncthreads();
    {
        int lmax = 1;
        for (int b = c.tid; b < A.batch; b += kThreads) lmax = max(lmax, ldcg_i32(A.b.seq_len + row_seq(A, b)) + row_off(A, b) + 1);
        lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, 16));
        lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, 8));
        lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, 4));
        lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, 2));
        lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, 1));
        if (c.lane == 0) atomicMax(&g_flag, lmax);
    }
    __syncthreads();
    const SplitPlan sp = split_plan(A, cap);
    const int s_cap = min(sp.count(min(g_flag, cap)), kMaxSplits);
    const int n_tasks = n_groups * Hkv * s_cap;
    const size_t head_stride = (size_t)ps * kHeadDim;
    const size_t page_stride = (size_t)M.n_layer * 2 * Hkv * head_stride;
    constexpr float kScale = 0.125f * 1.4426950408889634f;   // 1/sqrt(64) * log2(e): softmax in base 2

    for (int t = c.cta * kWarps + c.warp; t < n_tasks; t += c.n_ctas * kWarps) {
        const int s = t % s_cap, kvh = (t / s_cap) % Hkv, grp = t / (s_cap * Hkv);
        const int b0 = (grp / gps) * T + (grp % gps) * P;            // first batch row of the group
        const int nq = min(P, T - (grp % gps) * P);                   // its live query positions
        const int bs = row_seq(A, b0);
        const int len0 = ldcg_i32(A.b.seq_len + bs);
        const int L0 = len0 + row_off(A, b0) + 1;                     // context of the first row (its own position included)
        const int Lg = min(L0 + nq - 1, cap);                         // ... of the last one
        const int p0 = sp.lo(s);
        if (p0 >= Lg) continue;
        // cached positions that hold data: everything up to the group's last ACTIVE row (rows past the end of a prompt do
        // not append; their stale slots must not reach the PV product of the active rows as 0 x garbage)
        int Lload = Lg;
        if (A.mode == 1) {
            const int act = prompt_positions(A, bs) - (A.iter_base + c.iter * T);
            Lload = min(Lg, len0 + max(0, min(act, T)));
        }
        const int p1 = min(Lg, sp.lo(s + 1));
        const int pl = min(p1, Lload);
        // the two query rows of this lane: row r = (query position r / G, head r % G)
        const int ra = gq, rb = gq + 8;
        const int ia = ra / G, ib = rb / G;
        const bool va = ia < nq, vb = ib < nq;
        const int La = min(L0 + ia, cap), Lb = min(L0 + ib, cap);     // causal limits (positions < L are visible)
        uint32_t qa[4][4];
        {
            const uint4 z = make_uint4(0u, 0u, 0u, 0u);
            const uint16_t* qpa = M.q + ((size_t)(b0 + ia) * Hq + kvh * G + (ra - ia * G)) * kHeadDim + tq * 8;
            const uint16_t* qpb = M.q + ((size_t)(b0 + ib) * Hq + kvh * G + (rb - ib * G)) * kHeadDim + tq * 8;
            const uint4 a0 = va ? ldcg_v4(qpa) : z, a1 = va ? ldcg_v4(qpa + 32) : z;
            const uint4 c0 = vb ? ldcg_v4(qpb) : z, c1 = vb ? ldcg_v4(qpb + 32) : z;
            // k-step ks covers the dims {32 (ks >> 1) + 8 tq + 4 (ks & 1) + 0..3} of this lane (K uses the same map)
            qa[0][0] = a0.x; qa[0][1] = c0.x; qa[0][2] = a0.y; qa[0][3] = c0.y;
            qa[1][0] = a0.z; qa[1][1] = c0.z; qa[1][2] = a0.w; qa[1][3] = c0.w;
            qa[2][0] = a1.x; qa[2][1] = c1.x; qa[2][2] = a1.y; qa[2][3] = c1.y;
            qa[3][0] = a1.z; qa[3][1] = c1.z; qa[3][2] = a1.w; qa[3][3] = c1.w;
        }
        float o[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) { o[n][0] = 0.f; o[n][1] = 0.f; o[n][2] = 0.f; o[n][3] = 0.f; }
        float ma = -INFINITY, mb = -INFINITY, la = 0.f, lb = 0.f;      // running max (quad-uniform), this lane's share of the sums
        const int32_t* bt = A.b.block_table + (size_t)bs * A.b.max_pages;
        // page ids of the split: lane i holds the id of the i-th page the split touches (one coalesced load; a split longer
        // than 32 pages reloads).  A 16-position group never straddles a page (pages hold 16 or 32 positions).
        const int psh = ps == 32 ? 5 : 4;
        int pg_base = p0 >> psh;
        int my_page = ((pg_base + c.lane) << psh) < pl ? ldcg_i32(bt + pg_base + c.lane) : 0;
        // Addressing is the hot loop's other half (the phase is issue-bound): everything per-lane is a byte offset fixed
        // before the loop, a group costs one shuffle and one 64-bit multiply-add, full groups load without predicates.
        const char* pool = reinterpret_cast<const char*>(M.kv_pool) + ((size_t)ph.layer * 2 * Hkv + kvh) * head_stride * 2;
        const size_t page_bytes = page_stride * 2, v_delta = (size_t)Hkv * head_stride * 2;
        const uint32_t koff = (uint32_t)(gq * kHeadDim + tq * 8) * 2;        // K row gq (n-tile 1: + 8 rows), this lane's dims 8 tq .. (+ 32)
        const uint32_t voff = (uint32_t)(2 * tq * kHeadDim + gq * 8) * 2;    // V rows 2 tq (+ 1, + 8, + 9), dims 8 gq ..
        auto group_base = [&](int pb) -> const char* {
            const int pg = pb >> psh;
            if (pg - pg_base >= 32) {
                pg_base = pg;
                my_page = ((pg_base + c.lane) << psh) < pl ? ldcg_i32(bt + pg_base + c.lane) : 0;
            }
            const int page = __shfl_sync(0xffffffffu, my_page, (pg - pg_base) & 31);
            return pool + (size_t)page * page_bytes + ((size_t)(pb & (ps - 1)) << 7);
        };
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        uint4 kk[2][2], vv[4];
        auto load_k = [&](const char* gb, int pb) {      // K rows of n-tile j: position pb + 8 j + gq, this lane's 2 x 8 dims
            const char* kp = gb + koff;
            if (pb + 16 <= pl) {
                kk[0][0] = ldcg_v4(kp); kk[0][1] = ldcg_v4(kp + 64);
                kk[1][0] = ldcg_v4(kp + 1024); kk[1][1] = ldcg_v4(kp + 1088);
            } else {
                const bool ok0 = pb + gq < pl, ok1 = pb + 8 + gq < pl;
                kk[0][0] = ok0 ? ldcg_v4(kp) : z; kk[0][1] = ok0 ? ldcg_v4(kp + 64) : z;
                kk[1][0] = ok1 ? ldcg_v4(kp + 1024) : z; kk[1][1] = ok1 ? ldcg_v4(kp + 1088) : z;
            }
        };
        auto load_v = [&](const char* gb, int pb) {      // V rows pb + {2 tq, 2 tq + 1, 2 tq + 8, 2 tq + 9}, dims 8 gq .. 8 gq + 7
            const char* vp = gb + v_delta + voff;
            if (pb + 16 <= pl) {
                vv[0] = ldcg_v4(vp); vv[1] = ldcg_v4(vp + 128); vv[2] = ldcg_v4(vp + 1024); vv[3] = ldcg_v4(vp + 1152);
            } else {
                const int r = pb + 2 * tq;
                vv[0] = r < pl ? ldcg_v4(vp) : z; vv[1] = r + 1 < pl ? ldcg_v4(vp + 128) : z;
                vv[2] = r + 8 < pl ? ldcg_v4(vp + 1024) : z; vv[3] = r + 9 < pl ? ldcg_v4(vp + 1152) : z;
            }
        };
        // software pipeline without extra registers: the K fragments are dead after the QK products and the V fragments
        // after the PV products, so the next group's K loads are issued right after QK (covered by the softmax and PV of
        // this group) and its V loads right after PV (covered by the next group's QK and softmax)
        const char* gb = group_base(p0);
        load_k(gb, p0);
        load_v(gb, p0);
        for (int pb = p0; pb < p1; pb += 16) {
            const bool more = pb + 16 < p1;
            float sc[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                sc[j][0] = 0.f; sc[j][1] = 0.f; sc[j][2] = 0.f; sc[j][3] = 0.f;
                mma16816(sc[j], qa[0], kk[j][0].x, kk[j][0].y);
                mma16816(sc[j], qa[1], kk[j][0].z, kk[j][0].w);
                mma16816(sc[j], qa[2], kk[j][1].x, kk[j][1].y);
                mma16816(sc[j], qa[3], kk[j][1].z, kk[j][1].w);
            }
            if (more) { gb = group_base(pb + 16); load_k(gb, pb + 16); }
            // scores in the log2 domain, causal mask per row, one running-max update per row and 16 positions
            float mna = ma, mnb = mb;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int pc = pb + 8 * j + 2 * tq;
                sc[j][0] = pc < La ? sc[j][0] * kScale : -INFINITY;
                sc[j][1] = pc + 1 < La ? sc[j][1] * kScale : -INFINITY;
                sc[j][2] = pc < Lb ? sc[j][2] * kScale : -INFINITY;
                sc[j][3] = pc + 1 < Lb ? sc[j][3] * kScale : -INFINITY;
                mna = fmaxf(mna, fmaxf(sc[j][0], sc[j][1]));
                mnb = fmaxf(mnb, fmaxf(sc[j][2], sc[j][3]));
            }
            mna = fmaxf(mna, __shfl_xor_sync(0xffffffffu, mna, 1));
            mna = fmaxf(mna, __shfl_xor_sync(0xffffffffu, mna, 2));
            mnb = fmaxf(mnb, __shfl_xor_sync(0xffffffffu, mnb, 1));
            mnb = fmaxf(mnb, __shfl_xor_sync(0xffffffffu, mnb, 2));
            const float refa = (mna == -INFINITY) ? 0.f : mna, refb = (mnb == -INFINITY) ? 0.f : mnb;   // nothing visible yet: all factors 0
            const float ca = ex2(ma - refa), cb = ex2(mb - refb);
            ma = mna; mb = mnb;
            float sa = 0.f, sb = 0.f;
            uint32_t pa[4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float e0 = ex2(sc[j][0] - refa), e1 = ex2(sc[j][1] - refa);
                const float e2 = ex2(sc[j][2] - refb), e3 = ex2(sc[j][3] - refb);
                sa += e0 + e1; sb += e2 + e3;
                pa[2 * j] = pack_bf16(e0, e1);       // row a, k = 8 j + 2 tq, + 1
                pa[2 * j + 1] = pack_bf16(e2, e3);   // row b
            }
            la = fmaf(la, ca, sa); lb = fmaf(lb, cb, sb);
            if (__any_sync(0xffffffffu, (ca != 1.f) | (cb != 1.f))) {   // a row's maximum moved (rare after the first groups)
#pragma unroll
                for (int n = 0; n < 8; ++n) { o[n][0] *= ca; o[n][1] *= ca; o[n][2] *= cb; o[n][3] *= cb; }
            }
            // O += P V: n-tile n, column gq of the B fragment = dim 8 gq + n; k pairs (2 tq, 2 tq + 1) and (2 tq + 8, 2 tq + 9)
            const uint32_t v0[4] = {vv[0].x, vv[0].y, vv[0].z, vv[0].w}, v1[4] = {vv[1].x, vv[1].y, vv[1].z, vv[1].w};
            const uint32_t v2[4] = {vv[2].x, vv[2].y, vv[2].z, vv[2].w}, v3[4] = {vv[3].x, vv[3].y, vv[3].z, vv[3].w};
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const uint32_t sel = (n & 1) ? 0x7632u : 0x5410u;
                mma16816(o[n], pa, prmt(v0[n >> 1], v1[n >> 1], sel), prmt(v2[n >> 1], v3[n >> 1], sel));
            }
            if (more) load_v(gb, pb + 16);
        }
        la += __shfl_xor_sync(0xffffffffu, la, 1); la += __shfl_xor_sync(0xffffffffu, la, 2);
        lb += __shfl_xor_sync(0xffffffffu, lb, 1); lb += __shfl_xor_sync(0xffffffffu, lb, 2);
        // this lane holds, for rows a and b, the dims 16 tq + n (o[n][0], o[n][2]) and 16 tq + 8 + n (o[n][1], o[n][3])
        bool need_count = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool valid = h ? vb : va;
            const int r = h ? rb : ra, i = h ? ib : ia, Lr = h ? Lb : La;
            if (!valid || Lr <= p0) continue;            // padding row, or a row that ends before this split starts
            const int row = b0 + i, hq = kvh * G + (r - i * G);
            const float lsum = h ? lb : la, mrow = h ? mb : ma;
            if (sp.count(Lr) == 1) {
                float x0[8], x1[8];
#pragma unroll
                for (int n = 0; n < 8; ++n) { x0[n] = o[n][2 * h] / lsum; x1[n] = o[n][2 * h + 1] / lsum; }
                uint16_t* dst = M.attn + (size_t)row * Hq * kHeadDim + hq * kHeadDim + 16 * tq;
                *reinterpret_cast<uint4*>(dst) = pack8(x0);
                *reinterpret_cast<uint4*>(dst + 8) = pack8(x1);
            } else {
                need_count = true;
                float* dst = M.partial + (((size_t)row * Hq + hq) * kMaxSplits + s) * kPartialStride;
                if (tq == 0) { dst[0] = mrow; dst[1] = lsum; }
#pragma unroll
                for (int n = 0; n < 8; n += 2) {
                    *reinterpret_cast<float2*>(dst + 2 + 16 * tq + n) = make_float2(o[n][2 * h], o[n + 1][2 * h]);
                    *reinterpret_cast<float2*>(dst + 2 + 16 * tq + 8 + n) = make_float2(o[n][2 * h + 1], o[n + 1][2 * h + 1]);
                }
            }
        }
        if (!__any_sync(0xffffffffu, need_count)) continue;
        __threadfence();
        __syncwarp();
        // one arrival per (row, kv head); the last split of a row combines all of its splits in split order
        int ns_row = 0;
        uint32_t old = 0;
        if (c.lane < nq) {
            const int Lr = min(L0 + c.lane, cap);
            ns_row = sp.count(Lr);
            if (ns_row > 1 && Lr > p0) old = atomicAdd(M.split_count + (size_t)(b0 + c.lane) * Hkv + kvh, 1u);
            else ns_row = 0;
        }
        uint32_t last = __ballot_sync(0xffffffffu, ns_row > 1 && old == (uint32_t)(ns_row - 1));
        if (!last) continue;
        __threadfence();
        while (last) {
            const int i = __ffs(last) - 1;
            last &= last - 1;
            const int row = b0 + i, ns = __shfl_sync(0xffffffffu, ns_row, i);
            for (int g = 0; g < G; ++g) {  // lane j holds split j's (m, l); outputs: lane owns dims 2*lane, 2*lane+1
                const int hq = kvh * G + g;
                const float* base = M.partial + ((size_t)row * Hq + hq) * kMaxSplits * kPartialStride;
                const float m_l = c.lane < ns ? ldcg_f32(base + c.lane * kPartialStride) : -INFINITY;
                const float l_l = c.lane < ns ? ldcg_f32(base + c.lane * kPartialStride + 1) : 0.f;
                const float Mg = warp_max(m_l);
                const float sc_l = (m_l == -INFINITY) ? 0.f : ex2(m_l - Mg);
                float Lsum = 0.f, O0 = 0.f, O1 = 0.f;
                for (int si = 0; si < ns; si += 4) {
                    float2 ov[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        ov[u] = si + u < ns ? __ldcg(reinterpret_cast<const float2*>(base + (si + u) * kPartialStride + 2 + 2 * c.lane))
                                            : make_float2(0.f, 0.f);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float scu = __shfl_sync(0xffffffffu, sc_l, (si + u) & 31);
                        const float ll = __shfl_sync(0xffffffffu, l_l, (si + u) & 31);
                        if (si + u < ns) {
                            Lsum = fmaf(ll, scu, Lsum);
                            O0 = fmaf(ov[u].x, scu, O0);
                            O1 = fmaf(ov[u].y, scu, O1);
                        }
                    }
                }
                *reinterpret_cast<uint32_t*>(M.attn + (size_t)row * Hq * kHeadDim + hq * kHeadDim + 2 * c.lane) = pack_bf16(O0 / Lsum, O1 / Lsum);
            }
            if (c.lane == 0) M.split_count[(size_t)row * Hkv + kvh] = 0u;
        }
    }
}

// One weight phase on the tensor cores.  `target` is the grid barrier's running count: most phases start with a
// distributed pre-step (tc_norm_rows, or the depth attention before a fast wo) followed by an extra grid barrier;
// one-phase-per-launch mode runs the pre-step and the tiles as two launches instead (A.tc_part).
__device__ __forceinline__ void tile_gemm(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, umma::Bars* bars,
                              umma::Pipe& pipe, uint32_t& target, bool first_in_launch, bool next_in_launch) {
    const bool fast = ph.fast != 0;
    const int kind = ph.kind;
    const int D = fast ? M.fdim : M.dim, F = fast ? M.finter : M.inter;
    const int Hq = fast ? M.fn_head : M.n_head, Hkv = fast ? M.fn_kv : M.n_kv;
    const DevLayer& L = fast ? M.fast_layers[ph.layer] : M.layers[ph.layer];
    const int q_rows = Hq * kHeadDim, k_end = (Hq + Hkv) * kHeadDim;
    const int n_head_rows = fast ? M.codebook_size : M.vocab;
    const int K = (kind == PH_W2) ? F : D;
    const int n_out = kind == PH_QKV ? (Hq + 2 * Hkv) * kHeadDim : kind == PH_W13 ? F : kind == PH_HEAD ? n_head_rows : D;
    const uint16_t* table = fast ? M.fast_rope : M.rope;
    uint16_t* stream = fast ? M.xf : M.x;
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)c.xs + 1023) & ~(uintptr_t)1023);
    int* pos = reinterpret_cast<int*>(ring + umma::kRingBytes);
    // sub-phase timers of CTA 0 (tools/phase_profile.py): pre-step + barrier | tile setup | ring + MMA | epilogue
    const bool prof = (M.prof != nullptr) && c.cta == 0 && c.tid == 0;
    unsigned long long* seg = M.prof + 2 * kMaxProg + (size_t)(kind + (fast ? 8 : 0)) * 4;
    unsigned long long ts = 0;
    if (prof) ts = globaltimer_ns();

    // ---- distributed pre-step ----
    // (a normed phase that follows a wo / w2 inside one cooperative launch finds M.xn written by that phase's post-step)
    // (and the first QKV of a depth step finds its input written by the SAMPLE phase before it: phase_sample, tc_feed)
    const bool fed_by_post = A.cooperative && !first_in_launch &&
                             (kind == PH_W13 || kind == PH_HEAD || (kind == PH_QKV && ph.layer > 0) ||
                              (kind == PH_QKV && fast && ph.layer == 0 && !A.fast_from_xf));
    if (tile_has_prestep(ph) && !fed_by_post) {
        if (A.tc_part == 0 || A.tc_part == 1) {
            if (kind == PH_WO) {
                tile_depth_attention(M, A, c, ph.layer, ph.depth_pos);
            } else {
                int src_kind = 3;
                const uint16_t* base = kind == PH_W13 ? M.h : stream;
                uint16_t* spill = nullptr;
                if (kind == PH_QKV && ph.layer == 0) {
                    if (!fast) { src_kind = 0; spill = M.x; }
                    else if (!A.fast_from_xf) { src_kind = ph.depth_pos == 0 ? 1 : 2; spill = M.xf; }
                }
                const uint16_t* norm_w = kind == PH_QKV ? L.attention_norm : kind == PH_W13 ? L.ffn_norm : (fast ? M.fast_norm : M.norm);
                tile_norm_rows(M, A, c, ph, src_kind, base, spill, norm_w, D);
            }
        }
        if (A.cooperative) {
            fence_proxy_async_all();
            grid_arrive(M.barrier, target, (uint32_t)c.n_ctas);
            grid_wait(M.barrier, target);
            if (c.tid == umma::kTmaProducerA || c.tid == umma::kTmaProducerB) fence_proxy_async_all();   // the threads that issue TMA loads
        }
        if (A.tc_part == 1) return;
    }
    if (prof) { const unsigned long long t = globaltimer_ns(); seg[0] += t - ts; ts = t; }

    // ---- operands: activation tile and weight rows through TMA ----
    const unsigned char* tm = M.tmaps;
    const int box_idx = A.batch <= 32 ? 2 : A.batch <= 64 ? 1 : 0;   // activation box of 32 / 64 / 128 rows
    const int a_rows = umma::kM >> box_idx;
    const void* tm_a = tm + (size_t)kTensorMapBytes * (box_idx * TM_ACT_MAPS + (fast ? TM_FAST : 0) + (kind == PH_WO ? TM_ATTN : kind == PH_W2 ? TM_ACT : TM_XN));
    const int which = kind == PH_QKV ? 0 : kind == PH_WO ? 1 : kind == PH_W13 ? 2 : 4;
    const int layer = fast ? M.n_layer + ph.layer : ph.layer;
    const int w_index0 = kind == PH_HEAD ? (fast ? 1 : 0) : tm_weight_index(layer, which);
    const int w_index1 = kind == PH_W13 ? tm_weight_index(layer, 3) : -1;
    const int w_row_base = (kind == PH_HEAD && fast && M.depthwise_output) ? ph.depth_pos * n_head_rows : 0;

    // the residual phases (wo, w2) also cut K: their fp32 partials meet in the post-step
    const bool has_post = kind == PH_WO || kind == PH_W2;
    const int n_split = !has_post ? 1 : (K % (4 * umma::kBK) == 0) ? 4 : (K % (2 * umma::kBK) == 0) ? 2 : 1;
    const int k_len = K / n_split;
    const int m_tiles = (A.batch + umma::kM - 1) / umma::kM;
    const int blk_cap = kind == PH_W13 ? umma::kMaxN / 2 : umma::kMaxN;
    int blk = 16;
    while (blk < blk_cap && m_tiles * ((n_out + blk - 1) / blk) * n_split > c.n_ctas) blk += 16;
    const int n_blocks = (n_out + blk - 1) / blk;
    const int n_units = (A.tc_part == 0 || A.tc_part == 2) ? m_tiles * n_blocks * n_split : 0;

    for (int u = c.cta; u < n_units; u += c.n_ctas) {
        const int mt = u % m_tiles, un = u / m_tiles;       // the row tiles that share a weight block on neighbouring CTAs
        const int ks = un % n_split, nb = un / n_split;
        const int m0 = mt * umma::kM, n0 = nb * blk;
        if (kind == PH_QKV && c.tid < umma::kM) {
            const int bg = min(m0 + c.tid, A.batch - 1);
            pos[c.tid] = fast ? ph.depth_pos : ldcg_i32(A.b.seq_len + row_seq(A, bg)) + row_off(A, bg);
        }
        __syncthreads();
        if (prof) { const unsigned long long t = globaltimer_ns(); seg[1] += t - ts; ts = t; }
        umma::BSrc b0, b1;
        b0.tm = tm + (size_t)kTensorMapBytes * tm_weight_slot(w_index0, blk); b0.row0 = w_row_base + n0; b0.n = blk; b0.box = blk;
        b1.tm = w_index1 >= 0 ? tm + (size_t)kTensorMapBytes * tm_weight_slot(w_index1, blk) : nullptr;
        b1.row0 = n0; b1.n = w_index1 >= 0 ? blk : 0; b1.box = blk;
        umma::tile_mma_tma<kThreads>(ring, bars, pipe, k_len, tm_a, m0, b0, b1, ks * k_len, a_rows);
        if (prof) { const unsigned long long t = globaltimer_ns(); seg[2] += t - ts; ts = t; }

        if (kind == PH_W13) {
            umma::tile_epilogue_paired(bars, blk, [&](int row, int c0, const float (&ga)[8], const float (&up)[8]) {
                const int bg = m0 + row, u0 = n0 + c0;
                if (bg >= A.batch || u0 >= n_out) return;
                float o[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float a = bf16_round(ga[e]), g = bf16_round(up[e]);
                    // F.silu in fp32, bf16 out: a is a bf16 value, so the exactly rounded result is a table look-up (the
                    // exact exp / division made this epilogue issue-bound; a fast-math form moved 0.02 % of the results)
                    const float sg = __uint_as_float((uint32_t)__ldg(M.silu_lut + (__float_as_uint(a) >> 16)) << 16);
                    o[e] = __fmul_rn(sg, g);
                }
                *reinterpret_cast<uint4*>(M.act + (size_t)bg * F + u0) = pack8(o);
            }, b0.n + b1.n);
        } else {
            umma::tile_epilogue(bars, blk, [&](int row, int c0, const float (&acc)[8]) {
                const int bg = m0 + row, u0 = n0 + c0;
                if (bg >= A.batch || u0 >= n_out) return;
                if (kind == PH_HEAD) {
                    float* out = fast ? M.depth_logits + ((size_t)bg * M.depth + ph.depth_pos) * n_head_rows
                                      : M.token_logits + (size_t)bg * n_head_rows;
                    if (n_head_rows & 7) {   // (rows of logits that do not start on 16 bytes)
                        for (int e = 0; e < 8 && u0 + e < n_head_rows; ++e) out[u0 + e] = bf16_round(acc[e]);
                        return;
                    }
                    *reinterpret_cast<float4*>(out + u0) = make_float4(bf16_round(acc[0]), bf16_round(acc[1]), bf16_round(acc[2]), bf16_round(acc[3]));
                    *reinterpret_cast<float4*>(out + u0 + 4) = make_float4(bf16_round(acc[4]), bf16_round(acc[5]), bf16_round(acc[6]), bf16_round(acc[7]));
                    return;
                }
                if (kind != PH_QKV) {  // wo, w2: this K slice's partial sums (the post-step adds slices and residual)
                    float* pp = M.kpart + ((size_t)ks * M.ws_rows + bg) * D + u0;
                    *reinterpret_cast<float4*>(pp) = make_float4(acc[0], acc[1], acc[2], acc[3]);
                    *reinterpret_cast<float4*>(pp + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
                    return;
                }
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = bf16_round(acc[e]);
                const int p = pos[row];
                const int tp = fast ? p : min(p, M.max_seq_len - 1);  // never past the RoPE table (host checks bound p)
                if (u0 < k_end) {  // q and k rows: interleaved-pair RoPE with the bf16 table (P:616-640)
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const int j = ((u0 + e) & (kHeadDim - 1)) >> 1;
                        const uint32_t cs = __ldg(reinterpret_cast<const uint32_t*>(table + ((size_t)tp * (kHeadDim / 2) + j) * 2));
                        const float co = bf_lo(cs), si = bf_hi(cs);
                        const float r0 = bf16_round(__fsub_rn(__fmul_rn(v[e], co), __fmul_rn(v[e + 1], si)));
                        const float r1 = bf16_round(__fadd_rn(__fmul_rn(v[e + 1], co), __fmul_rn(v[e], si)));
                        v[e] = r0; v[e + 1] = r1;
                    }
                }
                const uint4 packed = pack8(v);
                if (u0 < q_rows) {
                    *reinterpret_cast<uint4*>(M.q + (size_t)bg * q_rows + u0) = packed;
                    return;
                }
                const int is_v = u0 >= k_end ? 1 : 0;
                const int n1 = u0 - (is_v ? k_end : q_rows);
                const int kvh = n1 / kHeadDim, d = n1 & (kHeadDim - 1);
                if (fast) {
                    uint16_t* dst = M.fkv + (((size_t)(bg * M.n_flayer + ph.layer) * 2 + is_v) * M.depth + ph.depth_pos) * (Hkv * kHeadDim)
                                    + kvh * kHeadDim + d;
                    *reinterpret_cast<uint4*>(dst) = packed;
                } else {
                    if (!seq_active(M, A, c, bg)) return;
                    const int ps = M.page_size;
                    if (p >= A.b.max_pages * ps) return;
                    const int page = ldcg_i32(A.b.block_table + (size_t)row_seq(A, bg) * A.b.max_pages + p / ps);
                    uint16_t* dst = M.kv_pool + ((((size_t)page * M.n_layer + ph.layer) * 2 + is_v) * Hkv + kvh) * ((size_t)ps * kHeadDim)
                                    + (size_t)(p % ps) * kHeadDim + d;
                    *reinterpret_cast<uint4*>(dst) = packed;
                }
            }, b0.n + b1.n);
        }
        if (prof) { const unsigned long long t = globaltimer_ns(); seg[3] += t - ts; ts = t; }
    }

    // ---- post-step of the residual phases: wo: h = stream + wo(attn) (P:499); w2: stream = h + w2(act) (P:500) ----
    if (has_post && A.tc_part != 2) {
        if (A.cooperative) {
            grid_arrive(M.barrier, target, (uint32_t)c.n_ctas);
            grid_wait(M.barrier, target);
        }
        const uint16_t* next_norm = nullptr;
        if (A.cooperative && next_in_launch) {
            const int n_net = fast ? M.n_flayer : M.n_layer;
            if (kind == PH_WO) next_norm = L.ffn_norm;
            else if (ph.layer + 1 < n_net) next_norm = (fast ? M.fast_layers[ph.layer + 1] : M.layers[ph.layer + 1]).attention_norm;
            else next_norm = fast ? M.fast_norm : M.norm;
        }
        tile_finish(M, A, c, kind == PH_WO ? stream : M.h, kind == PH_WO ? M.h : stream, D, n_split, next_norm);
        if (prof) { const unsigned long long t = globaltimer_ns(); seg[0] += t - ts; ts = t; }
    }
}

__shared__ __align__(8) umma::Bars g_tile_bars;

__global__ void __launch_bounds__(kThreads, 1)
smol_tiles_kernel(const __grid_constant__ DevModel M, const __grid_constant__ CallArgs A) {
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    Ctx c;
    c.cta = blockIdx.x; c.n_ctas = gridDim.x; c.tid = threadIdx.x;
    c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31;
    c.xs = reinterpret_cast<float*>(smem_dyn);
    c.stage = smem_dyn;
    c.iter = 0;
    uint32_t target = 0;
    if (A.cooperative) target = ldcg_u32(M.barrier + 1);
    umma::Pipe pipe;
    pipe.chunk = 0; pipe.tile = 0;
    umma::setup(&g_tile_bars, pipe, (uint32_t)umma::kAcc, 2u);
    const int per_iter = (A.mode == 1) ? phases_per_prefill_step(M.n_layer) : phases_per_frame(M.n_layer, M.n_flayer, M.depth);
    const bool prof_cta = M.prof != nullptr && c.cta == 0;  // CTA-uniform
    const bool prof = prof_cta && c.tid == 0;
    unsigned long long t0 = 0, t1 = 0;
    for (int it = 0; it < A.n_iter; ++it) {
        c.iter = it;
        for (int p = A.phase_begin; p < A.phase_end; ++p) {
            const Phase ph = unpack_phase(M.prog[p]);
            const bool first = p == A.phase_begin, more = p + 1 < A.phase_end;
            if (prof) t0 = globaltimer_ns();
            if (ph.kind == PH_ATTN) tile_attn(M, A, c, ph);
            else if (ph.kind == PH_SAMPLE) phase_sample(M, A, c, ph, A.cooperative && more && !A.fast_from_xf && !(ph.fast && ph.depth_pos == M.depth - 1));
            else tile_gemm(M, A, c, ph, &g_tile_bars, pipe, target, first, more);
            if (prof_cta) {
                __syncthreads();
                if (prof) t1 = globaltimer_ns();
            }
            // (one phase per launch: a phase may take up to three launches; bookkeeping runs in the last)
            const bool final_part = A.tc_part == 0 || A.tc_part == (tile_has_poststep(ph) ? 3 : 2);
            if (c.cta == 0 && p == per_iter - 1 && A.mode == 1 && final_part) {
                // prefill bookkeeping: every sequence advances by the positions of this tile that lie inside its prompt
                const int T = A.tile_t > 1 ? A.tile_t : 1;
                for (int b = c.tid; b < A.real_batch; b += kThreads) {
                    int n_act = prompt_positions(A, b) - (A.iter_base + c.iter * T);
                    n_act = n_act < 0 ? 0 : (n_act > T ? T : n_act);
                    if (n_act) A.b.seq_len[b] = ldcg_i32(A.b.seq_len + b) + n_act;
                }
            }
            if (c.cta == 0 && A.mode == 0 && A.advance && p == A.phase_end - 1) {
                for (int b = c.tid; b < A.batch; b += kThreads) A.b.seq_len[b] = ldcg_i32(A.b.seq_len + b) + 1;
            }
            if (A.cooperative && !(it == A.n_iter - 1 && p == A.phase_end - 1)) {
                fence_proxy_async_all();
                grid_arrive(M.barrier, target, (uint32_t)c.n_ctas);
                grid_wait(M.barrier, target);
                if (c.tid == umma::kTmaProducerA || c.tid == umma::kTmaProducerB) fence_proxy_async_all();   // the threads that issue TMA loads
            }
            if (prof) {  // [2p] CTA 0's own time in the phase, [2p+1] its wait at the barrier that follows
                const unsigned long long t2 = globaltimer_ns();
                M.prof[2 * p] += t1 - t0;
                M.prof[2 * p + 1] += t2 - t1;
            }
        }
    }
    if (A.mode == 1 && A.finalize && c.cta == 0) {
        // leave the last prompt column as the pending input of the first decode frame (G:66-73)
        for (int i = c.tid; i < A.real_batch * M.n_rows; i += kThreads) {
            const int b = i / M.n_rows, r = i - b * M.n_rows;
            A.b.tokens[i] = ldcg_i32(A.prompt + ((size_t)b * M.n_rows + r) * A.s_max + prompt_last(A, b));
        }
    }
    if (A.cooperative && c.cta == 0 && c.tid == 0) M.barrier[1] = target;
    umma::teardown(&g_tile_bars);
}

}  // namespace smol
