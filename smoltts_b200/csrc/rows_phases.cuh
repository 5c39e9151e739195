// Batched decode: the weight phases of decode_kernel.cu for 9 and more rows (sequences) as mma.sync tiles, plus the batch form of
// the paged attention (which prompts use too).  Included by decode_kernel.cu (uses its Ctx, grid barrier, embedding and row
// bookkeeping helpers).
//
// A frame is a chain of 196 dependent phases; a layer's weights (17 MB) take 2.7 us at the copy bandwidth, while a barrier of the
// grid takes 1.3 us and the exchange of 64 rows of 768 through L2 another 0.5 to 1.  What counts is how little else happens
// between two barriers.  So
//   * a phase is ONE step between two barriers: RMSNorm, the residual add and the depth attention happen inside the tiles
//     that read or write the rows (redundantly per tile), not in steps of their own;
//   * weights never wait for activations: a CTA's weight tiles of the next phase (one bulk copy, packed fragments) land in
//     shared memory while it finishes this phase and sits in the barrier; cached keys and values are fetched there, too;
//   * rows come by bulk copies, and a phase's pointers and sizes from tables in shared memory.
// Measured (150m, us per frame): 9 rows (contexts of up to 100) 1093, 33: 1288, 64 (up to 471): 1411; tcgen05 tiles (tile_phases.cuh:
// activation rows as the 128 lanes of an accumulator, 16 .. 96 weight rows as its columns, row steps between the phases) take 2024, 2094
// and 2216: with so few columns an MMA is bound by the 4 KB of its A operand, wo and w2 are cut over CTAs and added in a step of their
// own, and a frame has 380 barriers instead of 197.  Wide batches take several turns here and go there (in_groups, capi.cu).
//
// Summation order: four chains of MMAs per dot product (K steps 0, 4, 8 .. of 16 elements; 1, 5, 9 ..; ..), for wo and w2 per K
// slice, added in order: a function of K alone, so a row's bits depend neither on the number of rows nor on the tile plan.  (The
// tcgen05 tiles sum in the same order, and mma.sync and tcgen05 turn out to round alike: to the bit the same.)
#pragma once

namespace smol {

constexpr int kTcSplit = 128;  // cached positions per attention split of the batch attention (CallArgs.tc_split overrides it)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The thread's number, read where it is used: a phase's per-thread offsets must not be computed once for all phases (the
// compiler would, and keep them in local memory: with 227 KB of shared memory the L1 is too small for them).
__device__ __forceinline__ int tid_here() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 v;
    v.x = pack_bf16(f[0], f[1]); v.y = pack_bf16(f[2], f[3]); v.z = pack_bf16(f[4], f[5]); v.w = pack_bf16(f[6], f[7]);
    return v;
}

// A wait that runs out ends the launch and is reported by the model's next call (wait_over).
__device__ __forceinline__ void rows_wait(const DevModel& M, uint64_t* bar, uint32_t parity) {
    unsigned long long t0 = 0ull;
    for (uint32_t spin = 1; !mbar_try(bar, parity); ++spin) {
        if ((spin & 255u) == 0u) {
            t0 = wait_over(M.barrier, M.status, M.wait_ms, t0);
            if (t0 == kWaitOver) return;
        }
    }
}

// The grid barrier between phases, split: a CTA arrives at the end of a phase and waits inside the next one, behind what that
// one can do without its input (a w2 tile's weights -> registers, cached keys and values -> shared memory).
struct RowsSync {
    uint32_t target;         // arrivals the barrier completes at
    uint32_t par_w, par_x;   // parities of the weight and the row copies
    bool pending, failed;    // failed: the launch was given up (the same in all threads)
    int phase, next;         // this phase; the launch's next weight phase (-1: none), whose tiles this one fetches
    int waits_for;           // the phase whose barrier is pending
};
template <bool kTimed>
__device__ __forceinline__ void rows_sync_in(const DevModel& M, RowsSync& sy) {
    if (!sy.pending) return;
    const bool prof = kTimed && blockIdx.x == 0 && threadIdx.x == 0;
    unsigned long long t = 0;
    if (prof) t = globaltimer_ns();
    sy.failed = __syncthreads_or(threadIdx.x == 0 && grid_poll(M.barrier, M.status, M.wait_ms, sy.target)) != 0;
    sy.pending = false;
    if (prof) {   // belongs to the phase in front of the barrier, not to the one that waits
        t = globaltimer_ns() - t;
        M.prof[2 * sy.waits_for + 1] += t;
        M.prof[2 * sy.phase] -= t;
    }
}
// Profiling: ns in segment s of a weight phase's body (CTA 0, one thread), from the last stamp on.
__device__ __forceinline__ void rows_stamp(const DevModel& M, int kind, int fast, int s, unsigned long long& t) {
    const unsigned long long now = globaltimer_ns();
    M.prof[2 * kMaxProg + (kind + 8 * fast) * 4 + s] += now - t;
    t = now;
}
template <bool kTimed>
__device__ __forceinline__ void rows_arrive(const DevModel& M, const Ctx& c, RowsSync& sy) {
    rows_sync_in<kTimed>(M, sy);       // (a phase in which this CTA has no work may not have waited yet)
    // Shared memory used here is overwritten by copies.  (Rows written here are read by other CTAs' copies: the threads that issue those
    // fence global memory behind the barrier; a full fence.proxy.async here waits for
    // the stores of every thread: frames of 9 / 64 rows 1263 / 1520 us with it, 1188 / 1437 without.)
    fence_proxy_async();
    grid_arrive(M.barrier, sy.target, (uint32_t)c.n_ctas);
    sy.pending = true;
    if (kTimed) sy.waits_for = sy.phase;
}

// ---- batch attention on the tensor cores -------------------------------------------------------------------------
// mma.sync.m16n8k16 (bf16 x bf16 -> fp32): the 16 rows of the A operand are the query rows that share one kv head's
// cached K/V -- the G query heads of the kv head (GQA) times, in a prefill iteration, up to 16/G consecutive prompt
// positions of the sequence -- so one pass over a position's 256 bytes of K|V serves all of them.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    mma_bf16_16816(d, a[0], a[1], a[2], a[3], b0, b1);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Split schedule of the batch attention: ABSOLUTE position ranges, the same for every row whatever its length -- 16
// splits of s0 positions, then splits of 2*s0 -- so that rows of different lengths (the consecutive prompt positions of a
// prefill group) share their K/V passes and a row's result is still a function of its own context only (it combines, in
// split order, the splits that start below its length).  s0 = 128 covers 6144 positions with kMaxSplits = 32 splits.
struct SplitPlan {
    int s0, wide_from;   // splits [0, wide_from) hold s0 positions, later ones 2*s0
    __device__ __forceinline__ int lo(int k) const { return k <= wide_from ? k * s0 : wide_from * s0 + (k - wide_from) * 2 * s0; }
    __device__ __forceinline__ int count(int L) const {   // splits that start below position L
        if (L <= wide_from * s0) return (L + s0 - 1) / s0;
        return wide_from + (L - wide_from * s0 + 2 * s0 - 1) / (2 * s0);
    }
};
__device__ __forceinline__ SplitPlan split_plan(const CallArgs& A, int cap) {
    SplitPlan sp;
    if (A.tc_split >= 16) {   // the caller's override (tests): uniform splits, widened only if kMaxSplits would not cover cap
        sp.s0 = max(A.tc_split & ~15, (((cap + kMaxSplits - 1) / kMaxSplits) + 15) & ~15);
        sp.wide_from = kMaxSplits;
        return sp;
    }
    sp.s0 = kTcSplit;
    sp.wide_from = kMaxSplits / 2;
    while (sp.lo(kMaxSplits) < cap) sp.s0 *= 2;
    return sp;
}

// Warps per unit of the batch attention: as many as leave every unit a place at once.
__device__ __forceinline__ int attn_warps(int n_units, int n_ctas) {
    int wpt = kWarps;
    while (wpt > 4 && n_units * wpt > n_ctas * kWarps) wpt >>= 1;
    return wpt;
}

// Decode: the cached keys and values that this CTA's attention units will read -> L2, a phase ahead (64 rows at 471 positions
// hold 310 MB, so a layer's 31 MB come from HBM: 4.8 us at the copy bandwidth, which the QKV phase hides).
__device__ __forceinline__ void attn_prefetch(const DevModel& M, const CallArgs& A, const Ctx& c, int layer) {
    const int tid = tid_here(), warp = tid >> 5, lane = tid & 31;
    const int Hkv = M.n_kv, ps = M.page_size, n_units = A.batch * Hkv;
    const int wpt = attn_warps(n_units, c.n_ctas), per_cta = kWarps / wpt, slot = warp / wpt;
    for (int t = slot * c.n_ctas + c.cta; t < n_units; t += c.n_ctas * per_cta) {
        const int b = t / Hkv, kvh = t - b * Hkv;
        const int np = (min(ldcg_i32(A.b.seq_len + b), A.b.max_pages * ps) + ps - 1) / ps;
        for (int i = (warp - slot * wpt) * 32 + lane; i < 2 * np; i += wpt * 32) {
            const int page = ldcg_i32(A.b.block_table + (size_t)b * A.b.max_pages + (i >> 1));
            const uint16_t* src = M.kv_pool + ((((size_t)page * M.n_layer + layer) * 2 + (i & 1)) * Hkv + kvh) * ((size_t)ps * kHeadDim);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(ps * kHeadDim * 2) : "memory");
        }
    }
}

constexpr int kAttnStage = 8192;   // a warp's place in shared memory: two steps of keys and values; a split's state (36 floats per lane)
__shared__ __align__(8) uint64_t g_kvbar[2 * kWarps];   // a barrier per step buffer, and the parity of its next use
__shared__ uint32_t g_kvpar[2 * kWarps];
__device__ __forceinline__ void tma_kv(uint32_t dst, const void* map, int row, int page_layer, uint64_t* bar) {   // 16 rows of keys, 16 of values
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(page_layer) : "memory");
}

// Decode / prefill attention over the paged cache for a batch.  Unit = (query group, kv head); a
// query group is one decode row, or up to 16/G consecutive prompt positions of one sequence.  Per 16 cached positions:
// S = Q K^T (2 n-tiles x 4 k-steps), online softmax in base 2 with P rounded to bf16 for the PV product as the reference's
// SDPA does (P:559-566; the denominator sums the unrounded fp32 values), O += P V (8 n-tiles).  The k index of the QK product and
// the n index of the PV product are permuted so that every thread's fragment words are contiguous in memory (a dot product does
// not care about the order of its dims as long as both operands use the same one).  Keys and values come as swizzled 4 KB boxes:
// loaded straight into fragments (16 bytes of 8 rows at a time) they moved at 14 bytes per clock and SM.
// A unit's splits are shared out over `wpt` warps of a CTA, one split each per round.  Where one round is enough (up to 16
// splits, 2048 positions, in a batch of 37 rows) the splits' states (max, sum, O) meet in shared memory, else in M.partial;
// they are combined in split order, relative to the largest maximum, so the result does not depend on wpt.
// Decoding (kPrompt false): one position per unit, so only the fragments' first eight rows are in use, and a unit's cached keys and
// values are fetched before the barrier in front of the phase (all but the step that holds the newest position).
template <bool kPrompt, bool kTimed>
__device__ __forceinline__ void phase_attn_batch(const DevModel& M, const CallArgs& A, const Ctx& c, const Phase& ph, RowsSync& sy, const void* kv_map,
                                                 const int skip_row = -1) {   // kv_map: the pool's tensor map; skip_row: left alone
    const int tid = tid_here(), warp = tid >> 5, lane = tid & 31;
    const int Hq = M.n_head, Hkv = M.n_kv, ps = M.page_size, G = Hq / Hkv;
    const int cap = A.b.max_pages * ps;
    const int T = kPrompt && A.tile_t > 1 ? A.tile_t : 1;
    const int P = T > 1 ? 16 / G : 1;              // query positions per unit
    const int gps = (T + P - 1) / P;               // units (groups) per sequence
    const int n_groups = kPrompt ? (A.batch / T) * gps : A.batch;
    const int gq = lane >> 2, tq = lane & 3;       // fragment coordinates of this lane
    const SplitPlan sp = split_plan(A, cap);
    const int n_units = n_groups * Hkv;
    const int wpt = attn_warps(n_units, c.n_ctas);
    const int per_cta = kWarps / wpt, slot = warp / wpt, wi = warp - slot * wpt;
    if (kPrompt) rows_sync_in<kTimed>(M, sy);
    if (kPrompt && lane == 0) fence_proxy_async_global();    // keys and values written by other CTAs
    constexpr float kScale = 0.125f * 1.4426950408889634f;   // 1/sqrt(64) * log2(e): softmax in base 2

    // neighbouring units on different SMs; the trip count is the same for all warps of the CTA
    for (int t0 = 0; t0 < n_units; t0 += c.n_ctas * per_cta) {
        const int t = t0 + slot * c.n_ctas + c.cta;
        const bool work = t < n_units;
        const int grp = work ? t / Hkv : 0, kvh = work ? t - grp * Hkv : 0;
        const int sq = kPrompt ? grp / gps : grp, go = kPrompt ? (grp - sq * gps) * P : 0;
        const int b0 = sq * T + go;                                   // first batch row of the group
        const int nq = kPrompt ? min(P, T - go) : 1;                  // its live query positions
        const int bs = row_seq(A, b0);
        const int32_t* bt = A.b.block_table + (size_t)bs * A.b.max_pages;
        const int psh = ps == 32 ? 5 : 4;
        // page ids of the warp's first split, before its length is known (an entry past the sequence is not used)
        const int first_pg = sp.lo(wi) >> psh;
        const int first_page = first_pg + lane < A.b.max_pages ? ldcg_i32(bt + first_pg + lane) : 0;
        const int len0 = ldcg_i32(A.b.seq_len + bs);
        const int L0 = len0 + row_off(A, b0) + 1;                     // context of the first row (its own position included)
        const int Lg = min(L0 + nq - 1, cap);                         // ... of the last one
        // cached positions that hold data: everything up to the group's last ACTIVE row (rows past the end of a prompt do
        // not append; their stale slots must not reach the PV product of the active rows as 0 x garbage)
        int Lload = Lg;
        if (kPrompt) {
            const int act = prompt_positions(A, bs) - (A.iter_base + c.iter * T);
            Lload = min(Lg, len0 + max(0, min(act, T)));
        }
        const int ns = work ? min(sp.count(Lg), kMaxSplits) : 0;      // splits of the group's longest row
        // the two query rows of this lane: row r = (query position r / G, head r % G)
        const int ra = gq, rb = gq + 8;
        const int ia = kPrompt ? ra / G : (ra < G ? 0 : 1), ib = kPrompt ? rb / G : 1;
        const bool va = ia < nq, vb = kPrompt && ib < nq;
        const int La = min(L0 + ia, cap), Lb = min(L0 + ib, cap);     // causal limits (positions < L are visible)
        uint32_t qa[4][4];
        auto load_q = [&]() {
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
        };
        if (kPrompt) load_q();
        const bool two = kPrompt && nq * G > 8;                       // rows 8 .. 15 of the fragments are in use
        const bool one_round = ns <= wpt;
        // where a round has fewer splits than the unit has warps, each takes the step buffers of several
        int share = wpt;
        while (share > 1 && wpt / share < min(ns, wpt)) share >>= 1;
        const int depth = 2 * share;                                  // step buffers of an active warp
        const int buf0 = 2 * (slot * wpt + min(wi * share, wpt - share));
        unsigned char* stage = reinterpret_cast<unsigned char*>(c.xs) + buf0 * (kAttnStage / 2);
        float* st = reinterpret_cast<float*>(stage) + lane;           // then the split's state: [value][lane]
        for (int s0 = 0; s0 < ns; s0 += wpt) {
            const int s = s0 + wi;
            const int p0 = sp.lo(s), p1 = s < ns ? min(Lg, sp.lo(s + 1)) : p0;
            const int pl = min(p1, Lload);
            float o[8][4];
#pragma unroll
            for (int n = 0; n < 8; ++n) { o[n][0] = 0.f; o[n][1] = 0.f; o[n][2] = 0.f; o[n][3] = 0.f; }
            float ma = -INFINITY, mb = -INFINITY, la = 0.f, lb = 0.f;      // running max (quad-uniform), this lane's share of the sums
            if (s < ns) {
                // page ids of the split: lane i holds the id of the i-th page the split touches (one coalesced load; a split longer
                // than 32 pages reloads).  A 16-position step never straddles a page (pages hold 16 or 32 positions).
                int pg_base = p0 >> psh;
                int my_page = s0 == 0 ? first_page : ((pg_base + lane) << psh) < pl ? ldcg_i32(bt + pg_base + lane) : 0;
                // keys and values of a step: a box of 2 x 16 rows x 128 bytes, rows swizzled by the copy engine
                int in = 0, at = 0, fetched = p0;                              // buffers of the next step fetched / used; its position
                uint32_t par = lane < depth ? g_kvpar[buf0 + lane] : 0u;       // lane i: buffer i's parity
                auto fetch = [&]() {
                    const int pb = fetched, pg = pb >> psh;
                    if (pg - pg_base >= 32) {
                        pg_base = pg;
                        my_page = ((pg_base + lane) << psh) < pl ? ldcg_i32(bt + pg_base + lane) : 0;
                    }
                    const int page = __shfl_sync(0xffffffffu, my_page, (pg - pg_base) & 31);
                    if (lane == 0) {
                        uint64_t* bar = &g_kvbar[buf0 + in];
                        mbar_expect_tx(bar, 4096u);
                        tma_kv(smem_u32(stage) + (uint32_t)in * 4096u, kv_map, kvh * ps + (pb & (ps - 1)), page * M.n_layer + ph.layer, bar);
                    }
                    in = in + 1 < depth ? in + 1 : 0;
                    fetched += 16;
                };
                if (!kPrompt && sy.pending) {
                    for (int i = 0; i < depth && fetched + 16 <= min(pl, len0); ++i) fetch();
                    rows_sync_in<kTimed>(M, sy);
                }
                if (!kPrompt) {
                    if (lane == 0) fence_proxy_async_global();   // the newest position was written by other CTAs
                    load_q();
                }
                while (fetched < pl && fetched < p0 + 16 * depth) fetch();
                for (int pb = p0; pb < pl; pb += 16) {
                    rows_wait(M, &g_kvbar[buf0 + at], __shfl_sync(0xffffffffu, par, at));
                    const unsigned char* kt = stage + at * 4096;
                    if (lane == at) par ^= 1u;
                    at = at + 1 < depth ? at + 1 : 0;
                    float sc[2][4];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        // key 8 j + gq: 16-byte pieces tq and tq + 4 of its row, swizzled with the row; odd rows read the second one
                        // first, so that eight lanes never meet in a bank
                        const unsigned char* kr = kt + (8 * j + gq) * 128;
                        const uint4 e0 = *reinterpret_cast<const uint4*>(kr + ((tq + 4 * (gq & 1)) ^ gq) * 16);
                        const uint4 e1 = *reinterpret_cast<const uint4*>(kr + ((tq + 4 - 4 * (gq & 1)) ^ gq) * 16);
                        uint4 k0 = gq & 1 ? e1 : e0, k1 = gq & 1 ? e0 : e1;
                        if (pb + 16 > pl && pb + 8 * j + gq >= pl) { k0 = make_uint4(0u, 0u, 0u, 0u); k1 = k0; }   // past the end: whatever the slot holds
                        sc[j][0] = 0.f; sc[j][1] = 0.f; sc[j][2] = 0.f; sc[j][3] = 0.f;
                        mma16816(sc[j], qa[0], k0.x, k0.y);
                        mma16816(sc[j], qa[1], k0.z, k0.w);
                        mma16816(sc[j], qa[2], k1.x, k1.y);
                        mma16816(sc[j], qa[3], k1.z, k1.w);
                    }
                    // scores in the log2 domain, causal mask per row, one running-max update per row and 16 positions
                    float mna = ma, mnb = mb;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int pc = pb + 8 * j + 2 * tq;
                        sc[j][0] = pc < La ? sc[j][0] * kScale : -INFINITY;
                        sc[j][1] = pc + 1 < La ? sc[j][1] * kScale : -INFINITY;
                        mna = fmaxf(mna, fmaxf(sc[j][0], sc[j][1]));
                        if (kPrompt) {
                            sc[j][2] = pc < Lb ? sc[j][2] * kScale : -INFINITY;
                            sc[j][3] = pc + 1 < Lb ? sc[j][3] * kScale : -INFINITY;
                            mnb = fmaxf(mnb, fmaxf(sc[j][2], sc[j][3]));
                        }
                    }
                    mna = fmaxf(mna, __shfl_xor_sync(0xffffffffu, mna, 1));
                    mna = fmaxf(mna, __shfl_xor_sync(0xffffffffu, mna, 2));
                    if (kPrompt) {
                        mnb = fmaxf(mnb, __shfl_xor_sync(0xffffffffu, mnb, 1));
                        mnb = fmaxf(mnb, __shfl_xor_sync(0xffffffffu, mnb, 2));
                    }
                    const float refa = (mna == -INFINITY) ? 0.f : mna, refb = (mnb == -INFINITY) ? 0.f : mnb;   // nothing visible yet: all factors 0
                    const float ca = ex2(ma - refa), cb = kPrompt ? ex2(mb - refb) : 1.f;
                    ma = mna; mb = mnb;
                    float sa = 0.f, sb = 0.f;
                    uint32_t pa[4];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float e0 = ex2(sc[j][0] - refa), e1 = ex2(sc[j][1] - refa);
                        sa += e0 + e1;
                        pa[2 * j] = pack_bf16(e0, e1);       // row a, k = 8 j + 2 tq, + 1
                        pa[2 * j + 1] = 0u;
                        if (kPrompt) {
                            const float e2 = ex2(sc[j][2] - refb), e3 = ex2(sc[j][3] - refb);
                            sb += e2 + e3;
                            pa[2 * j + 1] = pack_bf16(e2, e3);   // row b
                        }
                    }
                    la = fmaf(la, ca, sa);
                    if (kPrompt) lb = fmaf(lb, cb, sb);
                    if (__any_sync(0xffffffffu, (ca != 1.f) | (cb != 1.f))) {   // a row's maximum moved (rare after the first groups)
#pragma unroll
                        for (int n = 0; n < 8; ++n) {
                            o[n][0] *= ca; o[n][1] *= ca;
                            if (kPrompt) { o[n][2] *= cb; o[n][3] *= cb; }
                        }
                    }
                    uint4 vv[4];   // rows 2 tq, 2 tq + 1, + 8, + 9: piece gq, swizzled
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int r = 2 * tq + (i & 1) + 8 * (i >> 1);
                        vv[i] = *reinterpret_cast<const uint4*>(kt + 2048 + r * 128 + ((gq ^ (r & 7)) * 16));
                        if (pb + 16 > pl && pb + r >= pl) vv[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    // O += P V: n-tile n, column gq of the B fragment = dim 8 gq + n; k pairs (2 tq, 2 tq + 1) and (2 tq + 8, 2 tq + 9)
                    const uint32_t v0[4] = {vv[0].x, vv[0].y, vv[0].z, vv[0].w}, v1[4] = {vv[1].x, vv[1].y, vv[1].z, vv[1].w};
                    const uint32_t v2[4] = {vv[2].x, vv[2].y, vv[2].z, vv[2].w}, v3[4] = {vv[3].x, vv[3].y, vv[3].z, vv[3].w};
#pragma unroll
                    for (int n = 0; n < 8; ++n) {
                        const uint32_t sel = (n & 1) ? 0x7632u : 0x5410u;
                        mma16816(o[n], pa, prmt(v0[n >> 1], v1[n >> 1], sel), prmt(v2[n >> 1], v3[n >> 1], sel));
                    }
                    __syncwarp();
                    if (fetched < pl) fetch();
                }
                if (lane < depth) g_kvpar[buf0 + lane] = par;
                __syncwarp();
                la += __shfl_xor_sync(0xffffffffu, la, 1); la += __shfl_xor_sync(0xffffffffu, la, 2);
                if (kPrompt) { lb += __shfl_xor_sync(0xffffffffu, lb, 1); lb += __shfl_xor_sync(0xffffffffu, lb, 2); }
            }
            // this lane holds, for rows a and b, the dims 16 tq + n (o[n][0], o[n][2]) and 16 tq + 8 + n (o[n][1], o[n][3])
            if (one_round) {
                if (s < ns) {
                    st[0] = ma; st[32] = la;
#pragma unroll
                    for (int n = 0; n < 8; ++n) { st[(4 + 2 * n) * 32] = o[n][0]; st[(5 + 2 * n) * 32] = o[n][1]; }
                    if (two) {
                        st[64] = mb; st[96] = lb;
#pragma unroll
                        for (int n = 0; n < 8; ++n) { st[(20 + 2 * n) * 32] = o[n][2]; st[(21 + 2 * n) * 32] = o[n][3]; }
                    }
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = h ? rb : ra, i = h ? ib : ia;
                    if (!(h ? vb : va) || (h ? Lb : La) <= p0 || s >= ns || b0 + i == skip_row) continue;      // padding row, or a row that ends before this split starts
                    float* dst = M.partial + (((size_t)(b0 + i) * Hq + kvh * G + (r - i * G)) * kMaxSplits + s) * kPartialStride;
                    if (tq == 0) { dst[0] = h ? mb : ma; dst[1] = h ? lb : la; }
#pragma unroll
                    for (int n = 0; n < 8; n += 2) {
                        *reinterpret_cast<float2*>(dst + 2 + 16 * tq + n) = make_float2(o[n][2 * h], o[n + 1][2 * h]);
                        *reinterpret_cast<float2*>(dst + 2 + 16 * tq + 8 + n) = make_float2(o[n][2 * h + 1], o[n + 1][2 * h + 1]);
                    }
                }
            }
        }
        rows_sync_in<kTimed>(M, sy);   // (warps without a split come by here)
        if (ns > 0) {
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(wpt * 32) : "memory");
            if (one_round && wi < 4) {
                // the unit's first four warps combine, one pair of n-tiles each: dims 16 tq + 2 wi, + 1 and + 8
                const float* sk0 = c.xs + (size_t)slot * wpt * (kAttnStage / 4) + lane;
                const int sk_step = share * (kAttnStage / 4);
                float mxa = -INFINITY, mxb = -INFINITY;
                for (int k = 0; k < ns; ++k) {
                    mxa = fmaxf(mxa, sk0[k * sk_step]);
                    if (two) mxb = fmaxf(mxb, sk0[k * sk_step + 64]);
                }
                float om[2][4], sa = 0.f, sb = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) { om[0][e] = 0.f; om[1][e] = 0.f; }
#pragma unroll 1
                for (int k = 0; k < ns; ++k) {
                    const float* sk = sk0 + k * sk_step;
                    const float fa = sk[0] == -INFINITY ? 0.f : ex2(sk[0] - mxa);
                    sa = fmaf(sk[32], fa, sa);
                    float fb = 0.f;
                    if (two) { fb = sk[64] == -INFINITY ? 0.f : ex2(sk[64] - mxb); sb = fmaf(sk[96], fb, sb); }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float* v = sk + (4 + 4 * wi + 2 * h) * 32;
                        om[h][0] = fmaf(v[0], fa, om[h][0]); om[h][1] = fmaf(v[32], fa, om[h][1]);
                        if (two) { om[h][2] = fmaf(v[16 * 32], fb, om[h][2]); om[h][3] = fmaf(v[17 * 32], fb, om[h][3]); }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = h ? rb : ra, i = h ? ib : ia;
                    if (!(h ? vb : va) || b0 + i == skip_row) continue;
                    const float l = fmaxf(h ? sb : sa, 1e-30f);   // (a visible row's sum is at least 1; rows past a prompt see nothing)
                    uint16_t* dst = M.attn + (size_t)(b0 + i) * Hq * kHeadDim + (kvh * G + (r - i * G)) * kHeadDim + 16 * tq + 2 * wi;
                    *reinterpret_cast<uint32_t*>(dst) = pack_bf16(om[0][2 * h] / l, om[1][2 * h] / l);
                    *reinterpret_cast<uint32_t*>(dst + 8) = pack_bf16(om[0][2 * h + 1] / l, om[1][2 * h + 1] / l);
                }
            }
            if (!one_round) {
                for (int pr = wi; pr < nq * G; pr += wpt) {   // a warp per (position, head): lane j holds split j's max and sum, dims 2 lane, 2 lane + 1
                    const int row = b0 + pr / G, hq = kvh * G + pr % G, nr = sp.count(min(L0 + pr / G, cap));
                    if (row == skip_row) continue;
                    const float* base = M.partial + ((size_t)row * Hq + hq) * kMaxSplits * kPartialStride;
                    const float m_l = lane < nr ? ldcg_f32(base + lane * kPartialStride) : -INFINITY;
                    const float l_l = lane < nr ? ldcg_f32(base + lane * kPartialStride + 1) : 0.f;
                    const float mx = warp_max(m_l), sc_l = m_l == -INFINITY ? 0.f : ex2(m_l - mx);
                    float l = 0.f, o0 = 0.f, o1 = 0.f;
                    for (int k = 0; k < nr; ++k) {
                        const float2 v = __ldcg(reinterpret_cast<const float2*>(base + k * kPartialStride + 2 + 2 * lane));
                        const float f = __shfl_sync(0xffffffffu, sc_l, k), w = __shfl_sync(0xffffffffu, l_l, k);
                        l = fmaf(w, f, l); o0 = fmaf(v.x, f, o0); o1 = fmaf(v.y, f, o1);
                    }
                    l = fmaxf(l, 1e-30f);
                    *reinterpret_cast<uint32_t*>(M.attn + (size_t)row * Hq * kHeadDim + hq * kHeadDim + 2 * lane) = pack_bf16(o0 / l, o1 / l);
                }
            }
            fence_proxy_async();   // the states are overwritten by the copy engine
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(wpt * 32) : "memory");
        }
    }
}

// ---- weight phases -------------------------------------------------------------------------------------------------
// A phase's n_out weight rows are tiles of 16 (w1|w3: 8 + 8 rows), packed as mma.m16n8k16 A fragments (smol_rows_pack_kernel:
// 512 bytes per 16 K elements).  A unit is a block of up to `mt` tiles times a group of up to `n` activation rows; both
// numbers come from the host's plan (rows_plan).  A CTA owns one tile block at a time and walks row groups with it.
constexpr int kRowsW = 147456;    // bytes of the weight region: 6 tiles of K = 768
constexpr int kRowsP = 73728;     // bytes of the region in front of it: activation rows, then partial sums; attention states; a logits row
constexpr int kRowsMax = 32;      // activation rows of a unit
constexpr int kRowsTiles = 6;     // tiles of a block
constexpr int kRowsTilesWo = 4;   // ... of the depth transformer's wo
constexpr int kRowsAttn = kWarps * kAttnStage - kRowsP;   // of the weight region that the attention before a slow wo uses
constexpr int kRowsTilesSlowWo = 3;   // tiles of a slow wo block: they lie behind that
static_assert(kRowsW - kRowsAttn >= kRowsTilesSlowWo * 16 * 768 * 2, "wo's tiles beside the attention's keys and values");
constexpr int kChainMax = 12;     // MMAs of a chain in one go (of 16 K elements each): K = 768 per slice; longer ones (odd widths of w2) loop

// What a phase needs and does not depend on data, worked out once per launch (a parameter or constant-bank miss and an
// integer division cost a phase more than its MMAs: 6000 issue slots per phase and SM quarter without these tables).
struct __align__(16) RowsStep {   // one per phase of the program
    const uint16_t* w;        // this CTA's first tile block
    const uint16_t* norm_w;
};
struct __align__(16) RowsKind {   // one per (slow / depth transformer, phase kind)
    const uint16_t* src;      // activation rows, K elements apart
    const uint16_t* res;      // residual rows (wo, w2)
    void* dst;
    int rows, K, tiles, n_out, split, nk;   // K slices of the chains; MMAs of a chain
    int mt, n, blocks, block0, g0, gstep, q_rows, k_end;   // block0 < 0: the CTA has no unit in such a phase
    uint32_t off;             // of the tiles in the weight region
    uint32_t bytes;           // of the first tile block, fetched a phase ahead (w2: 0, its one tile goes straight to registers)
};
__shared__ RowsKind g_rk[2][6];
__shared__ int g_rpos[kRowsMax], g_rpage[kRowsMax];

__device__ void rows_tables(const DevModel& M, const CallArgs& A, const Ctx& c, RowsStep* steps) {
    if (c.tid < 12) {
        const int f = c.tid / 6, kind = c.tid - f * 6;
        RowsKind r;
        const int D = f ? M.fdim : M.dim, F = f ? M.finter : M.inter, Hq = f ? M.fn_head : M.n_head, Hkv = f ? M.fn_kv : M.n_kv;
        uint16_t* stream = f ? M.xf : M.x;
        r.rows = A.batch;
        r.K = kind == PH_W2 ? F : D;
        r.n_out = kind == PH_QKV ? (Hq + 2 * Hkv) * kHeadDim : kind == PH_W13 ? F : kind == PH_HEAD ? (f ? M.codebook_size : M.vocab) : D;
        r.split = kind != PH_WO && kind != PH_W2 ? 1 : r.K % 256 == 0 ? 4 : r.K % 128 == 0 ? 2 : 1;
        r.nk = r.K / r.split / 64;
        r.tiles = kind == PH_W13 ? F >> 3 : (r.n_out + 15) >> 4;
        r.q_rows = Hq * kHeadDim; r.k_end = (Hq + Hkv) * kHeadDim;
        r.src = kind == PH_WO ? M.attn : kind == PH_W13 ? M.h : kind == PH_W2 ? M.act : stream;
        r.res = kind == PH_WO ? stream : M.h;
        r.dst = kind == PH_QKV ? (void*)M.q : kind == PH_WO ? (void*)M.h : kind == PH_W13 ? (void*)M.act
              : kind == PH_W2 ? (void*)stream : f ? (void*)M.depth_logits : (void*)M.token_logits;
        const RowsPlan pl = A.rows_plan[f][kind];
        r.mt = max(1, (int)pl.mt); r.n = max(1, (int)pl.n);
        r.blocks = (r.tiles + r.mt - 1) / r.mt;
        if (r.blocks <= c.n_ctas) {      // one tile block per CTA; the CTAs that share one take turns at the row groups
            r.gstep = c.n_ctas / r.blocks;
            r.g0 = c.cta / r.blocks;
            r.block0 = r.g0 < r.gstep && r.g0 * r.n < r.rows ? c.cta - r.g0 * r.blocks : -1;
        } else {
            r.gstep = 1; r.g0 = 0; r.block0 = c.cta;
        }
        r.off = kind == PH_WO && !f ? (uint32_t)kRowsAttn : 0u;
        r.bytes = kind == PH_W2 || r.block0 < 0 ? 0u : (uint32_t)(min(r.mt, r.tiles - r.block0 * r.mt) * r.K) * 32u;
        g_rk[f][kind] = r;
    }
    __syncthreads();
    for (int p = A.phase_begin + c.tid; p < A.phase_end; p += kThreads) {
        const Phase ph = unpack_phase(M.prog[p]);
        RowsStep s;
        s.w = nullptr; s.norm_w = nullptr;
        if (ph.kind != PH_ATTN && ph.kind != PH_SAMPLE) {
            const RowsKind& r = g_rk[ph.fast][ph.kind];
            const DevLayer& L = ph.fast ? M.fast_layers[ph.layer] : M.layers[ph.layer];
            const RowsLayer& W = ph.fast ? M.rows_fast_layers[ph.layer] : M.rows_layers[ph.layer];
            s.w = ph.kind == PH_QKV ? W.wqkv : ph.kind == PH_WO ? W.wo : ph.kind == PH_W13 ? W.w13 : ph.kind == PH_W2 ? W.w2
                : ph.fast ? M.rows_fast_output + (M.depthwise_output ? (size_t)ph.depth_pos * r.tiles * 16 * r.K : 0) : M.rows_head;
            s.norm_w = ph.kind == PH_QKV ? L.attention_norm : ph.kind == PH_W13 ? L.ffn_norm : ph.fast ? M.fast_norm : M.norm;
            if (r.block0 >= 0) s.w += (size_t)r.block0 * r.mt * 16 * r.K;
        }
        steps[p - A.phase_begin] = s;
    }
    __syncthreads();
}

// One thread: weight tiles -> the weight region, completing on g_mbar[0].  Nobody reads the region any more.
__device__ __forceinline__ void rows_issue(unsigned char* stage, const uint16_t* w, uint32_t bytes) {
    if (bytes == 0u) return;
    fence_proxy_async();
    mbar_expect_tx(&g_mbar[0], bytes);
    bulk_g2s(stage, w, bytes, &g_mbar[0]);
}
// The first tiles of the launch's next weight phase.
__device__ __forceinline__ void rows_issue_next(const DevModel& M, const RowsSync& sy, const RowsStep* step, unsigned char* stage) {
    if (sy.next < 0) return;
    const Phase ph = unpack_phase(M.prog[sy.next]);
    rows_issue(stage + g_rk[ph.fast][ph.kind].off, step[sy.next - sy.phase].w, g_rk[ph.fast][ph.kind].bytes);
}

// Token embedding of the pending columns -> the slow residual stream (P:205-221), once per frame.
// Gathered inside the QKV tiles it would be nine row loads per chunk in every tile block.
__device__ __noinline__ void rows_embed(const DevModel& M, const CallArgs& A, const Ctx& c) {
    const int nch = M.dim >> 3;
    for (int i = c.cta * kThreads + c.tid; i < A.batch * nch; i += c.n_ctas * kThreads) {
        const int bg = i / nch, ch = i - bg * nch;
        float x[8];
        embed_chunk(M, A, c, bg, ch, x);
        *reinterpret_cast<uint4*>(M.x + (size_t)bg * M.dim + ch * 8) = pack8(x);
    }
}

// Depth attention of one query head by a warp, in the arithmetic and the order of additions of fast_attention_rows: fp32 FMAs, four lanes per
// position with 16 dims each (position lane / 4, and + 8 where `deep`), one softmax with the true maximum, probabilities rounded to bf16 for
// P V while the row sum keeps the unrounded values (P:559-566).  Returns dims 2 lane, 2 lane + 1.  q: the lane's 16 dims; k: of its
// positions; v: its two dims of all positions (zeros past depth_pos).
template <bool deep>
__device__ __forceinline__ uint32_t depth_head(const uint4 (&q)[2], const uint4 (&k)[deep ? 2 : 1][2], const uint32_t (&v)[deep ? 16 : 8], int depth_pos, int lane) {
    constexpr int H = deep ? 2 : 1;
    const int jl = lane >> 2;
    float qf[16], sc[H];
    unpack8(q[0], *reinterpret_cast<float(*)[8]>(qf));
    unpack8(q[1], *reinterpret_cast<float(*)[8]>(qf + 8));
#pragma unroll
    for (int h = 0; h < H; ++h) {
        float k0[8], k1[8], s = 0.f;
        unpack8(k[h][0], k0);
        unpack8(k[h][1], k1);
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(qf[e], k0[e], s);
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(qf[8 + e], k1[e], s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        sc[h] = jl + 8 * h <= depth_pos ? s * 0.125f : -INFINITY;
    }
    float m = deep ? fmaxf(sc[0], sc[H - 1]) : sc[0];
    asm volatile("redux.sync.max.f32 %0, %0, 0xffffffff;" : "+f"(m));
    float pe[H], pb[H];
#pragma unroll
    for (int h = 0; h < H; ++h) { pe[h] = jl + 8 * h <= depth_pos ? expf(sc[h] - m) : 0.f; pb[h] = bf16_round(pe[h]); }
    float l = deep ? pe[0] + pe[H - 1] : pe[0];
    l += __shfl_xor_sync(0xffffffffu, l, 4);
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8 * H; ++j) {
        const float p = __shfl_sync(0xffffffffu, pb[j / 8], (j & 7) * 4);
        o0 = fmaf(p, bf_lo(v[j]), o0);
        o1 = fmaf(p, bf_hi(v[j]), o1);
    }
    const float inv = __frcp_rn(l);
    return pack_bf16(o0 * inv, o1 * inv);
}
// kp: a kv head's first key; `kvw` elements from position to position, the values behind `depth` keys
template <bool deep>
__device__ __forceinline__ void depth_load(const uint16_t* kp, int kvw, int depth, int depth_pos, int lane, uint4 (&k)[deep ? 2 : 1][2], uint32_t (&v)[deep ? 16 : 8]) {
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    const uint16_t* vp = kp + (size_t)depth * kvw + 2 * lane;
#pragma unroll
    for (int h = 0; h < (deep ? 2 : 1); ++h) {
        const int j = (lane >> 2) + 8 * h;
        const uint16_t* kr = kp + (size_t)j * kvw + (lane & 3) * 16;
        k[h][0] = j <= depth_pos ? ldcg_v4(kr) : z;
        k[h][1] = j <= depth_pos ? ldcg_v4(kr + 8) : z;
    }
#pragma unroll
    for (int j = 0; j < (deep ? 16 : 8); ++j) v[j] = j <= depth_pos ? ldcg_u32(vp + (size_t)j * kvw) : 0u;
}

// Depth attention of rows [r0, r0 + n_live) by one CTA, a warp per (row, kv head), which goes through the kv head's G query heads.  The
// result goes to shared memory as bf16 rows (`stride` bytes apart), where the wo tiles of this CTA read it, and, where `copy` is given,
// to its rows of M.attn.  Every tile block of wo repeats it: for 8 rows that is two tasks per warp, less than the barrier that a
// step of its own would need.  4.0 us of the 6.9 of such a phase at 64 rows (150m), a chain of loads, FMAs and shuffles per head; the heads side
// by side, two tasks at once, or more loads ahead spill and take longer (frames of 64, us: 1451, and 1513 to 1717).
template <bool deep>   // deep: positions 8 .. 15 exist
__device__ __forceinline__ void rows_depth_attention(const DevModel& M, int layer, int depth_pos, int r0, int n_live, unsigned char* out, int stride, uint16_t* copy) {
    const int Hq = M.fn_head, Hkv = M.fn_kv, G = Hq / Hkv, kvw = Hkv * kHeadDim, depth = M.depth, n_flayer = M.n_flayer;
    const uint16_t* q0 = M.q;
    const uint16_t* kv0 = M.fkv;
    const int tid = tid_here(), warp = tid >> 5, lane = tid & 31;
#pragma unroll 1
    for (int task = warp; task < n_live * Hkv; task += kWarps) {
        const int row = task / Hkv, kvh = task - row * Hkv;
        const uint16_t* qp = q0 + ((size_t)(r0 + row) * Hq + kvh * G) * kHeadDim + (lane & 3) * 16;
        uint4 k[deep ? 2 : 1][2], q[2] = {ldcg_v4(qp), ldcg_v4(qp + 8)};
        uint32_t v[deep ? 16 : 8];
        depth_load<deep>(kv0 + ((size_t)((r0 + row) * n_flayer + layer) * 2) * depth * kvw + kvh * kHeadDim, kvw, depth, depth_pos, lane, k, v);
        int at = kvh * G * kHeadDim + 2 * lane;
#pragma unroll 1
        for (int g = 0; g < G; ++g, at += kHeadDim) {
            uint4 next[2] = {q[0], q[1]};
            qp += kHeadDim;
            if (g + 1 < G) { next[0] = ldcg_v4(qp); next[1] = ldcg_v4(qp + 8); }
            const uint32_t r = depth_head<deep>(q, k, v, depth_pos, lane);
            *reinterpret_cast<uint32_t*>(out + (size_t)row * stride + at * 2) = r;
            if (copy != nullptr) *reinterpret_cast<uint32_t*>(copy + (size_t)row * Hq * kHeadDim + at) = r;
            q[0] = next[0]; q[1] = next[1];
        }
    }
}

// two fp32 numbers per instruction
__device__ __forceinline__ unsigned long long f2_pack(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void f2_split(unsigned long long v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
// RMSNorm of two elements (P:601-613): fp32 normalise, round to bf16, multiply by the bf16 weight, round again
__device__ __forceinline__ uint32_t rows_norm2(uint32_t x, unsigned long long r, uint32_t w) {
    float a, b;
    f2_split(f2_mul(f2_pack(bf_lo(x), bf_hi(x)), r), a, b);
    __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    p = __hmul2_rn(p, *reinterpret_cast<__nv_bfloat162*>(&w));
    return *reinterpret_cast<uint32_t*>(&p);
}

// A chain's partial sums of a tile: [16 weight rows][N activation rows] fp32.  Fragment stores (8 weight rows x 4 pairs) and the
// epilogue's loads (4 weight rows x 4 pairs of activation rows per half warp) meet different banks through an XOR of
// the activation row.
template <int N>
__device__ __forceinline__ int part_at(int w, int b) {
    return w * N + (b ^ (N == 32 ? 8 * ((w ^ (w >> 2)) & 3) : N == 16 ? 8 * ((w >> 1) & 1) : 0));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
constexpr int kNormSteps = 3;   // RMSNorm of a row by a warp: 256 elements per step

// One weight phase: tiles of 16 weight rows times groups of up to 8 NT activation rows.  A dot product is four chains of MMAs
// (K steps 0, 4, 8 .. of 16 elements; 1, 5, 9 ..; ..) for each K slice: one slice, or four for wo and w2.  Without slices the
// warps are the four chains x 4, which take every fourth tile; with slices a warp is one chain and takes all tiles.  The one
// tile of a w2 block sits in registers.
// kTimed: the profiling build of the kernel, which stamps rows in place | normed | chains | sums and epilogue.
template <int kind, bool kDepthAttn, int NT, bool kTimed>
__device__ __forceinline__ void rows_gemm(const DevModel& M, const CallArgs& A, const int iter, const uint32_t packed_phase, const RowsStep* step,
                                          unsigned char* stage, float* P, RowsSync& sy) {
    constexpr bool wide = kind == PH_W2;
    constexpr bool split = kind == PH_W2 || kind == PH_WO;
    constexpr int N = NT * 8;
    constexpr int kTile = N * 16;                              // floats of a chain's tile
    constexpr int TW = wide ? 1 : split ? kRowsTilesWo : (kRowsTiles + 3) / 4;   // tiles of a warp
    constexpr int KG = split ? 16 : 4;                         // chains, at most
    static_assert(N <= kRowsMax && (split ? 16 * kTile : 4 * kRowsTiles * kTile) * 4 <= kRowsP, "partial sums of a unit do not fit");
    constexpr bool normed = kind == PH_QKV || kind == PH_W13 || kind == PH_HEAD;
    const Phase ph = unpack_phase(packed_phase);
    const bool fast = ph.fast != 0;
    // (volatile: fields are read where they are used; kept in registers across the loops they would be spilled, and a spilled
    // value waits for the load that produced it)
    const volatile RowsKind& rk = g_rk[ph.fast][kind];
    unsigned char* rows_s = reinterpret_cast<unsigned char*>(P);
    const int tid = tid_here(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, cc = lane & 3;
    const int K = rk.K, nk = rk.nk;
    const int stride_s = K * 2 + 16;   // rows in shared memory: ldmatrix of 8 rows hits all banks
    // chain of MMAs: 16-element steps k0, k0 + 4, ..; tiles t_lo, t_lo + t_step, ..
    const int chain = split ? warp : (warp & 3), t_lo = split ? 0 : (warp >> 2), t_step = split ? 1 : 4;
    const int k0 = split ? (warp >> 2) * nk * 4 + (warp & 3) : chain;
    const bool idle = split && warp >= 4 * rk.split;
    // the first QKV of a depth step reads the slow hidden state or the previous code's embedding (G:136-140) and leaves the
    // row behind as the depth transformer's residual stream
    const bool depth_in = kind == PH_QKV && fast && ph.layer == 0 && !A.fast_from_xf;
    bool landed = false;

    int block = rk.block0, r0 = rk.g0 * rk.n;
#pragma unroll 1
    for (;;) {
        const int n_live = min(rk.n, rk.rows - r0);
        // ---- before the previous phase is complete: what does not depend on it ----
        uint4 af[wide ? kChainMax : 1];   // w2: the chain's part of the block's tile
        if (wide) {
            const uint4* wp = reinterpret_cast<const uint4*>(step->w + (size_t)(block - rk.block0) * 16 * K) + k0 * 32 + lane;
#pragma unroll
            for (int i = 0; i < kChainMax; ++i) af[i] = i < nk && !idle ? ldg_stream(wp + i * 128) : make_uint4(0u, 0u, 0u, 0u);
        }
        uint4 wv[normed ? kNormSteps : 1];
        if (normed) {
#pragma unroll
            for (int i = 0; i < kNormSteps; ++i)
                wv[i] = (lane + 32 * i) * 8 < K ? __ldg(reinterpret_cast<const uint4*>(step->norm_w) + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (kind == PH_QKV && !fast && tid >= kThreads - 32 && tid - (kThreads - 32) < n_live) {
            Ctx c;   // cache slot of the row (lengths and tables are settled a barrier before the frame's first layer): page (-1: nothing is appended) and position
            c.iter = iter;
            const int i = tid - (kThreads - 32), bg = r0 + i, bs = row_seq(A, bg);
            const int p = ldcg_i32(A.b.seq_len + bs) + row_off(A, bg);
            int page = -1;
            if (seq_active(M, A, c, bg) && p < A.b.max_pages * M.page_size)
                page = ldcg_i32(A.b.block_table + (size_t)bs * A.b.max_pages + p / M.page_size);
            g_rpos[i] = p; g_rpage[i] = page;
        }
        if (!wide && !landed) { rows_wait(M, &g_mbar[0], sy.par_w); sy.par_w ^= 1u; landed = true; }
        rows_sync_in<kTimed>(M, sy);
        const bool timed = kTimed && blockIdx.x == 0 && tid == 0;
        unsigned long long stamp = 0ull;
        if (timed) stamp = globaltimer_ns();
        // ---- the group's rows: bulk copies into shared memory (contiguous 16-byte loads take 3400 clocks for 96 KB on every SM
        // at once, loads straight into fragments -- 64 bytes of 8 rows each -- 7000, bulk copies 2000) ----
        if (kDepthAttn) {
            uint16_t* copy = block == 0 ? M.attn + (size_t)(uint32_t)(r0 * K) : nullptr;
            if (ph.depth_pos < 8) rows_depth_attention<false>(M, ph.layer, ph.depth_pos, r0, n_live, rows_s, stride_s, copy);
            else rows_depth_attention<true>(M, ph.layer, ph.depth_pos, r0, n_live, rows_s, stride_s, copy);
            __syncthreads();
        } else if (lane == 0) {
            if (warp < n_live) {
                fence_proxy_async_global();   // rows written by st.global in other CTAs, read by the copy engine
                if (warp == 0) mbar_expect_tx(&g_mbar[1], (uint32_t)(n_live * K) * 2u);
#pragma unroll 1
                for (int row = warp; row < n_live; row += kWarps) {
                    const uint16_t* src = rk.src + (size_t)(uint32_t)((r0 + row) * K);
                    if (depth_in) {
                        src = M.x + (size_t)(uint32_t)((r0 + row) * K);
                        if (ph.depth_pos > 0) {
                            const int code = ldcg_i32(M.frame_tokens + (size_t)(r0 + row) * M.n_rows + ph.depth_pos);
                            const int off = M.depthwise_wte ? (M.dup0 ? ph.depth_pos - 1 : ph.depth_pos) * M.codebook_size : 0;
                            src = M.fast_embeddings + (size_t)(uint32_t)((code + off) * K);
                        }
                    }
                    bulk_g2s(rows_s + row * stride_s, src, (uint32_t)K * 2u, &g_mbar[1]);
                }
            }
        }
        const int nt = wide ? 1 : min(rk.mt, rk.tiles - block * rk.mt);
        // An item of the epilogue: the sums of one weight row (w1|w3: of both) for two activation rows; then lanes of neighbouring
        // weight rows swap, and each finishes the pair of outputs of one activation row.
        constexpr int NB4 = N / 8, kWB = kind == PH_W13 ? 1 : 2;    // groups of four pairs of activation rows; of four weight rows: 2 kWB
        const auto item_w = [](int idx) { return (idx & 3) + 4 * ((idx >> 4) % (2 * kWB)); };
        const auto item_b = [](int idx) { return 2 * (((idx >> 2) & 3) + 4 * ((idx >> 4) / (2 * kWB) % NB4)); };
        const auto item_t = [](int idx) { return (idx >> 4) / (2 * kWB) / NB4; };
        uint32_t pre = 0u;                                          // the first item's residual pair: in flight before the sums exist
        if (split) {
            const int row = item_b(tid) + (tid & 1), t = item_t(tid);
            if (t < nt && row < n_live)
                pre = ldcg_u32(rk.res + (size_t)(uint32_t)((r0 + row) * rk.n_out + ((block * rk.mt + t) * 16 + (item_w(tid) & ~1))));
        }
        if (!kDepthAttn) { rows_wait(M, &g_mbar[1], sy.par_x); sy.par_x ^= 1u; }
        if (timed) rows_stamp(M, kind, ph.fast, 0, stamp);
        if (normed) {
            // a warp per row, two at a time: their chains of shuffles and divisions run side by side
            constexpr int NR = N > kWarps ? 2 : 1;
            unsigned char* rp[NR];
            uint4 v[NR][kNormSteps];       // (arrays are always written whole: one that a loop may leave as it was stays live through it)
            float ss[NR][kNormSteps];      // sums over 256 elements each, added in order
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                rp[u] = rows_s + min(warp + u * kWarps, n_live - 1) * stride_s + lane * 16;
#pragma unroll
                for (int i = 0; i < kNormSteps; ++i) {
                    v[u][i] = (lane + 32 * i) * 8 < K ? *reinterpret_cast<const uint4*>(rp[u] + i * 512) : make_uint4(0u, 0u, 0u, 0u);
                    float f[8], t = 0.f;
                    unpack8(v[u][i], f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) t = fmaf(f[e], f[e], t);
                    ss[u][i] = t;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int u = 0; u < NR; ++u) {
#pragma unroll
                    for (int i = 0; i < kNormSteps; ++i) ss[u][i] += __shfl_xor_sync(0xffffffffu, ss[u][i], o);
                }
            }
#pragma unroll
            for (int u = 0; u < NR; ++u) {
#pragma unroll
                for (int i = 1; i < kNormSteps; ++i) ss[u][0] = __fadd_rn(ss[u][0], ss[u][i]);
                ss[u][0] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss[u][0], (float)K), M.eps)));
            }
            const bool keep = depth_in && block == 0;
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int row = warp + u * kWarps;
                if (row < n_live) {
                    const unsigned long long r2 = f2_pack(ss[u][0], ss[u][0]);
                    uint16_t* kp = M.xf + (size_t)(uint32_t)((r0 + row) * K) + lane * 8;
#pragma unroll
                    for (int i = 0; i < kNormSteps; ++i) {
                        if ((lane + 32 * i) * 8 < K) {
                            uint4& w = v[u][i];
                            if (keep) *reinterpret_cast<uint4*>(kp + i * 256) = w;
                            w.x = rows_norm2(w.x, r2, wv[i].x); w.y = rows_norm2(w.y, r2, wv[i].y);
                            w.z = rows_norm2(w.z, r2, wv[i].z); w.w = rows_norm2(w.w, r2, wv[i].w);
                            *reinterpret_cast<uint4*>(rp[u] + i * 512) = w;
                        }
                    }
                }
            }
            __syncthreads();
            if (kind == PH_QKV) {   // the first item's RoPE pair (P:616-640): never past the table (host checks bound the position)
                const int row = item_b(tid) + (tid & 1), u0 = (block * rk.mt + item_t(tid)) * 16 + (item_w(tid) & ~1);
                if (u0 < rk.k_end && row < n_live)
                    pre = __ldg(reinterpret_cast<const uint32_t*>((fast ? M.fast_rope : M.rope) + (size_t)(fast ? ph.depth_pos : min(g_rpos[row], M.max_seq_len - 1)) * kHeadDim + (u0 & (kHeadDim - 1))));
            }
        }
        if (timed) rows_stamp(M, kind, ph.fast, 1, stamp);
        // ---- the warp's chains (columns past the group repeat its last row: nobody reads their sums) ----
        float acc[TW][NT][4];
#pragma unroll
        for (int t = 0; t < TW; ++t) {
#pragma unroll
            for (int j = 0; j < NT; ++j) { acc[t][j][0] = 0.f; acc[t][j][1] = 0.f; acc[t][j][2] = 0.f; acc[t][j][3] = 0.f; }
        }
        if (!idle) {
            // ldmatrix: lanes 0-7 the rows' first 16 bytes of a step, 8-15 the second; 16-31 the same of the next 8 rows
            uint32_t src[(NT + 1) / 2];
#pragma unroll
            for (int j = 0; j < (NT + 1) / 2; ++j)
                src[j] = smem_u32(rows_s) + (uint32_t)(min(16 * j + (lane & 7) + 8 * (lane >> 4), n_live - 1) * stride_s + ((lane >> 3) & 1) * 16 + k0 * 32);
            const unsigned char* wt = stage + rk.off + (uint32_t)(t_lo * (K >> 4) + k0) * 512u + lane * 16;
            const uint32_t tile_b = (uint32_t)(t_step * (K >> 4)) * 512u;
#pragma unroll 1
            for (int k = 0; k < nk; k += kChainMax) {
#pragma unroll
                for (int i = 0; i < kChainMax; ++i) {
                    if (wide && k > 0)
                        af[wide ? i : 0] = k + i < nk ? ldg_stream(reinterpret_cast<const uint4*>(step->w + (size_t)(block - rk.block0) * 16 * K) + k0 * 32 + lane + (k + i) * 128)
                                                      : make_uint4(0u, 0u, 0u, 0u);
                    if (k + i < nk) {
                        uint32_t x[(NT + 1) / 2][4];
#pragma unroll
                        for (int j = 0; j < (NT + 1) / 2; ++j) ldsm_x4(x[j], src[j] + (k + i) * 128);
#pragma unroll
                        for (int t = 0; t < TW; ++t) {
                            if (wide || t_lo + t * t_step < nt) {
                                const uint4 a = wide ? af[wide ? i : 0] : *reinterpret_cast<const uint4*>(wt + t * tile_b + (k + i) * 2048);
#pragma unroll
                                for (int j = 0; j < NT; ++j) mma_bf16_16816(acc[t][j], a.x, a.y, a.z, a.w, x[j >> 1][2 * (j & 1)], x[j >> 1][2 * (j & 1) + 1]);
                            }
                        }
                    }
                }
            }
        }
        // ---- partial sums of the chains, then their sum and the phase's epilogue ----
        const bool last_rows = r0 + rk.gstep * rk.n >= rk.rows;
        const int next_block = block + (rk.blocks <= (int)gridDim.x ? rk.blocks : (int)gridDim.x);
        __syncthreads();   // the rows have been read: their place takes the partial sums
        if (timed) rows_stamp(M, kind, ph.fast, 2, stamp);
        if (!idle) {
#pragma unroll
            for (int t = 0; t < TW; ++t) {
                const int tl = t_lo + t * t_step;
                if (!wide && tl >= nt) continue;
                float* pt = P + (tl * KG + chain) * kTile;
#pragma unroll
                for (int j = 0; j < NT; ++j) {   // weight rows g, g + 8 of activation rows 2 cc, 2 cc + 1
                    *reinterpret_cast<float2*>(pt + part_at<N>(g, 8 * j + 2 * cc)) = make_float2(acc[t][j][0], acc[t][j][1]);
                    *reinterpret_cast<float2*>(pt + part_at<N>(g + 8, 8 * j + 2 * cc)) = make_float2(acc[t][j][2], acc[t][j][3]);
                }
            }
        }
        __syncthreads();
        if (last_rows && tid == kThreads - 32) {   // the block's weights are used up: fetch the next ones
            if (next_block < rk.blocks) {
                if (!wide) rows_issue(stage + rk.off, step->w + (size_t)(next_block - rk.block0) * rk.mt * 16 * K, (uint32_t)(min(rk.mt, rk.tiles - next_block * rk.mt) * K) * 32u);
            } else {
                rows_issue_next(M, sy, step, stage);
            }
        }
        const int D = rk.n_out;
        unsigned char* const dst = reinterpret_cast<unsigned char*>(rk.dst);
#pragma unroll 1
        for (int idx = tid; idx < nt * (NB4 * kWB * 32); idx += kThreads) {   // (whole warps: a multiple of 32)
            const int wr = item_w(idx), rw = item_b(idx), t = item_t(idx), odd = idx & 1;
            const float* pp = P + t * KG * kTile;
            auto sum = [&](int w, float (&o)[2]) {
                const float* q = pp + part_at<N>(w, rw);
                unsigned long long v = 0ull;
#pragma unroll
                for (int k = 0; k < KG; k += 4) {   // a slice's four chains in order, the slices in order
                    if (split && k >= 4 * rk.split) continue;
                    unsigned long long u = *reinterpret_cast<const unsigned long long*>(q + k * kTile);
#pragma unroll
                    for (int e = 1; e < 4; ++e) u = f2_add(u, *reinterpret_cast<const unsigned long long*>(q + (k + e) * kTile));
                    v = k == 0 ? u : f2_add(v, u);
                }
                f2_split(v, o[0], o[1]);
            };
            float o[2];
            sum(wr, o);
            o[0] = bf16_round(o[0]); o[1] = bf16_round(o[1]);
            if (kind == PH_W13) {   // F.silu in fp32, bf16 out (P:581)
                float u[2];
                sum(wr + 8, u);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    o[h] = __fmul_rn(bf16_round(__fdiv_rn(o[h], __fadd_rn(1.0f, expf(-o[h])))), bf16_round(u[h]));
            }
            const float got = __shfl_xor_sync(0xffffffffu, odd ? o[0] : o[1], 1);
            float v0 = odd ? got : o[0], v1 = odd ? o[1] : got;   // outputs u0, u0 + 1 of one activation row
            const int row = rw + odd, b = r0 + row, tile = block * rk.mt + t;
            if (row >= n_live) continue;
            if (kind == PH_W13) {
                *reinterpret_cast<uint32_t*>(dst + (size_t)(uint32_t)(b * D + tile * 8 + (wr & ~1)) * 2) = pack_bf16(v0, v1);
                continue;
            }
            const int u0 = tile * 16 + (wr & ~1);
            if (kind == PH_HEAD) {
                float* out = reinterpret_cast<float*>(dst) + (fast ? ((size_t)b * M.depth + ph.depth_pos) * D : (size_t)b * D);
                if (u0 < D) out[u0] = v0;
                if (u0 + 1 < D) out[u0 + 1] = v1;
                continue;
            }
            uint32_t pv = pre;
            const bool ahead = idx == tid;
            if (kind != PH_QKV) {   // wo: h = stream + wo(attn) (P:499); w2: stream = h + w2(act) (P:500)
                const size_t at = (size_t)(uint32_t)(b * D + u0);
                if (!ahead) pv = ldcg_u32(rk.res + at);
                *reinterpret_cast<uint32_t*>(dst + 2 * at) = pack_bf16(__fadd_rn(bf_lo(pv), v0), __fadd_rn(bf_hi(pv), v1));
                continue;
            }
            const int p = fast ? ph.depth_pos : g_rpos[row], k_end = rk.k_end, q_rows = rk.q_rows;
            if (u0 < k_end) {  // q and k rows: interleaved-pair RoPE with the bf16 table (P:616-640)
                if (!ahead) pv = __ldg(reinterpret_cast<const uint32_t*>((fast ? M.fast_rope : M.rope) + (size_t)(fast ? p : min(p, M.max_seq_len - 1)) * kHeadDim + (u0 & (kHeadDim - 1))));
                const float co = bf_lo(pv), si = bf_hi(pv);
                const float r0f = bf16_round(__fsub_rn(__fmul_rn(v0, co), __fmul_rn(v1, si)));
                const float r1f = bf16_round(__fadd_rn(__fmul_rn(v1, co), __fmul_rn(v0, si)));
                v0 = r0f; v1 = r1f;
            }
            const uint32_t packed = pack_bf16(v0, v1);
            if (u0 < q_rows) {
                *reinterpret_cast<uint32_t*>(dst + (size_t)(uint32_t)(b * q_rows + u0) * 2) = packed;
                continue;
            }
            const int is_v = u0 >= k_end ? 1 : 0, kvw = k_end - q_rows;
            const int n1 = u0 - (is_v ? k_end : q_rows);
            if (fast) {
                *reinterpret_cast<uint32_t*>(M.fkv + (((size_t)(b * M.n_flayer + ph.layer) * 2 + is_v) * M.depth + ph.depth_pos) * kvw + n1) = packed;
            } else if (g_rpage[row] >= 0) {
                const int ps = M.page_size, kvh = n1 / kHeadDim, d = n1 & (kHeadDim - 1);
                *reinterpret_cast<uint32_t*>(M.kv_pool + ((((size_t)g_rpage[row] * M.n_layer + ph.layer) * 2 + is_v) * M.n_kv + kvh) * ((size_t)ps * kHeadDim)
                                             + (size_t)(p & (ps - 1)) * kHeadDim + d) = packed;
            }
        }
        if (timed) rows_stamp(M, kind, ph.fast, 3, stamp);
        if (!last_rows || next_block < rk.blocks) {   // the partial sums are overwritten, by copies
            fence_proxy_async();
            __syncthreads();
        }
        if (!last_rows) { r0 += rk.gstep * rk.n; continue; }
        if (next_block >= rk.blocks) break;
        block = next_block;
        r0 = rk.g0 * rk.n;
        landed = false;
    }
}

// One weight phase: the kernel form its plan names.  The CTA's first tiles are on their way (`step`); the tiles of
// the launch's next weight phase are fetched as soon as these are used up.
template <bool kTimed>
__device__ __forceinline__ void phase_rows(const DevModel& M, const CallArgs& A, const Ctx& c, uint32_t packed_phase, RowsSync& sy, const RowsStep* step) {
    const Phase ph = unpack_phase(packed_phase);
    if (tc_has_prestep(ph)) {
        rows_sync_in<kTimed>(M, sy);
        if (A.tc_part == 0 || A.tc_part == 1) rows_embed(M, A, c);
        if (A.cooperative) rows_arrive<kTimed>(M, c, sy);
        if (A.tc_part == 1) return;
    }
    if (ph.kind == PH_QKV && !ph.fast) attn_prefetch(M, A, c, ph.layer);
    if (g_rk[ph.fast][ph.kind].block0 < 0) {   // no unit here: the weight region is free for the phase that follows
        if (c.tid == kThreads - 32) rows_issue_next(M, sy, step, c.stage);
        rows_sync_in<kTimed>(M, sy);
        return;
    }
    const int n = g_rk[ph.fast][ph.kind].n;
#define ROWS_ARGS M, A, c.iter, packed_phase, step, c.stage, c.xs, sy
#define ROWS_CASE(kind, attn) \
    if (n <= 8) rows_gemm<kind, attn, 1, kTimed>(ROWS_ARGS); \
    else if (n <= 16) rows_gemm<kind, attn, 2, kTimed>(ROWS_ARGS); \
    else rows_gemm<kind, attn, 4, kTimed>(ROWS_ARGS);
    switch (ph.kind) {
        case PH_QKV: ROWS_CASE(PH_QKV, false) break;
        case PH_W13: ROWS_CASE(PH_W13, false) break;
        case PH_HEAD: ROWS_CASE(PH_HEAD, false) break;
        case PH_W2:
            if (n <= 8) rows_gemm<PH_W2, false, 1, kTimed>(ROWS_ARGS);
            else if (n <= 16) rows_gemm<PH_W2, false, 2, kTimed>(ROWS_ARGS);
            else rows_gemm<PH_W2, false, 3, kTimed>(ROWS_ARGS);
            break;
        default:
            if (ph.fast) { ROWS_CASE(PH_WO, true) }
            else { ROWS_CASE(PH_WO, false) }
    }
#undef ROWS_CASE
#undef ROWS_ARGS
}

}  // namespace smol
