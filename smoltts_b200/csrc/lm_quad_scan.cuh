// The recurrences' scan for short prompts, four tokens at a time (included by lm_kernels.cu after lm_delta_mlstm.cuh; long ones: lm_chunk_scan.cuh).  Everything is fp32.
//
// The generalized delta rule and the linear attentions act on a head's state S [d, dv] as
//     S <- diag(w) S - a (u^T S) + k v^T,     o = S^T r
// with per-token vectors over the d key channels (the generalized delta rule; the linear attentions without a and u).  With S the state before four tokens and W(i, j] the product of the
// decays of tokens i + 1 .. j, everything token t needs of the key channels follows from sums that all read the same S,
//     seen_t = (W(0, t-1] u_t)^T S + sum_(s<t) [-(W(s, t-1] u_t).a_s seen_s + (W(s, t-1] u_t).k_s v_s],
//     o_t    = (W(0, t] r_t)^T S   + sum_(s<=t) [-(W(s, t] r_t).a_s seen_s + (W(s, t] r_t).k_s v_s],
// and the four leave  S <- W(0, 4] S + sum_s [-(W(s, 4] a_s) seen_s + (W(s, 4] k_s) v_s].  The decays are at most one, so nothing is
// divided and nothing grows.
//
// quad_prep_kernel makes the scaled vectors and the products between a group's tokens, one record per (group, head); it is parallel over the
// whole prompt.  quad_scan_kernel is what is left to do in order: per group eight sums over the key channels, reduced across lanes side
// by side (the latency of the shuffles is paid once per four tokens), a small triangle, one update.
// What bounds it is that chain; a head's value columns never mix, so blocks take eight columns each on two warps, and a warp has its
// scheduler to itself.  Eight lanes share a column, each with DK / 8 state rows in registers as pairs for the packed FMA.  A third warp
// keeps the records coming through a ring, a few groups per bulk copy; the groups of a copy are unrolled without a barrier between them, so
// that the next group's vectors are read while the current one's sums are reduced.  (Measured and dropped: a barrier wait per group, 1390
// clocks a group against 760; block barriers and copies issued by the computing warps, 850; the vectors in registers a group ahead, 780.)
// 2048 tokens, 12 heads of 64 x 64: 197 us (and 23 for the records) against 370 token by token for the generalized delta rule; of 128 x 128,
// 1801 tokens: 364 (45) against 527; gated linear recurrence, 1024 tokens of 12 x 64 x 64: 66 (4) against 117.  The gated delta rule and the
// mLSTM stay on group_scan_kernel, whose records are smaller: 101 and 120 us per 1000 tokens there, 103 and 121 here.
#pragma once

namespace smol {
namespace lm {

constexpr int kQuad = 4;                 // tokens of a group
constexpr int kQuadMinTokens = 32;       // fewer tokens in every sequence: the scans without a record
constexpr int kQuadMeanTokens = 16;      // fewer tokens per sequence in the mean: likewise
constexpr int kQuadLanes = 8, kQuadCols = 8, kQuadThreads = kQuadLanes * kQuadCols + 32;
constexpr int kQuadRing = 4;             // copies of the ring
__host__ __device__ constexpr int quad_chunk(int DK) { return DK <= 64 ? 4 : DK <= 128 ? 2 : 1; }      // groups per copy
enum { kFormGeneral = 0, kFormAdd = 1 };      // with a and u, without them
// A record: vectors over the key channels, [.][DK] each, then the products.
//   general: W(0,t-1] u_t [4] | W(0,t] r_t [4] | -W(s,4] a_s [4] | W(s,4] k_s [4] | W(0,4];  products [4 t][-a.u [4 s] | k.u [4] | -a.r [4] | k.r [4]]
//   add:     W(0,t] r_t [4] | W(s,4] k_s [4] | W(0,4];                                        products [4 t][k.r [4 s]]
__host__ __device__ constexpr int quad_vecs(int form) { return form == kFormGeneral ? 17 : 9; }
__host__ __device__ constexpr int quad_products(int form) { return form == kFormGeneral ? 64 : 16; }
__host__ __device__ constexpr int quad_record(int form, int DK) { return quad_vecs(form) * DK + quad_products(form); }
__host__ __device__ constexpr int quad_pad(int d) { return d <= 32 ? 32 : d <= 64 ? 64 : d <= 128 ? 128 : 256; }
// The records of a head follow one another: record (head, group) is head * cap + group.  Number of the first group of sequence `seq`, whose first row is t0 (sequences' records never overlap: floor(t0 / 4) + seq grows by
// at least a sequence's number of groups)
__host__ __device__ constexpr int quad_first(int t0, int seq) { return t0 / kQuad + seq; }

enum { kQuadGeneralDelta = 0, kQuadChannelDecay = 1, kQuadHeadDecay = 2 };
constexpr int quad_form(int kind) { return kind == kQuadGeneralDelta ? kFormGeneral : kFormAdd; }
struct QuadSource {
    int H, share, d;                     // heads; heads that share a query / key head; key channels
    const float *q, *k;                  // token t, head h: q + t * q_ld + (h / share) * d
    int q_ld, k_ld;
    const float* decay;                  // per channel [T][H * d]
    const float *head_decay, *head_step; // per head: [t * head_ld + h * head_el] (head_step nullptr: 1)
    int head_ld, head_el;
    const float *rate, *rate_bias;       // generalized delta rule: a = sigmoid(rate + bias) u, u = k / sqrt(sum k^2 + unit_eps)
    float unit_eps;
    const int32_t* seq_start;
    int cap;                             // records per head
};

// Sums of N values over the warp, one value left per lane: lane l ends with value l (N 32) or l / 2 (N 16).
template <int N>
__device__ __forceinline__ float scatter_sum(float (&v)[N], int lane) {
    static_assert(N == 32 || N == 16, "a value per lane or per pair of lanes");
#pragma unroll
    for (int off = 16, n = N / 2; n > 0; off >>= 1, n >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    if (N == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

// One warp per (group, sequence, head).
template <int KIND, int DK>
__global__ void __launch_bounds__(128) quad_prep_kernel(const QuadSource A, float* __restrict__ rec) {
    dep_wait();
    dep_go();
    constexpr int FORM = quad_form(KIND), NV = quad_vecs(FORM), NP = quad_products(FORM), NS = FORM == kFormGeneral ? 32 : 16;
    const int h = blockIdx.z * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, seq = blockIdx.y;
    const int t0 = A.seq_start[seq], n_all = A.seq_start[seq + 1] - t0, r0 = blockIdx.x * kQuad;
    if (h >= A.H || r0 >= n_all) return;
    const int n = min(kQuad, n_all - r0), g = h / A.share, d = A.d;
    float* out = rec + ((size_t)h * A.cap + quad_first(t0, seq) + blockIdx.x) * quad_record(FORM, DK);
    const float *q = A.q + (size_t)(t0 + r0) * A.q_ld + g * d, *k = A.k + (size_t)(t0 + r0) * A.k_ld + g * d;
    float inv[kQuad], hw[kQuad], hs[kQuad];
#pragma unroll
    for (int t = 0; t < kQuad; ++t) {
        inv[t] = hs[t] = 0.0f;
        hw[t] = 1.0f;
        if (KIND == kQuadGeneralDelta && t < n) {
            float ss = 0.0f;
            for (int c = lane; c < d; c += 32) { const float v = k[(size_t)t * A.k_ld + c]; ss += v * v; }
            inv[t] = 1.0f / sqrtf(warp_sum(ss) + A.unit_eps);
        }
        if (KIND == kQuadHeadDecay && t < n) {
            const size_t at = (size_t)(t0 + r0 + t) * A.head_ld + h * A.head_el;
            hw[t] = A.head_decay[at];
            hs[t] = A.head_step ? A.head_step[at] : 1.0f;
        }
    }
    // products, in the order of the lanes that end up with them: a.u [6] | k.u [6] | a.r [10] | k.r [10] (those the form has)
    constexpr int iKU = 6, iAR = 12, iKR = FORM == kFormGeneral ? 22 : 0;
    float sum[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) sum[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < DK / 32; ++i) {
        const int c = lane + 32 * i;
        const bool in = c < d;
        float w[kQuad], u[kQuad], a[kQuad], kk[kQuad], r[kQuad];
#pragma unroll
        for (int t = 0; t < kQuad; ++t) {
            const bool on = in && t < n;
            const size_t row = t0 + r0 + t;
            const float kv = on ? k[(size_t)t * A.k_ld + c] : 0.0f;
            r[t] = on ? q[(size_t)t * A.q_ld + c] : 0.0f;
            w[t] = KIND != kQuadHeadDecay ? (on ? A.decay[row * A.H * d + h * d + c] : 1.0f) : hw[t];
            if (KIND == kQuadGeneralDelta) {
                u[t] = kv * inv[t];
                a[t] = on ? sigmoidf_(A.rate[row * A.k_ld + h * d + c] + A.rate_bias[h * d + c]) * u[t] : 0.0f;
                kk[t] = kv;
            } else {
                u[t] = a[t] = 0.0f;
                kk[t] = KIND == kQuadHeadDecay ? hs[t] * kv : kv;
            }
        }
        // what token s leaves at the end of the group, and the group's whole decay
        float tail = 1.0f;
#pragma unroll
        for (int s = kQuad - 1; s >= 0; --s) {
            if (FORM == kFormGeneral) out[(8 + s) * DK + c] = -(tail * a[s]);
            out[((FORM == kFormGeneral ? 12 : 4) + s) * DK + c] = tail * kk[s];
            tail *= w[s];
        }
        out[(NV - 1) * DK + c] = tail;
        // what token t reads of the state before the group, and of the group's earlier tokens
#pragma unroll
        for (int t = 0; t < kQuad; ++t) {
            float x = u[t], y = r[t] * w[t];          // decayed back to just after token s
            if (FORM == kFormGeneral) {
#pragma unroll
                for (int s = t - 1; s >= 0; --s) {
                    const int at = t * (t - 1) / 2 + s;
                    sum[at] = fmaf(x, a[s], sum[at]);
                    sum[iKU + at] = fmaf(x, kk[s], sum[iKU + at]);
                    x *= w[s];
                }
                out[t * DK + c] = x;
            }
            {
                const int at = t * (t + 1) / 2 + t;
                if (FORM == kFormGeneral) sum[iAR + at] = fmaf(r[t], a[t], sum[iAR + at]);
                sum[iKR + at] = fmaf(r[t], kk[t], sum[iKR + at]);
            }
#pragma unroll
            for (int s = t - 1; s >= 0; --s) {
                const int at = t * (t + 1) / 2 + s;
                if (FORM == kFormGeneral) sum[iAR + at] = fmaf(y, a[s], sum[iAR + at]);
                sum[iKR + at] = fmaf(y, kk[s], sum[iKR + at]);
                y *= w[s];
            }
            out[((FORM == kFormAdd ? 0 : 4) + t) * DK + c] = y;
        }
    }
    const float mine = scatter_sum<NS>(sum, lane);
    float* prod = out + NV * DK;
#pragma unroll
    for (int i = lane; i < NP; i += 32) prod[i] = 0.0f;
    __syncwarp();
    const int id = NS == 32 ? lane : lane >> 1;
    const bool has = (NS == 32 || (lane & 1) == 0) && id < (FORM == kFormAdd ? 10 : NS);
    if (has) {
        const bool strict = FORM == kFormGeneral && id < iAR;      // the triangle without its diagonal
        constexpr int per = NP / 4;
        int e = id, at = 0;
        float sign = 1.0f;
        if (FORM == kFormGeneral) {
            if (id < 6) sign = -1.0f;
            else if (id < 12) { e = id - 6; at = 4; }
            else if (id < 22) { e = id - 12; at = 8; sign = -1.0f; }
            else { e = id - 22; at = 12; }
        }
        int t, s;
        if (strict) { t = e < 1 ? 1 : e < 3 ? 2 : 3; s = e - t * (t - 1) / 2; }
        else { t = e < 1 ? 0 : e < 3 ? 1 : e < 6 ? 2 : 3; s = e - t * (t + 1) / 2; }
        prod[t * per + at + s] = sign * mine;
    }
}

struct QuadArgs {
    int H, d, dv;
    const float* rec;
    int cap;
    const float* v_src;                  // token t: v_src + t * v_ld + h * dv
    int v_ld;
    float q_scale;
    const int32_t *seq_start, *seq_pos0, *seq_slot;
    size_t slot_floats, state_off;
    int n_slots;
    int32_t* err;
};
__host__ __device__ constexpr size_t quad_smem(int form, int DK) { return (size_t)kQuadRing * quad_chunk(DK) * (quad_record(form, DK) + kQuad * kQuadCols) * sizeof(float); }

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long both(float x) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "r"(__float_as_uint(x)));
    return d;
}
__device__ __forceinline__ void bulk_copy(float* dst, const float* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(umma::s2u(dst)), "l"(src), "r"(bytes), "r"(umma::s2u(bar)) : "memory");
}

__device__ __forceinline__ void copy_float(float* dst, const float* src, bool in) {       // 4 bytes, or a zero
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(umma::s2u(dst)), "l"(src), "r"(in ? 4 : 0));
}

template <int DK, int FORM>
__global__ void __launch_bounds__(kQuadThreads, 1) quad_scan_kernel(const QuadArgs A, float* state_pool, float* __restrict__ o_raw) {
    dep_wait();
    dep_go();
    using f32t::fma2;
    constexpr int L = kQuadLanes, CB = kQuadCols, RV = DK / L / 4, NB = kQuadRing, NG = quad_chunk(DK), RF = quad_record(FORM, DK), NV = quad_vecs(FORM);
    constexpr int kAt = FORM == kFormGeneral ? 12 : 4;      // the k vectors
    constexpr int PW = quad_products(FORM) / 16;                                  // 16-byte pieces of a token's products
    constexpr int NQ = FORM == kFormAdd ? 4 : 8;                                  // vectors that read the state: u and r, or r alone
    extern __shared__ __align__(16) float sh[];
    __shared__ uint64_t full[NB], empty[NB];
    float* vs = sh + NB * NG * RF;                                                // [NB][NG * 4 tokens][CB]
    const int d = A.d, dv = A.dv, NS = (dv + CB - 1) / CB;
    const int part = blockIdx.x % (A.H * NS), seq = blockIdx.x / (A.H * NS);
    const int h = part / NS, j0 = (part % NS) * CB;
    const int t0 = A.seq_start[seq], t1 = A.seq_start[seq + 1];
    const int slot = A.seq_slot[seq];
    if (slot < 0 || slot >= A.n_slots) {
        if (threadIdx.x == 0) atomicExch(A.err, 2);
        return;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) { umma::bar_init(&full[i], 33); umma::bar_init(&empty[i], 2); }      // the copy and each lane's values; two warps
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int groups = (t1 - t0 + kQuad - 1) / kQuad, chunks = (groups + NG - 1) / NG, lane = threadIdx.x & 31;
    if (threadIdx.x >= L * CB) {
        const float* rec = A.rec + ((size_t)h * A.cap + quad_first(t0, seq)) * RF;
        const int c = j0 + lane % CB;
        for (int i = 0; i < chunks; ++i) {
            const int b = i % NB;
            if (i >= NB) umma::bar_wait(&empty[b], (i / NB - 1) & 1);
            if (lane == 0) {
                const uint32_t bytes = (uint32_t)min(NG, groups - i * NG) * RF * 4;
                umma::bar_expect_tx(&full[b], bytes);
                bulk_copy(sh + b * NG * RF, rec + (size_t)i * NG * RF, bytes, &full[b]);
            }
#pragma unroll
            for (int x = 0; x < NG; ++x) {
                const int t = t0 + (i * NG + x) * kQuad + lane / CB;
                const bool value = t < t1 && c < dv;
                copy_float(vs + (b * NG + x) * kQuad * CB + lane, value ? A.v_src + (size_t)t * A.v_ld + h * dv + c : A.v_src, value);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(umma::s2u(&full[b])) : "memory");
        }
        cp_async_commit();
        cp_async_wait<0>();
        return;
    }
    const int col = threadIdx.x / L, q = threadIdx.x % L, j = j0 + col;
    float* st = state_pool + (size_t)slot * A.slot_floats + A.state_off + (size_t)h * d * dv + j;
    __align__(16) float S0[RV][4];
    const bool fresh = A.seq_pos0[seq] == 0;
#pragma unroll
    for (int e = 0; e < RV; ++e)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * (e * L + q) + x;
            S0[e][x] = (!fresh && i < d && j < dv) ? st[(size_t)i * dv] : 0.0f;
        }
    ulonglong2 S[RV];
#pragma unroll
    for (int e = 0; e < RV; ++e) S[e] = *reinterpret_cast<const ulonglong2*>(S0[e]);
    // the lane that ends up with token t's output: 4 + t, or t where nothing is removed
    const int mt = q & 3;
    const bool stores = (FORM == kFormAdd ? q < 4 : q >= 4) && j < dv;
    float* out = o_raw + (size_t)h * dv + j;
    const size_t out_ld = (size_t)A.H * dv;
    auto group = [&](const float* R, const float* vp, int t_group) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(R) + q;        // piece e of vector x: p[x * DK / 4 + e * L]
        const float4* pr = reinterpret_cast<const float4*>(R + NV * DK);
        const float v[4] = {vp[0], vp[CB], vp[2 * CB], vp[3 * CB]};
        unsigned long long acc[NQ];
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
#pragma unroll
            for (int e = 0; e < RV; ++e) {
                const ulonglong2 y = p[x * (DK / 4) + e * L];
                acc[x] = e == 0 ? mul2(y.x, S[0].x) : fma2(y.x, S[e].x, acc[x]);
                acc[x] = fma2(y.y, S[e].y, acc[x]);
            }
        }
        // what does not wait for the sums: the decayed state, and the writes of the general and the adding form
#pragma unroll
        for (int e = 0; e < RV; ++e) {
            const ulonglong2 w = p[(NV - 1) * (DK / 4) + e * L];
            S[e].x = mul2(w.x, S[e].x);
            S[e].y = mul2(w.y, S[e].y);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const ulonglong2 y = p[(kAt + s) * (DK / 4) + e * L];
                S[e].x = fma2(y.x, both(v[s]), S[e].x);
                S[e].y = fma2(y.y, both(v[s]), S[e].y);
            }
        }
        float val[NQ];
#pragma unroll
        for (int x = 0; x < NQ; ++x) val[x] = f32t::pair_sum(acc[x]);
        // sums over the column's lanes, one left per lane: lane q ends with value q (adding form: q & 3)
        if (NQ == 8) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const bool up = q & 4;
                const float send = up ? val[x] : val[(x + 4) % NQ], keep = up ? val[(x + 4) % NQ] : val[x];
                val[x] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const bool up = q & 2;
            const float send = up ? val[x] : val[x + 2], keep = up ? val[x + 2] : val[x];
            val[x] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
        {
            const bool up = q & 1;
            const float send = up ? val[0] : val[1], keep = up ? val[1] : val[0];
            val[0] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
        float o = val[0];
        // of the tokens after mt the output takes nothing, also where they are not finite (their products in the record are zeros)
        const float v1 = mt >= 1 ? v[1] : 0.0f, v2 = mt >= 2 ? v[2] : 0.0f, v3 = mt >= 3 ? v[3] : 0.0f;
        if (FORM == kFormAdd) {
            o += __shfl_xor_sync(0xffffffffu, o, 4);
            const float4 kr = pr[mt];
            o = fmaf(kr.x, v[0], o); o = fmaf(kr.y, v1, o); o = fmaf(kr.z, v2, o); o = fmaf(kr.w, v3, o);
        } else {
            float b[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) b[t] = __shfl_sync(0xffffffffu, val[0], t, 8);
            // seen_t; the products with the values do not wait
            const float4 a1 = pr[PW], a2 = pr[2 * PW], a3 = pr[3 * PW], k1 = pr[PW + 1], k2 = pr[2 * PW + 1], k3 = pr[3 * PW + 1];
            const float s0 = b[0];
            const float s1 = fmaf(a1.x, s0, fmaf(k1.x, v[0], b[1]));
            const float s2 = fmaf(a2.y, s1, fmaf(a2.x, s0, fmaf(k2.y, v[1], fmaf(k2.x, v[0], b[2]))));
            const float s3 = fmaf(a3.z, s2, fmaf(a3.y, s1, fmaf(a3.x, s0, fmaf(k3.z, v[2], fmaf(k3.y, v[1], fmaf(k3.x, v[0], b[3]))))));
            const float4 ar = pr[mt * PW + 2], kr = pr[mt * PW + 3];
            o = fmaf(kr.x, v[0], o); o = fmaf(kr.y, v1, o); o = fmaf(kr.z, v2, o); o = fmaf(kr.w, v3, o);
            o = fmaf(ar.x, s0, o); o = fmaf(ar.y, mt >= 1 ? s1 : 0.0f, o); o = fmaf(ar.z, mt >= 2 ? s2 : 0.0f, o); o = fmaf(ar.w, mt >= 3 ? s3 : 0.0f, o);
            const unsigned long long z[4] = {both(s0), both(s1), both(s2), both(s3)};
#pragma unroll
            for (int e = 0; e < RV; ++e)
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const ulonglong2 y = p[(8 + s) * (DK / 4) + e * L];
                    S[e].x = fma2(y.x, z[s], S[e].x);
                    S[e].y = fma2(y.y, z[s], S[e].y);
                }
        }
        const int t = t_group + mt;
        if (stores && t < t1) out[(size_t)t * out_ld] = o * A.q_scale;
    };
    for (int i = 0; i < chunks; ++i) {
        const int b = i % NB;
        umma::bar_wait(&full[b], (i / NB) & 1);
        const float *R = sh + b * NG * RF, *vp = vs + b * NG * kQuad * CB + col;
        const int g0 = i * NG, tg = t0 + g0 * kQuad;
        if (g0 + NG <= groups) {
#pragma unroll
            for (int x = 0; x < NG; ++x) group(R + x * RF, vp + x * kQuad * CB, tg + x * kQuad);
        } else {
            for (int x = 0; x < groups - g0; ++x) group(R + x * RF, vp + x * kQuad * CB, tg + x * kQuad);
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[b]);
    }
#pragma unroll
    for (int e = 0; e < RV; ++e) {
        *reinterpret_cast<ulonglong2*>(S0[e]) = S[e];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * (e * L + q) + x;
            if (i < d && j < dv) st[(size_t)i * dv] = S0[e][x];
        }
    }
}

}  // namespace lm
}  // namespace smol
