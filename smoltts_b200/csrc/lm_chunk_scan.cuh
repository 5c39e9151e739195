// The recurrences' scan for prompts, sixteen tokens at a time (included by lm_kernels.cu after lm_quad_scan.cuh).  Everything is fp32.
//
// The recurrences act on a head's state S [d, dv] as
//     S <- diag(w) S - a (u^T S) + k v^T,     o = S^T r
// with per-token vectors over the d key channels (the generalized and the gated delta rule; the linear attentions and the mLSTM without a and u).
// With W(i, j] the product of the decays of tokens i + 1 .. j of a chunk and S the state before it, everything the chunk's tokens need is
//     seen = X_w S + V',   o = X_o S + O',   S <- W(0, 16] S + Y_v V + Y_a seen
// where, with the strict triangles L = (W(s, t-1] u_t).a_s and M = (W(s, t-1] u_t).k_s and the triangles with their diagonals A = (W(s, t] r_t).a_s and
// R = (W(s, t] r_t).k_s,
//     X_w = (1 + L)^-1 W(0, t-1] u_t      V' = (1 + L)^-1 M V        Y_v = W(s, 16] k_s
//     X_o = W(0, t] r_t - A X_w           O' = R V - A V'            Y_a = -W(s, 16] a_s
// (without a and u: X_o = W(0, t] r_t, O' = R V, no X_w, V', Y_a).  The decays are at most one, so nothing is divided and nothing grows; the inverse is a
// forward substitution.
//
// (The chunk-wise form of the delta rule: the triangular inverse is that of a product of Householder-like updates, its WY representation.)
//
// chunk_prep_kernel (one decay per head: chunk_prep_head_kernel) makes X, Y, V' and O' of a (chunk, head) in one block; it is parallel over the whole prompt.
// chunk_scan_kernel is what is left to do in order: two small matrix products per sixteen tokens.  A head's value columns never mix, so a block takes eight of them,
// and its four warps share the key channels.  Both products run on mma.sync m16n8k16: every fp32 operand as three bf16 parts, which hold all of its 24 bits, and the
// six products of parts that reach the last place (the split of a product over pieces of a shorter format): 170 multiply-adds per clock and SM against 128 on the FMA
// pipe, and without the shared-memory traffic and shuffles that those need for 16 x 8 results.
// The state's accumulator fragments become operand fragments through a patch of shared memory of the warp's own; the warps' shares of `seen` and o meet
// in shared memory, one barrier per chunk.  X, Y and V lie as the parts of their fragments, so a lane's share is three 16-byte (V: 8-byte) loads.
// What bounds the scan is the instructions of that chain (one warp per scheduler), no longer a chain per four tokens.
// Records and scan, 2048 tokens, 12 heads of 64 x 64: generalized delta rule 109 us (four tokens at a time 211), decay per channel 79 (135), gated delta rule 92 (207),
// mLSTM 76 (181); 1801 tokens of 128 x 128: 196 (408), 149 (220), 177 (307), 140 (266); 3 x 1000 of 64 x 64: 103 (172), 68 (84), 83 (107), 96 (140).
// Error of the outputs | of the state against 64 bits, 1100 tokens of 12 heads of 64 x 64 (four tokens at a time): generalized delta rule 1.16e-7 (1.36) | 0.90e-7 (1.17), decay
// per channel 1.08 (1.13) | 0.84 (0.90), gated delta rule 1.06 (1.18) | 0.81 (1.07), mLSTM 1.02 (1.16) | 0.80 (1.15); 9 to 256 channels, 210 to 2000 tokens: never above.
// With two tf32 parts per operand (three MMAs of 8, 99 us where it is 109 now) the outputs were at 1.62, 1.49, 1.63 and 1.53e-7.
#pragma once

namespace smol {
namespace lm {

constexpr int kChunk = 16;               // tokens of a chunk
constexpr int kChunkCols = 8;            // value columns of a block
enum { kScanGeneralDelta = 0, kScanChannelDecay = 1, kScanHeadDecay = 2, kScanGatedDelta = 3 };
constexpr bool scan_removes(int kind) { return kind == kScanGeneralDelta || kind == kScanGatedDelta; }      // has a and u
__host__ __device__ constexpr int chunk_pad(int d) { return d <= 32 ? 32 : d <= 64 ? 64 : d <= 128 ? 128 : 256; }
// Fragments of 16 x 16 lie as their three bf16 parts, made once beside the records instead of by every block that reads them; above 128 channels, where two such
// records do not fit an SM, as fp32.
__host__ __device__ constexpr bool chunk_split(int DK) { return DK <= 128; }
__host__ __device__ constexpr int chunk_frag(int DK) { return chunk_split(DK) ? 384 : 256; }      // words of a fragment
// A record holds the key side: X fragments [16 channels][seen, o] | Y fragments [16 channels][V, then seen] | W(0, 16]; the value side follows, per block of
// columns V' [16][8] (with removal; rows in the order of chunk_place) | O' [16][8] | V's three parts, an operand fragment each [32 lanes][2].
constexpr int kChunkVals = 3 * 64;
__host__ __device__ constexpr int chunk_key_floats(bool removes, int DK) { return (removes ? 4 : 2) * DK / 16 * chunk_frag(DK) + DK; }
__host__ __device__ constexpr int chunk_col_floats(bool removes) { return (removes ? 2 : 1) * kChunk * kChunkCols + kChunkVals; }
__host__ __device__ constexpr int chunk_blocks(int columns) { return (columns + kChunkCols - 1) / kChunkCols; }
__host__ __device__ constexpr int chunk_record(bool removes, int DK, int columns) { return chunk_key_floats(removes, DK) + chunk_blocks(columns) * chunk_col_floats(removes); }
// Where row k of a 16 x 8 operand lies in shared memory: lane (g, q) reads rows 2 q + b + 8 r of column g, and so finds them in banks of its own
__host__ __device__ constexpr int chunk_place(int k) { return (k >> 3) * 8 + (k & 1) * 4 + ((k >> 1) & 3); }
// The records of a head follow one another: record (head, chunk) is head * cap + chunk.  Number of the first chunk of sequence `seq`, whose first row is t0
// (sequences' records never overlap: floor(t0 / 16) + seq grows by at least a sequence's number of chunks)
__host__ __device__ constexpr int chunk_first(int t0, int seq) { return t0 / kChunk + seq; }

struct ChunkSource {
    int H, share, d, dv, columns;        // heads; heads that share a query / key head; key channels; value columns, and with the unit column behind them
    const float *q, *k;                  // token t, head h: q + t * q_ld + (h / share) * d
    int q_ld, k_ld;
    const float* v;                      // v + t * v_ld + h * dv
    int v_ld;
    const float* decay;                  // per channel [T][H * d]
    const float *head_decay, *head_step; // per head: [t * head_ld + h * head_el] (head_step nullptr: 1)
    int head_ld, head_el;
    const float *rate, *rate_bias;       // generalized delta rule: a = sigmoid(rate + bias) u, u = k / sqrt(sum k^2 + unit_eps)
    float unit_eps;
    const int32_t* seq_start;
    int cap;                             // records per head
};

// Sums of N values over each eight lanes: lane `sub` of the eight ends with values sub * N / 8 .. (N 16), or value sub / 2 (N 4).
template <int N>
__device__ __forceinline__ void scatter_sum8(float (&v)[N], int sub) {
    static_assert(N == 16 || N == 4, "two values per lane or one per pair of lanes");
#pragma unroll
    for (int off = 4, n = N / 2; off > (N == 4 ? 1 : 0); off >>= 1, n >>= 1) {
        const bool up = sub & off;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    if (N == 4) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// floats between the tokens' rows: r and u are gathered as operands whose rows are tokens, k and a as operands whose columns are; decays are read in pieces only
__host__ __device__ constexpr int chunk_xl(int DK) { return DK + 8; }
__host__ __device__ constexpr int chunk_yl(int DK) { return DK + 4; }
constexpr int kDecayLd = kChunk + 4;      // W(s, t] of a head: [16 tokens t][s = -1 .. 15], here and there four more
__host__ __device__ constexpr int chunk_prep_floats(int kind, int DK) {
    const int xl = chunk_xl(DK), yl = chunk_yl(DK);
    return kind == kScanGeneralDelta ? kChunk * (2 * xl + 2 * yl + DK + 4) + 4 * DK + 4 * kChunk * kChunk
           : kind == kScanChannelDecay ? kChunk * (xl + yl + DK + 4) + 4 * DK + kChunk * kChunk
           : kind == kScanGatedDelta ? kChunk * (2 * xl + yl + kDecayLd) + 2 * kChunk * kChunk
                                     : kChunk * (xl + yl + kDecayLd) + kChunk * kChunk;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// Two fp32 numbers as three pairs of bf16, eight bits each and cut off, so that nothing of the 24 is lost: x = p[0] + p[1] + p[2].
__device__ __forceinline__ void bf16_parts(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint32_t a = __float_as_uint(x), b = __float_as_uint(y);
        p[i] = __byte_perm(a, b, 0x7632);
        x -= __uint_as_float(a & 0xffff0000u);
        y -= __uint_as_float(b & 0xffff0000u);
    }
}
// Operands of mma.sync m16n8k16 in their three parts
struct PartsA {
    uint32_t p[3][4];
    // rows g, g + 8, g, g + 8; columns 2 q, 2 q + 1 (the last two: + 8)
    __device__ __forceinline__ void set(int i, float x, float y) {
        uint32_t z[3];
        bf16_parts(x, y, z);
#pragma unroll
        for (int k = 0; k < 3; ++k) p[k][i] = z[k];
    }
    template <bool SPLIT>
    __device__ __forceinline__ void load(const float* frag, int lane) {
        if (SPLIT) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint4 v = reinterpret_cast<const uint4*>(frag)[k * 32 + lane];
                p[k][0] = v.x; p[k][1] = v.y; p[k][2] = v.z; p[k][3] = v.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float4 v = reinterpret_cast<const float4*>(frag)[k * 32 + lane];
                set(2 * k, v.x, v.y);
                set(2 * k + 1, v.z, v.w);
            }
        }
    }
    template <bool SPLIT>
    __device__ static __forceinline__ void store(float* frag, int lane, const float (&v)[8]) {
        if (SPLIT) {
            PartsA a;
#pragma unroll
            for (int i = 0; i < 4; ++i) a.set(i, v[2 * i], v[2 * i + 1]);
#pragma unroll
            for (int k = 0; k < 3; ++k) reinterpret_cast<uint4*>(frag)[k * 32 + lane] = make_uint4(a.p[k][0], a.p[k][1], a.p[k][2], a.p[k][3]);
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) reinterpret_cast<float4*>(frag)[k * 32 + lane] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
    }
};
struct PartsB {
    uint32_t p[3][2];
    // rows 2 q, 2 q + 1 (the second: + 8) of column g
    __device__ __forceinline__ void set(int i, float x, float y) {
        uint32_t z[3];
        bf16_parts(x, y, z);
#pragma unroll
        for (int k = 0; k < 3; ++k) p[k][i] = z[k];
    }
    __device__ __forceinline__ void load(const float* parts, int lane) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint2 v = reinterpret_cast<const uint2*>(parts)[k * 32 + lane];
            p[k][0] = v.x; p[k][1] = v.y;
        }
    }
};
// sum = a b over N steps of 16: six of the nine products of parts (the others lie below the last place), those of one size in accumulators of their own, no more than
// two MMAs behind one another.  The tensor core cuts its sums off instead of rounding them; what the largest one loses by that in the mean, half a unit of its last place
// (0.5 to 1 x 2^-24 of it), is given back (outputs of the generalized delta rule with 0 / 0.72 / 1.0: 1.48, 1.32 and 1.31e-7 off, all else alike).
constexpr float kCutOff = 0.85f * 0x1p-24f;
template <int N>
__device__ __forceinline__ void mma_sum(float (&sum)[4], const PartsA (&a)[N], const PartsB (&b)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
        float big[4], s1[4], s2[4], s3[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) big[e] = s1[e] = s2[e] = s3[e] = 0.0f;
        mma_bf16(s1, a[k].p[0], b[k].p[2]);
        mma_bf16(s2, a[k].p[2], b[k].p[0]);
        mma_bf16(s3, a[k].p[1], b[k].p[1]);
        mma_bf16(big, a[k].p[0], b[k].p[0]);
        mma_bf16(s1, a[k].p[0], b[k].p[1]);
        mma_bf16(s2, a[k].p[1], b[k].p[0]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float t = big[e] + (fmaf(big[e], kCutOff, s3[e]) + (s1[e] + s2[e]));
            sum[e] = k == 0 ? t : sum[e] + t;
        }
    }
}

// acc += sign * sum_(s < upto) p[s] z[s] over the quad s = 4 i .., which is added up by itself
__device__ __forceinline__ void chunk_take(float& acc, const float4 p, const float (&z)[kChunk], int i, int upto, float sign) {
    float part = 0.0f;
    if (4 * i < upto) part = p.x * z[4 * i];
    if (4 * i + 1 < upto) part = fmaf(p.y, z[4 * i + 1], part);
    if (4 * i + 2 < upto) part = fmaf(p.z, z[4 * i + 2], part);
    if (4 * i + 3 < upto) part = fmaf(p.w, z[4 * i + 3], part);
    acc = fmaf(sign, part, acc);
}
__device__ __forceinline__ float2 two(const float* p) { return *reinterpret_cast<const float2*>(p); }
// value column j of a chunk's rows (a unit column is behind the value columns); V's parts of that column in its block's record
__device__ __forceinline__ void chunk_values(const ChunkSource& A, size_t row, int n, int h, int j, float (&v)[kChunk]) {
    const float* at = A.v + row * A.v_ld + h * A.dv + j;
#pragma unroll
    for (int t = 0; t < kChunk; ++t, at += A.v_ld) v[t] = t < n && j < A.columns ? (j < A.dv ? *at : 1.0f) : 0.0f;
}
template <bool REM>
__device__ __forceinline__ void chunk_value_parts(float* cols, int j, const float (&v)[kChunk]) {
    uint2* parts = reinterpret_cast<uint2*>(cols + (j / kChunkCols) * chunk_col_floats(REM) + (REM ? 2 : 1) * kChunk * kChunkCols) + j % kChunkCols * 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        PartsB b;
        b.set(0, v[2 * q], v[2 * q + 1]);
        b.set(1, v[2 * q + 8], v[2 * q + 9]);
#pragma unroll
        for (int k = 0; k < 3; ++k) parts[k * 32 + q] = make_uint2(b.p[k][0], b.p[k][1]);
    }
}
// The key side's fragments: X from rows of tokens, Y from columns of tokens (`removed`: the sign of the writes along a: 1, or -1 where a is k itself)
template <int DK, bool REM>
__device__ __forceinline__ void chunk_fragments(float* out, const float* s_u, const float* s_r, const float* s_k, const float* s_a, float removed) {
    constexpr int MX = REM ? 2 : 1, FR = chunk_frag(DK), XL = chunk_xl(DK), YL = chunk_yl(DK);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, q = lane & 3;
#pragma unroll 2
    for (int i = warp; i < DK / 16 * MX; i += 4) {
        const float* p = (REM && i % MX == 0 ? s_u : s_r) + gq * XL + i / MX * 16 + 2 * q;
        const float2 a = two(p), b = two(p + 8 * XL), c = two(p + 8), e = two(p + 8 * XL + 8);
        PartsA::store<chunk_split(DK)>(out + i * FR, lane, {a.x, a.y, b.x, b.y, c.x, c.y, e.x, e.y});
    }
#pragma unroll 2
    for (int i = warp; i < DK / 16 * MX; i += 4) {
        const bool of_a = i % MX != 0;
        const float* p = (of_a ? s_a : s_k) + 2 * q * YL + i / MX * 16 + gq;
        const float f = of_a ? removed : 1.0f;
        PartsA::store<chunk_split(DK)>(out + (DK / 16 * MX + i) * FR, lane,
                                       {f * p[0], f * p[YL], f * p[8], f * p[YL + 8], f * p[8 * YL], f * p[9 * YL], f * p[8 * YL + 8], f * p[9 * YL + 8]});
    }
}

// Decays per channel.  One block per (chunk, sequence, head); a warp has four tokens, the chunk four such quads.  The vectors lie in shared memory [16][DK].  Within a quad a warp
// makes the products on the FMA pipe, eight lanes per token, the decays multiplied in on the way back from token to token; products between two quads
// are made by MMAs (operands in three bf16 parts, as in the scan) from what each side is at the border: the later one's vectors decayed back to the
// start of its quad, the earlier one's writes decayed up to there.  Then a thread per column runs the substitutions, and the results leave as fragments.
template <int KIND, int DK>
__global__ void __launch_bounds__(128, DK <= 64 ? 5 : DK <= 128 ? 4 : 1) chunk_prep_kernel(const ChunkSource A, float* __restrict__ rec) {
    dep_wait();
    dep_go();
    using f32t::fma2;
    constexpr bool REM = scan_removes(KIND);
    static_assert(KIND == kScanGeneralDelta || KIND == kScanChannelDecay, "one decay per head: chunk_prep_head_kernel");
    constexpr int XL = chunk_xl(DK), YL = chunk_yl(DK), WL = DK + 4, NM = REM ? 4 : 1, E = DK / 32;
    constexpr int kR = NM - 1, kM = NM > 1 ? 1 : 0, kA = NM > 1 ? 2 : 0;         // products: L, M, A, R, or R alone
    extern __shared__ __align__(16) float sh[];
    float *s_r = sh, *s_u = s_r + kChunk * XL, *s_k = s_u + (REM ? kChunk * XL : 0), *s_a = s_k + kChunk * YL, *s_w = s_a + (REM ? kChunk * YL : 0);
    float *s_q = s_w + kChunk * WL, *s_m = s_q + 4 * DK;                         // a quad's decay [4][DK]; products [NM][16][16]
    const int h = blockIdx.z, seq = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = A.seq_start[seq], n_all = A.seq_start[seq + 1] - t0, r0 = blockIdx.x * kChunk;
    if (r0 >= n_all) return;
    const int n = min(kChunk, n_all - r0), g = h / A.share, d = A.d;
    const int nb = chunk_blocks(A.columns), n_cols = nb * kChunkCols;
    float* out = rec + ((size_t)h * A.cap + chunk_first(t0, seq) + blockIdx.x) * (chunk_key_floats(REM, DK) + nb * chunk_col_floats(REM));
    // value column j of the rows, every load on its way before the products are made (DK 64: on the threads that will have no key channel)
    const int j_first = DK <= 64 ? (int)(threadIdx.x + 128 - DK) % 128 : (int)threadIdx.x;
    float v[kChunk];
    constexpr bool EARLY = DK <= 64 && REM;
    if (EARLY) chunk_values(A, t0 + r0, n, h, j_first, v);
    // ---- the tokens' vectors ----
    {
        float kv[4][E], qv[4][E], wv[4][E], rv[4][E], bias[E];
#pragma unroll
        for (int e = 0; e < E; ++e) bias[e] = KIND == kScanGeneralDelta && lane + 32 * e < d ? A.rate_bias[h * d + lane + 32 * e] : 0.0f;
        const size_t row = t0 + r0 + warp * 4;
        const float *pk = A.k + row * A.k_ld + g * d + lane, *pq = A.q + row * A.q_ld + g * d + lane;
        const float *pw = A.decay + row * A.H * d + h * d + lane, *pr = KIND == kScanGeneralDelta ? A.rate + row * A.k_ld + h * d + lane : nullptr;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const bool on = warp * 4 + x < n;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const bool in = on && lane + 32 * e < d;
                kv[x][e] = in ? pk[32 * e] : 0.0f;
                qv[x][e] = in ? pq[32 * e] : 0.0f;
                wv[x][e] = in ? pw[32 * e] : 1.0f;
                rv[x][e] = KIND == kScanGeneralDelta && in ? pr[32 * e] : 0.0f;
            }
            pk += A.k_ld;
            pq += A.q_ld;
            pw += A.H * d;
            if (KIND == kScanGeneralDelta) pr += A.k_ld;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int t = warp * 4 + x;
            float inv = 0.0f;
            if (KIND == kScanGeneralDelta) {
                float ss = 0.0f;
#pragma unroll
                for (int e = 0; e < E; ++e) ss = fmaf(kv[x][e], kv[x][e], ss);
                inv = 1.0f / sqrtf(warp_sum(ss) + A.unit_eps);
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int c = lane + 32 * e;
                s_r[t * XL + c] = qv[x][e];
                s_w[t * WL + c] = wv[x][e];
                s_k[t * YL + c] = kv[x][e];
                if (REM) {
                    const float u = kv[x][e] * inv;
                    s_u[t * XL + c] = u;
                    s_a[t * YL + c] = t < n && c < d ? sigmoidf_(rv[x][e] + bias[e]) * u : 0.0f;
                }
            }
        }
    }
    __syncwarp();
    // ---- products within the quad: token t = 4 warp + lane / 8 with the tokens before it (R and A: itself too), channels 4 (8 e + lane % 8) .. + 3 ----
    {
        const int tg = lane >> 3, sub = lane & 7, t = warp * 4 + tg;
        ulonglong2 x[REM ? E : 1], y[E];
        auto piece = [&](float* p, int e) -> ulonglong2& { return *reinterpret_cast<ulonglong2*>(p + 4 * (e * 8 + sub)); };
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (REM) x[e] = piece(s_u + t * XL, e);
            y[e] = piece(s_r + t * XL, e);
        }
        float sum[4 * NM];
        ulonglong2 tail[E];                                // W(s, end of the quad] of s = t, then the whole quad's decay
#pragma unroll
        for (int i = 3; i >= 0; --i) {
            const int s = warp * 4 + i;
            const bool before = i < tg, reached = i <= tg;
            unsigned long long p[NM];
#pragma unroll
            for (int m = 0; m < NM; ++m) p[m] = 0ull;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const ulonglong2 kk = piece(s_k + s * YL, e), ww = piece(s_w + s * WL, e);
                p[kR] = fma2(y[e].x, kk.x, p[kR]); p[kR] = fma2(y[e].y, kk.y, p[kR]);
                if (REM) {
                    const ulonglong2 aa = piece(s_a + s * YL, e);
                    p[0] = fma2(x[e].x, aa.x, p[0]); p[0] = fma2(x[e].y, aa.y, p[0]);
                    p[kM] = fma2(x[e].x, kk.x, p[kM]); p[kM] = fma2(x[e].y, kk.y, p[kM]);
                    p[kA] = fma2(y[e].x, aa.x, p[kA]); p[kA] = fma2(y[e].y, aa.y, p[kA]);
                    const ulonglong2 xw = {mul2(x[e].x, ww.x), mul2(x[e].y, ww.y)};
                    if (before) x[e] = xw;
                }
                const ulonglong2 yw = {mul2(y[e].x, ww.x), mul2(y[e].y, ww.y)};
                if (reached) y[e] = yw;
            }
            // what lies behind the diagonal is dropped here, also where it is not finite
#pragma unroll
            for (int m = 0; m < NM; ++m) sum[i * NM + m] = (REM && m < 2 ? before : reached) ? f32t::pair_sum(p[m]) : 0.0f;
        }
        scatter_sum8<4 * NM>(sum, sub);
        if (REM) {
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const int id = 2 * sub + z;
                s_m[(id % NM) * kChunk * kChunk + t * kChunk + warp * 4 + id / NM] = sum[z];
            }
        } else if ((sub & 1) == 0) s_m[t * kChunk + warp * 4 + sub / 2] = sum[0];
        // the vectors at the quad's borders
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const ulonglong2 one = {0x3f8000003f800000ull, 0x3f8000003f800000ull};
            ulonglong2 all = one, mine = one;
#pragma unroll
            for (int i = 3; i >= 0; --i) {
                const ulonglong2 ww = piece(s_w + (warp * 4 + i) * WL, e);
                if (i == tg) mine = all;
                all = {mul2(all.x, ww.x), mul2(all.y, ww.y)};
            }
            tail[e] = mine;
            if (tg == 0) piece(s_q + warp * DK, e) = all;
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e) {
            ulonglong2 kk = piece(s_k + t * YL, e);
            piece(s_k + t * YL, e) = {mul2(tail[e].x, kk.x), mul2(tail[e].y, kk.y)};
            if (REM) {
                ulonglong2 aa = piece(s_a + t * YL, e);
                piece(s_a + t * YL, e) = {mul2(tail[e].x, aa.x), mul2(tail[e].y, aa.y)};
                piece(s_u + t * XL, e) = x[e];
            }
            piece(s_r + t * XL, e) = y[e];
        }
    }
    __syncthreads();
    // ---- products between quads: rows x (4 tokens) | y (4) of quad i, columns a (4) | k (4) of quad j < i; without removal y and k alone ----
    {
        const int gq = lane >> 2, q = lane & 3;
        for (int id = warp; id < 6; id += 4) {                             // (3,0) (3,1) (3,2) (2,0) (2,1) (1,0)
            const int i = id < 3 ? 3 : id < 5 ? 2 : 1, j = id < 3 ? id : id < 5 ? id - 3 : 0;
            const float *row = REM && gq < 4 ? s_u + (4 * i + gq) * XL : s_r + (4 * i + (gq & 3)) * XL;
            const float *col = REM && gq < 4 ? s_a + (4 * j + gq) * YL : s_k + (4 * j + (gq & 3)) * YL;
            float sum[2] = {0.0f, 0.0f};
#pragma unroll 4
            for (int k = 0; k < DK / 16; ++k) {
                PartsA a[1];
                PartsB z[1];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int c = 16 * k + 8 * x + 2 * q;
                    const float2 r2 = two(row + c);
                    float2 z2 = two(col + c);                              // ... times the decay of the quads between
                    if (i - j > 1) { const float2 w2 = two(s_q + (i - 1) * DK + c); z2.x *= w2.x; z2.y *= w2.y; }
                    if (i - j > 2) { const float2 w2 = two(s_q + (i - 2) * DK + c); z2.x *= w2.x; z2.y *= w2.y; }
                    a[0].set(2 * x, r2.x, r2.y);
                    a[0].set(2 * x + 1, 0.0f, 0.0f);
                    z[0].set(x, z2.x, z2.y);
                }
                float part[4];
                mma_sum<1>(part, a, z);
                sum[0] += part[0];
                sum[1] += part[1];
            }
            // row gq, columns 2 q, 2 q + 1
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 2 * q + e;
                if (REM) s_m[((gq >> 2) * 2 + (c >> 2)) * kChunk * kChunk + (4 * i + (gq & 3)) * kChunk + 4 * j + (c & 3)] = sum[e];
                else if (gq < 4 && c < 4) s_m[(4 * i + gq) * kChunk + 4 * j + c] = sum[e];
            }
        }
    }
    __syncthreads();
    // ---- columns: key channels first, then value columns; row t of a product, elements 4 i .. + 3 ----
    auto row4 = [&](int m, int t, int i) { return *reinterpret_cast<const float4*>(s_m + m * kChunk * kChunk + t * kChunk + 4 * i); };
    for (int c = threadIdx.x; c < DK; c += 128) {
        float xw[kChunk], p = 1.0f;
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
            float o = p * s_r[t * XL + c];
            if (REM) {
                xw[t] = p * s_u[t * XL + c];
#pragma unroll
                for (int i = 0; 4 * i < t; ++i) chunk_take(xw[t], row4(0, t, i), xw, i, t, -1.0f);
#pragma unroll
                for (int i = 0; 4 * i <= t; ++i) chunk_take(o, row4(kA, t, i), xw, i, t + 1, -1.0f);
                s_u[t * XL + c] = xw[t];
            }
            s_r[t * XL + c] = o;
            if (t % 4 == 3) p *= s_q[t / 4 * DK + c];
        }
        out[chunk_key_floats(REM, DK) - DK + c] = p;
        p = 1.0f;
#pragma unroll
        for (int s = kChunk - 1; s >= 0; --s) {
            s_k[s * YL + c] = p * s_k[s * YL + c];
            if (REM) s_a[s * YL + c] = -(p * s_a[s * YL + c]);
            if (s % 4 == 0) p *= s_q[s / 4 * DK + c];
        }
    }
    asm volatile("" ::: "memory");               // the products are read again: kept for both loops they do not fit the registers (DK 128)
    float* cols = out + chunk_key_floats(REM, DK);
    for (int j = j_first; j < n_cols; j += 128) {
        if (!EARLY || j != j_first) chunk_values(A, t0 + r0, n, h, j, v);
        float seen[kChunk];
        float* to = cols + (j / kChunkCols) * chunk_col_floats(REM) + j % kChunkCols;
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
            if (t % 4 == 0) asm volatile("" ::: "memory");      // (all rows read ahead would not fit either)
            float o = 0.0f;
            if (REM) {
                seen[t] = 0.0f;
#pragma unroll
                for (int i = 0; 4 * i < t; ++i) {
                    chunk_take(seen[t], row4(kM, t, i), v, i, t, 1.0f);
                    chunk_take(seen[t], row4(0, t, i), seen, i, t, -1.0f);
                }
                to[chunk_place(t) * kChunkCols] = seen[t];
            }
#pragma unroll
            for (int i = 0; 4 * i <= t; ++i) {
                chunk_take(o, row4(kR, t, i), v, i, t + 1, 1.0f);
                if (REM) chunk_take(o, row4(kA, t, i), seen, i, t + 1, -1.0f);
            }
            to[(REM ? kChunk + t : t) * kChunkCols] = o;
        }
        chunk_value_parts<REM>(cols, j, v);
    }
    __syncthreads();
    // ---- fragments ----
    chunk_fragments<DK, REM>(out, s_u, s_r, s_k, s_a, 1.0f);
}

// One decay per head and token: it leaves the products of vectors alone and multiplies them afterwards.  W(s, t] is a product of at most sixteen numbers in fp64,
// rounded once (multiplied up along the vectors, its roundings would be the same in all of a head's channels).  The gated delta rule, S <- w S + b k (v - k^T (w S))^T,
// removes along what it writes along: with L = W(s, t] (k_t . b_s k_s) and R likewise of r, and u_t = v_t - sum_(s < t) L u_s what a token writes,
//     X_w = W(0, t] k_t - L X_w      V' = L u      X_o = W(0, t] r_t - R X_w      O' = R u      Y_v = W(s, 16] b_s k_s = -Y_a.
// One block per (chunk, sequence, head).  All products are MMAs, a warp a triangle's half (eight columns; without removal two of the warps).
template <int KIND, int DK>
__global__ void __launch_bounds__(128, DK <= 64 ? 5 : DK <= 128 ? 4 : 1) chunk_prep_head_kernel(const ChunkSource A, float* __restrict__ rec) {
    dep_wait();
    dep_go();
    constexpr bool REM = scan_removes(KIND);
    constexpr int XL = chunk_xl(DK), YL = chunk_yl(DK), NM = REM ? 2 : 1, E = DK / 32, kR = NM - 1;
    extern __shared__ __align__(16) float sh[];
    float *s_r = sh, *s_u = s_r + kChunk * XL, *s_k = s_u + (REM ? kChunk * XL : 0), *s_m = s_k + kChunk * YL, *s_w = s_m + NM * kChunk * kChunk;
    const int h = blockIdx.z, seq = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = A.seq_start[seq], n_all = A.seq_start[seq + 1] - t0, r0 = blockIdx.x * kChunk;
    if (r0 >= n_all) return;
    const int n = min(kChunk, n_all - r0), g = h / A.share, d = A.d;
    const int nb = chunk_blocks(A.columns), n_cols = nb * kChunkCols;
    float* out = rec + ((size_t)h * A.cap + chunk_first(t0, seq) + blockIdx.x) * (chunk_key_floats(REM, DK) + nb * chunk_col_floats(REM));
    // value column j of the rows, every load on its way before the products are made (DK 64: on the threads that will have no key channel)
    const int j_first = DK <= 64 ? (int)(threadIdx.x + 128 - DK) % 128 : (int)threadIdx.x;
    float v[kChunk];
    constexpr bool EARLY = DK <= 64 && REM;
    if (EARLY) chunk_values(A, t0 + r0, n, h, j_first, v);
    // ---- the tokens' vectors, four tokens a warp; the decays ----
    {
        float kv[4][E], qv[4][E], hs[4];
        const size_t row = t0 + r0 + warp * 4;
        const float *pk = A.k + row * A.k_ld + g * d + lane, *pq = A.q + row * A.q_ld + g * d + lane, *ps = A.head_step ? A.head_step + row * A.head_ld + h * A.head_el : nullptr;
        float w = 1.0f;
        if (warp == 3 && lane < n) w = A.head_decay[(size_t)(t0 + r0 + lane) * A.head_ld + h * A.head_el];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const bool on = warp * 4 + x < n;
            hs[x] = on && ps ? *ps : 1.0f;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const bool in = on && lane + 32 * e < d;
                kv[x][e] = in ? pk[32 * e] : 0.0f;
                qv[x][e] = in ? pq[32 * e] : 0.0f;
            }
            pk += A.k_ld;
            pq += A.q_ld;
            if (ps) ps += A.head_ld;
        }
        if (warp == 3) {
            // lane t: W(s, t] for s = t down to -1, at s + 1
            double p = 1.0;
#pragma unroll
            for (int s = kChunk - 1; s >= 0; --s) {
                const float ws = __shfl_sync(0xffffffffu, w, s);
                if (s > lane || lane >= kChunk) continue;
                s_w[lane * kDecayLd + s + 1] = (float)p;
                p *= (double)ws;
            }
            if (lane < kChunk) s_w[lane * kDecayLd] = (float)p;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int t = warp * 4 + x, c = lane + 32 * e;
                s_r[t * XL + c] = qv[x][e];
                if (REM) s_u[t * XL + c] = kv[x][e];
                s_k[t * YL + c] = hs[x] * kv[x][e];
            }
    }
    __syncthreads();
    // ---- products: rows 16 tokens t, columns eight tokens s ----
    if (warp < 2 * NM) {
        const int gq = lane >> 2, q = lane & 3, m = warp >> 1, s0 = (warp & 1) * 8;
        const float *row = (REM && m == 0 ? s_u : s_r) + gq * XL + 2 * q, *col = s_k + (s0 + gq) * YL + 2 * q;
        float sum[4];
#pragma unroll 4
        for (int k = 0; k < DK / 16; ++k) {
            PartsA a[1];
            PartsB z[1];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float2 lo = two(row + 16 * k + 8 * x), hi = two(row + 8 * XL + 16 * k + 8 * x), b2 = two(col + 16 * k + 8 * x);
                a[0].set(2 * x, lo.x, lo.y);
                a[0].set(2 * x + 1, hi.x, hi.y);
                z[0].set(x, b2.x, b2.y);
            }
            float part[4];
            mma_sum<1>(part, a, z);
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[e] = k == 0 ? part[e] : sum[e] + part[e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = gq + 8 * (e >> 1), s = s0 + 2 * q + (e & 1);
            // what lies behind the diagonal is dropped, also where it is not finite
            s_m[m * kChunk * kChunk + t * kChunk + s] = (REM && m == 0 ? s < t : s <= t) ? sum[e] * s_w[t * kDecayLd + s + 1] : 0.0f;
        }
    }
    __syncthreads();
    // ---- columns: key channels first, then value columns; row t of a product, elements 4 i .. + 3 ----
    auto row4 = [&](int m, int t, int i) { return *reinterpret_cast<const float4*>(s_m + m * kChunk * kChunk + t * kChunk + 4 * i); };
    for (int c = threadIdx.x; c < DK; c += 128) {
        float xw[kChunk];
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
            const float w = s_w[t * kDecayLd];
            float o = w * s_r[t * XL + c];
            if (REM) {
                xw[t] = w * s_u[t * XL + c];
#pragma unroll
                for (int i = 0; 4 * i < t; ++i) chunk_take(xw[t], row4(0, t, i), xw, i, t, -1.0f);
#pragma unroll
                for (int i = 0; 4 * i <= t; ++i) chunk_take(o, row4(kR, t, i), xw, i, t + 1, -1.0f);
                s_u[t * XL + c] = xw[t];
            }
            s_r[t * XL + c] = o;
            s_k[t * YL + c] *= s_w[(kChunk - 1) * kDecayLd + t + 1];
        }
        out[chunk_key_floats(REM, DK) - DK + c] = s_w[(kChunk - 1) * kDecayLd];
    }
    asm volatile("" ::: "memory");               // the products are read again: kept for both loops they do not fit the registers (DK 128)
    float* cols = out + chunk_key_floats(REM, DK);
    for (int j = j_first; j < n_cols; j += 128) {
        if (!EARLY || j != j_first) chunk_values(A, t0 + r0, n, h, j, v);
        chunk_value_parts<REM>(cols, j, v);
        float* to = cols + (j / kChunkCols) * chunk_col_floats(REM) + j % kChunkCols;
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
            if (t % 4 == 0) asm volatile("" ::: "memory");      // (all rows read ahead would not fit either)
            float o = 0.0f;
            if (REM) {
                float seen = 0.0f;
#pragma unroll
                for (int i = 0; 4 * i < t; ++i) chunk_take(seen, row4(0, t, i), v, i, t, 1.0f);
                to[chunk_place(t) * kChunkCols] = seen;
                v[t] -= seen;                    // what the token writes
            }
#pragma unroll
            for (int i = 0; 4 * i <= t; ++i) chunk_take(o, row4(kR, t, i), v, i, t + 1, 1.0f);
            to[(REM ? kChunk + t : t) * kChunkCols] = o;
        }
    }
    __syncthreads();
    chunk_fragments<DK, REM>(out, s_u, s_r, s_k, s_k, -1.0f);
}

struct ChunkArgs {
    int H, d, dv;
    const float* rec;
    int cap;
    float q_scale;
    const int32_t *seq_start, *seq_pos0, *seq_slot;
    size_t slot_floats, state_off;
    int n_slots;
    int32_t* err;
    // A further state column per head whose value is 1 for every token, behind the value columns: its rows live at unit_off inside the slot ([H][d]), its
    // product with the query goes to unit_out[t * H + h].  nullptr: none.
    float* unit_out;
    size_t unit_off;
    ConvIo conv;                         // taps > 1: the blocks of a sequence also bring these inputs in the slot up to date
};
__host__ __device__ constexpr int chunk_warps(int DK) { return DK >= 64 ? 4 : DK / 16; }
__host__ __device__ constexpr int chunk_ring(int DK) { return DK <= 128 ? 3 : 2; }
// ring | the state [2][NT][DK][8] | V's writes, as much | shares of o, of seen [2][NT][warps][16][8]
__host__ __device__ constexpr size_t chunk_smem(bool removes, int DK, int NT) {
    return (chunk_ring(DK) * (chunk_key_floats(removes, DK) + NT * chunk_col_floats(removes)) + NT * kChunkCols * (4 * DK + (removes ? 4 : 2) * chunk_warps(DK) * kChunk)) * sizeof(float);
}

// Warps 0 .. NW - 1 carry the state from chunk to chunk, DK / NW channels each; warps NW .. 2 NW - 1 do for the same channels what that chain need not wait for
// -- V's writes of the next chunk, the outputs of this one --; the last warp copies records.  NT blocks of eight columns.
template <int DK, bool REM, int NT>
__global__ void __launch_bounds__(chunk_warps(DK) * 64 + 32, DK <= 32 ? 4 : DK <= 64 ? 2 : 1) chunk_scan_kernel(const ChunkArgs A, float* state_pool, float* __restrict__ o_raw) {
    dep_wait();
    dep_go();
    constexpr int NW = chunk_warps(DK), CW = DK / NW, MT = CW / 16, KS = CW / 16, NB = chunk_ring(DK), KF = chunk_key_floats(REM, DK), CF = chunk_col_floats(REM);
    constexpr int MX = REM ? 2 : 1, CB = kChunkCols, SH = kChunk * CB, SLOT = KF + NT * CF, FR = chunk_frag(DK), YF = DK / 16 * MX * FR;
    constexpr bool SPLIT = chunk_split(DK);
    extern __shared__ __align__(16) float sh[];
    __shared__ uint64_t full[NB], empty[NB];
    float* state = sh + NB * SLOT;                      // [2][NT][DK][CB]: the state before a chunk, on its way from result to operand
    float* writes = state + 2 * NT * DK * CB;           // [2][NW][NT][MT][32][4]: Y_v V
    float* share_o = writes + 2 * NT * DK * CB;         // [2][NT][NW][16][CB]
    float* share_s = share_o + 2 * NT * NW * SH;        // [2][NT][NW][16][CB]
    const int d = A.d, dv = A.dv, columns = dv + (A.unit_out ? 1 : 0), NS = chunk_blocks(columns), NC = (NS + NT - 1) / NT;
    const int item = blockIdx.x % (A.H * NC), seq = blockIdx.x / (A.H * NC);
    const int h = item / NC, blk = item % NC * NT, j0 = blk * CB;
    const int t0 = A.seq_start[seq], t1 = A.seq_start[seq + 1];
    const int slot = A.seq_slot[seq];
    if (slot < 0 || slot >= A.n_slots) {
        if (threadIdx.x == 0) atomicExch(A.err, 2);
        return;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) { umma::bar_init(&full[i], 1); umma::bar_init(&empty[i], 2 * NW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int chunks = (t1 - t0 + kChunk - 1) / kChunk;
    if (chunks == 0) return;
    const int lane = threadIdx.x & 31, gq = lane >> 2, q = lane & 3;
    const int role = (threadIdx.x >> 5) / NW, warp = (threadIdx.x >> 5) % NW, c0 = warp * CW;
    if (role == 2) {
        if (lane == 0) {
            const size_t stride = KF + (size_t)NS * CF;
            const float* rec = A.rec + ((size_t)h * A.cap + chunk_first(t0, seq)) * stride;
            const uint32_t col_bytes = (uint32_t)min(NT, NS - blk) * CF * 4;
            for (int i = 0, b = 0, round = 0; i < chunks; ++i, rec += stride) {
                if (round > 0) umma::bar_wait(&empty[b], (round - 1) & 1);
                umma::bar_expect_tx(&full[b], KF * 4 + col_bytes);
                bulk_copy(sh + b * SLOT, rec, KF * 4, &full[b]);
                bulk_copy(sh + b * SLOT + KF, rec + KF + blk * CF, col_bytes, &full[b]);
                if (++b == NB) { b = 0; ++round; }
            }
        }
        return;
    }
    auto all_barrier = [&] { asm volatile("bar.sync 1, %0;" ::"n"(NW * 64) : "memory"); };
    // operands whose rows lie in the order of chunk_place: of the state before a chunk, this warp's channels
    auto state_parts = [&](const float* at, PartsB (&sb)[KS]) {
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int x = 0; x < 2; ++x) sb[k].set(x, at[(16 * k + 8 * x + q) * CB + gq], at[(16 * k + 8 * x + 4 + q) * CB + gq]);
    };
    const int g_at = chunk_place(gq);
    auto put_share = [&](float* to, int row, const float (&sum)[4]) {
        *reinterpret_cast<float2*>(to + row * CB + 2 * q) = make_float2(sum[0], sum[1]);
        *reinterpret_cast<float2*>(to + (row + 8) * CB + 2 * q) = make_float2(sum[2], sum[3]);
    };
    int b = 0;                                          // the chunk's slot in the ring, and the parity of its round
    uint32_t parity = 0;
    auto next_slot = [&] {
        if (++b == NB) { b = 0; parity ^= 1u; }
    };
    if (role == 1) {
        auto make_writes = [&](const float* R, float* to) {
            PartsB vb[NT][1];
#pragma unroll
            for (int n = 0; n < NT; ++n) vb[n][0].load(R + KF + n * CF + MX * SH, lane);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                PartsA y[1];
                y[0].load<SPLIT>(R + YF + (warp * MT + m) * MX * FR, lane);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    float sum[4];
                    mma_sum<1>(sum, y, vb[n]);
                    reinterpret_cast<float4*>(to + ((warp * NT + n) * MT + m) * 128)[lane] = make_float4(sum[0], sum[1], sum[2], sum[3]);
                }
            }
        };
        const int first = threadIdx.x - NW * 32;
        if (A.conv.taps > 1)
            for (int c = item * NW * 32 + first; c < A.conv.ch; c += A.H * NC * NW * 32) conv_state_update(A.conv, state_pool, seq, c);
        umma::bar_wait(&full[0], 0);
        make_writes(sh, writes);
        for (int i = 0; i < chunks; ++i) {
            const float* R = sh + b * SLOT;
            const int now = b;
            PartsA X[KS];
#pragma unroll
            for (int k = 0; k < KS; ++k) X[k].template load<SPLIT>(R + ((warp * KS + k) * MX + MX - 1) * FR, lane);
            all_barrier();                               // the state before chunk i is there, V's writes of chunk i are
            float* part = share_o + (i & 1) * NT * NW * SH;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                PartsB sb[KS];
                state_parts(state + ((i & 1) * NT + n) * DK * CB + c0 * CB, sb);
                float sum[4];
                mma_sum<KS>(sum, X, sb);
                put_share(part + (n * NW + warp) * SH, gq, sum);
            }
            asm volatile("bar.sync 2, %0;" ::"n"(NW * 32) : "memory");
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int x = first; x < SH; x += NW * 32) {
                    float p[NW];
#pragma unroll
                    for (int w = 0; w < NW; ++w) p[w] = part[(n * NW + w) * SH + x];
                    const float o = (NW == 4 ? (p[0] + p[1]) + (p[NW - 2] + p[NW - 1]) : p[0] + p[NW - 1]) + R[KF + n * CF + (MX - 1) * SH + x];
                    const int t = t0 + i * kChunk + x / CB, j = j0 + n * CB + x % CB;
                    if (t < t1 && j < columns) (j < dv ? o_raw[((size_t)t * A.H + h) * dv + j] : A.unit_out[(size_t)t * A.H + h]) = o * A.q_scale;
                }
            __syncwarp();
            if (lane == 0) bar_arrive(&empty[now]);
            next_slot();
            if (i + 1 < chunks) {
                umma::bar_wait(&full[b], parity);
                make_writes(sh + b * SLOT, writes + ((i + 1) & 1) * NT * DK * CB);
            }
        }
        return;
    }
    // element (channel i, column j) of the state lives at
    float* slot_at = state_pool + (size_t)slot * A.slot_floats;
    auto state_at = [&](int i, int j) { return j < dv ? slot_at + A.state_off + ((size_t)h * d + i) * dv + j : slot_at + A.unit_off + (size_t)h * d + i; };
    const bool fresh = A.seq_pos0[seq] == 0;
    float S[NT][MT][4];                                 // rows c0 + 16 m + gq (+ 8), columns j0 + 8 n + 2 q (+ 1)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = c0 + 16 * m + gq + 8 * (e >> 1), j = j0 + 8 * n + 2 * q + (e & 1);
                S[n][m][e] = !fresh && i < d && j < columns ? *state_at(i, j) : 0.0f;
            }
    PartsA X[KS];
    auto load_x = [&](const float* R) {
        if (REM) {
#pragma unroll
            for (int k = 0; k < KS; ++k) X[k].template load<SPLIT>(R + (warp * KS + k) * MX * FR, lane);
        }
    };
    umma::bar_wait(&full[0], 0);
    load_x(sh);
    for (int i = 0; i < chunks; ++i) {
        const float *R = sh + b * SLOT, *W = R + KF - DK + c0;
        const int now = b;
        float *at = state + (i & 1) * NT * DK * CB + c0 * CB, *part = share_s + (i & 1) * NT * NW * SH;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                float* to = at + n * DK * CB + (16 * m + g_at) * CB + 2 * q;
                *reinterpret_cast<float2*>(to) = make_float2(S[n][m][0], S[n][m][1]);
                *reinterpret_cast<float2*>(to + 8 * CB) = make_float2(S[n][m][2], S[n][m][3]);
            }
        __syncwarp();
        if (REM) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                PartsB sb[KS];
                state_parts(at + n * DK * CB, sb);
                float sum[4];
                mma_sum<KS>(sum, X, sb);
                put_share(part + (n * NW + warp) * SH, g_at, sum);
            }
        }
        // what does not wait for the other warps' shares
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float w0 = W[16 * m + gq], w1 = W[16 * m + gq + 8];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][m][e] *= e < 2 ? w0 : w1;
        }
        PartsA Y[REM ? MT : 1][1];
        if (REM) {
#pragma unroll
            for (int m = 0; m < MT; ++m) Y[m][0].template load<SPLIT>(R + YF + ((warp * MT + m) * MX + MX - 1) * FR, lane);
        }
        next_slot();
        if (i + 1 < chunks) {
            umma::bar_wait(&full[b], parity);
            load_x(sh + b * SLOT);
        }
        all_barrier();
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (REM) {
                PartsB seen[1];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    float z[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int e = (8 * k + 4 * x + q) * CB + gq;
                        float p[NW];
#pragma unroll
                        for (int w = 0; w < NW; ++w) p[w] = part[(n * NW + w) * SH + e];
                        z[x] = (NW == 4 ? (p[0] + p[1]) + (p[NW - 2] + p[NW - 1]) : p[0] + p[NW - 1]) + R[KF + n * CF + e];
                    }
                    seen[0].set(k, z[0], z[1]);
                }
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    float sum[4];
                    mma_sum<1>(sum, Y[m], seen);
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[n][m][e] += sum[e];
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 w4 = reinterpret_cast<const float4*>(writes + (i & 1) * NT * DK * CB + ((warp * NT + n) * MT + m) * 128)[lane];
                S[n][m][0] += w4.x;
                S[n][m][1] += w4.y;
                S[n][m][2] += w4.z;
                S[n][m][3] += w4.w;
            }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[now]);
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = c0 + 16 * m + gq + 8 * (e >> 1), j = j0 + 8 * n + 2 * q + (e & 1);
                if (i < d && j < columns) *state_at(i, j) = S[n][m][e];
            }
}

}  // namespace lm
}  // namespace smol
