// The recurrences over a request's tokens: one matrix of state per head, S [dk, dv] in float32, whose columns (one value
// dimension each) go through the tokens in order, every column on its own:
//
//   gdr_recurrent           S <- g S;        u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q   (g: a number per head and token)
//   gdr_channel_recurrent   S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q   (g: one per key channel)
//   gla_recurrent           S <- diag(g) S;                         S <- S + k v^T;  o = S^T q
//
// Four tokens are taken at a time.  With S the state ahead of them, G(i..j) the product of the decays of tokens i to j,
//
//   a_j = S^T (G(1..j) k_j),  b_j = S^T (G(1..j) q_j)
//   u_j = beta_j (v_j - a_j - sum_{i<j} u_i (k_i . G(i+1..j) k_j));      o_j = b_j + sum_{i<=j} u_i (k_i . G(i+1..j) q_j)
//   S  <- G(1..4) S + sum_i (G(i+1..4) k_i) u_i^T
//
// which is the same arithmetic in another order: no quotient of decays is formed.  The scaled vectors and the sixteen
// products between tokens do not depend on the column: the CTA forms them once for its columns (one warp a stretch of four
// tokens) where the tokens lie in shared memory.  What is left per column is 13 multiply-adds a key channel for four tokens.
//
// LPC lanes share NC neighbouring columns, R key channels a lane: vectors leave shared memory as 16-byte loads that feed NC
// columns (the lanes that load the same vector are neighbours: measured, a warp's 16-byte load takes two cycles of shared
// memory where neighbouring lanes agree and four however else they agree), products run on pairs of channels
// (fma.rn.f32x2), and the lanes' sums are exchanged by halves.  Tokens arrive by asynchronous copies, a stage of some blocks
// at a time.
//
// Requests with fewer than four tokens in a step (decoded tokens) go token by token, fetched straight into registers: in a
// kernel of their own where a step has one token a request, beside the portions else.
//
// What a request's bits depend on: its tokens, its state and where its prompt was cut (blocks count from a portion's first
// token), not the requests that share its step or how many columns and channels a launch gives a lane.
//
// What bounds it: 13 multiply-adds a channel and column for four tokens are 97 us of 2,048 tokens on 32 heads of 128 x 128;
// with the exchange, the loads and the stages a warp issues 700 instructions for those 208, most of them depending on the one
// before, and one or two warps a scheduler are all that the columns give.  Measured there (decay per channel / per head /
// linear): 376 / 365 / 268 us; 830 / 800 / 670 with one column per 16 lanes, a full exchange per sum, one or two tokens at a time.
//
// A request's slot of state holds S as [heads][dv][dk] (a column's dk values side by side) at its start.  Rows of qkv are
// [q: G*dk | k: G*dk | v: H*dv]; head h of H reads q/k head h / (H / G).
#include <type_traits>

#include "async_copy.cuh"
#include "rows.cuh"

namespace {

enum Rule : int { DELTA_HEAD = 0, DELTA_CHANNEL = 1, LINEAR = 2 };

constexpr int TB = 4;                  // tokens of a block
constexpr int DOTS = 16;               // products between the tokens of a block: k_i k_j (i < j), then k_i q_j (i <= j)
__device__ constexpr int kk_at(int i, int j) { return i * 3 - i * (i - 1) / 2 + j - i - 1; }
__device__ constexpr int kq_at(int i, int j) { return 6 + i * 4 - i * (i - 1) / 2 + j - i; }

// Two float32 in one 64-bit register.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ float sum2(f2 v) {
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Sums of v[0..NV) over the LANES lanes whose numbers differ in li only (li: the lane's number over STEP), exchanged by
// halves: afterwards lane li holds, in v[0], v[1], ..., the sums of values li * NV / LANES and following (NV >= LANES), or in
// v[0] that of value li / (LANES / NV).
template <int NV, int LANES, int STEP>
__device__ __forceinline__ void scatter_sums(float* v, int li) {
    if constexpr (LANES > 1) {
        constexpr int off = LANES / 2;
        if constexpr (NV > 1) {
            const bool up = li & off;
#pragma unroll
            for (int i = 0; i < NV / 2; ++i) {
                const float send = up ? v[i] : v[i + NV / 2], keep = up ? v[i + NV / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off * STEP);
            }
            scatter_sums<NV / 2, off, STEP>(v, li);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off * STEP);
            scatter_sums<1, off, STEP>(v, li);
        }
    }
}

// How a launch cuts the work: THREADS of a CTA hold columns, ch tokens a stage (a multiple of TB).  SPLIT: as many threads
// more fetch and prepare the stages ahead.
template <int R, int LPC, int NC, int THREADS, bool SPLIT> struct Cut {
    static constexpr int DKP = R * LPC, COLS = THREADS / LPC * NC;
    static constexpr int CH = DKP <= 128 ? 16 : DKP <= 512 ? 8 : 4;
    static constexpr int STAGES = SPLIT ? 3 : 2;
    static constexpr int ALL = SPLIT ? 2 * THREADS : THREADS;
    // behind a stage's vectors and numbers: per block (and per token of an incomplete block) the block's decay and its products
    __host__ __device__ static constexpr int block_rows(int ch) { return ch / TB + TB - 1; }
    __host__ __device__ static constexpr int stage_floats(int ch) { return ch * (3 * DKP + COLS + 2) + block_rows(ch) * (DKP + DOTS); }
    __host__ __device__ static constexpr int floats(int ch) { return STAGES * stage_floats(ch); }
};

// A lane's share of a column's sum S^T x, x in groups of four channels: pairs of channels in float32x2.  Sixteen channels a lane
// are two chains of eight, so that 8 lanes of sixteen and 16 lanes of eight add in one order: what a step's launch gives a lane
// does not show in the result.
template <int R> __device__ __forceinline__ float lane_sum(const f2* s, const ulonglong2* x) {
    constexpr int CHAINS = R == 16 ? 2 : 1;
    float part[CHAINS];
#pragma unroll
    for (int h = 0; h < CHAINS; ++h) {
        f2 y = fma2(s[2 * h + 1], x[h].y, mul2(s[2 * h], x[h].x));
#pragma unroll
        for (int r = h + CHAINS; r < R / 4; r += CHAINS) y = fma2(s[2 * r + 1], x[r].y, fma2(s[2 * r], x[r].x, y));
        part[h] = sum2(y);
    }
    return CHAINS == 2 ? part[0] + part[CHAINS - 1] : part[0];
}

// Named barriers of a CTA: `count` threads meet, or come by.
__device__ __forceinline__ void meet(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void come_by(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

// The first channel of lane li's r-th group of four, LPC lanes a column.
template <int LPC> __device__ __forceinline__ int channel_of(int r, int li) { return r * (4 * LPC) + 4 * li; }

// Four channels of a row from d on, zeros beyond dk.
template <bool BY4> __device__ __forceinline__ ulonglong2 load_group(const float* row, int d, int dk) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (BY4) {
        if (d < dk) v = Vec4<float>::load(row + d);
    } else {
        if (d < dk) v.x = row[d];
        if (d + 1 < dk) v.y = row[d + 1];
        if (d + 2 < dk) v.z = row[d + 2];
        if (d + 3 < dk) v.w = row[d + 3];
    }
    return make_ulonglong2(pack2(v.x, v.y), pack2(v.z, v.w));
}
template <bool BY4> __device__ __forceinline__ void store_group(float* row, int d, int dk, f2 lo, f2 hi) {
    float x[4];
    unpack2(lo, x[0], x[1]);
    unpack2(hi, x[2], x[3]);
    if constexpr (BY4) {
        if (d < dk) Vec4<float>::store(row + d, make_float4(x[0], x[1], x[2], x[3]));
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (d + u < dk) row[d + u] = x[u];
    }
}

// Where the tokens, states and results of a launch lie.
struct Rows {
    const float* qkv; const float* beta; const float* decay;
    float* state; long state_stride;
    const int* seq_q_start; const int* seq_q_len; const int* seq_slot;
    float* o;
    int G, H, dk, dv;
};

// A request's tokens one by one, for a decoded token or a few (fewer than a block's): a lane fetches its channels of the
// token's vectors and of its columns' state from global memory, and nothing passes through shared memory.
template <int RULE, int R, int LPC, int NC, bool BY4>
__device__ __forceinline__ void few_tokens(const Rows& a, int seq, int head, int li, int col0, int L) {
    constexpr bool DELTA = RULE != LINEAR;
    constexpr int PW = 32 / LPC;
    const int dk = a.dk, dv = a.dv, qk = a.G * dk, C = 2 * qk + a.H * dv, g = head / (a.H / a.G);
    float* S = a.state + (size_t)a.seq_slot[seq] * a.state_stride + (size_t)head * dv * dk;
    f2 s[NC][R / 2];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
            const ulonglong2 v = load_group<BY4>(S + (size_t)(col0 + c) * dk, channel_of<LPC>(r, li), col0 + c < dv ? dk : 0);
            s[c][2 * r] = v.x;
            s[c][2 * r + 1] = v.y;
        }
#pragma unroll 1
    for (int t = 0; t < L; ++t) {
        const size_t row = (size_t)a.seq_q_start[seq] + t;
        const float* qp = a.qkv + row * C + (size_t)g * dk;
        ulonglong2 q[R / 4], k[R / 4], w[R / 4];
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
            const int d = channel_of<LPC>(r, li);
            q[r] = load_group<BY4>(qp, d, dk);
            k[r] = load_group<BY4>(qp + qk, d, dk);
            if constexpr (RULE == DELTA_HEAD) {
                const float x = a.decay[row * a.H + head];
                w[r].x = w[r].y = pack2(x, x);
            } else w[r] = load_group<BY4>(a.decay + (row * a.H + head) * dk, d, dk);
        }
        float v[NC], bt = 1.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = col0 + c < dv ? a.qkv[row * C + 2 * qk + (size_t)head * dv + col0 + c] : 0.0f;
        if constexpr (DELTA) bt = a.beta[row * a.H + head];
        constexpr int SUMS = 1 + NC * (DELTA ? 2 : 1);           // k.q, then S^T q and S^T k of every column
        float sum[SUMS];
        f2 kf[R / 2];
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
            kf[2 * r] = k[r].x;
            kf[2 * r + 1] = k[r].y;
        }
        sum[0] = lane_sum<R>(kf, q);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
                s[c][2 * r] = mul2(s[c][2 * r], w[r].x);
                s[c][2 * r + 1] = mul2(s[c][2 * r + 1], w[r].y);
            }
            sum[1 + c] = lane_sum<R>(s[c], q);
            if constexpr (DELTA) sum[1 + NC + c] = lane_sum<R>(s[c], k);
        }
#pragma unroll
        for (int off = LPC / 2; off > 0; off >>= 1)
#pragma unroll
            for (int i = 0; i < SUMS; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], off * PW);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            float u = v[c];
            if constexpr (DELTA) u = bt * (v[c] - sum[1 + NC + c]);
            const f2 uu = pack2(u, u);
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
                s[c][2 * r] = fma2(k[r].x, uu, s[c][2 * r]);
                s[c][2 * r + 1] = fma2(k[r].y, uu, s[c][2 * r + 1]);
            }
            if (li == 0 && col0 + c < dv) a.o[row * a.H * dv + (size_t)head * dv + col0 + c] = fmaf(u, sum[0], sum[1 + c]);
        }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < R / 4; ++r)
            if (col0 + c < dv) store_group<BY4>(S + (size_t)(col0 + c) * dk, channel_of<LPC>(r, li), dk, s[c][2 * r], s[c][2 * r + 1]);
}

// Steps of one token a request (decoding).
template <int RULE, int R, int LPC, int NC, bool BY4>
__global__ void __launch_bounds__(128)
one_token_kernel(const Rows a) {
    // The kernels behind are let in when the one ahead has ended, not before: CTAs of the output product, which hold an SM's
    // shared memory for their weights, else take the SMs that this kernel has not filled (three decoded tokens, a decay per
    // channel, 16 heads: a layer 37.7 us so, 35.2 in this order).  Portions are slower with it (linear, 700 tokens 279 and 332).
    fb_pdl_wait();
    fb_pdl_launch_dependents();
    constexpr int PW = 32 / LPC, COLS = 128 / LPC * NC;
    const int seq = blockIdx.x / a.H, head = blockIdx.x - seq * a.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = a.seq_q_len[seq];
    if (L > 0) few_tokens<RULE, R, LPC, NC, BY4>(a, seq, head, lane / PW, blockIdx.y * COLS + (warp * PW + lane % PW) * NC, L);
}

// BY4: rows of q, k, decay and the state start on 16-byte borders and dk is a multiple of 4.
template <int RULE, int R, int LPC, int NC, int THREADS, bool BY4, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 2 * THREADS : THREADS)
recurrent_kernel(const Rows a_, int ch) {
    const float* __restrict__ qkv = a_.qkv;
    const float* __restrict__ beta = a_.beta;
    const float* __restrict__ decay = a_.decay;
    float* __restrict__ o = a_.o;
    const int G = a_.G, H = a_.H, dk = a_.dk, dv = a_.dv;
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    using C_ = Cut<R, LPC, NC, THREADS, SPLIT>;
    constexpr int DKP = C_::DKP, COLS = C_::COLS, WARPS = THREADS / 32;
    constexpr bool DELTA = RULE != LINEAR;
    extern __shared__ __align__(16) float sh[];
    const int seq = blockIdx.x / H, head = blockIdx.x - seq * H;
    const int g = head / (H / G);
    const int tid = threadIdx.x & (THREADS - 1), warp = tid >> 5, lane = tid & 31;    // (THREADS: a power of two)
    constexpr int PW = 32 / LPC;                                 // groups of columns a warp; their lanes alternate
    const int li = lane / PW, group = warp * PW + lane % PW, col0 = blockIdx.y * COLS + group * NC;
    const int qk = G * dk, C = 2 * qk + H * dv;
    const int start = a_.seq_q_start[seq], L = a_.seq_q_len[seq];
    if (L < TB) {                                                // a decoded token beside portions
        if (L > 0 && threadIdx.x < THREADS) few_tokens<RULE, R, LPC, NC, BY4>(a_, seq, head, li, col0, L);
        return;
    }
    float* S = a_.state + (size_t)a_.seq_slot[seq] * a_.state_stride + (size_t)head * dv * dk;
    auto stage = [&](int i) { return sh + i % C_::STAGES * C_::stage_floats(ch); };
    auto ends_of = [&](float* st) { return st + ch * (3 * DKP + COLS + 2); };                 // [block rows][DKP]
    auto dots_of = [&](float* st) { return ends_of(st) + C_::block_rows(ch) * DKP; };         // [block rows][DOTS]

    // a stage: q, k, decay [ch][DKP] each (rows padded with zeros beyond dk; a decay per head leaves the third free),
    // v [ch][COLS], beta [ch], decay per head [ch]
    auto fetch = [&](int t0, float* st) {
        const int cnt = min(ch, L - t0);
        float* qs = st;
        float* ks = qs + ch * DKP;
        float* gs = ks + ch * DKP;
        float* vs = gs + ch * DKP;
        constexpr int W = BY4 ? 4 : 1;
        for (int e = tid * W; e < cnt * DKP; e += THREADS * W) {
            const int t = e / DKP, d = e - t * DKP;
            const size_t row = (size_t)(start + t0 + t);
            if (d < dk) {
                const float* rowp = qkv + row * C + (size_t)g * dk + d;
                const float* gp = decay + (row * H + head) * dk + d;
                if constexpr (BY4) {
                    cp_async16(qs + e, rowp);
                    cp_async16(ks + e, rowp + qk);
                    if constexpr (RULE != DELTA_HEAD) cp_async16(gs + e, gp);
                } else {
                    cp_async4(qs + e, rowp);
                    cp_async4(ks + e, rowp + qk);
                    if constexpr (RULE != DELTA_HEAD) cp_async4(gs + e, gp);
                }
            } else {
#pragma unroll
                for (int u = 0; u < W; ++u) qs[e + u] = ks[e + u] = gs[e + u] = 0.0f;
            }
        }
        for (int e = tid; e < cnt * COLS; e += THREADS) {
            const int t = e / COLS, c2 = blockIdx.y * COLS + (e - t * COLS);
            if (c2 < dv) cp_async4(vs + e, qkv + (size_t)(start + t0 + t) * C + 2 * qk + (size_t)head * dv + c2);
            else vs[e] = 0.0f;
        }
        if (DELTA && tid < cnt) {
            cp_async4(vs + ch * COLS + tid, beta + (size_t)(start + t0 + tid) * H + head);
            if constexpr (RULE == DELTA_HEAD) cp_async4(vs + ch * (COLS + 1) + tid, decay + (size_t)(start + t0 + tid) * H + head);
        }
        cp_async_commit();
    };

    // The vectors of the N tokens from `t` on made what the columns want of them, in place (q: G(1..j) q_j; k: G(1..j) k_j;
    // decay: G(j+1..N) k_j), the block's decay, and the products between its tokens, by one warp.
    auto prepare = [&](auto n_tokens, float* st, int t, int row) {
        constexpr int N = decltype(n_tokens)::value;
        float* qs = st + t * DKP;
        float* ks = qs + ch * DKP;
        float* gs = ks + ch * DKP;
        float kk[6] = {}, kq[10] = {};
        for (int d = 4 * lane; d < DKP; d += 128) {
            float q[N][4], k[N][4], w[N][4], all[4];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float4 a = Vec4<float>::load(qs + j * DKP + d), b = Vec4<float>::load(ks + j * DKP + d);
                q[j][0] = a.x; q[j][1] = a.y; q[j][2] = a.z; q[j][3] = a.w;
                k[j][0] = b.x; k[j][1] = b.y; k[j][2] = b.z; k[j][3] = b.w;
                if constexpr (RULE == DELTA_HEAD) {
                    const float x = (st + ch * (3 * DKP + COLS + 1))[t + j];
                    w[j][0] = w[j][1] = w[j][2] = w[j][3] = x;
                } else {
                    const float4 x = Vec4<float>::load(gs + j * DKP + d);
                    w[j][0] = x.x; w[j][1] = x.y; w[j][2] = x.z; w[j][3] = x.w;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float e[N];                            // G(i+1..j) k_i, in the end j = N
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    e[i] = k[i][u];
                    kq[kq_at(i, i) - 6] = fmaf(e[i], q[i][u], kq[kq_at(i, i) - 6]);
#pragma unroll
                    for (int j = i + 1; j < N; ++j) {
                        e[i] *= w[j][u];
                        if constexpr (DELTA) kk[kk_at(i, j)] = fmaf(e[i], k[j][u], kk[kk_at(i, j)]);
                        kq[kq_at(i, j) - 6] = fmaf(e[i], q[j][u], kq[kq_at(i, j) - 6]);
                    }
                }
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    all[u] = j == 0 ? w[0][u] : all[u] * w[j][u];
                    q[j][u] *= all[u];
                    k[j][u] *= all[u];
                    w[j][u] = e[j];
                }
            }
            Vec4<float>::store(ends_of(st) + row * DKP + d, make_float4(all[0], all[1], all[2], all[3]));
#pragma unroll
            for (int j = 0; j < N; ++j) {
                Vec4<float>::store(qs + j * DKP + d, make_float4(q[j][0], q[j][1], q[j][2], q[j][3]));
                if constexpr (DELTA) Vec4<float>::store(ks + j * DKP + d, make_float4(k[j][0], k[j][1], k[j][2], k[j][3]));
                Vec4<float>::store(gs + j * DKP + d, make_float4(w[j][0], w[j][1], w[j][2], w[j][3]));
            }
        }
        if constexpr (N == 1) {
            const float x = fb_warp_sum(kq[0]);
            if (lane == 0) dots_of(st)[row * DOTS + 6] = x;
        } else {
            float v[DOTS];
#pragma unroll
            for (int i = 0; i < 6; ++i) v[i] = kk[i];
#pragma unroll
            for (int i = 0; i < 10; ++i) v[6 + i] = kq[i];
            scatter_sums<DOTS, 32, 1>(v, lane);
            if (!(lane & 1)) dots_of(st)[row * DOTS + (lane >> 1)] = v[0];
        }
    };

    const int n_stages = (L + ch - 1) / ch;
    const std::integral_constant<int, TB> block_of;
    const std::integral_constant<int, 1> token;
    // A warp's share of a stage's blocks (and of the tokens behind them).
    auto prepare_stage = [&](int i) {
        const int cnt = min(ch, L - i * ch), blocks = cnt / TB, rows = blocks + cnt % TB;
        for (int x = warp; x < rows; x += WARPS) {
            if (x < blocks) prepare(block_of, stage(i), x * TB, x);
            else prepare(token, stage(i), blocks * TB + x - blocks, x);
        }
    };
    // Barriers: 1 + slot: the stage in that slot is prepared; 1 + STAGES + slot: its readers are through.
    if (SPLIT && threadIdx.x >= THREADS) {
        for (int i = 0; i < n_stages; ++i) {
            if (i == 0) fetch(0, stage(0));
            if (i + 1 < n_stages) {
                if (i + 1 >= C_::STAGES) meet(1 + C_::STAGES + (i + 1) % C_::STAGES, 2 * THREADS);
                fetch((i + 1) * ch, stage(i + 1));
                cp_async_wait<1>();
            } else cp_async_wait<0>();
            meet(1 + 2 * C_::STAGES, THREADS);           // every fetching thread's copies are there
            prepare_stage(i);
            come_by(1 + i % C_::STAGES, 2 * THREADS);
        }
        return;
    }

    f2 s[NC][R / 2];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
            const ulonglong2 v = load_group<BY4>(S + (size_t)(col0 + c) * dk, channel_of<LPC>(r, li), col0 + c < dv ? dk : 0);
            s[c][2 * r] = v.x;
            s[c][2 * r + 1] = v.y;
        }

    // The vectors of N tokens that the state is multiplied with, in registers.
    struct Vectors { ulonglong2 q[TB][R / 4], k[DELTA ? TB : 1][R / 4]; };
    auto load = [&](auto n_tokens, const float* st, int t, Vectors& x) {
        constexpr int N = decltype(n_tokens)::value;
        const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(st + t * DKP) + li;
        const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(st + (ch + t) * DKP) + li;
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
                if constexpr (DELTA) x.k[j][r] = k4[j * (DKP / 4) + r * LPC];
                x.q[j][r] = q4[j * (DKP / 4) + r * LPC];
            }
    };

    // N tokens of this lane's columns.
    auto advance = [&](auto n_tokens, float* st, int t, int row, long out_row) {
        constexpr int N = decltype(n_tokens)::value;
        constexpr int NV = NC * N, REM = NV >= LPC ? NV / LPC : 1, SPREAD = NV >= LPC ? 1 : LPC / NV;
        const ulonglong2* w4 = reinterpret_cast<const ulonglong2*>(st + (2 * ch + t) * DKP) + li;
        const ulonglong2* e4 = reinterpret_cast<const ulonglong2*>(ends_of(st) + row * DKP) + li;
        Vectors x;
        load(n_tokens, st, t, x);
        // a = S^T k (scaled), b = S^T q (scaled): value c * N + j of column c, token j
        float a[NV], b[NV];
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                b[c * N + j] = lane_sum<R>(s[c], x.q[j]);
                if constexpr (DELTA) a[c * N + j] = lane_sum<R>(s[c], x.k[j]);
            }
        float D[DOTS];
#pragma unroll
        for (int i = 0; i < DOTS / 4; ++i) {
            const float4 y = Vec4<float>::load(dots_of(st) + row * DOTS + 4 * i);
            D[4 * i] = y.x; D[4 * i + 1] = y.y; D[4 * i + 2] = y.z; D[4 * i + 3] = y.w;
        }
        const float* vs = st + 3 * ch * DKP;
        float u[NC][N];
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int c = 0; c < NC; ++c) u[c][j] = vs[(t + j) * COLS + group * NC + c];
        if constexpr (DELTA) {
            scatter_sums<NV, LPC, PW>(a, li);
            float all[NV];
#pragma unroll
            for (int m = 0; m < NV; ++m) all[m] = __shfl_sync(0xffffffffu, a[m % REM], m / REM * SPREAD * PW + lane % PW);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float bt = vs[ch * COLS + t + j];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float y = all[c * N + j];
#pragma unroll
                    for (int i = 0; i < j; ++i) y = fmaf(u[c][i], D[kk_at(i, j)], y);
                    u[c][j] = bt * (u[c][j] - y);
                }
            }
        }
        // S <- G S + sum_i (G(i+1..N) k_i) u_i^T
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
            const ulonglong2 ev = e4[r * LPC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                s[c][2 * r] = mul2(s[c][2 * r], ev.x);
                s[c][2 * r + 1] = mul2(s[c][2 * r + 1], ev.y);
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            f2 uu[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) uu[c] = pack2(u[c][j], u[c][j]);
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
                const ulonglong2 wv = w4[j * (DKP / 4) + r * LPC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    s[c][2 * r] = fma2(wv.x, uu[c], s[c][2 * r]);
                    s[c][2 * r + 1] = fma2(wv.y, uu[c], s[c][2 * r + 1]);
                }
            }
        }
        // o_j = b_j + sum_{i<=j} u_i (k_i . G q_j), by the lane that holds b_j
        scatter_sums<NV, LPC, PW>(b, li);
        const int first = li * REM / SPREAD;
#pragma unroll
        for (int y = 0; y < REM; ++y) {
            const int m = first + y, c = m / N, j = m - c * N;
            float w = 0.0f;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc)
#pragma unroll
                for (int jj = 0; jj < N; ++jj) {
                    float z = 0.0f;
#pragma unroll
                    for (int i = 0; i <= jj; ++i) z = fmaf(u[cc][i], D[kq_at(i, jj)], z);
                    if (m == cc * N + jj) w = z;
                }
            if (li % SPREAD == 0 && col0 + c < dv) o[(size_t)(out_row + j) * H * dv + (size_t)head * dv + col0 + c] = b[y] + w;
        }
    };

    if (!SPLIT && L > 0) fetch(0, stage(0));
    for (int i = 0; i < n_stages; ++i) {
        const int t0 = i * ch, cnt = min(ch, L - t0), blocks = cnt / TB, rows = blocks + cnt % TB;
        float* st = stage(i);
        if constexpr (SPLIT) {
            meet(1 + i % C_::STAGES, 2 * THREADS);
        } else {
            if (i + 1 < n_stages) {                      // (its last readers passed the barrier below)
                fetch(t0 + ch, stage(i + 1));
                cp_async_wait<1>();
            } else cp_async_wait<0>();
            __syncthreads();
            prepare_stage(i);
            __syncthreads();
        }
        for (int y = 0; y < blocks; ++y) advance(block_of, st, y * TB, y, (long)start + t0 + y * TB);
        for (int y = blocks; y < rows; ++y) {
            const int t = blocks * TB + y - blocks;
            advance(token, st, t, y, (long)start + t0 + t);
        }
        if constexpr (SPLIT) {
            if (i + C_::STAGES < n_stages) come_by(1 + C_::STAGES + i % C_::STAGES, 2 * THREADS);
        } else __syncthreads();                          // the stage may be overwritten by the fetch after next
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < R / 4; ++r)
            if (col0 + c < dv) store_group<BY4>(S + (size_t)(col0 + c) * dk, channel_of<LPC>(r, li), dk, s[c][2 * r], s[c][2 * r + 1]);
}

template <int RULE, int R, int LPC, int NC, int THREADS, bool BY4, bool SPLIT>
int launch(const Rows& a, int n_seqs, int rows, cudaStream_t stream) {
    using C_ = Cut<R, LPC, NC, THREADS, SPLIT>;
    auto kernel = recurrent_kernel<RULE, R, LPC, NC, THREADS, BY4, SPLIT>;
    constexpr int whole = C_::floats(C_::CH) * (int)sizeof(float), alone = 120 * 1024, most = whole > alone ? whole : alone;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return fb_fail(-2, "recurrence: cannot reserve %d bytes of shared memory: %s", most, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    const dim3 grid(n_seqs * a.H, (a.dv + C_::COLS - 1) / C_::COLS);
    const bool round = (long)grid.x * grid.y <= fb_sm_count();
    // A few tokens a request: stages of one block, so that many CTAs share an SM.  A portion that gives no SM two CTAs asks for
    // more shared memory than two can have: launched while the kernel ahead still runs, they would else fill the SMs that are
    // free first with two each (measured: 830 us instead of 480 when this kernel took 480).
    const int ch = rows <= 4L * n_seqs ? TB : C_::CH;
    const size_t smem = round && rows > 4L * n_seqs ? most : C_::floats(ch) * sizeof(float);
    fb_launch(kernel, grid, dim3(C_::ALL), smem, stream, a, ch);
    return fb_check_launch("recurrence");
}

template <int RULE, int R, int LPC, int NC, bool BY4>
int launch_one(const Rows& a, int n_seqs, cudaStream_t stream) {
    constexpr int COLS = 128 / LPC * NC, spread = 100 * 1024;
    auto kernel = one_token_kernel<RULE, R, LPC, NC, BY4>;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, spread);
        if (e != cudaSuccess) return fb_fail(-2, "recurrence: cannot reserve %d bytes of shared memory: %s", spread, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    // Where two CTAs an SM hold them all, they ask for the shared memory that lets two in, so that they spread over the SMs
    // (one request, a decay per channel, 32 heads: a layer 62.4 us without, 58.0 with it, 59.2 with the kernels behind held back
    // as well; eight requests 68.4 and 77.5).
    const dim3 grid(n_seqs * a.H, (a.dv + COLS - 1) / COLS);
    fb_launch(kernel, grid, dim3(128), (long)grid.x * grid.y <= 2L * fb_sm_count() ? spread : 0, stream, a);
    return fb_check_launch("recurrence");
}

// What a launch gives a lane must not show in the result: for one key size, lane_sum and the exchange between lanes add in one
// order in every instance below.
template <int RULE>
int run(const float* qkv, const float* beta, const float* decay, float* state, long state_stride, const int* seq_q_start,
        const int* seq_q_len, const int* seq_slot, int n_seqs, int rows, int longest, float* o, int G, int H, int dk, int dv,
        cudaStream_t stream) {
    const long C = 2L * G * dk + (long)H * dv;
    const bool by4 = dk % 4 == 0 && C % 4 == 0 && state_stride % 4 == 0 && (uintptr_t)qkv % 16 == 0 &&
                     (uintptr_t)state % 16 == 0 && (RULE == DELTA_HEAD || (uintptr_t)decay % 16 == 0);
    const Rows a = {qkv, beta, decay, state, state_stride, seq_q_start, seq_q_len, seq_slot, o, G, H, dk, dv};
#define FB_ONE(R, LPC, NC) return by4 ? launch_one<RULE, R, LPC, NC, true>(a, n_seqs, stream) : launch_one<RULE, R, LPC, NC, false>(a, n_seqs, stream)
    if (rows <= n_seqs || longest < TB) {
        if (dk <= 16) FB_ONE(4, 4, 2);
        if (dk <= 32) FB_ONE(4, 8, 2);
        if (dk <= 64) FB_ONE(4, 16, 2);
        if (dk <= 128) FB_ONE(8, 16, 2);
        if (dk <= 256) FB_ONE(8, 32, 2);
        if (dk <= 512) FB_ONE(16, 32, 1);
        FB_ONE(32, 32, 1);
    }
#undef FB_ONE
#define FB_RECURRENCE_OF(R, LPC, NC, THREADS, BY4, SPLIT) return launch<RULE, R, LPC, NC, THREADS, BY4, SPLIT>(a, n_seqs, rows, stream)
#define FB_RECURRENCE(R, LPC, NC, BY4, SPLIT) FB_RECURRENCE_OF(R, LPC, NC, 128, BY4, SPLIT)
#define FB_RECURRENCE_BY(R, LPC, NC)                  \
    do {                                              \
        if (by4) FB_RECURRENCE(R, LPC, NC, true, false); \
        FB_RECURRENCE(R, LPC, NC, false, false);      \
    } while (0)
    if (dk <= 16) FB_RECURRENCE_BY(4, 4, 2);
    if (dk <= 32) FB_RECURRENCE_BY(4, 8, 2);
    if (dk <= 64) FB_RECURRENCE_BY(4, 16, 2);
    if (dk <= 128 && by4) {
        // With a decay per channel, 2,048 tokens of 32 heads of 128 x 128 take 376 us on 32 columns a CTA and 450 on 16 (391
        // without threads of their own for the stages); 16 heads, which 32 columns spread over 64 SMs only, 373 and 288.
        // Few tokens are over before 32 columns pay: a layer of 64 takes 75.6 us on 16, 79.5 on 32 (linear, 32 heads), 17 take 80 and 84.
        if (rows <= 128 || (long)n_seqs * H * ((dv + 15) / 16) <= fb_sm_count()) FB_RECURRENCE(8, 16, 2, true, true);
        FB_RECURRENCE(16, 8, 2, true, true);
    }
    if (dk <= 128) FB_RECURRENCE(16, 8, 2, false, false);
    if (dk <= 256) FB_RECURRENCE_BY(16, 16, 2);
    if (dk <= 512) {
        // (a stage fills more than half of an SM's shared memory: more CTAs than SMs are better off with twice the columns each;
        // 1,024 tokens of 32 heads of 512 x 64, a decay per channel: 507 us, 807 on 8 columns)
        if (by4 && (long)n_seqs * H * ((dv + 7) / 8) > fb_sm_count()) FB_RECURRENCE_OF(16, 32, 2, 256, true, false);
        FB_RECURRENCE_BY(16, 32, 2);
    }
    FB_RECURRENCE_BY(32, 32, 1);
#undef FB_RECURRENCE_BY
#undef FB_RECURRENCE
#undef FB_RECURRENCE_OF
}

}  // namespace

// rows: tokens of the step over all requests; longest: of the request that has most (rows where that is not known).
FB_API int fb_gdr_recurrent(const float* qkv, const float* beta, const float* decay, float* state, long long state_stride,
                            const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int n_seqs, int rows, int longest,
                            float* o, int G, int H, int dk, int dv, cudaStream_t stream) {
    FB_REQUIRE(n_seqs >= 0 && rows >= 0 && G > 0 && H > 0 && H % G == 0 && dk > 0 && dv > 0, "gated delta: bad sizes");
    FB_REQUIRE(dk <= 1024, "gated delta: key size %d is larger than 1024", dk);
    if (n_seqs == 0) return 0;
    return run<DELTA_HEAD>(qkv, beta, decay, state, (long)state_stride, seq_q_start, seq_q_len, seq_slot, n_seqs, rows, longest, o, G, H,
                           dk, dv, stream);
}

// decay: float32 [rows][H][dk], one factor per head and key channel; the rest as in fb_gdr_recurrent.
FB_API int fb_gdr_channel_recurrent(const float* qkv, const float* beta, const float* decay, float* state,
                                    long long state_stride, const int* seq_q_start, const int* seq_q_len, const int* seq_slot,
                                    int n_seqs, int rows, int longest, float* o, int G, int H, int dk, int dv, cudaStream_t stream) {
    FB_REQUIRE(n_seqs >= 0 && rows >= 0 && G > 0 && H > 0 && H % G == 0 && dk > 0 && dv > 0, "gated delta: bad sizes");
    FB_REQUIRE(dk <= 1024, "gated delta: key size %d is larger than 1024", dk);
    if (n_seqs == 0) return 0;
    return run<DELTA_CHANNEL>(qkv, beta, decay, state, (long)state_stride, seq_q_start, seq_q_len, seq_slot, n_seqs, rows, longest, o, G,
                              H, dk, dv, stream);
}

FB_API int fb_gla_recurrent(const float* qkv, const float* decay, float* state, long long state_stride, const int* seq_q_start,
                            const int* seq_q_len, const int* seq_slot, int n_seqs, int rows, int longest, float* o, int H, int dk,
                            int dv, cudaStream_t stream) {
    FB_REQUIRE(n_seqs >= 0 && rows >= 0 && H > 0 && dk > 0 && dv > 0, "linear attention: bad sizes");
    FB_REQUIRE(dk <= 1024, "linear attention: key size %d is larger than 1024", dk);
    if (n_seqs == 0) return 0;
    return run<LINEAR>(qkv, nullptr, decay, state, (long)state_stride, seq_q_start, seq_q_len, seq_slot, n_seqs, rows, longest, o, H, H,
                       dk, dv, stream);
}
