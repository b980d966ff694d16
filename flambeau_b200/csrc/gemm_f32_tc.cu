// out[M,N] = X[M,K] * W[N,K]^T in float32 on the 5th-generation tensor cores.
//
// The tensor pipes have no float32 x float32 mode, but three bfloat16 numbers hold a float32 exactly (8 + 8 + 8 bits of
// mantissa, each the rounding of what the ones before it left): x = xh + xm + xl, w = wh + wm + wl.  Six of the nine
// products are formed, xh wh, xh wm, xm wh, xh wl, xl wh and xm wm; each is exact in float32, and what is left out is
// below 2^-25 of |x w|, half of what a single float32 rounding may lose.
//
// Accumulation.  The tensor pipe's float32 sums are cut off, not rounded, so long chains of them drift towards zero.
// The large product xh wh is therefore summed in tensor memory over 64 of K only (four instructions) and then added to a
// float32 register by the ordinary adder; the five small products, 2^-8 and less of it, over a share of 512 of K.  The
// shares are added in ascending order, by the thread that computed them or, where CTAs split K, by the one that arrives
// last.  Which CTA computes a share, how many rows a call has and how wide a token tile is change no bit of a result:
// the arithmetic of an element depends on its row, its column and K alone.
//
// Range.  Both operands are multiplied by 2^24 on their way into parts, so that every part of every float32 (subnormal ones
// too) is a normal bfloat16, and the result by 2^-48 on its way out.  What overflows thereby (operands from 2^103, sums from
// 2^79) and infinities, which have no parts (inf - inf), end as a result that is not finite; such a result is computed
// again by one thread in float32 multiply-adds.
//
// Layout.  One CTA owns 128 output features x up to 128 tokens ("swap-AB" as in gemm_tc.cu).  The weights arrive as
// float32 by TMA, 32 of K a stage; four warps, a thread a feature, split a row's 32 numbers and put the parts into tensor
// memory, where the MMA takes its A operand from: the parts never pass through shared memory, whose bandwidth the MMA's
// token operand needs.  The tokens are split once for all feature tiles by a kernel of their own into bfloat16 parts
// that TMA fetches (64-byte swizzle).  Weights stay 4 bytes in memory: a decode step reads them once.
//
// Warps: 0 weight copies, 1 MMA, 2 token copies, 3 tensor memory, 4..11 split (two groups of four take the stages in turn:
// a group needs 1,100 cycles a stage, nearly all of it latency), 12..19 sums (two warps a lane quarter).  One barrier says
// that a stage's parts of both operands are there, one that its MMAs are done: the issuing thread spends 100 cycles on
// every wait and commit, beside 768 of MMAs.
// Tensor memory (512 columns): xh wh in two buffers, the small products in one, two buffers of weight parts.
//
// What bounds it: with a tile of 128 tokens a stage of 32 k takes about 1,000 cycles, 768 of them MMA, the rest the issuing
// threads' waits; with few tokens 800, of which HBM's share of 16 KB is 720.  Measured with cold L2 (us, multiply-adds on the
// CUDA cores as in gemm_simt.cu / here): 301 x 6,144 x 4,096 575 / 95, 301 x 4,096 x 4,096 464 / 85, 2,048 x 28,672 x 4,096
// 14,160 / 2,290, 64 x 28,672 x 4,096 606 / 146, 16 x 4,096 x 14,336 482 / 84, 8 x 4,096 x 4,096 56 / 33, 1 x 28,672 x 4,096
// 145 / 139, 1 x 256 x 2,048 30 / 20.  Error against 64 bits (root mean square over the results', K = 512 / 4,096): 2.9e-7 /
// 8.1e-7 there, 0.9e-7 / 1.1e-7 here.
//
// Every mbarrier wait is bounded as in gemm_tc.cu.
#include "tensor_map.cuh"
#include "umma.cuh"

namespace {

constexpr int FBM = 128;                 // output features per CTA
constexpr int FBN = 128;                 // most tokens per CTA
constexpr int FBK = 32;                  // K per stage: 128 bytes of float32
constexpr int SUM_STAGES = 2;            // stages (of 32) whose large products are summed in tensor memory
constexpr int SHARE_STAGES = 16;         // stages of a share of K
constexpr int MAX_WS = 12, MAX_XS = 8;   // most stages of weights / of token parts in flight (fewer as the token tile grows)
constexpr int W_BYTES = FBM * FBK * 4;
constexpr int F_SMEM = 227 * 1024;       // [weight stages | token stages | sums of shares, bn x 128 float32 | barriers]
constexpr int F_RING = F_SMEM - 1024 - 512;
constexpr int F_THREADS = 640;
constexpr int COL_SMALL = 2 * FBN;       // tensor-memory columns: [large 0 | large 1 | small | parts 0 | parts 1]
constexpr int COL_PARTS = 3 * FBN;
constexpr int PART_COLS = FBK / 2;       // columns of one part of a stage (two bfloat16 a column)
static_assert(COL_PARTS + 2 * 3 * PART_COLS <= 512, "tensor memory");

// K-major operand with the 64-byte swizzle: rows of 32 bf16, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_64(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

constexpr float SCALE_IN = 16777216.0f;                              // 2^24
constexpr float SCALE_OUT = 1.0f / (SCALE_IN * SCALE_IN);

// Two float32, scaled, into their three bfloat16 parts.
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    split_bf16x3(a * SCALE_IN, b * SCALE_IN, h, m, l);
}

// Xp[part][m][k] for k below Kp (a multiple of 32; zeros behind K).
template <bool VEC>
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ X, long lda, __nv_bfloat16* __restrict__ Xp, int M, int K, int Kp) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const long quads = (long)M * (Kp / 4);
    for (long q = (long)blockIdx.x * 256 + threadIdx.x; q < quads; q += (long)gridDim.x * 256) {
        const int m = (int)(q / (Kp / 4)), k = 4 * (int)(q - (long)m * (Kp / 4));
        const float* row = X + (size_t)m * lda;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (k < K) v = *reinterpret_cast<const float4*>(row + k);          // (K is a multiple of 4)
        } else {
            if (k < K) v.x = row[k];
            if (k + 1 < K) v.y = row[k + 1];
            if (k + 2 < K) v.z = row[k + 2];
            if (k + 3 < K) v.w = row[k + 3];
        }
        uint2 h, mm, l;
        split2(v.x, v.y, h.x, mm.x, l.x);
        split2(v.z, v.w, h.y, mm.y, l.y);
        __nv_bfloat16* dst = Xp + (size_t)m * Kp + k;
        const size_t part = (size_t)M * Kp;
        *reinterpret_cast<uint2*>(dst) = h;
        *reinterpret_cast<uint2*>(dst + part) = mm;
        *reinterpret_cast<uint2*>(dst + 2 * part) = l;
    }
}

struct F32Tc {
    const float* X; long lda;
    const float* W; long ldw;
    float* out; long ldo;
    float* partials; int* counters;
    int M, N, K, bn, tiles_m, tiles_n, splits, shares, stages, n_units, ws, xs;
    int* status;
};

struct FUnit { int m0, n0, tile, first, last; };        // shares [first, last) of output tile `tile`
__device__ __forceinline__ FUnit f_unit(int u, const F32Tc& a) {
    FUnit w;
    const int tiles = a.tiles_m * a.tiles_n, split = u / tiles;
    w.tile = u - split * tiles;
    w.m0 = w.tile % a.tiles_m * a.bn;
    w.n0 = w.tile / a.tiles_m * FBM;
    w.first = (int)((long)split * a.shares / a.splits);
    w.last = (int)((long)(split + 1) * a.shares / a.splits);
    return w;
}

// One result in float32 multiply-adds, even and odd k on their own.
__device__ __noinline__ float f32_dot(const float* __restrict__ x, const float* __restrict__ w, int K) {
    float even = 0.0f, odd = 0.0f;
    for (int k = 0; k + 1 < K; k += 2) {
        even = fmaf(x[k], w[k], even);
        odd = fmaf(x[k + 1], w[k + 1], odd);
    }
    if (K & 1) even = fmaf(x[K - 1], w[K - 1], even);
    return even + odd;
}
__device__ __forceinline__ bool f32_again(float v) { return !(fabsf(v) <= 3.4028234e38f); }      // (infinite or NaN)

// Rows m .. m + rows - 1 of column n of the output: those that need it once more.
__device__ __noinline__ void f32_again_columns(const F32Tc& a, int m, int rows, int n) {
    for (int r = m; r < m + rows; ++r) {
        float* at = a.out + (size_t)r * a.ldo + n;
        if (f32_again(*at)) *at = f32_dot(a.X + (size_t)r * a.lda, a.W + (size_t)n * a.ldw, a.K);
    }
}

__global__ void __launch_bounds__(F_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const __grid_constant__ F32Tc a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int WS = a.ws, XS = a.xs;
    const uint32_t part_bytes = (uint32_t)a.bn * FBK * 2, x_bytes = 3 * part_bytes;
    uint8_t* xs_base = smem + (size_t)WS * W_BYTES;
    float* totals = (float*)(xs_base + (size_t)XS * x_bytes);
    uint64_t* bars = (uint64_t*)(smem + F_RING);
    // full[s]: the stage's token parts (bytes) and weight parts (128 arrivals) are there; done[s]: its MMAs are
    uint64_t *w_full = bars, *w_empty = w_full + MAX_WS, *full = w_empty + MAX_WS, *done = full + MAX_XS, *l_full = done + MAX_XS,
             *l_empty = l_full + 2, *s_full = l_empty + 2, *s_empty = s_full + 1;
    uint32_t* tmem_slot = (uint32_t*)(s_empty + 1);
    int* last_flag = (int*)(tmem_slot + 1);
    int* bail = last_flag + 1;                   // a bounded wait ran out somewhere in this CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(smem_u32(bar), parity, a.status); };
    auto bailed = [&]() { return *(volatile int*)bail != 0; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_WS; ++s) { mbar_init(smem_u32(&w_full[s]), 1); mbar_init(smem_u32(&w_empty[s]), 128); }
        for (int s = 0; s < MAX_XS; ++s) { mbar_init(smem_u32(&full[s]), 129); mbar_init(smem_u32(&done[s]), 2); }
        for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&l_full[s]), 1); mbar_init(smem_u32(&l_empty[s]), 256); }
        mbar_init(smem_u32(s_full), 1);
        mbar_init(smem_u32(s_empty), 256);
        *bail = 0;
        mbar_fence_init();
    }
    if (warp == 2) tmem_alloc(tmem_slot, 512);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    fb_pdl_launch_dependents();                  // (behind the allocation: see umma.cuh)
    const uint32_t tmem = *tmem_slot;
    auto stages_of = [&](const FUnit& w) { return min(w.last * SHARE_STAGES, a.stages) - w.first * SHARE_STAGES; };

    if (warp == 0) {
        // ---------------- weights: no other kernel writes them, so they are requested at once ----------------
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 1;
            for (int u = blockIdx.x; u < a.n_units && !bailed(); u += gridDim.x) {
                const FUnit w = f_unit(u, a);
                const int n = stages_of(w);
                for (int i = 0; i < n; ++i) {
                    if (!wait(&w_empty[s], phase)) { *bail = 1; break; }
                    mbar_expect_tx(smem_u32(&w_full[s]), W_BYTES);
                    tma_load_2d(smem_u32(smem + (size_t)s * W_BYTES), &map_w, smem_u32(&w_full[s]),
                                (w.first * SHARE_STAGES + i) * FBK, w.n0);
                    if (++s == WS) { s = 0; phase ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---------------- token parts ----------------
        if (elect_one()) {
            fb_pdl_wait();
            int s = 0;
            uint32_t phase = 1;
            for (int u = blockIdx.x; u < a.n_units && !bailed(); u += gridDim.x) {
                const FUnit w = f_unit(u, a);
                const int n = stages_of(w);
                for (int i = 0; i < n; ++i) {
                    if (!wait(&done[s], phase)) { *bail = 1; break; }
                    mbar_expect_tx(smem_u32(&full[s]), x_bytes);
#pragma unroll
                    for (int p = 0; p < 3; ++p)          // (rows beyond M are the next part's, or zeros: nobody stores them)
                        tma_load_2d(smem_u32(xs_base) + (uint32_t)s * x_bytes + p * part_bytes, &map_x, smem_u32(&full[s]),
                                    (w.first * SHARE_STAGES + i) * FBK, p * a.M + w.m0);
                    if (++s == XS) { s = 0; phase ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1 || warp == 3) {
        // ---------------- MMA: one thread issues the large products, another the small ones (each its own accumulators) ----
        if (elect_one()) {
            const bool large = warp == 3;
            const uint32_t idesc = umma_idesc(a.bn), part = part_bytes >> 4;
            int xs = 0;
            uint32_t phase = 0, ab = 0, sums = 0;        // sums: large sums, or shares, begun by this CTA
            bool ok = true;
            for (int u = blockIdx.x; u < a.n_units && ok && !bailed(); u += gridDim.x) {
                const int n = stages_of(f_unit(u, a));
                for (int i = 0; i < n; ++i) {
                    const int run = large ? SUM_STAGES : SHARE_STAGES;       // stages of a sum (powers of two)
                    const bool first = (i & (run - 1)) == 0, last = (i & (run - 1)) == run - 1 || i == n - 1;
                    const uint32_t A = tmem + (uint32_t)COL_PARTS + ab * (3 * PART_COLS);
                    const uint64_t xh = umma_desc_64(smem_u32(xs_base) + (uint32_t)xs * x_bytes);
                    if (large) {
                        const uint32_t lb = sums & 1u, d = tmem + lb * FBN;
                        if (first) ok = wait(&l_empty[lb], ((sums >> 1) & 1u) ^ 1u);
                        if (ok) ok = wait(&full[xs], phase);
                        if (!ok) break;
                        tmem_fence_after();
                        umma_bf16_ts(d, A, xh, idesc, first ? 0u : 1u);
                        umma_bf16_ts(d, A + 8, xh + 2, idesc, 1u);
                        umma_commit(smem_u32(&done[xs]));
                        if (last) { umma_commit(smem_u32(&l_full[lb])); ++sums; }
                    } else {
                        const uint32_t d = tmem + (uint32_t)COL_SMALL;
                        const uint64_t xm = xh + part, xl = xm + part;
                        if (first) ok = wait(s_empty, (sums & 1u) ^ 1u);
                        if (ok) ok = wait(&full[xs], phase);
                        if (!ok) break;
                        tmem_fence_after();
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const uint32_t ah = A + (uint32_t)(k * 8), am = ah + PART_COLS, al = am + PART_COLS;
                            umma_bf16_ts(d, ah, xm + (uint64_t)(k * 2), idesc, (first && k == 0) ? 0u : 1u);
                            umma_bf16_ts(d, am, xh + (uint64_t)(k * 2), idesc, 1u);
                            umma_bf16_ts(d, ah, xl + (uint64_t)(k * 2), idesc, 1u);
                            umma_bf16_ts(d, al, xh + (uint64_t)(k * 2), idesc, 1u);
                            umma_bf16_ts(d, am, xm + (uint64_t)(k * 2), idesc, 1u);
                        }
                        umma_commit(smem_u32(&done[xs]));
                        if (last) { umma_commit(smem_u32(s_full)); ++sums; }
                    }
                    ab ^= 1u;
                    if (++xs == XS) { xs = 0; phase ^= 1u; }
                }
            }
            if (!ok) *bail = 1;
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 12) {
        // ---------------- split: a thread per feature, its 32 numbers of a stage into tensor memory ----------------
        const int quarter = warp & 3, row = quarter * 32 + lane, ab = (warp - 4) >> 2;
        const uint32_t dst = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(COL_PARTS + ab * 3 * PART_COLS);
        // (counters of this group's stages: `it` over all stages, its weight and token slots with their phases)
        uint32_t it = 0, w_phase = 0, x_phase = 0;       // x: the slot of stage it - 2, whose MMAs read this buffer before
        int ws = 0, xs = 0, x_old = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < a.n_units && ok && !bailed(); u += gridDim.x) {
            const int n = stages_of(f_unit(u, a));
            for (int i = 0; i < n; ++i, ++it) {
                if ((int)(it & 1u) == ab) {
                    ok = wait(&w_full[ws], w_phase);
                    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                    const uint8_t* src = smem + (size_t)ws * W_BYTES + row * 128;
                    float4 v[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
                    uint32_t h[16], m[16], l[16];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        split2(v[c].x, v[c].y, h[2 * c], m[2 * c], l[2 * c]);
                        split2(v[c].z, v[c].w, h[2 * c + 1], m[2 * c + 1], l[2 * c + 1]);
                    }
                    if (it >= 2) {                           // the MMAs that read this buffer, two stages ago, are done
                        ok = wait(&done[x_old], x_phase);
                        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                        tmem_fence_after();
                    }
                    tmem_st16(dst, h);
                    tmem_st16(dst + PART_COLS, m);
                    tmem_st16(dst + 2 * PART_COLS, l);
                    // (behind the stores, which need every number of the row: an arrival ahead of them let the assembler move the
                    // row's last loads behind it, where the slot's next copy overtook them)
                    mbar_arrive(smem_u32(&w_empty[ws]));
                    tmem_wait_st();
                    tmem_fence_before();
                    mbar_arrive(smem_u32(&full[xs]));
                }
                if (++ws == WS) { ws = 0; w_phase ^= 1u; }
                if (++xs == XS) xs = 0;
                if (it >= 2 && ++x_old == XS) { x_old = 0; x_phase ^= 1u; }
            }
        }
        if (!ok) *bail = 1;
    } else if (warp >= 12) {
        // ---------------- sums: lanes are features, the two warps of a quarter take 32 columns in turn ----------------
        fb_pdl_wait();
        const int quarter = warp & 3, half = (warp - 12) >> 2, row = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        uint32_t sums = 0, shares = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < a.n_units; u += gridDim.x) {
            const FUnit w = f_unit(u, a);
            const int n_stages = stages_of(w), n = w.n0 + row;
            for (int sh = w.first; sh < w.last && ok; ++sh) {
                float acc[64];
#pragma unroll
                for (int c = 0; c < 64; ++c) acc[c] = 0.0f;
                const int left = n_stages - (sh - w.first) * SHARE_STAGES;
                const int n_sums = (min(left, SHARE_STAGES) + SUM_STAGES - 1) / SUM_STAGES;
                for (int i = 0; i <= n_sums; ++i) {                  // the large sums of the share, then the small one
                    const bool small = i == n_sums;
                    const int lb = (int)(sums & 1u);
                    ok = !bailed() && (small ? wait(s_full, shares & 1u) : wait(&l_full[lb], (sums >> 1) & 1u));
                    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                    tmem_fence_after();
                    const uint32_t from = lanes + (uint32_t)(small ? COL_SMALL : lb * FBN);
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        const int c0 = half * 32 + cc * 64;
                        if (c0 < a.bn) {                             // (columns behind bn are read and dropped)
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                float r[16];
                                tmem_ld16(from + (uint32_t)(c0 + 16 * hh), r);
#pragma unroll
                                for (int c = 0; c < 16; ++c) acc[cc * 32 + hh * 16 + c] += r[c];
                            }
                        }
                    }
                    tmem_fence_before();
                    mbar_arrive(smem_u32(small ? s_empty : &l_empty[lb]));
                    if (small) ++shares; else ++sums;
                }
                if (!ok) break;
                if (a.splits > 1) {
                    float* mine = a.partials + ((size_t)w.tile * a.shares + sh) * (size_t)(a.bn * FBM) + row;
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            const int col = half * 32 + cc * 64 + c;
                            if (col < a.bn && w.m0 + col < a.M) mine[(size_t)col * FBM] = acc[cc * 32 + c];
                        }
                } else {
                    // shares are added up in shared memory (a thread's own numbers), the last one on its way out
                    const bool first = sh == w.first, last = sh == w.last - 1;
                    const int all = min(a.bn, a.M - w.m0);
                    float* mine = totals + row;
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) {
                        const int c0 = half * 32 + (cc >> 1) * 64 + (cc & 1) * 16;
                        if (c0 >= all) continue;
                        if (!first) {
#pragma unroll
                            for (int c = 0; c < 16; ++c) acc[cc * 16 + c] = mine[(c0 + c) * FBM] + acc[cc * 16 + c];
                        }
                        if (!last) {
#pragma unroll
                            for (int c = 0; c < 16; ++c) mine[(c0 + c) * FBM] = acc[cc * 16 + c];
                        } else if (n < a.N) {
                            float* p = a.out + (size_t)(w.m0 + c0) * a.ldo + n;
                            bool again = false;
#pragma unroll
                            for (int c = 0; c < 16; ++c, p += a.ldo) {
                                if (c0 + c < all) {
                                    const float v = acc[cc * 16 + c] * SCALE_OUT;
                                    *p = v;
                                    again |= f32_again(v);
                                }
                                if (c % 8 == 7) asm volatile("" : "+l"(p)::"memory");      // (addresses of eight at a time)
                            }
                            if (again) f32_again_columns(a, w.m0 + c0, min(16, all - c0), n);
                        }
                    }
                }
            }
            if (!ok) *bail = 1;
            if (a.splits > 1) {
                // one warp says for all eight whether the unit is whole and whether this CTA is the tile's last
                __threadfence();
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (warp == 12 && lane == 0) *last_flag = bailed() ? 2 : (atomicAdd(&a.counters[w.tile], 1) == a.splits - 1 ? 1 : 0);
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (*last_flag == 2) break;
                if (*last_flag == 1) {
                    __threadfence();
                    const float* base = a.partials + (size_t)w.tile * a.shares * (size_t)(a.bn * FBM);
                    const int rows = min(a.bn, a.M - w.m0);
                    for (int e = (warp - 12) * 32 + lane; e < rows * (FBM / 4); e += 256) {
                        const int col = e / (FBM / 4), f = 4 * (e - col * (FBM / 4));
                        const float4* p = reinterpret_cast<const float4*>(base + (size_t)col * FBM + f);
                        const size_t step = (size_t)(a.bn * FBM) / 4;
                        float4 v = __ldcg(p);
                        for (int s0 = 1; s0 < a.shares; s0 += 8) {
                            float4 t[8];
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                t[q] = s0 + q < a.shares ? __ldcg(p + (size_t)(s0 + q) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (s0 + q < a.shares) { v.x += t[q].x; v.y += t[q].y; v.z += t[q].z; v.w += t[q].w; }
                        }
                        float* at = a.out + (size_t)(w.m0 + col) * a.ldo + w.n0 + f;
                        const float r[4] = {v.x * SCALE_OUT, v.y * SCALE_OUT, v.z * SCALE_OUT, v.w * SCALE_OUT};
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (w.n0 + f + q < a.N)
                                at[q] = f32_again(r[q]) ? f32_dot(a.X + (size_t)(w.m0 + col) * a.lda,
                                                                  a.W + (size_t)(w.n0 + f + q) * a.ldw, a.K) : r[q];
                    }
                    if (warp == 12 && lane == 0) a.counters[w.tile] = 0;       // ready for the next launch
                }
            }
            if (a.splits == 1 && (!ok || bailed())) break;
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 2) {
        tmem_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

struct FPlan { int bn, splits; };
// Token tiles and shares of K: the cheapest of the choices in cycles of an SM.  A stage costs its twelve MMAs (N / 2 cycles
// each), its bytes from L2 or the splitting warps' work, whichever is most; all CTAs together no less than the weights from
// HBM.  Splitting K costs a copy of the output per share of 512, written and read, and the join of the CTA that is last.
FPlan plan_f32_tc(long M, long N, int shares, int stages, long partial_floats, int n_counters) {
    const long sms = fb_sm_count(), tiles_n = (N + FBM - 1) / FBM;
    FPlan best = {FBN, 1};
    double best_cost = 1e300;
    const long least = (M + FBN - 1) / FBN;
    for (long tiles_m = least; tiles_m <= least + 2 && tiles_m * 16 < M + 16 * least; ++tiles_m) {
        const int bn = (int)((((M + tiles_m - 1) / tiles_m) + 15) / 16 * 16);
        const double stage = fmax(fmax(9.0 * bn, 600.0), 720.0 / (double)tiles_m);
        const long tiles = tiles_n * ((M + bn - 1) / bn);
        for (int splits = 1; splits <= shares; ++splits) {
            if (splits > 1 && (tiles > n_counters || tiles * shares * bn * FBM > partial_floats)) break;
            const long rounds = (tiles * splits + sms - 1) / sms;
            const double per_unit = fmin((double)((shares + splits - 1) / splits) * SHARE_STAGES, (double)stages);
            double cost = fmax((double)rounds * (per_unit * stage + 1500.0), (double)tiles * stages * 16384.0 / (23.0 * sms));
            if (splits > 1) cost += 2500.0 + (double)shares * (M < bn ? M : bn) * FBM * 4.0 * 2.0 / 24.0;
            if (cost < best_cost - 1e-6) { best_cost = cost; best = FPlan{bn, splits}; }
        }
    }
    return best;
}

constexpr long SPLIT_FLOATS = 16L << 20;         // most that the shares of one product may take

int stages_of_k(int K) { return (K + FBK - 1) / FBK; }
int shares_of_k(int K) { return (stages_of_k(K) + SHARE_STAGES - 1) / SHARE_STAGES; }

}  // namespace

// Floats of `partials` that fb_gemm_f32_tc wants for the same sizes with `n_counters` counters: 0 where K is not split.
FB_API long long fb_gemm_f32_tc_scratch_floats(int M, int N, int K, int n_counters) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int shares = shares_of_k(K);
    const FPlan p = plan_f32_tc(M, N, shares, stages_of_k(K), SPLIT_FLOATS, n_counters);
    if (p.splits == 1) return 0;
    return (long long)((M + p.bn - 1) / p.bn) * ((N + FBM - 1) / FBM) * shares * p.bn * FBM;
}

// X [M,K] and out [M,N] float32 with any strides of at least a row; W [N,K] float32 whose rows start on 16-byte borders, K a
// multiple of 4.  `parts` takes 3 M Kp bfloat16 (Kp: K rounded up to a multiple of 32), 16-byte aligned; `partials` and
// `counters` (zero before the call and after it) are the scratch of split K, as in fb_gemm_tc, of calls that run one after the
// other; without them, or with fewer floats than fb_gemm_f32_tc_scratch_floats asks for, K is split less or not at all.
FB_API int fb_gemm_f32_tc(const void* X, long long lda, const void* W, long long ldw, void* out, long long ldo, int M, int N,
                          int K, void* parts, long long parts_elems, float* partials, long long partial_floats, int* counters,
                          int n_counters, int* status, cudaStream_t stream) {
    FB_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    FB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_f32_tc: a row stride is shorter than its row");
    FB_REQUIRE(K % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)W & 15) == 0, "gemm_f32_tc: weight rows must start on 16-byte borders");
    FB_REQUIRE(((uintptr_t)X & 3) == 0 && ((uintptr_t)out & 3) == 0 && status, "gemm_f32_tc: unaligned operands, or no status word");
    if (M == 0) return 0;
    const int Kp = (K + FBK - 1) / FBK * FBK;
    FB_REQUIRE(parts && ((uintptr_t)parts & 15) == 0 && parts_elems >= 3LL * M * Kp, "gemm_f32_tc: scratch for the rows' parts missing");
    FB_REQUIRE(3LL * M < 2147483647LL, "gemm_f32_tc: too many rows (M=%d)", M);
    const int stages = stages_of_k(K), shares = shares_of_k(K);
    const FPlan plan = plan_f32_tc(M, N, shares, stages, partials && counters ? partial_floats : 0, counters ? n_counters : 0);
    F32Tc a = {};
    a.X = (const float*)X; a.lda = (long)lda; a.W = (const float*)W; a.ldw = (long)ldw; a.out = (float*)out; a.ldo = (long)ldo;
    a.partials = partials; a.counters = counters; a.M = M; a.N = N; a.K = K; a.bn = plan.bn;
    a.tiles_m = (M + plan.bn - 1) / plan.bn; a.tiles_n = (N + FBM - 1) / FBM;
    a.splits = plan.splits; a.shares = shares; a.stages = stages; a.status = status;
    // shared memory: the sums of shares where one CTA adds several, token stages for 2 us of MMAs, the rest for weights
    const int x_bytes = 3 * plan.bn * FBK * 2, room = F_RING - (a.splits == 1 && shares > 1 ? plan.bn * FBM * 4 : 0);
    a.xs = (room - 5 * W_BYTES) / x_bytes < MAX_XS ? (room - 5 * W_BYTES) / x_bytes : MAX_XS;
    a.ws = (room - a.xs * x_bytes) / W_BYTES < MAX_WS ? (room - a.xs * x_bytes) / W_BYTES : MAX_WS;
    const long n_units = (long)a.tiles_m * a.tiles_n * a.splits;
    FB_REQUIRE(n_units <= 2000000000L, "gemm_f32_tc: too many tiles (M=%d N=%d)", M, N);
    a.n_units = (int)n_units;
    CUtensorMap mw, mx;
    int rc = fb_tensor_map_rows(&mw, W, 4, N, K, (long)ldw, FBK, FBM);
    if (rc) return rc;
    rc = fb_tensor_map_rows(&mx, parts, 2, 3L * M, Kp, Kp, FBK, plan.bn);
    if (rc) return rc;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM);
        if (e != cudaSuccess) return fb_fail(-2, "gemm_f32_tc: cannot reserve %d bytes of shared memory: %s", F_SMEM, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    const long quads = (long)M * (Kp / 4), blocks = (quads + 255) / 256;
    const int split_grid = (int)(blocks < 8L * fb_sm_count() ? blocks : 8L * fb_sm_count());
    if (lda % 4 == 0 && ((uintptr_t)X & 15) == 0)
        fb_launch(split_rows_kernel<true>, split_grid, 256, 0, stream, a.X, a.lda, (__nv_bfloat16*)parts, M, K, Kp);
    else
        fb_launch(split_rows_kernel<false>, split_grid, 256, 0, stream, a.X, a.lda, (__nv_bfloat16*)parts, M, K, Kp);
    const int grid = (int)(n_units < fb_sm_count() ? n_units : fb_sm_count());
    fb_launch_class(M > 128 ? FB_LAUNCH_GEMM_WIDE : FB_LAUNCH_OTHER, gemm_f32_tc_kernel, grid, F_THREADS, F_SMEM, stream, mw, mx, a);
    return fb_check_launch("gemm_f32_tc");
}
