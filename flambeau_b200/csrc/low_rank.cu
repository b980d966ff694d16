// Maps through a narrow middle: y = f(W2 (W1 h)), W1 h being columns of a mixer's stacked projection (float32, possibly
// as split-K shares) and W2 [N, R] with R a few dozen.  One launch serves up to two such maps of the same rows, each
// with a function of its own behind it (the product never leaves the kernel unfinished):
//   FB_LR_PLAIN     y = z                                       z = W2 (W1 h) + bias   (bias [N], optional)
//   FB_LR_SIGMOID   y = 1 / (1 + exp(-z))
//   FB_LR_DECAY     y = exp(-exp(log_rate[c / group]) * log(1 + exp(z)))        (a decay per output, a rate per `group`
//                                                                                neighbouring outputs)
// y is float32 [rows, N].  What stands behind the product is float32 in both forms:
//   low_rank_tiles, low_rank_mma   bfloat16 W2: tensor cores (mma.sync m16n8k16, float32 accumulation), a CTA of four warps
//                  takes 64 rows x 64 outputs (or several such tiles one after the other); the middle is rounded once to
//                  bfloat16
//   low_rank_fma   any types: float32 multiply-adds, 32 rows x 64 outputs a CTA
#include <algorithm>
#include <climits>
#include <type_traits>

#include "attention_common.cuh"
#include "rows.cuh"

namespace {

enum FbLowRank : int { FB_LR_PLAIN = 0, FB_LR_SIGMOID = 1, FB_LR_DECAY = 2 };

struct LowRankMap {
    const void* w;             // [N, R]
    int mid_off, R, N;         // the middle's columns in the projection rows, and the sizes
    int act;                   // an FbLowRank code
    const void* bias;          // [N] or nullptr
    const void* log_rate;      // [ceil(N / group)] for FB_LR_DECAY
    int group;
    float* out;                // [rows, N]
};
struct LowRankArgs {
    const float* proj; long proj_stride; int n_partials; long partial_stride;
    int n;
    LowRankMap map[2];
    int tiles_first;           // blockIdx.y below this: map[0]
};

template <typename TW>
__device__ __forceinline__ float lr_finish(const LowRankMap& m, float z, int c) {
    if (m.bias) z += fb_to_float(static_cast<const TW*>(m.bias)[c]);
    if (m.act == FB_LR_SIGMOID) return 1.0f / (1.0f + expf(-z));
    if (m.act == FB_LR_DECAY) {
        const float softplus = z > 20.0f ? z : log1pf(expf(z));
        return expf(-expf(fb_to_float(static_cast<const TW*>(m.log_rate)[c / m.group])) * softplus);
    }
    return z;
}

constexpr int LM_T = 64, LM_KC = 64, LM_LD = LM_KC + 8;

__global__ void __launch_bounds__(128)
low_rank_mma_kernel(const LowRankArgs a) {
    using bf16 = __nv_bfloat16;
    fb_pdl_launch_dependents();
    __shared__ __align__(16) bf16 As[LM_T][LM_LD];
    __shared__ __align__(16) bf16 Ws[LM_T][LM_LD];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const bool second = (int)blockIdx.y >= a.tiles_first;
    const LowRankMap m = second ? a.map[1] : a.map[0];
    const int m0 = blockIdx.x * LM_T, n0 = ((int)blockIdx.y - (second ? a.tiles_first : 0)) * LM_T;
    const bf16* w = static_cast<const bf16*>(m.w);
    const bool w_vec = m.R % 8 == 0 && (uintptr_t)w % 16 == 0;
    const bool a_vec = m.R % 4 == 0 && m.mid_off % 4 == 0 && a.proj_stride % 4 == 0 && a.partial_stride % 4 == 0 &&
                       (uintptr_t)a.proj % 16 == 0;
    float acc[LM_T / 8][4];
#pragma unroll
    for (int j = 0; j < LM_T / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    bool waited = false;
    for (int k0 = 0; k0 < m.R; k0 += LM_KC) {
        // the weights first: they are not of this step and need not wait for the kernel before
        if (w_vec) {
#pragma unroll
            for (int u = 0; u < LM_T * (LM_KC / 8) / 128; ++u) {
                const int idx = tid + 128 * u, nn = idx / (LM_KC / 8), k = (idx - nn * (LM_KC / 8)) * 8;
                uint4 raw = make_uint4(0u, 0u, 0u, 0u);
                if (n0 + nn < m.N && k0 + k < m.R) raw = *reinterpret_cast<const uint4*>(w + (size_t)(n0 + nn) * m.R + k0 + k);
                *reinterpret_cast<uint4*>(&Ws[nn][k]) = raw;
            }
        } else {
            for (int idx = tid; idx < LM_T * LM_KC; idx += 128) {
                const int nn = idx / LM_KC, k = idx - nn * LM_KC;
                Ws[nn][k] = (n0 + nn < m.N && k0 + k < m.R) ? w[(size_t)(n0 + nn) * m.R + k0 + k] : __float2bfloat16(0.0f);
            }
        }
        if (!waited) { fb_pdl_wait(); waited = true; }
        if (a_vec) {
#pragma unroll
            for (int u = 0; u < LM_T * (LM_KC / 4) / 128; ++u) {
                const int idx = tid + 128 * u, r = idx / (LM_KC / 4), k = (idx - r * (LM_KC / 4)) * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (m0 + r < a.n && k0 + k < m.R)
                    v = slab_sum4(a.proj + (size_t)(m0 + r) * a.proj_stride + m.mid_off + k0 + k, a.n_partials, a.partial_stride);
                uint2 raw;
                raw.x = fb_attn::pack_bf16(v.x, v.y);
                raw.y = fb_attn::pack_bf16(v.z, v.w);
                *reinterpret_cast<uint2*>(&As[r][k]) = raw;
            }
        } else {
            for (int idx = tid; idx < LM_T * LM_KC; idx += 128) {
                const int r = idx / LM_KC, k = idx - r * LM_KC;
                float v = 0.0f;
                if (m0 + r < a.n && k0 + k < m.R)
                    v = fb_slab_sum(a.proj + (size_t)(m0 + r) * a.proj_stride, m.mid_off + k0 + k, a.n_partials, a.partial_stride);
                As[r][k] = __float2bfloat16(v);
            }
        }
        __syncthreads();
        if (m0 + warp * 16 < a.n) {
#pragma unroll
            for (int kk = 0; kk < LM_KC; kk += 16) {
                uint32_t af[4];
                af[0] = *reinterpret_cast<const uint32_t*>(&As[warp * 16 + g][kk + 2 * t]);
                af[1] = *reinterpret_cast<const uint32_t*>(&As[warp * 16 + g + 8][kk + 2 * t]);
                af[2] = *reinterpret_cast<const uint32_t*>(&As[warp * 16 + g][kk + 8 + 2 * t]);
                af[3] = *reinterpret_cast<const uint32_t*>(&As[warp * 16 + g + 8][kk + 8 + 2 * t]);
#pragma unroll
                for (int j = 0; j < LM_T / 8; ++j) {
                    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(&Ws[j * 8 + g][kk + 2 * t]);
                    const uint32_t b1 = *reinterpret_cast<const uint32_t*>(&Ws[j * 8 + g][kk + 8 + 2 * t]);
                    fb_attn::mma_bf16(acc[j], af, b0, b1);
                }
            }
        }
        __syncthreads();
    }
    const bool pairs = m.N % 2 == 0 && (uintptr_t)m.out % 8 == 0;
#pragma unroll
    for (int j = 0; j < LM_T / 8; ++j)
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) {
            const int r = m0 + warp * 16 + g + hi * 8, c = n0 + j * 8 + 2 * t;
            if (r >= a.n || c >= m.N) continue;
            float* dst = m.out + (size_t)r * m.N + c;
            const float y0 = lr_finish<bf16>(m, acc[j][2 * hi], c);
            if (c + 1 >= m.N) { dst[0] = y0; continue; }
            const float y1 = lr_finish<bf16>(m, acc[j][2 * hi + 1], c + 1);
            if (pairs) *reinterpret_cast<float2*>(dst) = make_float2(y0, y1);
            else { dst[0] = y0; dst[1] = y1; }
        }
}

// The same for middles of up to LT_MAX_R columns whose weights can be fetched 16 bytes at a time: the rows' middles stay in
// shared memory for all NT output tiles of the CTA, whose weights arrive by asynchronous copies one tile ahead.
constexpr int LT_MAX_R = 256;
__host__ __device__ constexpr int lt_pitch(int R) { return (R + 15) / 16 * 16 + 8; }
inline size_t lt_smem(int R) { return (size_t)3 * LM_T * lt_pitch(R) * 2 + 4 * LM_T * sizeof(float); }

__device__ __forceinline__ float lr_finish_fast(int act, float z, float bias, float rate) {
    z += bias;
    if (act == FB_LR_SIGMOID) return __fdividef(1.0f, 1.0f + __expf(-z));
    if (act == FB_LR_DECAY) {
        // log(1 + exp(z)) = max(z, 0) + log(1 + e), e = exp(-|z|); for small e the series, where 1 + e would lose e's digits
        const float e = __expf(-fabsf(z));
        const float l = e < 0.02f ? e * fmaf(e, fmaf(e, fmaf(e, -0.25f, 1.0f / 3.0f), -0.5f), 1.0f) : __logf(1.0f + e);
        return expf(-rate * (fmaxf(z, 0.0f) + l));
    }
    return z;
}

// What bounds it: the functions behind the products, some 25 instructions an output, beside stores of 4 bytes an output; for few
// rows the way of the middles into shared memory.  To 2 x 4,096 outputs (a decay and a sigmoid) through 128 columns of one share /
// of three: 2,048 rows 50 / 51 us, 343 rows 14 / 16, 65 rows 7.6 / 9.2; with the middles fetched one by one across branches,
// fragments by 4-byte loads and CTAs of four tiles 55 / 67, 26 / 31 and 24 / 28.  Through 16 columns 2,048 rows 27 (30 so), but
// 4,096 rows 54 (51): those CTAs had fewer registers, and six of them an SM hide the functions better than four.
__global__ void __launch_bounds__(128, 4)
low_rank_tiles_kernel(const LowRankArgs a, int NT) {
    using bf16 = __nv_bfloat16;
    fb_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char lt_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const bool second = (int)blockIdx.y >= a.tiles_first;
    const LowRankMap m = second ? a.map[1] : a.map[0];
    const int m0 = blockIdx.x * LM_T, tile0 = ((int)blockIdx.y - (second ? a.tiles_first : 0)) * NT;
    const int tiles = min(NT, (m.N + LM_T - 1) / LM_T - tile0);
    const int P = lt_pitch(m.R), K = P - 8;
    bf16* As = reinterpret_cast<bf16*>(lt_raw);                       // [64][P]
    bf16* Ws = As + LM_T * P;                                         // [2][64][P]
    float* col = reinterpret_cast<float*>(Ws + 2 * LM_T * P);         // [2][bias: 64 | rate: 64]
    const bf16* w = static_cast<const bf16*>(m.w);
    // (thread tid fetches the chunks tid, tid + 128, ... of 8 numbers: their places by addition)
    const int chunks = K / 8, r_first = tid / chunks, k_first = tid - r_first * chunks, r_step = 128 / chunks, k_step = 128 - r_step * chunks;
    auto fetch = [&](int tile) {
        bf16* dst = Ws + (tile & 1) * LM_T * P;
        const int n0 = (tile0 + tile) * LM_T;
        for (int r = r_first, k = k_first; r < LM_T;) {
            if (n0 + r < m.N && 8 * k < m.R)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * P + 8 * k)),
                             "l"(w + (size_t)(n0 + r) * m.R + 8 * k) : "memory");
            else
                *reinterpret_cast<uint4*>(dst + r * P + 8 * k) = make_uint4(0u, 0u, 0u, 0u);
            r += r_step;
            k += k_step;
            if (k >= chunks) {
                k -= chunks;
                ++r;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (tid < LM_T && n0 + tid < m.N) {
            float* c = col + (tile & 1) * 2 * LM_T + tid;
            c[0] = m.bias ? fb_to_float(static_cast<const bf16*>(m.bias)[n0 + tid]) : 0.0f;
            c[LM_T] = m.act == FB_LR_DECAY ? expf(fb_to_float(static_cast<const bf16*>(m.log_rate)[(n0 + tid) / m.group])) : 0.0f;
        }
    };
    fetch(0);                                          // (not of this step: it need not wait for the kernel before)
    fb_pdl_wait();
    const bool a_vec = m.mid_off % 4 == 0 && a.proj_stride % 4 == 0 && a.partial_stride % 4 == 0 && (uintptr_t)a.proj % 16 == 0;
    // The middles of a warp's 16 rows, four columns an item; an item's loads are unconditional, so that those of U items are on
    // their way at once.
    const int quads = K / 4, rows = min(16, a.n - m0 - warp * 16);                  // (rows behind the last are nobody's)
    const int r_more = 32 / quads, q_more = 32 - r_more * quads;                      // from an item to the lane's next
    const float* mids = a.proj + (size_t)(m0 + warp * 16) * a.proj_stride + m.mid_off;
    auto stage = [&](auto at_once) {
        constexpr int U = decltype(at_once)::value;
        for (int i = lane, r = lane / quads, q = lane - r * quads; i < rows * quads; i += 32 * U) {
            float4 v[U];
            const float* src[U];
            int to[U];
            bool there[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                there[u] = 4 * q < m.R;
                src[u] = mids + (size_t)min(r, rows - 1) * a.proj_stride + (there[u] ? 4 * q : 0);
                to[u] = r < rows ? (warp * 16 + r) * P + 4 * q : -1;
                r += r_more;
                q += q_more;
                if (q >= quads) { q -= quads; ++r; }
            }
            if (a_vec && a.n_partials == 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = Vec4<float>::load(src[u]);
            } else if (a_vec && a.n_partials <= 3 && U > 1) {     // (no loop between the loads of two items)
                const bool third = a.n_partials == 3;
                const long second_at = a.partial_stride, third_at = third ? 2 * a.partial_stride : 0;
#pragma unroll
                for (int u0 = 0; u0 + 4 <= U; u0 += 4) {
                    float4 x[4], y[4], z[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        x[u] = Vec4<float>::load(src[u0 + u]);
                        y[u] = Vec4<float>::load(src[u0 + u] + second_at);
                        z[u] = Vec4<float>::load(src[u0 + u] + third_at);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float4 s = make_float4(x[u].x + y[u].x, x[u].y + y[u].y, x[u].z + y[u].z, x[u].w + y[u].w);
                        v[u0 + u] = third ? make_float4(s.x + z[u].x, s.y + z[u].y, s.z + z[u].z, s.w + z[u].w) : s;
                    }
                }
            } else if (a_vec) {
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = slab_sum4(src[u], a.n_partials, a.partial_stride);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    v[u] = make_float4(fb_slab_sum(src[u], 0, a.n_partials, a.partial_stride), fb_slab_sum(src[u], 1, a.n_partials, a.partial_stride),
                                       fb_slab_sum(src[u], 2, a.n_partials, a.partial_stride), fb_slab_sum(src[u], 3, a.n_partials, a.partial_stride));
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (to[u] >= 0)
                    *reinterpret_cast<uint2*>(As + to[u]) = there[u] ? make_uint2(fb_attn::pack_bf16(v[u].x, v[u].y), fb_attn::pack_bf16(v[u].z, v[u].w))
                                                                     : make_uint2(0u, 0u);
        }
    };
    if (rows * quads <= 64) stage(std::integral_constant<int, 1>());
    else stage(std::integral_constant<int, 8>());
    const bool pairs = m.N % 2 == 0 && (uintptr_t)m.out % 8 == 0;
    // (ldmatrix: lane l gives the address of row l % 8 of the 8 x 8 block l / 8)
    const bf16* a_at = As + (warp * 16 + (lane & 15)) * P + (lane >> 4) * 8;
    const bf16* w_at = Ws + ((lane >> 4) * 8 + (lane & 7)) * P + ((lane >> 3) & 1) * 8;
    for (int tile = 0; tile < tiles; ++tile) {
        if (tile + 1 < tiles) {
            fetch(tile + 1);                           // (its buffer's last readers passed the barrier at the loop's end)
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int n0 = (tile0 + tile) * LM_T;
        if (m0 + warp * 16 < a.n) {                    // (warp-uniform)
            float acc[LM_T / 8][4];
#pragma unroll
            for (int j = 0; j < LM_T / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
            const bf16* w_tile = w_at + (tile & 1) * LM_T * P;
            for (int kk = 0; kk < K; kk += 16) {
                uint32_t af[4];
                fb_attn::ldmatrix_x4(af, a_at + kk);
#pragma unroll
                for (int j = 0; j < LM_T / 8; j += 2) {
                    uint32_t bf[4];                    // outputs 8 j .. and 8 (j + 1) .., channels kk .. and kk + 8 .. of each
                    fb_attn::ldmatrix_x4(bf, w_tile + j * 8 * P + kk);
                    fb_attn::mma_bf16(acc[j], af, bf[0], bf[1]);
                    fb_attn::mma_bf16(acc[j + 1], af, bf[2], bf[3]);
                }
            }
            const float* c0 = col + (tile & 1) * 2 * LM_T;
            auto finish = [&](auto act_of) {           // (the function is the map's: chosen once, not per output)
                constexpr int ACT = decltype(act_of)::value;
#pragma unroll
                for (int j = 0; j < LM_T / 8; ++j) {
                    const int cc = j * 8 + 2 * t, c = n0 + cc;
                    const float2 b = *reinterpret_cast<const float2*>(c0 + cc), rate = *reinterpret_cast<const float2*>(c0 + LM_T + cc);
#pragma unroll
                    for (int hi = 0; hi < 2; ++hi) {
                        const int r = m0 + warp * 16 + g + hi * 8;
                        if (r >= a.n || c >= m.N) continue;
                        float* dst = m.out + (size_t)r * m.N + c;
                        const float y0 = lr_finish_fast(ACT, acc[j][2 * hi], b.x, rate.x), y1 = lr_finish_fast(ACT, acc[j][2 * hi + 1], b.y, rate.y);
                        if (pairs) { *reinterpret_cast<float2*>(dst) = make_float2(y0, y1); continue; }
                        dst[0] = y0;
                        if (c + 1 < m.N) dst[1] = y1;
                    }
                }
            };
            if (m.act == FB_LR_DECAY) finish(std::integral_constant<int, FB_LR_DECAY>());
            else if (m.act == FB_LR_SIGMOID) finish(std::integral_constant<int, FB_LR_SIGMOID>());
            else finish(std::integral_constant<int, FB_LR_PLAIN>());
        }
        __syncthreads();
    }
}

constexpr int LF_TM = 32, LF_TN = 64, LF_KC = 16;

template <typename TW>
__global__ void __launch_bounds__(256)
low_rank_fma_kernel(const LowRankArgs a) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    __shared__ float As[LF_KC][LF_TM + 1];
    __shared__ float Ws[LF_KC][LF_TN + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const bool second = (int)blockIdx.y >= a.tiles_first;
    const LowRankMap m = second ? a.map[1] : a.map[0];
    const int m0 = blockIdx.x * LF_TM, n0 = ((int)blockIdx.y - (second ? a.tiles_first : 0)) * LF_TN;
    const TW* w = static_cast<const TW*>(m.w);
    float acc[2][4] = {};
    for (int k0 = 0; k0 < m.R; k0 += LF_KC) {
        for (int idx = tid; idx < LF_TM * LF_KC; idx += 256) {
            const int r = idx / LF_KC, k = idx - r * LF_KC;
            As[k][r] = (m0 + r < a.n && k0 + k < m.R)
                ? fb_slab_sum(a.proj + (size_t)(m0 + r) * a.proj_stride, m.mid_off + k0 + k, a.n_partials, a.partial_stride) : 0.0f;
        }
        for (int idx = tid; idx < LF_TN * LF_KC; idx += 256) {
            const int nn = idx / LF_KC, k = idx - nn * LF_KC;
            Ws[k][nn] = (n0 + nn < m.N && k0 + k < m.R) ? fb_to_float(w[(size_t)(n0 + nn) * m.R + k0 + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < LF_KC; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[0][i] = fmaf(As[k][ty], Ws[k][tx + 16 * i], acc[0][i]);
                acc[1][i] = fmaf(As[k][ty + 16], Ws[k][tx + 16 * i], acc[1][i]);
            }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = m0 + ty + 16 * j, c = n0 + tx + 16 * i;
            if (r < a.n && c < m.N) m.out[(size_t)r * m.N + c] = lr_finish<TW>(m, acc[j][i], c);
        }
}

}  // namespace

// Up to two maps of the same projection rows (count 1 or 2); the arrays hold one entry a map.  The weights, biases and
// rates of all maps share a dtype.
FB_API int fb_low_rank_maps(const float* proj, long long proj_stride, int n_partials, long long partial_stride, int n,
                            int count, const void* const* w, int w_dtype, const int* mid_off, const int* R, const int* N,
                            const int* act, const void* const* bias, const void* const* log_rate, const int* group,
                            float* const* out, cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && (count == 1 || count == 2), "low_rank_maps: one or two maps wanted");
    LowRankArgs a = {};
    a.proj = proj; a.proj_stride = (long)proj_stride; a.n = n;
    a.n_partials = n_partials < 1 ? 1 : n_partials; a.partial_stride = (long)partial_stride;
    int tiles = 0;
    for (int i = 0; i < count; ++i) {
        FB_REQUIRE(w[i] && out[i] && R[i] > 0 && N[i] > 0 && mid_off[i] >= 0 && proj_stride >= (long long)mid_off[i] + R[i],
                   "low_rank_maps: bad sizes");
        FB_REQUIRE(act[i] >= FB_LR_PLAIN && act[i] <= FB_LR_DECAY, "low_rank_maps: unknown function %d", act[i]);
        FB_REQUIRE(act[i] != FB_LR_DECAY || (log_rate[i] && group[i] > 0), "low_rank_maps: a decay wants its rates");
        a.map[i] = {w[i], mid_off[i], R[i], N[i], act[i], bias[i], log_rate[i], group[i] > 0 ? group[i] : 1, out[i]};
        if (i == 0) a.tiles_first = (N[i] + LM_T - 1) / LM_T;
        tiles += (N[i] + LM_T - 1) / LM_T;
    }
    static_assert(LM_T == LF_TN, "both kernels tile the outputs alike");
    FB_REQUIRE(tiles <= 65535, "low_rank_maps: too many outputs");
    if (n == 0) return 0;
    if (w_dtype == FB_BF16) {
        bool resident = true;
        int widest = 0;
        for (int i = 0; i < count; ++i) {
            resident = resident && R[i] % 8 == 0 && R[i] <= LT_MAX_R && (uintptr_t)w[i] % 16 == 0;
            widest = R[i] > widest ? R[i] : widest;
        }
        if (resident) {
            // Tiles a CTA, by the time of the fullest SM: its CTAs one after the other, a CTA's tiles and the fetch of its rows
            // (a tile's time for 48 columns); fewer than four CTAs on an SM do not keep it busy.  Measured over 1 to 16 tiles, 65
            // to 4,096 rows and middles of 16 to 256, three shares (us, one tile / the rule's / sixteen): 2,048 rows to 2 x 4,096
            // through 16 columns 43 / 30 (four) / 62, through 128 101 / 58 (eight) / 95, through 256 310 / 119 (sixteen); 343
            // rows through 128 28 / 21 (two) / 71; 65 rows 14 (one) / 71.
            const size_t smem = lt_smem(widest);
            const long blocks = (n + LM_T - 1) / LM_T, busy = std::min<long>(4, 220 * 1024 / (long)(smem + 1024));
            auto groups = [&](int i, int nt) { return ((N[i] + LM_T - 1) / LM_T + nt - 1) / nt; };
            int NT = 1;
            long best = LONG_MAX;
            for (int nt = 1; nt <= 16; ++nt) {
                const long ctas = blocks * (groups(0, nt) + (count > 1 ? groups(1, nt) : 0));
                const long cost = (48L * nt + widest) * std::max((ctas + fb_sm_count() - 1) / fb_sm_count(), busy);
                if (cost < best) { best = cost; NT = nt; }
            }
            a.tiles_first = groups(0, NT);
            const dim3 grid((unsigned)blocks, groups(0, NT) + (count > 1 ? groups(1, NT) : 0));
            if (smem > 48 * 1024) cudaFuncSetAttribute(low_rank_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            fb_launch(low_rank_tiles_kernel, grid, dim3(128), smem, stream, a, NT);
            return fb_check_launch("low_rank_maps");
        }
        fb_launch(low_rank_mma_kernel, dim3((n + LM_T - 1) / LM_T, tiles), dim3(128), 0, stream, a);
    } else {
        FB_REQUIRE(w_dtype == FB_F32, "low_rank_maps: unknown dtype code %d", w_dtype);
        fb_launch(low_rank_fma_kernel<float>, dim3((n + LF_TM - 1) / LF_TM, tiles), dim3(256), 0, stream, a);
    }
    return fb_check_launch("low_rank_maps");
}
