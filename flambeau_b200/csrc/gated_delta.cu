// The gated delta rule: a linear recurrence with one matrix of state per head, S [dk, dv] in float32, which a token
// first lets decay, then corrects along its key towards its value, then reads with its query:
//
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q        (g, beta: one number per head and token)
//
// or, with a decay per key channel, S <- diag(g) S with one number of g per row of S.
//
// Kernels, in the order a step runs them:
//   gdr_prepare      per (token, head of q, k or v): add the projection's split-K shares, the short causal convolution
//                    over time with its SiLU (inputs before the portion's start come from the request's kept tail),
//                    q and k made unit vectors per head (q also times `q_scale`), beta = sigmoid,
//                    g = exp(-exp(A_log) * softplus(a + dt_bias)) where a head has one; all float32 (decays per key
//                    channel come from a map through a narrow middle: low_rank.cu)
//   gdr_conv_tail    per request: the last taps-1 convolution inputs of the step become the kept tail
//   (then the recurrence: recurrence.cu)
//   gdr_out_norm     per (token, head): o / rms(o) * weight * act(gate) (silu, sigmoid, or the gate as it is), rounded to
//                    the engine's dtype
//
// A request's slot of state is one float32 array: S as [heads][dv][dk] (a column's dk values side by side), then the
// tail as [taps-1][channels]
// (oldest first).  Projection rows begin [q: G*dk | k: G*dk | v: H*dv]; where beta, the decay and the gate lie behind
// them are arguments; head h of H reads q/k head h / (H / G).
#include "rows.cuh"

__device__ __forceinline__ float gdr_slab_sum(const float* row, int c, int n_partials, long partial_stride) {
    float v = row[c];
    for (int p = 1; p < n_partials; ++p) v += row[(size_t)p * partial_stride + c];
    return v;
}
__device__ __forceinline__ float gdr_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float gdr_softplus(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

template <typename TW>
__global__ void __launch_bounds__(128)
gdr_prepare_kernel(const float* __restrict__ proj, long proj_stride, int n_partials, long partial_stride,
                   const TW* __restrict__ conv_w, int taps, int b_off, int a_off, const TW* __restrict__ a_log,
                   const TW* __restrict__ dt_bias, const float* __restrict__ state, long state_stride, long tail_off, const int* __restrict__ row_seq,
                   const int* __restrict__ seq_q_start, const int* __restrict__ seq_slot, float* __restrict__ qkv,
                   float* __restrict__ beta, float* __restrict__ decay, int G, int H, int dk, int dv, float q_scale,
                   float unit_eps) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    constexpr int PER = 8;                             // channels a thread takes: heads of up to 1024
    __shared__ float red[32];
    const int row = blockIdx.x, unit = blockIdx.y, tid = threadIdx.x;
    const int qk = G * dk, C = 2 * qk + H * dv;
    const bool is_v = unit >= 2 * G;
    const int width = is_v ? dv : dk;
    const int base = is_v ? 2 * qk + (unit - 2 * G) * dv : unit * dk;    // q heads, then k heads, then v heads
    const int seq = row_seq[row];
    const int i = row - seq_q_start[seq];              // place within the step's portion of this request
    const float* tail = state + (size_t)seq_slot[seq] * state_stride + tail_off;
    float y[PER];
    float sq = 0.0f;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
        const int d = tid + 128 * e;
        y[e] = 0.0f;
        if (d >= width) continue;
        const int c = base + d;
        float acc = 0.0f;
        for (int j = 0; j < taps; ++j) {
            const int src = i - (taps - 1 - j);
            const float x = src >= 0
                ? gdr_slab_sum(proj + (size_t)(row - (taps - 1 - j)) * proj_stride, c, n_partials, partial_stride)
                : tail[(size_t)(taps - 1 + src) * C + c];
            acc = fmaf(fb_to_float(conv_w[(size_t)c * taps + j]), x, acc);
        }
        y[e] = gdr_silu(acc);
        sq = fmaf(y[e], y[e], sq);
    }
    float f = 1.0f;
    if (!is_v) {                                       // block-uniform
        sq = fb_block_sum(sq, red);
        f = (unit < G ? q_scale : 1.0f) / sqrtf(sq + unit_eps);
    }
    float* out = qkv + (size_t)row * C + base;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
        const int d = tid + 128 * e;
        if (d < width) out[d] = y[e] * f;
    }
    if (is_v && tid == 0) {
        const int h = unit - 2 * G;
        const float* pr = proj + (size_t)row * proj_stride;
        const float b = gdr_slab_sum(pr, b_off + h, n_partials, partial_stride);
        beta[(size_t)row * H + h] = 1.0f / (1.0f + expf(-b));
        if (!decay) return;
        const float a = gdr_slab_sum(pr, a_off + h, n_partials, partial_stride);
        decay[(size_t)row * H + h] = expf(-expf(fb_to_float(a_log[h])) * gdr_softplus(a + fb_to_float(dt_bias[h])));
    }
}

// Sums over the warp of ROWS numbers a lane (ROWS a power of two, at most 32), every one in the order of fb_warp_sum: the
// lanes that differ in bit 16, then 8 and so on meet, and as long as there are several numbers left a lane sends those that it
// does not keep.  Lane l ends with the sum of number l / (32 / ROWS): five to nine exchanges instead of five a number.
template <int ROWS>
__device__ __forceinline__ float warp_sums(float (&v)[ROWS]) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int left = ROWS; left > 1; left >>= 1, o >>= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
            if (r >= left / 2) break;
            const float keep = upper ? v[r + left / 2] : v[r], give = upper ? v[r] : v[r + left / 2];
            v[r] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// The same for up to four taps and heads of up to 256 whose sizes are multiples of 4: a warp takes a head of ROWS
// neighbouring rows, four neighbouring channels a lane (16-byte loads and stores, NV groups of them), and the rows' inputs
// form a window in registers, so that a row's input is fetched once and not once a tap; an input ahead of the portion's first
// token is a load from the kept tail in its place.  The rows' norms are summed together and their factors formed by a lane
// each.  What bounds it is the SiLU's exponential and division.  2,048 rows of 96 heads of 128 took 97 us with every row's own
// sums, factors and choice between tail and input, now 62 (200 MB, 31 at the copy rate); 1,029 rows of 24 heads 31 and 16.
template <typename TW, int TAPS, int NV, int ROWS>
__global__ void __launch_bounds__(128)
gdr_prepare_vec_kernel(const float* __restrict__ proj, long proj_stride, int n_partials, long partial_stride,
                       const TW* __restrict__ conv_w, int b_off, int a_off, const TW* __restrict__ a_log,
                       const TW* __restrict__ dt_bias, const float* __restrict__ state, long state_stride, long tail_off,
                       const int* __restrict__ row_seq, const int* __restrict__ seq_q_start, const int* __restrict__ seq_slot,
                       float* __restrict__ qkv, float* __restrict__ beta, float* __restrict__ decay, int n, int G, int H,
                       int dk, int dv, float q_scale, float unit_eps) {
    fb_pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int units = 2 * G + H, qk = G * dk, C = 2 * qk + H * dv;
    const int unit = (int)blockIdx.y * 4 + warp, row0 = (int)blockIdx.x * ROWS;
    if (unit >= units) return;
    const bool is_v = unit >= 2 * G;
    const int width = is_v ? dv : dk;
    const int base = is_v ? 2 * qk + (unit - 2 * G) * dv : unit * dk;    // q heads, then k heads, then v heads
    float w[NV][4 * TAPS];                             // [channel][tap]
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int d = 4 * lane + 128 * i;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const float4 v = d < width ? Vec4<TW>::load(conv_w + (size_t)(base + d) * TAPS + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
            w[i][4 * j] = v.x; w[i][4 * j + 1] = v.y; w[i][4 * j + 2] = v.z; w[i][4 * j + 3] = v.w;
        }
    }
    fb_pdl_wait();
    const int rows = min(ROWS, n - row0);
    const int seq = row_seq[row0];
    // x[m], m < count: the inputs of rows row + m - (TAPS - 1) of request `of`, which has `place` of its portion's rows ahead of
    // row `row`: the projection's or, ahead of the portion, the kept ones.  Addresses first, so that every load is in flight.
    auto fetch = [&](float4* x, int count, int row, int place, int of, int c, bool in) {
        const float* kept = state + (size_t)seq_slot[of] * state_stride + tail_off + c;
        const float* fresh = proj + c;
        if (ROWS == 1 && n_partials > 1) {              // one number a tap, its shares eight at a time
#pragma unroll
            for (int m = 0; m < TAPS; ++m) {
                const int off = m - (TAPS - 1);
                x[m] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!in) continue;
                if (place + off >= 0) x[m] = slab_sum4(fresh + (long)(row + off) * proj_stride, n_partials, partial_stride);
                else x[m] = Vec4<float>::load(kept + (long)(TAPS - 1 + place + off) * C);
            }
            return;
        }
#pragma unroll
        for (int m = 0; m < ROWS + TAPS - 1; ++m) {
            const int off = m - (TAPS - 1);
            const float* p = place + off >= 0 ? fresh + (long)(row + off) * proj_stride : kept + (long)(TAPS - 1 + place + off) * C;
            x[m] = in && m < count ? Vec4<float>::load(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (n_partials > 1 && in) {
            for (int s = 1; s < n_partials; ++s)
#pragma unroll
                for (int m = 0; m < ROWS + TAPS - 1; ++m) {
                    if (m >= count) break;
                    const int off = m - (TAPS - 1);
                    if (place + off < 0) continue;
                    const float4 v = Vec4<float>::load(fresh + (size_t)s * partial_stride + (long)(row + off) * proj_stride);
                    x[m].x += v.x; x[m].y += v.y; x[m].z += v.z; x[m].w += v.w;
                }
        }
    };
    auto mix = [&](int i, const float4* x) -> float4 {  // the convolution over x[0 .. TAPS) with its SiLU
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            acc[0] = fmaf(w[i][j], x[j].x, acc[0]);
            acc[1] = fmaf(w[i][TAPS + j], x[j].y, acc[1]);
            acc[2] = fmaf(w[i][2 * TAPS + j], x[j].z, acc[2]);
            acc[3] = fmaf(w[i][3 * TAPS + j], x[j].w, acc[3]);
        }
        return make_float4(gdr_silu(acc[0]), gdr_silu(acc[1]), gdr_silu(acc[2]), gdr_silu(acc[3]));
    };
    float4 y[NV][ROWS];
    float sq[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) sq[r] = 0.0f;
    const bool one = ROWS == 1 || row_seq[row0 + rows - 1] == seq;       // (a request's rows lie side by side)
    const int place0 = row0 - seq_q_start[seq];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int d = 4 * lane + 128 * i;
        const bool in = d < width;
        if (one) {
            float4 x[ROWS + TAPS - 1];                 // x[m]: the input of row row0 + m - (TAPS - 1)
            fetch(x, rows + TAPS - 1, row0, place0, seq, base + d, in);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) y[i][r] = mix(i, x + r);
        } else {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                float4 x[ROWS + TAPS - 1];
                const int row = row0 + min(r, rows - 1), of = row_seq[row], place = row - seq_q_start[of];
                fetch(x, TAPS, row, place, of, base + d, in);
                y[i][r] = mix(i, x);
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            sq[r] = fmaf(y[i][r].x, y[i][r].x, sq[r]);
            sq[r] = fmaf(y[i][r].y, y[i][r].y, sq[r]);
            sq[r] = fmaf(y[i][r].z, y[i][r].z, sq[r]);
            sq[r] = fmaf(y[i][r].w, y[i][r].w, sq[r]);
        }
    }
    float f = 1.0f;
    if (!is_v) f = (unit < G ? q_scale : 1.0f) / sqrtf(warp_sums<ROWS>(sq) + unit_eps);       // (warp-uniform)
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const float fr = is_v ? 1.0f : __shfl_sync(0xffffffffu, f, r * (32 / ROWS));
        if (r >= rows) break;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int d = 4 * lane + 128 * i;
            if (d < width)
                Vec4<float>::store(qkv + (size_t)(row0 + r) * C + base + d,
                                   make_float4(y[i][r].x * fr, y[i][r].y * fr, y[i][r].z * fr, y[i][r].w * fr));
        }
    }
    if (is_v && lane < rows) {
        const int h = unit - 2 * G, row = row0 + lane;
        const float* pr = proj + (size_t)row * proj_stride;
        beta[(size_t)row * H + h] = 1.0f / (1.0f + expf(-fb_slab_sum(pr, b_off + h, n_partials, partial_stride)));
        if (decay) {
            const float a = fb_slab_sum(pr, a_off + h, n_partials, partial_stride);
            decay[(size_t)row * H + h] = expf(-expf(fb_to_float(a_log[h])) * gdr_softplus(a + fb_to_float(dt_bias[h])));
        }
    }
}

__global__ void gdr_conv_tail_kernel(const float* __restrict__ proj, long proj_stride, int n_partials, long partial_stride,
                                     int taps, float* __restrict__ state, long state_stride, long tail_off,
                                     const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                                     const int* __restrict__ seq_slot, int C) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const int seq = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int L = seq_q_len[seq], start = seq_q_start[seq];
    float* tail = state + (size_t)seq_slot[seq] * state_stride + tail_off;
    // ascending m: an entry taken from the old tail lies above the one being written
    for (int m = 0; m < taps - 1; ++m) {
        const int src = L - (taps - 1) + m;
        tail[(size_t)m * C + c] = src >= 0
            ? gdr_slab_sum(proj + (size_t)(start + src) * proj_stride, c, n_partials, partial_stride)
            : tail[(size_t)(taps - 1 + src) * C + c];
    }
}

enum FbGdrGate : int { FB_GDR_SILU = 0, FB_GDR_SIGMOID = 1, FB_GDR_AS_IS = 2 };

__device__ __forceinline__ float gdr_gate(int gate_act, float gate) {
    if (gate_act == FB_GDR_SILU) return gdr_silu(gate);
    if (gate_act == FB_GDR_SIGMOID) return 1.0f / (1.0f + expf(-gate));
    return gate;
}

template <typename TW, typename T>
__global__ void __launch_bounds__(128)
gdr_out_norm_kernel(const float* __restrict__ o, const float* __restrict__ proj, long proj_stride, int n_partials,
                    long partial_stride, int gate_off, int gate_act, const TW* __restrict__ weight, float eps, T* __restrict__ out,
                    int n, int H, int dv) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long item = (long)blockIdx.x * 4 + warp;
    if (item >= (long)n * H) return;
    const int row = (int)(item / H), head = (int)(item - (long)row * H);
    const float* x = o + (size_t)row * H * dv + (size_t)head * dv;
    float s = 0.0f;
    for (int d = lane; d < dv; d += 32) s = fmaf(x[d], x[d], s);
    s = fb_warp_sum(s);
    const float inv = 1.0f / sqrtf(s / (float)dv + eps);
    const float* pr = proj + (size_t)row * proj_stride;
    for (int d = lane; d < dv; d += 32) {
        float gate = gdr_slab_sum(pr, gate_off + head * dv + d, n_partials, partial_stride);
        gate = gdr_gate(gate_act, gate);
        out[(size_t)row * H * dv + (size_t)head * dv + d] =
            fb_from_float<T>(x[d] * inv * fb_to_float(weight[d]) * gate);
    }
}

// The same for heads of up to 512 whose sizes are multiples of 4, rows on 16-byte borders: four neighbouring channels a lane,
// NV groups of them, held between the sum and the output.  2,048 rows of 32 heads of 128: 32 us before (one number a load, the
// head read twice), 20 here for 84 MB.
template <typename TW, typename T, int NV>
__global__ void __launch_bounds__(128)
gdr_out_norm_vec_kernel(const float* __restrict__ o, const float* __restrict__ proj, long proj_stride, int n_partials,
                        long partial_stride, int gate_off, int gate_act, const TW* __restrict__ weight, float eps, T* __restrict__ out,
                        int n, int H, int dv) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const int lane = threadIdx.x & 31, head = (int)blockIdx.y * 4 + (threadIdx.x >> 5), row = blockIdx.x;
    if (head >= H) return;
    const size_t at = (size_t)row * H * dv + (size_t)head * dv;
    const float* gates = proj + (size_t)row * proj_stride + gate_off + (size_t)head * dv;
    float4 x[NV], g[NV];
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int d = 4 * lane + 128 * i;
        x[i] = g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d >= dv) continue;
        x[i] = Vec4<float>::load(o + at + d);
        g[i] = slab_sum4(gates + d, n_partials, partial_stride);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) s += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
    const float inv = 1.0f / sqrtf(fb_warp_sum(s) / (float)dv + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int d = 4 * lane + 128 * i;
        if (d >= dv) continue;
        const float4 w = Vec4<TW>::load(weight + d);
        Vec4<T>::store(out + at + d, make_float4(x[i].x * inv * w.x * gdr_gate(gate_act, g[i].x), x[i].y * inv * w.y * gdr_gate(gate_act, g[i].y),
                                                 x[i].z * inv * w.z * gdr_gate(gate_act, g[i].z), x[i].w * inv * w.w * gdr_gate(gate_act, g[i].w)));
    }
}

// decay (with a_log, dt_bias and the columns from a_off on) may be null: no decay per head.
FB_API int fb_gdr_prepare(const float* proj, long long proj_stride, int n_partials, long long partial_stride,
                          const void* conv_w, int taps, int b_off, int a_off, const void* a_log, const void* dt_bias, int w_dtype,
                          float* state, long long state_stride, long long tail_off, const int* row_seq,
                          const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int n_seqs, float* qkv,
                          float* beta, float* decay, int n, int G, int H, int dk, int dv, float q_scale,
                          float unit_eps, cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && G > 0 && H > 0 && H % G == 0 && dk > 0 && dv > 0 && taps >= 1, "gated delta: bad sizes");
    const long long C = 2LL * G * dk + (long long)H * dv;
    FB_REQUIRE(b_off >= C && proj_stride >= (long long)b_off + H, "gated delta: projection rows are too short");
    FB_REQUIRE(!decay || (a_log && dt_bias && a_off >= C && proj_stride >= (long long)a_off + H),
               "gated delta: a decay per head wants its columns and parameters");
    if (n == 0) return 0;
    if (n_partials < 1) n_partials = 1;
    FB_REQUIRE(dk <= 1024 && dv <= 1024, "gated delta: head sizes up to 1024 (key %d, value %d)", dk, dv);
    FB_REQUIRE(2 * G + H <= 65535, "gated delta: too many heads");
    const size_t wsize = w_dtype == FB_BF16 ? 2 : 4;
    const int widest = dk > dv ? dk : dv;
    auto aligned = [](const void* p, size_t to) { return (uintptr_t)p % to == 0; };
    const bool vec = taps <= 4 && dk % 4 == 0 && dv % 4 == 0 && widest <= 256 && proj_stride % 4 == 0 && partial_stride % 4 == 0 &&
                     state_stride % 4 == 0 && tail_off % 4 == 0 && aligned(proj, 16) && aligned(state, 16) && aligned(qkv, 16) &&
                     aligned(conv_w, 4 * wsize);
    if (vec) {
        // (a few rows: one a warp, so that the heads spread over the device; a portion: four, which share their windows and
        // sums; eight leave half as many warps, of twice the registers: 2,048 rows 62 us either way, 1,029 rows 16 / 34)
#define FB_GDP_LAUNCH(TAPS_, NV_, ROWS_)                                                                                     \
        FB_DISPATCH_DTYPE(w_dtype, TW,                                                                                       \
            (fb_launch((gdr_prepare_vec_kernel<TW, TAPS_, NV_, ROWS_>),                                                      \
                       dim3((unsigned)((n + ROWS_ - 1) / ROWS_), (unsigned)((2 * G + H + 3) / 4)), dim3(128), 0, stream, proj, \
                       (long)proj_stride, n_partials, (long)partial_stride, (const TW*)conv_w, b_off, a_off, (const TW*)a_log, \
                       (const TW*)dt_bias, (const float*)state, (long)state_stride, (long)tail_off, row_seq, seq_q_start,     \
                       seq_slot, qkv, beta, decay, n, G, H, dk, dv, q_scale, unit_eps)))
#define FB_GDP_TAPS(TAPS_)                                                                                                   \
        case TAPS_:                                                                                                          \
            if (widest <= 128) { if (n <= 64) FB_GDP_LAUNCH(TAPS_, 1, 1); else FB_GDP_LAUNCH(TAPS_, 1, 4); }                   \
            else { if (n <= 64) FB_GDP_LAUNCH(TAPS_, 2, 1); else FB_GDP_LAUNCH(TAPS_, 2, 4); }                                \
            break;
        switch (taps) { FB_GDP_TAPS(1) FB_GDP_TAPS(2) FB_GDP_TAPS(3) FB_GDP_TAPS(4) }
#undef FB_GDP_TAPS
#undef FB_GDP_LAUNCH
    } else
    FB_DISPATCH_DTYPE(w_dtype, TW, {
        auto kernel = gdr_prepare_kernel<TW>;
        fb_launch(kernel, dim3(n, 2 * G + H), dim3(128), 0, stream, proj, (long)proj_stride, n_partials, (long)partial_stride,
                  (const TW*)conv_w, taps, b_off, a_off, (const TW*)a_log, (const TW*)dt_bias, (const float*)state, (long)state_stride,
                  (long)tail_off, row_seq, seq_q_start, seq_slot, qkv, beta, decay, G, H, dk, dv, q_scale, unit_eps);
    });
    int rc = fb_check_launch("gdr_prepare");
    if (rc || taps < 2) return rc;
    fb_launch(gdr_conv_tail_kernel, dim3(n_seqs, (unsigned)((C + 127) / 128)), dim3(128), 0, stream, proj,
              (long)proj_stride, n_partials, (long)partial_stride, taps, state, (long)state_stride, (long)tail_off,
              seq_q_start, seq_q_len, seq_slot, (int)C);
    return fb_check_launch("gdr_conv_tail");
}

FB_API int fb_gdr_out_norm(const float* o, const float* proj, long long proj_stride, int n_partials,
                           long long partial_stride, int gate_off, int gate_act, const void* weight, int w_dtype, float eps,
                           void* out, int out_dtype, int n, int H, int dv, cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && H > 0 && dv > 0, "gated delta: bad sizes");
    FB_REQUIRE(gate_act >= FB_GDR_SILU && gate_act <= FB_GDR_AS_IS, "gated delta: unknown gate %d", gate_act);
    if (n == 0) return 0;
    if (n_partials < 1) n_partials = 1;
    const long items = (long)n * H;
    const size_t wsize = w_dtype == FB_BF16 ? 2 : 4, osize = out_dtype == FB_BF16 ? 2 : 4;
    if (dv % 4 == 0 && dv <= 512 && gate_off % 4 == 0 && proj_stride % 4 == 0 && partial_stride % 4 == 0 && (uintptr_t)o % 16 == 0 &&
        (uintptr_t)proj % 16 == 0 && (uintptr_t)weight % (4 * wsize) == 0 && (uintptr_t)out % (4 * osize) == 0 && (H + 3) / 4 <= 65535) {
#define FB_GON_LAUNCH(NV_)                                                                                                    \
        FB_DISPATCH_DTYPE(w_dtype, TW, FB_DISPATCH_DTYPE(out_dtype, T,                                                        \
            (fb_launch((gdr_out_norm_vec_kernel<TW, T, NV_>), dim3(n, (unsigned)((H + 3) / 4)), dim3(128), 0, stream, o, proj, \
                       (long)proj_stride, n_partials, (long)partial_stride, gate_off, gate_act, (const TW*)weight, eps, (T*)out, n, H, dv))))
        if (dv <= 128) FB_GON_LAUNCH(1);
        else if (dv <= 256) FB_GON_LAUNCH(2);
        else FB_GON_LAUNCH(4);
#undef FB_GON_LAUNCH
        return fb_check_launch("gdr_out_norm");
    }
    FB_DISPATCH_DTYPE(w_dtype, TW, FB_DISPATCH_DTYPE(out_dtype, T,
        (fb_launch((gdr_out_norm_kernel<TW, T>), dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, o, proj,
                   (long)proj_stride, n_partials, (long)partial_stride, gate_off, gate_act, (const TW*)weight, eps, (T*)out, n, H,
                   dv))));
    return fb_check_launch("gdr_out_norm");
}
