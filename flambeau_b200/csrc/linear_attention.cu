// Gated linear attention: a linear recurrence with one matrix of state per head, S [dk, dv] in float32, whose rows
// (one per key channel) decay each by a factor of its own before a token adds its key times its value:
//
//     S <- diag(alpha) S + k v^T;   o = S^T q          (alpha: one number per head, key channel and token)
//     alpha = sigmoid(z)^(1/tau),   z = W2 (W1 h) + b  (a map through a narrow middle, W1 h being part of the
//                                                        mixer's stacked projection)
//
// Kernels, in the order a step runs them:
//   gla_prepare      per (token, head): add the projection's split-K shares; q times `q_scale`, k and v as they are;
//                    z from the narrow middle, log sigmoid(z) / tau and its exponential; all float32
//   (then the recurrence: recurrence.cu)
// The head norm and output gate that follow are those of the gated delta rule (gdr_out_norm).
//
// A request's slot of state holds S as [heads][dv][dk] (a column's dk values side by side) at its start.
// Projection rows are [q: H*dk | k: H*dk | v: H*dv | gate: H*dv | middle: R].
#include "common.cuh"

__device__ __forceinline__ float gla_slab_sum(const float* row, int c, int n_partials, long partial_stride) {
    return fb_slab_sum(row, c, n_partials, partial_stride);
}

template <typename TW>
__global__ void __launch_bounds__(128)
gla_prepare_kernel(const float* __restrict__ proj, long proj_stride, int n_partials, long partial_stride,
                   const TW* __restrict__ w2, const TW* __restrict__ b2, int R, float inv_tau, float q_scale,
                   float* __restrict__ qkv, float* __restrict__ decay, int H, int dk, int dv) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    extern __shared__ float mid[];                     // the narrow middle of the decay's map, [R]
    const int row = blockIdx.x, head = blockIdx.y, tid = threadIdx.x;
    const int qk = H * dk, C = 2 * qk + H * dv;
    const float* pr = proj + (size_t)row * proj_stride;
    for (int r = tid; r < R; r += blockDim.x) mid[r] = gla_slab_sum(pr, C + H * dv + r, n_partials, partial_stride);
    __syncthreads();
    float* out = qkv + (size_t)row * C;
    for (int d = tid; d < dk; d += blockDim.x) {
        const int c = head * dk + d;
        out[c] = gla_slab_sum(pr, c, n_partials, partial_stride) * q_scale;
        out[qk + c] = gla_slab_sum(pr, qk + c, n_partials, partial_stride);
        float z = fb_to_float(b2[c]);
        const TW* wr = w2 + (size_t)c * R;
        for (int r = 0; r < R; ++r) z = fmaf(fb_to_float(wr[r]), mid[r], z);
        // log sigmoid(z) = min(z, 0) - log(1 + exp(-|z|))
        const float ls = fminf(z, 0.0f) - log1pf(expf(-fabsf(z)));
        decay[(size_t)row * qk + c] = expf(ls * inv_tau);
    }
    for (int d = tid; d < dv; d += blockDim.x) {
        const int c = 2 * qk + head * dv + d;
        out[c] = gla_slab_sum(pr, c, n_partials, partial_stride);
    }
}

FB_API int fb_gla_prepare(const float* proj, long long proj_stride, int n_partials, long long partial_stride,
                          const void* w2, const void* b2, int w_dtype, int R, float tau, float q_scale, float* qkv,
                          float* decay, int n, int H, int dk, int dv, cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && H > 0 && dk > 0 && dv > 0 && R > 0, "linear attention: bad sizes");
    FB_REQUIRE(tau > 0.0f, "linear attention: tau must be positive");
    FB_REQUIRE(proj_stride >= 2LL * H * dk + 2LL * H * dv + R, "linear attention: projection rows are too short");
    FB_REQUIRE(H <= 65535 && R <= 8192, "linear attention: too many heads, or a middle wider than 8192");
    if (n == 0) return 0;
    if (n_partials < 1) n_partials = 1;
    FB_DISPATCH_DTYPE(w_dtype, TW,
        (fb_launch((gla_prepare_kernel<TW>), dim3(n, H), dim3(128), (size_t)R * sizeof(float), stream, proj,
                   (long)proj_stride, n_partials, (long)partial_stride, (const TW*)w2, (const TW*)b2, R, 1.0f / tau,
                   q_scale, qkv, decay, H, dk, dv)));
    return fb_check_launch("gla_prepare");
}
