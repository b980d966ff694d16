// A map per head over a portion's rows on the 5th-generation tensor cores: out[t, h, :N] = W_h [N, K] . a[t, h, :K] in
// bfloat16 (latent_attention.cu describes what it is for; its mma.sync kernel keeps steps of few rows and other sizes).
//
// A CTA takes 128 rows of one head: the head's weights by TMA (they do not wait for the kernel before), the rows by TMA where
// they are bfloat16, else float32 shares that all threads add, round once and place as the MMA wants them.  One tcgen05.mma
// chain of K / 16 instructions of M = 128 rows, N outputs; the results pass through the weights' shared memory into boxes of
// 64 outputs x 128 rows that TMA stores (rows beyond the portion are not written).
//
// What bounds it: memory, 66 MB for 2,048 rows of 32 heads of 128 -> 256 from float32 (10 us at the copy rate).  With 64 x 64
// tiles of mma.sync, which fetch a head's weights for every 64 rows and its rows for every 64 outputs, this took 44 us, now 16;
// 256 -> 128 from bfloat16 38, now 17.
#include "tensor_map.cuh"
#include "umma.cuh"

namespace {

constexpr int HT_ROWS = 128, HT_KB = 64;               // rows of a CTA; K of a swizzled block (128 bytes)
constexpr int HT_BLOCK = HT_ROWS * HT_KB * 2;          // bytes of such a block of rows
constexpr int HT_THREADS = 256;

__host__ __device__ inline int ht_smem(int N, int K) {
    const int weights = N * K * 2, staged = N / HT_KB * HT_BLOCK;
    return K / HT_KB * HT_BLOCK + (weights > staged ? weights : staged) + 1024 + 64;
}

template <typename TA>
__global__ void __launch_bounds__(HT_THREADS)
head_linear_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                      const __grid_constant__ CUtensorMap map_o, const TA* __restrict__ a, long a_stride, long a_head, int n_partials,
                      long partial_stride, int o_head, int n, int N, int K, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* As = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* Ws = As + K / HT_KB * HT_BLOCK;
    const int weights = N * K * 2, staged = N / HT_KB * HT_BLOCK;
    uint64_t* bars = (uint64_t*)(Ws + (weights > staged ? weights : staged));      // [operands there, products done]
    uint32_t* tmem_slot = (uint32_t*)(bars + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * HT_ROWS, h = blockIdx.y;
    constexpr bool BY_TMA = sizeof(TA) == 2;
    uint32_t cols = 32;
    while ((int)cols < N) cols *= 2;

    if (tid == 0) {
        mbar_init(smem_u32(&bars[0]), 1);
        mbar_init(smem_u32(&bars[1]), 1);
        mbar_fence_init();
        mbar_expect_tx(smem_u32(&bars[0]), (uint32_t)(weights + (BY_TMA ? K / HT_KB * HT_BLOCK : 0)));
        for (int k = 0; k < K; k += HT_KB)
            tma_load_2d(smem_u32(Ws + (size_t)(k / HT_KB) * N * 128), &map_w, smem_u32(&bars[0]), k, h * N);
    }
    fb_pdl_wait();
    if (BY_TMA && tid == 0)
        for (int k = 0; k < K; k += HT_KB)
            tma_load_2d(smem_u32(As + k / HT_KB * HT_BLOCK), &map_a, smem_u32(&bars[0]), (int)(h * a_head) + k, m0);
    // (behind the wait, so that it waits for no column of the kernel before; dependents behind it, who could hold theirs for good)
    if (warp == 1) tmem_alloc(tmem_slot, cols);
    tmem_fence_before();
    __syncthreads();
    fb_pdl_launch_dependents();
    if (!BY_TMA) {
        constexpr int U = 8;                            // groups of four numbers a thread has in flight
        const float* from = reinterpret_cast<const float*>(a) + (size_t)h * a_head;
        const int per_row = K / 4, groups = HT_ROWS * per_row;
        for (int g0 = tid; g0 < groups; g0 += U * HT_THREADS) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int g = g0 + u * HT_THREADS, row = g / per_row, k = 4 * (g - row * per_row);
                v[u] = g < groups && m0 + row < n ? *reinterpret_cast<const float4*>(from + (size_t)(m0 + row) * a_stride + k)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            for (int p = 1; p < n_partials; ++p)
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int g = g0 + u * HT_THREADS, row = g / per_row, k = 4 * (g - row * per_row);
                    if (g < groups && m0 + row < n) {
                        const float4 m = *reinterpret_cast<const float4*>(from + (size_t)p * partial_stride + (size_t)(m0 + row) * a_stride + k);
                        v[u].x += m.x; v[u].y += m.y; v[u].z += m.z; v[u].w += m.w;
                    }
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int g = g0 + u * HT_THREADS, row = g / per_row, k = 4 * (g - row * per_row);
                if (g >= groups) continue;
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v[u].x, v[u].y), hi = __floats2bfloat162_rn(v[u].z, v[u].w);
                const int byte = 2 * (k % HT_KB);
                *reinterpret_cast<uint2*>(As + k / HT_KB * HT_BLOCK + row * 128 + (((byte >> 4) ^ (row & 7)) << 4) + (byte & 15)) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            ok = mbar_wait(smem_u32(&bars[0]), 0, status);
            tmem_fence_after();
            if (ok) {
                const uint32_t idesc = umma_idesc(N);
                for (int k = 0; k < K; k += UMMA_K) {
                    const uint64_t da = umma_desc(smem_u32(As + k / HT_KB * HT_BLOCK)) + (uint64_t)((k % HT_KB) / 8);
                    const uint64_t db = umma_desc(smem_u32(Ws + (size_t)(k / HT_KB) * N * 128)) + (uint64_t)((k % HT_KB) / 8);
                    umma_bf16(tmem, da, db, idesc, k > 0 ? 1u : 0u);
                }
            }
            umma_commit(smem_u32(&bars[1]));            // (without products: at once)
        }
        __syncwarp();
    }
    const bool done = mbar_wait(smem_u32(&bars[1]), 0, status);
    tmem_fence_after();
    if (done) {
        // lanes are rows, the two warps of a quarter take 32 outputs in turn; a row's 64 outputs of a box are 128 swizzled bytes
        const int quarter = warp & 3, row = quarter * 32 + lane;
        for (int c0 = (warp >> 2) * 32; c0 < N; c0 += 64) {
            uint32_t r[32];
            tmem_ld32_nowait(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
            tmem_wait_ld();
            uint8_t* dst = Ws + c0 / HT_KB * HT_BLOCK + row * 128;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(r[8 * q + 2 * e]), __uint_as_float(r[8 * q + 2 * e + 1]));
                    w[e] = *reinterpret_cast<const uint32_t*>(&b);
                }
                const int chunk = (c0 % HT_KB) / 8 + q;
                *reinterpret_cast<uint4*>(dst + ((chunk ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    tmem_fence_before();
    __syncthreads();
    if (tid == 0 && done) {
        for (int c = 0; c < N; c += HT_KB)
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                         ::"l"(&map_o), "r"(smem_u32(Ws + c / HT_KB * HT_BLOCK)), "r"(h * o_head + c), "r"(m0) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (warp == 1) {
        tmem_fence_after();
        tmem_dealloc(tmem, cols);
    }
}

template <typename TA>
int launch(const TA* a, long a_stride, long a_head, int n_partials, long partial_stride, const void* w, void* out, long o_stride, long o_head,
           int n, int H, int N, int K, int* status, cudaStream_t stream) {
    CUtensorMap mw, ma, mo;
    int rc = fb_tensor_map_bf16(&mw, w, (long)H * N, K, K, HT_KB, N);
    if (rc) return rc;
    rc = fb_tensor_map_bf16(&mo, out, n, (long)(H - 1) * o_head + N, o_stride, HT_KB, HT_ROWS);
    if (rc) return rc;
    if (sizeof(TA) == 2) rc = fb_tensor_map_bf16(&ma, a, n, (long)(H - 1) * a_head + K, a_stride, HT_KB, HT_ROWS);
    else ma = mw;                                       // (not used)
    if (rc) return rc;
    auto kernel = head_linear_tc_kernel<TA>;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return fb_fail(-2, "head_linear: cannot reserve shared memory: %s", cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    fb_launch(kernel, dim3((n + HT_ROWS - 1) / HT_ROWS, H), dim3(HT_THREADS), (size_t)ht_smem(N, K), stream, mw, ma, mo, a, a_stride, a_head,
              n_partials, partial_stride, (int)o_head, n, N, K, status);
    return fb_check_launch("head_linear_tc");
}

}  // namespace

// Bfloat16 weights [H, N, K] and outputs, inputs in bfloat16 or as float32 shares: portions of at least 128 rows (fewer leave a
// tile half empty), sizes that are multiples of 64, at most 256 outputs, rows and heads on 16-byte borders, and as many tiles of
// 128 rows as it takes to be faster than 64 x 64 tiles, whose CTAs share a few rows' work among more SMs.  Measured over 2 to
// 1,024 tiles (us there / here, inputs -> outputs):
//   bfloat16: wherever there are as many inputs as outputs (256 -> 128: 8 tiles 5.8 / 4.4, 256 30.4 / 15.8), else from a quarter
//   of the SMs on (64 -> 256: 8 tiles 1.4 times as long, 32 1.1, 40 even; 128 -> 256: 16 tiles 1.2 times, 40 0.8)
//   float32: no more inputs than outputs, of which 128 at least, from half of the SMs on (128 -> 256: 8 tiles 4.1 / 7.4, 64 6.9 /
//   7.5, 80 8.9 / 7.5, 512 39.0 / 17.6; 64 -> 64: 80 tiles 3.5 / 4.4, 448 7.1 / 7.8; 256 -> 128: 448 tiles 1.1 times as long)
//   several float32 shares: from a tile for every SM on (130 rows of 32 heads, three shares, 128 -> 256: 21 us here, 16 there;
//   800 rows 8.6 and 17)
// Returns 1, nothing done, for anything else: the caller takes fb_head_linear.
FB_API int fb_head_linear_tc(const void* a, int a_dtype, long long a_stride, long long a_head, int n_partials, long long partial_stride,
                             const void* w, void* out, long long o_stride, long long o_head, int n, int H, int N, int K, int* status,
                             cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && H > 0 && N > 0 && K > 0 && status, "head_linear: bad sizes");
    FB_REQUIRE(n_partials <= 1 || a_dtype == FB_F32, "head_linear: only float32 inputs come as shares");
    if (n_partials < 1) n_partials = 1;
    const long long per = a_dtype == FB_F32 ? 4 : 8;
    auto aligned = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
    const long tiles = (long)((n + HT_ROWS - 1) / HT_ROWS) * H;
    const bool enough = n_partials > 1 ? tiles >= fb_sm_count()
                        : a_dtype == FB_F32 ? N >= 128 && K <= N && tiles >= fb_sm_count() / 2 : K >= N || tiles >= fb_sm_count() / 4;
    const bool takes = n >= 128 && enough && N % HT_KB == 0 && N <= 256 && K % HT_KB == 0 && K <= 4096 && ht_smem(N, K) <= 227 * 1024 && H <= 65535 &&
                       (long long)H * N < 2147483647LL && a_head >= 0 && a_head < 2147483647LL / H && o_head >= N && o_head < 2147483647LL / H &&
                       a_stride >= (H - 1) * a_head + K && o_stride >= (H - 1) * o_head + N && a_stride % per == 0 && a_head % per == 0 &&
                       (n_partials == 1 || partial_stride % per == 0) && o_stride % 8 == 0 && o_head % 8 == 0 && aligned(a) && aligned(w) &&
                       aligned(out);
    if (!takes) return 1;
    if (a_dtype == FB_F32)
        return launch<float>((const float*)a, (long)a_stride, (long)a_head, n_partials, (long)partial_stride, w, out, (long)o_stride,
                             (long)o_head, n, H, N, K, status, stream);
    if (a_dtype == FB_BF16)
        return launch<__nv_bfloat16>((const __nv_bfloat16*)a, (long)a_stride, (long)a_head, 1, 0, w, out, (long)o_stride, (long)o_head, n, H,
                                     N, K, status, stream);
    return fb_fail(-1, "head_linear: unknown dtype code %d", a_dtype);
}
