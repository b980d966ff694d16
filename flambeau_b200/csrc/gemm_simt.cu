// out[M,N] = A[M,K] * W[N,K]^T with float32 FMA accumulation on the CUDA cores.
//
// This is the matrix product of the true 32-bit path for the shapes that
// gemm_f32_tc.cu does not take (fewer than 64 outputs or 512 inputs, weight
// rows off 16-byte borders) and the fallback of the bfloat16 path for shapes
// the tensor-core kernel refuses.  Each output
// element is summed in one thread in ascending k (even and odd k on their own
// where 16-byte copies fetch the rows), so the result of a row does not depend
// on how many rows the call has.
// Weight layout as in the reference: rows = outputs, columns = inputs
// (crates/kernels-hip/src/kernels/mmq_f16_tile.cu:34-39).
#include "async_copy.cuh"

template <typename TA, typename TW, typename TO, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_kernel(const TA* __restrict__ A, long lda, const TW* __restrict__ W, long ldw,
                 TO* __restrict__ out, long ldo, int M, int N, int K) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = tid; e < BM * BK; e += THREADS) {
            const int row = e / BK, kk = e - row * BK;
            const int m = m0 + row, k = k0 + kk;
            As[kk][row] = (m < M && k < K) ? fb_to_float(A[(size_t)m * lda + k]) : 0.0f;
        }
#pragma unroll
        for (int e = tid; e < BN * BK; e += THREADS) {
            const int row = e / BK, kk = e - row * BK;
            const int n = n0 + row, k = k0 + kk;
            Ws[kk][row] = (n < N && k < K) ? fb_to_float(W[(size_t)n * ldw + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) out[(size_t)m * ldo + n] = fb_from_float<TO>(acc[i][j]);
        }
    }
}

// The same for float32 rows that start on 16-byte borders: A and W tiles of BK along k arrive by 16-byte asynchronous copies
// in STAGES stages as they lie in memory, four k a load.  Thread (ty, tx) of BM / TM x BN / TN holds rows ty TM and following
// and columns tx, tx + BN / TN, ...: neighbouring lanes read one row of A (two cycles of shared memory) and rows of W in
// different banks.  Each output element is summed in one thread, even and odd k on their own (fma.rn.f32x2: half the issue
// slots, the same rate) and in ascending order, whatever the tile: a row's result does not depend on how many rows there are.
// 48 cycles of shared memory stand beside 256 multiply-adds of a warp at 8 x 8 a thread; the two overlap to about 30 TFLOP/s
// of the 74 that the multiply-adds alone would give.  Measured (us, before / here): 301 x 6,144 x 4,096 961 / 571, 301 x 4,096
// x 4,096 903 / 557, 64 x 28,672 x 4,096 954 / 601, 8 x 4,096 x 4,096 188 / 53.
template <int BM, int BN, int BK, int STAGES, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw, float* __restrict__ out, long ldo,
                int M, int N, int K) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    constexpr int COLS = BN / TN, THREADS = (BM / TM) * COLS, LD = BK + 4, STAGE = (BM + BN) * LD;
    extern __shared__ __align__(16) float sh[];
    const int tid = threadIdx.x, tx = tid % COLS, ty = tid / COLS;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int n_steps = (K + BK - 1) / BK;
    auto fetch = [&](int step) {
        if (step < n_steps) {
            float* st = sh + step % STAGES * STAGE;
            const int k0 = step * BK;
            for (int e = tid; e < (BM + BN) * (BK / 4); e += THREADS) {
                const int r = e / (BK / 4), k = 4 * (e - r * (BK / 4));
                const bool in = k0 + k < K && (r < BM ? m0 + r < M : n0 + r - BM < N);      // (K is a multiple of 4)
                float* dst = st + r * LD + k;
                if (in) cp_async16(dst, (r < BM ? A + (size_t)(m0 + r) * lda : W + (size_t)(n0 + r - BM) * ldw) + k0 + k);
                else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        cp_async_commit();
    };
    unsigned long long acc[TM][TN];                    // (sum over even k, sum over odd k)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int step = 0; step < n_steps; ++step) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                               // this step's stage is there; the one before it is free
        fetch(step + STAGES - 1);
        const float* as = sh + step % STAGES * STAGE + ty * TM * LD;
        const float* ws = sh + step % STAGES * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            ulonglong2 a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + i * LD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + j * COLS * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i].x), "l"(w[j].x));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i].y), "l"(w[j].y));
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * COLS;
            float even, odd;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(acc[i][j]));
            if (n < N) out[(size_t)m * ldo + n] = even + odd;
        }
    }
}

template <int BM, int BN, int BK, int STAGES, int TM, int TN>
static int launch_gemm_f32(const float* A, long lda, const float* W, long ldw, float* out, long ldo, int M, int N, int K,
                           cudaStream_t stream) {
    auto kernel = gemm_f32_kernel<BM, BN, BK, STAGES, TM, TN>;
    constexpr int smem = STAGES * (BM + BN) * (BK + 4) * (int)sizeof(float);
    static bool configured[FB_MAX_DEVICES] = {};
    if (smem > 48 * 1024 && fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fb_fail(-2, "gemm_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    fb_launch(kernel, dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3((BM / TM) * (BN / TN)), (size_t)smem, stream, A, lda, W, ldw,
              out, ldo, M, N, K);
    return fb_check_launch("gemm_f32");
}

// The tile whose busiest SM has the least to do: tiles an SM times a tile's size, smaller tiles counted dearer by what their
// extra loads cost.
static int run_gemm_f32(const float* A, long lda, const float* W, long ldw, float* out, long ldo, int M, int N, int K, cudaStream_t stream) {
#define FB_F32(BM, BN, BK, ST, TM, TN) return launch_gemm_f32<BM, BN, BK, ST, TM, TN>(A, lda, W, ldw, out, ldo, M, N, K, stream)
    if (M <= 8) FB_F32(8, 32, 64, 4, 2, 2);
    if (M <= 16) FB_F32(16, 32, 64, 4, 4, 2);
    const long sms = fb_sm_count();
    auto load = [&](int bm, int bn, double dearer) {
        const long tiles = (long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
        return (double)((tiles + sms - 1) / sms) * bm * bn * dearer;
    };
    const double c0 = load(128, 128, 1.0), c1 = load(64, 128, 1.05), c2 = load(64, 64, 1.15), c3 = load(32, 64, 1.4);
    const double best = fmin(fmin(c0, c1), fmin(c2, c3));
    if (c0 == best) FB_F32(128, 128, 16, 3, 8, 8);
    if (c1 == best) FB_F32(64, 128, 16, 4, 8, 8);
    if (c2 == best) FB_F32(64, 64, 16, 4, 8, 4);
    FB_F32(32, 64, 32, 4, 4, 4);
#undef FB_F32
}

template <typename TA, typename TW, typename TO>
static int launch_gemm_simt(const void* A, long lda, const void* W, long ldw, void* out, long ldo, int M, int N,
                            int K, cudaStream_t stream) {
    if (M >= 256 && N >= 128) {
        constexpr int BM = 128, BN = 128, BK = 8, TM = 8, TN = 8;
        dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
        fb_launch((gemm_simt_kernel<TA, TW, TO, BM, BN, BK, TM, TN>), grid, (BM / TM) * (BN / TN), 0, stream, 
            (const TA*)A, lda, (const TW*)W, ldw, (TO*)out, ldo, M, N, K);
    } else if (M > 16) {
        constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
        dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
        fb_launch((gemm_simt_kernel<TA, TW, TO, BM, BN, BK, TM, TN>), grid, (BM / TM) * (BN / TN), 0, stream, 
            (const TA*)A, lda, (const TW*)W, ldw, (TO*)out, ldo, M, N, K);
    } else {
        constexpr int BM = 16, BN = 64, BK = 32, TM = 2, TN = 2;
        dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
        fb_launch((gemm_simt_kernel<TA, TW, TO, BM, BN, BK, TM, TN>), grid, (BM / TM) * (BN / TN), 0, stream, 
            (const TA*)A, lda, (const TW*)W, ldw, (TO*)out, ldo, M, N, K);
    }
    return fb_check_launch("gemm_simt");
}

FB_API int fb_gemm_simt(const void* A, int a_dtype, long long lda, const void* W, int w_dtype, long long ldw,
                        void* out, int o_dtype, long long ldo, int M, int N, int K, cudaStream_t stream) {
    FB_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    FB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm: a row stride is shorter than its row");
    if (M == 0) return 0;
    FB_REQUIRE((N + 15) / 16 <= 2147483647 && (M + 15) / 16 <= 65535, "gemm: too many rows (M=%d)", M);
    if (a_dtype == FB_F32 && w_dtype == FB_F32 && o_dtype == FB_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0 && (M + 7) / 8 <= 65535)
        return run_gemm_f32((const float*)A, (long)lda, (const float*)W, (long)ldw, (float*)out, (long)ldo, M, N, K, stream);
    FB_DISPATCH_DTYPE(a_dtype, TA, FB_DISPATCH_DTYPE(w_dtype, TW, FB_DISPATCH_DTYPE(o_dtype, TO,
        return (launch_gemm_simt<TA, TW, TO>(A, (long)lda, W, (long)ldw, out, (long)ldo, M, N, K, stream)))));
    return 0;
}

// ---------------------------------------------------------------------------
// The grouped form: the rows are cut into tiles of BM, and every tile multiplies with the weights of its own group
// (an expert): W + tile_group[tile] * group_stride.  A tile whose group is negative is skipped.  Row m of A is row
// row_index[m] of the caller's matrix (negative: a row of zeros; nullptr: row m itself), so tokens that were
// sorted by expert need not be copied side by side first.  `act` (an FbPlainAct code) is applied to every output.
// Each output element still sums its K products in ascending k in one thread.
// ---------------------------------------------------------------------------
template <typename TA, typename TW, typename TO, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_grouped_kernel(const TA* __restrict__ A, long lda, const int* __restrict__ row_index,
                         const TW* __restrict__ W, long ldw, long group_stride, const int* __restrict__ tile_group,
                         TO* __restrict__ out, long ldo, int M, int N, int K, int act) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ int src_row[BM];
    const int group = tile_group[blockIdx.y];
    if (group < 0) return;
    const TW* Wg = W + (size_t)group * group_stride;
    const int tid = threadIdx.x;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    for (int r = tid; r < BM; r += THREADS) {
        const int m = m0 + r;
        src_row[r] = m < M ? (row_index ? row_index[m] : m) : -1;
    }
    __syncthreads();
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = tid; e < BM * BK; e += THREADS) {
            const int row = e / BK, kk = e - row * BK;
            const int src = src_row[row], k = k0 + kk;
            As[kk][row] = (src >= 0 && k < K) ? fb_to_float(A[(size_t)src * lda + k]) : 0.0f;
        }
#pragma unroll
        for (int e = tid; e < BN * BK; e += THREADS) {
            const int row = e / BK, kk = e - row * BK;
            const int n = n0 + row, k = k0 + kk;
            Ws[kk][row] = (n < N && k < K) ? fb_to_float(Wg[(size_t)n * ldw + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) out[(size_t)m * ldo + n] = fb_from_float<TO>(fb_plain_act(act, acc[i][j]));
        }
    }
}

// M = rows of the padded order (a multiple of `tile`); tile_group has M / tile entries.  `tile` is 16 or 64.
FB_API int fb_gemm_simt_grouped(const void* A, int a_dtype, long long lda, const int* row_index, const void* W,
                                int w_dtype, long long ldw, long long group_stride, const int* tile_group, int tile,
                                void* out, int o_dtype, long long ldo, int M, int N, int K, int act,
                                cudaStream_t stream) {
    FB_REQUIRE(M >= 0 && N > 0 && K > 0, "grouped gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    FB_REQUIRE(tile == 16 || tile == 64, "grouped gemm: row tiles of 16 or 64, not %d", tile);
    FB_REQUIRE(M % tile == 0 && tile_group, "grouped gemm: the rows must be whole tiles with a group each");
    FB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "grouped gemm: a row stride is shorter than its row");
    FB_REQUIRE(fb_plain_act_known(act), "grouped gemm: unknown activation code %d", act);
    if (M == 0) return 0;
    FB_REQUIRE(M / tile <= 65535, "grouped gemm: too many row tiles (M=%d)", M);
    if (tile == 64) {
        constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
        dim3 grid((N + BN - 1) / BN, M / BM);
        FB_DISPATCH_DTYPE(a_dtype, TA, FB_DISPATCH_DTYPE(w_dtype, TW, FB_DISPATCH_DTYPE(o_dtype, TO,
            (fb_launch((gemm_simt_grouped_kernel<TA, TW, TO, BM, BN, BK, TM, TN>), grid, (BM / TM) * (BN / TN), 0, stream,
                       (const TA*)A, (long)lda, row_index, (const TW*)W, (long)ldw, (long)group_stride, tile_group,
                       (TO*)out, (long)ldo, M, N, K, act)))));
    } else {
        constexpr int BM = 16, BN = 64, BK = 32, TM = 2, TN = 2;
        dim3 grid((N + BN - 1) / BN, M / BM);
        FB_DISPATCH_DTYPE(a_dtype, TA, FB_DISPATCH_DTYPE(w_dtype, TW, FB_DISPATCH_DTYPE(o_dtype, TO,
            (fb_launch((gemm_simt_grouped_kernel<TA, TW, TO, BM, BN, BK, TM, TN>), grid, (BM / TM) * (BN / TN), 0, stream,
                       (const TA*)A, (long)lda, row_index, (const TW*)W, (long)ldw, (long)group_stride, tile_group,
                       (TO*)out, (long)ldo, M, N, K, act)))));
    }
    return fb_check_launch("gemm_simt_grouped");
}
