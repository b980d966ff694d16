// Paged causal (sliding-window) attention in float32 on the CUDA cores, in tiles: the attention of the true 32-bit path for
// head sizes that are multiples of 4 up to 256 (attention_simt.cu takes every other size and the bfloat16 forms).
//
// A CTA of 128 threads owns one key/value head, BM query rows = (BM / G) tokens x the G query heads that share the head, and a
// stretch of the 32-key tiles that its rows see.  K and V tiles come through the block table by 16-byte asynchronous copies, V
// under the scores and the next K under the product.  Thread (ty, tx) of 8 x 16 holds rows ty * BM / 8 and following: their
// scores of keys tx and tx + 16, then their output columns 4 tx + 64 c; so a row's maximum and sum are agreed on by 16 lanes
// and its rescaling needs no memory.  Rows up to 16 (decoded tokens) run with BM 16, others with BM 64, in two launches.
//
// Where that gives too few CTAs the tiles are cut into stretches: every CTA leaves its rows' maximum, sum and unnormalised
// output, and a warp per (row, head) merges them.
//
// What bounds it: multiply-adds over portions (2 x 128 x 128 a row and tile of 32 keys at heads of 128; the scores read 24
// cycles of shared memory for 64 multiply-adds of a warp), the stream of keys and values for decoded tokens.  301 tokens
// behind 500 (32 heads of 128 on 8): 3,340 us with a warp a (row, head), about 140 here.
//
// Sums run in float32 throughout; sinks, caps, gates, slopes and kept first keys as in attention_simt.cu.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int THREADS = 128;
constexpr int KEYS = 32;                // keys of a tile
constexpr int MAX_SPLITS = 32;

struct F32Args {
    const float* q; long q_stride;
    float* out; long out_stride;
    const float* k_pool; const float* v_pool;
    int page_size, n_pages;
    const int* block_table; int table_stride; const int* table_base; int table_head;
    const int* seq_q_start; const int* seq_q_len; const int* seq_pos_start;
    int n_seqs, n, nh, nkv, hd, vd, window, keep_first;
    float scale, softcap;
    const float* score_slopes; const float* sinks;
    const float* head_gate; long gate_stride; int gate_partials; long gate_partial_stride;
    int token_tiles;                    // CTAs that the tokens of a (sequence, key/value head) are laid over
    int short_rows;                     // sequences with at most this many rows (tokens x G) run with BM 16
    int n_splits;
    float* part_o; float* part_ml;      // [split][row][head] x vd, and x (maximum, sum)
    int* status;
};

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

template <int BM, int VDP>
__global__ void __launch_bounds__(THREADS, VDP <= 128 ? 3 : 1)
attention_f32_kernel(const F32Args a) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    constexpr int RPT = BM / 8, NC = VDP / 64;                   // rows and groups of four columns a thread
    extern __shared__ __align__(16) float sh[];
    const int G = a.nh / a.nkv, hd = a.hd, vd = a.vd;
    const int pair = blockIdx.x / a.token_tiles, tile = blockIdx.x - pair * a.token_tiles;
    const int seq = pair / a.nkv, kvh = pair - seq * a.nkv;
    const int q_len = a.seq_q_len[seq];
    if ((q_len * G <= a.short_rows) != (BM == 16)) return;
    const int TQ = BM / G;
    const int tok0 = (a.token_tiles - 1 - tile) * TQ;      // later tokens see more keys: start them first
    if (tok0 >= q_len) return;
    const int ntok = min(TQ, q_len - tok0), rows = ntok * G;
    const int q_start = a.seq_q_start[seq] + tok0, pos0 = a.seq_pos_start[seq] + tok0;

    const int LQ = hd + 4;                                       // row stride of Q and K
    float* Qs = sh;                                              // [BM][LQ]
    float* Ks = Qs + BM * LQ;                                    // [KEYS][LQ]
    float* Vs = Ks + KEYS * LQ;                                  // [KEYS][VDP]
    float* Ps = Vs + KEYS * VDP;                                 // [KEYS][BM + 4]: the weights, key by key
    int* has_page = reinterpret_cast<int*>(Ps + KEYS * (BM + 4));      // [2][KEYS]

    // ---- the tiles: those that hold kept first keys and lie before the window's first, then the window's ----
    const int t_hi = pos0 + ntok - 1, t_lo = fb_first_key(pos0, a.window, 0);
    const int keep = a.window > 0 ? a.keep_first : 0;
    const int tile_lo = t_lo / KEYS * KEYS, head_tiles = min((keep + KEYS - 1) / KEYS, t_lo / KEYS);
    const int n_tiles = head_tiles + (t_hi - tile_lo) / KEYS + 1;
    const int per = (n_tiles + a.n_splits - 1) / a.n_splits;
    const int first_tile = blockIdx.z * per, last_tile = min(first_tile + per, n_tiles) - 1;
    auto tile_start = [&](int i) { return i < head_tiles ? i * KEYS : tile_lo + (i - head_tiles) * KEYS; };

    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int* table = a.block_table + (size_t)seq * a.table_stride;
    const int base_page = a.table_base ? a.table_base[seq] : 0;

    // four threads fetch a key's row; the page of its key in tile i: -2 where no query sees the key, -1 where there is none
    const int fr = tid >> 2, fs = tid & 3;
    auto lookup = [&](int i) -> int {
        if (i > last_tile) return -2;
        const int t = tile_start(i) + fr;
        if (t > t_hi || (t < t_lo && t >= keep)) return -2;
        const int e = fb_table_column(t / a.page_size, base_page, a.table_head);
        const int page = (e >= 0 && e < a.table_stride) ? table[e] : -1;
        return (page < 0 || page >= a.n_pages) ? -1 : page;
    };
    auto fetch = [&](const float* pool, int i, int page, int width, float* dst_row) {
        const int t = tile_start(i) + fr;
        if (page >= 0) {
            const float* src = pool + (((size_t)page * a.nkv + kvh) * a.page_size + t % a.page_size) * width;
            for (int c = 4 * fs; c < width; c += 16) copy16(dst_row + c, src + c);
        } else {
            for (int c = 4 * fs; c < width; c += 16) *reinterpret_cast<float4*>(dst_row + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto fetch_k = [&](int i, int page) {
        if (fs == 0) {
            has_page[(i & 1) * KEYS + fr] = page >= 0;
            if (page == -1) atomicOr(a.status, FB_STATUS_BAD_PAGE);
        }
        fetch(a.k_pool, i, page, hd, Ks + fr * LQ);
    };

    int page = lookup(first_tile), next_page = lookup(first_tile + 1);
    if (first_tile <= last_tile) fetch_k(first_tile, page);
    copies_commit();
    for (int e = tid; e < BM * (hd / 4); e += THREADS) {         // Q, zeros beyond the CTA's rows
        const int r = e / (hd / 4), c = 4 * (e - r * (hd / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) v = *reinterpret_cast<const float4*>(a.q + (size_t)(q_start + r / G) * a.q_stride + (size_t)(kvh * G + r % G) * hd + c);
        *reinterpret_cast<float4*>(Qs + r * LQ + c) = v;
    }
    if (vd < VDP)                                                // columns that no value fills
        for (int e = tid; e < KEYS * (VDP - vd); e += THREADS) Vs[e / (VDP - vd) * VDP + vd + e % (VDP - vd)] = 0.0f;

    int p_row[RPT], t0_row[RPT];
    float slope[RPT], m[RPT], l[RPT], o[RPT][4 * NC];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = ty * RPT + i;
        p_row[i] = r < rows ? pos0 + r / G : -1;
        t0_row[i] = r < rows ? fb_first_key(p_row[i], a.window, 0) : 0;
        slope[i] = a.score_slopes && r < rows ? a.score_slopes[kvh * G + r % G] : 0.0f;
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < 4 * NC; ++c) o[i][c] = 0.0f;
    }

    for (int it = first_tile; it <= last_tile; ++it) {
        fetch(a.v_pool, it, page, vd, Vs + fr * VDP);
        copies_commit();
        const int page2 = lookup(it + 2);
        copies_wait<1>();
        __syncthreads();                                         // K (and, the first time, Q) is there
        float s[RPT][2];
#pragma unroll
        for (int i = 0; i < RPT; ++i) s[i][0] = s[i][1] = 0.0f;
        const float* k0 = Ks + tx * LQ;
        const float* k1 = k0 + 16 * LQ;
        const float* qr = Qs + ty * RPT * LQ;
#pragma unroll 2
        for (int d = 0; d < hd; d += 4) {
            const float4 x = *reinterpret_cast<const float4*>(k0 + d), y = *reinterpret_cast<const float4*>(k1 + d);
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const float4 z = *reinterpret_cast<const float4*>(qr + i * LQ + d);
                s[i][0] = fmaf(z.x, x.x, s[i][0]); s[i][1] = fmaf(z.x, y.x, s[i][1]);
                s[i][0] = fmaf(z.y, x.y, s[i][0]); s[i][1] = fmaf(z.y, y.y, s[i][1]);
                s[i][0] = fmaf(z.z, x.z, s[i][0]); s[i][1] = fmaf(z.z, y.z, s[i][1]);
                s[i][0] = fmaf(z.w, x.w, s[i][0]); s[i][1] = fmaf(z.w, y.w, s[i][1]);
            }
        }
        const int t0 = tile_start(it) + tx, t1 = t0 + 16;
        const bool there0 = has_page[(it & 1) * KEYS + tx], there1 = has_page[(it & 1) * KEYS + tx + 16];
        float p[RPT][2];
        bool see[RPT][2];
        bool whole_tile = there0 && there1;                      // every row of this warp sees every key of the tile
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            whole_tile = whole_tile && (ty * RPT + i >= rows || (tile_start(it) + KEYS - 1 <= p_row[i] && tile_start(it) >= t0_row[i]));
            float x = s[i][0] * a.scale, y = s[i][1] * a.scale;
            if (a.softcap > 0.0f) {
                x = a.softcap * tanhf(x / a.softcap);
                y = a.softcap * tanhf(y / a.softcap);
            }
            x += slope[i] * (float)(t0 - p_row[i]);
            y += slope[i] * (float)(t1 - p_row[i]);
            see[i][0] = there0 && t0 <= p_row[i] && (t0 >= t0_row[i] || t0 < keep);
            see[i][1] = there1 && t1 <= p_row[i] && (t1 >= t0_row[i] || t1 < keep);
            x = see[i][0] ? x : -INFINITY;
            y = see[i][1] ? y : -INFINITY;
            float top = fmaxf(x, y);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float m_new = fmaxf(m[i], top), m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_use);
            p[i][0] = see[i][0] ? expf(x - m_use) : 0.0f;
            p[i][1] = see[i][1] ? expf(y - m_use) : 0.0f;
            l[i] = l[i] * corr + (p[i][0] + p[i][1]);            // (this lane's keys; the lanes' sums meet at the end)
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * NC; ++c) o[i][c] *= corr;
        }
        whole_tile = __all_sync(0xffffffffu, whole_tile);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            Ps[tx * (BM + 4) + ty * RPT + i] = see[i][0] ? p[i][0] : -1.0f;     // (below zero: a key that the row does not see)
            Ps[(tx + 16) * (BM + 4) + ty * RPT + i] = see[i][1] ? p[i][1] : -1.0f;
        }
        __syncthreads();                                         // the weights are there, K is free
        if (it < last_tile) fetch_k(it + 1, next_page);
        copies_commit();
        copies_wait<1>();
        __syncthreads();                                         // V is there
        const float* pr = Ps + ty * RPT;
        const float* vr = Vs + 4 * tx;
        auto weigh = [&](auto whole_, int k) {
            constexpr bool whole = decltype(whole_)::value;
            float w[RPT];
#pragma unroll
            for (int i = 0; i < RPT; i += (RPT % 4 == 0 ? 4 : 2)) {
                if constexpr (RPT % 4 == 0) {
                    const float4 x = *reinterpret_cast<const float4*>(pr + k * (BM + 4) + i);
                    w[i] = x.x; w[i + 1] = x.y; w[i + 2] = x.z; w[i + 3] = x.w;
                } else {
                    const float2 x = *reinterpret_cast<const float2*>(pr + k * (BM + 4) + i);
                    w[i] = x.x; w[i + 1] = x.y;
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(vr + k * VDP + 64 * c);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    if (!whole && w[i] < 0.0f) continue;         // (what a row does not see must not reach it as 0 * NaN; what it
                                                                 // sees does, also with a weight that has become 0)
                    o[i][4 * c] = fmaf(w[i], v.x, o[i][4 * c]);
                    o[i][4 * c + 1] = fmaf(w[i], v.y, o[i][4 * c + 1]);
                    o[i][4 * c + 2] = fmaf(w[i], v.z, o[i][4 * c + 2]);
                    o[i][4 * c + 3] = fmaf(w[i], v.w, o[i][4 * c + 3]);
                }
            }
        };
        if (whole_tile)
#pragma unroll 2
            for (int k = 0; k < KEYS; ++k) weigh(std::true_type(), k);
        else
#pragma unroll 1
            for (int k = 0; k < KEYS; ++k) weigh(std::false_type(), k);
        page = next_page;
        next_page = page2;
        __syncthreads();                                         // V and the weights are free
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
        const int r = ty * RPT + i;
        if (r >= rows) continue;
        const int row = q_start + r / G, head = kvh * G + r % G;
        if (a.n_splits > 1) {
            const size_t at = ((size_t)blockIdx.z * a.n + row) * a.nh + head;
            if (tx == 0) {
                a.part_ml[2 * at] = m[i];
                a.part_ml[2 * at + 1] = l[i];
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (4 * tx + 64 * c < vd)
                    *reinterpret_cast<float4*>(a.part_o + at * vd + 4 * tx + 64 * c) = make_float4(o[i][4 * c], o[i][4 * c + 1], o[i][4 * c + 2], o[i][4 * c + 3]);
            continue;
        }
        float f = 1.0f, sum = l[i];
        if (a.sinks) {                                           // the slot without key and value
            const float sk = a.sinks[head], m_new = fmaxf(m[i], sk);
            f = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_new);
            sum = sum * f + expf(sk - m_new);
        }
        f = sum > 0.0f ? f / sum : 0.0f;
        if (a.head_gate)
            f /= 1.0f + expf(-fb_slab_sum(a.head_gate + (size_t)row * a.gate_stride, head, a.gate_partials, a.gate_partial_stride));
        float* op = a.out + (size_t)row * a.out_stride + (size_t)head * vd;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (4 * tx + 64 * c < vd)
                *reinterpret_cast<float4*>(op + 4 * tx + 64 * c) = make_float4(o[i][4 * c] * f, o[i][4 * c + 1] * f, o[i][4 * c + 2] * f, o[i][4 * c + 3] * f);
    }
}

// One warp a (row, head): the stretches' results made one.
__global__ void __launch_bounds__(128)
attention_f32_merge_kernel(const F32Args a) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const long item = (long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (item >= (long)a.n * a.nh) return;
    const int lane = threadIdx.x & 31, row = (int)(item / a.nh), head = (int)(item - (long)row * a.nh);
    const size_t stride = (size_t)a.n * a.nh;
    float ms = -INFINITY, ls = 0.0f;                             // stretch `lane`
    if (lane < a.n_splits) {
        ms = a.part_ml[2 * (item + lane * stride)];
        ls = a.part_ml[2 * (item + lane * stride) + 1];
    }
    float top = fb_warp_max(ms);
    if (a.sinks) top = fmaxf(top, a.sinks[head]);
    const float w = ms == -INFINITY ? 0.0f : expf(ms - top);
    float sum = fb_warp_sum(w * ls);
    if (a.sinks) sum += expf(a.sinks[head] - top);
    float f = sum > 0.0f ? 1.0f / sum : 0.0f;
    if (a.head_gate)
        f /= 1.0f + expf(-fb_slab_sum(a.head_gate + (size_t)row * a.gate_stride, head, a.gate_partials, a.gate_partial_stride));
    float* op = a.out + (size_t)row * a.out_stride + (size_t)head * a.vd;
    for (int d = lane; d < (a.vd + 31) / 32 * 32; d += 32) {
        float acc = 0.0f;
        for (int s = 0; s < a.n_splits; ++s) {
            const float ws = __shfl_sync(0xffffffffu, w, s);
            if (d < a.vd && ws > 0.0f) acc = fmaf(ws, a.part_o[(item + s * stride) * a.vd + d], acc);
        }
        if (d < a.vd) op[d] = acc * f;
    }
}

size_t smem_bytes(int bm, int hd, int vdp) {
    return ((size_t)(bm + KEYS) * (hd + 4) + (size_t)KEYS * vdp + (size_t)KEYS * (bm + 4) + 2 * KEYS) * sizeof(float);
}

template <int BM, int VDP>
int launch(F32Args a, int max_q_len, cudaStream_t stream) {
    auto kern = attention_f32_kernel<BM, VDP>;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        const int most = (int)smem_bytes(BM, 256, VDP);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return fb_fail(-2, "attention_f32: cannot reserve %d bytes of shared memory: %s", most, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    const int TQ = BM / (a.nh / a.nkv);
    const int longest = BM == 16 ? min(max_q_len, TQ) : max_q_len;     // (a sequence with BM 16 is one tile)
    a.token_tiles = (longest + TQ - 1) / TQ;
    fb_launch(kern, dim3((unsigned)((long)a.token_tiles * a.n_seqs * a.nkv), 1, a.n_splits), dim3(THREADS), smem_bytes(BM, a.hd, VDP), stream, a);
    return fb_check_launch("attention_f32");
}

template <int BM>
int launch(const F32Args& a, int max_q_len, cudaStream_t stream) {
    if (a.vd <= 64) return launch<BM, 64>(a, max_q_len, stream);
    if (a.vd <= 128) return launch<BM, 128>(a, max_q_len, stream);
    return launch<BM, 256>(a, max_q_len, stream);
}

}  // namespace

// Into how many stretches the tiles of a step are cut: as many as make four CTAs a multiprocessor, at least two tiles each,
// at most 32.  (One CTA a multiprocessor leaves its four warps waiting on each other's loads, and CTAs that start while the
// kernel ahead still runs then share the SMs that are free first: 301 tokens behind 500 took 560 us so.)
FB_API int fb_attention_f32_splits(int n_seqs, int nkv, int G, int max_q_len, int max_keys) {
    const long rows = (long)max_q_len * G;
    const long ctas = (long)n_seqs * nkv * (rows <= 16 ? 1 : (max_q_len + 64 / G - 1) / (64 / G));
    long s = ctas > 0 ? 4L * fb_sm_count() / ctas : 1;
    const long most = max_keys / (2 * KEYS);
    if (s > most) s = most;
    if (s > MAX_SPLITS) s = MAX_SPLITS;
    return s < 1 ? 1 : (int)s;
}

// q, out: float32 [rows, nh * hd] / [rows, nh * vd]; pools float32.  part: n_splits * n * nh * (vd + 2) floats (n_splits > 1).
FB_API int fb_paged_attention_f32(const float* q, long long q_stride, float* out, long long out_stride, const float* k_pool,
                                  const float* v_pool, int page_size, int n_pages, const int* block_table, int table_stride,
                                  const int* table_base, int table_head, const int* seq_q_start, const int* seq_q_len,
                                  const int* seq_pos_start, int n_seqs, int max_q_len, int any_short, int any_long, int n, int nh,
                                  int nkv, int hd, int vd, int window, int keep_first, float scale, float softcap,
                                  const float* score_slopes, const float* sinks, const float* head_gate, long long gate_stride,
                                  int gate_partials, long long gate_partial_stride, int n_splits, float* part,
                                  long long part_floats, int* status, cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && n_seqs >= 0 && nh > 0 && nkv > 0 && nh % nkv == 0, "attention_f32: bad head counts");
    FB_REQUIRE(hd % 4 == 0 && hd >= 4 && hd <= 256 && vd % 4 == 0 && vd >= 4 && vd <= 256 && nh / nkv <= 64,
               "attention_f32: sizes (key %d, value %d) are multiples of 4 up to 256, up to 64 heads a key/value head", hd, vd);
    FB_REQUIRE(q_stride % 4 == 0 && out_stride % 4 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)out % 16 == 0 &&
               (uintptr_t)k_pool % 16 == 0 && (uintptr_t)v_pool % 16 == 0, "attention_f32: unaligned operands");
    FB_REQUIRE(page_size > 0 && n_pages > 0 && window >= 0 && keep_first >= 0, "attention_f32: bad cache geometry");
    FB_REQUIRE(softcap >= 0.0f && (!head_gate || gate_stride >= nh), "attention_f32: bad cap or gate");
    FB_REQUIRE((long long)n_seqs * nkv * max_q_len < (1LL << 31), "attention_f32: too many sequences and tokens for one grid");
    if (n == 0 || n_seqs == 0) return 0;
    if (n_splits < 1) n_splits = 1;
    if (n_splits > MAX_SPLITS) n_splits = MAX_SPLITS;
    const long long items = (long long)n * nh;
    FB_REQUIRE(n_splits == 1 || (part && part_floats >= n_splits * items * (vd + 2)), "attention_f32: too little scratch");
    F32Args a;
    a.q = q; a.q_stride = (long)q_stride; a.out = out; a.out_stride = (long)out_stride;
    a.k_pool = k_pool; a.v_pool = v_pool; a.page_size = page_size; a.n_pages = n_pages;
    a.block_table = block_table; a.table_stride = table_stride; a.table_base = table_base;
    a.table_head = table_head > 0 ? table_head : 0;
    a.seq_q_start = seq_q_start; a.seq_q_len = seq_q_len; a.seq_pos_start = seq_pos_start;
    a.n_seqs = n_seqs; a.n = n; a.nh = nh; a.nkv = nkv; a.hd = hd; a.vd = vd; a.window = window; a.keep_first = keep_first;
    a.scale = scale; a.softcap = softcap; a.score_slopes = score_slopes; a.sinks = sinks;
    a.head_gate = head_gate; a.gate_stride = (long)gate_stride;
    a.gate_partials = gate_partials < 1 ? 1 : gate_partials; a.gate_partial_stride = (long)gate_partial_stride;
    a.short_rows = nh / nkv <= 16 ? 16 : 0;                      // (a token of more than 16 heads takes BM 64)
    a.n_splits = n_splits;
    a.part_o = part; a.part_ml = part ? part + n_splits * items * vd : nullptr;
    a.status = status;
    if (any_long) {
        const int rc = launch<64>(a, max_q_len, stream);
        if (rc) return rc;
    }
    if (any_short && a.short_rows > 0) {
        const int rc = launch<16>(a, max_q_len, stream);
        if (rc) return rc;
    }
    if (n_splits > 1) {
        fb_launch(attention_f32_merge_kernel, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, a);
        return fb_check_launch("attention_f32_merge");
    }
    return 0;
}
