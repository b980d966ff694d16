// Paged causal (sliding-window) attention in float32 on the CUDA cores, in tiles: the attention of the true 32-bit path for
// head sizes that are multiples of 4 up to 256 (attention_f32_tc.cu takes heads of 128 without caps, slopes and kept first keys,
// attention_simt.cu every other size and the bfloat16 forms).
//
// A CTA of 128 threads owns one key/value head, BM query rows = (BM / G) tokens x the G query heads that share the head, and
// some of the 32-key tiles that its rows see.  K and V tiles come through the block table by 16-byte asynchronous copies, V
// under the scores and the next K under the product.  Thread (ty, tx) of 8 x 16 holds rows ty * BM / 8 and following: their
// scores of keys tx and tx + 16, then their output columns 4 tx + 64 c; so a row's maximum and sum are agreed on by 16 lanes
// and its rescaling needs no memory.  Rows up to 16 (decoded tokens) run with BM 16, others with BM 64, in two launches.
//
// A row's bits depend on its position and its keys alone, not on the rows that share its step, on how its prompt was cut, or on
// how the work was laid over CTAs: tiles begin at multiples of 32 positions, stretches of tiles at multiples of 256, a stretch
// is summed on its own, and the stretches are joined in their order by one rule (join).  A CTA that takes all stretches of its
// rows joins them in its output rows; where that gives too few CTAs each takes some, leaves every stretch's maximum, sum and
// unnormalised output, and a warp per row joins them.
//
// What bounds it: multiply-adds over portions (2 x 32 x 128 a row and tile of 32 keys at heads of 128; the scores read 24
// cycles of shared memory for 64 multiply-adds of a warp), the stream of keys and values for decoded tokens.  301 tokens
// behind 500 (32 heads of 128 on 8), launched behind itself: 3,330 us with a warp a (row, head), 195 here; 8 decoded tokens
// of 8,000 keys 7,700 and 312.  (Stretches cut by the step's rows took 192 and 215: the latter in one round of CTAs.)
//
// Sums run in float32 throughout; sinks, caps, gates, slopes and kept first keys as in attention_simt.cu.
#include <type_traits>

#include "attention_f32.cuh"

namespace {

constexpr int THREADS = 128;
constexpr int KEYS = 32;                // keys of a tile
constexpr int TPS = STRETCH / KEYS;

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

template <int BM, int VDP>
__global__ void __launch_bounds__(THREADS, VDP == 64 ? 3 : VDP == 128 ? 2 : 1)
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
    float* run = Ps + KEYS * (BM + 4);                           // [2][2][BM]: maxima and sums of the stretches joined so far,
                                                                 // read from one half and left in the other
    int* has_page = reinterpret_cast<int*>(run + 4 * BM);        // [2][KEYS]

    // ---- the tiles: those that hold kept first keys and lie before the window's first, then the window's ----
    const int t_hi = pos0 + ntok - 1, t_lo = fb_first_key(pos0, a.window, 0);
    const int keep = a.window > 0 ? a.keep_first : 0;
    const int tile_lo = t_lo / KEYS * KEYS, head_tiles = min((keep + KEYS - 1) / KEYS, t_lo / KEYS);
    const int n_tiles = head_tiles + (t_hi - tile_lo) / KEYS + 1;
    // ---- its stretches, numbered from the first that holds a tile ----
    const int head_last = (head_tiles - 1) / TPS, window_first = tile_lo / STRETCH;
    const int shift = (head_tiles > 0 ? head_last + (window_first > head_last) : 0) - window_first;
    auto tile_of = [&](int s) {                                  // the first tile of stretch s
        if (s >= a.slots) return n_tiles;
        if (head_tiles > 0 && s <= head_last) return s * TPS;
        return min(n_tiles, head_tiles + max(0, (s - shift) * TPS - tile_lo / KEYS));
    };
    const int slot_end = min((int)(blockIdx.z + 1) * a.per, a.slots);
    int slot = blockIdx.z * a.per, stretch_end = tile_of(slot + 1);
    const int first_tile = tile_of(slot), last_tile = tile_of(slot_end) - 1;
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
            const bool see0 = there0 && t0 <= p_row[i] && (t0 >= t0_row[i] || t0 < keep);
            const bool see1 = there1 && t1 <= p_row[i] && (t1 >= t0_row[i] || t1 < keep);
            x = see0 ? x : -INFINITY;
            y = see1 ? y : -INFINITY;
            float top = fmaxf(x, y);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float m_new = fmaxf(m[i], top), m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_use);
            const float px = see0 ? expf(x - m_use) : 0.0f, py = see1 ? expf(y - m_use) : 0.0f;
            l[i] = l[i] * corr + (px + py);                      // (this lane's keys; the lanes' sums meet at the end)
            p[i][0] = see0 ? px : -1.0f;                         // (below zero: a key that the row does not see)
            p[i][1] = see1 ? py : -1.0f;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * NC; ++c) o[i][c] *= corr;
        }
        whole_tile = __all_sync(0xffffffffu, whole_tile);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            Ps[tx * (BM + 4) + ty * RPT + i] = p[i][0];
            Ps[(tx + 16) * (BM + 4) + ty * RPT + i] = p[i][1];
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
        if (it + 1 == stretch_end || it == last_tile) {          // the stretch is complete
            const bool first = slot == 0;
            const float* run_in = run + (slot & 1) * 2 * BM;
            float* run_out = run + (~slot & 1) * 2 * BM;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
                const int r = ty * RPT + i;
                if (r >= rows) continue;
                const int row = q_start + r / G, head = kvh * G + r % G;
                if (a.part_o) {
                    const size_t at = part_at<BM>(a, slot, pair, row, head, r);
                    if (tx == 0) *reinterpret_cast<float2*>(a.part_ml + 2 * at) = make_float2(m[i], l[i]);
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (4 * tx + 64 * c < vd)
                            *reinterpret_cast<float4*>(a.part_o + at * vd + 4 * tx + 64 * c) = make_float4(o[i][4 * c], o[i][4 * c + 1], o[i][4 * c + 2], o[i][4 * c + 3]);
                    continue;
                }
                float M = first ? -INFINITY : run_in[r], L = first ? 0.0f : run_in[BM + r];
                const Join j = join(M, L, m[i], l[i]);
                const float f = it == last_tile ? finish(a, row, head, M, L) : 1.0f;
                if (tx == 0) {
                    run_out[r] = M;
                    run_out[BM + r] = L;
                }
                float* op = a.out + (size_t)row * a.out_stride + (size_t)head * vd + 4 * tx;     // (read by the thread that wrote it)
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (4 * tx + 64 * c < vd) {
                        const float4 b = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(op + 64 * c);
                        *reinterpret_cast<float4*>(op + 64 * c) = make_float4(joined(j, b.x, o[i][4 * c]) * f, joined(j, b.y, o[i][4 * c + 1]) * f,
                                                                              joined(j, b.z, o[i][4 * c + 2]) * f, joined(j, b.w, o[i][4 * c + 3]) * f);
                    }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                m[i] = -INFINITY;
                l[i] = 0.0f;
#pragma unroll
                for (int c = 0; c < 4 * NC; ++c) o[i][c] = 0.0f;
            }
            stretch_end = tile_of(++slot + 1);
        }
        __syncthreads();                                         // V and the weights are free
    }
    if (a.part_o && tx == 0)                                     // stretches that these rows do not have
        for (; slot < slot_end; ++slot)
            for (int r = ty * RPT; r < min((ty + 1) * RPT, rows); ++r)
                *reinterpret_cast<float2*>(a.part_ml + 2 * part_at<BM>(a, slot, pair, q_start + r / G, kvh * G + r % G, r)) = make_float2(-INFINITY, 0.0f);
}

size_t smem_bytes(int bm, int hd, int vdp) {
    return ((size_t)(bm + KEYS) * (hd + 4) + (size_t)KEYS * vdp + (size_t)KEYS * (bm + 4) + 4 * bm + 2 * KEYS) * sizeof(float);
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
    const unsigned ctas = (unsigned)((long)a.token_tiles * a.n_seqs * a.nkv);
    fb_launch(kern, dim3(ctas, 1, (a.slots + a.per - 1) / a.per), dim3(THREADS), smem_bytes(BM, a.hd, VDP), stream, a);
    const int rc = fb_check_launch("attention_f32");
    if (rc || !a.part_o) return rc;
    fb_launch((attention_f32_join_kernel<BM>), dim3(ctas, BM / 4), dim3(128), 0, stream, a);
    return fb_check_launch("attention_f32_join");
}

template <int BM>
int launch(const F32Args& a, int max_q_len, cudaStream_t stream) {
    if (a.vd <= 64) return launch<BM, 64>(a, max_q_len, stream);
    if (a.vd <= 128) return launch<BM, 128>(a, max_q_len, stream);
    return launch<BM, 256>(a, max_q_len, stream);
}

// How a step's stretches are laid over CTAs.
struct Plan {
    int slots, per_short, per_long;     // stretches of a row at most; those a CTA takes, with BM 16 and BM 64
    long long short_floats, long_floats;                         // scratch (0: every CTA takes all stretches)
};

// short_tiles, long_tiles: CTAs a key/value head of the sequences that run with BM 16 and BM 64.  Stretches are spread until
// there are about four CTAs a multiprocessor.  (One leaves its four warps waiting on each other's loads, and CTAs that start
// while the kernel ahead still runs then share the SMs that are free first: 301 tokens behind 500 took 560 us so.)  A row's
// stretches: those of its window's keys, which begin anywhere in one and end anywhere in another, and of the kept first keys.
Plan plan_of(int n_seqs, int n, int nh, int nkv, int vd, int max_q_len, int max_kv_len, int window, int keep_first, long long short_tiles,
             long long long_tiles) {
    Plan p = {};
    long long slots = (max_kv_len + STRETCH - 1) / STRETCH;
    if (window > 0) {
        const long long most = (keep_first + (long long)STRETCH - 1) / STRETCH + (window + 62LL) / STRETCH + 2;
        if (most < slots) slots = most;
    }
    p.slots = (int)(slots < 1 ? 1 : slots);
    const int G = nh / nkv;
    auto spread = [&](long long ctas, long long floats_a_slot, int& per, long long& floats) {
        per = p.slots;
        floats = 0;
        if (ctas <= 0 || p.slots == 1) return;
        const long long want = 4LL * fb_sm_count(), each = (p.slots * ctas + want / 2) / want;
        if (each >= p.slots || p.slots * floats_a_slot > SCRATCH_FLOATS) return;
        per = each < 1 ? 1 : (int)each;
        floats = p.slots * floats_a_slot;                        // (slots x rows x (vd + 2))
    };
    spread(short_tiles * nkv, (long long)n_seqs * nkv * (max_q_len == 1 ? G : 16) * (vd + 2), p.per_short, p.short_floats);
    spread(long_tiles * nkv, (long long)n * nh * (vd + 2), p.per_long, p.long_floats);
    return p;
}

}  // namespace

// Floats of scratch that fb_paged_attention_f32 wants for the same numbers.
FB_API long long fb_attention_f32_scratch_floats(int n_seqs, int n, int nh, int nkv, int vd, int max_q_len, int max_kv_len, int window,
                                                 int keep_first, long long short_tiles, long long long_tiles) {
    if (n_seqs <= 0 || n <= 0 || nkv <= 0 || nh % nkv != 0) return 0;
    const Plan p = plan_of(n_seqs, n, nh, nkv, vd, max_q_len, max_kv_len, window, keep_first, short_tiles, long_tiles);
    return p.short_floats + border4(p.long_floats);
}

// q, out: float32 [rows, nh * hd] / [rows, nh * vd]; pools float32.  short_tiles: sequences with at most 16 rows (tokens x query
// heads a key/value head; none where that is more than 16 heads); long_tiles: over the others, 64-row tiles of their tokens.
FB_API int fb_paged_attention_f32(const float* q, long long q_stride, float* out, long long out_stride, const float* k_pool,
                                  const float* v_pool, int page_size, int n_pages, const int* block_table, int table_stride,
                                  const int* table_base, int table_head, const int* seq_q_start, const int* seq_q_len,
                                  const int* seq_pos_start, int n_seqs, int max_q_len, int max_kv_len, long long short_tiles,
                                  long long long_tiles, int n, int nh, int nkv, int hd, int vd, int window, int keep_first, float scale,
                                  float softcap, const float* score_slopes, const float* sinks, const float* head_gate,
                                  long long gate_stride, int gate_partials, long long gate_partial_stride, float* part,
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
    const Plan p = plan_of(n_seqs, n, nh, nkv, vd, max_q_len, max_kv_len, window, keep_first, short_tiles, long_tiles);
    const long long wanted = p.short_floats + border4(p.long_floats);
    FB_REQUIRE(wanted == 0 || (part && (uintptr_t)part % 16 == 0 && part_floats >= wanted),
               "attention_f32: too little scratch");
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
    a.slots = p.slots;
    a.part_rows = max_q_len == 1 ? nh / nkv : 16;
    a.status = status;
    auto parts = [&](float* at, long long floats, int per) {     // (outputs first: they are read four at a time)
        a.per = per;
        a.part_o = floats ? at : nullptr;
        a.part_ml = floats ? at + floats / (vd + 2) * vd : nullptr;
    };
    if (long_tiles > 0) {
        parts(part, p.long_floats, p.per_long);
        const int rc = launch<64>(a, max_q_len, stream);
        if (rc) return rc;
    }
    if (short_tiles > 0 && a.short_rows > 0) {
        parts(part + border4(p.long_floats), p.short_floats, p.per_short);
        return launch<16>(a, max_q_len, stream);
    }
    return 0;
}
