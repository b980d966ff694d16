// Paged causal (sliding-window) attention in float32 on the 5th-generation tensor cores, for heads of 128: float32 numbers as
// three bfloat16 each and six products, as in gemm_f32_tc.cu (exactness and the sums' precision are described there).
// attention_f32.cu keeps other sizes, caps, slopes and kept first keys; which of the two computes a row depends on the model's
// sizes and options alone, never on the rows of a step.
//
// A CTA owns one key/value head, 128 query rows (128 / G tokens x the G query heads that share the head) and some of the
// stretches of 256 keys that its rows see, in tiles of 64 keys.  Tiles and stretches begin at multiples of 64 and 256
// positions, a stretch is summed on its own and the stretches are joined in their order (attention_f32.cuh), so a row's bits
// depend on its position and its keys alone.
//
// Decoded tokens are the same work on few of the 128 rows: there five of the softmax warps bring keys and values as well.
//
// Warps: 0..7 softmax, a row's 64 scores and 128 outputs by two threads; 8..10 keys and values, copied from their pages into a
// stage while the tile before is split into parts in shared memory (K-major for the scores, MN-major for the product: the same
// bytes); 11 MMA.  Per tile: S = Q K^T into two accumulators (large products, small products), weights split into parts in tensor
// memory, O = P V of the tile alone into two accumulators, added to float32 registers by the softmax threads with the rescaling
// that the tile's maximum asks for: nothing is summed in tensor memory over more than 128 channels or 64 keys.
//
// Numbers from 1e18 on, infinities and NaN, whose parts or products may overflow: a tile that holds one, or a row whose query
// does, is computed by the row's threads in float32 multiply-adds, key by key, and what a row does not see does not reach it.
// Values are multiplied by 2^48 on their way into parts and their products by 2^-48 on the way out, so that every part of every
// float32 (subnormal ones too) is a normal bfloat16; what queries, keys and weights lose below bfloat16's range changes a score
// by less than 1e-20.
//
// What bounds it: shared memory, 4,900 cycles a tile (72 MMAs' operands 3,070, the stage and the parts written and read 1,800);
// decoded tokens take 4,800 a tile, full rows 6,700, the three warps that split being the longest chain there.  What a loop runs
// has to fit the instruction cache: with the split expanded twice, and again for the helping warps, decoding took twice as long.
// 301 tokens behind 500 (32 heads of 128 on 8): 197 us on the CUDA cores, 60 here; 8 decoded tokens of 4,096 keys 142 and 130.
#include "attention_f32.cuh"
#include "umma.cuh"

#include <algorithm>

namespace {

constexpr int TROWS = 128, TKEYS = 64, THD = 128;
constexpr int TILES_PER_STRETCH = STRETCH / TKEYS;
constexpr int T_THREADS = 12 * 32;       // (three warps a scheduler: 168 registers a thread)
constexpr int FEW_ROWS = 32;             // up to here softmax has two warps' work: five of its others bring keys and values too
constexpr int Q_PART = TROWS * THD * 2, KV_PART = TKEYS * THD * 2;       // bytes of one part
constexpr int STAGE = TKEYS * THD * 4;                                   // a tile's keys or values as they lie in the pages
constexpr int T_SMEM = 3 * Q_PART + 6 * KV_PART + STAGE + 2048 + 640;
static_assert(T_SMEM <= 227 * 1024, "shared memory of an SM");
constexpr int COL_SL = 0, COL_SS = 64, COL_P = 128, COL_OL = 256, COL_OS = 384;
constexpr int BAD_K = 1, BAD_V = 2, GAPS = 4;    // a tile with keys or values that have no parts; with keys that nobody sees or without a page
constexpr float T_MOST = 1.0e18f;        // (2^60)
constexpr float V_IN = 281474976710656.0f, V_OUT = 1.0f / V_IN;          // (2^48: sums of 64 weighted values stay below 2^114)

// The largest magnitude, NaN if there was one.
__device__ __forceinline__ float larger(float a, float b) {
    float c;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(c) : "f"(fabsf(a)), "f"(fabsf(b)));
    return c;
}
__device__ __forceinline__ float most_of(float4 v) { return larger(larger(v.x, v.y), larger(v.z, v.w)); }
// Channels 4 lane .. 4 lane + 3 of row r into the three parts of [ROWS][128] (two blocks of 64 channels, 128-byte swizzle).
template <int ROWS>
__device__ __forceinline__ void place(uint32_t parts, int r, int lane, float4 v) {
    constexpr uint32_t PART = ROWS * THD * 2;
    uint2 h, m, l;
    split_bf16x3(v.x, v.y, h.x, m.x, l.x);
    split_bf16x3(v.z, v.w, h.y, m.y, l.y);
    const uint32_t at = parts + (uint32_t)((lane >> 4) * ROWS * 128 + r * 128 + ((((lane >> 1) & 7) ^ (r & 7)) << 4) + (lane & 1) * 8);
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(h.x), "r"(h.y) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + PART), "r"(m.x), "r"(m.y) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + 2 * PART), "r"(l.x), "r"(l.y) : "memory");
}
// Sixteen columns from each of two places, waited for once.
__device__ __forceinline__ void tmem_ld16_two(uint32_t at, uint32_t too, float* x, float* y) {
    uint32_t r[16], q[16];
    tmem_ld16_nowait(at, r);
    tmem_ld16_nowait(too, q);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        x[i] = __uint_as_float(r[i]);
        y[i] = __uint_as_float(q[i]);
    }
}
// What is rare is called, not expanded: a loop's instructions have to stay in the cache.
// A key's place in the pools, in rows, or a negative number.
__device__ __noinline__ long pool_row(const F32Args& a, int seq, int kvh, int t) {
    const int base_page = a.table_base ? a.table_base[seq] : 0, e = fb_table_column(t / a.page_size, base_page, a.table_head);
    const int page = (e >= 0 && e < a.table_stride) ? a.block_table[(size_t)seq * a.table_stride + e] : -1;
    return page < 0 || page >= a.n_pages ? -1 : ((long)page * a.nkv + kvh) * a.page_size + t % a.page_size;
}
// A score in float32 multiply-adds.
__device__ __noinline__ float slow_score(const F32Args& a, const float* q, int seq, int kvh, int t) {
    const long at = pool_row(a, seq, kvh, t);
    if (at < 0) return 0.0f;
    const float* k = a.k_pool + (size_t)at * THD;
    float s = 0.0f;
    for (int d = 0; d < THD; ++d) s = fmaf(q[d], k[d], s);
    return s * a.scale;
}

__global__ void __launch_bounds__(T_THREADS, 1)
attention_f32_tc_kernel(const __grid_constant__ F32Args a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];        // (the swizzle's blocks; nothing is left to align it by hand)
    uint8_t* Qs = smem_raw;
    uint8_t* Ks = Qs + 3 * Q_PART;
    uint8_t* Vs = Ks + 3 * KV_PART;
    uint8_t* stage = Vs + 3 * KV_PART;
    float* red = (float*)(stage + STAGE);                        // [2][128]: a row's maximum (sum) over either thread's keys
    float* run = red + 2 * TROWS;                                // [2][128]: maximum and sum of the stretches joined so far
    uint64_t* bars = (uint64_t*)(run + 2 * TROWS);
    uint64_t *k_full = bars, *v_full = bars + 1, *s_full = bars + 2, *s_empty = bars + 3, *p_full = bars + 4, *pv_done = bars + 5;
    uint64_t *q_full = bars + 6, *staged = bars + 7;             // staged: [8], of each warp that brings keys and values
    uint32_t* tmem_slot = (uint32_t*)(bars + 15);
    int* bail = (int*)(tmem_slot + 1);
    int* flags = bail + 1;                                       // [8]: of a tile
    uint8_t* bad_q = (uint8_t*)(flags + 8);                      // [128]
    uint8_t* has_page = bad_q + TROWS;                           // [4][64]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = a.nh / a.nkv;
    const int pair = blockIdx.x / a.token_tiles, tile = blockIdx.x - pair * a.token_tiles;
    const int seq = pair / a.nkv, kvh = pair - seq * a.nkv;
    fb_pdl_wait();
    const int q_len = a.seq_q_len[seq], TQ = TROWS / G;
    const int tok0 = (a.token_tiles - 1 - tile) * TQ;            // later tokens see more keys: start them first
    if (tok0 >= q_len) return;
    const int ntok = min(TQ, q_len - tok0), rows = ntok * G;
    const int q_start = a.seq_q_start[seq] + tok0, pos0 = a.seq_pos_start[seq] + tok0;

    // ---- the tiles, and the stretches numbered from the first that holds one ----
    const int t_hi = pos0 + ntok - 1, t_lo = fb_first_key(pos0, a.window, 0);
    const int tile_lo = t_lo / TKEYS * TKEYS, n_tiles = (t_hi - tile_lo) / TKEYS + 1, window_first = tile_lo / STRETCH;
    auto tile_of = [&](int s) {                                  // the first tile of stretch s
        return s >= a.slots ? n_tiles : min(n_tiles, max(0, (s + window_first) * TILES_PER_STRETCH - tile_lo / TKEYS));
    };
    const int slot0 = blockIdx.z * a.per, slot_end = min(slot0 + a.per, a.slots);
    const int first_tile = tile_of(slot0), T = tile_of(slot_end) - first_tile;       // tiles of this CTA
    auto tile_start = [&](int i) { return tile_lo + (first_tile + i) * TKEYS; };
    const int* table = a.block_table + (size_t)seq * a.table_stride;
    const int base_page = a.table_base ? a.table_base[seq] : 0;
    const bool few = rows <= FEW_ROWS;
    const int fetchers = few ? 256 : 96;                         // threads that bring keys and values
    if (tid == 0) {
        mbar_init(smem_u32(k_full), fetchers);
        mbar_init(smem_u32(v_full), fetchers);
        mbar_init(smem_u32(s_full), 1);
        mbar_init(smem_u32(s_empty), 64 * ((rows + 31) / 32));   // (the softmax warps that have rows)
        mbar_init(smem_u32(p_full), 64 * ((rows + 31) / 32));
        mbar_init(smem_u32(pv_done), 1);
        mbar_init(smem_u32(q_full), few ? 64 : 256);
        for (int i = 0; i < 8; ++i) mbar_init(smem_u32(staged + i), 1);
        *bail = 0;
        for (int i = 0; i < 8; ++i) flags[i] = 0;
        mbar_fence_init();
    }
    if (warp == 11) tmem_alloc(tmem_slot, 512);                  // (behind the wait: the kernels ahead have given theirs back)
    tmem_fence_before();
    __syncthreads();
    fb_pdl_launch_dependents();                                  // (behind the allocation: see umma.cuh)
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto wait_for = [&](uint32_t bar, int phase) { return mbar_wait(bar, (uint32_t)phase & 1u, a.status); };
    auto wait = [&](uint64_t* bar, int phase) { return wait_for(smem_u32(bar), phase); };
    auto bailed = [&]() { return *(volatile int*)bail != 0; };

    // ---------------- keys and values: warp w takes `count` rows of a tile from r0 on, a lane four channels ----------------
    auto bring = [&](auto rows_of, int r0, int count) {
        constexpr int R = decltype(rows_of)::value;
        // lane l: where row r0 + l of a tile lies in a pool, in rows (-2: no query sees it, -1: it has no page); the tile's entry of
        // the table is read a tile ahead.
        int key = tile_start(0) + r0 + lane, column = key / a.page_size, in_page = key - column * a.page_size, entry = -1;
        const int columns = TKEYS / a.page_size, in_pages = TKEYS - columns * a.page_size;
        auto look = [&]() {
            const int e = fb_table_column(column, base_page, a.table_head);
            const bool there = e >= 0 && e < a.table_stride;
            entry = *(there ? table + e : a.seq_q_len);
            if (!there) entry = -1;
        };
        auto place_of = [&]() -> long {                          // (then the next tile's)
            const long at = lane >= count || key > t_hi || key < t_lo ? -2
                            : (entry < 0 || entry >= a.n_pages) ? -1 : ((long)entry * a.nkv + kvh) * a.page_size + in_page;
            key += TKEYS;
            column += columns;
            in_page += in_pages;
            if (in_page >= a.page_size) {
                in_page -= a.page_size;
                ++column;
            }
            return at;
        };
        // The rows on their way into the warp's part of the stage, those that follow one another in the pool as one copy.
        const uint32_t mine = smem_u32(stage) + (uint32_t)(r0 * THD * 4);
        const uint32_t landed = smem_u32(staged + (count <= 8 ? r0 >> 3 : warp - 8));
        int copies = 0;
        auto copy = [&](const float* pool, long at) {
            const uint32_t present = __ballot_sync(0xffffffffu, at >= 0);
            const long before = __shfl_up_sync(0xffffffffu, at, 1);
            const bool first = lane == 0 || at != before + 1 || before < 0;
            const uint32_t later = __ballot_sync(0xffffffffu, at < 0 || first) & (0xfffffffeu << lane);
            if (lane == 0) mbar_expect_tx(landed, (uint32_t)__popc(present) * THD * 4);
            __syncwarp();
            if (at >= 0 && first)
                bulk_copy_g2s(mine + lane * THD * 4, pool + at * THD, (uint32_t)((later ? __ffs(later) - 1 : 32) - lane) * THD * 4, landed);
        };
        // The rows that have arrived (zeros without a place), and their largest magnitude.
        bool ok = true;                  // (a wait that ran out ends the waiting, not the loop: the warps meet at barriers of their own)
        auto settle = [&](bool got) { ok = __all_sync(0xffffffffu, got); };
        auto take = [&](float4* v, uint32_t missing) {
            const bool got = wait_for(landed, copies++);
            if (!__all_sync(0xffffffffu, got)) ok = false;
#pragma unroll
            for (int j = 0; j < R; ++j)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w)
                             : "r"(mine + (j < count ? j : 0) * THD * 4 + lane * 16) : "memory");
            if (missing)
#pragma unroll
                for (int j = 0; j < R; ++j)
                    if (j >= count || (missing >> j & 1u)) v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 top = v[0];                                   // (four chains: one would take as long as the rest)
#pragma unroll
            for (int j = 1; j < R; ++j) top = make_float4(larger(top.x, v[j].x), larger(top.y, v[j].y), larger(top.z, v[j].z), larger(top.w, v[j].w));
            const float most = most_of(top);
            asm volatile("" ::"f"(most) : "memory");             // (all of them have been read: the next copy may land)
            __syncwarp();
            return most;
        };
        auto put = [&](uint32_t parts, const float4* v) {
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (j < count) place<TKEYS>(parts, r0 + j, lane, v[j]);
        };
        const uint32_t k_at = smem_u32(Ks), v_at = smem_u32(Vs);
        // The keys of tile i + 1 go ahead of the values of tile i: the scores before them are done early, the product later.
        const uint32_t some = 0xffffffffu >> (32 - count);
        look();
        long at = -2, at_k = place_of();
        uint32_t missing_k = __ballot_sync(0xffffffffu, at_k < 0) & some, missing_v = 0;
        look();
        if (T > 0) copy(a.k_pool, at_k);
        for (int i = -1; i < T; ++i) {
            const long after = place_of();                       // of the keys of tile i + 2
            look();
            // (one body for both: its instructions, twice, would not stay in the cache beside the softmax warps')
#pragma unroll 1
            for (int values = i + 1 == T; values <= (i >= 0); ++values) {
                float4 v[R];
                const float most = take(v, values ? missing_v : missing_k);
                const bool next_k = values ? i + 2 < T : i < 0 && T > 1;
                const long next = next_k ? after : values || i < 0 ? at_k : at;
                if (!values || i + 1 < T) copy(next_k ? a.k_pool : a.v_pool, next);
                if ((values ? i > 0 : i >= 0) && ok) settle(!bailed() && wait(values ? pv_done : s_full, i - values));
                int flag = __any_sync(0xffffffffu, !(most < T_MOST)) ? (values ? BAD_V : BAD_K) : 0;
                if (values) {
#pragma unroll
                    for (int j = 0; j < R; ++j) v[j] = make_float4(v[j].x * V_IN, v[j].y * V_IN, v[j].z * V_IN, v[j].w * V_IN);
                } else {
                    if (missing_k) flag |= GAPS;
                    // (set next by whom these keys' scores have reached; read last six tiles ago)
                    if (lane == 0 && warp == 8) flags[(i + 2) & 7] = 0;
                    if (lane < count) {
                        has_page[((i + 1) & 3) * TKEYS + r0 + lane] = at_k >= 0;
                        if (at_k == -1) atomicOr(a.status, FB_STATUS_BAD_PAGE);
                    }
                }
                put(values ? v_at : k_at, v);
                if (lane == 0 && flag) atomicOr(&flags[(i + !values) & 7], flag);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive(smem_u32(values ? v_full : k_full));
            }
            at = at_k;
            at_k = after;
            missing_v = missing_k;
            missing_k = __ballot_sync(0xffffffffu, after < 0) & some;
        }
        if (!ok) *bail = 1;
    };
    // ---------------- queries: sixteen rows a warp (zeros beyond the CTA's), while the first keys are on their way ----------------
    if (T > 0 && (few ? warp == 0 || warp == 4 : warp < 8)) {
        const int q0 = few ? warp * 4 : warp * 16;               // (what lies in the quarters that nobody reads does not matter)
#pragma unroll 1
        for (int r0 = q0; r0 < q0 + 16; r0 += 8) {
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = min(r0 + j, rows - 1);
                v[j] = *reinterpret_cast<const float4*>(a.q + (size_t)(q_start + r / G) * a.q_stride + (size_t)(kvh * G + r % G) * THD + 4 * lane);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (r0 + j >= rows) v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                const bool bad = __any_sync(0xffffffffu, !(most_of(v[j]) < T_MOST));
                if (lane == 0) bad_q[r0 + j] = bad;
                place<TROWS>(smem_u32(Qs), r0 + j, lane, v[j]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(smem_u32(q_full));
    }
    const std::integral_constant<int, 8> eight;
    const std::integral_constant<int, 22> most_rows;

    if (warp == 11) {
        // ---------------- MMA ----------------
        if (elect_one()) {
            const uint32_t idesc_s = umma_idesc(TKEYS), idesc_o = umma_idesc(THD, true);
            // (addresses stand in a descriptor in units of 16 bytes: a part, a block or a step further is an addition)
            const uint64_t q_desc = umma_desc(smem_u32(Qs)), k_desc = umma_desc(smem_u32(Ks)), v_desc = umma_desc_mn(smem_u32(Vs), TKEYS * 128, 1024);
            auto scores = [&](int t) {
                bool ok = wait(k_full, t) && (t == 0 || wait(s_empty, t - 1));
                if (!ok) return false;
                tmem_fence_after();
#pragma unroll
                for (int kk = 0; kk < THD / UMMA_K; ++kk) {
                    const uint64_t qs = (uint64_t)((kk >> 2) * (Q_PART / 2 / 16) + (kk & 3) * 2), ks = (uint64_t)((kk >> 2) * (KV_PART / 2 / 16) + (kk & 3) * 2);
                    const uint64_t qh = q_desc + qs, qm = qh + Q_PART / 16, ql = qm + Q_PART / 16;
                    const uint64_t kh = k_desc + ks, km = kh + KV_PART / 16, kl = km + KV_PART / 16;
                    const uint32_t more = kk > 0 ? 1u : 0u;
                    umma_bf16(tmem + COL_SL, qh, kh, idesc_s, more);
                    umma_bf16(tmem + COL_SS, qh, km, idesc_s, more);
                    umma_bf16(tmem + COL_SS, qm, kh, idesc_s, 1u);
                    umma_bf16(tmem + COL_SS, qh, kl, idesc_s, 1u);
                    umma_bf16(tmem + COL_SS, ql, kh, idesc_s, 1u);
                    umma_bf16(tmem + COL_SS, qm, km, idesc_s, 1u);
                }
                umma_commit(smem_u32(s_full));                   // (also: the keys' slot is free)
                return true;
            };
            bool ok = T <= 0 || (wait(q_full, 0) && scores(0));
            for (int t = 0; t < T && ok && !bailed(); ++t) {
                if (t + 1 < T) ok = scores(t + 1);
                if (ok) ok = wait(v_full, t) && wait(p_full, t);
                if (!ok) break;
                tmem_fence_after();
                const uint32_t p0 = tmem + COL_P;
#pragma unroll
                for (int kk = 0; kk < TKEYS / UMMA_K; ++kk) {
                    const uint64_t vh = v_desc + kk * (16 * 128 / 16), vm = vh + KV_PART / 16, vl = vm + KV_PART / 16;
                    const uint32_t ph = p0 + (uint32_t)(kk * 8), pm = ph + 32, pl = pm + 32, more = kk > 0 ? 1u : 0u;
                    umma_bf16_ts(tmem + COL_OL, ph, vh, idesc_o, more);
                    umma_bf16_ts(tmem + COL_OS, ph, vm, idesc_o, more);
                    umma_bf16_ts(tmem + COL_OS, pm, vh, idesc_o, 1u);
                    umma_bf16_ts(tmem + COL_OS, ph, vl, idesc_o, 1u);
                    umma_bf16_ts(tmem + COL_OS, pl, vh, idesc_o, 1u);
                    umma_bf16_ts(tmem + COL_OS, pm, vm, idesc_o, 1u);
                }
                umma_commit(smem_u32(pv_done));                  // (also: the values' and the weights' places are free)
            }
            if (!ok) *bail = 1;
        }
        __syncwarp();
    } else if (few && warp != 7 && (warp >= 8 || (warp & 3) * 32 >= rows)) {     // (five warps without rows help)
        bring(eight, 8 * (warp >= 8 ? warp - 8 : warp < 4 ? warp + 2 : warp + 1), 8);
    } else if (warp >= 8) {
        bring(most_rows, 21 * (warp - 8) + (warp > 8), warp == 8 ? 22 : 21);
    } else {
        // ---------------- softmax: thread (half, row) has keys 32 half + and outputs 64 half + of its row ----------------
        const int quarter = warp & 3, half = warp >> 2, r = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const bool real = r < rows;
        const int row = q_start + r / G, head = kvh * G + r % G;
        const int p_row = real ? pos0 + r / G : 0x7fffffff, t0_row = real ? fb_first_key(p_row, a.window, 0) : 0;
        bool ok = true, ended = false;   // (a wait that ran out ends the waiting, not the loop)
        auto settle = [&](bool got) { ok = __all_sync(0xffffffffu, got); };
        if (T > 0) settle(wait(q_full, 0));
        const bool slow_row = T > 0 && real && bad_q[r];
        const float* q_row = a.q + (size_t)(real ? row : q_start) * a.q_stride + (size_t)(real ? head : 0) * THD;
        auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); };      // a row's two threads
        float m = -INFINITY, l = 0.0f, corr_before = 1.0f, m_before = 0.0f, m_end = -INFINITY, l_end = 0.0f, o[64];
#pragma unroll
        for (int c = 0; c < 64; ++c) o[c] = 0.0f;
        int slot = slot0, stretch_end = tile_of(slot + 1) - first_tile;
        // What the product of tile i left, added to the outputs with the rescaling that came with its weights; a tile (or a row)
        // with numbers that have no parts key by key instead.
        auto collect = [&](int i, float corr, float m_use) {
            const bool slow = slow_row || (real && (flags[i & 7] & (BAD_K | BAD_V)));
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 16) {
                float x[16], y[16];
                tmem_ld16_two(lanes + (uint32_t)(COL_OL + half * 64 + c0), lanes + (uint32_t)(COL_OS + half * 64 + c0), x, y);
#pragma unroll
                for (int c = 0; c < 16; ++c) o[c0 + c] = fmaf(o[c0 + c], corr, slow ? 0.0f : (x[c] + y[c]) * V_OUT);
            }
            if (slow)
                for (int t = max(tile_start(i), t0_row); t <= min(tile_start(i) + TKEYS - 1, p_row); ++t) {
                    const long at = pool_row(a, seq, kvh, t);
                    if (at < 0) continue;
                    const float w = expf(slow_score(a, q_row, seq, kvh, t) - m_use);
                    const float* v = a.v_pool + (size_t)at * THD + half * 64;
#pragma unroll
                    for (int c = 0; c < 64; ++c) o[c] = fmaf(w, v[c], o[c]);
                }
            __syncwarp();
        };
        // The outputs of a complete stretch (slot `slot`, maximum m_end, this thread's sum l_end) on their way; last: of the CTA.
        // Four threads exchange theirs, so that 64 bytes of a row go at a time: a quarter of the accesses.
        auto finalize = [&](float m_end, float l_end, bool last) {
            red[half * TROWS + r] = l_end;
            meet();
            const float l_all = red[r] + red[TROWS + r];
            const bool parts = a.part_o != nullptr, first = slot == 0;
            float M = -INFINITY, L = 0.0f, f = 1.0f;
            Join j = {0.0f, 1.0f};
            long at = 0;
            if (real && parts) {
                const size_t p = part_at<64>(a, slot, pair, row, head, r);
                if (half == 0) *reinterpret_cast<float2*>(a.part_ml + 2 * p) = make_float2(m_end, l_all);
                at = (long)p * THD + half * 64;
            } else if (real) {
                M = first ? -INFINITY : run[r], L = first ? 0.0f : run[TROWS + r];
                j = join(M, L, m_end, l_all);
                if (last) f = finish(a, row, head, M, L);
                at = (long)row * a.out_stride + (long)head * THD + half * 64;
            }
            meet();                                              // (red and run have been read)
            if (half == 0) {
                run[r] = M;
                run[TROWS + r] = L;
            }
            float* to = (parts ? a.part_o : a.out) + 4 * (lane & 3);             // (read by the thread that wrote it)
            const uint32_t reals = __ballot_sync(0xffffffffu, real) >> (lane & 28);
#pragma unroll
            for (int c = 0; c < 64; c += 16) {                   // lane 4 g + i: channels c + 4 i .. of the rows 4 g ..
#pragma unroll
                for (int k = 0; k < 16; ++k) {                   // [row][4 channels] <-> the four threads
                    if ((k >> 2) & 1) continue;
                    const float give = lane & 1 ? o[c + k] : o[c + k + 4], got = __shfl_xor_sync(0xffffffffu, give, 1);
                    if (lane & 1) o[c + k] = got; else o[c + k + 4] = got;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float give = lane & 2 ? o[c + k] : o[c + k + 8], got = __shfl_xor_sync(0xffffffffu, give, 2);
                    if (lane & 2) o[c + k] = got; else o[c + k + 8] = got;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int from = (lane & 28) + i;
                const Join ji = {__shfl_sync(0xffffffffu, j.before, from), __shfl_sync(0xffffffffu, j.own, from)};
                const float fi = __shfl_sync(0xffffffffu, f, from);
                float* op = to + __shfl_sync(0xffffffffu, at, from);
                float4 b[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = parts || first ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(op + 16 * c);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float* x = o + 16 * c + 4 * i;
                    float4 y = make_float4(x[0], x[1], x[2], x[3]);
                    if (!parts)
                        y = make_float4(joined(ji, b[c].x, y.x) * fi, joined(ji, b[c].y, y.y) * fi, joined(ji, b[c].z, y.z) * fi, joined(ji, b[c].w, y.w) * fi);
                    if (reals >> i & 1u) *reinterpret_cast<float4*>(op + 16 * c) = y;
                }
            }
#pragma unroll
            for (int c = 0; c < 64; ++c) o[c] = 0.0f;
            ++slot;
        };
        // (a quarter without rows: what its lanes hold concerns no other row)
        const bool idle = quarter * 32 >= rows;
        for (int i = 0; !idle && i < T; ++i) {
            if (ok) settle(!bailed() && wait(s_full, i));
            tmem_fence_after();
            float s[32];
#pragma unroll
            for (int c0 = 0; c0 < 32; c0 += 16) {
                float x[16], y[16];
                tmem_ld16_two(lanes + (uint32_t)(COL_SL + half * 32 + c0), lanes + (uint32_t)(COL_SS + half * 32 + c0), x, y);
#pragma unroll
                for (int c = 0; c < 16; ++c) s[c0 + c] = (x[c] + y[c]) * a.scale;
            }
            tmem_fence_before();
            mbar_arrive(smem_u32(s_empty));
            const int flag = flags[i & 7];
            const bool slow = slow_row || (real && (flag & BAD_K));              // the row's scores of this tile one by one
            const int key0 = tile_start(i) + half * 32;
            uint32_t seen = 0xffffffffu;
            // (a warp whose rows see all of their keys, as most do, has nothing to leave out)
            if (__any_sync(0xffffffffu, (real && (flag & GAPS)) || key0 + 31 > p_row || key0 < t0_row)) {
                const uint8_t* there = has_page + (i & 3) * TKEYS + half * 32;
                seen = 0;
#pragma unroll
                for (int c = 0; c < 32; ++c) seen |= (key0 + c <= p_row && key0 + c >= t0_row && there[c]) ? 1u << c : 0u;
            }
            if (__any_sync(0xffffffffu, slow)) {
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    if (slow && (seen >> c & 1u)) s[c] = slow_score(a, q_row, seq, kvh, key0 + c);
            }
            float top = -INFINITY;
            if (__all_sync(0xffffffffu, seen == 0xffffffffu)) {
#pragma unroll
                for (int c = 0; c < 16; ++c) top = fmaxf(top, fmaxf(s[c], s[c + 16]));
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    if (!(seen >> c & 1u)) s[c] = -INFINITY;     // (its weight: exp(-inf) = 0)
                    top = fmaxf(top, s[c]);
                }
            }
            red[half * TROWS + r] = top;
            meet();
            const float m_new = fmaxf(m, fmaxf(top, red[(half ^ 1) * TROWS + r])), m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = m == -INFINITY ? 0.0f : expf(m - m_use);
            float sum = 0.0f;
            uint32_t ph[16], pm[16], pl[16];
#pragma unroll
            for (int c = 0; c < 32; c += 2) {
                const float x = expf(s[c] - m_use), y = expf(s[c + 1] - m_use);
                sum += x + y;
                split_bf16x3(x, y, ph[c / 2], pm[c / 2], pl[c / 2]);
            }
            l = l * corr + sum;
            m = m_new;
            meet();                                              // (red has been read by both)
            if (i > 0) {                                         // the product before has read its weights
                if (ok) settle(!bailed() && wait(pv_done, i - 1));
                tmem_fence_after();
            }
            tmem_st16(lanes + (uint32_t)(COL_P + half * 16), ph);
            tmem_st16(lanes + (uint32_t)(COL_P + 32 + half * 16), pm);
            tmem_st16(lanes + (uint32_t)(COL_P + 64 + half * 16), pl);
            if (i > 0) collect(i - 1, corr_before, m_before);
            tmem_wait_st();
            tmem_fence_before();
            mbar_arrive(smem_u32(p_full));
            if (ended) finalize(m_end, l_end, false);            // (of the tile before: beside this tile's product)
            m_before = m_use;
            corr_before = corr;
            ended = i + 1 == stretch_end;
            if (ended) {
                m_end = m;
                l_end = l;
                m = -INFINITY;
                l = 0.0f;
                stretch_end = tile_of(slot + 2) - first_tile;
            }
        }
        if (!idle && T > 0) {
            if (ok) settle(!bailed() && wait(pv_done, T - 1));
            tmem_fence_after();
            collect(T - 1, corr_before, m_before);
            tmem_fence_before();
            finalize(ended ? m_end : m, ended ? l_end : l, true);
        }
        if (!ok) *bail = 1;
        if (a.part_o && half == 0 && real)                       // stretches that these rows do not have
            for (; slot < slot_end; ++slot)
                *reinterpret_cast<float2*>(a.part_ml + 2 * part_at<64>(a, slot, pair, row, head, r)) = make_float2(-INFINITY, 0.0f);
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 11) {
        tmem_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

struct TcPlan { int slots, per; long long floats; };
// Stretches that a CTA takes: what is over first by an estimate of the longest CTA, of the SMs' share of all tiles and of the
// joining (`tiles`: CTAs a key/value head).  Measured: a tile of full rows takes 3.6 us, with one warp of rows 2.6, a CTA's start
// and end 10 and 7, joining 3 and a microsecond for 10 MB written and read.  301 tokens behind 500: 62 us in one piece, 52 in
// two, 59 in four; 2,048 tokens 321 in one, 384 in two; 8 decoded ones of 8,000 keys 220 in two, 363 in one, 219 in five.
TcPlan tc_plan(int n, int nh, int nkv, int max_q_len, int max_kv_len, int window, long long tiles) {
    TcPlan p = {};
    const int TQ = TROWS / (nh / nkv), token_tiles = std::max(1, (max_q_len + TQ - 1) / TQ);
    long long slots = ((long long)max_kv_len + STRETCH - 1) / STRETCH, key_tiles = std::max(1LL, ((long long)max_kv_len + TKEYS - 1) / TKEYS);
    if (window > 0) {
        slots = std::min(slots, (window + TROWS - 2LL) / STRETCH + 2);
        key_tiles = std::min(key_tiles, (window + TQ - 2LL) / TKEYS + 2);
    }
    p.slots = (int)(slots < 1 ? 1 : slots);
    p.per = p.slots;
    const bool few = (long long)max_q_len * (nh / nkv) <= FEW_ROWS;
    const double tile_us = few ? 2.6 : 3.6, cta_us = few ? 7.0 : 10.0, ctas = (double)tiles * nkv, sms = fb_sm_count();
    const double mean_tiles = std::max(1.0, key_tiles - (window > 0 && window < max_kv_len ? 0.0 : 0.5 * (token_tiles - 1) * TQ / TKEYS));
    const double join_us = 3.0 + (double)p.slots * n * nh * (THD + 2) * 8.0 * 1e-7;
    double best = 1e300;
    for (int per = p.slots; per >= 1; --per) {
        const int z = (p.slots + per - 1) / per;
        if (z > 65535 || (z > 1 && (long long)p.slots * n * nh * (THD + 2) > SCRATCH_FLOATS)) break;
        const double longest = std::min((double)per * TILES_PER_STRETCH, (double)key_tiles) * tile_us + cta_us;
        const double last = std::max(1.0, mean_tiles - (double)(z - 1) * per * TILES_PER_STRETCH) * tile_us + cta_us;    // (of a row of keys)
        const double share = ctas * (mean_tiles * tile_us + z * cta_us) / sms + 0.5 * last;
        const double cost = (ctas * z <= sms ? longest : std::max(longest, share)) + (z > 1 ? join_us : 0.0);
        if (cost < 0.95 * best) { best = cost; p.per = per; }    // (more pieces only where they clearly pay)
    }
    p.floats = p.per < p.slots ? border4((long long)p.slots * n * nh * (THD + 2)) : 0;
    return p;
}

}  // namespace

// Floats of scratch that fb_attention_f32_tc wants for the same numbers.
FB_API long long fb_attention_f32_tc_scratch_floats(int n, int nh, int nkv, int max_q_len, int max_kv_len, int window, long long tiles) {
    if (n <= 0 || nh <= 0 || nkv <= 0 || nh % nkv != 0 || nh / nkv > 64 || tiles <= 0) return 0;
    return tc_plan(n, nh, nkv, max_q_len, max_kv_len, window, tiles).floats;
}

// As fb_paged_attention_f32, for heads of 128 (keys and values), without caps, slopes or kept first keys.  tiles: tiles of 128
// rows (tokens x query heads a key/value head) over all sequences.
FB_API int fb_attention_f32_tc(const float* q, long long q_stride, float* out, long long out_stride, const float* k_pool,
                               const float* v_pool, int page_size, int n_pages, const int* block_table, int table_stride,
                               const int* table_base, int table_head, const int* seq_q_start, const int* seq_q_len,
                               const int* seq_pos_start, int n_seqs, int max_q_len, int max_kv_len, long long tiles, int n, int nh,
                               int nkv, int window, float scale, const float* sinks, const float* head_gate, long long gate_stride,
                               int gate_partials, long long gate_partial_stride, float* part, long long part_floats, int* status,
                               cudaStream_t stream) {
    FB_REQUIRE(n >= 0 && n_seqs >= 0 && nh > 0 && nkv > 0 && nh % nkv == 0 && nh / nkv <= 64, "attention_f32: bad head counts");
    FB_REQUIRE(q_stride % 4 == 0 && out_stride % 4 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)out % 16 == 0 &&
               (uintptr_t)k_pool % 16 == 0 && (uintptr_t)v_pool % 16 == 0, "attention_f32: unaligned operands");
    FB_REQUIRE(page_size > 0 && n_pages > 0 && window >= 0 && (!head_gate || gate_stride >= nh), "attention_f32: bad cache geometry or gate");
    if (n == 0 || n_seqs == 0) return 0;
    F32Args a = {};
    a.q = q; a.q_stride = (long)q_stride; a.out = out; a.out_stride = (long)out_stride;
    a.k_pool = k_pool; a.v_pool = v_pool; a.page_size = page_size; a.n_pages = n_pages;
    a.block_table = block_table; a.table_stride = table_stride; a.table_base = table_base;
    a.table_head = table_head > 0 ? table_head : 0;
    a.seq_q_start = seq_q_start; a.seq_q_len = seq_q_len; a.seq_pos_start = seq_pos_start;
    a.n_seqs = n_seqs; a.n = n; a.nh = nh; a.nkv = nkv; a.hd = a.vd = THD; a.window = window;
    a.scale = scale; a.sinks = sinks; a.head_gate = head_gate; a.gate_stride = (long)gate_stride;
    a.gate_partials = gate_partials < 1 ? 1 : gate_partials; a.gate_partial_stride = (long)gate_partial_stride;
    a.status = status;
    const TcPlan p = tc_plan(n, nh, nkv, max_q_len, max_kv_len, window, tiles);
    FB_REQUIRE(p.floats == 0 || (part && (uintptr_t)part % 16 == 0 && part_floats >= p.floats), "attention_f32: too little scratch");
    a.slots = p.slots;
    a.per = p.per;
    a.part_o = p.floats ? part : nullptr;
    a.part_ml = p.floats ? part + (long long)p.slots * n * nh * THD : nullptr;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(attention_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T_SMEM);
        if (e != cudaSuccess) return fb_fail(-2, "attention_f32: cannot reserve %d bytes of shared memory: %s", T_SMEM, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    const int G = nh / nkv;
    a.token_tiles = (max_q_len + TROWS / G - 1) / (TROWS / G);
    FB_REQUIRE((long long)a.token_tiles * n_seqs * nkv < (1LL << 31) && (p.slots + p.per - 1) / p.per <= 65535, "attention_f32: too many CTAs for one grid");
    fb_launch(attention_f32_tc_kernel, dim3((unsigned)((long)a.token_tiles * n_seqs * nkv), 1, (p.slots + p.per - 1) / p.per), dim3(T_THREADS),
              (size_t)T_SMEM, stream, a);
    const int rc = fb_check_launch("attention_f32_tc");
    if (rc || !a.part_o) return rc;
    a.token_tiles = (max_q_len + 64 / G - 1) / (64 / G);         // (short_rows = 0: every sequence is joined by 64 rows)
    FB_REQUIRE((long long)a.token_tiles * n_seqs * nkv < (1LL << 31), "attention_f32: too many CTAs for one grid");
    fb_launch((attention_f32_join_kernel<64>), dim3((unsigned)((long)a.token_tiles * n_seqs * nkv), 16), dim3(128), 0, stream, a);
    return fb_check_launch("attention_f32_join");
}
