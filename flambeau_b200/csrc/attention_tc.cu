// Paged causal (sliding-window) attention for portions of prompts on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory), for heads of 64 or 128 bfloat16 and pages that tile 64 keys, and for heads
// of 256 whose key rows are the values as well (attention over latents).
//
// A CTA owns one key/value head and 256 query rows = (256 / G) tokens x the G query heads that share the head, as
// two row tiles of 128 that use every K/V tile fetched (one row tile when two would leave SMs without work), and
// walks the visible keys in tiles of 64.  CTAs are numbered heaviest first over all heads and sequences.
//
//   S = Q K^T      tcgen05.mma, Q and K K-major in shared memory (128-byte swizzle), S in tensor memory, two
//                  buffers per row tile: the scores run two key tiles ahead of the softmax;
//   softmax        one thread per row (the row = its tensor-memory lane): the row's 64 scores in one tcgen05.ld
//                  round trip, base-2 online softmax in float32, P rounded to bfloat16 and stored with tcgen05.st
//                  over the scores it came from; where the caller wants more bits of mantissa, what the rounding left is
//                  stored as one or two bfloat16 numbers more (two fill the columns that one score had), and the
//                  product runs over all;
//   O += P V       tcgen05.mma with P read from tensor memory and V as it lies in the cache ([key][dim], the
//                  MN-major operand); O in tensor memory.
//
// O is rescaled only when a row's maximum has grown by more than 2^8 since the exponentials' reference point was
// last moved (the sum l is kept against the same reference, so O / l is exact either way); the first tile sets
// the reference.  Warps: 0 fetches K and V pages with tensor-map copies through four-slot rings of their own (page
// ids read from the block table 32 at a time); 1 owns tensor memory; 1 and 2 issue the MMAs of row tiles 0 and 1;
// 4..7 and 8..11 are the softmax of the two row tiles (a warp reads the quarter of the lanes given by its index
// modulo 4).  A wait names a phase of an mbarrier only by its parity, so every barrier here is waited on for the
// phase that is current or just completed: one barrier per buffer, and one of its own for the last product.  Every
// wait is bounded in time; when one runs out the kernel flags it, leaves its loops, frees its tensor memory and
// returns.
//
// Heads of 256 (one row tile: O takes 256 columns): a tile is fetched once and serves as K and as V, its slot is free when
// its product is through.  An MMA of 64 columns takes as long as one of 128 (62 to 72 cycles), so a key tile costs 16 x 65 for
// the scores and 3 x 4 x 130 for the product with the three parts of the weights: 75 us of 2,048 tokens of 32 heads of 256 over
// one latent row, which take about 170 (570 on the mma.sync kernel, 153 with two parts).  The softmax bounds it, one thread a
// row: a quarter more MMAs, the third part's, cost a layer 1 to 4 %.
//
// Decoded tokens over latents (SPLIT): the rows of a sequence are fewer than a row tile, which costs a key tile no more; a CTA
// takes a stretch of a sequence's key tiles and leaves its rows' maximum, sum and unnormalised O, and a warp per row merges them.
//
// Differential attention (two score maps of 64 a head over values of 128): the row tiles are the two maps of the same 128
// rows, each with its column block of Q and K and both on one V tile.  At the end the threads of both take half of the
// columns each, read both maps' O from tensor memory and form the difference, its norm and the gate.  A key tile costs 8 x 65
// for the scores and 16 x 65 for the products, 45 us of 2,048 tokens of 32 heads, which take about 153 (373 on the mma.sync
// kernel, 141 with a reference that lags): the softmax threads again.
//
// Formulas: crates/kernels-hip/src/kernels/attention_prefill_flash_tile_f16.cu:73-213 (tile + online softmax).
#include "attention_common.cuh"
#include "umma.cuh"

namespace {

using namespace fb_attn;

constexpr int BM = 128;            // query rows per row tile (the M of the MMAs)
constexpr int BN = 64;             // keys per tile
// Threads of a CTA with RT row tiles: warp 0 fetches, warps 1 and 2 issue the MMAs of row tiles 0 and 1 (warp 3 has no
// work), warps 4..7 (and 8..11) are the softmax of row tile 0 (and 1).
__host__ __device__ constexpr int tc_threads(int rt) { return 128 + BM * rt; }
constexpr int NKV = 4;             // K slots and V slots
constexpr int TMEM_COLS = 512;     // S/P buffer b of row tile t at (2t + b) * 64; O of row tile t at RT * 128 + t * 128

// Softmax weights of more than one bfloat16 number (HILO) are three, 24 bits of mantissa, where tensor memory has 32 columns
// more a buffer: behind everything else, at heads of 64 behind O.  Two row tiles at heads of 128 fill it: there they are two,
// and the reference point of the exponentials follows a row's maximum at every step, so that the largest weight is 1 and
// loses nothing in two parts, as on the mma.sync kernels.  (A reference that lags leaves that weight up to 2^8, rounded to 16
// bits as the others are.  Results that are not the rounding of the exact ones, uneven weights: over latents 0.19 % so, 0.14
// with three parts, 0.16 on the mma.sync kernel; decoded tokens 0.16, 0.06 and 0.08; two maps 0.22, at every step 0.17, 0.17.
// The third part costs up to 4 % of a layer, a reference that follows at every step 5 to 40 % over latents, whose O is 256
// columns, and up to 6 % with two maps.)
template <int HD, int RT, bool HILO> struct Weights {
    static constexpr int PARTS = !HILO ? 1 : HD == 128 && RT == 2 ? 2 : 3;
    static constexpr float RESCALE_STEP = PARTS == 2 ? 0.0f : 8.0f;         // how far (base 2) a maximum may pass the reference
    __device__ static constexpr int third(int t, int b) {                   // the columns of the third parts
        return HD == 64 ? RT * 128 + t * 128 + 64 + b * (BN / 2) : RT * 128 + RT * HD + (2 * t + b) * (BN / 2);
    }
    static_assert(PARTS < 3 || HD == 64 || RT * 128 + RT * HD + RT * BN <= TMEM_COLS, "tensor memory");
};

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Key tiles a CTA takes of a sequence that `splits` CTAs share: a stretch of fewer than four would be mostly set-up.
__host__ __device__ __forceinline__ int split_tiles(int n_tiles, int splits) {
    const int per = (n_tiles + splits - 1) / splits;
    return per < 4 ? 4 : per;
}

template <int HD, int RT, bool SHARED, bool DIFF> struct TcSmem {
    static constexpr int Q_TILES = DIFF ? 1 : RT;               // (the maps' rows lie side by side in one)
    static constexpr int Q_BYTES = BM * HD * 2;                 // one row tile: [HD/64 column blocks][128 rows][128 bytes]
    static constexpr int KV_BYTES = BN * HD * 2;                // one K or V tile: [HD/64][64 keys][128 bytes]
    static constexpr int TAIL_BYTES = 256 + (DIFF ? 4 * BM * 4 : 0);                      // barriers, tensor-memory address, flag
    static constexpr int USED = Q_TILES * Q_BYTES + NKV * (SHARED ? 1 : 2) * KV_BYTES + TAIL_BYTES + 1024 /* alignment */;
    // one CTA per SM: two would both want all of tensor memory
    static constexpr int BYTES = USED > 120 * 1024 ? USED : 120 * 1024;
};

// RT row tiles of 128 rows per CTA: with two, both use every K/V tile that is fetched and the tensor pipe works for
// one under the softmax of the other; with one, a short portion still spreads over enough CTAs.
// HILO: the weights enter the product as two or three bfloat16 numbers each (Weights).  SHARED: the key rows are the values as well.
// DIFF: differential attention; the row tiles are the two maps of the same rows.  SPLIT: a stretch of the keys of a sequence
// whose rows fit a row tile.
template <int HD, int RT, bool HILO, bool SHARED, bool DIFF, bool SPLIT>
__global__ void __launch_bounds__(tc_threads(RT), 1)
attention_tc_kernel(const __grid_constant__ AttnArgs a) {
    static_assert(RT * 128 + RT * (HD > 128 ? HD : 128) <= TMEM_COLS, "tensor memory");
    static_assert(!DIFF || (HD == 128 && RT == 2 && !SHARED), "two maps of 64 over values of 128");
    using SM = TcSmem<HD, RT, SHARED, DIFF>;
    constexpr int ROWS = DIFF ? BM : RT * BM;                   // query rows of the CTA
    constexpr int CB = HD / 64;                                 // 64-column blocks of a head
    using W = Weights<HD, RT, HILO>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    uint8_t* Qs = smem;                                         // [RT] row tiles
    uint8_t* Ks = Qs + SM::Q_TILES * SM::Q_BYTES;                        // [NKV] tiles
    uint8_t* Vs = SHARED ? Ks : Ks + NKV * SM::KV_BYTES;        // [NKV] tiles
    uint8_t* tail = Vs + NKV * SM::KV_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail);
    uint64_t* k_full = bars;                                    // [NKV] a K tile has landed
    uint64_t* k_empty = bars + NKV;                             // [NKV] both row tiles' scores are computed
    uint64_t* v_full = bars + 2 * NKV;                          // [NKV] a V tile has landed
    uint64_t* v_empty = bars + 3 * NKV;                         // [NKV] both row tiles' products are computed
    uint64_t* s_full = bars + 4 * NKV;                          // [RT][2] S of a row tile is in tensor memory (two buffers)
    uint64_t* p_full = bars + 4 * NKV + 2 * RT;                 // [RT][2] P of a row tile is in tensor memory, per buffer:
                                                                //       the softmax may be two tiles ahead of the products
    uint64_t* pv_done = bars + 4 * NKV + 4 * RT;                // [RT]  O of a row tile holds the key tile's product
    uint64_t* o_done = bars + 4 * NKV + 5 * RT;                 // [RT]  O of a row tile holds all products (used once)
    uint64_t* q_full = bars + 4 * NKV + 6 * RT;                 //       Q is staged
    uint64_t* v_clean = bars + 4 * NKV + 6 * RT + 1;            //       row tile 0 has cleared a V tile's unseen rows (at most twice)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * NKV + 6 * RT + 2);
    int* bail = reinterpret_cast<int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = a.nh / a.nkv, hd = a.hd;

    // ---- what this CTA has to do: query tokens [tok0, tok0 + ntok) of a sequence, one key/value head ----
    // CTAs are numbered heaviest first over the whole step: the last tokens of every sequence and head (they see
    // the most keys) get the first SMs, whatever head or sequence they belong to
    const int pairs = a.nkv * (SPLIT ? a.n_seqs : portion_seqs(a));
    const int rank = SPLIT ? 0 : blockIdx.x / pairs, pair = SPLIT ? blockIdx.x / a.k_splits : blockIdx.x - rank * pairs;
    const int seq = SPLIT ? pair / a.nkv : portion_seq(a, pair / a.nkv), kvh = pair % a.nkv;
    const int q_tiles = SPLIT ? 1 : gridDim.x / pairs;
    const int q_len = a.seq_q_len[seq];
    if ((q_len * G <= a.short_rows) != SPLIT) return;           // the other arrangement's
    const int TQ = ROWS / G;
    const int tok0 = (q_tiles - 1 - rank) * TQ;               // later tokens see more keys: start them first
    if (tok0 >= q_len) return;
    const int ntok = min(TQ, q_len - tok0);
    const int q_start = a.seq_q_start[seq], pos0 = a.seq_pos_start[seq];
    const int rows_valid = ntok * G;                            // of the CTA's rows
    const int p_first = pos0 + tok0, p_last = pos0 + tok0 + ntok - 1;
    const int t_lo = fb_first_key(p_first, a.window, DIFF ? a.chunk : 0);
    const int t_hi = p_last;
    int k_begin = (t_lo / BN) * BN, k_end = t_hi + 1;
    if constexpr (SPLIT) {                                      // this CTA's stretch
        const int per = split_tiles((k_end - k_begin + BN - 1) / BN, a.k_splits);
        k_begin += (int)(blockIdx.x % a.k_splits) * per * BN;
        if (k_begin >= k_end) return;
        k_end = min(k_end, k_begin + per * BN);
    }
    const int n_tiles = (k_end - k_begin + BN - 1) / BN;        // both row tiles walk all of them
    const int* table = a.block_table + (size_t)seq * a.table_stride;
    const int pages_per_tile = BN / a.page_size;
    const int n_ops = pages_per_tile * CB;                      // copies per K or V tile: (page, column block)
    // Value rows no query of the CTA sees: pages of the first tile wholly before the window, keys of the last tile
    // behind the last position.  Whole pages arrive, the slots behind the last position included, and what a page
    // holds there was never written by this request; pages wholly before the window or behind the last position do
    // not arrive at all, and their slots hold whatever was there.  The probabilities of such keys are 0, but
    // 0 * NaN is NaN: the softmax of row tile 0 clears those rows, 128 bytes per key and column block, before it
    // lets its product start, and says so on a barrier that the thread of row tile 1's products waits for.
    const int dead_lo_first = max(0, t_lo - k_begin) / a.page_size * a.page_size;      // rows [0, dead_lo_first) of tile 0
    const int dead_hi_last = k_end - (k_begin + (n_tiles - 1) * BN);               // rows [dead_hi_last, BN) of the last tile
    auto dead_lo_of = [&](int j) { return j == 0 ? dead_lo_first : 0; };
    auto dead_hi_of = [&](int j) { return j == n_tiles - 1 ? dead_hi_last : BN; };
    auto has_dead = [&](int j) { return dead_lo_of(j) > 0 || dead_hi_of(j) < BN; };

    if (tid == 0) {
        for (int s = 0; s < NKV; ++s) {
            mbar_init(smem_u32(&k_full[s]), n_ops);
            mbar_init(smem_u32(&k_empty[s]), RT);
            mbar_init(smem_u32(&v_full[s]), n_ops);
            mbar_init(smem_u32(&v_empty[s]), RT);
        }
        for (int t = 0; t < RT; ++t) {
            mbar_init(smem_u32(&s_full[2 * t]), 1);
            mbar_init(smem_u32(&s_full[2 * t + 1]), 1);
            mbar_init(smem_u32(&p_full[2 * t]), BM);
            mbar_init(smem_u32(&p_full[2 * t + 1]), BM);
            mbar_init(smem_u32(&pv_done[t]), 1);
            mbar_init(smem_u32(&o_done[t]), 1);
        }
        mbar_init(smem_u32(q_full), RT * BM);
        mbar_init(smem_u32(v_clean), BM);
        *bail = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_fence_before();
    __syncthreads();
    fb_pdl_launch_dependents();                                 // (behind the allocation: see umma.cuh)
    tmem_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    fb_pdl_wait();                                              // from here on: Q and the cache

    // a wait that ran out anywhere ends every loop of the CTA
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        if (mbar_try_wait(smem_u32(bar), parity)) return true;  // a wait that passes costs one round trip to shared memory
        if (*(volatile int*)bail) return false;
        if (mbar_wait(smem_u32(bar), parity, a.status)) return true;
        *(volatile int*)bail = 1;
        return false;
    };

    if (warp == 0) {
        // ================= fetch: lane l copies (page l / CB, column block l % CB) of every K and V tile ==========
        // K tiles and V tiles run through rings of their own: a K slot is free as soon as its scores are computed
        // (a tile ahead of the softmax), a V slot after the tile's products, so a copy has two tiles' time to land.
        // Page ids come from the block table 32 at a time (one per lane, the next 32 already on their way), so a
        // tile does not wait for the table: -2 = nothing to fetch (no query of the CTA sees the page), -1 = the
        // table has no page although one is needed.
        const int first_entry = k_begin / a.page_size - table_base_of(a, seq);   // the table entry of tile 0's first page
        auto entries = [&](int block) -> int {                  // table entries first_entry + 32 * block + lane
            const int e = first_entry + 32 * block + lane;      // (below 0: a page before the row's first, never needed)
            return (e >= 0 && e < a.table_stride) ? table[e] : -1;
        };
        int ids_block = 0, ids_cur = entries(0), ids_next = entries(1);
        auto lookup = [&](int j) -> int {
            const int rel = j * pages_per_tile + lane / CB;     // this lane's page of tile j, counted from tile 0
            const int block = (j * pages_per_tile) / 32;        // the same for all lanes: a tile's pages share a block
            if (block != ids_block) {                           // tiles come in order: the next block
                ids_cur = ids_next;
                ids_next = entries(block + 1);
                ids_block = block;
            }
            const int page = __shfl_sync(0xffffffffu, ids_cur, rel & 31);
            if (lane >= n_ops || j >= n_tiles) return -2;
            const int t_first = k_begin + rel * a.page_size;
            if (!(t_first + a.page_size > t_lo && t_first < k_end)) return -2;
            return (page < 0 || page >= a.n_pages) ? -1 : page;
        };
        auto issue = [&](uint8_t* tile, const CUtensorMap* map, uint64_t* full, int page) {
            if (lane >= n_ops) return;
            const uint32_t bar = smem_u32(full);
            if (page >= 0) {
                const int cb = lane % CB, pj = lane / CB;
                mbar_expect_tx(bar, (uint32_t)(a.page_size * 128));
                tma_load_2d(smem_u32(tile + cb * (BN * 128) + pj * a.page_size * 128), map, bar, cb * 64,
                            (page * a.nkv + kvh) * a.page_size);
            } else {
                if (page == -1) atomicOr(a.status, FB_STATUS_BAD_PAGE);
                mbar_arrive(bar);                               // whatever lies in the slot stays; it is masked
            }
        };
        int page = lookup(0);
        for (int j = 0; j < n_tiles; ++j) {
            const int s = j % NKV;
            const uint32_t reuse = (uint32_t)(j / NKV - 1) & 1u;
            if constexpr (SHARED) {                             // (the tile's product is the last to read it)
                if (j >= NKV && !wait(&v_empty[s], reuse)) break;
                issue(Ks + s * SM::KV_BYTES, &a.map_k, &k_full[s], page);
            } else {
                if (j >= NKV && !wait(&k_empty[s], reuse)) break;
                issue(Ks + s * SM::KV_BYTES, &a.map_k, &k_full[s], page);
                if (j >= NKV && !wait(&v_empty[s], reuse)) break;
                issue(Vs + s * SM::KV_BYTES, &a.map_v, &v_full[s], page);
            }
            page = lookup(j + 1);                               // in flight while this warp waits for the next slot
        }
    } else if (warp < 4) {
        // ================= MMA issue: warp 1 for row tile 0, warp 2 for row tile 1 =================
        // Scores run two key tiles ahead of the softmax (two buffers per row tile), so a row tile's softmax never
        // waits for the tensor pipe.  Per key tile: O += P V, then the scores of the tile after next into the
        // columns P lay in (the MMAs of one thread run in the order of their issue, so the product has read P by
        // then), then every commit of the step at one point.  Measured on one SM with back-to-back instructions:
        // a thread that issues MMAs runs in step with the tensor pipe (its queue is a few instructions deep), so
        // the pipe stands still while that thread waits for a barrier, and every point of the instruction stream
        // where tcgen05.commit stands costs the pipe about 170 cycles, however many commits stand there.  Hence a
        // thread for each row tile (the pipe has the other's MMAs meanwhile), the waits for K and V ahead of the
        // wait for P (they pass at once unless the cache is late), and one point of commits per key tile.
        const int t = warp - 1;
        if (t < RT && elect_one()) {
            constexpr uint32_t idesc_s = umma_idesc(BN);
            constexpr uint32_t idesc_o = umma_idesc(HD, true);
            const uint32_t q_addr = smem_u32(Qs + t * (DIFF ? BM * 128 : SM::Q_BYTES));
            auto issue_s = [&](int j) {                         // S buffer j & 1 of the row tile = Q_t K_j^T
                const uint32_t k_addr = smem_u32(Ks + (j % NKV) * SM::KV_BYTES + (DIFF ? t * (BN * 128) : 0));
                const uint32_t d = tmem_base + (uint32_t)((2 * t + (j & 1)) * BN);
#pragma unroll
                for (int kk = 0; kk < (DIFF ? 64 : HD) / UMMA_K; ++kk)
                    umma_bf16(d, umma_desc(q_addr + (uint32_t)((kk / 4) * (BM * 128) + (kk % 4) * 32)),
                              umma_desc(k_addr + (uint32_t)((kk / 4) * (BN * 128) + (kk % 4) * 32)), idesc_s,
                              kk > 0 ? 1u : 0u);
            };
            bool ok = wait(q_full, 0);
            for (int j = 0; ok && j < 2 && j < n_tiles; ++j) {
                ok = wait(&k_full[j % NKV], (uint32_t)(j / NKV) & 1u);
                if (!ok) break;
                tmem_fence_after();
                issue_s(j);
                umma_commit(smem_u32(&s_full[2 * t + (j & 1)]));
                if (!SHARED) umma_commit(smem_u32(&k_empty[j % NKV]));
            }
            for (int j = 0; ok && j < n_tiles; ++j) {
                const bool more = j + 2 < n_tiles;              // there are scores left to compute
                if (!SHARED) ok = wait(&v_full[j % NKV], (uint32_t)(j / NKV) & 1u);
                if (ok && more) ok = wait(&k_full[(j + 2) % NKV], (uint32_t)((j + 2) / NKV) & 1u);
                // (the barrier's first phase is tile 0's clearing if tile 0 has rows to clear, else the last tile's)
                if (ok && t > 0 && has_dead(j)) ok = wait(v_clean, (j > 0 && has_dead(0)) ? 1u : 0u);
                if (ok) ok = wait(&p_full[2 * t + (j & 1)], (uint32_t)(j >> 1) & 1u);
                if (!ok) break;
                tmem_fence_after();
                const uint32_t v_addr = smem_u32(Vs + (j % NKV) * SM::KV_BYTES);
                const uint32_t p_addr = tmem_base + (uint32_t)((2 * t + (j & 1)) * BN);     // bf16 pairs over the scores
                const uint32_t d = tmem_base + (uint32_t)(RT * 128 + t * 128);
#pragma unroll
                for (int kk = 0; kk < BN / UMMA_K; ++kk) {      // 16 keys = 8 columns of P each
                    const uint64_t db = umma_desc_mn(v_addr + (uint32_t)(kk * 16 * 128), BN * 128, 1024);
                    umma_bf16_ts(d, p_addr + (uint32_t)(kk * 8), db, idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
                    if (HILO) umma_bf16_ts(d, p_addr + (uint32_t)(BN / 2 + kk * 8), db, idesc_o, 1u);
                    if (W::PARTS == 3) umma_bf16_ts(d, tmem_base + (uint32_t)(W::third(t, j & 1) + kk * 8), db, idesc_o, 1u);
                }
                if (more) issue_s(j + 2);
                umma_commit(smem_u32(&pv_done[t]));
                if (j == n_tiles - 1) umma_commit(smem_u32(&o_done[t]));
                umma_commit(smem_u32(&v_empty[j % NKV]));
                if (more) {
                    umma_commit(smem_u32(&s_full[2 * t + (j & 1)]));
                    if (!SHARED) umma_commit(smem_u32(&k_empty[(j + 2) % NKV]));
                }
            }
        }
        __syncwarp();
    } else {
        // ================= softmax: thread = query row = tensor-memory lane; warps 4..7 row tile 0, 8..11 row tile 1 =====
        const int quarter = warp & 3;                           // the lanes this warp may read
        const int t = (warp - 4) >> 2;                          // its row tile
        const int r = (DIFF ? 0 : t * BM) + quarter * 32 + lane;   // row of the CTA
        const bool valid = r < rows_valid;
        const int token = q_start + tok0 + r / G, head = kvh * G + r % G;
        // ---- stage Q (zero rows beyond the CTA's share) ----
        {
            const __nv_bfloat16* src = a.q + (size_t)token * a.q_stride + (size_t)head * hd + (DIFF ? t * 64 : 0);
            uint8_t* qrow = Qs + t * (DIFF ? BM * 128 : SM::Q_BYTES) + (quarter * 32 + lane) * 128;
#pragma unroll
            for (int c = 0; c < (DIFF ? 64 : HD) / 8; ++c) {
                uint4 v = make_uint4(0, 0, 0, 0);
                if (valid) v = *reinterpret_cast<const uint4*>(src + c * 8);
                *reinterpret_cast<uint4*>(qrow + (c / 8) * (BM * 128) + (((c & 7) ^ (r & 7)) << 4)) = v;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(smem_u32(q_full));
        }
        const int p_row = valid ? pos0 + tok0 + r / G : -1;     // a row beyond the share sees nothing
        const int t0_row = valid ? fb_first_key(p_row, a.window, DIFF ? a.chunk : 0) : 0;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t o_addr = lane_addr + (uint32_t)(RT * 128 + t * 128); // O of this row
        float m_ref = -INFINITY;                                // reference point of the exponentials (scaled, base 2)
        float l = 0.0f;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int tile_start = k_begin + j * BN;
            const uint32_t s_addr = lane_addr + (uint32_t)((2 * t + (j & 1)) * BN);   // S, and P over it, of this row
            ok = ok && __all_sync(0xffffffffu, wait(&s_full[2 * t + (j & 1)], (uint32_t)(j >> 1) & 1u));
            if (!ok) continue;
            tmem_fence_after();
            // every key of the tile is visible to every row of the warp, or each is compared
            const bool plain = __all_sync(0xffffffffu, tile_start + BN - 1 <= p_row && tile_start >= t0_row);
            // ---- the row's 64 scores into registers (one round trip), masked where needed; their maximum ----
            uint32_t v[BN / 32][32];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tmem_ld32_nowait(s_addr + (uint32_t)(c * 32), v[c]);
            tmem_wait_ld();
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (plain) {
#pragma unroll
                for (int c = 0; c < BN / 32; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[c][i]));
            } else {
#pragma unroll
                for (int c = 0; c < BN / 32; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = tile_start + c * 32 + i;
                        if (!(key >= t0_row && key <= p_row)) v[c][i] = 0xff800000u;      // -inf
                        mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[c][i]));
                    }
            }
            const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * a.scale_log2e);
            if (j == 0) {
                m_ref = m_new;                                  // O is overwritten by the first product
            } else if (__any_sync(0xffffffffu, m_new > m_ref + W::RESCALE_STEP || (m_ref == -INFINITY && m_new > m_ref))) {
                // move the reference point: O *= 2^(old - new), for the whole warp at once.  (The product of tile
                // j - 2 is complete, that of tile j cannot start before this thread is through: the phase asked
                // for is the current one or the one just completed.)
                ok = __all_sync(0xffffffffu, wait(&pv_done[t], (uint32_t)(j - 1) & 1u));
                if (!ok) continue;
                tmem_fence_after();
                const float f = m_new == -INFINITY ? 1.0f : exp2f(m_ref - m_new);
#pragma unroll 1
                for (int c = 0; c < HD / 32; ++c) {
                    uint32_t w[32];
                    tmem_ld32_nowait(o_addr + (uint32_t)(c * 32), w);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * f);
                    tmem_st32(o_addr + (uint32_t)(c * 32), w);
                }
                tmem_wait_st();
                l *= f;
                m_ref = m_new;
            }
            // ---- P = 2^(s - reference), rounded to bfloat16, over the scores it came from: keys 32c .. 32c + 31
            // go to columns 16c .. 16c + 15 ----
            const float neg_ref = m_ref == -INFINITY ? 0.0f : -m_ref;
            float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t pk[16], rest[16], third[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    // a masked score is -inf: 2^-inf = 0
                    const float p0 = fast_exp2(fmaf(__uint_as_float(v[c][2 * i]), a.scale_log2e, neg_ref));
                    const float p1 = fast_exp2(fmaf(__uint_as_float(v[c][2 * i + 1]), a.scale_log2e, neg_ref));
                    sum4[i & 3] += p0 + p1;
                    pk[i] = pack_bf16(p0, p1);
                    if (HILO) {
                        const float r0 = p0 - bf16_low(pk[i]), r1 = p1 - bf16_high(pk[i]);
                        rest[i] = pack_bf16(r0, r1);
                        if (W::PARTS == 3) third[i] = pack_bf16(r0 - bf16_low(rest[i]), r1 - bf16_high(rest[i]));
                    }
                }
                tmem_st16(s_addr + (uint32_t)(c * 16), pk);
                if (HILO) tmem_st16(s_addr + (uint32_t)(BN / 2 + c * 16), rest);
                if (W::PARTS == 3) tmem_st16(lane_addr + (uint32_t)(W::third(t, j & 1) + c * 16), third);
            }
            l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            if (t == 0 && has_dead(j)) {                        // (only the first and the last tile can)
                const int dead_lo = dead_lo_of(j), dead_hi = dead_hi_of(j);
                ok = __all_sync(0xffffffffu, wait(SHARED ? &k_full[j % NKV] : &v_full[j % NKV], (uint32_t)(j / NKV) & 1u));
                if (!ok) continue;
                uint8_t* vt = Vs + (j % NKV) * SM::KV_BYTES;
                const int n_dead = dead_lo + (BN - dead_hi);
                for (int idx = tid - 128; idx < n_dead * 8 * CB; idx += BM) {
                    const int cb = idx / (n_dead * 8), rest = idx - cb * (n_dead * 8);
                    const int k = rest / 8, row = k < dead_lo ? k : dead_hi + (k - dead_lo);
                    *reinterpret_cast<uint4*>(vt + cb * (BN * 128) + row * 128 + (rest & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (RT > 1) mbar_arrive(smem_u32(v_clean));
            }
            tmem_wait_st();
            tmem_fence_before();
            mbar_arrive(smem_u32(&p_full[2 * t + (j & 1)]));
        }
        // ---- O / l, written as bfloat16 ----
        // (a barrier of its own: pv_done may be one or two phases on by now, and a wait names a phase by its parity)
        if (ok) ok = __all_sync(0xffffffffu, wait(&o_done[t], 0));
        if constexpr (DIFF) {
            // out = (a_1 - lambda a_2) / rms * out_scale * gate with a_m = O_m / l_m: this thread's half of the columns
            float* inv_of = reinterpret_cast<float*>(tail + 256);       // [2 maps][128 rows]
            float* squares = inv_of + 2 * BM;                           // [2 halves][128 rows]
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            inv_of[t * BM + r] = inv;
            if (ok) ok = __all_sync(0xffffffffu, wait(&o_done[1 - t], 0));
            asm volatile("bar.sync 1, 256;" ::: "memory");
            tmem_fence_after();
            const float inv1 = inv_of[r], inv2 = a.lambda * inv_of[BM + r];
            const uint32_t o1 = lane_addr + (uint32_t)(RT * 128 + t * 64), o2 = o1 + 128;
            float d[64], ss = 0.0f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t v1[32], v2[32];
                tmem_ld32_nowait(o1 + (uint32_t)(c * 32), v1);
                tmem_ld32_nowait(o2 + (uint32_t)(c * 32), v2);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    d[c * 32 + i] = __uint_as_float(v1[i]) * inv1 - inv2 * __uint_as_float(v2[i]);
                    ss = fmaf(d[c * 32 + i], d[c * 32 + i], ss);
                }
            }
            squares[t * BM + r] = ss;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (ok && valid) {
                const float f = a.out_scale * (a.row_gate ? a.row_gate[(size_t)token * a.nh + head] : 1.0f) /
                                sqrtf((squares[r] + squares[BM + r]) * (1.0f / HD) + a.eps);
                __nv_bfloat16* dst = a.out + (size_t)token * a.out_stride + (size_t)head * HD + t * 64;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[e] = pack_bf16(d[8 * c + 2 * e] * f, d[8 * c + 2 * e + 1] * f);
                    *reinterpret_cast<uint4*>(dst + 8 * c) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        } else if constexpr (SPLIT) {
            if (ok) {
                tmem_fence_after();
                const size_t at = (size_t)blockIdx.x * a.split_rows + r;
                if (valid) *reinterpret_cast<float2*>(a.part_ml + 2 * at) = make_float2(m_ref, l);
                float* po = a.part_o + at * HD;
#pragma unroll
                for (int c = 0; c < HD / 32; ++c) {
                    uint32_t v[32];
                    tmem_ld32_nowait(o_addr + (uint32_t)(c * 32), v);
                    tmem_wait_ld();
                    if (valid) {
#pragma unroll
                        for (int e = 0; e < 32; e += 4)
                            *reinterpret_cast<uint4*>(po + c * 32 + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
                    }
                }
            }
        } else if (ok) {
            tmem_fence_after();
            l += sink_term(a, head, m_ref);
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            __nv_bfloat16* dst = a.out + (size_t)token * a.out_stride + (size_t)head * hd;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) {
                uint32_t v[32];
                tmem_ld32_nowait(o_addr + (uint32_t)(c * 32), v);
                tmem_wait_ld();
                if (valid) {
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = pack_bf16(__uint_as_float(v[8 * q4 + 2 * e]) * inv,
                                             __uint_as_float(v[8 * q4 + 2 * e + 1]) * inv);
                        *reinterpret_cast<uint4*>(dst + c * 32 + q4 * 8) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 1) {
        tmem_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// One warp per (pair, row) of sequences whose keys were cut into stretches: their results made one.
template <int HD>
__global__ void __launch_bounds__(128)
attention_tc_merge_kernel(const __grid_constant__ AttnArgs a) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int pair = item / a.split_rows, r = item - pair * a.split_rows, seq = pair / a.nkv, kvh = pair - seq * a.nkv;
    if (seq >= a.n_seqs) return;
    const int G = a.nh / a.nkv, q_len = a.seq_q_len[seq], pos0 = a.seq_pos_start[seq];
    if (q_len * G > a.short_rows || r >= q_len * G) return;
    const int k_begin = fb_first_key(pos0, a.window, 0) / BN * BN, n_tiles = (pos0 + q_len - k_begin + BN - 1) / BN;
    const int per = split_tiles(n_tiles, a.k_splits), chunks = (n_tiles + per - 1) / per;
    const size_t slot0 = ((size_t)pair * a.k_splits) * a.split_rows + r;
    float m = -INFINITY;
    for (int s = lane; s < chunks; s += 32) m = fmaxf(m, a.part_ml[2 * (slot0 + (size_t)s * a.split_rows)]);
    m = fb_warp_max(m);
    float acc[HD / 32], l = 0.0f;
#pragma unroll
    for (int i = 0; i < HD / 32; ++i) acc[i] = 0.0f;
    if (m > -INFINITY) {
#pragma unroll 4
        for (int s = 0; s < chunks; ++s) {
            const size_t at = slot0 + (size_t)s * a.split_rows;
            const float2 ml = *reinterpret_cast<const float2*>(a.part_ml + 2 * at);
            const float w = exp2f(ml.x - m);                    // 0 where a stretch saw nothing
            l = fmaf(w, ml.y, l);
#pragma unroll
            for (int i = 0; i < HD / 128; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(a.part_o + at * HD + 128 * i + 4 * lane);
                acc[4 * i] = fmaf(w, v.x, acc[4 * i]); acc[4 * i + 1] = fmaf(w, v.y, acc[4 * i + 1]);
                acc[4 * i + 2] = fmaf(w, v.z, acc[4 * i + 2]); acc[4 * i + 3] = fmaf(w, v.w, acc[4 * i + 3]);
            }
        }
    }
    const int token = a.seq_q_start[seq] + r / G, head = kvh * G + r % G;
    l += sink_term(a, head, m);
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    __nv_bfloat16* dst = a.out + (size_t)token * a.out_stride + (size_t)head * HD;
#pragma unroll
    for (int i = 0; i < HD / 128; ++i)
        *reinterpret_cast<uint2*>(dst + 128 * i + 4 * lane) = make_uint2(pack_bf16(acc[4 * i] * inv, acc[4 * i + 1] * inv),
                                                                         pack_bf16(acc[4 * i + 2] * inv, acc[4 * i + 3] * inv));
}

template <int HD, int RT, bool HILO, bool SHARED, bool DIFF = false, bool SPLIT = false>
int launch_tc(const AttnArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    auto kern = attention_tc_kernel<HD, RT, HILO, SHARED, DIFF, SPLIT>;
    using SM = TcSmem<HD, RT, SHARED, DIFF>;
    static bool configured[FB_MAX_DEVICES] = {};
    if (fb_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::BYTES);
        if (e != cudaSuccess) return fb_fail(-2, "attention_tc: cannot reserve %d bytes of shared memory: %s",
                                             SM::BYTES, cudaGetErrorString(e));
        fb_setup_done(configured);
    }
    const int TQ = (DIFF ? 1 : RT) * BM / (a.nh / a.nkv);
    const dim3 grid(SPLIT ? n_seqs * a.nkv * a.k_splits : ((max_q_len + TQ - 1) / TQ) * a.nkv * portion_seqs(a));
    fb_launch_class(FB_LAUNCH_ATTENTION_TC, (kern), grid, tc_threads(RT), (size_t)SM::BYTES, stream, a);
    return fb_check_launch("attention_tc");
}

// Two row tiles per CTA when that still gives every SM a CTA, else one.
template <int HD, bool HILO>
int launch_tc(const AttnArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    const int sms = fb_sm_count();
    const int TQ2 = 2 * BM / (a.nh / a.nkv);
    const long ctas2 = (long)((max_q_len + TQ2 - 1) / TQ2) * a.nkv * portion_seqs(a);   // an upper bound: short ones leave early
    return ctas2 >= sms ? launch_tc<HD, 2, HILO, false>(a, n_seqs, max_q_len, stream)
                        : launch_tc<HD, 1, HILO, false>(a, n_seqs, max_q_len, stream);
}

template <bool HILO>
int launch_tc(const AttnArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    return a.hd == 64    ? launch_tc<64, HILO>(a, n_seqs, max_q_len, stream)
           : a.hd == 128 ? launch_tc<128, HILO>(a, n_seqs, max_q_len, stream)
                         : launch_tc<256, 1, HILO, true>(a, n_seqs, max_q_len, stream);
}

}  // namespace

bool fb_attention_tc_takes(const AttnArgs& a, bool tma) {
    const int G = a.nh / a.nkv;
    // (it does not walk kept first keys behind a window, cap scores or gate heads)
    return tma && !a.score_slopes && a.keep_first == 0 && a.cap_log2e == 0.0f && !a.head_gate &&
           (a.hd == 64 || a.hd == 128 || (a.hd == 256 && a.k_pool == a.v_pool)) && G <= BM && BN % a.page_size == 0 &&
           a.out_stride % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
}

int fb_launch_attention_tc(const AttnArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    return a.weights_hi_lo ? launch_tc<true>(a, n_seqs, max_q_len, stream) : launch_tc<false>(a, n_seqs, max_q_len, stream);
}

// Differential attention over portions: maps of 64, values of 128, pages that tile 64 keys, rows that leave in 16-byte pieces.
bool fb_diff_attention_tc_takes(int nh, int nkv, int kd, int vd, int page_size, const void* out, long out_stride) {
    return kd == 64 && vd == 128 && nh / nkv <= BM && page_size >= 8 && page_size <= BN && BN % page_size == 0 &&
           out_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
}

int fb_launch_diff_attention_tc(const AttnArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    return launch_tc<128, 2, true, false, true>(a, n_seqs, max_q_len, stream);
}

// Decoded tokens (rows up to 16 a stretch of heads, short_rows in all) over rows of 256 that are keys and values at once.
// Measured with 8 sequences of 8,172 rows and 32 heads: 54 us on the split-key kernel, which fetches a row four times (as key
// and as value, for two stretches of 16 heads), 25 here with the merge.  A layer of 1 to 64 sequences of 60 to 8,000 rows takes
// 0.58 to 0.99 of the time with 32 heads and 0.71 to 1.00 with 16; no size was found where the split-key kernel is faster.
bool fb_attention_tc_split_takes(const AttnArgs& a, bool tma) { return a.hd == 256 && fb_attention_tc_takes(a, tma) && a.short_rows <= BM; }

// Into how many stretches the keys of a sequence are cut, at most `most`: the count whose rounds of CTAs (one a
// multiprocessor) times the tiles of a stretch are fewest, three tiles counted for a CTA's set-up and end; at least three
// stretches where there are tiles for them, so that sequences of different lengths spread.  38 sequences of 8,000 rows, 16
// heads, a layer: four stretches are 152 CTAs and a second round for four of them, 158 us; seven take 125, the
// split-key kernel 136.
FB_API int fb_attention_tc_stretches(long long pairs, int tiles, int most, int sms) {
    int best = 0;
    long long best_cost = 0;
    for (int s = 1; s <= most && s <= 64; ++s) {
        const int per = split_tiles(tiles, s), there = (tiles + per - 1) / per;
        if (there < s) continue;                       // (more stretches than the tiles make)
        if (s < 3 && s < most && split_tiles(tiles, s + 1) < per) continue;
        const long long cost = (pairs * s + sms - 1) / sms * (per + 3);
        if (best == 0 || cost < best_cost) { best = s; best_cost = cost; }
    }
    return best > 0 ? best : most >= 1 ? 1 : 0;
}

// part: room for partial results, `floats` of them; 1 where it does not do (nothing was launched).
int fb_launch_attention_tc_split(AttnArgs& a, int n_seqs, int max_kv_len, float* part, long long floats, cudaStream_t stream) {
    const long pairs = (long)n_seqs * a.nkv;
    a.split_rows = a.short_rows;
    const long long each = pairs * a.split_rows * (a.hd + 2), most = floats / each;
    const int keys = a.window > 0 ? min(max_kv_len, a.window + BM) : max_kv_len;
    const long splits = fb_attention_tc_stretches(pairs, (keys + BN - 1) / BN, (int)(most < 64 ? most : 64), fb_sm_count());
    if (splits < 1) return 1;
    a.k_splits = (int)splits;
    a.part_o = part;
    a.part_ml = part + splits * pairs * a.split_rows * a.hd;
    const int rc = a.weights_hi_lo ? launch_tc<256, 1, true, true, false, true>(a, n_seqs, 1, stream)
                                   : launch_tc<256, 1, false, true, false, true>(a, n_seqs, 1, stream);
    if (rc) return rc;
    fb_launch((attention_tc_merge_kernel<256>), dim3((unsigned)((pairs * a.split_rows + 3) / 4)), dim3(128), 0, stream, a);
    return fb_check_launch("attention_tc_merge");
}
