// What the two kernels of float32 attention (attention_f32.cu on the CUDA cores, attention_f32_tc.cu on the tensor cores) share:
// their arguments, and how stretches of keys are joined.
#pragma once

#include "common.cuh"

#include <type_traits>

namespace {

constexpr int STRETCH = 256;            // keys of a stretch: joined on their own, whoever takes them
constexpr long long SCRATCH_FLOATS = 1LL << 25;      // most that stretches of one launch may leave for joining

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
    int slots, per;                     // stretches that a row's keys have at most, and that a CTA takes
    int part_rows;                      // rows of a pair in the parts of BM 16
    float* part_o; float* part_ml;      // per stretch and row: output x vd, and (maximum, sum); nullptr: a CTA takes all
    int* status;
};

// What a stretch (maximum m, sum l) adds to the stretches before it (M, L): the factors of the output so far and of its own.
struct Join { float before, own; };
__device__ __forceinline__ Join join(float& M, float& L, float m, float l) {
    const float top = fmaxf(M, m);
    Join j;
    j.before = M == -INFINITY ? 0.0f : expf(M - top);
    j.own = m == -INFINITY ? 0.0f : expf(m - top);
    L = fmaf(L, j.before, __fmul_rn(l, j.own));
    M = top;
    return j;
}
__device__ __forceinline__ float joined(const Join& j, float before, float own) { return fmaf(before, j.before, __fmul_rn(own, j.own)); }

// What a row's joined output is multiplied with in the end.
__device__ __forceinline__ float finish(const F32Args& a, int row, int head, float M, float L) {
    float f = 1.0f, sum = L;
    if (a.sinks) {                                               // the slot without key and value
        const float sk = a.sinks[head], top = fmaxf(M, sk);
        f = M == -INFINITY ? 0.0f : expf(M - top);
        sum = fmaf(sum, f, expf(sk - top));
    }
    f = sum > 0.0f ? f / sum : 0.0f;
    if (a.head_gate)
        f /= 1.0f + expf(-fb_slab_sum(a.head_gate + (size_t)row * a.gate_stride, head, a.gate_partials, a.gate_partial_stride));
    return f;
}

// Row r of a CTA, in the parts of a stretch.
template <int BM>
__device__ __forceinline__ size_t part_at(const F32Args& a, int slot, int pair, int row, int head, int r) {
    return BM == 16 ? ((size_t)slot * a.n_seqs * a.nkv + pair) * a.part_rows + r : ((size_t)slot * a.n + row) * a.nh + head;
}

// One warp a row of the CTAs above (blockIdx.y: four rows each): its stretches joined.
template <int BM>
__global__ void __launch_bounds__(128)
attention_f32_join_kernel(const F32Args a) {
    fb_pdl_launch_dependents();
    fb_pdl_wait();
    const int G = a.nh / a.nkv, lane = threadIdx.x & 31, r = blockIdx.y * 4 + (threadIdx.x >> 5);
    const int pair = blockIdx.x / a.token_tiles, tile = blockIdx.x - pair * a.token_tiles;
    const int seq = pair / a.nkv, kvh = pair - seq * a.nkv, q_len = a.seq_q_len[seq];
    if ((q_len * G <= a.short_rows) != (BM == 16)) return;
    const int TQ = BM / G, tok0 = (a.token_tiles - 1 - tile) * TQ;
    if (tok0 >= q_len || r >= min(TQ, q_len - tok0) * G) return;
    const int row = a.seq_q_start[seq] + tok0 + r / G, head = kvh * G + r % G;
    // (a row's stretches are numbered in the order of their positions, the first at most by its own number: those behind the row's
    // position are empty.  A step may have room for many more of them: decoded tokens have it for the longest context.  8 x 32 rows
    // of 100 keys where contexts of 131,072 are allowed: attention 101 us with all of them read, 21 so)
    const int slots = min(a.slots, (a.seq_pos_start[seq] + tok0 + r / G) / STRETCH + 1);
    float M = -INFINITY, L = 0.0f;
    float4 acc[2] = {};
    // Several stretches' numbers on their way at once, four where there are no more: one after the other, 17 of 8 x 32 rows took
    // 18 us, eight at a time 12.
    auto all = [&](auto ahead, auto pieces) {
        constexpr int A = decltype(ahead)::value, P = decltype(pieces)::value;
        for (int s0 = 0; s0 < slots; s0 += A) {
            float2 ml[A];
            float4 x[A][P];
#pragma unroll
            for (int i = 0; i < A; ++i) {
                const size_t at = part_at<BM>(a, min(s0 + i, slots - 1), pair, row, head, r);
                ml[i] = *reinterpret_cast<const float2*>(a.part_ml + 2 * at);
#pragma unroll
                for (int c = 0; c < P; ++c) x[i][c] = *reinterpret_cast<const float4*>(a.part_o + at * a.vd + min(4 * lane + 128 * c, a.vd - 4));
            }
#pragma unroll
            for (int i = 0; i < A; ++i) {
                if (s0 + i >= slots || (ml[i].x == -INFINITY && ml[i].y == 0.0f)) continue;    // nothing was seen there (and nothing left)
                const Join j = join(M, L, ml[i].x, ml[i].y);
#pragma unroll
                for (int c = 0; c < P; ++c)
                    acc[c] = make_float4(joined(j, acc[c].x, x[i][c].x), joined(j, acc[c].y, x[i][c].y), joined(j, acc[c].z, x[i][c].z),
                                         joined(j, acc[c].w, x[i][c].w));
            }
        }
    };
    const std::integral_constant<int, 1> one;
    const std::integral_constant<int, 2> two;
    const std::integral_constant<int, 4> four;
    const std::integral_constant<int, 8> eight;
    if (a.vd > 128) all(four, two);
    else if (slots > 4) all(eight, one);
    else all(four, one);
    const float f = finish(a, row, head, M, L);
    float* op = a.out + (size_t)row * a.out_stride + (size_t)head * a.vd;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int d = 4 * lane + 128 * c;
        if (d < a.vd) *reinterpret_cast<float4*>(op + d) = make_float4(acc[c].x * f, acc[c].y * f, acc[c].z * f, acc[c].w * f);
    }
}

// (vd + 2 floats a row are no multiple of 16 bytes, the outputs are read by 16)
long long border4(long long floats) { return (floats + 3) / 4 * 4; }

}  // namespace
