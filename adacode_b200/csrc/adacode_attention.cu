// Fused unpack + single-query ("decode") attention over a float11-packed KV cache.
//
// The packed planes are read straight from HBM (1 + n/8 + p bytes per cached element instead of
// 2 for dense bf16), decoded tile by tile on the chip, and consumed there: scores against
// the G query heads that share a KV head, online softmax in fp32, weighted sum of the decoded V
// tile.  The cache is split along the sequence (flash-decoding): each CTA owns a run of 128-token tiles of one
// (batch, kv head), or of several that follow each other, and leaves (max, sum, numerator)
// partials that a second kernel combines.  Every call takes the pipelined tensor-core kernel, which decodes in
// registers.  The plain one, which comes first, is a second opinion on it for tests and for failure analysis, with
// other arithmetic (fp32 on the CUDA cores) and another decode (tables, tiles in shared memory); it runs only with
// ADACODE_ATTN_SIMPLE=1.
//
// The reference has no such kernel (its attention path materialises dense K/V first; the module
// its validation script imports, ops/kv_attention.py, is absent from its tree), so numerics are
// checked against an fp32 PyTorch attention over the dense cache.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "adacode.h"

#include <stdlib.h>

#include <atomic>
#include <mutex>

namespace {

#include "adacode_device.cuh"
#define ADACODE_PIPELINE_UNPACK_ONLY
#include "adacode_pipeline.cuh"

constexpr int kAttnThreads = 128;
constexpr int kTileTokens = 128;
constexpr int kMaxGroup = 8;      // query heads per KV head
constexpr int kMaxD = 128;

struct AttnArgs {
    const uint16_t *q;            // [B][Hq][D]
    long long q_sb, q_sh;
    const adacode_segment *kseg, *vseg;
    int n_seg;
    const uint16_t *k_tail, *v_tail;   // dense residual [B][Hkv][tail_len][D]
    int tail_len;
    long long t_sb, t_sh, t_ss;
    int B, Hq, Hkv, G, D;
    float scale;
    int n_splits;                 // partial results kept per (batch, KV head): as many as its row is cut into, or more
    float *part_o;                // [B*Hkv][splits][G][D]
    float *part_ml;               // [B*Hkv][splits][G][2]
    int32_t *status;
    // The work is rows (batch, KV head, group of query heads) of `items` tiles each, one after the other.  A CTA takes a
    // run of consecutive items: every `cut_items` of them are cut into `cut_ctas` runs, the r-th from cut_items r / cut_ctas
    // on.  cut_items is either one row (whole splits) or all rows together, in which case a run may end in one row
    // and go on in the next.  (cut_items x cut_ctas < 2**31)
    int items, head_groups, heads_per_row;
    int cut_items, cut_ctas;
    Quotient by_items, by_head_groups, by_heads, by_cut_items, by_cut_ctas;      // (by_heads: Hkv)
};

// Item at which the run of CTA c begins, and the CTA whose run holds item x.
__device__ __forceinline__ int run_begin(const AttnArgs &a, int c) {
    const int cut = (uint32_t)c / a.by_cut_ctas, r = c - cut * a.cut_ctas;
    return cut * a.cut_items + (int)((uint32_t)(a.cut_items * r) / a.by_cut_ctas);
}
__device__ __forceinline__ int cta_of(const AttnArgs &a, int x) {
    const int cut = (uint32_t)x / a.by_cut_items, y = x - cut * a.cut_items;
    return cut * a.cut_ctas + (int)((uint32_t)((y + 1) * a.cut_ctas - 1) / a.by_cut_items);
}

struct AttnSmem {
    alignas(16) uint8_t sm[kTileTokens * kMaxD];          // staged sign/mantissa plane of one tile
    alignas(16) uint8_t codes[kTileTokens * kMaxD / 2];   // staged code plane
    alignas(16) uint16_t tile[kTileTokens * (kMaxD + 2)]; // decoded (or dense) tile, rows padded by 2
    alignas(16) float q[kMaxGroup][kMaxD];
    alignas(16) float p[kTileTokens][kMaxGroup];       // softmax numerators, [token][query head]
    alignas(16) uint32_t lut[2][1024];                    // decode tables: [0] keys, [1] values
    int lut_left[2], lut_nbits[2];
    float red[kMaxGroup][4];
    int scan[4];
};

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Decode tile `bh` of one packed segment into s.tile (row stride D + 2 elements).
template <int N>
__device__ __forceinline__ void decode_tile(AttnSmem &s, const adacode_segment &sg, int bh, int D, const uint32_t *lut,
                                            int32_t *status) {
    constexpr int CB = 2 * N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile_elems = kTileTokens * D;
    const int chunks = tile_elems >> 4;
    const int per_thread = chunks / kAttnThreads;             // 8 at D = 128, 4 at D = 64
    const uint8_t *gsm = sg.sign_mant + (long long)bh * tile_elems;
    const uint8_t *gcd = sg.codes + (long long)bh * (tile_elems * N / 8);
    // stage both planes with coalesced 16-byte loads
    for (int i = tid; i < tile_elems / 16; i += kAttnThreads)
        reinterpret_cast<uint4 *>(s.sm)[i] = __ldg(reinterpret_cast<const uint4 *>(gsm) + i);
    for (int i = tid; i < tile_elems * N / 128; i += kAttnThreads)
        reinterpret_cast<uint4 *>(s.codes)[i] = __ldg(reinterpret_cast<const uint4 *>(gcd) + i);
    __syncthreads();

    // pass 1: escapes in this thread's run of chunks, then an exclusive scan over the block
    const int c0 = tid * per_thread;
    int cnt = 0;
    for (int k = 0; k < per_thread; ++k) {
        uint32_t g[2];
        load_chunk_codes<N, 16>(s.codes + (c0 + k) * CB, g);
        cnt += __popc(zero_slots<N>(g[0])) + __popc(zero_slots<N>(g[1]));
    }
    int x = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += u;
    }
    if (lane == 31) s.scan[warp] = x;
    __syncthreads();
    int rank = x - cnt;
    for (int i = 0; i < warp; ++i) rank += s.scan[i];
    const long long esc0 = bh > 0 ? sg.tile_base[bh - 1] : 0;

    // pass 2: decode, write the padded rows, patch escapes
    const int row_stride = D + 2;
    for (int k = 0; k < per_thread; ++k) {
        const int c = c0 + k;
        uint32_t g[2];
        load_chunk_codes<N, 16>(s.codes + c * CB, g);
        const uint4 sv = *reinterpret_cast<const uint4 *>(s.sm + c * 16);
        const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
        const int e0 = c * 16;
        const int row = e0 / D, col = e0 - row * D;
        uint32_t *dst = reinterpret_cast<uint32_t *>(s.tile + row * row_stride + col);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t ew[4];
            decode_group<N>(lut, g[q], ew);
            const uint32_t s0 = sw[2 * q], s1 = sw[2 * q + 1];
            dst[4 * q + 0] = ew[0] | (__byte_perm(s0, 0u, 0x1100) & 0x807F807Fu);
            dst[4 * q + 1] = ew[1] | (__byte_perm(s0, 0u, 0x3322) & 0x807F807Fu);
            dst[4 * q + 2] = ew[2] | (__byte_perm(s1, 0u, 0x1100) & 0x807F807Fu);
            dst[4 * q + 3] = ew[3] | (__byte_perm(s1, 0u, 0x3322) & 0x807F807Fu);
        }
        uint16_t *row16 = reinterpret_cast<uint16_t *>(dst);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t z = zero_slots<N>(g[q]);
            while (z) {
                const int pos = 31 - __clz(z);
                z ^= 1u << pos;
                const int el = q * 8 + 7 - pos / N;
                uint32_t e = 0;
                const long long idx = esc0 + rank;
                if (idx < sg.escapes_len) e = sg.escapes[idx];
                else atomicOr(status, ADACODE_STATUS_ESCAPE_UNDERRUN);
                ++rank;
                row16[el] = (uint16_t)((row16[el] & 0x807Fu) | (e << 7));
            }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void decode_dispatch(AttnSmem &s, const adacode_segment &sg, int bh, int D, int which,
                                                int32_t *status) {
    if (s.lut_nbits[which] != sg.nbits || s.lut_left[which] != sg.left) {
        __syncthreads();
        build_decode_lut(s.lut[which], sg.nbits, sg.left, kAttnThreads);
        if (threadIdx.x == 0) {
            s.lut_nbits[which] = sg.nbits;
            s.lut_left[which] = sg.left;
        }
        __syncthreads();
    }
    switch (sg.nbits) {
        case 1: decode_tile<1>(s, sg, bh, D, s.lut[which], status); break;
        case 2: decode_tile<2>(s, sg, bh, D, s.lut[which], status); break;
        case 3: decode_tile<3>(s, sg, bh, D, s.lut[which], status); break;
        default: decode_tile<4>(s, sg, bh, D, s.lut[which], status); break;
    }
}

// Dense tile from the residual: rows [t0, t0 + 128) of `base`, zero beyond `len`.
__device__ __forceinline__ void load_dense_tile(AttnSmem &s, const uint16_t *base, long long ss, int t0, int len, int D) {
    const int row_stride = D + 2;
    const int words_per_row = D / 2;
    for (int i = threadIdx.x; i < kTileTokens * words_per_row; i += kAttnThreads) {
        const int row = i / words_per_row, w = i - row * words_per_row;
        uint32_t v = 0;
        if (t0 + row < len) v = *reinterpret_cast<const uint32_t *>(base + (long long)(t0 + row) * ss + 2 * w);
        *reinterpret_cast<uint32_t *>(s.tile + row * row_stride + 2 * w) = v;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kAttnThreads) k_decode_attn(const AttnArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    AttnSmem &s = *reinterpret_cast<AttnSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (it always takes whole splits)
    const int r = blockIdx.x / a.n_splits, split = blockIdx.x - r * a.n_splits;
    const int bh = r / a.head_groups;
    const int b = bh / a.Hkv, hkv = bh - b * a.Hkv;
    // query heads of the group are handled eight at a time
    const int Gt = a.G, gz = (r - bh * a.head_groups) * kMaxGroup;
    const int G = Gt - gz < kMaxGroup ? Gt - gz : kMaxGroup, D = a.D;

    // queries of this KV head's group, as fp32, pre-multiplied by the softmax scale
    for (int i = tid; i < G * D; i += kAttnThreads) {
        const int g = i / D, d = i - g * D;
        const uint16_t raw = a.q[(long long)b * a.q_sb + (long long)(hkv * Gt + gz + g) * a.q_sh + d];
        s.q[g][d] = __uint_as_float((uint32_t)raw << 16) * a.scale;
    }
    for (int i = tid; i < kTileTokens * kMaxGroup; i += kAttnThreads) (&s.p[0][0])[i] = 0.f;
    if (tid == 0) s.lut_nbits[0] = s.lut_nbits[1] = 0;
    __syncthreads();

    const int first = run_begin(a, blockIdx.x) - r * a.items, last = run_begin(a, blockIdx.x + 1) - r * a.items;

    float m[kMaxGroup], l[kMaxGroup], o[kMaxGroup];     // o: column `tid` of the numerator
#pragma unroll
    for (int g = 0; g < kMaxGroup; ++g) m[g] = -INFINITY, l[g] = 0.f, o[g] = 0.f;
    const int row_words = (D + 2) / 2;

    for (int it = first; it < last; ++it) {
        const bool packed = it < a.n_seg;
        const int t0 = packed ? 0 : (it - a.n_seg) * kTileTokens;
        const int valid = packed ? kTileTokens : min(kTileTokens, a.tail_len - t0);
        // ---- K tile -> scores
        if (packed) decode_dispatch(s, a.kseg[it], bh, D, 0, a.status);
        else load_dense_tile(s, a.k_tail + (long long)b * a.t_sb + (long long)hkv * a.t_sh, a.t_ss, t0, a.tail_len, D);
        float sc[kMaxGroup];
#pragma unroll
        for (int g = 0; g < kMaxGroup; ++g) sc[g] = 0.f;
        const uint32_t *krow = reinterpret_cast<const uint32_t *>(s.tile) + tid * row_words;
        for (int j = 0; j < D / 2; ++j) {
            const uint32_t kw = krow[j];
            const float k0 = bf16_lo(kw), k1 = bf16_hi(kw);
#pragma unroll
            for (int g = 0; g < kMaxGroup; ++g)
                if (g < G) sc[g] = fmaf(s.q[g][2 * j], k0, fmaf(s.q[g][2 * j + 1], k1, sc[g]));
        }
        // ---- online softmax over the tile's 128 tokens (thread = token)
#pragma unroll
        for (int g = 0; g < kMaxGroup; ++g) {
            if (g < G) {
                float v = tid < valid ? sc[g] : -INFINITY;
                sc[g] = v;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, d));
                if (lane == 0) s.red[g][warp] = v;
            }
        }
        __syncthreads();
        float alpha[kMaxGroup];
#pragma unroll
        for (int g = 0; g < kMaxGroup; ++g) {
            alpha[g] = 1.f;
            if (g < G) {
                const float tmax = fmaxf(fmaxf(s.red[g][0], s.red[g][1]), fmaxf(s.red[g][2], s.red[g][3]));
                const float mn = fmaxf(m[g], tmax);
                alpha[g] = (m[g] == -INFINITY) ? 0.f : __expf(m[g] - mn);
                const float pv = (sc[g] == -INFINITY) ? 0.f : __expf(sc[g] - mn);
                s.p[tid][g] = pv;
                m[g] = mn;
                sc[g] = pv;
            }
        }
        __syncthreads();          // s.red is read, s.p is written
#pragma unroll
        for (int g = 0; g < kMaxGroup; ++g) {
            if (g < G) {
                float v = sc[g];
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
                if (lane == 0) s.red[g][warp] = v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < kMaxGroup; ++g)
            if (g < G) l[g] = l[g] * alpha[g] + (s.red[g][0] + s.red[g][1] + s.red[g][2] + s.red[g][3]);
        // ---- V tile -> numerator (thread = output column)
        __syncthreads();          // everyone is done with the K tile and s.red
        if (packed) decode_dispatch(s, a.vseg[it], bh, D, 1, a.status);
        else load_dense_tile(s, a.v_tail + (long long)b * a.t_sb + (long long)hkv * a.t_sh, a.t_ss, t0, a.tail_len, D);
        if (tid < D) {
#pragma unroll
            for (int g = 0; g < kMaxGroup; ++g) o[g] *= alpha[g];
            for (int t = 0; t < valid; ++t) {
                const float v = __uint_as_float((uint32_t)s.tile[t * (D + 2) + tid] << 16);
                const float4 p0 = *reinterpret_cast<const float4 *>(&s.p[t][0]);
                const float4 p1 = *reinterpret_cast<const float4 *>(&s.p[t][4]);
                o[0] = fmaf(p0.x, v, o[0]), o[1] = fmaf(p0.y, v, o[1]), o[2] = fmaf(p0.z, v, o[2]), o[3] = fmaf(p0.w, v, o[3]);
                o[4] = fmaf(p1.x, v, o[4]), o[5] = fmaf(p1.y, v, o[5]), o[6] = fmaf(p1.z, v, o[6]), o[7] = fmaf(p1.w, v, o[7]);
            }
        }
        __syncthreads();          // the tile and s.p are reused by the next item
    }

    const long long slot = (long long)bh * a.n_splits + split;
#pragma unroll
    for (int g = 0; g < kMaxGroup; ++g) {
        if (g < G) {
            if (tid < D) a.part_o[(slot * Gt + gz + g) * D + tid] = o[g];
            if (tid == g) {
                a.part_ml[(slot * Gt + gz + g) * 2 + 0] = m[g];
                a.part_ml[(slot * Gt + gz + g) * 2 + 1] = l[g];
            }
        }
    }
}

// The terms of a probability after the first may be 0 or negative (and weights may underflow), so a value that is
// not finite leaves a sum that is not finite but not always the right one (0 x inf, inf - inf).  What is right follows from
// the values alone: NaN for a NaN or for infinities of both signs, the infinity otherwise.  A warp of the combine
// kernel that ends with such sums (`odd`, a column each) looks its columns up here; sums that overflowed stay.
// A block whose window ends below 255 and whose escapes hold no 255 is done with its escape bytes.
template <int D>
__device__ __noinline__ void settle_columns(const AttnArgs &a, int bh, bool odd, unsigned *flags, uint16_t *out) {
    const int lane = threadIdx.x & 31, d0 = threadIdx.x & ~31;
    flags += d0;                                           // this warp's columns: bit 0 inf, bit 1 -inf, bit 2 NaN
    flags[lane] = 0;
    __syncwarp();
    const auto note = [flags, d0](int d, bool negative, bool nan) {
        if ((d & ~31) == d0) atomicOr(flags + (d - d0), nan ? 4u : negative ? 2u : 1u);
    };
    for (int t = 0; t < a.n_seg; ++t) {
        const adacode_segment &sg = a.vseg[t];
        const int nbits = sg.nbits;
        int64_t rank = bh > 0 ? sg.tile_base[bh - 1] : 0;
        int64_t end = sg.tile_base[bh];
        if (end > sg.escapes_len) end = sg.escapes_len;
        bool has = sg.left + (1 << nbits) - 1 >= 255;
#pragma unroll 8
        for (int64_t i = rank + lane; i < end; i += 32) has |= sg.escapes[i] == 255;
        if (!__any_sync(kFull, has)) continue;
        const uint8_t *sm = sg.sign_mant + (int64_t)bh * (kTileTokens * D);
        const uint8_t *codes = sg.codes + (int64_t)bh * (kTileTokens * D / 8 * nbits);
        for (int g = lane; g < kTileTokens * D / 8; g += 32) {           // groups of eight elements
            uint32_t x = 0;
            for (int i = 0; i < nbits; ++i) x = (x << 8) | codes[g * nbits + i];
            int escapes = 0;
            for (int k = 0; k < 8; ++k) escapes += ((x >> (k * nbits)) & ((1u << nbits) - 1)) == 0;
            int incl = escapes;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(kFull, incl, d);
                if (lane >= d) incl += u;
            }
            int64_t r = rank + incl - escapes;
            for (int k = 0; k < 8; ++k) {
                const uint32_t code = (x >> ((7 - k) * nbits)) & ((1u << nbits) - 1);
                uint32_t e = (code + (uint32_t)sg.left) & 0xFFu;
                if (code == 0) e = r < end ? sg.escapes[r] : 0u, ++r;
                const uint8_t b = sm[g * 8 + k];
                if (e == 255) note((g * 8 + k) % D, (b & 0x80) != 0, (b & 0x7F) != 0);
            }
            rank += __shfl_sync(kFull, incl, 31);
        }
    }
    const int b = bh / a.Hkv, hkv = bh - b * a.Hkv;
    const uint16_t *col = a.v_tail + b * a.t_sb + hkv * a.t_sh + d0 + lane;
#pragma unroll 8
    for (int t = 0; t < a.tail_len; ++t) {
        const uint32_t v = col[t * a.t_ss];
        if ((v & 0x7F80u) == 0x7F80u) note(d0 + lane, (v & 0x8000u) != 0, (v & 0x7Fu) != 0);
    }
    __syncwarp();
    const unsigned f = flags[lane];
    if (odd && f != 0) out[lane] = f == 1 ? 0x7F80 : f == 2 ? 0xFF80 : 0x7FFF;
}

// out[b][hq][d] = sum_s w_s o_s / sum_s w_s l_s, w_s = exp(m_s - max m).  One CTA per query head, bound by the
// latency of its reads: the weights of all splits are found at once, and the D columns are summed by
// GROUPS groups of threads that share the splits.  [1, 8, 20480, 128] with 37 splits, attention and combine:
// 47.3 us with one thread per column that walked all splits twice, 43.4 us with four groups.  Up to
// kFewSplits splits the extra threads only cost ([16, 4, 4096, 64] with 16 heads per group, nine splits: 53.9 us
// with one group, 57.0 us with eight).
constexpr int kCombineThreads = 512;
constexpr int kFewSplits = 16;
constexpr int kMaxSplits = 128;

template <int D, int GROUPS>
__global__ void __launch_bounds__(GROUPS * D) k_decode_attn_combine(const __grid_constant__ AttnArgs a, uint16_t *__restrict__ out) {
    __shared__ float s_w[kMaxSplits], s_den[kMaxSplits], s_num[GROUPS][D];
    __shared__ unsigned s_flags[D];
    const float *__restrict__ part_o = a.part_o;
    const float *__restrict__ part_ml = a.part_ml;
    const int G = a.G;
    const int tid = threadIdx.x, lane = tid & 31;
    const int bhq = blockIdx.x;
    const int b = bhq / a.Hq, hq = bhq - b * a.Hq;
    const int hkv = hq / G, g = hq - hkv * G, bh = b * a.Hkv + hkv;
    const long long base = (long long)bh * a.n_splits;
    // parts that this head's row was cut into
    const int x = (bh * a.head_groups + g / a.heads_per_row) * a.items;
    const int n_splits = cta_of(a, x + a.items - 1) - cta_of(a, x) + 1;
    // launched as a programmatic dependent of the attention kernel: wait for its partial results
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float mx = -INFINITY;
    for (int s = lane; s < n_splits; s += 32) mx = fmaxf(mx, part_ml[((base + s) * G + g) * 2]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, d));
    for (int s = tid; s < n_splits; s += GROUPS * D) {
        const float m = part_ml[((base + s) * G + g) * 2], l = part_ml[((base + s) * G + g) * 2 + 1];
        const float w = __expf(m - mx);
        s_w[s] = m == -INFINITY ? -1.f : w;                // (negative: a split without tokens, not read)
        s_den[s] = m == -INFINITY ? l : w * l;             // (without a maximum l is 0, or NaN if all scores are)
    }
    __syncthreads();
    const int d = tid % D, grp = tid / D;
    float num = 0.f;
#pragma unroll 4
    for (int s = grp; s < n_splits; s += GROUPS) {
        const float w = s_w[s];
        if (!(w < 0.f)) num = fmaf(w, part_o[((base + s) * G + g) * D + d], num);
    }
    s_num[grp][d] = num;
    __syncthreads();
    if (tid < D) {
        float n = 0.f, den = 0.f;
#pragma unroll
        for (int i = 0; i < GROUPS; ++i) n += s_num[i][tid];
        for (int s = 0; s < n_splits; ++s) den += s_den[s];
        // (no weight at all, every score minus infinity: 0; a NaN score makes den NaN)
        const float r = den == 0.f ? 0.f : n / den;
        out[(long long)bhq * D + tid] = __bfloat16_as_ushort(__float2bfloat16_rn(r));
        const bool odd = !isfinite(n) && isfinite(den);
        if (__any_sync(kFull, odd)) settle_columns<D>(a, bh, odd, s_flags, out + (long long)bhq * D + (tid & ~31));
    }
}

// =======================================================================================
// Pipelined tensor-core variant: bulk copies into a ring of units (one unit = one tile, as in the
// unpack pipeline) feeding mma.sync straight from registers.  A tile of 128 tokens is split over the
// eight warps, sixteen tokens each, and what a thread decodes is what the
// tensor core wants from that thread, so a decoded tile never goes through shared memory:
//   scores  S^T[g][t] = sum_d q[g][d] K[t][d]  : A = q, B = K^T.  Thread (i, j) = (lane / 4, lane % 4)
//           owns D / 4 consecutive elements of token i; the order of the contraction over d is free,
//           so k-step s takes elements 4 s .. 4 s + 3 of the four threads of a token.
//   output  O^T[d][g] = sum_t V[t][d] P[t][g]  : A = V^T, B = P^T.  The scores' accumulators are the B
//           operand as they are.  Thread (i, j) owns columns i D / 8 .. of tokens 4 j .. 4 j + 3 and
//           pairs up tokens with byte permutes.
// The online softmax is each warp's own (running maximum, sum and numerator over its sixteen-token
// slabs); the warps meet once per unit, for the escape counts before each one's first element, and
// once at the end, to merge.  Behind a unit's barrier the unit before it has been read by everyone, so
// its stage is refilled after that, by one warp in turn: no producer warp (whose registers the others can
// use) and no barrier for free stages.
// Keys and values of [16, 8, 8192, 128], 3 bits, 5 % escapes: 4 query heads per KV head 301 -> 215 us, 16
// 588 -> 251 us; [16, 4, 8192, 64] (the plain kernel before) 221 -> 78 and 423 -> 90 us.  The floor is the packed
// bytes, 58 us; what bounds it is the integer pipe (47 % busy) and, with sixteen warps per SM, instruction
// latency and fetches.  The version before put every decoded tile into shared memory, let half of its warps
// multiply and met four times per tile.
// =======================================================================================

constexpr int kAWarps = 8;
constexpr int kAThreads = kAWarps * 32;
constexpr int kAStages = 3;
constexpr float kLog2e = 1.4426950408889634f;

template <int D>
struct alignas(128) AttnStage {
    static constexpr int kEscStage = kTileTokens * D / 2;
    alignas(128) uint8_t sm[kTileTokens * D];
    alignas(128) uint8_t codes[kTileTokens * D / 2];
    alignas(128) uint8_t esc[kEscStage + kEscSlack];
};

template <int D>
struct AttnPipeSmem {
    AttnStage<D> stage[kAStages];
    alignas(16) UnitMeta meta[kAStages];
    alignas(16) uint16_t q[16 * (D + 8)];         // queries (sixteen heads per CTA only)
    alignas(16) TileSrc src[32];                  // where the current 32 units lie
    float m[kAWarps][16];                         // running max per warp and head (log2 domain)
    float l[kAWarps][16];
    alignas(8) uint64_t full[kAStages];
    alignas(16) int warp_tot[2][kAWarps];         // escapes per warp of a unit, by the unit's parity
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two fp32 rounded to bf16, `lo` in the low half
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Elements from one query row to the next in shared memory (padded: the rows start in different banks).
template <int D>
constexpr int kQRow = D + 8;

// What a warp carries along.  HG: groups of eight query heads (1 or 2).
template <int D, int HG>
struct AttnState {
    // O^T: [HG][d pair][c0: (d, head 2 j), c1: (d, head 2 j + 1), c2, c3: d + 1], d = i D / 8 + 2 pair
    float o[HG][D / 16][4];
    float m[HG], l[HG];                           // head i (+ 8): running max, this thread's part of the sum
    uint32_t q[HG == 1 ? D / 8 : 1];              // one group: q[head i][j D / 4 ..], bf16 pairs
    const uint16_t *q_smem;                       // two (too many registers): the same in shared memory, head i
    uint32_t p[HG][2];                            // probabilities of the current slab, tokens 4 j .. 4 j + 3
    uint32_t p2[HG][2], p3[HG][2];                // what rounding p to bf16 (once, twice) left over
};

// Bf16 terms of a probability that go through the tensor core, which has time to spare: two at head_dim
// 128 (17 bits or more), three, all of the 24 bits, at head_dim 64 (whose kernel worked in fp32 before).
// The denominators sum p as it is.
template <int D>
constexpr int kTermsP = D == 64 ? 3 : 2;

// Scores += k-step `step` of the token this thread owns: its elements 4 step .. 4 step + 3.
template <int D, int HG>
__device__ __forceinline__ void score_words(const AttnState<D, HG> &st, int step, uint32_t w0, uint32_t w1, float (&c)[4]) {
    if constexpr (HG == 1) {
        mma_bf16(c, st.q[2 * step], 0u, st.q[2 * step + 1], 0u, w0, w1);
    } else {
        const uint2 lo = *reinterpret_cast<const uint2 *>(st.q_smem + 4 * step);
        const uint2 hi = *reinterpret_cast<const uint2 *>(st.q_smem + 8 * kQRow<D> + 4 * step);
        mma_bf16(c, lo.x, hi.x, lo.y, hi.y, w0, w1);
    }
}

// Online softmax of one slab: c[a] holds S^T of n-tile a (heads i and i + 8, tokens 4 j + 2 a, + 1);
// `valid`: tokens of the slab that exist (16 for a packed one).
template <int D, int HG>
__device__ __forceinline__ void softmax_slab(AttnState<D, HG> &st, const float (&c)[2][4], float sc2, int valid) {
    const int j = threadIdx.x & 3;
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        float s[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float v = c[t >> 1][2 * h + (t & 1)] * sc2;
            s[t] = 4 * j + t < valid ? v : -INFINITY;
        }
        float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
        mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, 2));
        const float mn = fmaxf(st.m[h], mx);
        const float ref = mn == -INFINITY ? 0.f : mn;         // (all scores so far minus infinity: weights 0, not NaN)
        const float alpha = exp2f(st.m[h] - ref);
        st.m[h] = mn;
        float sum = 0.f;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float p0 = exp2f(s[2 * u] - ref), p1 = exp2f(s[2 * u + 1] - ref);
            sum += p0 + p1;
            st.p[h][u] = bf16_pair(p0, p1);
            const float r0 = p0 - bf16_lo(st.p[h][u]), r1 = p1 - bf16_hi(st.p[h][u]);
            st.p2[h][u] = bf16_pair(r0, r1);
            if (kTermsP<D> == 3) st.p3[h][u] = bf16_pair(r0 - bf16_lo(st.p2[h][u]), r1 - bf16_hi(st.p2[h][u]));
        }
        st.l[h] = st.l[h] * alpha + sum;
        // the accumulators hold heads 2 j and 2 j + 1: fetch those heads' factors
        const float a0 = __shfl_sync(kFull, alpha, 8 * j), a1 = __shfl_sync(kFull, alpha, 8 * j + 4);
        if (__any_sync(kFull, alpha != 1.f)) {
#pragma unroll
            for (int e = 0; e < D / 16; ++e) {
                st.o[h][e][0] *= a0, st.o[h][e][1] *= a1;
                st.o[h][e][2] *= a0, st.o[h][e][3] *= a1;
            }
        }
    }
}

// One pair of columns of the slab's V: w[m] = columns (2 e, 2 e + 1) of token 4 j + m.
template <int D, int HG>
__device__ __forceinline__ void accumulate_words(AttnState<D, HG> &st, int e, const uint32_t (&w)[4]) {
    const uint32_t a0 = __byte_perm(w[0], w[1], 0x5410), a1 = __byte_perm(w[0], w[1], 0x7632);
    const uint32_t a2 = __byte_perm(w[2], w[3], 0x5410), a3 = __byte_perm(w[2], w[3], 0x7632);
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        if (kTermsP<D> == 3) mma_bf16(st.o[h][e], a0, a1, a2, a3, st.p3[h][0], st.p3[h][1]);
        mma_bf16(st.o[h][e], a0, a1, a2, a3, st.p2[h][0], st.p2[h][1]);
        mma_bf16(st.o[h][e], a0, a1, a2, a3, st.p[h][0], st.p[h][1]);
    }
}

// Escapes of the tile before this warp's first one: the warps' counts, through shared memory.
__device__ __forceinline__ int escapes_before_warp(int *warp_tot, int mine) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) warp_tot[warp] = mine;
    __syncthreads();
    return (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? warp_tot[lane & (kAWarps - 1)] : 0));
}

// Escape bytes of one group into its exponent bytes, from the staged window or, beyond it, from global memory.
__device__ __forceinline__ void fill_escapes(uint32_t z, int rank, bool staged, const uint8_t *esc, const UnitMeta &meta,
                                             int32_t *status, uint32_t (&e)[2]) {
    const int shift = meta.esc_shift;
    if (staged) {
        const uint32_t *words = reinterpret_cast<const uint32_t *>(esc);
        place_escapes(z, shift + rank, [words](int i) { return words[i]; }, e);
    } else {
        const uint2 g = gather_escapes(z, rank, esc + shift, meta.esc_staged, meta, status);
        e[0] |= g.x, e[1] |= g.y;
    }
}

// Scores of a staged K tile: this warp's sixteen tokens.
template <int N, int D, int HG>
__device__ __forceinline__ void score_unit(AttnState<D, HG> &st, const AttnStage<D> &stage, const UnitMeta &meta, int *warp_tot,
                                           float sc2, int32_t *status) {
    constexpr int NG = D / 32;                    // groups of eight elements in a thread's quarter of a token
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ExpTable tab = exp_table<N>(meta.left);
    // n-tile a, column i is token 4 (i / 2) + 2 a + i % 2: a thread's probabilities are then those of tokens 4 j ..
    const int tok0 = warp * 16 + 4 * (lane >> 3) + ((lane >> 2) & 1);
    const int base = tok0 * D + (lane & 3) * (D / 4);
    uint32_t nib[2][NG];
    int cnt[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int off = base + 2 * a * D;
        uint32_t x[NG];
        if constexpr (NG == 4) load_codes32<N>(stage.codes + off * N / 8, x);
        else load_codes16<N>(stage.codes + off * N / 8, x);
        cnt[a] = 0;
#pragma unroll
        for (int q = 0; q < NG; ++q) {
            nib[a][q] = spread8<N>(x[q]);
            cnt[a] += escapes_of(escape_mask<N>(nib[a][q]));
        }
    }
    // ranks: four tokens at a time, eight lanes each; tile a = 0 comes before a = 1 in every four
    uint32_t x = (uint32_t)cnt[0] | ((uint32_t)cnt[1] << 16);
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, x, d, 8);
        if ((lane & 7) >= d) x += u;
    }
    const uint32_t tot = __shfl_sync(kFull, x, 7, 8);
    const int t0 = (int)(tot & 0xFFFFu), four = t0 + (int)(tot >> 16);
    int pre = four;
#pragma unroll
    for (int d = 8; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(kFull, pre, d);
        if (lane >= d) pre += u;
    }
    const int mine = __shfl_sync(kFull, pre, 31);
    pre += escapes_before_warp(warp_tot, mine) - four;
    const int rank[2] = {pre + (int)(x & 0xFFFFu) - cnt[0], pre + t0 + (int)(x >> 16) - cnt[1]};
    // (a warp none of whose escapes lies beyond the window, i.e. nearly every one)
    const bool staged = __all_sync(kFull, rank[1] + cnt[1] <= meta.esc_staged);
    float c[2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        c[a][0] = c[a][1] = c[a][2] = c[a][3] = 0.f;
        const int off = base + 2 * a * D;
        int r = rank[a];
#pragma unroll
        for (int q = 0; q < NG; q += 2) {
            const uint4 sv = *reinterpret_cast<const uint4 *>(stage.sm + off + 8 * q);
            const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t z = escape_mask<N>(nib[a][q + u]);
                uint32_t e[2];
                lookup8<N>(nib[a][q + u], tab, e);
                fill_escapes(z, r, staged, stage.esc + kEscFront, meta, status, e);
                r += escapes_of(z);
                uint32_t w[4];
                assemble4(sw[2 * u], e[0], w[0], w[1]);
                assemble4(sw[2 * u + 1], e[1], w[2], w[3]);
                score_words(st, 2 * (q + u), w[0], w[1], c[a]);
                score_words(st, 2 * (q + u) + 1, w[2], w[3], c[a]);
            }
        }
    }
    softmax_slab(st, c, sc2, 16);
}

// Weighted sum over a staged V tile: this warp's sixteen tokens.
template <int N, int D, int HG>
__device__ __forceinline__ void accumulate_unit(AttnState<D, HG> &st, const AttnStage<D> &stage, const UnitMeta &meta,
                                                int *warp_tot, int32_t *status) {
    constexpr int NG = D / 64;                    // groups of eight elements in a thread's columns of a token
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = lane >> 2, j = lane & 3;
    const ExpTable tab = exp_table<N>(meta.left);
    const int base = (warp * 16 + 4 * j) * D + i * (D / 8);
    uint32_t nib[4][NG];
    uint32_t x = 0;                               // escapes of this thread's four pieces, a byte each (at most 16)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int off = base + m * D;
        uint32_t raw[NG];
        if constexpr (NG == 2) load_codes16<N>(stage.codes + off * N / 8, raw);
        else raw[0] = load_codes8<N>(stage.codes + off * N / 8);
        uint32_t cnt = 0;
#pragma unroll
        for (int q = 0; q < NG; ++q) {
            nib[m][q] = spread8<N>(raw[q]);
            cnt += (uint32_t)escapes_of(escape_mask<N>(nib[m][q]));
        }
        x |= cnt << (8 * m);
    }
    const uint32_t own = x;
    // ranks: token by token, the eight threads of a token one after the other (sums of at most 128)
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += u;
    }
    const uint32_t rows = __shfl_sync(kFull, x, 28 + j);
    const int rt[4] = {(int)(rows & 0xFFu), (int)((rows >> 8) & 0xFFu), (int)((rows >> 16) & 0xFFu), (int)(rows >> 24)};
    const int four = rt[0] + rt[1] + rt[2] + rt[3];
    int pre = four;
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        const int u = __shfl_up_sync(kFull, pre, d, 4);
        if (j >= d) pre += u;
    }
    const int mine = __shfl_sync(kFull, pre, 3);
    pre += escapes_before_warp(warp_tot, mine) - four;
    const bool staged = __all_sync(kFull, pre + four <= meta.esc_staged);
    int rank[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        rank[m] = pre + (int)((x >> (8 * m)) & 0xFFu) - (int)((own >> (8 * m)) & 0xFFu);
        pre += rt[m];
    }
#pragma unroll
    for (int q = 0; q < NG; ++q) {
        uint32_t w[4][4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const uint2 sv = *reinterpret_cast<const uint2 *>(stage.sm + base + m * D + 8 * q);
            const uint32_t z = escape_mask<N>(nib[m][q]);
            uint32_t e[2];
            lookup8<N>(nib[m][q], tab, e);
            fill_escapes(z, rank[m], staged, stage.esc + kEscFront, meta, status, e);
            rank[m] += escapes_of(z);
            assemble4(sv.x, e[0], w[0][m], w[1][m]);
            assemble4(sv.y, e[1], w[2][m], w[3][m]);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) accumulate_words(st, 4 * q + p, w[p]);
    }
}

// WORDS 32-bit words from a row that starts on a 16-byte boundary (wide) or only on a 4-byte one.
template <int WORDS>
__device__ __forceinline__ void load_row(const uint16_t *p, bool wide, uint32_t (&w)[WORDS]) {
    if (wide) {
#pragma unroll
        for (int i = 0; i < WORDS / 4; ++i) {
            const uint4 v = reinterpret_cast<const uint4 *>(p)[i];
            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < WORDS; ++i) w[i] = reinterpret_cast<const uint32_t *>(p)[i];
    }
}

// One slab of sixteen tokens of the dense residual, straight from global memory; `valid` of them exist.
template <int D, int HG>
__device__ __forceinline__ void dense_slab(AttnState<D, HG> &st, const uint16_t *k, const uint16_t *v, long long ss, int valid,
                                           bool wide, float sc2) {
    const int lane = threadIdx.x & 31, i = lane >> 2, j = lane & 3;
    float c[2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int t = 4 * (i >> 1) + 2 * a + (i & 1);
        uint32_t w[D / 8];
#pragma unroll
        for (int u = 0; u < D / 8; ++u) w[u] = 0u;
        if (t < valid) load_row(k + t * ss + j * (D / 4), wide, w);
        c[a][0] = c[a][1] = c[a][2] = c[a][3] = 0.f;
#pragma unroll
        for (int s = 0; s < D / 16; ++s) score_words(st, s, w[2 * s], w[2 * s + 1], c[a]);
    }
    softmax_slab(st, c, sc2, valid);
#pragma unroll
    for (int part = 0; part < D / 64; ++part) {
        uint32_t w[4][4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
#pragma unroll
            for (int u = 0; u < 4; ++u) w[m][u] = 0u;
            if (4 * j + m < valid) load_row(v + (4 * j + m) * ss + i * (D / 8) + 8 * part, wide, w[m]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t col[4] = {w[0][e], w[1][e], w[2][e], w[3][e]};
            accumulate_words(st, 4 * part + e, col);
        }
    }
}

// See the merge of the warps: a permutation of the D / 16 pairs of a column group (of eight) for heads 2 j and 2 j + 1.
template <int D>
__device__ __forceinline__ int merge_swizzle(int i, int j) {
    return D == 128 ? (i >> 1) ^ ((j & 1) * 4) : (i >> 2) ^ ((j & 1) * 2);
}

// ROWS: a run of items may go on in the next rows (see AttnArgs); otherwise a CTA has one split of one row, and nothing
// of the loop over rows, whose counters cost registers: spill loads 60 -> 44 bytes at <128, 1>, 244 -> 172 at <128, 2>;
// keys and values [1, 8, 20557, 128], 4 heads each, 41.4 -> 40.4 us, [16, 8, 1500, 128], 8 heads, 46.4 -> 45.1 us.
template <int D, int HG, bool ROWS>
__global__ void __launch_bounds__(kAThreads, 2) k_decode_attn_pipe(const __grid_constant__ AttnArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    AttnPipeSmem<D> &s = *reinterpret_cast<AttnPipeSmem<D> *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kAStages; ++i) {
            mbar_init(&s.full[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kAStages) {
        // an empty unit: what a consumer sees if it gives up waiting before the first description is written
        UnitMeta &m = s.meta[tid];
        m.dst = nullptr, m.esc = nullptr, m.esc_len = 0, m.esc_tile_start = 0, m.esc_staged = 0, m.esc_shift = 0;
        m.elems = 0, m.left = 0, m.nbits = 1, m.first_unit_of_tile = 1, m.ds = 0;
    }
    __syncthreads();
    // this CTA's items [begin, end), and the units that are to be decoded for them (two per packed item)
    const int begin = run_begin(a, blockIdx.x), end = run_begin(a, blockIdx.x + 1);
    const int row0 = ROWS ? (uint32_t)begin / a.by_items : blockIdx.x / a.by_cut_ctas, item0 = begin - row0 * a.items;
    const int row1 = ROWS ? (uint32_t)end / a.by_items : row0;
    const int n_units = 2 * ((row1 - row0) * a.n_seg + min(end - row1 * a.items, a.n_seg) - min(item0, a.n_seg));
    // launched as a programmatic dependent of its predecessor in the stream: no global memory is touched above
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int i = lane >> 2, j = lane & 3;
    const float sc2 = a.scale * kLog2e;                      // scores are kept in the log2 domain

    // Start the copies of unit n (a whole warp; units in ascending order): K tile, V tile, K tile, ... of the packed items
    // of the run, from one row on to the next.  The sources of 32 units are looked up at a time, one per lane:
    // two dependent round trips to global memory for all of them.
    const auto issue = [&](int n) {
        if (n >= n_units) return;
        if ((n & 31) == 0) {
            const int pair = (n + lane) >> 1;
            if (n + lane < n_units) {
                int row = row0, item = item0 + pair;
                if (ROWS && item >= a.n_seg) {                       // beyond the first row's (n_units > 0: there are packed items)
                    const int more = pair - max(0, a.n_seg - item0);
                    row += 1 + more / a.n_seg;
                    item = more % a.n_seg;
                }
                const adacode_segment sg = ((n + lane) & 1 ? a.vseg : a.kseg)[item];
                s.src[lane] = resolve_segment_tile(sg, (uint32_t)row / a.by_head_groups, kTileTokens * D, nullptr, 0);
            }
            __syncwarp();
        }
        const TileSrc &t = s.src[n & 31];
        const EscWindow w = esc_window(t, AttnStage<D>::kEscStage);
        const int stg = n % kAStages;
        AttnStage<D> &st = s.stage[stg];
        issue_unit(st.sm, st.codes, st.esc + kEscFront, s.meta[stg], &s.full[stg], t, w, 0, kTileTokens, D, nullptr, true, a.status);
    };
    if (warp == 0) {
#pragma unroll 1
        for (int n = 0; n < kAStages - 1; ++n) issue(n);
    }
    int u = 0;                                               // units of this CTA so far
    int x = begin;
    do {
        // the part [first, last) of one row's items
        const int row = ROWS ? (uint32_t)x / a.by_items : row0, first = x - row * a.items;
        const int last = ROWS ? min(a.items, first + (end - x)) : end - row * a.items;
        x += last - first;
        const int bh = (uint32_t)row / a.by_head_groups;
        const int b = (uint32_t)bh / a.by_heads, hkv = bh - b * a.Hkv;
        const int gz = (row - bh * a.head_groups) * (8 * HG);    // 8 or 16 query heads of the group at a time
        const int G = min(a.G - gz, 8 * HG);
        const int u1 = u + 2 * (min(last, a.n_seg) - min(first, a.n_seg));

        AttnState<D, HG> st;
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            st.m[h] = -INFINITY, st.l[h] = 0.f;
#pragma unroll
            for (int e = 0; e < D / 16; ++e) st.o[h][e][0] = st.o[h][e][1] = st.o[h][e][2] = st.o[h][e][3] = 0.f;
        }
        const uint16_t *qb = a.q + (long long)b * a.q_sb + (long long)(hkv * a.G + gz) * a.q_sh;
        if constexpr (HG == 1) {
            const uint16_t *qrow = qb + (long long)i * a.q_sh + j * (D / 4);
#pragma unroll
            for (int w = 0; w < D / 8; ++w) st.q[w] = 0u;
            if (i < G) {
                if (((uintptr_t)qrow & 15) == 0) load_row(qrow, true, st.q);
                else                                             // (query rows are only known to be 2-byte aligned)
#pragma unroll
                    for (int w = 0; w < D / 8; ++w) st.q[w] = (uint32_t)qrow[2 * w] | ((uint32_t)qrow[2 * w + 1] << 16);
            }
        } else {
            for (int n = tid; n < 16 * D; n += kAThreads) {
                const int g = n / D, d = n - g * D;
                s.q[g * kQRow<D> + d] = g < G ? qb[(long long)g * a.q_sh + d] : (uint16_t)0;
            }
            st.q_smem = s.q + i * kQRow<D> + j * (D / 4);
            __syncthreads();
        }
        for (; u < u1; ++u) {
            const int stg = u % kAStages;
            mbar_wait(&s.full[stg], (u / kAStages) & 1, a.status);      // (every lane: the ready case is three instructions)
            __syncwarp();
            const AttnStage<D> &stage = s.stage[stg];
            const UnitMeta &meta = s.meta[stg];
            int *wt = s.warp_tot[u & 1];
            if ((u & 1) == 0) {
                switch (meta.nbits) {
                    case 1: score_unit<1, D, HG>(st, stage, meta, wt, sc2, a.status); break;
                    case 2: score_unit<2, D, HG>(st, stage, meta, wt, sc2, a.status); break;
                    case 3: score_unit<3, D, HG>(st, stage, meta, wt, sc2, a.status); break;
                    default: score_unit<4, D, HG>(st, stage, meta, wt, sc2, a.status); break;
                }
            } else {
                switch (meta.nbits) {
                    case 1: accumulate_unit<1, D, HG>(st, stage, meta, wt, a.status); break;
                    case 2: accumulate_unit<2, D, HG>(st, stage, meta, wt, a.status); break;
                    case 3: accumulate_unit<3, D, HG>(st, stage, meta, wt, a.status); break;
                    default: accumulate_unit<4, D, HG>(st, stage, meta, wt, a.status); break;
                }
            }
            // every warp has passed this unit's barrier, so the stage of the unit before it is free
            if (warp == (u & (kAWarps - 1))) issue(u + kAStages - 1);
        }
        // dense residual tiles that fall into this part, a slab per warp
        const int tl_first = first > a.n_seg ? first - a.n_seg : 0;
        const int tl_last = last > a.n_seg ? last - a.n_seg : 0;
        const long long toff = (long long)b * a.t_sb + (long long)hkv * a.t_sh;
        const bool wide = ((((uintptr_t)a.k_tail | (uintptr_t)a.v_tail) & 15) | (uintptr_t)((a.t_sb | a.t_sh | a.t_ss) & 7)) == 0;
        for (int t = tl_first; t < tl_last; ++t) {
            const int t0 = t * kTileTokens + warp * 16;
            const int valid = a.tail_len - t0 < 16 ? a.tail_len - t0 : 16;
            if (valid > 0)
                dense_slab(st, a.k_tail + toff + t0 * a.t_ss, a.v_tail + toff + t0 * a.t_ss, a.t_ss, valid, wide, sc2);
        }

        // the combine kernel may be set up from here on (it waits for this launch to complete before it reads)
        if (!ROWS || x >= end) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        // ---------------- merge the warps ----------------
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            st.l[h] += __shfl_xor_sync(kFull, st.l[h], 1);
            st.l[h] += __shfl_xor_sync(kFull, st.l[h], 2);
            if (j == 0) {
                s.m[warp][8 * h + i] = st.m[h];
                s.l[warp][8 * h + i] = st.l[h];
            }
        }
        __syncthreads();                       // also: every unit so far has been read
        // Numerators of all warps, one group of eight heads at a time: [warp][head][d], in the stage that comes after those
        // which the next row's first units are on their way to.  The pairs of a column group of sixteen are
        // permuted so that a warp's writes, eight column groups of four heads, spread over the banks.
        float *acc = reinterpret_cast<float *>(&s.stage[(u + kAStages - 1) % kAStages]);
        static_assert(sizeof(AttnStage<D>) >= sizeof(float) * kAWarps * 8 * D, "a stage holds the numerators of the merge");
        const long long slot = (long long)bh * a.n_splits + ((int)blockIdx.x - (ROWS ? cta_of(a, row * a.items) : row * a.cut_ctas));
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            float f[2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int g = 8 * h + 2 * j + w;
                float mx = s.m[0][g];
#pragma unroll
                for (int k = 1; k < kAWarps; ++k) mx = fmaxf(mx, s.m[k][g]);
                f[w] = s.m[warp][g] == -INFINITY ? 0.f : exp2f(s.m[warp][g] - mx);
            }
#pragma unroll
            for (int e = 0; e < D / 16; ++e) {
                float *r0 = acc + (warp * 8 + 2 * j) * D + i * (D / 8) + 2 * (e ^ merge_swizzle<D>(i, j)), *r1 = r0 + D;
                *reinterpret_cast<float2 *>(r0) = make_float2(st.o[h][e][0] * f[0], st.o[h][e][2] * f[0]);
                *reinterpret_cast<float2 *>(r1) = make_float2(st.o[h][e][1] * f[1], st.o[h][e][3] * f[1]);
            }
            __syncthreads();
            for (int n = tid; n < 8 * D; n += kAThreads) {
                const int g = n / D, d = n - g * D;
                if (8 * h + g < G) {
                    const int at = d ^ (2 * merge_swizzle<D>(d / (D / 8), g >> 1));
                    float v = 0.f;
#pragma unroll
                    for (int w = 0; w < kAWarps; ++w) v += acc[(w * 8 + g) * D + at];
                    a.part_o[(slot * a.G + gz + 8 * h + g) * D + d] = v;
                }
            }
            if (h + 1 < HG) __syncthreads();
        }
        if (tid < G) {
            float mx = s.m[0][tid];
#pragma unroll
            for (int w = 1; w < kAWarps; ++w) mx = fmaxf(mx, s.m[w][tid]);
            float l = 0.f;
#pragma unroll
            for (int w = 0; w < kAWarps; ++w) l += s.m[w][tid] == -INFINITY ? s.l[w][tid] : s.l[w][tid] * exp2f(s.m[w][tid] - mx);
            a.part_ml[(slot * a.G + gz + tid) * 2 + 0] = mx == -INFINITY ? -INFINITY : mx / kLog2e;   // natural-log domain
            a.part_ml[(slot * a.G + gz + tid) * 2 + 1] = l;
        }
        if (ROWS && x < end) {
            // (the stage is written again, by a copy, behind the next unit's barrier; the warps' sums by the next row)
            fence_async_smem();
            __syncthreads();
        }
    } while (ROWS && x < end);
    // do not leave while a copy into this CTA's shared memory may still be in flight (see k_unpack_pipe)
    if (warp == 0 && launch_timed_out(a.status))
        for (int n = u > kAStages ? u - kAStages : 0; n < u; ++n)
            mbar_wait(&s.full[n % kAStages], (n / kAStages) & 1, a.status);
}

static_assert(sizeof(AttnPipeSmem<128>) <= 113 * 1024, "two CTAs of the pipelined kernel must fit one SM");

// CTAs of the pipelined kernel that are resident at a time: two per SM.
long long resident_ctas() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148 * 2;
    int sms = known[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148 * 2;
        known[dev].store(sms, std::memory_order_relaxed);
    }
    return (long long)sms * 2;
}

// CTAs that the items of all rows are dealt out to evenly: the n that are resident at a time, fewer if there are
// fewer items or if a row would be cut into more than kMaxSplits parts (at most n / rows + 2, or n / rows where
// that is a whole number).
long long even_ctas(long long n, long long rows, int items) {
    if (n > rows * items) n = rows * items;
    if (n >= rows * kMaxSplits) n = rows * kMaxSplits;
    else if (n > rows * (kMaxSplits - 1)) n = rows * (kMaxSplits - 1);
    return n;
}

// Whole splits per (batch, KV head), for workspaces that hold no more: the grid should fill a whole number of waves
// of resident CTAs.  One, two and three waves are
// tried and the fullest wins; fewer waves on ties (more tiles per CTA, less per-CTA overhead).
int pick_splits(long long slots, int B, int Hkv, int items) {
    const long long bh = (long long)B * Hkv;
    int best = 1;
    double best_fill = 0.0;
    for (int waves = 1; waves <= 3; ++waves) {
        long long sp = waves * slots / bh;
        if (sp < 1) sp = 1;
        if (sp > items) sp = items;
        if (sp > kMaxSplits) sp = kMaxSplits;
        const long long ctas = bh * sp;
        const double fill = (double)ctas / (double)(((ctas + slots - 1) / slots) * slots);
        if (fill > best_fill + 0.02) best_fill = fill, best = (int)sp;
    }
    return best;
}

}  // namespace

namespace {
// Programmatic dependent launch: the kernel may be set up while its predecessor in the stream drains;
// it executes griddepcontrol.wait before it reads or writes global memory.
template <typename... KArgs, typename... Args>
cudaError_t launch_as_dependent(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                                Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <int D, int HG, bool ROWS>
int launch_attn_pipe(const AttnArgs &a, dim3 grid, cudaStream_t st) {
    // the kernel's limit of dynamic shared memory is raised once per device
    static std::atomic<bool> done[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ADACODE_ERR_CUDA;
    if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(k_decode_attn_pipe<D, HG, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(AttnPipeSmem<D>)) != cudaSuccess)
            return ADACODE_ERR_CUDA;
        if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    }
    return launch_as_dependent(k_decode_attn_pipe<D, HG, ROWS>, grid, kAThreads, sizeof(AttnPipeSmem<D>), st, a) == cudaSuccess
               ? ADACODE_OK
               : ADACODE_ERR_CUDA;
}

template <bool ROWS>
int launch_attn_heads(const AttnArgs &a, bool two_groups, dim3 grid, cudaStream_t st) {
    if (a.D == 128) return two_groups ? launch_attn_pipe<128, 2, ROWS>(a, grid, st) : launch_attn_pipe<128, 1, ROWS>(a, grid, st);
    return two_groups ? launch_attn_pipe<64, 2, ROWS>(a, grid, st) : launch_attn_pipe<64, 1, ROWS>(a, grid, st);
}
}  // namespace

extern "C" {

size_t adacode_decode_attn_workspace_bytes(int B, int Hq, int D, int n_splits) {
    if (B <= 0 || Hq <= 0 || D <= 0) return 0;
    if (n_splits <= 0 || n_splits > kMaxSplits) n_splits = kMaxSplits;
    return (size_t)B * Hq * n_splits * ((size_t)D + 2) * sizeof(float);
}

int adacode_decode_attn(const void *q_bf16, int64_t q_stride_b, int64_t q_stride_h,
                        const adacode_segment *k_segments_dev, const adacode_segment *v_segments_dev, int n_segments,
                        const void *k_tail_bf16, const void *v_tail_bf16, int tail_len, int64_t tail_stride_b,
                        int64_t tail_stride_h, int64_t tail_stride_s, int B, int Hq, int Hkv, int seq_tile, int D,
                        float scale, void *out_bf16, void *workspace, size_t workspace_bytes, int n_splits,
                        int32_t *status, void *stream) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0 || n_segments < 0 || tail_len < 0) return ADACODE_ERR_INVALID_ARG;
    const int G = Hq / Hkv;
    if (seq_tile != kTileTokens || (D != 64 && D != 128)) return ADACODE_ERR_INVALID_ARG;
    // ADACODE_ATTN_SIMPLE=1 forces the plain kernel
    static const bool force_simple = [] {
        const char *v = getenv("ADACODE_ATTN_SIMPLE");
        return v && v[0] == '1';
    }();
    // Rows of work per KV head: up to eight query heads share a CTA, or up to sixteen: what costs is the decode of the
    // cache, which they share.  The plain kernel takes eight.
    const bool two_groups = G > 8 && !force_simple;
    const int heads_per_cta = two_groups ? 16 : kMaxGroup;
    const int head_groups = (G + heads_per_cta - 1) / heads_per_cta;
    if (head_groups > 65535) return ADACODE_ERR_INVALID_ARG;
    if (!q_bf16 || !out_bf16 || !workspace || !status) return ADACODE_ERR_INVALID_ARG;
    if (n_segments > 0 && (!k_segments_dev || !v_segments_dev)) return ADACODE_ERR_INVALID_ARG;
    if (tail_len > 0 && (!k_tail_bf16 || !v_tail_bf16 || ((uintptr_t)k_tail_bf16 & 3) || ((uintptr_t)v_tail_bf16 & 3) ||
                         ((tail_stride_b | tail_stride_h | tail_stride_s) & 1)))
        return ADACODE_ERR_INVALID_ARG;
    const int items = n_segments + (tail_len + kTileTokens - 1) / kTileTokens;
    if (items == 0) return ADACODE_ERR_INVALID_ARG;
    const long long rows = (long long)B * Hkv * head_groups;
    if (rows * items >= (1ll << 31)) return ADACODE_ERR_INVALID_ARG;
    const bool given = n_splits > 0;
    const long long slots = given ? 0 : resident_ctas();
    if (!given) n_splits = pick_splits(slots, B, Hkv * head_groups, items);
    if (n_splits > kMaxSplits) n_splits = kMaxSplits;
    if (workspace_bytes < adacode_decode_attn_workspace_bytes(B, Hq, D, n_splits)) return ADACODE_ERR_WORKSPACE;
    if (n_splits > items) n_splits = items;                // (the others would be empty)
    if ((long long)items * n_splits >= (1ll << 31)) n_splits = 1;
    // Whole splits of every row, or one cut through all rows where that makes the longest run of items shorter: it is worth
    // the time of about one item to end a row and to begin the next.  256 rows of 33 items on 296 CTAs (keys and values
    // [32, 8, 4146, 128], 4 heads each): 33 items per CTA and 206 us, or 29 and 192 us; 20 rows of 71 items ([5, 4, 9000, 128],
    // 7 heads each): 6 items and 54.3 us, or 5 and a row's end, which counts as 6 and stays whole (cut 52.6 us);
    // 128 rows of 3 items ([64, 2, 300, 128]): 2 either way, 18.4 us whole, 21.1 us cut.
    long long n_ctas = rows * n_splits, cut_items = items, cut_ctas = n_splits;
    if (!given && !force_simple) {
        const long long even = even_ctas(slots, rows, items);
        const int parts = (int)(even % rows == 0 ? even / rows : even / rows + 2);
        const long long whole_run = (n_ctas + slots - 1) / slots * ((items + n_splits - 1) / n_splits);
        const long long even_run = (rows * items + even - 1) / even + (even % rows != 0);
        // (a caller's workspace may be for the whole splits only)
        if (even_run < whole_run && rows * items * even < (1ll << 31) &&
            workspace_bytes >= adacode_decode_attn_workspace_bytes(B, Hq, D, parts))
            n_ctas = cut_ctas = even, cut_items = rows * items, n_splits = parts;
    }
    if (n_ctas >= (1ll << 31)) return ADACODE_ERR_INVALID_ARG;
    AttnArgs a;
    a.items = items, a.head_groups = head_groups, a.heads_per_row = heads_per_cta;
    a.cut_items = (int)cut_items, a.cut_ctas = (int)cut_ctas;
    a.by_items = quotient_by(items), a.by_head_groups = quotient_by(head_groups), a.by_heads = quotient_by(Hkv);
    a.by_cut_items = quotient_by(cut_items), a.by_cut_ctas = quotient_by(cut_ctas);
    a.q = (const uint16_t *)q_bf16, a.q_sb = q_stride_b, a.q_sh = q_stride_h;
    a.kseg = k_segments_dev, a.vseg = v_segments_dev, a.n_seg = n_segments;
    a.k_tail = (const uint16_t *)k_tail_bf16, a.v_tail = (const uint16_t *)v_tail_bf16, a.tail_len = tail_len;
    a.t_sb = tail_stride_b, a.t_sh = tail_stride_h, a.t_ss = tail_stride_s;
    a.B = B, a.Hq = Hq, a.Hkv = Hkv, a.G = G, a.D = D, a.scale = scale, a.n_splits = n_splits;
    a.part_o = (float *)workspace;
    a.part_ml = a.part_o + (size_t)B * Hq * n_splits * D;
    a.status = status;
    cudaStream_t st = (cudaStream_t)stream;
    // Two launches that hand partial results on in the workspace: threads that share a stream and a workspace must not come
    // between them.
    static std::mutex locks[64];
    const std::lock_guard<std::mutex> both(locks[((uintptr_t)workspace >> 9) * 0x9E3779B97F4A7C15ull >> 58]);
    if (!force_simple) {
        const dim3 grid((unsigned)n_ctas);
        const int rc = cut_items > items ? launch_attn_heads<true>(a, two_groups, grid, st) : launch_attn_heads<false>(a, two_groups, grid, st);
        if (rc != ADACODE_OK) return rc;
    } else {
        if (cudaFuncSetAttribute(k_decode_attn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AttnSmem)) !=
            cudaSuccess)
            return ADACODE_ERR_CUDA;
        k_decode_attn<<<dim3((unsigned)n_ctas), kAttnThreads, sizeof(AttnSmem), st>>>(a);
    }
    if (cudaGetLastError() != cudaSuccess) return ADACODE_ERR_CUDA;
    const bool few = n_splits <= kFewSplits;
    auto combine = D == 128 ? (few ? k_decode_attn_combine<128, 1> : k_decode_attn_combine<128, kCombineThreads / 128>)
                            : (few ? k_decode_attn_combine<64, 1> : k_decode_attn_combine<64, kCombineThreads / 64>);
    if (launch_as_dependent(combine, dim3(B * Hq), few ? D : kCombineThreads, 0, st, a, (uint16_t *)out_bf16) != cudaSuccess)
        return ADACODE_ERR_CUDA;
    return ADACODE_OK;
}

}  // extern "C"
