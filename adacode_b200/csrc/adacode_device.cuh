// Device helpers shared by the float11 kernels (pack, unpack, fused decode attention): bit
// manipulation of bf16 words, zero-slot masks of packed code words, serialisation of a chunk's
// codes, block copies and the warp scan of escape counts.  Included inside an anonymous
// namespace by each .cu file.
#pragma once

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kCPT = 4;                          // chunks per thread per slab
constexpr int kSlabChunks = kThreads * kCPT;     // 1024
constexpr unsigned kFull = 0xFFFFFFFFu;

// Quotients of numbers below 2**31 by a divisor that the host knows, by multiplication (Granlund and Montgomery,
// Division by invariant integers using multiplication, 1994: 2**l >= d, m = 2**31 (2**l - d) / d + 2**31 + 1 rounded
// down, n / d = n m >> (31 + l)).
struct Quotient {
    uint32_t d, m, shift;
};
Quotient quotient_by(int64_t d) {
    int l = 0;
    while ((1ll << l) < d) ++l;
    return {(uint32_t)d, (uint32_t)(((1ull << 31) * ((1ull << l) - (uint64_t)d)) / (uint64_t)d + (1ull << 31) + 1), (uint32_t)(31 + l)};
}
__device__ __forceinline__ uint32_t operator/(uint32_t n, const Quotient &q) { return (uint32_t)((uint64_t)n * q.m >> q.shift); }

// ---------------------------------------------------------------------------------------
// bit helpers
// ---------------------------------------------------------------------------------------

// sign/mantissa bytes of two bf16 held in one 32-bit word, one byte per 16-bit lane
__device__ __forceinline__ uint32_t signmant_lanes(uint32_t w) {
    return ((w >> 8) & 0x00800080u) | (w & 0x007F007Fu);
}
// four sign/mantissa bytes from four consecutive bf16 (two words)
__device__ __forceinline__ uint32_t signmant4(uint32_t w0, uint32_t w1) {
    return __byte_perm(signmant_lanes(w0), signmant_lanes(w1), 0x6420);
}

// Mask with one bit at the least significant bit of each of the eight N-bit code slots.
template <int N>
struct SlotLsb;
template <>
struct SlotLsb<1> { static constexpr uint32_t v = 0xFFu; };
template <>
struct SlotLsb<2> { static constexpr uint32_t v = 0x5555u; };
template <>
struct SlotLsb<3> { static constexpr uint32_t v = 0x249249u; };
template <>
struct SlotLsb<4> { static constexpr uint32_t v = 0x11111111u; };

// Bit (at the slot LSB) for every code slot of the group word that holds code 0.
template <int N>
__device__ __forceinline__ uint32_t zero_slots(uint32_t g) {
    uint32_t m = g;
#pragma unroll
    for (int i = 1; i < N; ++i) m |= g >> i;
    return ~m & SlotLsb<N>::v;
}

// The eight slot bits of zero_slots<N>() (one per N-bit slot, at the slot's least significant bit)
// moved next to each other: slot j -> bit j, so element k of the group sits at bit 7 - k.
template <int N>
__device__ __forceinline__ uint32_t compress_slots(uint32_t z) {
    if constexpr (N == 1) {
        return z;
    } else if constexpr (N == 2) {
        z = (z | (z >> 1)) & 0x3333u;
        z = (z | (z >> 2)) & 0x0F0Fu;
        return (z | (z >> 4)) & 0xFFu;
    } else if constexpr (N == 3) {
        z = (z | (z >> 2)) & 0x0C30C3u;
        z = (z | (z >> 4)) & 0x00F00Fu;
        return (z | (z >> 8)) & 0xFFu;
    } else {
        z = (z | (z >> 3)) & 0x03030303u;
        z = (z | (z >> 6)) & 0x000F000Fu;
        return (z | (z >> 12)) & 0xFFu;
    }
}

// Eight exponent codes of eight consecutive bf16 (four words) as one group word:
// element k sits at bits [(7-k)*N, (8-k)*N).  Out-of-window exponents code as 0.
template <int N>
__device__ __forceinline__ uint32_t encode_group(const uint32_t w[4], int left) {
    constexpr uint32_t kMax = (1u << N) - 1u;
    uint32_t g = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t c0 = ((w[i] >> 7) & 0xFFu) - (uint32_t)left;
        uint32_t c1 = ((w[i] >> 23) & 0xFFu) - (uint32_t)left;
        c0 = c0 > kMax ? 0u : c0;
        c1 = c1 > kMax ? 0u : c1;
        g |= c0 << ((7 - 2 * i) * N);
        g |= c1 << ((6 - 2 * i) * N);
    }
    return g;
}

// In-window histogram: cnt[v] += number of slots of g holding code v (v = 1 .. 2^N-1).
template <int N>
__device__ __forceinline__ void count_codes(uint32_t g, uint32_t (&cnt)[1 << N]) {
    constexpr uint32_t M = SlotLsb<N>::v;
    uint32_t plane[N];
#pragma unroll
    for (int i = 0; i < N; ++i) plane[i] = (g >> i) & M;
#pragma unroll
    for (int v = 1; v < (1 << N); ++v) {
        uint32_t m = M;
#pragma unroll
        for (int i = 0; i < N; ++i) m &= ((v >> i) & 1) ? plane[i] : ~plane[i];
        cnt[v] += __popc(m);
    }
}

// ---------------------------------------------------------------------------------------
// code-byte (de)serialisation: a chunk of CH elements owns CH*N/8 bytes, each group of 8
// codes stored as an N-byte big-endian word
// ---------------------------------------------------------------------------------------

template <int N, int CH>
__device__ __forceinline__ void store_chunk_codes(uint8_t *s, const uint32_t g[CH / 8]) {
    if constexpr (CH == 16) {
        if constexpr (N == 1) {
            *reinterpret_cast<uint16_t *>(s) = (uint16_t)(g[0] | (g[1] << 8));
        } else if constexpr (N == 2) {
            *reinterpret_cast<uint32_t *>(s) = __byte_perm(g[0], g[1], 0x4501);
        } else if constexpr (N == 3) {
            const uint32_t lo = __byte_perm(g[0], g[1], 0x6012);
            const uint32_t hi = __byte_perm(g[1], 0u, 0x4401);
            uint16_t *p = reinterpret_cast<uint16_t *>(s);
            p[0] = (uint16_t)lo;
            p[1] = (uint16_t)(lo >> 16);
            p[2] = (uint16_t)hi;
        } else {
            uint2 v;
            v.x = __byte_perm(g[0], 0u, 0x0123);
            v.y = __byte_perm(g[1], 0u, 0x0123);
            *reinterpret_cast<uint2 *>(s) = v;
        }
    } else {
        if constexpr (N == 1) {
            s[0] = (uint8_t)g[0];
        } else if constexpr (N == 2) {
            *reinterpret_cast<uint16_t *>(s) = (uint16_t)__byte_perm(g[0], 0u, 0x4401);
        } else if constexpr (N == 3) {
            s[0] = (uint8_t)(g[0] >> 16);
            s[1] = (uint8_t)(g[0] >> 8);
            s[2] = (uint8_t)g[0];
        } else {
            *reinterpret_cast<uint32_t *>(s) = __byte_perm(g[0], 0u, 0x0123);
        }
    }
}

template <int N, int CH>
__device__ __forceinline__ void load_chunk_codes(const uint8_t *s, uint32_t g[CH / 8]) {
    if constexpr (CH == 16) {
        if constexpr (N == 1) {
            const uint32_t v = *reinterpret_cast<const uint16_t *>(s);
            g[0] = v & 0xFFu;
            g[1] = v >> 8;
        } else if constexpr (N == 2) {
            const uint32_t v = *reinterpret_cast<const uint32_t *>(s);
            g[0] = __byte_perm(v, 0u, 0x4401);
            g[1] = __byte_perm(v, 0u, 0x4423);
        } else if constexpr (N == 3) {
            const uint16_t *p = reinterpret_cast<const uint16_t *>(s);
            const uint32_t lo = (uint32_t)p[0] | ((uint32_t)p[1] << 16);
            const uint32_t hi = p[2];
            g[0] = __byte_perm(lo, 0u, 0x4012);
            g[1] = __byte_perm(lo, hi, 0x6345);
        } else {
            const uint2 v = *reinterpret_cast<const uint2 *>(s);
            g[0] = __byte_perm(v.x, 0u, 0x0123);
            g[1] = __byte_perm(v.y, 0u, 0x0123);
        }
    } else {
        if constexpr (N == 1) {
            g[0] = s[0];
        } else if constexpr (N == 2) {
            g[0] = __byte_perm((uint32_t) * reinterpret_cast<const uint16_t *>(s), 0u, 0x4401);
        } else if constexpr (N == 3) {
            g[0] = ((uint32_t)s[0] << 16) | ((uint32_t)s[1] << 8) | s[2];
        } else {
            g[0] = __byte_perm(*reinterpret_cast<const uint32_t *>(s), 0u, 0x0123);
        }
    }
}

// Copy `bytes` bytes between shared and global memory with the whole block, 16 bytes at a
// time when both ends allow it.
__device__ __forceinline__ void block_copy_out(uint8_t *dst, const uint8_t *s_src, int bytes) {
    if ((((uintptr_t)dst | (uintptr_t)bytes) & 15) == 0) {
        const uint4 *s4 = reinterpret_cast<const uint4 *>(s_src);
        uint4 *d4 = reinterpret_cast<uint4 *>(dst);
        for (int i = threadIdx.x; i < bytes / 16; i += kThreads) d4[i] = s4[i];
    } else {
        for (int i = threadIdx.x; i < bytes; i += kThreads) dst[i] = s_src[i];
    }
}
__device__ __forceinline__ void block_copy_in(uint8_t *s_dst, const uint8_t *src, int bytes) {
    if ((((uintptr_t)src | (uintptr_t)bytes) & 15) == 0) {
        const uint4 *g4 = reinterpret_cast<const uint4 *>(src);
        uint4 *s4 = reinterpret_cast<uint4 *>(s_dst);
        for (int i = threadIdx.x; i < bytes / 16; i += kThreads) s4[i] = __ldg(g4 + i);
    } else {
        for (int i = threadIdx.x; i < bytes; i += kThreads) s_dst[i] = src[i];
    }
}

// Inclusive warp scans of four counters per lane, walked in (k, lane) order.  Counters are
// at most 16, so two share one register as 16-bit fields.  On return incl[k] is the
// inclusive rank of (k, lane) within the warp's 4x32 chunks; the return value is the total.
__device__ __forceinline__ int warp_scan4(const int cnt[kCPT], int incl[kCPT]) {
    uint32_t a = (uint32_t)cnt[0] | ((uint32_t)cnt[1] << 16);
    uint32_t b = (uint32_t)cnt[2] | ((uint32_t)cnt[3] << 16);
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t ua = __shfl_up_sync(kFull, a, d);
        const uint32_t ub = __shfl_up_sync(kFull, b, d);
        if (lane >= d) {
            a += ua;
            b += ub;
        }
    }
    const uint32_t ta = __shfl_sync(kFull, a, 31);
    const uint32_t tb = __shfl_sync(kFull, b, 31);
    const int t0 = ta & 0xFFFF, t1 = ta >> 16, t2 = tb & 0xFFFF, t3 = tb >> 16;
    incl[0] = (int)(a & 0xFFFF);
    incl[1] = (int)(a >> 16) + t0;
    incl[2] = (int)(b & 0xFFFF) + t0 + t1;
    incl[3] = (int)(b >> 16) + t0 + t1 + t2;
    return t0 + t1 + t2 + t3;
}

// ---- table-driven decode -------------------------------------------------------------------
// One shared-memory lookup per pair (or quadruple, or octet) of codes: the table maps a run of packed
// code bits to the finished exponent fields of the corresponding bf16 pairs, `(e0 << 7) | (e1 << 23)`,
// with the window's left edge already added (and 0 for code 0).  Index width: 8 bits for N = 1, 2, 4; 6 bits
// for N = 3.  Only the plain attention kernel decodes this way, which makes it independent of the decode
// in registers below that it is there to check.
__device__ __forceinline__ void build_decode_lut(uint32_t *lut, int N, int left, int n_threads) {
    const int index_bits = (N == 3) ? 6 : 8;
    const int words = (index_bits / N) / 2;
    const int total = (1 << index_bits) * words;
    const uint32_t mask = (1u << N) - 1u;
    for (int w = threadIdx.x; w < total; w += n_threads) {
        const uint32_t e = (uint32_t)(w / words), p = (uint32_t)(w % words);
        const uint32_t c_even = (e >> (index_bits - (2 * p + 1) * N)) & mask;
        const uint32_t c_odd = (e >> (index_bits - (2 * p + 2) * N)) & mask;
        // code 0 (an escape) decodes to exponent field 0, so that the escaped exponent can be OR-ed in
        const uint32_t e_even = c_even ? ((c_even + (uint32_t)left) & 0xFFu) : 0u;
        const uint32_t e_odd = c_odd ? ((c_odd + (uint32_t)left) & 0xFFu) : 0u;
        lut[w] = (e_even << 7) | (e_odd << 23);
    }
}

// Exponent fields of the four bf16 pairs of group word g (element 0 in the most significant bits).
template <int N>
__device__ __forceinline__ void decode_group(const uint32_t *lut, uint32_t g, uint32_t (&ew)[4]) {
    if constexpr (N == 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ew[i] = lut[(g >> (24 - 8 * i)) & 0xFFu];
    } else if constexpr (N == 3) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ew[i] = lut[(g >> (18 - 6 * i)) & 0x3Fu];
    } else if constexpr (N == 2) {
        const uint2 hi = reinterpret_cast<const uint2 *>(lut)[(g >> 8) & 0xFFu];
        const uint2 lo = reinterpret_cast<const uint2 *>(lut)[g & 0xFFu];
        ew[0] = hi.x, ew[1] = hi.y, ew[2] = lo.x, ew[3] = lo.y;
    } else {
        const uint4 v = reinterpret_cast<const uint4 *>(lut)[g & 0xFFu];
        ew[0] = v.x, ew[1] = v.y, ew[2] = v.z, ew[3] = v.w;
    }
}


// ---- decode in registers ---------------------------------------------------------------------
// Eight codes at a time, without shared-memory lookups and without a loop over the escapes.  The
// exponent fields are put together as bytes, four elements to a 32-bit word:
//   1. the codes are spread to one nibble per element.  The first element's code has the most
//      significant bits of a group, so element k lies in nibble 7 - k, and in the words below the
//      last of four elements has the lowest byte;
//   2. a byte permute looks four exponents up at once in a table of at most eight bytes that lives
//      in two registers (N = 4 has sixteen values and adds the window's left edge bytewise);
//   3. z has one bit per element that escaped (code 0).  A product with 0x11111111 gives every
//      nibble the number of escapes from its element to the last one, and from it the selector with
//      which a byte permute drops the escape bytes that end here into their places (zero bytes
//      elsewhere);
//   4. sign, mantissa and exponent bytes are merged and interleaved into bf16 pairs.
// Nothing of it is divergent, and all of it runs on the full-rate integer and multiply pipes (bringing the
// elements into ascending order with one bit reversal per group made that unit, a quarter as fast, the
// bottleneck at 85 % busy).  The unpack kernel executes 15.7 instructions per element whatever the share of
// escapes; with the table lookups and the per-escape loop that this replaces it was 15.8 at 6 % escapes and
// more with more of them.

struct ExpTable { uint32_t a, b; };

// bits of a where the mask has ones, of b elsewhere: one instruction
__device__ __forceinline__ uint32_t bit_select(uint32_t mask, uint32_t a, uint32_t b) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(r) : "r"(a), "r"(b), "r"(mask));
    return r;
}

template <int N>
__device__ __forceinline__ ExpTable exp_table(int left) {
    ExpTable t = {0u, 0u};
    if constexpr (N == 4) {
        t.a = (uint32_t)left;
    } else {
        const auto v = [left](int c) { return (uint32_t)(c + left) & 0xFFu; };
        t.a = (v(1) << 8) | (v(2) << 16) | (v(3) << 24);
        t.b = v(4) | (v(5) << 8) | (v(6) << 16) | (v(7) << 24);
    }
    return t;
}

// __byte_perm by a selector that is computed: the intrinsic masks it first, these have no bit to mask (unpack and
// attention 3-4 % faster without).
__device__ __forceinline__ uint32_t permute(uint32_t a, uint32_t b, uint32_t selector) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(selector));
    return r;
}

// The codes of two consecutive groups, as spread8 takes them, from a 16-element chunk's code bytes.
template <int N>
__device__ __forceinline__ void load_codes16(const uint8_t *s, uint32_t (&x)[2]) {
    if constexpr (N == 1) {
        const uint32_t v = *reinterpret_cast<const uint16_t *>(s);
        x[0] = v & 0xFFu, x[1] = v >> 8;
    } else if constexpr (N == 2) {
        const uint32_t v = *reinterpret_cast<const uint32_t *>(s);
        x[0] = __byte_perm(v, 0u, 0x4041), x[1] = __byte_perm(v, 0u, 0x4243);
    } else if constexpr (N == 3) {
        const uint16_t *p = reinterpret_cast<const uint16_t *>(s);
        const uint32_t lo = (uint32_t)p[0] | ((uint32_t)p[1] << 16), hi = p[2];
        x[0] = __byte_perm(lo, 0u, 0x4012);
        x[1] = __byte_perm(lo, hi, 0x6345);
    } else {
        const uint2 v = *reinterpret_cast<const uint2 *>(s);
        x[0] = __byte_perm(v.x, 0u, 0x0123), x[1] = __byte_perm(v.y, 0u, 0x0123);
    }
}

// The same for the eight elements of one group, whose N code bytes lie on an N-byte boundary
// (N = 3: anywhere).
template <int N>
__device__ __forceinline__ uint32_t load_codes8(const uint8_t *s) {
    if constexpr (N == 1) return s[0];
    else if constexpr (N == 2) return __byte_perm((uint32_t) * reinterpret_cast<const uint16_t *>(s), 0u, 0x4041);
    else if constexpr (N == 3) return ((uint32_t)s[0] << 16) | ((uint32_t)s[1] << 8) | s[2];
    else return __byte_perm(*reinterpret_cast<const uint32_t *>(s), 0u, 0x0123);
}

// The same for 32 elements (four groups) whose 4 N code bytes lie on a 4 N-byte boundary (N = 3: 4 bytes).
template <int N>
__device__ __forceinline__ void split_codes32(const uint32_t (&w)[N], uint32_t (&x)[4]) {
    if constexpr (N == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = (w[0] >> (8 * q)) & 0xFFu;
    } else if constexpr (N == 2) {
        x[0] = __byte_perm(w[0], 0u, 0x4041), x[1] = __byte_perm(w[0], 0u, 0x4243);
        x[2] = __byte_perm(w[1], 0u, 0x4041), x[3] = __byte_perm(w[1], 0u, 0x4243);
    } else if constexpr (N == 3) {
        // (the highest byte is arbitrary: spread8 ignores it)
        x[0] = __byte_perm(w[0], 0u, 0x4012);
        x[1] = __byte_perm(w[0], w[1], 0x5345);
        x[2] = __byte_perm(w[1], w[2], 0x4234);
        x[3] = __byte_perm(w[2], 0u, 0x4123);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = __byte_perm(w[q], 0u, 0x0123);
    }
}
template <int N>
__device__ __forceinline__ void load_codes32(const uint8_t *s, uint32_t (&x)[4]) {
    uint32_t w[N];
    if constexpr (N == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(s);
        w[0] = v.x, w[1] = v.y;
    } else if constexpr (N == 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(s);
        w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = reinterpret_cast<const uint32_t *>(s)[i];
    }
    split_codes32<N>(w, x);
}

// One nibble per element.
template <int N>
__device__ __forceinline__ uint32_t spread8(uint32_t x) {
    uint32_t nib = x;
    if constexpr (N == 3) {
        // (what a step leaves between the fields it moves is cleared by the last mask)
        nib = bit_select(0xFFFF0000u, x << 4, x);
        nib = bit_select(0xFF00FF00u, nib << 2, nib);
        nib = bit_select(0xF0F0F0F0u, nib << 1, nib) & 0x77777777u;
    } else if constexpr (N == 2) {                     // x: eight bits in each half
        nib = (x | (x << 4)) & 0x0F0F0F0Fu;
        nib = (nib | (nib << 2)) & 0x33333333u;
    } else if constexpr (N == 1) {
        nib = (x | (x << 12)) & 0x000F000Fu;
        nib = (nib | (nib << 6)) & 0x03030303u;
        nib = (nib | (nib << 3)) & 0x11111111u;
    }
    return nib;
}

// z: bit 4 (7 - k) set where element k escaped
template <int N>
__device__ __forceinline__ uint32_t escape_mask(uint32_t nib) {
    if constexpr (N == 4) {
        const uint32_t t = nib | (nib >> 1);
        return ~(t | (t >> 2)) & 0x11111111u;
    } else if constexpr (N == 3) {
        return (~(nib + 0x77777777u) & 0x88888888u) >> 3;
    } else if constexpr (N == 2) {
        return (~(nib + 0x33333333u) & 0x44444444u) >> 2;
    } else {
        return ~nib & 0x11111111u;
    }
}

// e[0], e[1]: exponent bytes of elements 0..3 and 4..7 (the last one lowest), zero where the element escaped
template <int N>
__device__ __forceinline__ void lookup8(uint32_t nib, const ExpTable &t, uint32_t (&e)[2]) {
    if constexpr (N == 4) {
        const uint32_t even = (nib >> 4) & 0x0F0F0F0Fu, odd = nib & 0x0F0F0F0Fu;
        const uint32_t ne = ((even + 0x0F0F0F0Fu) >> 4) & 0x01010101u;      // code != 0
        const uint32_t no = ((odd + 0x0F0F0F0Fu) >> 4) & 0x01010101u;
        // (no carry between bytes: a code that was written stands for an exponent of 0..255)
        const uint32_t ee = ne * t.a + even, eo = no * t.a + odd;
        e[0] = __byte_perm(ee, eo, 0x3726);
        e[1] = __byte_perm(ee, eo, 0x1504);
    } else {
        e[0] = permute(t.a, t.b, nib >> 16);
        e[1] = permute(t.a, t.b, nib);
    }
}

// escapes among the eight elements of z
__device__ __forceinline__ int escapes_of(uint32_t z) { return (int)((z * 0x11111111u) >> 28); }

// Put the escape bytes of these eight elements, which begin at byte `r` of a stream, into e (as lookup8
// left it).  `word(i)` is the stream's aligned 32-bit word i; of the words from the one before r's to
// two behind it three are read, whether they are needed or not.
template <typename Words>
__device__ __forceinline__ void place_escapes(uint32_t z, int r, const Words &word, uint32_t (&e)[2]) {
    const uint32_t suffix = z * 0x11111111u;               // nibble 7 - k: escapes among elements k..7 (at most 8)
    const uint32_t last8 = (suffix >> 9) & 0x78u;          // 8 x escapes among elements 4..7
    const int mid8 = 8 * r + (int)(suffix >> 28) * 8 - (int)last8;       // 8 x where those begin
    const int i = (mid8 >> 5) - 1;
    const uint32_t w0 = word(i), w1 = word(i + 1), w2 = word(i + 2);
    const uint32_t a = __funnelshift_r(w0, w1, (uint32_t)mid8);          // the four bytes before that place
    const uint32_t b = __funnelshift_r(w1, w2, (uint32_t)mid8);
    const uint32_t c = __funnelshift_rc(a, b, last8);                    // the four bytes before the end
    // a nibble of a selector: the s-th escape from the end of four elements takes byte 4 - s of the word
    // (bytes 4..7 of the pair), any other element a zero byte (0..3)
    e[0] |= permute(0u, a, 0x3333u - (z >> 16) * (0x1111u - 5u));
    e[1] |= permute(0u, c, 0x3333u - z * (0x1111u - 5u));
}

// Two bf16 pairs from four sign/mantissa bytes and their exponent bytes (the last one lowest).
__device__ __forceinline__ void assemble4(uint32_t sm, uint32_t e, uint32_t &w0, uint32_t &w1) {
    // exponents to bits 7..14 of each half (the product runs on the multiply pipe), the rest from the byte
    // of sign and mantissa doubled
    w0 = bit_select(0x7F807F80u, __byte_perm(e, 0u, 0x4243) * 128u, __byte_perm(sm, 0u, 0x1100));
    w1 = bit_select(0x7F807F80u, __byte_perm(e, 0u, 0x4041) * 128u, __byte_perm(sm, 0u, 0x3322));
}

// ---- encode in registers ---------------------------------------------------------------------
// The exponents of a word's two bf16 as codes in its 16-bit halves, 0 outside the window: one packed
// add-and-minimum takes exponent - left, where everything below the window wraps to a large value and
// everything beyond it is cut to 2**N, whose low N bits are 0 again.  `neg_left` is -left in both halves.
// (A table in shared memory, one byte lookup per element, took a load and two bank conflicts each: pack of keys and
// values [16, 8, 8192, 128] at 3 bits 222.6 us with it, 209.8 us without; with the histogram 241 and 219 us.)
template <int N>
__device__ __forceinline__ uint32_t encode_pair(uint32_t w, uint32_t neg_left) {
    constexpr uint32_t kTop = (1u << N) * 0x10001u;
    return __viaddmin_u16x2((w >> 7) & 0x00FF00FFu, neg_left, kTop) & (kTop - 0x10001u);
}

// Eight codes (four words of encode_pair) as one group word, element 0 in the most significant bits.
template <int N>
__device__ __forceinline__ uint32_t join_codes(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3) {
    constexpr uint32_t kStep = 1u << (2 * N);
    const uint32_t u = p0 * kStep + p1, v = p2 * kStep + p3;       // low half: elements 0, 2 (4, 6), high half: 1, 3 (5, 7)
    constexpr uint32_t kWeights = (1u << N) | (1u << 8);           // low half x 2**N + high half
    return __dp2a_lo(v, kWeights, __dp2a_lo(u, kWeights, 0u) * (kStep * kStep));
}
