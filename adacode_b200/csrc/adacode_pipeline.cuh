// Pipelined pack / unpack kernels: tiles are staged through shared memory with asynchronous
// bulk copies (the untiled form of TMA) so that the loads of the next units are in flight
// while the current unit is processed.  Unpacked rows and the sign/mantissa plane are stored straight from
// registers, packed codes and escapes leave through shared memory with bulk stores.  Included by
// adacode_kernels.cu and, without the pack part, by adacode_attention.cu inside their anonymous namespaces.
//
// One CTA = W consumer warps + 1 producer warp, persistent over tiles.  A "unit" is a run of
// whole token rows of one tile, at most W x 1024 elements.  Two geometries are built: the wide one
// (16 warps, units of a whole 128 x 128 tile, 2 CTAs per SM) for the pack kernel, the narrow one
// (8 warps, units of 8192 elements, 4 CTAs per SM) for the unpack kernel, which measured 5-8 % faster
// with four smaller pipelines per SM than with two large ones.
// The pack kernel measured 7 % slower that way (twice the escape slots and unit counts to
// compact) and takes the narrow geometry only for tiles of at most 8192 elements, which would
// leave half the threads of a wide unit idle.
//   producer warp : waits for a free stage, issues the unit's bulk loads (sign/mantissa and
//                   code planes, or source rows) against the stage's "full" mbarrier, and
//                   stages the tile's escape bytes with plain loads
//   consumer warps: wait on "full", work out of shared memory, signal "empty"
// The pack kernel's codes and escapes of a unit leave through ONE bulk store each: the copy engine has a
// sizeable cost per operation, and a variant in which every consumer warp stored its own slice (no
// CTA-wide barrier inside a unit) ran 40 % slower.
// Every mbarrier wait is bounded: after kMaxPolls failed polls the waiter records
// ADACODE_STATUS_TIMEOUT in the status word and carries on (the result is then wrong but the
// kernel still reaches every barrier and terminates).
#pragma once

constexpr int kPCPT = 2;                                   // 16-element chunks per consumer thread and unit

template <int W, int CTAS>
struct PipeGeom {
    static constexpr int kWarps = W;                        // consumer warps
    static constexpr int kConsumers = W * 32;
    static constexpr int kThreads = kConsumers + 32;        // + the producer warp
    static constexpr int kUnit = kConsumers * kPCPT * 16;   // elements per unit
    static constexpr int kCtasPerSm = CTAS;
    static constexpr int kEscStage = 8192;                  // bytes of a tile's escape stream staged with a unit
};
using WideGeom = PipeGeom<16, 2>;
using NarrowGeom = PipeGeom<8, 4>;

// the wide geometry under the names that the helpers default to
constexpr int kConsumerThreads = WideGeom::kConsumers;
constexpr int kUnitElems = WideGeom::kUnit;
constexpr int kStages = 2;
constexpr uint32_t kMaxPolls = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait; on expiry flags the status word and returns anyway (false: the barrier did not
// complete).  Once any wait of the launch has timed out, the others stop waiting as well (they look
// at the status word now and then), so that a broken launch ends in about the time of one expired
// wait.  A consumer whose wait failed keeps computing (it must reach every barrier) but stores
// nothing to global memory any more: it may be looking at a half-written unit description.
__device__ __forceinline__ bool launch_timed_out(const int32_t *status) {
    return (*reinterpret_cast<const volatile int32_t *>(status) & ADACODE_STATUS_TIMEOUT) != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int32_t *status,
                                          uint32_t limit = kMaxPolls) {
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 4095u) == 4095u && launch_timed_out(status)) return false;
    }
    atomicOr(status, ADACODE_STATUS_TIMEOUT);
    return false;
}
// global -> shared bulk copy, completion counted in bytes on `bar`; 16-byte aligned, size % 16 == 0
__device__ __forceinline__ void bulk_load(void *sdst, const void *gsrc, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(sdst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// the box of a four-dimensional tensor map that begins at element 0 of row `row` of (head, batch)
__device__ __forceinline__ void tensor_load(void *sdst, const CUtensorMap *map, int row, int head, int batch, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            smem_u32(sdst)),
        "l"(map), "r"(0), "r"(row), "r"(head), "r"(batch), "r"(smem_u32(bar))
        : "memory");
}
// shared -> global bulk copy, tracked by the issuing thread's bulk group
__device__ __forceinline__ void bulk_store(void *gdst, const void *ssrc, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(ssrc)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// makes shared-memory writes of this thread visible to the async proxy (bulk stores)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
template <int THREADS = kConsumerThreads>
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }

// Inclusive warp scan of kPCPT per-lane counters walked in (k, lane) order (counters <= 16 each, so
// they travel as 16-bit fields).  incl[k] = inclusive rank of (k, lane) within the warp's
// kPCPT x 32 chunks; returns the warp total.
__device__ __forceinline__ int warp_scan_counts(const int (&cnt)[kPCPT], int (&incl)[kPCPT]) {
    static_assert(kPCPT == 2 || kPCPT == 4, "two or four chunks per thread");
    const int lane = threadIdx.x & 31;
    uint32_t a = (uint32_t)cnt[0] | ((uint32_t)cnt[1] << 16);
    uint32_t b = 0;
    if (kPCPT == 4) b = (uint32_t)cnt[kPCPT - 2] | ((uint32_t)cnt[kPCPT - 1] << 16);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t ua = __shfl_up_sync(kFull, a, d);
        uint32_t ub = 0;
        if (kPCPT == 4) ub = __shfl_up_sync(kFull, b, d);
        if (lane >= d) {
            a += ua;
            b += ub;
        }
    }
    const uint32_t ta = __shfl_sync(kFull, a, 31);
    const int t0 = ta & 0xFFFF, t1 = ta >> 16;
    incl[0] = (int)(a & 0xFFFF);
    incl[1] = (int)(a >> 16) + t0;
    int total = t0 + t1;
    if (kPCPT == 4) {
        const uint32_t tb = __shfl_sync(kFull, b, 31);
        incl[kPCPT - 2] = (int)(b & 0xFFFF) + total;
        incl[kPCPT - 1] = (int)(b >> 16) + total + (int)(tb & 0xFFFF);
        total += (int)(tb & 0xFFFF) + (int)(tb >> 16);
    }
    return total;
}

// Rows of one tile handled per unit: whole rows, a multiple of 8 (so that code bytes per unit are a
// multiple of 16), at most UNIT elements (D <= UNIT / 8).
template <int UNIT = kUnitElems>
__host__ __device__ inline int unit_rows_for(int seq_tile, int D) {
    int r = (UNIT / D) & ~7;
    if (r < 8) r = 8;
    return r < seq_tile ? r : seq_tile;
}

// ---------------------------------------------------------------------------------------
// unpack
// ---------------------------------------------------------------------------------------

// Bytes of an escape buffer that are not for escapes: kEscFront in front of the first granule, because
// place_escapes reads the word before an escape, and behind the last one a granule and the words it
// reads ahead.
constexpr int kEscFront = 16;
constexpr int kEscSlack = kEscFront + 32;

struct UnitMeta {
    uint16_t *dst;            // first element of the unit in the destination
    const uint8_t *esc;       // the segment's escape stream
    long long esc_len;
    long long esc_tile_start; // index in esc of the tile's first escape
    int esc_staged;           // escapes of the tile present in shared memory (from index 0 of the tile)
    int esc_shift;            // offset of escape 0 inside the staged bytes
    int elems;
    int left;
    int nbits;
    int first_unit_of_tile;
    long long ds;             // destination row stride in elements
};

// bulk copies need 16-byte aligned shared addresses: every buffer starts on a 128-byte boundary
template <class G>
struct alignas(128) UnpackStageT {
    alignas(128) uint8_t sm[G::kUnit];
    alignas(128) uint8_t codes[G::kUnit / 2];
    alignas(128) uint8_t esc[G::kEscStage + kEscSlack];
};

template <class G>
struct alignas(128) UnpackSmemT {
    UnpackStageT<G> stage[kStages];
    // Unit descriptions live in a ring of their own, twice as deep as the stages: a consumer reads
    // the destination of unit i after it has released stage i % kStages, and the producer writes
    // the description of unit i + 2 * kStages only after every consumer has released unit
    // i + kStages, i.e. after it is done with unit i altogether.  So nobody has to keep a
    // description in registers through a unit.
    alignas(16) UnitMeta meta_ring[2 * kStages];
    alignas(8) uint64_t full[kStages];
    alignas(8) uint64_t empty[kStages];
    // escapes per consumer warp of a unit, by the unit's parity: a warp writes those of unit i + 2 only
    // behind the barrier of unit i + 1, which no warp reaches before it has read those of unit i
    int warp_tot[2][G::kWarps];
};
static_assert(sizeof(UnpackStageT<WideGeom>) % 128 == 0 && sizeof(UnpackStageT<NarrowGeom>) % 128 == 0,
              "stage buffers must stay 128-byte aligned");

struct UnpackPipeArgs {
    // uniform form (seg == nullptr): planes as adacode_pack_tiles wrote them
    const uint8_t *sign_mant;
    const uint8_t *codes;
    const uint8_t *escapes;
    long long escapes_len;
    const int32_t *tile_base;
    const int64_t *seg_off;
    int left, nbits;
    int tb_stride;            // tile t's inclusive base is tile_base[(t + 1) * tb_stride - 1] (1: one entry per tile)
    // table form
    const adacode_segment *seg;
    // common
    int H, BH, seq_tile, D, tile_elems;
    Quotient by_BH, by_H;
    long long n_tiles;
    uint16_t *dst;
    long long db, dh, ds;
    int32_t *status;
};

// Everything the producer needs to know about tile `tile`.
struct TileSrc {
    const uint8_t *sm, *codes, *esc;
    long long esc_len, esc_start;
    int esc_cnt, left, nbits;
    uint16_t *dst;
    long long ds;
};

// Tile bh of a segment (its destination, for a caller that has one, is `base` and the segment's offset).
__device__ __forceinline__ TileSrc resolve_segment_tile(const adacode_segment &sg, int bh, int tile_elems, uint16_t *base, long long ds) {
    TileSrc t;
    t.nbits = sg.nbits, t.left = sg.left;
    t.sm = sg.sign_mant + (long long)bh * tile_elems;
    t.codes = sg.codes + (long long)bh * (tile_elems * sg.nbits / 8);
    t.esc = sg.escapes, t.esc_len = sg.escapes_len;
    const int prev = bh > 0 ? sg.tile_base[bh - 1] : 0;
    t.esc_start = prev;
    t.esc_cnt = sg.tile_base[bh] - prev;
    t.dst = base + sg.dst_seq_offset * ds;
    t.ds = ds;
    return t;
}

__device__ __forceinline__ TileSrc resolve_tile(const UnpackPipeArgs &a, long long tile) {
    TileSrc t;
    const long long blk = (uint32_t)tile / a.by_BH;       // (fewer than 2**31 tiles: their planes fit a GPU)
    const int bh = (int)(tile - blk * a.BH);
    const int b = (uint32_t)bh / a.by_H, h = bh - b * a.H;
    uint16_t *base = a.dst + (long long)b * a.db + (long long)h * a.dh;
    t.ds = a.ds;
    if (a.seg) {
        const adacode_segment sg = a.seg[blk];
        t = resolve_segment_tile(sg, bh, a.tile_elems, base, a.ds);
    } else {
        t.nbits = a.nbits, t.left = a.left;
        t.sm = a.sign_mant + tile * a.tile_elems;
        t.codes = a.codes + tile * (a.tile_elems * a.nbits / 8);
        t.esc = a.escapes, t.esc_len = a.escapes_len;
        const long long seg_start = a.seg_off ? a.seg_off[blk] : 0;
        const long long ts = a.tb_stride > 1 ? a.tb_stride : 1;
        const int prev = bh > 0 ? a.tile_base[tile * ts - 1] : 0;
        t.esc_start = seg_start + prev;
        t.esc_cnt = a.tile_base[tile * ts + ts - 1] - prev;
        t.dst = base + blk * a.seq_tile * a.ds;
    }
    return t;
}

__device__ __forceinline__ long long shfl_ll(long long v, int src) {
    const int lo = __shfl_sync(kFull, (int)(v & 0xFFFFFFFFll), src);
    const int hi = __shfl_sync(kFull, (int)(v >> 32), src);
    return ((long long)hi << 32) | (unsigned int)lo;
}
template <typename T>
__device__ __forceinline__ T *shfl_ptr(T *p, int src) {
    return reinterpret_cast<T *>(shfl_ll((long long)(uintptr_t)p, src));
}
// Lane `src`'s tile description, in every lane of the warp.
__device__ __forceinline__ TileSrc shfl_tile(const TileSrc &m, int src) {
    TileSrc t;
    t.sm = shfl_ptr(m.sm, src), t.codes = shfl_ptr(m.codes, src), t.esc = shfl_ptr(m.esc, src);
    t.esc_len = shfl_ll(m.esc_len, src), t.esc_start = shfl_ll(m.esc_start, src);
    t.esc_cnt = __shfl_sync(kFull, m.esc_cnt, src);
    t.left = __shfl_sync(kFull, m.left, src), t.nbits = __shfl_sync(kFull, m.nbits, src);
    t.dst = shfl_ptr(m.dst, src);
    t.ds = shfl_ll(m.ds, src);
    return t;
}

// The part of a tile's escape stream that is staged in shared memory with each of its units.
// The window [a0, a0 + win) of whole 16-byte granules is fetched with one bulk copy.  It may
// begin up to 15 bytes before the tile's first escape (same granule, ignored), but never reaches
// past the last whole granule of the stream: what lies in the stream's final partial granule
// (`tail` bytes) is fetched with plain loads.
struct EscWindow {
    const uint8_t *a0;
    int win, tail, staged, shift;
};

__device__ __forceinline__ EscWindow esc_window(const TileSrc &t, int most) {
    EscWindow w;
    // stage no more than the stream really holds, so that a short stream is reported as such
    long long avail = t.esc_len - t.esc_start;
    if (avail > t.esc_cnt) avail = t.esc_cnt;
    if (avail > most) avail = most;
    w.staged = avail > 0 ? (int)avail : 0;
    const uint8_t *ea = t.esc + t.esc_start;
    w.shift = (int)((uintptr_t)ea & 15);
    w.a0 = ea - w.shift;
    w.win = (w.shift + w.staged + 15) & ~15;
    w.tail = 0;
    const uintptr_t stream_end = (uintptr_t)(t.esc + t.esc_len);
    if (w.staged > 0 && (uintptr_t)w.a0 + (uintptr_t)w.win > stream_end) {
        w.win -= 16;
        w.tail = (int)(stream_end & 15);
    }
    if (w.staged == 0) w.win = 0;
    return w;
}

// One warp, stage known to be free: describe the unit (rows [row0, row0 + rows) of tile t) in `m` and
// start its bulk copies against `full_bar`.
__device__ __forceinline__ void issue_unit(uint8_t *s_sm, uint8_t *s_codes, uint8_t *s_esc, UnitMeta &m, uint64_t *full_bar,
                                           const TileSrc &t, const EscWindow &w, int row0, int rows, int D, uint16_t *dst,
                                           bool first_unit, int32_t *status, bool withhold = false) {
    const int lane = threadIdx.x & 31;
    if (w.tail > 0) {
        if (lane < w.tail) s_esc[w.win + lane] = w.a0[w.win + lane];
        __syncwarp();
    }
    if (lane == 0) {
        const int elems = rows * D;
        const uint8_t *src_sm = t.sm + (long long)row0 * D;
        const uint8_t *src_cd = t.codes + (long long)row0 * D * t.nbits / 8;
        m.dst = dst;
        m.esc = t.esc, m.esc_len = t.esc_len, m.esc_tile_start = t.esc_start;
        m.esc_staged = w.staged, m.esc_shift = w.shift;
        m.elems = elems, m.left = t.left, m.nbits = t.nbits;
        m.first_unit_of_tile = first_unit;
        m.ds = t.ds;
        const uint32_t cbytes = (uint32_t)elems * t.nbits / 8;
        if (withhold) {
            // testing aid: an empty unit whose "loaded" signal never comes; the consumers' bounded
            // wait runs out, they flag ADACODE_STATUS_TIMEOUT and carry on with nothing to do
            m.elems = 0;
            m.nbits = 1;
        } else if ((((uintptr_t)src_sm | (uintptr_t)src_cd | (uintptr_t)dst) & 15) != 0 || (cbytes & 15) != 0 || t.nbits < 1 ||
            t.nbits > 4) {
            // never start a misaligned bulk copy: flag it and hand over an empty unit
            atomicOr(status, ADACODE_STATUS_MISALIGNED);
            m.elems = 0;
            m.nbits = 1;
            mbar_arrive_expect_tx(full_bar, 0);
        } else {
            mbar_arrive_expect_tx(full_bar, (uint32_t)elems + cbytes + (uint32_t)w.win);
            bulk_load(s_sm, src_sm, (uint32_t)elems, full_bar);
            bulk_load(s_codes, src_cd, cbytes, full_bar);
            if (w.win > 0) bulk_load(s_esc, w.a0, (uint32_t)w.win, full_bar);
        }
    }
}

// A 16-element chunk of a destination row.  32 bytes leave in one instruction where they are aligned
// (a warp then writes 1 KB of whole sectors at once), in two otherwise.
__device__ __forceinline__ void store_chunk(uint16_t *dst, const uint32_t (&w)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]),
                     "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// Escapes of one group whose bytes are not (all) staged in shared memory: byte by byte, from global
// memory beyond the window; a stream that is too short is flagged and gives exponent 0.  Returns the
// bytes in their places (elements 0..3, 4..7, the last one lowest).
__device__ __noinline__ uint2 gather_escapes(uint32_t z, int r, const uint8_t *esc_smem, int staged, const UnitMeta &m,
                                                int32_t *status) {
    const uint8_t *g_esc = m.esc;
    const long long g_len = m.esc_len, g_start = m.esc_tile_start;
    uint2 e = make_uint2(0u, 0u);
#pragma unroll 1
    for (; z != 0; ++r) {
        const int at = 31 - __clz((int)z);                 // the first element has the highest nibble
        z ^= 1u << at;
        uint32_t v = 0;
        if (r < staged) v = esc_smem[r];
        else if (g_start + r < g_len) v = g_esc[g_start + r];
        else atomicOr(status, ADACODE_STATUS_ESCAPE_UNDERRUN);
        const uint32_t b = v << (2 * (at & 15));
        if (at >= 16) e.x |= b;
        else e.y |= b;
    }
    return e;
}

// One unit: staged planes -> registers -> global memory.  The codes are expanded, the escapes placed
// and the bf16 words put together in registers (see spread8), and
// whole sectors are stored straight from there.  The only CTA-wide barrier is the one between the
// escape counts of the warps and their sum.
// Keys and values of [16, 8, 8192, 128] in one launch (268 M elements), with the lookups, the escape loop and the
// bulk store that were here before and now: n = 3, 5 % escapes 188.6 -> 177.7 us (5.2 TB/s, 81 % of what a plain
// copy reaches), n = 2, 34 % escapes 340 -> 177 us, n = 4, 0.1 % escapes 169.7 -> 170.8 us; [1, 8, 20480, 128]
// 38.8 -> 35.0 us; 4 % less each since computed permutes go without the intrinsic's mask, and 4-5 % less since the
// escape masks are found again behind the barrier from the codes' nibbles, and a chunk's row and column share a
// register (spills 72 / 104 -> 68 / 96 bytes of stores / loads, which is not where the time went; what it is has not been measured): n = 3 161.9 -> 154.5 us, n = 2 160.0 -> 154.7 us, n = 4 161.5 -> 160.9 us, the flat
// form of 4096 x 14336 40.2 -> 38.2 us.  What is left over a plain copy (143 us) is waiting at the barrier and for loads, and
// the last round of a launch.  Tried and slower: no producer warp (one warp in turn refills; the others wait for it at the next
// barrier) 201 us; one tile per warp without shared memory or barriers 217-219 us; the finished unit through
// shared memory and a bulk store, which leaves room for three CTAs per SM, 229 us; five CTAs per SM (spills) 223 us;
// four chunks per thread in eight warps, three CTAs per SM, 168 us, in four warps, six CTAs, 220 us.
template <int N, class G>
__device__ __forceinline__ void unpack_unit(const UnpackStageT<G> &st, const UnitMeta &meta, int *warp_tot, int &consumed,
                                            const ExpTable &tab, const uint32_t (&at)[kPCPT],
                                            uint64_t *empty_bar, int32_t *status, bool broken) {
    constexpr int CB = 2 * N;   // code bytes per 16-element chunk
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (meta.first_unit_of_tile) consumed = 0;
    const int chunks = meta.elems >> 4;
    const int c0 = warp * (kPCPT * 32) + lane;

    uint32_t nib[kPCPT][2];
    int zc[kPCPT];
#pragma unroll
    for (int k = 0; k < kPCPT; ++k) {
        const int c = c0 + k * 32;
        uint32_t x[2];
        load_codes16<N>(st.codes + c * CB, x);             // (beyond the unit's end: what lies there, not used)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            nib[k][q] = c < chunks ? spread8<N>(x[q]) : 0x11111111u;      // (beyond the end: no escapes)
        }
        zc[k] = escapes_of(escape_mask<N>(nib[k][0])) + escapes_of(escape_mask<N>(nib[k][1]));
    }
    int incl[kPCPT];
    const int wtot = warp_scan_counts(zc, incl);
    if (lane == 0) warp_tot[warp] = wtot;
    consumer_sync<G::kConsumers>();
    const int others = warp_tot[lane & (G::kWarps - 1)];
    const int before = consumed + (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? others : 0));
    consumed += (int)__reduce_add_sync(kFull, (unsigned)(lane < G::kWarps ? others : 0));
    const uint8_t *const esc = st.esc + kEscFront;
    const int staged = meta.esc_staged, shift = meta.esc_shift;
    uint16_t *const dst = meta.dst;
    const long long ds = meta.ds;
    const bool wide = ((((uintptr_t)dst) | ((uintptr_t)ds * 2)) & 31) == 0;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(esc);
    const auto word = [words](int i) { return words[i]; };
    // (a warp none of whose escapes lies beyond the window, i.e. nearly every one)
    const bool in_window = __all_sync(kFull, before + incl[kPCPT - 1] <= staged);
#pragma unroll
    for (int k = 0; k < kPCPT; ++k) {
        const int r0 = before + incl[k] - zc[k];               // rank inside the tile of the chunk's first escape
        // (hidden from the compiler, which would keep the masks from before the barrier)
        asm volatile("" : "+r"(nib[k][0]), "+r"(nib[k][1]));
        const uint32_t z0 = escape_mask<N>(nib[k][0]), z1 = escape_mask<N>(nib[k][1]);
        const int r1 = r0 + escapes_of(z0);
        uint32_t e0[2], e1[2];
        lookup8<N>(nib[k][0], tab, e0);
        lookup8<N>(nib[k][1], tab, e1);
        if (in_window) {
            place_escapes(z0, shift + r0, word, e0);
            place_escapes(z1, shift + r1, word, e1);
        } else {
            const uint2 g0 = gather_escapes(z0, r0, esc + shift, staged, meta, status);
            e0[0] |= g0.x, e0[1] |= g0.y;
            const uint2 g1 = gather_escapes(z1, r1, esc + shift, staged, meta, status);
            e1[0] |= g1.x, e1[1] |= g1.y;
        }
        const uint4 sv = *reinterpret_cast<const uint4 *>(st.sm + (c0 + k * 32) * 16);
        uint32_t w[8];
        assemble4(sv.x, e0[0], w[0], w[1]);
        assemble4(sv.y, e0[1], w[2], w[3]);
        assemble4(sv.z, e1[0], w[4], w[5]);
        assemble4(sv.w, e1[1], w[6], w[7]);
        if (c0 + k * 32 < chunks && !broken) store_chunk(dst + (long long)(at[k] >> 16) * ds + (at[k] & 0xFFFFu), w, wide);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_bar);    // this warp no longer reads the stage
}

// Consumer warp: wait (bounded) until unit `it` is loaded; false if the wait gave up.
template <class G>
__device__ __forceinline__ bool wait_loaded(UnpackSmemT<G> &s, uint32_t it, int32_t *status, uint32_t poll_limit) {
    // (every lane waits: the ready case is three instructions)
    return __all_sync(kFull, mbar_wait(&s.full[it % kStages], (it / kStages) & 1, status, poll_limit));
}

// Units it, it + 1, ... as long as they carry code length N and window `left`; returns the first unit
// that does not, already waited for, or n_units.
template <int N, class G>
__device__ __forceinline__ uint32_t unpack_run(UnpackSmemT<G> &s, uint32_t it, uint32_t n_units, int left, int &consumed,
                                               const uint32_t (&at)[kPCPT], bool &broken,
                                               int32_t *status, uint32_t poll_limit) {
    const ExpTable tab = exp_table<N>(left);
    for (;;) {
        const int stg = it % kStages;
        unpack_unit<N>(s.stage[stg], s.meta_ring[it % (2 * kStages)], s.warp_tot[it & 1], consumed, tab, at,
                       &s.empty[stg], status, broken);
        if (++it >= n_units) return it;
        broken |= !wait_loaded(s, it, status, poll_limit);
        const UnitMeta &next = s.meta_ring[it % (2 * kStages)];
        if (next.nbits != N || next.left != left) return it;
    }
}

constexpr int kMaxJobs = 8;

// A dense copy of bf16 rows (adacode_row_copy), by `n_workers` threads of which this is `worker`.
__device__ __forceinline__ void copy_rows(const adacode_row_copy &c, uint32_t worker, uint32_t n_workers) {
    const uint32_t vec = (uint32_t)c.D / 8, rows = (uint32_t)c.rows;
    const uint32_t total = (uint32_t)c.B * (uint32_t)c.H * rows * vec;      // (checked by the host: below 2**31)
#pragma unroll 2
    for (uint32_t i = worker; i < total; i += n_workers) {
        const uint32_t r = i / vec, v = i - r * vec, bh = r / rows, t = r - bh * rows;
        const uint32_t b = bh / (uint32_t)c.H, h = bh - b * (uint32_t)c.H;
        const uint16_t *src = (const uint16_t *)c.src_bf16 + b * c.src_b + h * c.src_h + t * c.src_s;
        uint16_t *dst = (uint16_t *)c.dst_bf16 + b * c.dst_b + h * c.dst_h + t * c.dst_s;
        reinterpret_cast<uint4 *>(dst)[v] = reinterpret_cast<const uint4 *>(src)[v];
    }
}

struct RowCopies {
    adacode_row_copy copy[kMaxJobs];
    int n;
};

// The end of a flat tensor that is less than a tile: `blocks` blocks of `block_elems` elements from block `first` on, the last
// one of last_elems (a multiple of 8).
struct FlatRest {
    const uint8_t *sign_mant, *codes, *escapes;            // of the whole tensor
    long long escapes_len;
    const int32_t *block_base;
    uint16_t *dst;
    int first, blocks, block_elems, last_elems, left, nbits;
};

// One of those blocks by the consumer threads of a CTA, eight elements per thread (a block has 1024 at most): bound by
// the latency of its loads, beside the tiles of the same launch.
template <class G>
__device__ __noinline__ void unpack_flat_block(const FlatRest &f, int b, int *warp_tot, int32_t *status) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbits = f.nbits, groups = (b == f.blocks - 1 ? f.last_elems : f.block_elems) / 8;
    const long long blk = f.first + b, g = blk * (f.block_elems / 8) + tid;        // this thread's group of the tensor
    const uint32_t mask = (1u << nbits) - 1u;
    uint32_t x = 0;
    uint2 sv = make_uint2(0u, 0u);
    long long start = 0;
    int count = 0;
    if (tid < groups) {
        for (int i = 0; i < nbits; ++i) x = (x << 8) | f.codes[g * nbits + i];
        sv = *reinterpret_cast<const uint2 *>(f.sign_mant + g * 8);
        for (int k = 0; k < 8; ++k) count += ((x >> (k * nbits)) & mask) == 0u;
    }
    if (blk > 0) start = f.block_base[blk - 1];
    int incl = count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += u;
    }
    if (lane == 31) warp_tot[warp] = incl;
    consumer_sync<G::kConsumers>();
    for (int w = 0; w < warp; ++w) incl += warp_tot[w];
    if (tid < groups) {
        long long r = start + incl - count;
        alignas(16) uint16_t out[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t code = (x >> ((7 - k) * nbits)) & mask, s = ((k < 4 ? sv.x : sv.y) >> (8 * (k & 3))) & 0xFFu;
            uint32_t e = (code + (uint32_t)f.left) & 0xFFu;
            if (code == 0u) {
                if (r < f.escapes_len) e = f.escapes[r];
                else e = 0u, atomicOr(status, ADACODE_STATUS_ESCAPE_UNDERRUN);
                ++r;
            }
            out[k] = (uint16_t)(((s & 0x80u) << 8) | (e << 7) | (s & 0x7Fu));
        }
        *reinterpret_cast<uint4 *>(f.dst + g * 8) = *reinterpret_cast<const uint4 *>(out);
    }
    consumer_sync<G::kConsumers>();                        // (the counts are read)
}

// Up to kMaxJobs destinations in one launch; job j owns the tiles [tile0[j], tile0[j + 1]).
struct UnpackJobsArgs {
    UnpackPipeArgs job[kMaxJobs];
    RowCopies rows;           // dense rows that go along
    FlatRest rest;            // blocks that go along (rest.blocks == 0: none)
    long long tile0[kMaxJobs + 1];
    int n_jobs;
    uint32_t poll_limit;      // bound of every on-chip wait (kMaxPolls unless a test lowered it)
    int withhold_unit;        // testing aid: CTA 0's producer never signals this unit as loaded (-1: off)
};

template <class G>
__global__ void __launch_bounds__(G::kThreads, G::kCtasPerSm) k_unpack_pipe(const __grid_constant__ UnpackJobsArgs ja) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    UnpackSmemT<G> &s = *reinterpret_cast<UnpackSmemT<G> *>(smem_raw);
    const int tid = threadIdx.x;
    const UnpackPipeArgs &a0 = ja.job[0];          // geometry and status word are common to all jobs
    const long long n_tiles = ja.tile0[ja.n_jobs];
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], G::kWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 2 * kStages) {
        // an empty unit: what a consumer sees if it gives up waiting before the first description is written
        UnitMeta &m = s.meta_ring[tid];
        m.dst = nullptr, m.esc = nullptr, m.esc_len = 0, m.esc_tile_start = 0, m.esc_staged = 0, m.esc_shift = 0;
        m.elems = 0, m.left = 0, m.nbits = 1, m.first_unit_of_tile = 1, m.ds = 0;
    }
    __syncthreads();
    // launched as a programmatic dependent of its predecessor in the stream: no global memory is touched above
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int unit_rows = unit_rows_for<G::kUnit>(a0.seq_tile, a0.D);
    const int units_per_tile = (a0.seq_tile + unit_rows - 1) / unit_rows;

    if (tid >= G::kConsumers) {
        // ---------------- producer warp ----------------
        // Tile metadata sits behind two dependent global loads (segment record, then the tile's
        // escape range).  Each lane resolves one of this CTA's next 32 tiles, so those round trips
        // are paid once per 32 tiles and never between "stage free" and "loads issued".
        const int lane = tid & 31;
        uint32_t it = 0;
        const long long my_tiles =
            n_tiles > (long long)blockIdx.x ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
        for (long long base = 0; base < my_tiles; base += 32) {
            TileSrc mine = {};
            if (base + lane < my_tiles) {
                const long long tile = blockIdx.x + (base + lane) * (long long)gridDim.x;
                int j = 0;
                while (j + 1 < ja.n_jobs && tile >= ja.tile0[j + 1]) ++j;
                mine = resolve_tile(ja.job[j], tile - ja.tile0[j]);
            }
            const int n_here = (int)(my_tiles - base < 32 ? my_tiles - base : 32);
            for (int j = 0; j < n_here; ++j) {
                const TileSrc t = shfl_tile(mine, j);
                const EscWindow w = esc_window(t, G::kEscStage);
                for (int u = 0; u < units_per_tile; ++u, ++it) {
                    const int stg = it % kStages;
                    mbar_wait(&s.empty[stg], ((it / kStages) & 1) ^ 1, a0.status, ja.poll_limit);
                    const int row0 = u * unit_rows;
                    const int rows = min(unit_rows, a0.seq_tile - row0);
                    UnpackStageT<G> &st = s.stage[stg];
                    issue_unit(st.sm, st.codes, st.esc + kEscFront, s.meta_ring[it % (2 * kStages)], &s.full[stg], t, w, row0, rows, a0.D,
                               t.dst + (long long)row0 * t.ds,
                               u == 0, a0.status, blockIdx.x == 0 && (int)it == ja.withhold_unit);
                }
            }
        }
        // Do not leave while a copy into this CTA's shared memory may still be in flight: after a
        // timed-out launch the consumers can be ahead of the data (a bounded wait, like all others).
        if (launch_timed_out(a0.status))
            for (uint32_t k = it > kStages ? it - kStages : 0; k < it; ++k)
                if (!(blockIdx.x == 0 && (int)k == ja.withhold_unit))
                    mbar_wait(&s.full[k % kStages], (k / kStages) & 1, a0.status, ja.poll_limit);
        return;
    }

    // ---------------- consumer warps ----------------
    // the dense rows first, while the first units are on their way
    for (int j = 0; j < ja.rows.n; ++j)
        copy_rows(ja.rows.copy[j], blockIdx.x * (uint32_t)G::kConsumers + tid, gridDim.x * (uint32_t)G::kConsumers);
    for (int b = blockIdx.x; b < ja.rest.blocks; b += gridDim.x) unpack_flat_block<G>(ja.rest, b, s.warp_tot[0], a0.status);
    int consumed = 0;
    bool broken = false;                  // a wait of this warp ran out: compute on, store nothing
    // row (upper half) and column of this thread's chunks inside a unit (a chunk never crosses a row: D % 16 == 0)
    uint32_t at[kPCPT];
#pragma unroll
    for (int k = 0; k < kPCPT; ++k) {
        const int e0 = ((tid >> 5) * (kPCPT * 32) + k * 32 + (tid & 31)) * 16;
        at[k] = ((uint32_t)(e0 / a0.D) << 16) | (uint32_t)(e0 % a0.D);
    }
    // (the consumers only count units: which tile a unit belongs to is in its description)
    const uint32_t my_units =
        n_tiles > (long long)blockIdx.x
            ? (uint32_t)((n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) * (uint32_t)units_per_tile
            : 0u;
    // Units of one code length and window are handled by a loop of their own (unpack_run<N>), so
    // that the compiler schedules each code length's loop body by itself; this outer loop only
    // takes over when the code length or the window changes.
    uint32_t it = 0;
    while (it < my_units) {
        broken |= !wait_loaded(s, it, a0.status, ja.poll_limit);      // returns at once if unpack_run waited already
        const UnitMeta &meta = s.meta_ring[it % (2 * kStages)];
        const int lf = meta.left;
        switch (meta.nbits) {
            case 1: it = unpack_run<1>(s, it, my_units, lf, consumed, at, broken, a0.status, ja.poll_limit); break;
            case 2: it = unpack_run<2>(s, it, my_units, lf, consumed, at, broken, a0.status, ja.poll_limit); break;
            case 3: it = unpack_run<3>(s, it, my_units, lf, consumed, at, broken, a0.status, ja.poll_limit); break;
            default: it = unpack_run<4>(s, it, my_units, lf, consumed, at, broken, a0.status, ja.poll_limit); break;
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

#ifndef ADACODE_PIPELINE_UNPACK_ONLY
// ---------------------------------------------------------------------------------------
// pack
// ---------------------------------------------------------------------------------------

// In-window histogram over several group words at once.  Bit i of a code lands on the least
// significant bit of its N-bit slot, so N groups (4 for N <= 2) can be overlaid on one 32-bit
// word: plane[i] then holds bit i of up to 32 codes.
//
// What is counted is not "how many codes equal v" (one three-input AND with complements, a mask
// and a population count per value) but, for every non-empty proper subset m of the N code bits,
// "how many codes have all bits of m set" (f(m): one AND of the planes named by m, no AND at all
// for single bits).  Together with the number of elements f(0) and the number of escapes x(0),
// which the kernel knows anyway, the per-value counts follow at flush time by inverting the
// superset sums: f(full) = (-1)^N (x(0) - sum_{m != full} (-1)^|m| f(m)), then
// x(c) = sum_{m >= c} (-1)^(|m|-|c|) f(m).  For N = 3 that is 6 population counts and 3 ANDs per
// 24 elements instead of 7 and 14; for N = 1 nothing at all.
template <int N>
struct GroupsPerWord { static constexpr int v = (N == 3) ? 3 : 4; };

template <int N>
__device__ __forceinline__ uint32_t overlay_shift(int j) {
    if (N >= 3) return (uint32_t)j;                           // sub-slot offsets 0..N-1
    if (N == 2) return (uint32_t)((j & 1) + 16 * (j >> 1));   // 16-bit halves, two sub-slot offsets
    return (uint32_t)(8 * j);                                 // N == 1: one byte per group
}

// Counters live in registers, two 16-bit fields per register: field 0 counts elements, field m
// (0 < m < 2^N - 1) the codes with all bits of m set, field 2^N - 1 the escapes.  A thread adds at
// most 32 to a field per unit, so the fields are flushed every 1024 units at the latest.
template <int N>
struct HistRegs { static constexpr int v = (1 << N) / 2 > 0 ? (1 << N) / 2 : 1; };

template <int N>
__device__ __forceinline__ void bump_field(uint32_t (&cnt2)[HistRegs<N>::v], int field, uint32_t by) {
    cnt2[field >> 1] = by * ((field & 1) ? 65536u : 1u) + cnt2[field >> 1];
}

template <int N, int NG>
__device__ __forceinline__ void count_codes_overlaid(const uint32_t (&g)[NG], uint32_t (&cnt2)[HistRegs<N>::v]) {
    constexpr int GPW = GroupsPerWord<N>::v;
    constexpr int FULL = (1 << N) - 1;
    constexpr uint32_t M = SlotLsb<N>::v;
#pragma unroll
    for (int base = 0; base < NG; base += GPW) {
        uint32_t plane[N];
#pragma unroll
        for (int i = 0; i < N; ++i) plane[i] = 0;
#pragma unroll
        for (int j = 0; j < GPW; ++j) {
            if (base + j < NG) {
                const uint32_t sh = overlay_shift<N>(j);
#pragma unroll
                for (int i = 0; i < N; ++i) plane[i] = ((g[base + j] >> i) & M) * (1u << sh) + plane[i];
            }
        }
#pragma unroll
        for (int m = 1; m < FULL; ++m) {
            uint32_t all = 0xFFFFFFFFu;
#pragma unroll
            for (int i = 0; i < N; ++i)
                if ((m >> i) & 1) all &= plane[i];
            bump_field<N>(cnt2, m, (uint32_t)__popc(all));
        }
    }
}

struct PackUnitMeta {
    uint8_t *sm_dst;       // sign/mantissa bytes of the unit
    uint8_t *code_dst;     // code bytes of the unit
    uint8_t *esc_dst;      // the unit's escape slot in the scratch
    int32_t *unit_count;   // where the unit's escape count goes
    int32_t *tile_count;   // where the tile's escape count goes (written with the last unit)
    int32_t *block_counts; // flat layout: where the counts of the unit's blocks go
    int elems;
    int first_unit_of_tile;
    int last_unit_of_tile;
    int job;               // index into PackPipeArgs::job
};

template <class G>
struct alignas(128) PackStageT {
    alignas(128) uint16_t in[G::kUnit];
};

template <class G>
struct alignas(128) PackSmemT {
    PackStageT<G> stage[kStages];
    alignas(128) uint8_t codes[G::kUnit / 2];
    alignas(128) uint8_t esc[G::kUnit];      // worst case: every element of a unit escapes
    alignas(16) PackUnitMeta meta_ring[2 * kStages];   // unit descriptions (see UnpackSmemT::meta_ring)
    alignas(8) uint64_t full[kStages];
    alignas(8) uint64_t empty[kStages];
    int warp_tot[G::kWarps];
    int hist[256];
    int is_last;
    long long carry;
    long long job_off[kMaxJobs];
    int scan[G::kWarps];
};
static_assert(sizeof(PackStageT<WideGeom>) % 128 == 0 && sizeof(PackStageT<NarrowGeom>) % 128 == 0,
              "stage buffers must stay 128-byte aligned");

// One tensor of a pack launch.  All jobs of a launch share B, H, seq_tile, D and the code length;
// job j owns the global tiles [tile0, tile0 + BH * n_blocks) and the global blocks [blk0, blk0 + n_blocks).
struct PackJob {
    const uint16_t *src;
    int64_t sb, sh, ss;
    uint8_t *sign_mant, *codes, *escapes;
    int64_t capacity;
    int32_t *tile_base;
    int64_t *seg_off;
    int32_t *hist;           // nullable
    int64_t tile0;
    int blk0, n_blocks, left, pad;
};

// A small device buffer that goes to page-locked host memory, every word (low half of 64 bits) together with a token that says
// it has arrived: a flag behind the words would have to wait for them to cross the bus.
struct Report {
    const uint32_t *src;
    uint64_t *dst;
    uint32_t words, token;
};

// By a whole CTA.  Word and token are ONE scalar store: the parts of a vector store may become visible in any order, and the
// host would take an old word for the one that its token announces.  The caller has seen to it that everything else that its
// kernel writes (outputs, the scratch's counters) is written for the whole GPU by now: the host goes on when it has the
// words, not when the kernel ends.  (A fence at the system's scope here costs 1.7 us of 45 for one block, 4 us of 107 for 20 480 tokens.)
__device__ __forceinline__ void send_report(const Report &r) {
    for (uint32_t i = threadIdx.x; i < r.words; i += blockDim.x) {
        const uint64_t v = (uint64_t)r.token << 32 | __ldcg(r.src + i);
        asm volatile("st.relaxed.sys.global.b64 [%0], %1;" ::"l"(r.dst + i), "l"(v) : "memory");
    }
}

struct PackPipeArgs {
    PackJob job[kMaxJobs];
    int n_jobs;
    int H, BH, seq_tile, D, tile_elems;
    Quotient by_BH, by_H;
    int64_t n_tiles;          // over all jobs
    uint8_t *esc_scratch;     // n_tiles * tile_elems bytes, global tile t owns [t * tile_elems, ...)
    int32_t *tile_counts;     // n_tiles
    int32_t *unit_counts;     // n_tiles * units_per_tile
    int64_t *blk_off;         // over all blocks of the launch: escapes before global block i (n_blocks_total + 1)
    unsigned int *done;       // two counters (CTAs of the pack, of the compaction), zero on entry, zero on exit
    int unit_rows, units_per_tile;
    // Flat layout (one job): a tile holds several escape-base blocks.  The pack kernel leaves block_counts, for every 1024
    // elements the inclusive counts of their blocks (1024 / block_elems of them), the compaction makes block_base of them.
    int32_t *block_counts, *block_base;
    int block_per_1024;
    int scan_in_pack;         // offsets by the pack kernel's last CTA (else by the compaction's CTAs)
    Report report;            // what the compaction's last CTA hands to the host (words == 0: nothing)
    int32_t *status;
    uint32_t poll_limit;      // bound of every on-chip wait (kMaxPolls unless a test lowered it)
};

// What the pack kernel gets.  map[j] describes job j's source as rows of D elements over (row, head, batch) if
// use_map[j]: sources whose rows do not follow each other, e.g. a [B, S, H, D] projection seen as [B, H, S, D].
struct PackKernelArgs {
    PackPipeArgs pa;
    int use_map[kMaxJobs];
    alignas(64) CUtensorMap map[kMaxJobs];
};

__device__ __forceinline__ int job_of_tile(const PackPipeArgs &pa, int64_t tile) {
    int j = 0;
    while (j + 1 < pa.n_jobs && tile >= pa.job[j + 1].tile0) ++j;
    return j;
}

// Turn per-tile escape counts into per-segment inclusive tile bases and segment offsets (per job).
// Run by the consumer threads of the CTA that finished last, while the rest of the GPU is idle,
// so it is kept short: every thread takes a run of kScanRun consecutive tiles; the counts of the
// next pass (threads x kScanRun tiles) are fetched while the current pass is worked on, so the
// memory round trip of a pass is hidden; one block scan of the run totals gives every tile its
// prefix; and the escape offsets of the blocks that begin inside the pass travel through shared
// memory (`boff`, one entry per block touched by the pass, in the idle staging buffers), not
// through global memory.
constexpr int kScanRun = 8;

template <class G>
__device__ __forceinline__ void scan_tile_counts(const PackPipeArgs &pa, long long *s_carry, int *s_scan,
                                                 long long *s_job_off, long long *boff_raw) {
    // All offsets of a launch fit 32 bits (it has fewer than 2**31 elements), and a thread walks
    // consecutive tiles, so block index, position in the block and job advance by comparison:
    // one division per thread and pass.  (One SM does all of this while the others wait.)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per_pass = G::kConsumers * kScanRun;
    const int n_tiles = (int)pa.n_tiles, BH = pa.BH;
    int *carry = reinterpret_cast<int *>(s_carry);
    int *job_off = reinterpret_cast<int *>(s_job_off);
    int *boff = reinterpret_cast<int *>(boff_raw);
    if (tid == 0) {
        *carry = 0;
        pa.blk_off[0] = 0;
        boff[0] = 0;
    }
    if (tid < kMaxJobs) job_off[tid] = 0;
    if (tid < pa.n_jobs) pa.job[tid].seg_off[0] = 0;
    int c[kScanRun], nxt[kScanRun];
#pragma unroll
    for (int i = 0; i < kScanRun; ++i) {
        const int t = tid * kScanRun + i;
        c[i] = t < n_tiles ? __ldcg(pa.tile_counts + t) : 0;
    }
    consumer_sync<G::kConsumers>();
    for (int pass = 0; pass < n_tiles; pass += per_pass) {
        const int t0 = pass + tid * kScanRun;
#pragma unroll
        for (int i = 0; i < kScanRun; ++i) {
            const int t = t0 + per_pass + i;
            nxt[i] = t < n_tiles ? __ldcg(pa.tile_counts + t) : 0;
        }
        int run = 0;
#pragma unroll
        for (int i = 0; i < kScanRun; ++i) run += c[i];
        int x = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += u;
        }
        if (lane == 31) s_scan[warp] = x;
        consumer_sync<G::kConsumers>();
        int wp = 0, tot = 0;
#pragma unroll
        for (int i = 0; i < G::kWarps; ++i) {
            const int v = s_scan[i];
            wp += (i < warp) ? v : 0;
            tot += v;
        }
        const int gb0 = pass / BH;                        // the block the pass begins in; boff[0] is its offset
        const int gb_first = t0 / BH, rem_first = t0 - gb_first * BH;
        int incl = *carry + wp + (x - run);               // escapes before this thread's run
        int inc[kScanRun];
        {
            int gb = gb_first, rem = rem_first;
#pragma unroll
            for (int i = 0; i < kScanRun; ++i) {
                incl += c[i];
                inc[i] = incl;                            // inclusive prefix over the whole launch
                if (++rem == BH) {                        // tile t0 + i ends block gb
                    rem = 0;
                    ++gb;
                    if (t0 + i < n_tiles) {
                        pa.blk_off[gb] = incl;
                        boff[gb - gb0] = incl;
                        for (int j = 1; j < pa.n_jobs; ++j)
                            if (pa.job[j].blk0 == gb) job_off[j] = incl;
                    }
                }
            }
        }
        consumer_sync<G::kConsumers>();                   // the offsets of the blocks of this pass are in boff
        if (t0 < n_tiles) {
            int gb = gb_first, rem = rem_first;
            int j = job_of_tile(pa, t0);
            int j_end = j + 1 < pa.n_jobs ? (int)pa.job[j + 1].tile0 : n_tiles;
            int32_t *tb = pa.job[j].tile_base - pa.job[j].tile0;
            int start = boff[gb - gb0];                   // offset at which block gb begins
#pragma unroll
            for (int i = 0; i < kScanRun; ++i) {
                const int t = t0 + i;
                if (t < n_tiles) {
                    if (t == j_end) {
                        ++j;
                        j_end = j + 1 < pa.n_jobs ? (int)pa.job[j + 1].tile0 : n_tiles;
                        tb = pa.job[j].tile_base - pa.job[j].tile0;
                    }
                    tb[t] = inc[i] - start;
                    if (++rem == BH) {
                        rem = 0;
                        ++gb;
                        pa.job[j].seg_off[gb - pa.job[j].blk0] = (long long)(inc[i] - job_off[j]);
                        start = inc[i];                   // = boff[gb - gb0]
                    }
                }
            }
        }
        // the block the next pass begins in may have begun in this one
        const int gb1 = (pass + per_pass) / BH;
        const int carry_off = boff[gb1 - gb0];
        consumer_sync<G::kConsumers>();
        if (tid == 0) {
            *carry += tot;
            boff[0] = carry_off;
        }
#pragma unroll
        for (int i = 0; i < kScanRun; ++i) c[i] = nxt[i];
        // (no barrier here: what thread 0 just wrote is read after the next pass's first barrier)
    }
    if (tid == 0) *pa.done = 0u;
}

// Per-thread counter fields -> the CTA's shared histogram: the fields are summed over the warp, the
// superset sums inverted (see count_codes_overlaid) and the per-value counts added by lane 0.
template <int N>
__device__ __forceinline__ void flush_code_counts(uint32_t (&cnt2)[HistRegs<N>::v], int left, int *s_hist) {
    constexpr int FULL = (1 << N) - 1;
    const int lane = threadIdx.x & 31;
    int f[1 << N];
#pragma unroll
    for (int m = 0; m <= FULL; ++m)
        f[m] = (int)__reduce_add_sync(kFull, (cnt2[m >> 1] >> (16 * (m & 1))) & 0xFFFFu);
    // f[FULL] holds the escapes x(0); f(full) follows from x(0) = sum_m (-1)^|m| f(m)
    int alt = 0;
#pragma unroll
    for (int m = 0; m < FULL; ++m) alt += (__builtin_popcount(m) & 1) ? -f[m] : f[m];
    f[FULL] = (N & 1) ? alt - f[FULL] : f[FULL] - alt;
    // inverse of the superset sums, one code bit at a time
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int m = 0; m <= FULL; ++m)
            if (!((m >> i) & 1)) f[m] -= f[m | (1 << i)];
#pragma unroll
    for (int v = 1; v <= FULL; ++v) {
        const int bin = left + v;
        if (lane == 0 && f[v] != 0 && bin >= 0 && bin < 256) atomicAdd(&s_hist[bin], f[v]);
    }
#pragma unroll
    for (int v = 0; v < HistRegs<N>::v; ++v) cnt2[v] = 0;
}

// FULL: the unit has G::kUnit elements (every thread has both of its chunks), so nothing is predicated.
template <int N, bool HIST, bool FLAT, class G, bool FULL>
__device__ __forceinline__ void pack_unit(PackSmemT<G> &s, const PackStageT<G> &st, const PackUnitMeta &m,
                                          uint64_t *empty_bar, int &running, uint32_t (&cnt2)[HistRegs<N>::v],
                                          uint32_t neg_left, bool broken) {
    constexpr int CB = 2 * N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (m lives in the description ring: its destination fields are read where the unit is stored)
    if (m.first_unit_of_tile) running = 0;
    const int chunks = FULL ? G::kUnit / 16 : m.elems >> 4;

    uint32_t g[kPCPT * 2], zm[kPCPT][2];
    int zc[kPCPT];
#pragma unroll
    for (int k = 0; k < kPCPT; ++k) {
        const int c = warp * (kPCPT * 32) + k * 32 + lane;
        const bool valid = FULL || c < chunks;
        uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
        if (valid) {
            const uint4 *p = reinterpret_cast<const uint4 *>(st.in + c * 16);
            w0 = p[0];
            w1 = p[1];
        }
        const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
        uint32_t smw[4], pair[8];
#pragma unroll
        for (int q = 0; q < 4; ++q)       // four elements: their low bytes [e0 m6..m0] and high bytes [s e7..e1]
            smw[q] = bit_select(0x80808080u, __byte_perm(w[2 * q], w[2 * q + 1], 0x7531), __byte_perm(w[2 * q], w[2 * q + 1], 0x6420));
#pragma unroll
        for (int i = 0; i < 8; ++i) pair[i] = encode_pair<N>(w[i], neg_left);
        const uint32_t gg[2] = {join_codes<N>(pair[0], pair[1], pair[2], pair[3]),
                                join_codes<N>(pair[4], pair[5], pair[6], pair[7])};
        g[2 * k] = valid ? gg[0] : 0u;
        g[2 * k + 1] = valid ? gg[1] : 0u;
        zm[k][0] = valid ? zero_slots<N>(gg[0]) : 0u;
        zm[k][1] = valid ? zero_slots<N>(gg[1]) : 0u;
        zc[k] = __popc(zm[k][0]) + __popc(zm[k][1]);
        if (valid && !broken) *reinterpret_cast<uint4 *>(m.sm_dst + c * 16) = make_uint4(smw[0], smw[1], smw[2], smw[3]);
    }
    if (HIST) {
        count_codes_overlaid<N, kPCPT * 2>(g, cnt2);
        const int first = warp * (kPCPT * 32) + lane;
        const int mine = FULL ? 32 : (first < chunks ? 16 : 0) + (first + 32 < chunks ? 16 : 0);  // elements this thread encoded
        bump_field<N>(cnt2, 0, (uint32_t)mine);
        bump_field<N>(cnt2, (1 << N) - 1, (uint32_t)(zc[0] + zc[1]));
    }

    int incl[kPCPT];
    const int wtot = warp_scan_counts(zc, incl);
    if (lane == 0) s.warp_tot[warp] = wtot;
    if (FLAT && !broken && m.elems > 0) {
        // this warp's 1024 elements are one block (N = 1, 3), two of 512 (2) or four of 256 (4)
        if (N == 2) {
            if (lane == 31) *reinterpret_cast<int2 *>(m.block_counts + 2 * warp) = make_int2(incl[0], incl[1]);
        } else if (N == 4) {
            if ((lane & 15) == 15) {
                m.block_counts[4 * warp + (lane >> 4)] = incl[0];
                m.block_counts[4 * warp + 2 + (lane >> 4)] = incl[1];
            }
        } else if (lane == 0) {
            m.block_counts[warp] = wtot;
        }
    }
    bulk_wait_read();      // the previous unit's stores have finished reading the out buffers
    consumer_sync<G::kConsumers>();
    const int others = s.warp_tot[lane & (G::kWarps - 1)];
    const int wprefix = (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? others : 0));
    const int unit_tot = (int)__reduce_add_sync(kFull, (unsigned)(lane < G::kWarps ? others : 0));
    static_assert(kPCPT == 2, "the escape loop below walks the two chunks of a thread together");
    const int c0 = warp * (kPCPT * 32) + lane;
#pragma unroll
    for (int k = 0; k < kPCPT; ++k) {
        const int c = c0 + k * 32;
        if (FULL || c < chunks) {
            const uint32_t gg[2] = {g[2 * k], g[2 * k + 1]};
            store_chunk_codes<N, 16>(s.codes + c * CB, gg);
        }
    }
    if (zc[0] + zc[1] != 0) {
        // One loop over the escapes of both chunks: chunk 0 elements 0..15, then chunk 1 elements 0..15, from the
        // most significant bit of the mask.  A warp iterates as often as its busiest lane has escapes, and counts over
        // 32 elements vary much less than those over 8, so this takes about half the iterations of four loops.
        uint32_t todo = (compress_slots<N>(zm[0][0]) << 24) | (compress_slots<N>(zm[0][1]) << 16) |
                        (compress_slots<N>(zm[1][0]) << 8) | compress_slots<N>(zm[1][1]);
        uint8_t *out = s.esc + wprefix + incl[0] - zc[0];
        const int skip = incl[1] - zc[1] - incl[0];        // from chunk 0's escape bytes to chunk 1's
        const uint16_t *src = st.in + c0 * 16;
        // The mask is shifted up past each escape (pos: elements behind us): keys and values [64, 8, 4096, 128] at 3 bits with
        // histograms 372 -> 363 us, [16, 8, 8192, 128] at 2 bits 193 -> 189 us against clearing the bit that was found.
        int pos = 0;
        while (todo) {
            const int z = __clz(todo);
            todo = (todo << z) << 1;
            pos += z;
            // (chunk 1 lies 32 chunks = 512 elements further on)
            const uint32_t e = src[pos + (pos >> 4) * 496] >> 7;
            out[(pos >> 4) * skip] = (uint8_t)e;
            ++out, ++pos;
        }
    }
    mbar_arrive(empty_bar);
    fence_async_smem();
    consumer_sync<G::kConsumers>();
    running += unit_tot;
    if (tid == 0 && !broken) {
        if (m.elems > 0) {
            bulk_store(m.code_dst, s.codes, (uint32_t)m.elems * N / 8);
            if (unit_tot > 0) bulk_store(m.esc_dst, s.esc, (uint32_t)((unit_tot + 15) & ~15));
            bulk_commit();
        }
        *m.unit_count = unit_tot;
        if (m.last_unit_of_tile) *m.tile_count = running;
    }
}

template <int N, bool HIST, bool FLAT, class G>
__global__ void __launch_bounds__(G::kThreads, G::kCtasPerSm) k_pack_pipe(const __grid_constant__ PackKernelArgs ka) {
    const PackPipeArgs &pa = ka.pa;
    static_assert(G::kConsumers >= 256, "one consumer thread per histogram bin");
    extern __shared__ __align__(128) uint8_t smem_raw[];
    PackSmemT<G> &s = *reinterpret_cast<PackSmemT<G> *>(smem_raw);
    const int tid = threadIdx.x;
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], G::kConsumers);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (HIST && tid < 256) s.hist[tid] = 0;
    if (tid < 2 * kStages) {
        // an empty unit: what a consumer sees if it gives up waiting before the first description is written
        PackUnitMeta &m = s.meta_ring[tid];
        m.sm_dst = m.code_dst = m.esc_dst = nullptr, m.unit_count = m.tile_count = m.block_counts = nullptr;
        m.elems = 0, m.first_unit_of_tile = 1, m.last_unit_of_tile = 0, m.job = 0;
    }
    __syncthreads();
    // launched as a programmatic dependent of its predecessor in the stream: no global memory is touched above
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int unit_rows = pa.unit_rows, upt = pa.units_per_tile;

    if (tid >= G::kConsumers) {
        // ---------------- producer warp ----------------
        const int lane = tid & 31;
        uint32_t it = 0;
        for (int64_t tile = blockIdx.x; tile < pa.n_tiles; tile += gridDim.x) {
            const int j = job_of_tile(pa, tile);
            const PackJob &jb = pa.job[j];
            const int64_t lt = tile - jb.tile0;
            const int64_t blk = (uint32_t)lt / pa.by_BH;
            const int bh = (int)(lt - blk * pa.BH);
            const int b = (uint32_t)bh / pa.by_H, h = bh - b * pa.H;
            const uint16_t *tsrc = jb.src + (int64_t)b * jb.sb + (int64_t)h * jb.sh + blk * pa.seq_tile * jb.ss;
            const bool rows_contig = (jb.ss == pa.D), use_map = ka.use_map[j] != 0;
            for (int u = 0; u < upt; ++u, ++it) {
                const int stg = it % kStages;
                PackStageT<G> &st = s.stage[stg];
                mbar_wait(&s.empty[stg], ((it / kStages) & 1) ^ 1, pa.status, pa.poll_limit);
                const int row0 = u * unit_rows;
                const int rows = min(unit_rows, pa.seq_tile - row0);
                const int elems = rows * pa.D;
                if (lane == 0) {
                    PackUnitMeta &m = s.meta_ring[it % (2 * kStages)];
                    const int64_t e0 = lt * pa.tile_elems + (int64_t)row0 * pa.D;
                    m.sm_dst = jb.sign_mant + e0;
                    m.code_dst = jb.codes + e0 * N / 8;
                    m.esc_dst = pa.esc_scratch + tile * pa.tile_elems + (int64_t)row0 * pa.D;
                    m.unit_count = pa.unit_counts + tile * upt + u;
                    m.tile_count = pa.tile_counts + tile;
                    constexpr int kPer1024 = N == 2 ? 2 : N == 4 ? 4 : 1;
                    if (FLAT) m.block_counts = pa.block_counts + (e0 >> 10) * kPer1024;
                    m.elems = elems;
                    m.first_unit_of_tile = (u == 0);
                    m.last_unit_of_tile = (u == upt - 1);
                    m.job = j;
                    // (a box is a whole unit; what lies behind the last rows of a tile is loaded and not used)
                    mbar_arrive_expect_tx(&s.full[stg], (uint32_t)(use_map ? unit_rows * pa.D : elems) * 2u);
                }
                __syncwarp();
                const uint16_t *usrc = tsrc + (int64_t)row0 * jb.ss;
                if (rows_contig) {
                    if (lane == 0) bulk_load(st.in, usrc, (uint32_t)elems * 2u, &s.full[stg]);
                } else if (use_map) {
                    if (lane == 0) tensor_load(st.in, &ka.map[j], (int)(blk * pa.seq_tile) + row0, h, b, &s.full[stg]);
                } else {
                    for (int r = lane; r < rows; r += 32)
                        bulk_load(st.in + r * pa.D, usrc + (int64_t)r * jb.ss, (uint32_t)pa.D * 2u, &s.full[stg]);
                }
            }
        }
        // do not leave while a copy into this CTA's shared memory may still be in flight (see k_unpack_pipe)
        if (launch_timed_out(pa.status))
            for (uint32_t k = it > kStages ? it - kStages : 0; k < it; ++k)
                mbar_wait(&s.full[k % kStages], (k / kStages) & 1, pa.status, pa.poll_limit);
        return;
    }

    // ---------------- consumer warps ----------------
    const int lane = tid & 31;
    uint32_t cnt2[HistRegs<N>::v];
#pragma unroll
    for (int v = 0; v < HistRegs<N>::v; ++v) cnt2[v] = 0;
    int running = 0;
    bool broken = false;                  // a wait of this warp ran out: compute on, store nothing
    int cur_job = -1, cur_left = 0;
    // (the consumers only count units: which tile a unit belongs to is in its description)
    const uint32_t my_units =
        pa.n_tiles > (int64_t)blockIdx.x
            ? (uint32_t)((pa.n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) * (uint32_t)upt
            : 0u;
    // Units of one job run in an inner loop of their own; this outer loop only takes over when the
    // job (and with it the window and the histogram) changes.
    auto wait_loaded = [&](uint32_t u) {
        bool loaded = true;
        if (lane == 0) loaded = mbar_wait(&s.full[u % kStages], (u / kStages) & 1, pa.status, pa.poll_limit);
        loaded = __shfl_sync(kFull, loaded, 0);
        __syncwarp();      // orders the other lanes' reads of the stage after lane 0's wait
        return loaded;
    };
    uint32_t it = 0;
    while (it < my_units) {
        broken |= !wait_loaded(it);               // returns at once if the inner loop waited already
        const int job = s.meta_ring[it % (2 * kStages)].job;
        if (job != cur_job) {
            // Uniform over the CTA (every consumer reads the same sequence of units): hand the finished
            // job's histogram over.
            if (HIST && cur_job >= 0) flush_code_counts<N>(cnt2, cur_left, s.hist);
            consumer_sync<G::kConsumers>();
            if (HIST && cur_job >= 0 && tid < 256) {
                const int hv = s.hist[tid];
                if (hv != 0 && pa.job[cur_job].hist) atomicAdd(pa.job[cur_job].hist + tid, hv);
                s.hist[tid] = 0;
            }
            cur_job = job;
            cur_left = pa.job[job].left;
            consumer_sync<G::kConsumers>();
        }
        const uint32_t neg_left = ((uint32_t)(-cur_left) & 0xFFFFu) * 0x10001u;
        for (;;) {
            const int stg = it % kStages;
            const PackUnitMeta &meta = s.meta_ring[it % (2 * kStages)];
            if (meta.elems == G::kUnit) pack_unit<N, HIST, FLAT, G, true>(s, s.stage[stg], meta, &s.empty[stg], running, cnt2, neg_left, broken);
            else pack_unit<N, HIST, FLAT, G, false>(s, s.stage[stg], meta, &s.empty[stg], running, cnt2, neg_left, broken);
            // the per-thread counters are 16-bit fields and grow by at most 32 per unit
            if (HIST && (it & 1023u) == 1023u) flush_code_counts<N>(cnt2, cur_left, s.hist);
            if (++it >= my_units) break;
            broken |= !wait_loaded(it);
            if (s.meta_ring[it % (2 * kStages)].job != cur_job) break;
        }
    }
    if (HIST && cur_job >= 0) {
        flush_code_counts<N>(cnt2, cur_left, s.hist);
        consumer_sync<G::kConsumers>();
        if (tid < 256) {
            const int hv = s.hist[tid];
            if (hv != 0 && pa.job[cur_job].hist) atomicAdd(pa.job[cur_job].hist + tid, hv);
        }
    }
    bulk_wait_all();
    // the compaction pass may be set up from here on (it waits for this launch to complete before it reads)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!pa.scan_in_pack) return;
    __threadfence();
    consumer_sync<G::kConsumers>();
    if (tid == 0) {
        const unsigned ticket = atomicAdd(pa.done, 1u);
        s.is_last = (ticket == gridDim.x - 1);
    }
    consumer_sync<G::kConsumers>();
    if (!s.is_last) return;
    __threadfence();
    // (the staging buffers are idle by now: every unit of this CTA has been consumed and stored)
    scan_tile_counts<G>(pa, &s.carry, s.scan, s.job_off, reinterpret_cast<long long *>(&s.stage[0]));
}

// One warp copies the escape bytes of tile t (its units follow each other in the scratch, `count` bytes in all) to `dst`
// of its job's stream, a kilobyte at a time whose loads are all under way together.  The bytes move as aligned 32-bit words,
// one per lane: a destination word is put together from a lane's source word and its neighbour's; only the first and
// last word of a run use byte stores.  With do_hist the escaped exponents are counted into `my_hist` (256 bins in shared
// memory).
// Pack and compaction together, in steps of 16 bytes per lane with a load of the word before each, four copies of the bins
// per warp, four CTAs per SM (64 registers) and now: keys and values [64, 8, 4096, 128] at 3 bits with histograms 440 -> 416 us,
// [16, 8, 8192, 128] at 2 bits, 34 % escapes, 249 -> 224 us; the compaction is bound by the latency of its reads.
constexpr int kCompactWords = 8;               // words per lane under way

__device__ __forceinline__ void compact_tile_units(const PackPipeArgs &pa, const PackJob &jb, int64_t t, int64_t dst,
                                                   int count, int *my_hist, bool do_hist) {
    const int lane = threadIdx.x & 31;
    const int upt = pa.units_per_tile;
    const int unit_elems = pa.unit_rows * pa.D;
    const bool fits = dst >= 0 && dst + count <= jb.capacity;
    if (!fits && lane == 0) atomicOr(pa.status, ADACODE_STATUS_ESCAPE_OVERFLOW);
    for (int u = 0; u < upt; ++u) {
        const int cu = upt == 1 ? count : __ldcg(pa.unit_counts + t * upt + u);
        // unit slots start on 16-byte boundaries
        const uint32_t *src = reinterpret_cast<const uint32_t *>(pa.esc_scratch + t * pa.tile_elems + (int64_t)u * unit_elems);
        uint8_t *d8 = jb.escapes + dst;
        const int r = (int)((uintptr_t)d8 & 3);
        uint32_t *dst32 = reinterpret_cast<uint32_t *>(d8 - r);
        const int n_words = (r + cu + 3) >> 2;             // destination words touched
        uint32_t carry = 0;                                // lane 0: the source word before its next one
#pragma unroll 1
        for (int base = 0; base < n_words; base += 32 * kCompactWords) {
            uint32_t w[kCompactWords];
#pragma unroll
            for (int k = 0; k < kCompactWords; ++k) {
                const int j = base + 32 * k + lane;
                w[k] = 4 * j < cu ? __ldcg(src + j) : 0u;
            }
#pragma unroll
            for (int k = 0; k < kCompactWords; ++k) {
                if (base + 32 * k >= n_words) break;       // (uniform)
                const int j = base + 32 * k + lane;
                const uint32_t turned = __shfl_sync(kFull, w[k], (lane + 31) & 31);
                const uint32_t prev = lane == 0 ? carry : turned;
                carry = turned;
                // bytes 4 j - r .. 4 j - r + 3 of the unit
                const uint32_t v = __funnelshift_lc(prev, w[k], 8 * r);
                const int s0 = 4 * j - r;
                if (fits && s0 >= 0 && s0 + 4 <= cu) {
                    dst32[j] = v;
                } else if (fits && j < n_words) {
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (s0 + b >= 0 && s0 + b < cu) reinterpret_cast<uint8_t *>(dst32 + j)[b] = (uint8_t)(v >> (8 * b));
                }
                if (do_hist) {
                    // source word j holds source bytes 4 j .. 4 j + 3: each source byte is counted once
                    const int left = cu - 4 * j;
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (b < left) atomicAdd(my_hist + ((w[k] >> (8 * b)) & 0xFFu), 1);
                }
            }
        }
        dst += cu;
    }
}

// Flat layout: the inclusive escape counts of tile t's blocks, whose first escape is number `start` of the tensor; one warp.
__device__ __forceinline__ void write_block_bases(const PackPipeArgs &pa, int64_t t, int64_t start) {
    const int lane = threadIdx.x & 31, per = pa.block_per_1024;
    const int64_t first = t * (pa.tile_elems >> 10);
    for (int g0 = 0, groups = pa.tile_elems >> 10; g0 < groups; g0 += 32) {
        const int32_t *counts = pa.block_counts + (first + g0 + lane) * per;
        int32_t *base = pa.block_base + (first + g0 + lane) * per;
        const bool mine = g0 + lane < groups;
        const int all = mine ? __ldcg(counts + per - 1) : 0;
        int incl = all;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += u;
        }
        if (mine)
            for (int i = 0; i < per; ++i) base[i] = (int32_t)start + incl - all + __ldcg(counts + i);
        start += __shfl_sync(kFull, incl, 31);
    }
}

// Offsets of the escapes of tiles [lt0, lt0 + n) of a job (n <= kThreads), by the whole CTA: their inclusive
// counts inside the segment and the segments' offsets go to the caller's arrays, s_off[i] is tile lt0 + i's
// first byte in the job's stream and s_cnt[i] its count.  Every CTA adds up all the counts before its own
// tiles: with at most kSumTiles of them that is a microsecond of reads from L2, while one CTA that
// scans them alone keeps the others waiting.  Keys and values in one launch, 3 bits: [16, 8, 8192, 128] (16 384 tiles)
// 209.8 -> 193.3 us, [1, 8, 20480, 128] (2560 tiles) 43.4 -> 39.1 us, one block of [1, 8, 128, 128] 14.2 -> 10.4 us.
constexpr int64_t kSumTiles = 65536;

__device__ __forceinline__ void tile_offsets(const PackPipeArgs &pa, const PackJob &jb, int lt0, int n, int *s_off, int *s_cnt,
                                             int *s_red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int seg0 = lt0 / pa.BH, seg0_tile = seg0 * pa.BH;
    const int first = (int)jb.tile0, mid = first + seg0_tile, last = first + lt0;
    // counts before segment seg0 and from there to lt0, four at a time (the array starts on a 256-byte boundary)
    int before_seg = 0, in_seg = 0;
#pragma unroll 4
    for (int v = (first >> 2) + tid; v < (last + 3) >> 2; v += kThreads) {
        const int4 q = __ldcg(reinterpret_cast<const int4 *>(pa.tile_counts) + v);
        const int c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = 4 * v + i;
            before_seg += t >= first && t < mid ? c[i] : 0;
            in_seg += t >= mid && t < last ? c[i] : 0;
        }
    }
    const int c = tid < n ? __ldcg(pa.tile_counts + last + tid) : 0;
    int incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += u;
    }
    before_seg = (int)__reduce_add_sync(kFull, (unsigned)before_seg);
    in_seg = (int)__reduce_add_sync(kFull, (unsigned)in_seg);
    if (lane == 31) s_red[warp] = before_seg, s_red[kWarps + warp] = in_seg, s_red[2 * kWarps + warp] = incl;
    __syncthreads();
    int seg_start = 0, start = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        seg_start += s_red[w];
        start += s_red[w] + s_red[kWarps + w];
        if (w < warp) incl += s_red[2 * kWarps + w];
    }
    const int off = start + incl - c;                     // escapes of the job before tile lt0 + tid
    s_off[tid] = off;
    s_cnt[tid] = c;
    __syncthreads();
    if (tid < n) {
        const int lt = lt0 + tid, seg = lt / pa.BH;
        const int at = seg == seg0 ? seg_start : s_off[seg * pa.BH - lt0];
        jb.tile_base[lt] = off + c - at;
        if (lt - seg * pa.BH == pa.BH - 1) jb.seg_off[seg + 1] = (int64_t)(off + c);
        if (lt == 0) jb.seg_off[0] = 0;
    }
}

// Gather every unit's escape bytes from its scratch slot into the compact per-segment stream.
// With scan_in_pack tile t of global block i starts at blk_off[i] - blk_off[first block of the job] + tile_base[t] -
// count[t] in its job's stream.  blockIdx.y is the job; one warp per tile; all of a tile's metadata
// is fetched with independent loads (one memory round trip).
// With HIST the escaped exponents are counted here (whole warps of escape bytes) rather than one
// by one inside the pack kernel, into one set of 256 bins per CTA.
template <bool HIST, bool FLAT>
__global__ void __launch_bounds__(kThreads) k_compact_units(const __grid_constant__ PackPipeArgs pa) {
    __shared__ int s_hist[HIST ? 256 : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const PackJob &jb = pa.job[blockIdx.y];
    int32_t *hist = jb.hist;
    const bool do_hist = HIST && hist != nullptr;
    if (HIST) {
        for (int i = tid; i < 256; i += kThreads) s_hist[i] = 0;
        __syncthreads();
    }
    // launched as a programmatic dependent of the pack kernel: nothing that kernel wrote is read above
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int *my_hist = s_hist;
    const int64_t job_tiles = (int64_t)jb.n_blocks * pa.BH;
    if (!pa.scan_in_pack) {
        __shared__ int s_off[kThreads], s_cnt[kThreads], s_red[3 * kWarps];
        const int per = (int)((job_tiles + gridDim.x - 1) / gridDim.x);
        const int64_t lt0 = (int64_t)blockIdx.x * per;
        const int n = (int)(job_tiles - lt0 < per ? job_tiles - lt0 : per);
        if (n > 0) {                                       // (uniform over the CTA)
            tile_offsets(pa, jb, (int)lt0, n, s_off, s_cnt, s_red);
            for (int i = warp; i < n; i += kWarps) {
                if (FLAT) write_block_bases(pa, lt0 + i, s_off[i]);
                if (s_cnt[i] != 0) compact_tile_units(pa, jb, jb.tile0 + lt0 + i, s_off[i], s_cnt[i], my_hist, do_hist);
            }
        }
    } else {
        const int64_t warp_global = (int64_t)blockIdx.x * kWarps + warp;
        const int64_t n_warps = (int64_t)gridDim.x * kWarps;
        const int64_t job_off = __ldg(pa.blk_off + jb.blk0);
        for (int64_t lt = warp_global; lt < job_tiles; lt += n_warps) {
            const int64_t t = jb.tile0 + lt;
            // independent loads: one round trip
            const int c = __ldg(pa.tile_counts + t);
            const int tb = __ldg(jb.tile_base + lt);
            const int64_t so = __ldg(pa.blk_off + t / pa.BH) - job_off;
            if (FLAT) write_block_bases(pa, t, so + tb - c);
            if (c == 0) continue;
            compact_tile_units(pa, jb, t, so + tb - c, c, my_hist, do_hist);
        }
    }
    if (do_hist) {
        __syncthreads();
        const int total = s_hist[tid];
        if (total != 0) atomicAdd(hist + tid, total);
    }
    if (pa.report.words != 0) {
        // The CTA that comes last has everyone's offsets, counts and status bits before it.  (A launch that only copies them
        // took 4.2 us behind the compaction, and its host side as long; this takes less than one, 7 us with fences
        // at the system's scope around a single flag.)
        __shared__ bool last;
        __syncthreads();
        if (tid == 0) {
            // (the last one's increment brings the counter back to zero: the scratch is free before the host hears of it.  By it the
            // outputs of all CTAs are written for the whole GPU, which send_report asks for)
            const unsigned ctas = gridDim.x * gridDim.y;
            unsigned before;
            asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(before) : "l"(pa.done + 1), "r"(ctas - 1) : "memory");
            last = before == ctas - 1;
        }
        __syncthreads();
        if (last) send_report(pa.report);
    }
}

#endif  // ADACODE_PIPELINE_UNPACK_ONLY
