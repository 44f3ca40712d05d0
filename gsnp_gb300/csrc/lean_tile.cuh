/*
 * lean_tile.cuh - the pileup and the sort of a tile in the short form
 * (lean.cuh), which the FP32 and the FP64 kernels share.
 */
#ifndef GSNP_LEAN_TILE_CUH
#define GSNP_LEAN_TILE_CUH

#include "lean.cuh"
#include "tile.cuh"

namespace gsnp {

/* Per-warp shared memory of the short form: the tile's unique reads as the
 * pileup broadcasts them, and a 16-bit entry per (strand, start or end) that
 * a covering read can have in a tile: its reads in the low byte, the number of
 * their group in the high one. */
struct LeanRead {
    int32_t c0;        /* column of the read at the tile's first site */
    int32_t off;       /* its element there, from the first read's row */
    uint32_t low;      /* bits 23:0 of its lean record there: cycle, strand, 4 * group */
    int32_t len;       /* bits 7:0; while the groups are formed, its table entry above */
};
/* record slots of the short form in a bin of that many: whole chunks of 16 */
__host__ __device__ constexpr int lean_slots(int slots) { return (slots + 15) & ~15; }
/* unique reads that a tile of the short form holds, with room to pad both lists */
__host__ __device__ constexpr int lean_reads(int slots) { return 2 * lean_slots(slots); }
__host__ __device__ constexpr int lean_table_words(int L) { return L + kTile; }
__host__ __device__ constexpr size_t lean_smem_bytes(int slots, int L) {
    /* the table is done with before the first record is written, and lies in
     * the records' place */
    return ((size_t)lean_slots(slots) * kTile > (size_t)lean_table_words(L) ? (size_t)lean_slots(slots) * kTile
                                                                           : (size_t)lean_table_words(L)) * 4 +
           (size_t)lean_reads(slots) * sizeof(LeanRead);
}
constexpr int kLeanGroups = 15;   /* most groups, and most reads of one (a 4-bit count each) */

/* Whether the short form took a tile: else a site deeper than its slots, or
 * something that no number of slots mends. */
enum LeanTook : int { kLeanTook = 0, kLeanDeep = 1, kLeanNever = 2 };

/* The pileup of a warp's tile (as warp_pileup) in the short form: not taken, for
 * the whole warp, when the tile needs the general one - a site deeper than
 * SLOTS records, more reads than the lists hold (both kLeanDeep), a quality above
 * 64, or more repeated keys than the walk's counts hold (kLeanNever).
 *
 * What bounds it is the number of instructions per read, since every lane
 * looks at every read of the tile.  What depends on the read only is worked
 * out once, by one lane, and broadcast with one 128-bit shared load; a lane
 * then needs its column, the element's address, and two additions for the
 * record word: the element is the word's top byte, and the cycle runs up
 * (forward reads) or down (reverse ones) with the site.  The records are
 * sorted afterwards and no site reaches the 255-record cap, so the reads may be
 * taken in any order: forward ones from a list at the front, reverse ones from
 * one at the back, and the few reads of several hits, which leave no record,
 * as they are met.  A base of quality 0 makes its record like any other (its
 * element has the spilled base's bits); the sites that have one go over the reads
 * once more to count them by their own base.  Left to the general form, tiles
 * with such a base cost more than before there was a short one: 8 Mbp at 30x,
 * one base in 100 of quality 0, recalled: FP32 6.04 ms (3.68 without the short
 * form) -> 2.55, FP64 8.58 (7.01) -> 3.57. */
template <int SLOTS>
__device__ __forceinline__ LeanTook lean_pileup(const CallArgs& a, int64_t s0, int64_t r_lo, int64_t r_hi,
                                            uint32_t* recs_all, LeanRead* reads, LeanPile* out) {
    constexpr int kReads = lean_reads(SLOTS);
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int L = a.L;
    uint32_t* const recs = recs_all + lane;
    uint32_t* const table = recs_all;
    if (r_hi - r_lo > kReads - 8) return kLeanDeep;
    const int n = (int)(r_hi - r_lo);
    for (int i = lane; i < lean_table_words(L); i += 32) table[i] = 0u;
    __syncwarp();
    const uint16_t* row = a.bq + r_lo * L + lane;
    uint32_t depth = 0, extra_hits = 0;
    uint64_t extra4 = 0;
    int groups = 0, fwd = 0, rev = 0;
    bool bad = false;
#pragma unroll 1
    for (int c = 0; c < n; c += 32) {
        bool uni = false, minus = false, second = false;
        int c0 = 0, len = 0, at = 0;
        uint32_t hit = 0;
        if (c + lane < n) {
            const int64_t r = r_lo + c + lane;
            c0 = (int)(s0 - __ldg(a.pos + r));
            const uint32_t lh = (uint32_t)__ldg(a.lenhit + r);
            len = (int)(lh >> 16);
            if (c0 < len) {   /* it covers a site of the tile */
                hit = lh & 0xffffu;
                uni = hit == 1u;
                minus = __ldg(a.strand + r) != '+';
            }
        }
        const unsigned covers = __ballot_sync(kFull, c0 < len);
        unsigned multi = covers & ~__ballot_sync(kFull, uni);
        const unsigned mr = __ballot_sync(kFull, uni && minus), mf = __ballot_sync(kFull, uni && !minus);
        if (uni) {
            /* entry of the read in the table: starts s0 - L + 1 .. s0 + 31 of the
             * forward reads, then ends s0 + 1 .. s0 + 31 + L of the reverse ones */
            at = minus ? L + kTile + (len - c0) - 1 : L - 1 - c0;
            const int sh = (at & 1) * 16;
            const uint32_t before = (atomicAdd(table + (at >> 1), 1u << sh) >> sh) & 0xffu;
            second = before == 1u;
            bad |= before >= (uint32_t)kLeanGroups;
            LeanRead m;
            m.c0 = c0;
            m.off = (c + lane) * L + c0;
            m.low = ((uint32_t)(minus ? len - 1 - c0 : c0) << 16) + (minus ? 0x8000u : 0u);
            m.len = len | at << 8;
            reads[minus ? kReads - 1 - rev - __popc(mr & lt) : fwd + __popc(mf & lt)] = m;
        }
        const unsigned b = __ballot_sync(kFull, second);
        if (second) reinterpret_cast<uint8_t*>(table)[at * 2 + 1] = (uint8_t)(groups + __popc(b & lt) + 1);
        groups += __popc(b);
        fwd += __popc(mf);
        rev += __popc(mr);
        for (; multi; multi &= multi - 1) {
            const int src = __ffs(multi) - 1;
            const int x = __shfl_sync(kFull, c0, src) + lane;
            const uint32_t h = __shfl_sync(kFull, hit, src);
            if ((uint32_t)x < (uint32_t)__shfl_sync(kFull, len, src)) {
                const uint32_t e = __ldg(a.bq + (r_lo + c + src) * L + x);
                depth += 1;
                extra_hits += h - 1u;
                if (elem_valid(e)) extra4 += 1ull << (elem_base(e) * 16);
            }
        }
        __syncwarp();
    }
    if (__any_sync(kFull, bad) || groups > kLeanGroups) return kLeanNever;
    /* each read's group; both lists are padded to whole steps of four */
    if (lane < 4) {
        reads[fwd + lane].len = 0;
        reads[kReads - 1 - rev - lane].len = 0;
    }
    for (int i = lane; i < fwd + rev; i += 32) {
        LeanRead* m = reads + (i < fwd ? i : kReads - 1 - (i - fwd));
        const int x = m->len;
        m->low |= (uint32_t)reinterpret_cast<const uint8_t*>(table)[(x >> 8) * 2 + 1] << 2;
        m->len = x & 0xff;
    }
    __syncwarp();
    uint32_t seen_bits = 0;
    int num = 0;
#pragma unroll 1
    for (int strand = 0; strand < 2; ++strand) {
        const int cnt = strand ? rev : fwd;
        const uint32_t step = strand ? 0u - ((uint32_t)lane << 16) : (uint32_t)lane << 16;
        const int4* list = reinterpret_cast<const int4*>(strand ? reads + (kReads - ((rev + 3) & ~3)) : reads);
#pragma unroll 1
        for (int k0 = 0; k0 < cnt; k0 += 4) {
            uint32_t e[4], low[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int4 rd = list[k0 + u];
                const bool cov = (uint32_t)(rd.x + lane) < (uint32_t)rd.w;
                low[u] = (uint32_t)rd.z + step;
                e[u] = kElemInvalid;
                if (cov) {
                    e[u] = __ldg(row + rd.y);
                    depth += 1;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                seen_bits |= e[u];
                if (e[u] < kElemWide) {
                    if (num < SLOTS) recs[num * kTile] = (e[u] << 24) + low[u];
                    num += 1;
                }
            }
        }
    }
    if (__any_sync(kFull, num > SLOTS || (seen_bits & kElemWide)))
        return __any_sync(kFull, (seen_bits & kElemWide) != 0) ? kLeanNever : kLeanDeep;
    if (seen_bits & kElemZero) {
        /* all slots of the two lists, the unused ones skipped: a loop over the
         * used ones ran a tenth shorter here but cost every other tile of the
         * FP64 kernel, which has no register to spare, another half percent */
#pragma unroll 1
        for (int i = 0; i < kReads; ++i) {
            const int4 rd = reinterpret_cast<const int4*>(reads)[i];
            uint32_t x = kElemInvalid;
            if ((i < fwd || i >= kReads - rev) && (uint32_t)(rd.x + lane) < (uint32_t)rd.w) x = __ldg(row + rd.y);
            if ((x & (kElemInvalid | kElemZero)) == kElemZero) extra4 += 1ull << (elem_base(x) * 16 + kLeanExtraBits);
        }
    }
    out->depth = depth;
    out->repeat = depth + extra_hits;
    out->extra4 = extra4;
    out->num = num;
    return kLeanTook;
}

/* The sorted columns of a tile: lean_pileup, padded and sorted, when that takes
 * it. */
template <int SLOTS>
__device__ __forceinline__ LeanTook lean_columns(const CallArgs& a, int64_t s0, int64_t r_lo, int64_t r_hi,
                                             uint32_t* recs_all, uint32_t* scratch, LeanPile* pile) {
    static_assert(SLOTS <= kLeanG && SLOTS % 16 == 0, "a walk counts at most kLeanG distinct keys; chunks of 16");
    const LeanTook took = lean_pileup<SLOTS>(a, s0, r_lo, r_hi, recs_all, reinterpret_cast<LeanRead*>(scratch), pile);
    if (took != kLeanTook) return took;
    uint32_t* recs = recs_all + (threadIdx.x & 31);
    const int most = __reduce_max_sync(kFull, pile->num);
    for (int i = pile->num; i < ((most + 15) & ~15); ++i) recs[i * kTile] = kLeanPad;
    lean_sort<kTile>(recs, pile->num, most);
    return kLeanTook;
}

}  // namespace gsnp

#endif
