/*
 * calling_fast.cu - the FP32 calling kernels: the tile kernels in the short
 * form (lean.cuh) and the general one, the persistent kernel over a segment's
 * tiles, and the warp-per-site kernel of the deepest bin.
 */
#include <cuda_runtime.h>

#include "calling.cuh"
#include "lean.cuh"
#include "lean_tile.cuh"
#include "deep.cuh"
#include "site_math.cuh"
#include "tile.cuh"
#include "tma.cuh"

namespace gsnp {

namespace {

/* resident CTAs per SM the kernels are compiled for; this caps their
 * registers at 64 (32 warps per SM; a few spilled words cost less than the
 * latency the extra warps hide) */
constexpr int kFastCtasPerSm = 32 * 32 / kTile;

/* The reads of a tile staged in shared memory by the persistent kernel: per
 * read its start, (len << 16) | hit with the strand in bit 31, and the byte
 * offset in `rows` that column 0 of its row would have; the bulk copy of the
 * read holds the columns that cover the tile. */
struct StagedReads {
    const int32_t* pos;
    const uint32_t* lhs;
    const int32_t* rbase;
    const uint8_t* rows;
    int n;
};

/* warp_pileup over staged reads: the same records and counts, read from
 * shared memory (broadcast loads of the per-read values, one 16-bit load
 * per covering read and lane). */
template <int SLOTS>
__device__ __forceinline__ PackedPileup warp_pileup_staged(const CallArgs& a, const StagedReads& sr, int64_t site,
                                                          bool active, uint32_t* recs, bool* report_overflow) {
    PileupAcc acc;
    for (int k = 0; k < sr.n; ++k) {
        const int32_t start = sr.pos[k];
        const uint32_t lhs = sr.lhs[k];
        const int coord = (int)(site - start);
        const uint32_t lh = lhs & 0x7fffffffu;
        if (active && coord >= 0 && coord < (int)(lh >> 16)) {
            const uint32_t bq = *reinterpret_cast<const uint16_t*>(sr.rows + sr.rbase[k] + 2 * coord);
            acc.take<SLOTS>(bq, lh, coord, (int)(lhs >> 31), recs);
        }
    }
    return acc.finish(a, report_overflow);
}

}  // namespace

/* ------------------------------------------------------------------------ */
/* the fast calling kernel                                                   */
/* ------------------------------------------------------------------------ */

/* The end of a site's FP32 call: prove(&call) decides it from its sums, or the
 * site is appended to the deferred pool with its counts p and sorted records
 * (record() gives a column word as a record word of occurrence 1).  Every lane of the warp calls it (the
 * appends are warp-aggregated). */
template <class Prove, class Record>
__device__ __forceinline__ void finish_fast_site(const CallArgs& a, int64_t site, bool active, uint8_t ori,
                                                 uint8_t wflags, int32_t snp_row, const SitePileup& p,
                                                 const uint32_t* recs, Prove&& prove, Record&& record) {
    const int lane = threadIdx.x & 31;
    uint8_t dflags = 0;
    if (active) {
        if (wflags & kWinKeepCounts) store_counts(a, site, p);
        CallWords call;
        if ((site & 4095) == 0 && a.stats) dflags = kCallSampled;
        const bool empty = p.num == 0 && (p.ca[0] | p.ca[1] | p.ca[2] | p.ca[3]) == 0 && a.empty_valid[ori];
        if (empty) {
            /* no record and no count: the call depends on the site code only */
            const uint4* src = reinterpret_cast<const uint4*>(a.empty_calls + ori);
            call.a = __ldg(src);
            call.b = __ldg(src + 1);
            call.b.x = p.depth;
            call.b.y = p.repeat;
        } else if (!prove(&call)) {
            call.a = call.b = make_uint4(0u, 0u, 0u, 0u);
            dflags |= kCallPending;
        }
        call.a.y |= (uint32_t)dflags << 16;
        uint4* dst = reinterpret_cast<uint4*>(a.out + site);
        dst[0] = call.a;
        dst[1] = call.b;
    }
    /* append the deferred sites of the warp */
    const unsigned m = __ballot_sync(kFull, dflags != 0);
    if (m == 0) return;
    unsigned long long base = 0;
    const int leader = __ffs(m) - 1;
    if (lane == leader) base = atomicAdd(a.dcount, (unsigned long long)__popc(m));
    base = __shfl_sync(kFull, base, leader);
    if (!dflags) return;
    const unsigned long long slot = base + __popc(m & ((1u << lane) - 1u));
    const unsigned long long off = atomicAdd(a.dcount + 1, (unsigned long long)p.num);
    if ((int64_t)slot >= a.dsite_cap || (int64_t)(off + p.num) > a.dpool_cap) return;
    DeferredSite d;
    d.site = site;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        d.cu[i] = (uint16_t)p.cu[i];
        d.qs[i] = (uint16_t)p.qs[i];
        d.ca[i] = p.ca[i];
    }
    d.depth = p.depth;
    d.repeat = p.repeat;
    d.rec_off = (uint32_t)off;
    d.num = (uint16_t)p.num;
    d.dep_uni = (uint16_t)p.dep_uni;
    d.snp_row = snp_row;
    d.flags = dflags;
#pragma unroll
    for (int i = 0; i < 3; ++i) d.pad[i] = 0;
    a.dsites[slot] = d;
    uint32_t* dst = a.dpool + off;
    for (int i = 0; i < p.num; ++i) dst[i] = record(recs[i * kTile]);
}

/* The FP32 work on one site of a tile after its pileup and sort, in the
 * general form: the dependency walk, the compensated sums and the FP32
 * posterior.  Every lane of the warp calls it. */
template <int SLOTS>
__device__ __forceinline__ void fast_site(const CallArgs& a, int64_t site, bool active, uint8_t ori, uint8_t wflags,
                                          int32_t snp_row, const SitePileup& p, uint32_t* recs, uint32_t* seen) {
    Kahan10 k;
    k.init();
    if (active) {
        /* adjusted quality of each record, written over its occurrence byte */
        walk_records<true, kPcrBits(SLOTS, true)>(a, recs, seen, kTile, p.num, [&](int i, int qa, int, int) {
            recs[i * kTile] = (recs[i * kTile] & ~0xffu) | (uint32_t)qa;
        });
        /* FP32 sums, four records per compensated step (the grouping of
         * likelihood_fp32) */
        for (int i = 0; i < p.num; i += 4) {
            float x[10], y[10];
            uint32_t w = recs[i * kTile];
            lik32_row(a, (int)(w & 0xffu), rec_coord(w), rec_base(w), x);
            if (i + 1 < p.num) {
                w = recs[(i + 1) * kTile];
                lik32_row(a, (int)(w & 0xffu), rec_coord(w), rec_base(w), y);
#pragma unroll
                for (int v = 0; v < 10; ++v) x[v] = __fadd_rn(x[v], y[v]);
            }
            if (i + 2 < p.num) {
                float z[10];
                w = recs[(i + 2) * kTile];
                lik32_row(a, (int)(w & 0xffu), rec_coord(w), rec_base(w), y);
                if (i + 3 < p.num) {
                    w = recs[(i + 3) * kTile];
                    lik32_row(a, (int)(w & 0xffu), rec_coord(w), rec_base(w), z);
#pragma unroll
                    for (int v = 0; v < 10; ++v) y[v] = __fadd_rn(y[v], z[v]);
                }
#pragma unroll
                for (int v = 0; v < 10; ++v) x[v] = __fadd_rn(x[v], y[v]);
            }
            k.add(x);
        }
    }
    finish_fast_site(a, site, active, ori, wflags, snp_row, p, recs,
                     [&](CallWords* call) {
                         SiteCall c;
                         if (!fast_posterior(a, snp_row, ori, p, k.s, p.num, &c)) return false;
                         *call = call_words(c);
                         return true;
                     },
                     [](uint32_t w) { return (w & ~0xffu) | 1u; });
}

/* A tile in the short form; every lane of the warp calls it.  Nothing is written
 * when lean_pileup leaves it. */
template <int SLOTS>
__device__ __forceinline__ LeanTook lean_tile(const CallArgs& a, int64_t tile, int64_t r_lo, int64_t r_hi, uint8_t wflags,
                                          uint32_t* recs_all, uint32_t* scratch) {
    const int t = threadIdx.x & 31;
    const int64_t s0 = tile * kTile, site = s0 + t;
    const bool active = site < a.chr_len;
    uint32_t* recs = recs_all + t;
    LeanPile pile;
    /* a read's columns end before the chromosome does, so sites past the end
     * have no covering read */
    const LeanTook took = lean_columns<SLOTS>(a, s0, r_lo, r_hi, recs_all, scratch, &pile);
    if (took != kLeanTook) return took;
    const uint8_t ori = active ? __ldg(a.ori + site) : 0;
    const int32_t snp_row = tile_snp_row(a, tile, (ori & 8) != 0);
    LeanSums z;
    lean_walk<kTile>(a, recs, pile.num, ori & 3, &z);
    lean_zeros(pile, &z);
    const SitePileup p = lean_counts(pile, z);
    finish_fast_site(a, site, active, ori, wflags, snp_row, p, recs,
                     [&](CallWords* call) { return lean_posterior(a, snp_row, ori, pile, z, call); },
                     [](uint32_t w) { return lean_to_record(w); });
    return kLeanTook;
}

/* Sites whose call is not proven in FP32 (and every 4096th site, sampled for
 * the FP32 accuracy figure) are appended to the deferred pool: counts and the
 * sorted records with their occurrence byte restored.  The append counters
 * keep counting past the capacities so that the host can size the pool and
 * run the pass again. */
template <int SLOTS>
__device__ __forceinline__ void fast_tile(const CallArgs& a, int32_t entry, uint32_t* recs_all, uint32_t* seen_all) {
    const int t = threadIdx.x;
    const int64_t tile = entry & ~kTileGeneral, s0 = tile * kTile;
    const int win = (int)(s0 / kWin);
    const uint8_t wflags = a.win_flags[win];
    const int64_t r_lo = a.warp_rng[tile * 2];
    const int64_t r_hi = a.warp_rng[tile * 2 + 1];
    if constexpr (SLOTS <= kLeanG) {
        if (a.lean_q && !(entry & kTileGeneral) &&
            lean_tile<lean_slots(SLOTS)>(a, tile, r_lo, r_hi, wflags, recs_all, recs_all + lean_slots(SLOTS) * kTile) ==
                kLeanTook)
            return;
        __syncwarp();
    }
    const int64_t site = s0 + t;
    const bool active = site < a.chr_len;
    const uint8_t ori = active ? __ldg(a.ori + site) : 0;
    const int32_t snp_row = tile_snp_row(a, tile, (ori & 8) != 0);
    const SitePileup p = warp_pileup<SLOTS>(a, r_lo, r_hi, site, active, recs_all + t).unpack();
    uint32_t* recs = recs_all + t;
    uint32_t* seen = seen_all + t;
    if (active) sort_column<SLOTS>(recs, p.num);

    fast_site<SLOTS>(a, site, active, ori, wflags, snp_row, p, recs, seen);
}

/* The tiles of one depth bin, as call_tiles_kernel takes them. */
template <int SLOTS>
__global__ void __launch_bounds__(kTile, kFastCtasPerSm) call_fast_kernel(const __grid_constant__ CallArgs a, const int32_t* __restrict__ tiles,
                                                                          const int* __restrict__ count, int* next) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t* recs_all = reinterpret_cast<uint32_t*>(smem);
    uint32_t* seen_all = recs_all + SLOTS * kTile;
    if (!count) {
        fast_tile<SLOTS>(a, tiles[blockIdx.x], recs_all, seen_all);
        return;
    }
    for_each_listed(count, next, [&](int i) { fast_tile<SLOTS>(a, tiles[i], recs_all, seen_all); });
}

/* ------------------------------------------------------------------------ */
/* the deep bin of the FP32 form: a warp's lanes on one site's records         */
/* ------------------------------------------------------------------------ */

/* Tiles with a site of more than 128 records (hotspots of hundreds of reads)
 * are called by warps of kDeepBatch neighbouring sites each: a site's hundreds
 * of records are spread over 32 lanes instead of walked by one, one site
 * after another, and the posteriors of the batch are taken together, a site
 * per lane.  What bounds the kernel is instruction issue; c2, 4 Mbp, some
 * 9,000 tiles: 2.26 ms with a warp per site that scanned all the tile's reads
 * for its depth, 1.87 in batches that count the depth of their sites in one
 * pass and end each site's own scan at its 255th record. */
constexpr int kDeepThreads = 32 * kTile;

/* a warp's shared memory */
struct DeepWarp32 {
    uint32_t recs[kDeepCap];
    uint8_t cnt[kDeepKeys];
    float sum[kDeepBatch][12];
    SitePileup pile[kDeepBatch];
    uint32_t span[2 * (kDeepBatch + 1)];
    uint32_t pad[2];
};
static_assert(sizeof(DeepWarp32) % 16 == 0, "16-byte aligned per warp");
constexpr size_t kDeepSmem = (size_t)kTile * sizeof(DeepWarp32);

/* The FP32 sums of a sorted column by its warp: each lane sums its records'
 * rows with compensation; the 32 sums are then added in a tree (the bound of
 * fast_posterior's k_units 9). */
__device__ __forceinline__ void deep_walk_sums(const CallArgs& a, const uint32_t* recs, uint8_t* cnt, int num,
                                               float* s) {
    Kahan10 k;
    k.init();
    deep_walk(a, recs, cnt, num, [&](int, bool valid, int qa, int coord, int o) {
        if (!valid) return;
        float x[10];
        lik32_row(a, qa, coord, o, x);
        k.add(x);
    });
#pragma unroll
    for (int v = 0; v < 10; ++v) {
        float t = k.s[v];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) t = __fadd_rn(t, __shfl_xor_sync(kFull, t, d));
        s[v] = t;
    }
}

/* Sites [first, first + sites) of a deep tile, called by one warp (as
 * fast_site: counts kept for later gap windows, the FP32 posterior, or the
 * site deferred with its records, which are piled up and sorted once more for
 * that: one site in some hundreds). */
__device__ __forceinline__ void deep_batch(const CallArgs& a, int64_t tile, int first, int sites, DeepWarp32& sm) {
    const int lane = threadIdx.x & 31;
    const int64_t s0 = tile * kTile, b0 = s0 + first;
    const uint8_t ori_t = s0 + lane < a.chr_len ? __ldg(a.ori + s0 + lane) : 0;
    const int32_t snp_t = tile_snp_row(a, tile, (ori_t & 8) != 0);
    const int n = (int)min((int64_t)sites, a.chr_len - b0);
    if (n <= 0) return;
    const uint8_t wflags = a.win_flags[s0 / kWin];
    const int64_t r_lo = a.warp_rng[tile * 2], r_hi = a.warp_rng[tile * 2 + 1];
    const DeepSpan span = deep_spans(a, r_lo, r_hi, b0, sm.span);
    auto pileup = [&](int j) {
        const SitePileup p = deep_pileup(a, r_lo + __shfl_sync(kFull, span.skip, j), r_hi, b0 + j,
                                         __shfl_sync(kFull, span.depth, j), __shfl_sync(kFull, span.repeat, j), sm.recs);
        __syncwarp();
        deep_sort(sm.recs, p.num);
        return p;
    };
    for (int j = 0; j < n; ++j) {
        const SitePileup p = pileup(j);
        if (lane == 0) sm.pile[j] = p;
        float s[10];
        deep_walk_sums(a, sm.recs, sm.cnt, p.num, s);
        if (lane == 0) {
#pragma unroll
            for (int v = 0; v < 10; ++v) sm.sum[j][v] = s[v];
        }
        __syncwarp();
    }
    /* lane j < n: site b0 + j */
    const int64_t site = b0 + lane;
    const uint8_t ori = (uint8_t)__shfl_sync(kFull, ori_t, (first + lane) & 31);
    const int32_t snp_row = __shfl_sync(kFull, snp_t, (first + lane) & 31);
    uint8_t dflags = 0;
    if (lane < n) {
        const SitePileup p = sm.pile[lane];
        if (p.depth > 0xffff) atomicExch(a.error, 1);
        if (wflags & kWinKeepCounts) store_counts(a, site, p);
        SiteCall call;
        if ((site & 4095) == 0 && a.stats) dflags = kCallSampled;
        const bool empty = p.num == 0 && (p.ca[0] | p.ca[1] | p.ca[2] | p.ca[3]) == 0 && a.empty_valid[ori];
        if (empty) {
            call = a.empty_calls[ori];
            call.depth = p.depth;
            call.repeat_time = p.repeat;
            call.flags |= dflags;
        } else {
            float s[10];
#pragma unroll
            for (int v = 0; v < 10; ++v) s[v] = sm.sum[lane][v];
            if (fast_posterior(a, snp_row, ori, p, s, p.num, &call, 9.0f)) {
                call.flags |= dflags;
            } else {
                call = SiteCall{};
                dflags |= kCallPending;
                call.flags = dflags;
            }
        }
        a.out[site] = call;
    }
    /* the deferred sites and their sorted records to the pool */
    for (unsigned m = __ballot_sync(kFull, dflags != 0); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const SitePileup p = pileup(j);
        const uint8_t fl = (uint8_t)__shfl_sync(kFull, dflags, j);
        const int32_t row = __shfl_sync(kFull, snp_row, j);
        unsigned long long slot = 0, off = 0;
        if (lane == 0) {
            slot = atomicAdd(a.dcount, 1ull);
            off = atomicAdd(a.dcount + 1, (unsigned long long)p.num);
        }
        slot = __shfl_sync(kFull, slot, 0);
        off = __shfl_sync(kFull, off, 0);
        if ((int64_t)slot >= a.dsite_cap || (int64_t)(off + p.num) > a.dpool_cap) continue;
        for (int i = lane; i < p.num; i += 32) a.dpool[off + i] = sm.recs[i];
        if (lane == 0) {
            DeferredSite d;
            d.site = b0 + j;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                d.cu[b] = (uint16_t)p.cu[b];
                d.qs[b] = (uint16_t)p.qs[b];
                d.ca[b] = p.ca[b];
            }
            d.depth = p.depth;
            d.repeat = p.repeat;
            d.rec_off = (uint32_t)off;
            d.num = (uint16_t)p.num;
            d.dep_uni = (uint16_t)p.dep_uni;
            d.snp_row = row;
            d.flags = fl;
#pragma unroll
            for (int b = 0; b < 3; ++b) d.pad[b] = 0;
            a.dsites[slot] = d;
        }
        __syncwarp();
    }
    __syncwarp();
}

/* The first n tiles of the list, or with count the first *count, some
 * sites (deep_sites) at a time to each warp: from *next (zero before the launch), or in
 * strides of the grid. */
__global__ void __launch_bounds__(kDeepThreads, 1) call_deep_kernel(const __grid_constant__ CallArgs a, const int32_t* __restrict__ tiles,
                                                                    int n, const int* __restrict__ count, int* next) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    DeepWarp32& sm = reinterpret_cast<DeepWarp32*>(smem)[w];
    if (count) n = *count;
    const unsigned step = gridDim.x * (kDeepThreads / 32);
    const int sites = deep_sites(n, (int)step);
    const unsigned per = (unsigned)(kTile / sites), items = (unsigned)n * per;
    unsigned item = blockIdx.x * (kDeepThreads / 32) + w;
    while (item < items) {
        deep_batch(a, tiles[item / per] & ~kTileGeneral, (int)(item % per) * sites, sites, sm);
        unsigned nx = item + step;
        if (next) {
            if (lane == 0) nx = (unsigned)atomicAdd(next, 1) + step;
            nx = __shfl_sync(kFull, nx, 0);
        }
        item = nx;
    }
}

/* ------------------------------------------------------------------------ */
/* the persistent FP32 calling kernel                                        */
/* ------------------------------------------------------------------------ */

/* Reads of a tile staged in shared memory by the persistent kernel, and the
 * bytes of each read's row window (32 columns of 16-bit base|quality plus up
 * to 14 bytes before them, to start the copy on a 16-byte boundary).  A tile
 * with more reads than this (deep pileups) reads its rows from global memory
 * instead. */
constexpr int kStageReads = 56;
constexpr int kStageSlot = 80;
constexpr uint64_t kStageWaitNs = 1000000000ull;   /* bound on one wait for a tile's bulk copies */
constexpr int kStageHeader = 16 + kStageReads * 12;
/* how the persistent kernel fetches a tile's reads */
constexpr int kStreamPlain = 0;      /* loads from global memory (through L1/L2) */
constexpr int kStreamPrefetch = 1;   /* the same, after a bulk prefetch of the rows into L2 */
constexpr int kStreamStaged = 2;     /* bulk copies into shared memory, one tile ahead */
static_assert(kStageHeader % 16 == 0 && kStageSlot % 16 == 0, "staging buffers are 16-byte aligned");

/* records [slots][kTile] and the pcr state of the general form; the bins that
 * try the short form first: its records and scratch in the same place */
__host__ __device__ constexpr size_t call_smem_bytes(int slots, int L) {
    const size_t general = ((size_t)slots * kTile + (size_t)pcr_smem_words(slots, L, true)) * 4;
    const size_t lean = slots <= kLeanG ? lean_smem_bytes(slots, L) : 0;
    return general > lean ? general : lean;
}

/* shared memory of one warp of the persistent kernel (a multiple of 16) */
__host__ __device__ constexpr size_t stream_warp_smem(int slots, int L, int mode) {
    const size_t n = mode != kStreamStaged ? lean_smem_bytes(slots, L)
                                           : call_smem_bytes(slots, L) + (size_t)kStageHeader + (size_t)kStageReads * kStageSlot;
    return (n + 15) & ~(size_t)15;
}

/* One launch over the FP32 windows' tiles of a segment: each warp takes
 * kStreamChunk consecutive tiles at a time from a counter, so the tiles in
 * flight are neighbours and the read rows they share are fetched from DRAM
 * about once and then served by L2.  The grid is sized to the resident CTAs,
 * whatever the segment's length.  A tile whose window needs the FP64 form
 * (its likelihood is kept for, or taken from, another window), or one with a
 * site of more than SLOTS records, is appended to the leftover list for the
 * binned kernels instead.
 *
 * MODE kStreamPrefetch: as soon as a warp takes a tile, it asks the
 * bulk-copy unit to prefetch the next tile's read rows into L2
 * (cp.async.bulk.prefetch), which costs no shared memory.
 * MODE kStreamStaged: as soon as a tile's pileup is done, the warp stages the
 * next tile's reads in shared memory - their start, length and strand with plain
 * loads, and each covering read's 32-column row window with one bulk copy
 * (cp.async.bulk) completing on the warp's mbarrier - so that the copies run
 * while the current tile is sorted, walked and summed, and the next pileup
 * reads only shared memory.  A wait for the copies that does not complete
 * within kStageWaitNs sets error code 5 and ends the warp. */
template <int SLOTS, int MODE>
__global__ void __launch_bounds__(32 * kStreamWarps, kFastCtasPerSm / kStreamWarps) call_stream_kernel(const __grid_constant__ CallArgs a, StreamQueue q) {
    constexpr bool STAGED = MODE == kStreamStaged;
    extern __shared__ __align__(16) uint8_t smem[];
    const int t = threadIdx.x & 31;
    uint8_t* base = smem + (threadIdx.x >> 5) * stream_warp_smem(SLOTS, a.L, MODE);
    uint64_t* bar = nullptr;
    int32_t* s_pos = nullptr;
    uint32_t* s_lhs = nullptr;
    int32_t* s_rbase = nullptr;
    uint8_t* s_rows = nullptr;
    if (STAGED) {
        bar = reinterpret_cast<uint64_t*>(base);
        s_pos = reinterpret_cast<int32_t*>(base + 16);
        s_lhs = reinterpret_cast<uint32_t*>(s_pos + kStageReads);
        s_rbase = reinterpret_cast<int32_t*>(s_lhs + kStageReads);
        s_rows = base + kStageHeader;
        base = s_rows + kStageReads * kStageSlot;
    }
    uint32_t* recs_all = reinterpret_cast<uint32_t*>(base);
    uint32_t* seen_all = recs_all + SLOTS * kTile;
    uint32_t* recs = recs_all + t;
    uint32_t* seen = seen_all + t;
    const int64_t n = q.t_end - q.t_begin;

    /* tiles in order: kStreamChunk at a time from the counter; -1 at the end */
    int64_t chunk_next = 0, chunk_end = 0;
    auto next_tile = [&]() -> int64_t {
        if (chunk_next >= chunk_end) {
            unsigned long long first = 0;
            if (t == 0) first = atomicAdd(q.next, (unsigned long long)kStreamChunk);
            first = __shfl_sync(kFull, first, 0);
            chunk_next = (int64_t)first;
            chunk_end = min(chunk_next + (int64_t)kStreamChunk, n);
            if (chunk_next >= n) {
                chunk_end = 0;
                return -1;
            }
        }
        return q.t_begin + chunk_next++;
    };
    auto fp64_window = [&](int64_t tile) {
        return (a.win_flags[(int)(tile * kTile / kWin)] & (kWinKeepLik | kWinExternalLik)) != 0;
    };
    /* stage the reads of `tile` (see above); their count, or -1 when the
     * tile is not staged.  Every lane calls it, after its last read of the
     * buffers. */
    auto stage = [&](int64_t tile) -> int {
        if (!STAGED || tile < 0 || fp64_window(tile)) return -1;
        const int64_t r_lo = a.tile_rng[tile * 2], r_hi = a.tile_rng[tile * 2 + 1];
        const int64_t nr = r_hi - r_lo;
        if (nr > kStageReads) return -1;
        const int64_t s0 = tile * kTile;
        uint32_t bytes[2] = {0u, 0u}, total = 0;
        const uint8_t* src[2] = {nullptr, nullptr};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int k = t + 32 * j;
            if (k >= nr) continue;
            const int64_t r = r_lo + k;
            const int32_t pos = __ldg(a.pos + r);
            const uint32_t lh = (uint32_t)__ldg(a.lenhit + r);
            const uint32_t minus = __ldg(a.strand + r) != '+';
            const int len = (int)(lh >> 16);
            const int c_lo = max(0, (int)(s0 - pos));
            const int c_hi = min(len, (int)(s0 + kTile - pos));
            const int64_t e_lo = (r * a.L + c_lo) * 2;   /* byte offset of column c_lo in the rows */
            const int m = (int)(e_lo & 15);
            if (c_hi > c_lo) {
                bytes[j] = (uint32_t)((m + 2 * (c_hi - c_lo) + 15) & ~15);
                src[j] = reinterpret_cast<const uint8_t*>(a.bq) + (e_lo - m);
            }
            s_pos[k] = pos;
            s_lhs[k] = lh | (minus << 31);
            s_rbase[k] = k * kStageSlot + m - 2 * c_lo;
            total += bytes[j];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(kFull, total, off);
        /* this lane's reads of the rows are done before the copies overwrite them */
        fence_proxy_async_smem();
        if (t == 0) mbar_arrive_expect_tx(bar, total);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (bytes[j]) bulk_copy_g2s(s_rows + (t + 32 * j) * kStageSlot, src[j], bytes[j], bar);
        return (int)nr;
    };

    /* the read rows of `tile` into L2 (the rows of a tile's reads are one
     * contiguous block; the bulk unit wants 16-byte bounds, and the row
     * array has slack past its end for the rounding) */
    auto prefetch_l2 = [&](int64_t tile) {
        if (MODE != kStreamPrefetch || tile < 0 || t != 0) return;
        const int64_t r_lo = a.tile_rng[tile * 2], r_hi = a.tile_rng[tile * 2 + 1];
        if (r_hi <= r_lo) return;
        const uintptr_t lo = reinterpret_cast<uintptr_t>(a.bq + r_lo * a.L) & ~(uintptr_t)15;
        const uintptr_t hi = (reinterpret_cast<uintptr_t>(a.bq + r_hi * a.L) + 15) & ~(uintptr_t)15;
        bulk_prefetch_l2(reinterpret_cast<const void*>(lo), (uint32_t)(hi - lo));
    };

    uint32_t phase = 0;
    if (STAGED) {
        if (t == 0) mbar_init(bar, 1);
        __syncwarp();
    }
    int64_t tile = next_tile();
    int staged_n = stage(tile);
    while (tile >= 0) {
        const int64_t s0 = tile * kTile;
        const int win = (int)(s0 / kWin);
        const uint8_t wflags = a.win_flags[win];
        const int64_t nxt = next_tile();
        prefetch_l2(nxt);
        if (wflags & (kWinKeepLik | kWinExternalLik)) {
            if (t == 0) q.leftover[atomicAdd(q.n_leftover, 1)] = (int32_t)tile | kTileGeneral;
            tile = nxt;
            staged_n = stage(tile);
            continue;
        }
        int staged_next = -1;
        LeanTook took;
        if (STAGED) {
            const int64_t site = s0 + t;
            const bool active = site < a.chr_len;
            const uint8_t ori = active ? __ldg(a.ori + site) : 0;
            const int32_t snp_row = tile_snp_row(a, tile, (ori & 8) != 0);
            bool overflow = false;
            SitePileup p;
            if (staged_n >= 0) {
                if (!mbar_wait_bounded(bar, phase, kStageWaitNs)) {
                    if (t == 0) atomicExch(a.error, 5);
                    (void)mbar_wait_bounded(bar, phase, kStageWaitNs);
                    return;
                }
                phase ^= 1u;
                const StagedReads sr{s_pos, s_lhs, s_rbase, s_rows, staged_n};
                p = warp_pileup_staged<SLOTS>(a, sr, site, active, recs, &overflow).unpack();
            } else {
                p = warp_pileup<SLOTS>(a, a.tile_rng[tile * 2], a.tile_rng[tile * 2 + 1], site, active, recs, &overflow)
                        .unpack();
            }
            /* the staging buffers are free: stage the next tile now, so that its
             * copies run while this one is sorted, walked and summed */
            staged_next = stage(nxt);
            took = __any_sync(kFull, overflow) ? kLeanDeep : kLeanTook;
            if (took == kLeanTook) {
                /* one sort network for every tile: specialised networks per
                 * tile depth made the kernel's code larger and it ran slower */
                if (active) sort_column<SLOTS>(recs, p.num);
                fast_site<SLOTS>(a, site, active, ori, wflags, snp_row, p, recs, seen);
            }
        } else {
            took = lean_tile<SLOTS>(a, tile, a.tile_rng[tile * 2], a.tile_rng[tile * 2 + 1], wflags, recs_all, seen_all);
        }
        if (took != kLeanTook && t == 0)
            q.leftover[atomicAdd(q.n_leftover, 1)] = (int32_t)tile | (took == kLeanNever ? kTileGeneral : 0);
        tile = nxt;
        staged_n = staged_next;
        __syncwarp();
    }
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */

template <int SLOTS, int MODE>
static cudaError_t stream_attr(int L, int* ctas_per_sm, int carveout = 0) {
    const int smem = (int)(kStreamWarps * stream_warp_smem(SLOTS, L, MODE));
    cudaError_t e =
        cudaFuncSetAttribute(call_stream_kernel<SLOTS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    /* a preferred shared-memory carveout (percent; 0 leaves the default) is a
     * hint: a refusal only costs speed, and its error is cleared */
    if (e == cudaSuccess && carveout > 0 &&
        cudaFuncSetAttribute(call_stream_kernel<SLOTS, MODE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             carveout) != cudaSuccess)
        (void)cudaGetLastError();
    if (e == cudaSuccess && ctas_per_sm)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, call_stream_kernel<SLOTS, MODE>,
                                                          32 * kStreamWarps, smem);
    return e;
}

template <int SLOTS, int MODE>
static cudaError_t launch_stream_one(const CallArgs& a, const StreamQueue& q, int ctas, int carveout,
                                     cudaStream_t stream) {
    cudaError_t e = g_launch_attributes ? stream_attr<SLOTS, MODE>(a.L, nullptr, carveout) : cudaSuccess;
    if (e != cudaSuccess) return e;
    call_stream_kernel<SLOTS, MODE>
        <<<ctas, 32 * kStreamWarps, kStreamWarps * stream_warp_smem(SLOTS, a.L, MODE), stream>>>(a, q);
    return cudaGetLastError();
}

template <int SLOTS>
static cudaError_t stream_dispatch(int mode, const CallArgs* a, const StreamQueue* q, int ctas, int carveout,
                                   cudaStream_t stream, int L, int* ctas_per_sm) {
    if (!a) {
        return mode == kStreamStaged     ? stream_attr<SLOTS, kStreamStaged>(L, ctas_per_sm, carveout)
               : mode == kStreamPrefetch ? stream_attr<SLOTS, kStreamPrefetch>(L, ctas_per_sm, carveout)
                                         : stream_attr<SLOTS, kStreamPlain>(L, ctas_per_sm, carveout);
    }
    return mode == kStreamStaged     ? launch_stream_one<SLOTS, kStreamStaged>(*a, *q, ctas, carveout, stream)
           : mode == kStreamPrefetch ? launch_stream_one<SLOTS, kStreamPrefetch>(*a, *q, ctas, carveout, stream)
                                     : launch_stream_one<SLOTS, kStreamPlain>(*a, *q, ctas, carveout, stream);
}

/* resident CTAs on one SM of the persistent kernel with `slots` record
 * slots (48 or 64) and read mode `mode` (0 plain, 1 L2 prefetch, 2 staged
 * in shared memory) */
int stream_ctas_per_sm(int slots, int L, int mode, int carveout) {
    int n = 0;
    const cudaError_t e = slots <= 48 ? stream_dispatch<48>(mode, nullptr, nullptr, 0, carveout, nullptr, L, &n)
                                      : stream_dispatch<64>(mode, nullptr, nullptr, 0, carveout, nullptr, L, &n);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

/* The persistent FP32 kernel over q's tiles with `ctas` CTAs; slots is 48 or
 * 64.  q.next and q.n_leftover must be zero. */
cudaError_t launch_stream(const CallArgs& a, const StreamQueue& q, int slots, int mode, int ctas, int carveout,
                          cudaStream_t stream) {
    if (q.t_end <= q.t_begin) return cudaSuccess;
    return slots <= 48 ? stream_dispatch<48>(mode, &a, &q, ctas, carveout, stream, a.L, nullptr)
                       : stream_dispatch<64>(mode, &a, &q, ctas, carveout, stream, a.L, nullptr);
}

/* set the bin kernel's shared-memory size and carveout (percent; 0 leaves the
 * default); with ctas_per_sm, its resident CTAs on one SM */
template <int SLOTS>
static cudaError_t fast_attr(int L, int carveout, int* ctas_per_sm) {
    /* the deep bin has its own kernel (call_deep_kernel) */
    constexpr bool deep = SLOTS >= kDeepSlots;
    const int smem = deep ? (int)kDeepSmem : (int)call_smem_bytes(SLOTS, L);
    const void* fn;
    if constexpr (deep) fn = reinterpret_cast<const void*>(call_deep_kernel);
    else fn = reinterpret_cast<const void*>(call_fast_kernel<SLOTS>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    /* the carveout is a hint: a refusal only costs speed, and its error is
     * cleared so that it is not taken for the launch's */
    if (carveout > 0 && cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, carveout) != cudaSuccess)
        (void)cudaGetLastError();
    if (ctas_per_sm) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, deep ? kDeepThreads : kTile, smem);
    return cudaSuccess;
}

template <int SLOTS>
static cudaError_t launch_fast(const CallArgs& a, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream) {
    cudaError_t e = g_launch_attributes ? fast_attr<SLOTS>(a.L, bl.carveout, nullptr) : cudaSuccess;
    if (e != cudaSuccess) return e;
    constexpr int64_t kWarps = kDeepThreads / 32;
    const unsigned grid = (unsigned)(bl.d_count                ? bl.grid
                                     : SLOTS >= kDeepSlots ? ((int64_t)bl.count * kDeepBatches + kWarps - 1) / kWarps
                                                           : bl.count);
    if (grid == 0) return cudaSuccess;
    if constexpr (SLOTS >= kDeepSlots)
        call_deep_kernel<<<grid, kDeepThreads, kDeepSmem, stream>>>(a, tiles, bl.count, bl.d_count,
                                                                    bl.d_count ? bl.d_next : nullptr);
    else
        call_fast_kernel<SLOTS><<<grid, kTile, call_smem_bytes(SLOTS, a.L), stream>>>(a, tiles, bl.d_count,
                                                                                            bl.d_next);
    return cudaGetLastError();
}

cudaError_t launch_fast_bin(const CallArgs& a, int bin, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream) {
    switch (bin) {
        case 0: return launch_fast<32>(a, tiles, bl, stream);
        case 1: return launch_fast<40>(a, tiles, bl, stream);
        case 2: return launch_fast<48>(a, tiles, bl, stream);
        case 3: return launch_fast<64>(a, tiles, bl, stream);
        case 4: return launch_fast<96>(a, tiles, bl, stream);
        case 5: return launch_fast<128>(a, tiles, bl, stream);
        default: return launch_fast<256>(a, tiles, bl, stream);
    }
}

cudaError_t fast_bin_attr(int bin, int L, int carveout, int* ctas_per_sm) {
    switch (bin) {
        case 0: return fast_attr<32>(L, carveout, ctas_per_sm);
        case 1: return fast_attr<40>(L, carveout, ctas_per_sm);
        case 2: return fast_attr<48>(L, carveout, ctas_per_sm);
        case 3: return fast_attr<64>(L, carveout, ctas_per_sm);
        case 4: return fast_attr<96>(L, carveout, ctas_per_sm);
        case 5: return fast_attr<128>(L, carveout, ctas_per_sm);
        default: return fast_attr<256>(L, carveout, ctas_per_sm);
    }
}

}  // namespace gsnp
