/*
 * tile.cuh - what the FP64 and the FP32 calling kernels share: the general
 * pileup of a warp's 32 sites, a tile's known-SNP rows, the counts kept for
 * gap windows, the next site's quality sum, and the hand-out of listed tiles.
 */
#ifndef GSNP_TILE_CUH
#define GSNP_TILE_CUH

#include "calling.cuh"
#include "site_math.cuh"

namespace gsnp {

constexpr unsigned kFull = 0xffffffffu;

/* bits of pcr occurrence count per (strand, cycle) key (walk_records) in the
 * bins of each record-slot capacity, for the FP32 (fast) or the FP64 kernel.
 * Two bits leave a scan back over the group only for a key seen three
 * times; at 30x one record in about fourteen repeats a key, and with one bit
 * the scans of single lanes held the whole warp (c1 at 25% scale:
 * fast<40> 2.63 -> 2.37 ms, tiles<40> 5.26 -> 4.97 ms).  The FP32 kernel's
 * 32-slot bin ran 3% slower with them and keeps one bit. */
__host__ __device__ constexpr int kPcrBits(int slots, bool fast) {
    return slots >= 96 ? 4 : (fast && slots <= 32) ? 1 : 2;
}

/* Running pileup of one site: per-base counters packed - count_uni 4 x 8
 * bits (at most 255 unique bases), q_sum and count_all 4 x 16 bits (a site
 * deeper than 65535 is a capacity error) - and its record column. */
struct PileupAcc {
    uint32_t cu4 = 0;
    uint64_t qs4 = 0, ca4 = 0;
    uint32_t depth = 0, repeat = 0;
    int dep_uni = 0, num = 0;
    bool overflow = false;

    /* one covering read's base (kernel/update_kernel.cu:278-325): e is its
     * element at the site, lh its (len << 16) | hit */
    template <int SLOTS>
    __device__ __forceinline__ void take(uint32_t e, uint32_t lh, int coord, int minus, uint32_t* recs) {
        const int rlen = (int)(lh >> 16);
        const uint32_t hit = lh & 0xffffu;
        depth += 1;
        repeat += hit;
        if (!elem_valid(e) || dep_uni >= 0xFF) return;
        const uint32_t base = (uint32_t)elem_base(e);
        const int sh = (int)base * 16;
        if (hit == 1) {
            dep_uni += 1;
            const int q = elem_q(e);
            const uint32_t coord_val = minus ? (uint32_t)(rlen - 1 - coord) : (uint32_t)coord;
            const uint32_t w = make_record_of(base, q, coord_val, (uint32_t)minus);
            if (num < SLOTS) {
                recs[num * kTile] = w;
                num += 1;
            } else {
                overflow = true;
            }
            cu4 += 1u << (sh >> 1);
            qs4 += (uint64_t)(uint32_t)q << sh;
        }
        ca4 += 1ull << sh;
    }

    __device__ __forceinline__ PackedPileup finish(const CallArgs& a, bool* report_overflow) const {
        if (report_overflow) *report_overflow = overflow;
        else if (overflow) atomicExch(a.error, 2);
        if (depth > 0xffff) atomicExch(a.error, 1);
        PackedPileup pk;
        pk.cu4 = cu4;
        pk.qs4 = qs4;
        pk.ca4 = ca4;
        pk.depth = depth;
        pk.repeat = repeat;
        pk.dep_uni = (uint16_t)dep_uni;
        pk.num = (uint16_t)num;
        return pk;
    }
};

/* Pileup of one warp's 32 consecutive sites (kernel/update_kernel.cu:260-325).
 * Reads [r_lo, r_hi) are those starting in [w0 - L + 1, w0 + 31]; their
 * positions, lengths and strands are loaded 32 at a time and broadcast, and
 * each lane takes the reads that cover its own site.  Records are appended to
 * the site's column in pileup order.  Lanes with !active only keep the warp's
 * loop going. */
template <int SLOTS>
__device__ __forceinline__ PackedPileup warp_pileup(const CallArgs& a, int64_t r_lo, int64_t r_hi, int64_t site,
                                                   bool active, uint32_t* recs, bool* report_overflow = nullptr) {
    /* records are appended in pileup order; sort_column puts them in
     * ascending order after the pileup */
    const int lane = threadIdx.x & 31;
    const int L = a.L;
    PileupAcc acc;
    for (int64_t rb = r_lo; rb < r_hi; rb += 32) {
        const int64_t r = rb + lane;
        int32_t mpos = 0;
        uint32_t mlh = 0;
        int mminus = 0;
        if (r < r_hi) {
            mpos = __ldg(a.pos + r);
            mlh = (uint32_t)__ldg(a.lenhit + r);
            mminus = __ldg(a.strand + r) != '+';
        }
        const int cnt = (int)((r_hi - rb) < 32 ? (r_hi - rb) : 32);
        const uint16_t* rows = a.bq + rb * L;
        /* four reads at a time: their row loads are issued together, then
         * the covering ones are taken in order */
        for (int k0 = 0; k0 < cnt; k0 += 4) {
            uint32_t bqv[4], lhv[4];
            int coordv[4], minusv[4];
            bool covv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u;
                const int32_t start = __shfl_sync(kFull, mpos, k & 31);
                lhv[u] = __shfl_sync(kFull, mlh, k & 31);
                minusv[u] = __shfl_sync(kFull, mminus, k & 31);
                coordv[u] = (int)(site - start);
                covv[u] = active && k < cnt && coordv[u] >= 0 && coordv[u] < (int)(lhv[u] >> 16);
                bqv[u] = covv[u] ? (uint32_t)__ldg(rows + k * L + coordv[u]) : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (covv[u]) acc.take<SLOTS>(bqv[u], lhv[u], coordv[u], minusv[u], recs);
        }
    }
    return acc.finish(a, report_overflow);
}

/* dbSNP row of each flagged site of a tile: the rows before the tile plus the
 * flagged sites before it in the tile (the rows are the flagged sites in
 * position order).  Every lane of the tile's warp calls it. */
__device__ __forceinline__ int32_t tile_snp_row(const CallArgs& a, int64_t tile, bool flagged) {
    const unsigned b = __ballot_sync(kFull, flagged);
    const int lane = threadIdx.x & 31;
    return flagged ? a.tile_snp[tile] + __popc(b & ((1u << lane) - 1u)) : -1;
}

__device__ __forceinline__ void store_counts(const CallArgs& a, int64_t site, const SitePileup& p) {
    SiteCounts c;
#pragma unroll
    for (int i = 0; i < 4; ++i) { c.cu[i] = (uint16_t)p.cu[i]; c.qs[i] = (uint16_t)p.qs[i]; c.ca[i] = p.ca[i]; }
    c.depth = p.depth;
    c.repeat_time = p.repeat;
    a.counts[site] = c;
}

/* q_sum[b] of site + 1 as the reference's window array holds it when site is
 * called: every deposited read covering site + 1, except that at the last
 * site of a window the next entry is the window's tail, which holds only the
 * reads starting inside the window (kernel/update_kernel.cu:260-325). */
static __device__ __noinline__ int neighbour_qsum(const CallArgs& a, int64_t site, int b) {
    const int64_t p = site + 1;
    const int64_t win_end = (site / kWin + 1) * (int64_t)kWin;
    const int64_t max_start = (p == win_end) ? win_end - 1 : p;
    const int64_t t = p / kTile;
    int64_t lo, hi;
    if (p < win_end && t >= a.tile_lo && t < a.n_tiles) {
        /* p's tile's read range, [lower_bound(32 t - L + 1), lower_bound(32 t
         * + 32)): the same reads in the same order and a few more, which the
         * checks below skip, without two searches over every read.  (The
         * window's end is left to the searches: its next site can lie in a
         * tile the pass has not ranged.) */
        lo = a.tile_rng[t * 2];
        hi = a.tile_rng[t * 2 + 1];
    } else {
        lo = a.read_lo + lower_bound_g(a.pos + a.read_lo, a.n_reads - a.read_lo, p - a.L + 1);
        hi = a.read_lo + lower_bound_g(a.pos + a.read_lo, a.n_reads - a.read_lo, max_start + 1);
    }
    int dep_uni = 0, qsum = 0;
    for (int64_t r = lo; r < hi; ++r) {
        const int64_t start = __ldg(a.pos + r);
        if (start > max_start) break;   /* the starts ascend */
        const int coord = (int)(p - start);
        const uint32_t lh = (uint32_t)__ldg(a.lenhit + r);
        if (coord >= (int)(lh >> 16)) continue;
        const uint32_t e = __ldg(a.bq + r * a.L + coord);
        if (!elem_valid(e) || dep_uni >= 0xFF) continue;
        if ((lh & 0xffffu) == 1) {
            dep_uni += 1;
            if (elem_base(e) == b) qsum += elem_q(e);
        }
    }
    return qsum;
}

/* The list entries [0, *count) of a grid sized to the resident CTAs (one
 * warp each): every CTA takes entry blockIdx.x first, then the next entry not
 * yet taken from the counter *next (zero before the launch), so that the
 * entries in flight stay neighbours and a CTA that drew cheap tiles takes
 * more of them. */
template <typename F>
__device__ __forceinline__ void for_each_listed(const int* __restrict__ count, int* next, F&& f) {
    const int n = *count;
    int i = blockIdx.x;
    while (i < n) {
        f(i);
        __syncwarp();
        int j = 0;
        if ((threadIdx.x & 31) == 0) j = atomicAdd(next, 1);
        i = __shfl_sync(0xffffffffu, j, 0) + (int)gridDim.x;
    }
}

/* warps of a CTA of the persistent kernels: each works by itself; several share
 * the CTA's reserved shared memory */
constexpr int kStreamWarps = 4;

/* record-slot capacity of each depth bin */
constexpr int kSlots[kNumBins] = {32, 40, 48, 64, 96, 128, 256};
static_assert(kSlots[kDeeperBin] == kLeanG && kSlots[kGeneralBin] == 48, "the bins after a persistent kernel");

/* 32-bit words of shared memory a bin's kernel keeps its pcr counts in */
__host__ __device__ constexpr int pcr_smem_words(int slots, int L, bool fast) {
    return (2 * L + 32 / kPcrBits(slots, fast) - 1) / (32 / kPcrBits(slots, fast)) * kTile;
}

/* Launchers set their kernel's shared-memory size and carveout before each
 * launch, except while this thread captures a graph: the attributes were set
 * when the grids were sized, before the capture. */
extern thread_local bool g_launch_attributes;

/* launchers of the FP32 kernels (calling_fast.cu) behind launch_bin */
cudaError_t fast_bin_attr(int bin, int L, int carveout, int* ctas_per_sm);

/* the FP64 kernel of the deep bin (calling_deep64.cu) */
cudaError_t launch_deep64(const CallArgs& a, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream);
cudaError_t deep64_attr(int* ctas_per_sm);
cudaError_t launch_fast_bin(const CallArgs& a, int bin, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream);

}  // namespace gsnp

#endif
