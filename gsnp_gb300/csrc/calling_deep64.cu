/*
 * calling_deep64.cu - the FP64 form of the deep bin: tiles with a site of more
 * than 128 records.
 *
 * A lane per site needs 32 KB of record columns a warp there, so six warps an
 * SM walked columns of hundreds of records one load after another: 0.5 us a
 * tile over the whole chip.  Here a warp takes kBatch neighbouring sites of a
 * tile.  One after another it piles up, sorts and walks each of them, a record
 * per lane (deep.cuh), and keeps of each record the table row its walk led to,
 * 16 bits in shared memory, and the base of its word in two bit planes (the
 * word's, not the read's: a quality of 0 or above 64 spills into it).  Then it adds the FP64 terms in the reference's
 * order, a genotype per lane and three sites at a time - an FP64 instruction
 * costs a warp 16 cycles of the SM's pipe however many lanes have work - and
 * takes the posterior of all of them at once, a site per lane.  Heterozygous
 * candidates, about one site in a thousand, have their column piled up again
 * for the rank sums, which saves holding the qualities of every site.
 * c2, 3 Mbp, 14,470 tiles of the bin: 7.2 -> 4.1 ms.  While its SMs are busy
 * half of their issue slots and of their FP64 pipe's are taken; the rest is the
 * latency of a site's shuffles and table rows (loading the next eight terms
 * ahead of the additions changed nothing).
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "calling.cuh"
#include "deep.cuh"
#include "lean.cuh"
#include "site_math.cuh"
#include "tile.cuh"

namespace gsnp {

namespace {

constexpr int kBatch = kDeepBatch;            /* sites a warp holds */
constexpr int kAtOnce = 3;                    /* sites summed together, ten lanes each */
constexpr int kDeep64Warps = 24;

/* a warp's shared memory; the counters of the walk, the sums and the rank
 * histogram are used one after another */
struct DeepWarp {
    uint16_t row[kBatch][kDeepCap];           /* adjusted quality * L + cycle of each record */
    uint2 base[kBatch][kDeepCap / 32];        /* bits 0 and 1 of 32 records' bases */
    uint32_t recs[kDeepCap];
    union {
        uint8_t cnt[kDeepKeys];
        struct {
            double sum[kBatch][10];           /* by table column */
            int32_t hist[2][66];
        } s;
    } u;
    uint32_t span[2 * (kBatch + 1)];
    uint32_t pad[2];
    int32_t rank2[kBatch][2];                 /* twice the rank sums of the candidate's alleles */
    uint16_t num[kBatch];                     /* records */
};
static_assert(sizeof(DeepWarp) % 16 == 0, "16-byte aligned per warp");

/* rank: the rank sums of genotype cand */
__device__ __noinline__ void deep_posterior(const CallArgs& a, int64_t site, uint8_t ori, int32_t snp_row,
                                            const SitePileup& p, const double* sum, const double* lp,
                                            const int32_t* rank2) {
    double tl[16];
    GSNP_ROLLED
    for (int g = 0; g < 16; ++g) tl[g] = 0.0;
    GSNP_ROLLED
    for (int v = 0; v < 10; ++v) tl[genotype_of(v)] = sum[v];
    auto nq = [&](int b) { return neighbour_qsum(a, site, b); };
    auto rank = [&](int g, bool* normal) -> double {
        const int ia = g & 3, ib = (g >> 2) & 3;
        if (ia == ib) return 1.0;
        if (p.cu[ia] == 0 || p.cu[ib] == 0) return 0.0;
        return rank_value(a.p_rank, p.cu[ia], p.cu[ib], 0.5 * (double)rank2[0], 0.5 * (double)rank2[1], normal);
    };
    SiteCall call;
    site_posterior_ranked<true>(a, ori, p, tl, nullptr, lp, rank, nq, &call);
    a.out[site] = call;
}

/* Sites [first, first + sites) of a tile, sites <= kBatch, by one warp. */
__device__ __forceinline__ void deep_batch(const CallArgs& a, int64_t tile, int first, int sites, DeepWarp& sm) {
    const int lane = threadIdx.x & 31;
    const int64_t s0 = tile * kTile;
    const uint8_t ori_t = s0 + lane < a.chr_len ? __ldg(a.ori + s0 + lane) : 0;
    const int32_t snp_t = tile_snp_row(a, tile, (ori_t & 8) != 0);
    const int n = (int)min((int64_t)sites, a.chr_len - (s0 + first));
    if (n <= 0) return;
    /* lane j < n owns site s0 + first + j */
    const int64_t site = s0 + first + lane;
    const uint8_t ori = (uint8_t)__shfl_sync(kFull, ori_t, (first + lane) & 31);
    const int32_t snp_row = __shfl_sync(kFull, snp_t, (first + lane) & 31);
    const int win = (int)(s0 / kWin);
    const uint8_t wflags = a.win_flags[win];
    const int64_t r_lo = a.warp_rng[tile * 2], r_hi = a.warp_rng[tile * 2 + 1];
    const bool external = (wflags & kWinExternalLik) != 0;
    const DeepSpan span = deep_spans(a, r_lo, r_hi, s0 + first, sm.span);
    auto pileup = [&](int j) {
        const SitePileup p = deep_pileup(a, r_lo + __shfl_sync(kFull, span.skip, j), r_hi, s0 + first + j,
                                         __shfl_sync(kFull, span.depth, j), __shfl_sync(kFull, span.repeat, j), sm.recs);
        __syncwarp();
        return p;
    };
    SitePileup mine = {};
    for (int j = 0; j < n; ++j) {
        const SitePileup p = pileup(j);
        if (lane == j) mine = p;
        if (lane == 0) sm.num[j] = (uint16_t)p.num;
        if (external) continue;
        deep_sort(sm.recs, p.num);
        deep_walk(a, sm.recs, sm.u.cnt, p.num, [&](int c0, bool valid, int qa, int coord, int o) {
            if (valid) sm.row[j][c0 + lane] = (uint16_t)(qa * a.L + coord);
            const uint2 planes = make_uint2(__ballot_sync(kFull, o & 1), __ballot_sync(kFull, o & 2));
            if (lane == 0) sm.base[j][c0 / 32] = planes;
        });
        __syncwarp();
    }
    if (lane < n) {
        if (mine.depth > 0xffff) atomicExch(a.error, 1);
        if (wflags & kWinKeepCounts) store_counts(a, site, mine);
    }
    /* the sums: lane 10 u + v has column v of site j0 + u */
    const int u = lane / 10, v = lane % 10;
    for (int j0 = 0; j0 < n; j0 += kAtOnce) {
        const int j = j0 + u;
        const bool has = u < kAtOnce && j < n;
        double s = 0.0;
        if (external) {
            const int src = a.win_lik_src[win];
            if (has && src >= 0)
                s = a.lik_keep[((int64_t)src * kWin + (s0 + first + j - (int64_t)win * kWin)) * 10 + v];
        } else {
            const int jj = has ? j : 0;
            const int num = has ? sm.num[jj] : 0;
            const int most = (int)__reduce_max_sync(kFull, (unsigned)num);
            const uint16_t* rows = sm.row[jj];
            const double* col = a.lik64 + v;
            for (int i0 = 0; i0 < most; i0 += 8) {
                double x[8];
                const uint2 planes = sm.base[jj][i0 / 32];
                const uint32_t p0 = planes.x >> (i0 & 31), p1 = planes.y >> (i0 & 31);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int i = i0 + k;
                    x[k] = 0.0;
                    if (i < num)
                        x[k] = __ldg(col + ((int)rows[i] * 4 + (int)((p0 >> k & 1u) | (p1 >> k & 1u) << 1)) * 10);
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (i0 + k < num) s = GSNP_DADD(s, x[k]);
            }
        }
        if (has) {
            sm.u.s.sum[j][v] = s;
            if ((wflags & kWinKeepLik) && !external) a.lik_keep[(s0 + first + j) * 10 + v] = s;
        }
    }
    __syncwarp();
    /* the best genotype of each site, as site_posterior_ranked finds it, and
     * the rank sums of the heterozygous ones */
    double lp[16];
    bool het = false;
    int best = 16;
    if (lane < n) {
        load_log_prior(a, snp_row, ori, lp);
        if (a.rank_sum && !a.monoploid) {
            double top = 0.0;
#pragma unroll
            for (int g = 0; g < 16; ++g) {
                if ((g >> 2) > (g & 3)) continue;
                const double t = GSNP_DADD(sm.u.s.sum[lane][col_of(g >> 2, g & 3)], lp[g]);
                if (best == 16 || t >= top) {
                    best = g;
                    top = t;
                }
            }
            het = (best >> 2) != (best & 3);
        }
    }
    for (unsigned m = __ballot_sync(kFull, het); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int g = __shfl_sync(kFull, best, j);
        const SitePileup p = pileup(j);
        warp_ranks(a, sm.recs, p.num, g, sm.u.s.hist, sm.rank2[j]);
    }
    if (lane < n) deep_posterior(a, site, ori, snp_row, mine, sm.u.s.sum[lane], lp, sm.rank2[lane]);
    __syncwarp();
}

/* The first n tiles of the list, or with count the first *count, some
 * sites (deep_sites) at a time to each warp; from *next (zero before the launch), or in strides
 * of the grid. */
__global__ void __launch_bounds__(32 * kDeep64Warps, 1)
    call_deep64_kernel(const __grid_constant__ CallArgs a, const int32_t* __restrict__ tiles, int n,
                       const int* __restrict__ count, int* next) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    DeepWarp& sm = reinterpret_cast<DeepWarp*>(smem)[w];
    if (count) n = *count;
    const unsigned step = gridDim.x * kDeep64Warps;
    const int sites = deep_sites(n, (int)step);
    const unsigned per = (unsigned)(kTile / sites), items = (unsigned)n * per;
    unsigned item = blockIdx.x * kDeep64Warps + w;
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

constexpr int kDeep64Smem = kDeep64Warps * (int)sizeof(DeepWarp);
static_assert(kDeep64Smem <= 227 * 1024, "one CTA an SM");

}  // namespace

cudaError_t deep64_attr(int* ctas_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(call_deep64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDeep64Smem);
    if (e != cudaSuccess) return e;
    if (ctas_per_sm)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, call_deep64_kernel, 32 * kDeep64Warps,
                                                             kDeep64Smem);
    return cudaSuccess;
}

cudaError_t launch_deep64(const CallArgs& a, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream) {
    const cudaError_t e = g_launch_attributes ? deep64_attr(nullptr) : cudaSuccess;
    if (e != cudaSuccess) return e;
    const unsigned grid = bl.d_count ? (unsigned)bl.grid
                                     : (unsigned)(((int64_t)bl.count * kDeepBatches + kDeep64Warps - 1) / kDeep64Warps);
    if (grid == 0) return cudaSuccess;
    call_deep64_kernel<<<grid, 32 * kDeep64Warps, kDeep64Smem, stream>>>(a, tiles, bl.count, bl.d_count,
                                                                       bl.d_count ? bl.d_next : nullptr);
    return cudaGetLastError();
}

}  // namespace gsnp
