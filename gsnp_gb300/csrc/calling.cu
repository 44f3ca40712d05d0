/*
 * calling.cu - fused consensus calling on sm_103a: pileup, per-site record
 * sort, dependency-adjusted likelihood, posterior, rank-sum test.
 *
 * One CTA handles a tile of kTile consecutive reference sites, one thread per
 * site.  The reference runs the same work as five kernels and a Thrust sort per
 * 262,144-site window, with every intermediate in global memory:
 *   kernel/update_kernel.cu:233-326     updateSparse_kernel (pileup)
 *   kernel/batchsort.cu:245-291         batchSortMP2 (per-site sort)
 *   kernel/likelihood_kernel.cu:168-256 likelihoodSparse_kernel
 *   kernel/posterior_kernel.cu:635-866  posterior_kernel, posterior_kernel2
 * Here the records of a site stay on the SM: the pileup appends them to the
 * site's column ([slot][site] layout, so a warp's accesses fall in 32 distinct
 * banks whatever slot each lane is at), the column is sorted in place
 * (column.cuh), the likelihood walks it in that order, and only the 32-byte
 * SiteCall leaves the SM.
 *
 * The pileup of a site is every deposited read that covers it, in (start, file)
 * order.  That equals the reference's window-resident pileup: its carried-over
 * tail holds the previous window's reads first and the 255-record cap is
 * applied in that same order (kernel/update_kernel.cu:265-268,288).  A warp
 * walks the reads that can cover any of its 32 sites once, in that order; each
 * read's row is read with one coalesced load per lane band.
 *
 * Most tiles are called in the short form (lean.cuh, lean_tile.cuh), which sums
 * only the genotypes that can decide a call; the rest in the general form of
 * tile.cuh.  The kernels:
 *   call_stream64_kernel, call_stream_kernel (calling_fast.cu)  persistent, one
 *                      launch per segment, tiles in genome order: FP64 sums,
 *                      or FP32 sums and an FP32 posterior for homozygous calls
 *                      that the error bound proves; tiles they cannot take go
 *                      to the binned kernels;
 *   call_tiles_kernel  FP64 sums in the reference's order, the tiles of a depth
 *                      bin (and windows whose likelihood another window reuses);
 *   call_fast_kernel   (calling_fast.cu) the FP32 form of a depth bin; a site it
 *                      cannot prove is deferred: its counts and sorted records
 *                      are appended to a small pool.  It runs no FP64
 *                      instruction;
 *   call_deep64_kernel, call_deep_kernel  (calling_deep64.cu, calling_fast.cu)
 *                      the deepest bin;
 *   deferred_sites_kernel  (deferred.cu) the deferred sites: the FP32 sums
 *                      again with the double-precision bound checks, the FP64
 *                      sums where those fail, the rank-sum test.
 * Tiles are binned by their deepest site (kNumBins record-slot capacities) so
 * that shared memory is sized for the tile, not for the worst case.
 */
#include <cuda_runtime.h>

#include "calling.cuh"
#include "lean.cuh"
#include "lean_tables.cuh"
#include "lean_tile.cuh"
#include "site_math.cuh"
#include "tile.cuh"

namespace gsnp {

namespace {

/* resident CTAs per SM the FP64 kernel is compiled for, which caps its
 * registers at 128 */
constexpr int kFp64CtasPerSm = 16 * 32 / kTile;
/* warps an SM the persistent FP64 kernel is compiled for (c1, 4 Mbp: 1.49 ms at
 * 16, 1.37 at 20, 1.35 at 24) */
constexpr int kStream64Warps = 24;

__device__ __forceinline__ int lower_bound_s(const int32_t* a, int n, int64_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

}  // namespace

/* ------------------------------------------------------------------------ */
/* tile classification                                                       */
/* ------------------------------------------------------------------------ */

/* Read range of every tile, [lower_bound(s0 - L + 1), lower_bound(s0 + kTile)),
 * in one pass over the sorted starts: read r is the lower bound of every
 * boundary b with pos[r - 1] < b <= pos[r].  Threads r_begin .. r_end; the
 * start of read r_end is next_pos (kNoRead past the last read), so that a
 * segment of the reads can be done before the next segment is on the device:
 * consecutive segments share their boundary thread, which writes the same
 * values twice.  Only tiles [tile_lo, n_tiles) are written.  When the device
 * holds reads from read_lo > 0 on (a streamed chunk, whose first read is the
 * lower bound of its first tile's first boundary), the start before read_lo
 * is taken as tile_lo * kTile - L: it is at least that read's start and below
 * every boundary of the chunk's tiles. */
__global__ void tile_bounds_kernel(const int32_t* __restrict__ pos, int64_t r_begin, int64_t r_end, int64_t next_pos,
                                   int64_t tile_lo, int64_t n_tiles, int64_t read_lo, int L,
                                   int64_t* __restrict__ rng) {
    const int64_t r = r_begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > r_end) return;
    const int64_t lo = r == 0 ? -kNoRead : r == read_lo ? tile_lo * kTile - L : (int64_t)pos[r - 1];
    const int64_t hi = r == r_end ? next_pos : (int64_t)pos[r];
    if (lo >= hi) return;
    auto fdiv = [](int64_t x) { return x >= 0 ? x / kTile : -((-x + kTile - 1) / kTile); };
    /* first boundaries t*kTile - L + 1 in (lo, hi] */
    int64_t t0 = fdiv(lo + L - 1) + 1, t1 = fdiv(hi + L - 1);
    if (t0 < tile_lo) t0 = tile_lo;
    if (t1 > n_tiles - 1) t1 = n_tiles - 1;
    for (int64_t t = t0; t <= t1; ++t) rng[t * 2] = r;
    /* second boundaries (t + 1)*kTile in (lo, hi] */
    t0 = fdiv(lo);
    t1 = fdiv(hi) - 1;
    if (t0 < tile_lo) t0 = tile_lo;
    if (t1 > n_tiles - 1) t1 = n_tiles - 1;
    for (int64_t t = t0; t <= t1; ++t) rng[t * 2 + 1] = r;
}

cudaError_t launch_tile_bounds(const CallArgs& a, int64_t r_begin, int64_t r_end, int64_t next_pos,
                               cudaStream_t stream) {
    const int64_t n = r_end - r_begin + 1;
    tile_bounds_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(a.pos, r_begin, r_end, next_pos, a.tile_lo,
                                                                         a.n_tiles, a.read_lo, a.L, a.tile_rng);
    return cudaGetLastError();
}

/* The FP64 call of a site with no record and no count for each of the 16
 * site codes (site_posterior over zero likelihoods), kept where it is
 * homozygous and does not depend on a dbSNP row. */
__global__ void empty_calls_kernel(CallArgs a, SiteCall* calls, uint8_t* valid) {
    const int code = threadIdx.x;
    if (code >= 16) return;
    SitePileup p;
#pragma unroll
    for (int i = 0; i < 4; ++i) { p.cu[i] = 0; p.qs[i] = 0; p.ca[i] = 0; }
    p.depth = 0;
    p.repeat = 0;
    p.dep_uni = 0;
    p.num = 0;
    double tl[16], lp[16];
    for (int i = 0; i < 16; ++i) {
        tl[i] = 0.0;
        lp[i] = a.log_prior[((code & 7) << 4) + i];
    }
    bool used_next = false;
    auto nq = [&](int) {
        used_next = true;
        return 0;
    };
    SiteCall c;
    site_posterior(a, (uint8_t)code, p, tl, nullptr, lp, nullptr, 1, nq, &c);
    const bool hom = (c.type1 >> 2) == (c.type1 & 3);
    valid[code] = hom && !used_next && !((code & 8) && a.refine);
    calls[code] = c;
}

cudaError_t launch_empty_calls(const CallArgs& a, SiteCall* calls, uint8_t* valid, cudaStream_t stream) {
    empty_calls_kernel<<<1, 32, 0, stream>>>(a, calls, valid);
    return cudaGetLastError();
}

/* Per tile: the deepest site's record need (reads starting in [site - L + 1,
 * site], capped at 255) picks the depth bin; the window's mode picks the FP64
 * kernel (bins 0 .. kNumBins-1) or the fast one (the next kNumBins).  The bins
 * start at min_bin, for a listed tile marked kTileGeneral at general_bin.  Each
 * warp's read range is stored for the calling kernels.  A CTA classifies
 * kClassifyTiles tiles and adds its bin counts to the global ones with one
 * atomic per bin. */
constexpr int kClassifyThreads = 256;
constexpr int kClassifyTiles = kClassifyThreads / kTile;
constexpr int kClassifyStage = 256;   /* read starts staged in shared memory per tile */
static_assert(kClassifyThreads % kTile == 0, "a classify CTA holds whole tiles");

__global__ void __launch_bounds__(kClassifyThreads) classify_tiles_kernel(CallArgs a, int pass, int min_bin,
                                                                          int general_bin, int64_t t_begin,
                                                                          int64_t t_end, int* bin_count,
                                                                          int32_t* bin_tiles,
                                                                          const int32_t* __restrict__ list,
                                                                          const int* __restrict__ d_count) {
    __shared__ int32_t spos[kClassifyTiles][kClassifyStage];
    __shared__ int smax[kClassifyThreads / 32];
    __shared__ int sbin_count[2 * kNumBins], sbin_base[2 * kNumBins];
    const int lt = threadIdx.x / kTile, tt = threadIdx.x % kTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    /* the tiles [t_begin, t_end), or with a list the tiles list[t_begin,
     * t_end); with d_count, t_end is t_begin + *d_count.  The CTAs take
     * kClassifyTiles tiles at a time, every gridDim.x-th group. */
    const int64_t end = d_count ? t_begin + *d_count : t_end;
    for (int64_t gbase = t_begin + (int64_t)blockIdx.x * kClassifyTiles; gbase < end;
         gbase += (int64_t)gridDim.x * kClassifyTiles) {
    const int64_t idx = gbase + lt;
    if (threadIdx.x < 2 * kNumBins) sbin_count[threadIdx.x] = 0;
    bool part = idx < end;
    const int32_t entry = list ? (part ? list[idx] : 0) : (int32_t)idx;
    const int64_t tile = entry & ~kTileGeneral;
    const int64_t s0 = tile * kTile;
    uint8_t wflags = 0;
    if (part) {
        wflags = a.win_flags[(int)(s0 / kWin)];
        part = ((wflags & kWinExternalLik) != 0) == (pass == 1);
    }
    int64_t r_lo = 0, r_hi = 0;
    if (part) {
        r_lo = a.tile_rng[tile * 2];
        r_hi = a.tile_rng[tile * 2 + 1];
    }
    const int n = (int)(r_hi - r_lo);
    const bool staged = r_hi - r_lo <= kClassifyStage;
    if (part && staged)
        for (int i = tt; i < n; i += kTile) spos[lt][i] = __ldg(a.pos + r_lo + i);
    __syncthreads();
    auto lb = [&](int64_t v) -> int64_t {
        return staged ? r_lo + lower_bound_s(spos[lt], n, v) : r_lo + lower_bound_g(a.pos + r_lo, r_hi - r_lo, v);
    };
    const int64_t site = s0 + tt;
    int need = 0;
    if (part && site < a.chr_len) {
        const int64_t c = lb(site + 1) - lb(site - a.L + 1);
        need = (int)(c < kMaxRecords ? c : kMaxRecords);
    }
    if (part && lane < 2) a.warp_rng[tile * 2 + lane] = lane == 0 ? lb(s0 - a.L + 1) : lb(s0 + kTile);
    for (int off = 16; off > 0; off >>= 1) need = max(need, __shfl_xor_sync(kFull, need, off));
    if (lane == 0) smax[warp] = need;
    __syncthreads();
    int my_bin = -1, my_rank = 0;
    if (part && tt == 0) {
        const int m = smax[lt];
        const bool fast = a.precision == 1 && !(wflags & (kWinKeepLik | kWinExternalLik));
        int bin = entry & kTileGeneral ? general_bin : min_bin;
        while (bin < kNumBins - 1 && m > a.bin_limit[bin]) ++bin;
        my_bin = bin + (fast ? kNumBins : 0);
        my_rank = atomicAdd(&sbin_count[my_bin], 1);
    }
    __syncthreads();
    if (threadIdx.x < 2 * kNumBins) {
        const int cnt = sbin_count[threadIdx.x];
        sbin_base[threadIdx.x] = cnt ? atomicAdd(&bin_count[threadIdx.x], cnt) : 0;
    }
    __syncthreads();
    if (my_bin >= 0) bin_tiles[(int64_t)my_bin * a.bin_stride + sbin_base[my_bin] + my_rank] = entry;
    __syncthreads();
    }
}

/* log10 genotype priors of every dbSNP row (kernel/posterior_kernel.cu:575-633,
 * the device version: no check of the number of listed alleles).  Run once per
 * reference and parameter set so that the calling kernels only load them; the
 * FP32 copy is by table column. */
__global__ void snp_log_prior_kernel(CallArgs a, double* out, float* out32) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n_snp) return;
    const DbSnpEntry e = a.snp[k];
    const int ori = a.ori[e.pos];
    const int ori7 = ori & 7;
    double lp[16];
    for (int i = 0; i < 16; ++i) lp[i] = a.log_prior[(ori7 << 4) + i];
    if (!e.indel) {
        const int t_base = ori & 3;
        for (int a1 = 0; a1 != 4; ++a1)
            for (int a2 = a1; a2 != 4; ++a2) {
                if (!(e.freq[a1] > 0 && e.freq[a2] > 0)) continue;
                double pr;
                if (!e.hapmap) {
                    if (a1 == a2 && a1 == t_base) pr = 1;
                    else if (a1 == t_base || a2 == t_base) pr = e.validated ? a.het_val : a.het_unval;
                    else if (a1 == a2) pr = e.validated ? a.althom_val : a.althom_unval;
                    else pr = e.validated ? a.het_val : a.het_unval;
                } else {
                    pr = GSNP_DMUL(GSNP_DMUL((a1 == a2 ? 1.0 : GSNP_DMUL(2.0, a.het_val)), e.freq[a1]), e.freq[a2]);
                }
                lp[(a1 << 2) | a2] = cr_log10(pr);
            }
    }
    for (int i = 0; i < 16; ++i) out[k * 16 + i] = lp[i];
    for (int t = 0; t < 12; ++t) out32[k * 12 + t] = t < 10 ? (float)lp[genotype_of(t)] : 0.f;
}

cudaError_t launch_snp_log_prior(const CallArgs& a, double* out, float* out32, cudaStream_t stream) {
    if (a.n_snp == 0) return cudaSuccess;
    snp_log_prior_kernel<<<(unsigned)((a.n_snp + 127) / 128), 128, 0, stream>>>(a, out, out32);
    return cudaGetLastError();
}

/* the short form's tables, once per table load */
__global__ void lean_tables_kernel(const double* lik64, const uint8_t* qadj, int tmax, int gmax, int qa_rows, int L,
                                   const int8_t* gap, uint32_t* lean_q, float4* lean4, double2* lean2d) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = first; i < kLeanQ; i += step) lean_q[i] = lean_q_entry(qadj, tmax, gmax, L, gap, i);
    for (int64_t i = first; i < lean4_rows(qa_rows, L); i += step) {
        float v[4];
        lean4_row(lik64, qa_rows, L, i, v);
        lean4[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
    for (int64_t i = first; i < lean2d_rows(qa_rows, L); i += step) {
        double v[2];
        lean2d_row(lik64, qa_rows, L, i, v);
        lean2d[i] = make_double2(v[0], v[1]);
    }
}

cudaError_t launch_lean_tables(const double* lik64, const uint8_t* qadj, int tmax, int gmax, int qa_rows, int L,
                               const int8_t* gap, uint32_t* lean_q, float* lean4, double* lean2d, cudaStream_t stream) {
    lean_tables_kernel<<<256, 256, 0, stream>>>(lik64, qadj, tmax, gmax, qa_rows, L, gap, lean_q,
                                                reinterpret_cast<float4*>(lean4), reinterpret_cast<double2*>(lean2d));
    return cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* the FP64 calling kernel                                                   */
/* ------------------------------------------------------------------------ */

/* A site of a tile in the short form that needs all ten genotypes (its best is
 * not (maj, maj), or the bounds do not name the second): the sums in the
 * reference's order over its walked column, then the general posterior.  Out of
 * line: about one site in a thousand comes here.  The column becomes record
 * words, which the rank-sum test reads. */
static __device__ __noinline__ void lean_general64(const CallArgs& a, int64_t site, uint8_t ori, int32_t snp_row,
                                                   LeanPile pile, uint32_t cu4, uint64_t qs4, uint32_t* recs) {
    LeanSums z;
    z.cu4 = cu4;
    z.qs4 = qs4;
    const SitePileup p = lean_counts(pile, z);
    double s[10];
#pragma unroll
    for (int v = 0; v < 10; ++v) s[v] = 0.0;
    for (int i = 0; i < pile.num; ++i) {
        const uint32_t w = recs[i * kTile];
        const double2* row = reinterpret_cast<const double2*>(
            a.lik64 + ((size_t)lean_qa(w) * a.L + ((w >> 16) & 0xffu)) * 40 + (w >> 30) * 10);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            const double2 x = __ldg(row + v);
            s[2 * v] = GSNP_DADD(s[2 * v], x.x);
            s[2 * v + 1] = GSNP_DADD(s[2 * v + 1], x.y);
        }
        recs[i * kTile] = lean_to_record(w);
    }
    double tl[16], lp[16];
#pragma unroll
    for (int g = 0; g < 16; ++g) tl[g] = 0.0;
#pragma unroll
    for (int v = 0; v < 10; ++v) tl[genotype_of(v)] = s[v];
    load_log_prior(a, snp_row, ori, lp);
    auto nq = [&](int b) { return neighbour_qsum(a, site, b); };
    SiteCall call;
    site_posterior<true>(a, ori, p, tl, nullptr, lp, recs, kTile, nq, &call);
    a.out[site] = call;
}

/* A tile in the short form (lean.cuh) with FP64 sums; every lane of the warp
 * calls it.  Nothing is written when lean_pileup leaves it.
 *
 * The FP64 pipe bounds the FP64 form (an FP64 instruction of a warp takes 16
 * cycles of the SM's pipe): the short form adds two terms a record instead of
 * ten, those of the best genotype and of the second, which FP32 sums with
 * their bounds name beforehand on the idle FP32 pipes.  c1, 4 Mbp: 3.2 ms in
 * the general form, 1.73 with four FP64 sums (73% of the FP64 pipe), 1.35 with
 * two (44%). */
template <int SLOTS>
__device__ __forceinline__ LeanTook lean_tile64(const CallArgs& a, int64_t tile, int64_t r_lo, int64_t r_hi, uint8_t wflags,
                                            uint32_t* recs_all, uint32_t* scratch) {
    const int t = threadIdx.x & 31;
    const int64_t s0 = tile * kTile, site = s0 + t;
    const bool active = site < a.chr_len;
    uint32_t* recs = recs_all + t;
    LeanPile pile;
    const LeanTook took = lean_columns<SLOTS>(a, s0, r_lo, r_hi, recs_all, scratch, &pile);
    if (took != kLeanTook) return took;
    const uint8_t ori = active ? __ldg(a.ori + site) : 0;
    const int32_t snp_row = tile_snp_row(a, tile, (ori & 8) != 0);
    LeanSums z;
    lean_walk<kTile, true>(a, recs, pile.num, ori & 3, &z);
    lean_zeros(pile, &z);
    if (active) {
        if (wflags & kWinKeepCounts) store_counts(a, site, lean_counts(pile, z));
        CallWords call;
        bool decided = true;
        if (pile.num == 0 && pile.extra4 == 0 && a.empty_valid[ori]) {
            /* no record and no count: the call depends on the site code only */
            const uint4* src = reinterpret_cast<const uint4*>(a.empty_calls + ori);
            call.a = __ldg(src);
            call.b = __ldg(src + 1);
            call.b.x = pile.depth;
            call.b.y = pile.repeat;
        } else {
            decided = lean_posterior64<kTile>(a, snp_row, ori, pile, z, recs, &call);
        }
        if (decided) {
            uint4* dst = reinterpret_cast<uint4*>(a.out + site);
            dst[0] = call.a;
            dst[1] = call.b;
        } else {
            lean_general64(a, site, ori, snp_row, pile, z.cu4, z.qs4, recs);
        }
    }
    return kLeanTook;
}

/* One tile of the FP64 kernel; every lane of the warp calls it. */
template <int SLOTS>
__device__ __forceinline__ void fp64_tile(const CallArgs& a, int32_t entry, uint32_t* recs_all, uint32_t* seen_all) {
    const int t = threadIdx.x;
    const int64_t tile = entry & ~kTileGeneral, s0 = tile * kTile;
    const int win = (int)(s0 / kWin);
    const uint8_t wflags = a.win_flags[win];
    const int64_t r_lo = a.warp_rng[tile * 2];
    const int64_t r_hi = a.warp_rng[tile * 2 + 1];
    if constexpr (SLOTS <= kLeanG) {
        if (a.lean_q && !(entry & kTileGeneral) && !(wflags & (kWinKeepLik | kWinExternalLik)) &&
            lean_tile64<lean_slots(SLOTS)>(a, tile, r_lo, r_hi, wflags, recs_all,
                                           recs_all + lean_slots(SLOTS) * kTile) == kLeanTook)
            return;
        __syncwarp();
    }
    const int64_t site = s0 + t;
    const bool active = site < a.chr_len;
    const uint8_t ori = active ? __ldg(a.ori + site) : 0;
    const int32_t snp_row = tile_snp_row(a, tile, (ori & 8) != 0);
    const SitePileup p = warp_pileup<SLOTS>(a, r_lo, r_hi, site, active, recs_all + t).unpack();
    if (!active) return;
    uint32_t* recs = recs_all + t;
    uint32_t* seen = seen_all + t;
    sort_column<SLOTS>(recs, p.num);

    double tl[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) tl[i] = 0.0;
    if (wflags & kWinExternalLik) {
        const int src = a.win_lik_src[win];
        if (src >= 0) {
            const double* srcp = a.lik_keep + ((int64_t)src * kWin + (site - (int64_t)win * kWin)) * 10;
#pragma unroll
            for (int i = 0; i < 10; ++i) tl[genotype_of(i)] = srcp[i];
        }
    } else {
        likelihood_fp64<kPcrBits(SLOTS, false)>(a, recs, seen, kTile, p.num, tl);
        if (wflags & kWinKeepLik) {
            double* dst = a.lik_keep + site * 10;
#pragma unroll
            for (int i = 0; i < 10; ++i) dst[i] = tl[genotype_of(i)];
        }
    }
    if (wflags & kWinKeepCounts) store_counts(a, site, p);

    double lp[16];
    load_log_prior(a, snp_row, ori, lp);
    auto nq = [&](int b) { return neighbour_qsum(a, site, b); };
    SiteCall call;
    site_posterior<true>(a, ori, p, tl, nullptr, lp, recs, kTile, nq, &call);
    a.out[site] = call;
}

/* The tiles of one depth bin: tiles[blockIdx.x] with count == nullptr (one
 * CTA per tile), else the first *count tiles of the list, handed out by
 * for_each_listed (a grid sized to the resident CTAs, whatever the count the
 * device holds). */
template <int SLOTS>
__global__ void __launch_bounds__(kTile, kFp64CtasPerSm)
    call_tiles_kernel(const __grid_constant__ CallArgs a, const int32_t* __restrict__ tiles,
                      const int* __restrict__ count, int* next) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t* recs_all = reinterpret_cast<uint32_t*>(smem);                   /* [SLOTS][kTile] */
    uint32_t* seen_all = reinterpret_cast<uint32_t*>(smem) + SLOTS * kTile;    /* [nw][kTile] */
    if (!count) {
        fp64_tile<SLOTS>(a, tiles[blockIdx.x], recs_all, seen_all);
        return;
    }
    for_each_listed(count, next, [&](int i) { fp64_tile<SLOTS>(a, tiles[i], recs_all, seen_all); });
}

/* The persistent kernel of the FP64 form: call_stream_kernel's hand-out of
 * tiles in genome order, each in the short form; the tiles it cannot take go to
 * the leftover list for the binned kernels. */
template <int SLOTS>
__global__ void __launch_bounds__(32 * kStreamWarps, kStream64Warps / kStreamWarps)
    call_stream64_kernel(const __grid_constant__ CallArgs a, StreamQueue q) {
    extern __shared__ __align__(16) uint8_t smem[];
    const size_t warp_bytes = (lean_smem_bytes(SLOTS, a.L) + 15) & ~(size_t)15;
    uint32_t* recs_all = reinterpret_cast<uint32_t*>(smem + (threadIdx.x >> 5) * warp_bytes);
    const int t = threadIdx.x & 31;
    const int64_t n = q.t_end - q.t_begin;
    for (;;) {
        unsigned long long first = 0;
        if (t == 0) first = atomicAdd(q.next, (unsigned long long)kStreamChunk);
        first = __shfl_sync(kFull, first, 0);
        if ((int64_t)first >= n) return;
        const int64_t end = min((int64_t)first + (int64_t)kStreamChunk, n);
        for (int64_t i = (int64_t)first; i < end; ++i) {
            const int64_t tile = q.t_begin + i;
            const uint8_t wflags = a.win_flags[(int)(tile * kTile / kWin)];
            const LeanTook took =
                wflags & (kWinKeepLik | kWinExternalLik)
                    ? kLeanNever
                    : lean_tile64<SLOTS>(a, tile, a.tile_rng[tile * 2], a.tile_rng[tile * 2 + 1], wflags, recs_all,
                                         recs_all + SLOTS * kTile);
            if (took != kLeanTook && t == 0)
                q.leftover[atomicAdd(q.n_leftover, 1)] = (int32_t)tile | (took == kLeanNever ? kTileGeneral : 0);
            __syncwarp();
        }
    }
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */

thread_local bool g_launch_attributes = true;
void set_launch_attributes(bool on) { g_launch_attributes = on; }

static size_t fp64_smem_bytes(int slots, int L) {
    /* records [slots][kTile], then the pcr state; the bins that try the short
     * form first: its records and scratch in the same place */
    const size_t general = ((size_t)slots * kTile + (size_t)pcr_smem_words(slots, L, false)) * 4;
    const size_t lean = slots <= kLeanG ? lean_smem_bytes(slots, L) : 0;
    return general > lean ? general : lean;
}

/* Classify tiles [t_begin, t_end) (with a list, list[t_begin, t_end); with
 * d_count, list[0, *d_count) read on the device, by a fixed grid of `grid`
 * CTAs) into the depth bins from min_bin, marked tiles from general_bin on;
 * d_bin_count's kBinCountInts ints are zero. */
cudaError_t launch_classify(const CallArgs& a, int pass, int min_bin, int general_bin, int64_t t_begin, int64_t t_end,
                            int* d_bin_count, int32_t* d_bin_tiles, cudaStream_t stream, const int32_t* list,
                            const int* d_count, int grid) {
    const unsigned blocks =
        d_count ? (unsigned)grid : (unsigned)((t_end - t_begin + kClassifyTiles - 1) / kClassifyTiles);
    if (blocks == 0) return cudaSuccess;
    classify_tiles_kernel<<<blocks, kClassifyThreads, 0, stream>>>(a, pass, min_bin, general_bin, t_begin, t_end,
                                                                   d_bin_count, d_bin_tiles, list, d_count);
    return cudaGetLastError();
}

template <int SLOTS>
static cudaError_t stream64_attr(int L, int carveout, int* ctas_per_sm) {
    const int smem = (int)(kStreamWarps * ((lean_smem_bytes(SLOTS, L) + 15) & ~(size_t)15));
    cudaError_t e = cudaFuncSetAttribute(call_stream64_kernel<SLOTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess && carveout > 0 &&
        cudaFuncSetAttribute(call_stream64_kernel<SLOTS>, cudaFuncAttributePreferredSharedMemoryCarveout, carveout) !=
            cudaSuccess)
        (void)cudaGetLastError();
    if (e == cudaSuccess && ctas_per_sm)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, call_stream64_kernel<SLOTS>, 32 * kStreamWarps, smem);
    return e;
}

/* resident CTAs on one SM of the persistent FP64 kernel with 48 or 64 record
 * slots */
int stream64_ctas_per_sm(int slots, int L, int carveout) {
    int n = 0;
    const cudaError_t e = slots <= 48 ? stream64_attr<48>(L, carveout, &n) : stream64_attr<64>(L, carveout, &n);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

template <int SLOTS>
static cudaError_t launch_stream64_one(const CallArgs& a, const StreamQueue& q, int ctas, int carveout,
                                       cudaStream_t stream) {
    cudaError_t e = g_launch_attributes ? stream64_attr<SLOTS>(a.L, carveout, nullptr) : cudaSuccess;
    if (e != cudaSuccess) return e;
    const size_t smem = kStreamWarps * ((lean_smem_bytes(SLOTS, a.L) + 15) & ~(size_t)15);
    call_stream64_kernel<SLOTS><<<ctas, 32 * kStreamWarps, smem, stream>>>(a, q);
    return cudaGetLastError();
}

/* The persistent FP64 kernel over q's tiles (as launch_stream); a.lean_q must
 * be set. */
cudaError_t launch_stream64(const CallArgs& a, const StreamQueue& q, int slots, int ctas, int carveout,
                            cudaStream_t stream) {
    if (q.t_end <= q.t_begin) return cudaSuccess;
    return slots <= 48 ? launch_stream64_one<48>(a, q, ctas, carveout, stream)
                       : launch_stream64_one<64>(a, q, ctas, carveout, stream);
}

/* set the FP64 bin kernel's shared-memory size and carveout (percent; 0
 * leaves the default); with ctas_per_sm, its resident CTAs on one SM */
template <int SLOTS>
static cudaError_t bin_attr(int L, int carveout, int* ctas_per_sm) {
    const int smem = (int)fp64_smem_bytes(SLOTS, L);
    const void* fn = reinterpret_cast<const void*>(call_tiles_kernel<SLOTS>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    /* the carveout is a hint: a refusal only costs speed, and its error is
     * cleared so that it is not taken for the launch's */
    if (carveout > 0 && cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, carveout) != cudaSuccess)
        (void)cudaGetLastError();
    if (ctas_per_sm) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, kTile, smem);
    return cudaSuccess;
}

template <int SLOTS>
static cudaError_t launch_one(const CallArgs& a, const int32_t* tiles, const BinLaunch& bl, cudaStream_t stream) {
    cudaError_t e = g_launch_attributes ? bin_attr<SLOTS>(a.L, bl.carveout, nullptr) : cudaSuccess;
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned)(bl.d_count ? bl.grid : bl.count);
    if (grid == 0) return cudaSuccess;
    call_tiles_kernel<SLOTS><<<grid, kTile, fp64_smem_bytes(SLOTS, a.L), stream>>>(a, tiles, bl.d_count, bl.d_next);
    return cudaGetLastError();
}

/* Launch the FP64 or the fast calling kernel over the tiles of depth bin
 * `bin` (see BinLaunch). */
cudaError_t launch_bin(const CallArgs& a, int kind, int bin, const int32_t* tiles, const BinLaunch& bl,
                       cudaStream_t stream) {
    if (kind == kKindFast) return launch_fast_bin(a, bin, tiles, bl, stream);
    switch (bin) {
        case 0: return launch_one<32>(a, tiles, bl, stream);
        case 1: return launch_one<40>(a, tiles, bl, stream);
        case 2: return launch_one<48>(a, tiles, bl, stream);
        case 3: return launch_one<64>(a, tiles, bl, stream);
        case 4: return launch_one<96>(a, tiles, bl, stream);
        case 5: return launch_one<128>(a, tiles, bl, stream);
        default: return launch_deep64(a, tiles, bl, stream);
    }
}

/* resident CTAs on one SM of bin `bin` of kernel `kind` at a carveout */
int bin_ctas_per_sm(int kind, int bin, int L, int carveout) {
    int n = 0;
    cudaError_t e;
    if (kind == kKindFast) e = fast_bin_attr(bin, L, carveout, &n);
    else switch (bin) {
        case 0: e = bin_attr<32>(L, carveout, &n); break;
        case 1: e = bin_attr<40>(L, carveout, &n); break;
        case 2: e = bin_attr<48>(L, carveout, &n); break;
        case 3: e = bin_attr<64>(L, carveout, &n); break;
        case 4: e = bin_attr<96>(L, carveout, &n); break;
        case 5: e = bin_attr<128>(L, carveout, &n); break;
        default: e = deep64_attr(&n); break;
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

int bin_slots(int bin) { return kSlots[bin]; }

}  // namespace gsnp
