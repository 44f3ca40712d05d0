/*
 * deferred.cu - the FP64 pass over the sites the FP32 kernels deferred: their
 * FP32 sums again with the double-precision bound checks, the FP64 sums where
 * those fail, the rank-sum test (calling.cu).
 *
 * A deferred site is a few dozen records of serial work, and there are few of
 * them (about one in a thousand at 30x), so the pass is bound by latency: of its
 * loads, and of its code, which is fetched cold.  A warp takes its sites one
 * after another for what is parallel inside a site - the dependency walk a
 * record per lane, the sums a genotype per lane, the quality histogram of the
 * rank-sum test - and then all of them at once, a site per lane, for the FP64
 * posterior.  (GB300 issues an FP64 instruction of a warp over 16 cycles
 * however many lanes it has, so a posterior per warp would cost 32 times as
 * much of the pipe.)  With few sites every warp takes one.  A thread per site, with
 * its walk in local memory and 290 KB of inlined code, took 310-380 us at 33
 * sites and at 20,000 alike, and 1.1 ms where the columns are deep (c2); this
 * form takes 43 us at 36 sites, 105 us at 5,000 (4 Mbp of c1), 260 us at 12,000
 * of c2.
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "calling.cuh"
#include "deep.cuh"
#include "site_math.cuh"
#include "tile.cuh"

namespace gsnp {

namespace {

constexpr int kDefWarps = 4;     /* warps of a CTA, each by itself */
constexpr int kDefBatch = 16;    /* most sites a warp holds at a time */

/* a warp's shared memory */
struct DefWarp {
    uint8_t cnt[kDeepKeys];             /* occurrences by (base, strand, cycle) key */
    int32_t hist[2][66];               /* records by quality of the candidate's two alleles */
    float tl32[kDefBatch][10];         /* FP32 sums by table column */
    double tl64[kDefBatch][10];        /* FP64 sums, where they are wanted */
    int32_t rank2[kDefBatch][2];       /* twice the rank sums of the candidate's alleles */
    int32_t cand[kDefBatch];           /* best genotype of the FP32 values, -1: no rank sums */
};

/* The dependency walk and the sums of a sorted column by a warp: the walk's 32
 * records a step, of which lane v < 10 adds column v in order.  T = float:
 * groups of four added pairwise and compensated, the values of
 * likelihood_fp32; T = double: the reference's order.  Returns column `lane`'s
 * sum on lanes 0-9. */
template <class T>
__device__ __forceinline__ T deferred_sum(const CallArgs& a, const uint32_t* recs, int num, uint8_t* cnt) {
    constexpr bool kSingle = sizeof(T) == 4;
    const int lane = threadIdx.x & 31;
    /* where column `lane` of a row lies */
    const int col = lane < 10 ? lane : 0;
    const T* base;
    int stride;
    if constexpr (kSingle) {
        base = col < 8 ? a.lik32 + col : a.lik32b + (col - 8);
        stride = col < 8 ? 8 : 2;
    } else {
        base = a.lik64 + col;
        stride = 10;
    }
    T s = 0, c = 0;
    deep_walk(a, recs, cnt, num, [&](int c0, bool valid, int qa, int coord, int o) {
        const int row = valid ? (qa * a.L + coord) * 4 + o : 0;
        const int n = num - c0 < 32 ? num - c0 : 32;
        for (int j = 0; j < n; j += 8) {
            T x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = __shfl_sync(kFull, row, j + u);
                x[u] = 0;
                if (j + u < n) x[u] = __ldg(base + (size_t)r * stride);
            }
            if constexpr (kSingle) {
#pragma unroll
                for (int u = 0; u < 8; u += 4)
                    if (j + u < n) {
                        const float g = __fadd_rn(__fadd_rn(x[u], x[u + 1]), __fadd_rn(x[u + 2], x[u + 3]));
                        const float y = __fsub_rn(g, c), t = __fadd_rn(s, y);
                        c = __fsub_rn(__fsub_rn(t, s), y);
                        s = t;
                    }
            } else {
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (j + u < n) s = GSNP_DADD(s, x[u]);
            }
        }
    });
    __syncwarp();
    return s;
}

/* The posterior of deferred site d by one lane: from its FP32 sums with their
 * bounds (t32), or from its FP64 sums (t64). */
__device__ __noinline__ bool deferred_posterior(const CallArgs& a, const DeferredSite& d, const float* t32,
                                                const double* t64, int cand, const int32_t* rank2, SiteCall* call) {
    const int64_t site = d.site;
    SitePileup p;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        p.cu[b] = d.cu[b];
        p.qs[b] = d.qs[b];
        p.ca[b] = d.ca[b];
    }
    p.depth = d.depth;
    p.repeat = d.repeat;
    p.dep_uni = d.dep_uni;
    p.num = d.num;
    double tl[16], eps[16], lp[16];
    const double kk = GSNP_FP32_K(p.num);
    GSNP_ROLLED
    for (int g = 0; g < 16; ++g) tl[g] = eps[g] = 0.0;
    GSNP_ROLLED
    for (int i = 0; i < 10; ++i) {
        const int g = genotype_of(i);
        tl[g] = t64 ? t64[i] : (double)t32[i];
        eps[g] = isinf(tl[g]) ? 0.0 : fabs(tl[g]) * kk;
    }
    const uint8_t ori = __ldg(a.ori + site);
    load_log_prior(a, d.snp_row, ori, lp);
    auto nq = [&](int b) { return neighbour_qsum(a, site, b); };
    auto rank = [&](int g, bool* normal) -> double {
        const int ia = g & 3, ib = (g >> 2) & 3;
        if (g != cand) return rank_test(a.p_rank, a.q_max_min, a.dpool + d.rec_off, 1, p.num, p.cu, g, normal);
        if (ia == ib) return 1.0;
        if (p.cu[ia] == 0 || p.cu[ib] == 0) return 0.0;
        return rank_value(a.p_rank, p.cu[ia], p.cu[ib], 0.5 * (double)rank2[0], 0.5 * (double)rank2[1], normal);
    };
    return site_posterior_ranked<true>(a, ori, p, tl, t64 ? nullptr : eps, lp, rank, nq, call);
}

}  // namespace

/* n sites, or with d_n = a.dcount the sites the fast kernels requested.  A pool
 * that did not hold all of them has slots nobody wrote (a site whose records
 * found no room keeps its slot); the host reads the counts after the pass,
 * grows the pool and runs the whole pass again, so nothing is done here.  Sampled sites also get the FP64 sums for the
 * accuracy figure, and when the fast kernel had decided them its call is
 * compared with this one. */
__global__ void __launch_bounds__(32 * kDefWarps) deferred_sites_kernel(const __grid_constant__ CallArgs a, int64_t n,
                                                                        const unsigned long long* d_n) {
    __shared__ __align__(16) DefWarp warps[kDefWarps];
    DefWarp& sm = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    if (d_n) {
        n = (int64_t)d_n[0];
        if (n > a.dsite_cap || (int64_t)d_n[1] > a.dpool_cap) return;
    }
    const int64_t n_warps = (int64_t)gridDim.x * kDefWarps;
    const int64_t warp = (int64_t)blockIdx.x * kDefWarps + (threadIdx.x >> 5);
    const int batch = (int)min((int64_t)kDefBatch, max((int64_t)1, (n + n_warps - 1) / n_warps));
    for (int64_t first = warp * batch; first < n; first += n_warps * batch) {
        const int k = (int)min((int64_t)batch, n - first);
        /* the FP32 sums, and the rank sums of the genotype they favour */
        for (int j = 0; j < k; ++j) {
            const DeferredSite& d = a.dsites[first + j];
            const uint32_t* recs = a.dpool + d.rec_off;
            const int num = d.num;
            const float s = deferred_sum<float>(a, recs, num, sm.cnt);
            const uint8_t ori = __ldg(a.ori + d.site);
            const double* prior = (ori & 8) && a.refine ? a.snp_lp + (int64_t)d.snp_row * 16 : a.log_prior + ((ori & 7) << 4);
            const int g = genotype_of(lane < 10 ? lane : 0);
            const bool counts = lane < 10 && !(a.monoploid && (g >> 2) != (g & 3));
            float v = counts ? s + (float)__ldg(prior + g) : -INFINITY;
            int best = g;
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) {
                const float y = __shfl_xor_sync(kFull, v, off);
                const int yg = __shfl_xor_sync(kFull, best, off);
                if (y > v || (y == v && yg > best)) { v = y; best = yg; }
            }
            best = __shfl_sync(kFull, best, 0);
            if (lane < 10) sm.tl32[j][lane] = s;
            if (lane == 0) sm.cand[j] = best;
            if (a.rank_sum && (best >> 2) != (best & 3)) warp_ranks(a, recs, num, best, sm.hist, sm.rank2[j]);
        }
        __syncwarp();
        DeferredSite d;
        SiteCall call;
        bool want64 = false, done = true;
        if (lane < k) {
            d = a.dsites[first + lane];
            done = deferred_posterior(a, d, sm.tl32[lane], nullptr, sm.cand[lane], sm.rank2[lane], &call);
            want64 = !done || (d.flags & kCallSampled);
        }
        for (unsigned m = __ballot_sync(kFull, want64); m; m &= m - 1) {
            const int j = __ffs(m) - 1;
            const DeferredSite& dj = a.dsites[first + j];
            const double s = deferred_sum<double>(a, a.dpool + dj.rec_off, dj.num, sm.cnt);
            if (lane < 10) sm.tl64[j][lane] = s;
        }
        __syncwarp();
        if (lane < k) {
            if (d.flags & kCallSampled) {
                double m = 0.0;
                GSNP_ROLLED
                for (int i = 0; i < 10; ++i) m = fmax(m, fabs(sm.tl64[lane][i] - (double)sm.tl32[lane][i]));
                atomicMax(a.stats + 3, (unsigned long long)__double_as_longlong(m));
                atomicAdd(a.stats + 2, 1ull);
            }
            if (!done) {
                /* FP64 fixup: the FP32 likelihood is too close to a decision boundary */
                deferred_posterior(a, d, nullptr, sm.tl64[lane], sm.cand[lane], sm.rank2[lane], &call);
                call.flags |= kCallFixup;
                atomicAdd(a.stats + 1, 1ull);
            }
            if (d.flags & kCallPending) {
                atomicAdd(a.stats + 4, 1ull);
            } else if (!same_call(a.out[d.site], call)) {
                /* a sampled site the fast kernel decided differs from the FP64 call */
                atomicAdd(a.stats + 5, 1ull);
            }
            a.out[d.site] = call;
        }
        __syncwarp();
    }
}

/* The FP64 pass over n deferred sites, or with d_n (a.dcount) over those the
 * fast kernels requested (read on the device) with a grid of the resident CTAs. */
cudaError_t launch_deferred(const CallArgs& a, int64_t n, cudaStream_t stream, const unsigned long long* d_n,
                            int grid) {
    if (!d_n && n <= 0) return cudaSuccess;
    const unsigned blocks = d_n ? (unsigned)grid : (unsigned)std::min<int64_t>((n + kDefWarps - 1) / kDefWarps, grid);
    if (blocks == 0) return cudaSuccess;
    deferred_sites_kernel<<<blocks, 32 * kDefWarps, 0, stream>>>(a, n, d_n);
    return cudaGetLastError();
}

/* resident CTAs of the pass on one SM */
int deferred_ctas_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, deferred_sites_kernel, 32 * kDefWarps, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

}  // namespace gsnp
