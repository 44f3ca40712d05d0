/*
 * deep.cuh - one site by one warp: the pileup of its column, the sort, the
 * dependency walk and the rank sums, for the columns of hundreds of records
 * (calling_fast.cu in FP32, calling_deep64.cu in FP64) and the deferred sites
 * (deferred.cu).
 */
#ifndef GSNP_DEEP_CUH
#define GSNP_DEEP_CUH

#include "calling.cuh"
#include "site_math.cuh"
#include "tile.cuh"

namespace gsnp {

constexpr int kDeepCap = 256;              /* records of a column (at most 255), a power of two */
constexpr int kDeepKeys = 4 * 2 * 256;     /* (base, strand, cycle) keys */

/* neighbouring sites of a tile that a warp takes together */
constexpr int kDeepBatch = 8;
constexpr int kDeepBatches = kTile / kDeepBatch;
constexpr int kDeepAhead = 2;

/* Sites a warp takes at a time of n tiles over `warps` warps: a power of two,
 * halved from kDeepBatch while there are not two rounds of work - a segment
 * with a few hundred deep tiles would otherwise take eight sites' latency. */
__device__ __forceinline__ int deep_sites(int n, int warps) {
    int sites = kDeepBatch;
    while (sites > 1 && (int64_t)n * (kTile / sites) < 2 * (int64_t)warps) sites >>= 1;
    return sites;
}

/* What the reads [r_lo, r_hi) are to the kDeepBatch sites from s0 on, lane j < kDeepBatch
 * site s0 + j: how many cover it, their hits' sum, and how many of the first
 * ones end before it whatever their length (they start at site - L or before).
 * One pass over the reads' starts and lengths for all the sites: a read that
 * covers them all is counted by ballot; the others add where they begin and
 * take away where they end, in shared memory.  scratch: 2 (kDeepBatch + 1)
 * words. */
struct DeepSpan {
    uint32_t depth, repeat;
    int skip;
};
__device__ __forceinline__ DeepSpan deep_spans(const CallArgs& a, int64_t r_lo, int64_t r_hi, int64_t s0,
                                               uint32_t* scratch) {
    const int lane = threadIdx.x & 31;
    uint32_t* const dep = scratch;
    uint32_t* const rep = scratch + kDeepBatch + 1;
    if (lane < 2 * (kDeepBatch + 1)) scratch[lane] = 0u;
    __syncwarp();
    uint32_t whole_n = 0, whole_rep = 0;
    DeepSpan out = {0u, 0u, 0};
    for (int64_t rb = r_lo; rb < r_hi; rb += 32 * kDeepAhead) {
        int32_t st[kDeepAhead];
        uint32_t lh[kDeepAhead];
#pragma unroll
        for (int u = 0; u < kDeepAhead; ++u) {
            const int64_t r = rb + 32 * u + lane;
            st[u] = r < r_hi ? __ldg(a.pos + r) : 0;
            lh[u] = r < r_hi ? (uint32_t)__ldg(a.lenhit + r) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kDeepAhead; ++u) {
            const bool in = rb + 32 * u + lane < r_hi;
            const int t = (int)(st[u] - s0);
            const int from = max(t, 0), to = min(t + (int)(lh[u] >> 16), kDeepBatch);
            const uint32_t hit = lh[u] & 0xffffu;
            const bool some = in && from < to, whole = some && to - from == kDeepBatch;
            whole_n += (uint32_t)__popc(__ballot_sync(kFull, whole));
            whole_rep += whole ? hit : 0u;
            if (some && !whole) {
                atomicAdd(dep + from, 1u);
                atomicAdd(rep + from, hit);
                atomicSub(dep + to, 1u);
                atomicSub(rep + to, hit);
            }
            const int past = in ? t + a.L : kDeepBatch;   /* the first site out of reach */
            if (__any_sync(kFull, past < kDeepBatch))
#pragma unroll
                for (int j = 0; j < kDeepBatch; ++j) {
                    const int n = __popc(__ballot_sync(kFull, past <= j));
                    if (lane == j) out.skip += n;
                }
        }
    }
    whole_rep = __reduce_add_sync(kFull, whole_rep);
    __syncwarp();
    out.depth = whole_n;
    out.repeat = whole_rep;
#pragma unroll
    for (int j = 0; j < kDeepBatch; ++j) {
        if (j > lane) continue;
        out.depth += dep[j];
        out.repeat += rep[j];
    }
    return out;
}

/* The pileup of one site by its warp (kernel/update_kernel.cu:260-325, as
 * PileupAcc::take): the reads [r_lo, r_hi) 32 at a time, in order, whose
 * depth and repeat the caller has (deep_spans).  A covering read that is not
 * N and reaches q_min is taken while the site has fewer than 255 unique
 * records, and a unique one (hit 1) adds a record.  Whether the cap still
 * admits a read depends only on the unique valid reads before it, which a
 * ballot gives, so the 32 reads of a step are decided together with the
 * reference's result.  The scan ends once the cap is reached, or at the first
 * step whose reads all start past the site.
 *
 * Its loads run ahead of the decisions (each step's base and quality load
 * depends on the read's start): an iteration loads the starts and lengths of
 * its kDeepAhead steps' reads in the iteration before, and their bases,
 * qualities and strands all at its start.  The steps are then decided in
 * order, as above. */
__device__ __forceinline__ SitePileup deep_pileup(const CallArgs& a, int64_t r_lo, int64_t r_hi, int64_t site,
                                                  uint32_t depth, uint32_t repeat, uint32_t* recs) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int L = a.L;
    int num = 0;   /* records so far */
    /* Counts by base per lane, added over the warp after the scan: records in
     * bytes (their total is at most 255), accepted reads and quality sums (at
     * most 255 x 255) in half words.  Counting each step's by ballots takes a
     * popc a base, which the SM issues at a quarter of the rate. */
    uint32_t cu_l = 0, ca_l[2] = {0u, 0u}, qs_l[2] = {0u, 0u};
    int32_t nst[kDeepAhead];
    uint32_t nlh[kDeepAhead];
#pragma unroll
    for (int u = 0; u < kDeepAhead; ++u) {
        const int64_t r = r_lo + 32 * u + lane;
        nst[u] = r < r_hi ? __ldg(a.pos + r) : 0;
        nlh[u] = r < r_hi ? (uint32_t)__ldg(a.lenhit + r) : 0u;
    }
    for (int64_t rb = r_lo; rb < r_hi && num < 0xFF; rb += 32 * kDeepAhead) {
        int coord[kDeepAhead];
        uint32_t lh[kDeepAhead], bq[kDeepAhead];
        bool cov[kDeepAhead], minus[kDeepAhead];
#pragma unroll
        for (int u = 0; u < kDeepAhead; ++u) {
            const int64_t r = rb + 32 * u + lane;
            const bool in = r < r_hi;
            coord[u] = in ? (int)(site - nst[u]) : -1;
            lh[u] = nlh[u];
            cov[u] = in && coord[u] >= 0 && coord[u] < (int)(lh[u] >> 16);
            bq[u] = 0;
            minus[u] = false;
            if (cov[u]) {
                bq[u] = __ldg(a.bq + r * L + coord[u]);
                minus[u] = __ldg(a.strand + r) != '+';
            }
            const int64_t rn = r + 32 * kDeepAhead;
            nst[u] = rn < r_hi ? __ldg(a.pos + rn) : 0;
            nlh[u] = rn < r_hi ? (uint32_t)__ldg(a.lenhit + rn) : 0u;
        }
        bool past = false;
#pragma unroll
        for (int u = 0; u < kDeepAhead; ++u) {
            if (__all_sync(kFull, coord[u] < 0)) {   /* every read from here on starts past the site */
                past = true;
                break;
            }
            if (num >= 0xFF) break;
            const bool valid = cov[u] && elem_valid(bq[u]);
            const int bi = elem_base(bq[u]), q = elem_q(bq[u]);
            const bool uni = valid && (lh[u] & 0xffffu) == 1;
            const unsigned mu = __ballot_sync(kFull, uni);
            const int uni_before = num + __popc(mu & lt);
            const bool acc = valid && uni_before < 0xFF;
            const bool rec = acc && uni;
            if (rec) {
                const uint32_t cv =
                    minus[u] ? (uint32_t)((int)(lh[u] >> 16) - 1 - coord[u]) : (uint32_t)coord[u];
                recs[uni_before] = make_record_of((uint32_t)bi, q, cv, (uint32_t)minus[u]);
            }
            num = min(0xFF, num + __popc(mu));   /* the unique valid ones below the cap */
            const uint32_t half = 16u * (bi & 1);
            cu_l += rec ? 1u << (8 * bi) : 0u;
            ca_l[0] += acc && bi < 2 ? 1u << half : 0u;
            ca_l[1] += acc && bi >= 2 ? 1u << half : 0u;
            qs_l[0] += rec && bi < 2 ? (uint32_t)q << half : 0u;
            qs_l[1] += rec && bi >= 2 ? (uint32_t)q << half : 0u;
        }
        if (past) break;
    }
    SitePileup p;
    p.depth = depth;
    p.repeat = repeat;
    p.dep_uni = num;
    p.num = num;
    cu_l = __reduce_add_sync(kFull, cu_l);
#pragma unroll
    for (int b = 0; b < 4; ++b) p.cu[b] = (int)((cu_l >> (8 * b)) & 0xffu);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t ca = __reduce_add_sync(kFull, ca_l[h]), qs = __reduce_add_sync(kFull, qs_l[h]);
        p.ca[2 * h] = ca & 0xffffu;
        p.ca[2 * h + 1] = ca >> 16;
        p.qs[2 * h] = (int)(qs & 0xffffu);
        p.qs[2 * h + 1] = (int)(qs >> 16);
    }
    return p;
}

/* Ascending bitonic sort of v[0, n), n <= kDeepCap = 256, by the lanes of a
 * warp in registers: lane l holds elements 8l .. 8l+7 (padded with
 * 0xFFFFFFFF, which no record word equals).  The network's stages of
 * distance j < 8 are compare-exchanges within a lane; those of distance
 * j >= 8 pair lane l with lane l ^ (j / 8), which keeps the smaller or the
 * larger of each of its eight elements.  Every loop bound is a constant, so
 * the 36 stages unroll into straight code with no index arithmetic and no
 * shared-memory traffic between them. */
__device__ __forceinline__ void deep_sort(uint32_t* v, int n) {
    static_assert(kDeepCap == 256, "eight elements a lane");
    const int lane = threadIdx.x & 31;
    uint32_t x[8];
    const uint4 lo4 = reinterpret_cast<const uint4*>(v)[lane * 2];
    const uint4 hi4 = reinterpret_cast<const uint4*>(v)[lane * 2 + 1];
    x[0] = lo4.x, x[1] = lo4.y, x[2] = lo4.z, x[3] = lo4.w;
    x[4] = hi4.x, x[5] = hi4.y, x[6] = hi4.z, x[7] = hi4.w;
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if (lane * 8 + e >= n) x[e] = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 2; k <= 256; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 8) {
                const int d = j >> 3;
                const bool keep_min = (((lane * 8) & k) == 0) == ((lane & d) == 0);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t y = __shfl_xor_sync(kFull, x[e], d);
                    x[e] = keep_min ? min(x[e], y) : max(x[e], y);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (e & j) continue;
                    const int f = e | j;
                    const bool asc = ((lane * 8 + e) & k) == 0;
                    const uint32_t a = min(x[e], x[f]), b = max(x[e], x[f]);
                    x[e] = asc ? a : b;
                    x[f] = asc ? b : a;
                }
            }
        }
    }
    __syncwarp();
    reinterpret_cast<uint4*>(v)[lane * 2] = make_uint4(x[0], x[1], x[2], x[3]);
    reinterpret_cast<uint4*>(v)[lane * 2 + 1] = make_uint4(x[4], x[5], x[6], x[7]);
    __syncwarp();
}

/* The dependency walk of a sorted column by its warp, 32 records a step,
 * record c0 + lane on that lane; cnt is kDeepKeys bytes, 16-byte aligned.  The
 * walk's two counts (walk_records) come from the whole step at once:
 *   - tmp, the earlier records of the same (base, strand, cycle) key: the
 *     key's counter from the steps before plus the lower lanes with that key
 *     (match-any); the highest of them then stores the new count;
 *   - gdc, the first occurrences of a key (tmp = 0) so far in the record's
 *     base group, less one: a ballot prefix, from the lane where the base
 *     group starts, or carried over from the step before.
 * f(c0, valid, adjusted quality, cycle, base) is called by every lane for each
 * step. */
template <class F>
__device__ __forceinline__ void deep_walk(const CallArgs& a, const uint32_t* recs, uint8_t* cnt, int num, F&& f) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u, le = (lt << 1) | 1u;
    for (int i = lane; i < kDeepKeys / 16; i += 32) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    int carry_firsts = 0, carry_base = -1;
    for (int c0 = 0; c0 < num; c0 += 32) {
        const bool valid = c0 + lane < num;
        const uint32_t w = valid ? recs[c0 + lane] : 0u;
        const int o = rec_base(w), coord = rec_coord(w);
        const int key = valid ? (o << 9) | (rec_strand(w) << 8) | coord : kDeepKeys + lane;
        const unsigned peers = __match_any_sync(kFull, key);
        const int seen = valid ? (int)cnt[key] : 0;
        __syncwarp();
        const int tmp = seen + __popc(peers & lt);
        if (valid && (peers >> lane) == 1u) cnt[key] = (uint8_t)(seen + __popc(peers));
        __syncwarp();
        const int prev_o = __shfl_up_sync(kFull, o, 1);
        const bool brk = valid && o != (lane == 0 ? carry_base : prev_o);
        const unsigned bm = __ballot_sync(kFull, brk) & le;
        const unsigned fm = __ballot_sync(kFull, valid && tmp == 0) & le;
        const int firsts = bm ? __popc(fm & ~((1u << (31 - __clz(bm))) - 1u)) : carry_firsts + __popc(fm);
        carry_firsts = __shfl_sync(kFull, firsts, 31);
        carry_base = __shfl_sync(kFull, o, 31);
        int qa = 0;
        if (valid) {
            const int gdc = firsts - 1, t1 = tmp + 1;
            qa = (t1 < a.tmax && gdc < a.gmax) ? (int)__ldg(a.qadj + ((size_t)t1 * a.gmax + gdc) * 65 + rec_q(w)) : 1;
        }
        f(c0, valid, qa, coord, o);
    }
}

/* Twice the rank sums of genotype g's two alleles over the site's records
 * (rank_test's Ta and Tb are half-integers far below 2^52, so its FP64 sums are
 * exact and any order gives them): a histogram by quality, and the rank of a
 * quality from the counts below it. */
__device__ __forceinline__ void warp_ranks(const CallArgs& a, const uint32_t* recs, int num, int g, int32_t (*hist)[66],
                                           int32_t* rank2) {
    const int lane = threadIdx.x & 31;
    const int ia = g & 3, ib = (g >> 2) & 3;
    for (int i = lane; i < 132; i += 32) hist[0][i] = 0;
    __syncwarp();
    for (int i = lane; i < num; i += 32) {
        const uint32_t w = recs[i];
        const int o = rec_base(w);
        if (o == ia) atomicAdd(&hist[0][rec_q(w)], 1);
        else if (o == ib) atomicAdd(&hist[1][rec_q(w)], 1);
    }
    __syncwarp();
    /* qualities above q_max - q_min + 1 keep rank 0 as in the reference */
    const int top = a.q_max_min + 1 < 64 ? a.q_max_min + 1 : 64;
    int below = 0, ta = 0, tb = 0;
    for (int q0 = 0; q0 <= 64; q0 += 32) {
        const int q = q0 + lane;
        const int ca = q <= top ? hist[0][q] : 0, cb = q <= top ? hist[1][q] : 0;
        int before = ca + cb;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(kFull, before, d);
            if (lane >= d) before += y;
        }
        const int total = __shfl_sync(kFull, before, 31);
        const int ra = 2 * (below + before - ca - cb) + 1 + ca + cb;   /* twice the average rank */
        ta += ra * ca;
        tb += ra * cb;
        below += total;
    }
    ta = __reduce_add_sync(kFull, ta);
    tb = __reduce_add_sync(kFull, tb);
    if (lane == 0) {
        rank2[0] = ta;
        rank2[1] = tb;
    }
    __syncwarp();
}

}  // namespace gsnp

#endif
