/*
 * lean.cuh - the short form of a site's FP32 call, used for the tiles it can
 * prove (calling_fast.cu falls back to the general form for the others).
 * Host-compilable, so that its decisions are checked against the FP64
 * posterior on the CPU.
 *
 * The general form walks a site's sorted records with a table of occurrence
 * counts in shared memory and sums all ten genotypes from two loads per
 * record.  Two facts make most of that unnecessary:
 *
 *   - Repeats of a (strand, cycle) key are a property of the reads, not of the
 *     site: two records share a key exactly when their reads have the same
 *     strand and the same start (+) or the same end (-).  So the pileup numbers
 *     the few groups of such reads of a tile once (1 .. 15; a record's group is
 *     in its low bits, 0 for none), and the walk counts them in one 64-bit
 *     register, four bits a group: no shared memory, no scan back.
 *
 *   - A call needs the best genotype and the value of the second best.  With
 *     `maj` the base of most records, those are among the four genotypes that
 *     contain maj, unless the site is one for the FP64 pass anyway.  So for
 *     maj's records only those four are summed, from one 16-byte load per
 *     record.  The other six enter the proof as one upper bound: for a record of
 *     base maj,
 *       term[xy] <= min(term[maj x], term[maj y]) - gap(q_adj),
 *     gap being the least difference over all cycles and bases of the table
 *     (tables.cpp, negative where the table has none).  The few records of
 *     another base are summed in full.
 *
 * Every lane of a warp runs this code for its own site, so its time is its
 * instructions and the rows' loads (each lane's row is a cache line of its own),
 * and straight-line code that does not fit the instruction cache stalls all
 * warps of the SM: the sort is one 16-record network used for every chunk, and
 * the posterior works on four genotypes and one bound.  c1's persistent kernel
 * (8 Mbp, 30x, 100 bp) took 3.00 ms in the general form (261 warp
 * instructions and 86 L1 wavefronts a site) and takes 1.54 ms in this one (150
 * and 43); a first version of it that kept the 32-record network, ten
 * columns in the posterior and arrays in local memory ran at 2.94 ms, a third
 * of its issue slots waiting for instructions.
 *
 * Lean records: the element (base << 6 | 64 - q) in bits 31:24, the read cycle
 * in bits 23:16, the strand in bit 15, 4 * the group in bits 5:2.  Their
 * order is the record words' order.
 */
#ifndef GSNP_LEAN_CUH
#define GSNP_LEAN_CUH

#include "site_math.cuh"

namespace gsnp {

/* a lean record as a record word of occurrence 1 */
GSNP_HDI uint32_t lean_to_record(uint32_t w) { return (w >> 15) << 8 | 1u; }
constexpr uint32_t kLeanPad = 0xFFFFFFFFu;   /* sorts after every record */

/* column of the genotype (a, b), a <= b, of the likelihood tables */
GSNP_HDI constexpr int col_of(int a, int b) { return a * (7 - a) / 2 + b; }
static_assert(col_of(0, 3) == 3 && col_of(1, 1) == 4 && col_of(2, 2) == 7 && col_of(3, 3) == 9, "column order");

/* Compare-exchanges of Batcher's odd-even merge of the sorted halves of v[0, N)
 * (Batcher 1968), and of the merge sort made of them (63 for 16 records, 128
 * more with their merge for 32; the bitonic network has 240 for 32). */
GSNP_HDI void lean_exchange(uint32_t& x, uint32_t& y) {
    const uint32_t a = x, b = y;
    x = a < b ? a : b;
    y = a < b ? b : a;
}
template <int N>
GSNP_HDI void odd_even_merge(uint32_t* v) {
#pragma unroll
    for (int k = N / 2; k > 0; k >>= 1)
#pragma unroll
        for (int i = 0; i + k < N; ++i)
            if (k == N / 2 ? i < k : (i / k) % 2 == 1) lean_exchange(v[i], v[i + k]);
}
template <int N>
GSNP_HDI void odd_even_sort(uint32_t* v) {
    if constexpr (N > 1) {
        odd_even_sort<N / 2>(v);
        odd_even_sort<N / 2>(v + N / 2);
        odd_even_merge<N>(v);
    }
}

/* Ascending sort of a lean column (kStride words apart) padded with kLeanPad to
 * the next multiple of 16 records; most is the largest count of the warp's
 * lanes, so that every lane runs the same chunks.  The first two chunks are of
 * 16 records, sorted by one network in registers and then merged by another;
 * the rest come 8 at a time and are merged from the back (most columns past
 * 32 have a few records more). */
template <int kStride>
GSNP_HDI void lean_sort(uint32_t* recs, int num, int most) {
    uint32_t v[32];
    const int end = most > 16 ? 32 : 16;
#pragma unroll 1
    for (int c0 = 0; c0 < end; c0 += 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = recs[(c0 + i) * kStride];
        odd_even_sort<16>(v);
#pragma unroll
        for (int i = 0; i < 16; ++i) recs[(c0 + i) * kStride] = v[i];
    }
    if (end == 16) return;
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = recs[i * kStride];
    odd_even_merge<32>(v);
#pragma unroll
    for (int i = 0; i < 32; ++i) recs[i * kStride] = v[i];
#pragma unroll 1
    for (int c0 = 32; c0 < most; c0 += 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = recs[(c0 + i) * kStride];
        odd_even_sort<8>(v);
        if (num > c0) merge_back<8, kStride>(recs, c0, v, num - c0 < 8 ? num - c0 : 8);
    }
}

/* What the pileup leaves besides the records.  extra4 has 16 bits a base: in the
 * low nine count_all beyond the records, in the high seven the records of
 * quality 0 among the base's reads, which lie under base | 1 (lean_zeros). */
struct LeanPile {
    uint32_t depth, repeat;
    uint64_t extra4;
    int num;
};
constexpr int kLeanExtraBits = 9;
constexpr uint64_t kLeanExtraOf4 = 0x01ff01ff01ff01ffull;
GSNP_HDI uint32_t lean_extra(uint64_t extra4, int base) {
    return (uint32_t)(extra4 >> (16 * base)) & ((1u << kLeanExtraBits) - 1u);
}

/* what the walk leaves of a site's column */
struct LeanSums {
    float s4[4];       /* sums of the genotypes (maj, 0..3) over maj's records */
    float mn[10];      /* all ten over the records of another base */
    int gap;           /* sum of gaps over maj's records, in kLeanGapUnit */
    uint32_t cu4;      /* records per base, 4 x 8 bits */
    uint64_t qs4;      /* quality sums per base, 4 x 16 bits */
    int maj, n_minor;
};

/* The walk counts a record by the base of its word.  One of quality 0 lies
 * under base | 1 with a score of 64: its count goes back to its read's base, its
 * score away. */
GSNP_HDI void lean_zeros(const LeanPile& pile, LeanSums* z) {
    const uint64_t zeros = pile.extra4 & ~kLeanExtraOf4;
    if (zeros == 0) return;
    auto of = [&](int base) { return (uint32_t)(zeros >> (16 * base + kLeanExtraBits)) & 0x7fu; };
    const uint32_t a = of(0), t = of(2);
    z->cu4 += a - (a << 8) + (t << 16) - (t << 24);
    z->qs4 -= (uint64_t)(kMaxQ * (a + of(1))) << 16 | (uint64_t)(kMaxQ * (t + of(3))) << 48;
}

/* The counts of one base group's walk: the earlier records of a record's key,
 * and 64 * (distinct keys so far - 1) */
struct LeanCounts {
    uint64_t cnt = 0;
    int g64 = -64;
    /* the record's index in lean_q, by its 64 - q in the last place */
    GSNP_HDI int next(uint32_t w) {
        const uint32_t sh = w & 0x3cu;
        const int tmp = (int)((uint32_t)(cnt >> sh) & 15u);
        cnt += (1ull << sh) & ~1ull;   /* group 0 is never counted */
        if (tmp == 0) g64 += 64;
        return tmp * (kLeanG * 64) + g64;
    }
};

/* sum of the signed (unsigned) top bytes: acc + top byte of x */
GSNP_HDI int add_top_signed(uint32_t x, int acc) {
#ifdef __CUDA_ARCH__
    return __dp4a((int)x, 0x01000000, acc);
#else
    return acc + ((int)x >> 24);
#endif
}
GSNP_HDI uint32_t add_top(uint32_t x, uint32_t acc) {
#ifdef __CUDA_ARCH__
    return __dp4a(x, 0x01000000u, acc);
#else
    return acc + (x >> 24);
#endif
}

/* a lean record with the q_adj of its lean_q entry in bits 13:6 (for a second
 * walk over the column) */
GSNP_HDI uint32_t lean_with_qa(uint32_t w, uint32_t e) { return (w & ~0x3fc0u) | ((e >> 10) & 0x3fc0u); }
GSNP_HDI int lean_qa(uint32_t w) { return (int)((w >> 6) & 0xffu); }

/* The walk over a sorted lean column of num records (kStride words apart, at
 * most kLeanG of them; up to three words past the last one are read and not
 * used).  none is the maj of a site without records; KEEP_QA leaves each
 * record's q_adj in it.  lean_q's entries hold
 * q_adj * L in bits 15:0, q_adj in bits 23:16 and the gap (signed) in bits
 * 31:24. */
template <int kStride, bool KEEP_QA = false>
__device__ __forceinline__ void lean_walk(const CallArgs& a, uint32_t* recs, int num, int none, LeanSums* o) {
    const int maj = num > 0 ? (int)(recs[(num >> 1) * kStride] >> 30) : none;
    /* maj's records are [gb, ge) */
    int gb = 0, ge = num;
    while (gb < num && (int)(recs[gb * kStride] >> 30) != maj) ++gb;
    while (ge > gb && (int)(recs[(ge - 1) * kStride] >> 30) != maj) --ge;
    const int m = ge - gb;
    o->maj = maj;
    o->n_minor = num - m;
    o->cu4 = (uint32_t)m << (8 * maj);
    float s[4] = {0.f, 0.f, 0.f, 0.f}, c[4] = {0.f, 0.f, 0.f, 0.f};
    int gap = 0;
    uint32_t tops = 0;
    {
        /* four records a step; the next step's q_adj entries are loaded while
         * this one's rows are on their way */
        LeanCounts k;
        const uint32_t* lq = a.lean_q - maj * 64;
        uint32_t* p = recs + gb * kStride;
        const float4* rows = reinterpret_cast<const float4*>(a.lean4) + (size_t)(maj * (a.qa_rows * a.L + 1));
        uint32_t w[4], e[4];
        auto entries = [&](int i) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = i + u < m;
                w[u] = p[u * kStride];
                const int at = k.next(w[u]);
                e[u] = 0;
                if (ok) {
                    e[u] = GSNP_LDG(lq + at + (int)(w[u] >> 24));
                    tops = add_top(w[u], tops);
                }
            }
            p += 4 * kStride;
        };
        entries(0);
#pragma unroll 1
        for (int i = 0; i < m; i += 4) {
            float4 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                gap = add_top_signed(e[u], gap);
                const uint32_t row = (e[u] & 0xffffu) + ((w[u] >> 16) & 0xffu) + 1u;
                x[u] = GSNP_LDG(rows + (i + u < m ? row : 0u));   /* row 0 is all zero */
                if (KEEP_QA && i + u < m) recs[(gb + i + u) * kStride] = lean_with_qa(w[u], e[u]);
            }
            if (i + 4 < m) entries(i + 4);
            const float v[4] = {__fadd_rn(__fadd_rn(x[0].x, x[1].x), __fadd_rn(x[2].x, x[3].x)),
                                __fadd_rn(__fadd_rn(x[0].y, x[1].y), __fadd_rn(x[2].y, x[3].y)),
                                __fadd_rn(__fadd_rn(x[0].z, x[1].z), __fadd_rn(x[2].z, x[3].z)),
                                __fadd_rn(__fadd_rn(x[0].w, x[1].w), __fadd_rn(x[2].w, x[3].w))};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float y = __fsub_rn(v[j], c[j]);
                const float t = __fadd_rn(s[j], y);
                c[j] = __fsub_rn(__fsub_rn(t, s[j]), y);
                s[j] = t;
            }
        }
    }
    /* top byte = maj * 64 + 64 - q */
    const uint32_t q_maj = (uint32_t)((maj * 64 + kMaxQ) * m) - tops;
    o->qs4 = (uint64_t)q_maj << (16 * maj);
    o->gap = gap;
#pragma unroll
    for (int j = 0; j < 4; ++j) o->s4[j] = s[j];
#pragma unroll
    for (int k = 0; k < 10; ++k) o->mn[k] = 0.f;
    /* the records of other bases, each base's group in order */
    LeanCounts k;
    int last = -1;
#pragma unroll 1
    for (int i = gb > 0 ? 0 : ge; i < num;) {
        const uint32_t w = recs[i * kStride];
        const int ob = (int)(w >> 30);
        if (ob != last) {
            k = LeanCounts();
            last = ob;
        }
        const uint32_t e = GSNP_LDG(a.lean_q + k.next(w) + (int)((w >> 24) & 63u));
        float x[10];
        lik32_row(a, (int)((e >> 16) & 0xffu), (int)((w >> 16) & 0xffu), ob, x);
#pragma unroll
        for (int t = 0; t < 10; ++t) o->mn[t] = __fadd_rn(o->mn[t], x[t]);
        o->cu4 += 1u << (8 * ob);
        o->qs4 += (uint64_t)(kMaxQ - ((w >> 24) & 63u)) << (16 * ob);
        if (KEEP_QA) recs[i * kStride] = lean_with_qa(w, e);
        ++i;
        if (i == gb) i = ge;
    }
}

/* The FP64 sums of the genotypes (maj, maj) and (maj, win) over a column that
 * lean_walk<KEEP_QA> has walked, every record in the reference's order: bit
 * for bit likelihood_fp64's.  maj's records take both terms in one 16-byte
 * load (lean2d), the others one each from the general table. */
template <int kStride>
__device__ __forceinline__ void lean_sums64(const CallArgs& a, const uint32_t* recs, int num, const LeanSums& z, int win,
                                            double* best, double* second) {
    const int maj = z.maj, lo = maj < win ? maj : win, hi = maj < win ? win : maj;
    const double* t0 = a.lik64 + col_of(maj, maj);
    const double* t1 = a.lik64 + col_of(lo, hi);
    const double2* rows = reinterpret_cast<const double2*>(a.lean2d) + (size_t)((maj * 4 + win) * a.qa_rows) * a.L;
    double s0 = 0.0, s1 = 0.0;
    const int m = num - z.n_minor;
    /* the other bases' records before maj's, maj's, and those after: one loop
     * each, so that the lanes of a warp run maj's together */
    auto other = [&](int i) {
        const uint32_t w = recs[i * kStride];
        const size_t row = ((size_t)(lean_qa(w) * a.L) + ((w >> 16) & 0xffu)) * 40 + (w >> 30) * 10;
        s0 = GSNP_DADD(s0, GSNP_LDG(t0 + row));
        s1 = GSNP_DADD(s1, GSNP_LDG(t1 + row));
    };
    int gb = 0;
#pragma unroll 1
    for (; gb < num && (int)(recs[gb * kStride] >> 30) != maj; ++gb) other(gb);
    const uint32_t* p = recs + gb * kStride;
#pragma unroll 1
    for (int i = 0; i < m; i += 4, p += 4 * kStride) {
        double2 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            x[u] = double2{0.0, 0.0};   /* adding it changes nothing: the sums are not -0 */
            if (i + u < m) {
                const uint32_t v = p[u * kStride];
                x[u] = GSNP_LDG(rows + lean_qa(v) * a.L + (int)((v >> 16) & 0xffu));
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (u == 0 || i + u < m) {
                s0 = GSNP_DADD(s0, x[u].x);
                s1 = GSNP_DADD(s1, x[u].y);
            }
    }
#pragma unroll 1
    for (int i = gb + m; i < num; ++i) other(i);
    *best = s0;
    *second = s1;
}

__device__ __forceinline__ SitePileup lean_counts(const LeanPile& pile, const LeanSums& z) {
    SitePileup p;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        p.cu[b] = (int)((z.cu4 >> (8 * b)) & 0xffu);
        p.qs[b] = (int)((z.qs4 >> (16 * b)) & 0xffffu);
        p.ca[b] = (uint32_t)p.cu[b] + lean_extra(pile.extra4, b);
    }
    p.depth = pile.depth;
    p.repeat = pile.repeat;
    p.dep_uni = p.num = pile.num;
    return p;
}

/* fill_call of a homozygous call from the packed counts (no indexed arrays).
 * The average quality is the integer quotient: a quotient of q <= 65535 by
 * c <= 255 that is not whole is 1/255 away from the next integer, and
 * (q + 1/4) / c stays on its side under the few ulps of the fast division. */
__device__ __forceinline__ void lean_fill(CallWords* out, const LeanPile& pile, const LeanSums& z, const TopBases& tb,
                                          int type1, int q) {
#ifdef __CUDA_ARCH__
    auto avg = [](uint32_t s, uint32_t n) { return (uint32_t)__fdividef((float)s + 0.25f, (float)n); };
#else
    auto avg = [](uint32_t s, uint32_t n) { return (uint32_t)(((float)s + 0.25f) / (float)n); };
#endif
    const bool b1 = tb.base1 < 4, b2 = tb.base2 < 4;
    const uint32_t cu1 = b1 ? (z.cu4 >> (8 * tb.base1)) & 0xffu : 0u, cu2 = b2 ? (z.cu4 >> (8 * tb.base2)) & 0xffu : 0u;
    const uint32_t qs1 = b1 ? (uint32_t)(z.qs4 >> (16 * tb.base1)) & 0xffffu : 0u;
    const uint32_t qs2 = b2 ? (uint32_t)(z.qs4 >> (16 * tb.base2)) & 0xffffu : 0u;
    const uint32_t ca1 = cu1 + (b1 ? lean_extra(pile.extra4, tb.base1) : 0u);
    const uint32_t ca2 = cu2 + (b2 ? lean_extra(pile.extra4, tb.base2) : 0u);
    out->a.x = (uint32_t)type1 | (uint32_t)tb.base1 << 8 | (uint32_t)tb.base2 << 16 | (uint32_t)q << 24;
    out->a.y = (qs1 ? avg(qs1, cu1) : 0u) | (qs2 ? avg(qs2, cu2) : 0u) << 8;
    out->a.z = cu1 | ca1 << 16;
    out->a.w = cu2 | ca2 << 16;
    out->b.x = pile.depth;
    out->b.y = pile.repeat;
    out->b.z = 0u;   /* rank-sum value 1.0 */
    out->b.w = 0x3ff00000u;
}

/* The values and bounds behind a lean call, for diploid calls.  With tp_j the
 * value of (maj, j) and v2 the largest for j != maj (j = win):
 *
 *   |tp_j - tp64_j| <= E_j: maj's sum carries 6 u and the record count's term
 *   (likelihood_fp32's grouping), the minor sum n_minor u, and the three
 *   additions and the prior's rounding one u of their operands each.
 *
 *   Any of the other six is at most M = max_j(s4_j) - gap + max(minor sum +
 *   prior over the six), within E_M, j over the three others.
 */
struct LeanBounds {
    float v1, e1, v2, e2;   /* (maj, maj), and the best of the other three */
    float rest;             /* the largest of tp_j + E_j - v2 over the two after it, and M + E_M - v2 */
    float ball;             /* the same over all three and M */
    float slack;            /* of E_j and E_M: covers the roundings of such differences */
    int win;
};

__device__ __forceinline__ LeanBounds lean_bounds(const CallArgs& a, int64_t snp_row, uint8_t ori, const LeanSums& z,
                                                  int num) {
    const float inf = INFINITY, u = 0x1p-24f;
    float t[10];
    load_log_prior32(a, snp_row, ori, t);
    float lp_mag = 0.f, mn_mag = 0.f;
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        lp_mag = fmaxf(lp_mag, fabsf(t[k]));
        mn_mag = fmaxf(mn_mag, fabsf(z.mn[k]));
        t[k] = __fadd_rn(z.mn[k], t[k]);
    }
    /* minor sums and priors of the four genotypes, and the six's largest */
    float t4[4] = {t[0], t[1], t[2], t[3]};
    float six = -inf;
#pragma unroll
    for (int b1 = 0; b1 < 4; ++b1)
#pragma unroll
        for (int b2 = b1; b2 < 4; ++b2) {
            const int k = col_of(b1, b2);
            const bool has = z.maj == b1 || z.maj == b2;
            six = fmaxf(six, has ? -inf : t[k]);
            if (b1 > 0 && z.maj == b1) t4[b2] = t[k];
            if (b2 > 0 && z.maj == b2) t4[b1] = t[k];
        }
    const float gap = __fmul_rn((float)z.gap, kLeanGapUnit);
    /* what every bound shares: the minor sum's error and every rounding after it */
    const float rest = __fadd_rn(__fmul_rn(mn_mag, (float)(z.n_minor + 8) * u), __fmul_rn(lp_mag, 8.f * u));
    const float kk = __fadd_rn(9.f * u, __fmul_rn((float)num, 0x1p-45f));
    LeanBounds b;
    b.v1 = b.e1 = b.e2 = 0.f;
    b.v2 = -inf;
    b.win = 0;
    float top = -inf, e_top = 0.f, tp[4], E[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        tp[j] = __fadd_rn(z.s4[j], t4[j]);
        E[j] = __fadd_rn(__fmul_rn(fabsf(z.s4[j]), kk), rest);
        if (z.maj == j) {
            b.v1 = tp[j];
            b.e1 = E[j];
            tp[j] = -inf;
        } else {
            if (tp[j] >= b.v2) { b.v2 = tp[j]; b.e2 = E[j]; b.win = j; }
            top = fmaxf(top, z.s4[j]);
            e_top = fmaxf(e_top, E[j]);
        }
    }
    /* M and its bound: three more additions of at most these magnitudes */
    const float M = __fadd_rn(__fsub_rn(top, gap), six);
    const float e_m = __fadd_rn(e_top, __fmul_rn(__fadd_rn(__fadd_rn(fabsf(top), fabsf(gap)), fabsf(six)), 4.f * u));
    b.rest = __fadd_rn(__fsub_rn(M, b.v2), e_m);
    b.ball = b.rest;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float x = __fadd_rn(__fsub_rn(tp[j], b.v2), E[j]);
        b.ball = fmaxf(b.ball, x);
        if (j != b.win) b.rest = fmaxf(b.rest, x);
    }
    b.slack = __fadd_rn(e_top, e_m);
    return b;
}

/* fast_posterior's proof (prove_hom) over the walk's sums: with d = v1 - v2 and
 * B = ball, tp64[maj maj] - max(other tp64) lies in [d - E1 - B, d + E1 + E2]. */
__device__ __forceinline__ bool lean_posterior(const CallArgs& a, int64_t snp_row, uint8_t ori, const LeanPile& pile,
                                               const LeanSums& z, CallWords* out) {
    const float grow = 1.0f + 0x1p-18f;
    const LeanBounds b = lean_bounds(a, snp_row, ori, z, pile.num);
    /* the roundings of the differences: 2^-23 of quantities of E's size where
     * B is small, and of B itself where a bound lies above v2 */
    const float B = __fmul_rn(__fadd_rn(fmaxf(b.ball, 0.f), __fmul_rn(b.slack, 0x1p-20f)), grow);
    if (!(isfinite(b.v1) && isfinite(b.v2) && isfinite(B))) return false;
    const float d = __fsub_rn(b.v1, b.v2);
    const float below = __fmul_rn(__fadd_rn(b.e1, B), grow);
    const float above = __fmul_rn(__fadd_rn(b.e1, b.e2), grow);
    if (!(__fsub_rn(__fmul_rn(d, 1.0f - 0x1p-22f), below) > 0.f)) return false;
    const TopBases tb = top_bases(lean_counts(pile, z), ori & 7);
    const float raw_lo = __fmul_rn(10.f, __fsub_rn(d, below));
    const float raw_hi = __fmul_rn(10.f, __fadd_rn(d, above));
    const float slack = __fmul_rn(__fadd_rn(fabsf(raw_hi), 1.f), 0x1p-19f);
    const int g1 = z.maj << 2 | z.maj;
    const int q = finalize_q(__float2int_rz(__fsub_rn(raw_lo, slack)), true, false, tb, g1);
    if (q != finalize_q(__float2int_rz(__fadd_rn(raw_hi, slack)), true, false, tb, g1)) return false;
    lean_fill(out, pile, z, tb, g1, q);
    return true;
}

/* The FP64 form's call from the FP64 sums of two genotypes, for diploid calls.
 * The FP32 sums only say which two: (maj, win) is the best of the genotypes
 * other than (maj, maj) when every other one's bound lies below its own.  Its
 * FP64 value is then the second best, and the best one's too if that is
 * larger.  False, writing nothing, when they do not say it, or when the best
 * genotype is not (maj, maj): the site then takes all ten in FP64. */
template <int kStride>
__device__ __forceinline__ bool lean_posterior64(const CallArgs& a, int64_t snp_row, uint8_t ori, const LeanPile& pile,
                                                 const LeanSums& z, const uint32_t* recs, CallWords* out) {
    const float grow = 1.0f + 0x1p-18f;
    const LeanBounds b = lean_bounds(a, snp_row, ori, z, pile.num);
    const float rest = __fadd_rn(b.rest, __fmul_rn(__fadd_rn(b.slack, fabsf(b.rest)), 0x1p-18f));
    if (!(isfinite(b.v2) && __fadd_rn(rest, __fmul_rn(b.e2, grow)) < 0.f && b.v1 > b.v2)) return false;
    const double* prior = (ori & 0x8) && a.refine ? a.snp_lp + snp_row * 16 : a.log_prior + ((ori & 7) << 4);
    double s0, s1;
    lean_sums64<kStride>(a, recs, pile.num, z, b.win, &s0, &s1);
    const int g1 = z.maj << 2 | z.maj, g2 = z.maj <= b.win ? z.maj << 2 | b.win : b.win << 2 | z.maj;
    const double best = GSNP_DADD(s0, GSNP_LDG(prior + g1)), second = GSNP_DADD(s1, GSNP_LDG(prior + g2));
    if (!(best > second)) return false;
    /* the rank-sum value of a homozygous call is 1 and its log10 0 */
    const TopBases tb = top_bases(lean_counts(pile, z), ori & 7);
    const double raw = GSNP_DMUL(10.0, GSNP_DSUB(best, second));
    lean_fill(out, pile, z, tb, g1, finalize_q((int)raw, true, false, tb, g1));
    return true;
}

}  // namespace gsnp

#endif
