/*
 * lean_check.cpp - the short form of a site's FP32 call (lean.cuh, compiled
 * for the host) against the general form and the FP64 posterior, with the
 * library's own tables (tables.cpp), on random sites:
 *
 *  1. lean_sort puts the records in their order, the walk's sums lie within
 *     their bounds of the FP64 ones (the main base's records and the others
 *     apart), and its counts and quality sums are the column's;
 *  2. every call lean_posterior decides equals the FP64 posterior's;
 *  3. its proof holds for adversarial sums: FP64 sums of the four genotypes
 *     that contain the main base anywhere within their bounds, those of
 *     the other six anywhere from -infinity to their upper bounds.
 *
 * Sites as posterior_check.cpp's, at depths 0 to 64 (kLeanG) with qualities 1
 * to 63, under calibrations from plain to noisy (rows in which another base is
 * likelier than the read's own, so that gaps are negative).
 * The FP64 form's two sums are checked beside it bit for bit, and its calls.
 * Prints "sites <n> decided <d> of <h> homozygous adversarial <a> decided64
 * <e>" and exits 0, or names the first failing site and exits 1.
 * Usage: lean_check <sites> <seed> <read length>
 */
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <map>
#include <random>
#include <string>
#include <vector>

#include "lean.cuh"
#include "lean_tables.cuh"
#include "tables.h"

using namespace gsnp;

static int pair_col(int a, int b) { return a < b ? col_of(a, b) : col_of(b, a); }

int main(int argc, char** argv) {
    const long n_sites = argc > 1 ? atol(argv[1]) : 100000;
    const unsigned long seed = argc > 2 ? strtoul(argv[2], nullptr, 10) : 1;
    gsnp_params p{};
    p.read_length = argc > 3 ? atoi(argv[3]) : 100;
    p.q_min = 64;
    p.q_max = 64 + 63;
    p.pcr_dependency = log10(0.5);
    p.global_dependency = log10(0.9);
    p.het_val = 0.1;
    p.het_unval = 0.02;
    p.althom_val = 0.05;
    p.althom_unval = 0.01;
    p.rank_sum = 1;
    p.precision = 1;
    p.het_novel = 0.0010;
    p.althom_novel = 0.0005;
    p.transition_dominant = 1;
    std::mt19937_64 rng(seed);
    auto uni = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
    auto below = [&](int n) { return (int)(rng() % (uint64_t)n); };
    std::vector<double> prior(128), rank(64UL * 64UL * 2048UL);
    prior_table(p, p.transition_dominant, p.het_novel, p.althom_novel, prior.data());
    rank_table(rank.data());
    std::vector<uint32_t> seen(64);
    long decided = 0, hom = 0, adversarial = 0, decided64 = 0;
    constexpr int kCalibrations = 4;
    for (int cal = 0; cal < kCalibrations; ++cal) {
        /* error 10^(-q/10) over the three other bases, varying with the cycle
         * and, from calibration to calibration, more and more at random */
        std::vector<double> pm(256UL * 256UL * 16UL, 1.0);
        for (int q = 0; q <= p.q_max - p.q_min; ++q)
            for (int coord = 0; coord < p.read_length; ++coord)
                for (int ref = 0; ref < 4; ++ref) {
                    const double e = std::min(0.75, pow(10.0, -q / 10.0) * (1.0 + 0.3 * coord / p.read_length));
                    for (int obs = 0; obs < 4; ++obs)
                        pm[((size_t)q << 12) | ((size_t)coord << 4) | (size_t)(ref << 2) | (size_t)obs] =
                            (obs == ref ? 1.0 - e : e / 3.0) * pow(10.0, cal == 0 ? 0.0 : -uni(0.0, 0.25 * cal));
                }
        p.pcr_dependency = log10(cal == 2 ? 0.9 : 0.5);
        p.global_dependency = log10(cal == 3 ? 0.99 : 0.9);
        HostTables t;
        std::string err;
        if (build_tables(p, pm.data(), prior.data(), &t, &err) != 0 || !t.lean_ok || !t.all_nonpositive) {
            printf("tables of calibration %d: %s\n", cal, err.c_str());
            return 1;
        }
        CallArgs a{};
        a.L = t.L;
        a.lik64 = t.lik64.data();
        a.lik32 = t.lik32.data();
        a.lik32b = t.lik32.data() + (size_t)t.qa_rows * t.L * 4 * 8;
        std::vector<uint32_t> lean_q((size_t)kLeanQ);
        std::vector<float> lean4((size_t)lean4_rows(t.qa_rows, t.L) * 4);
        std::vector<double> lean2d((size_t)lean2d_rows(t.qa_rows, t.L) * 2);
        for (size_t i = 0; i < lean_q.size(); ++i)
            lean_q[i] = lean_q_entry(t.qadj.data(), t.tmax, t.gmax, t.L, t.lean_gap.data(), (int64_t)i);
        for (size_t i = 0; i < lean4.size() / 4; ++i) lean4_row(t.lik64.data(), t.qa_rows, t.L, (int64_t)i, &lean4[i * 4]);
        for (size_t i = 0; i < lean2d.size() / 2; ++i)
            lean2d_row(t.lik64.data(), t.qa_rows, t.L, (int64_t)i, &lean2d[i * 2]);
        a.lean_q = lean_q.data();
        a.lean4 = lean4.data();
        a.lean2d = lean2d.data();
        a.qa_rows = t.qa_rows;
        a.qadj = t.qadj.data();
        a.tmax = t.tmax;
        a.gmax = t.gmax;
        a.log_prior = t.log_prior.data();
        a.log_prior32 = t.log_prior32.data();
        a.p_rank = rank.data();
        a.q_max_min = p.q_max - p.q_min;
        a.rank_sum = 1;
        a.precision = 1;
        std::vector<uint32_t> recs, lean;
        for (long site = 0; site < n_sites / kCalibrations; ++site) {
            const int ref = below(4);
            const uint8_t ori = (uint8_t)(below(50) == 0 ? 4 + ref : ref);
            const int kind = below(10);
            const int alt = (ref + 1 + below(3)) & 3;
            const double frac = kind < 6 ? 0.0 : kind < 8 ? 1.0 : kind < 9 ? uni(0.3, 0.7) : uni(0.02, 0.3);
            const int depth = below(6) == 0 ? below(6) : below(kLeanG + 1);
            std::map<std::pair<int, int>, int> keys;   /* (strand, cycle): records */
            SitePileup sp{};
            recs.clear();
            for (int i = 0; i < depth; ++i) {
                const int q = below(10) == 0 ? 1 + below(15) : below(20) == 0 ? 41 + below(23) : 20 + below(21);
                int base = uni(0, 1) < frac ? alt : ref;
                if (uni(0, 1) < pow(10.0, -q / 10.0)) base = (base + 1 + below(3)) & 3;
                int coord = below(p.read_length), strand = below(2);
                if (!recs.empty() && below(8) == 0) {
                    const uint32_t w = recs[(size_t)below((int)recs.size())];
                    coord = rec_coord(w);
                    strand = rec_strand(w);
                }
                int repeats = 0;
                for (auto& k : keys) repeats += k.second > 1;
                int& k = keys[{strand, coord}];
                if (k >= 15 || (k == 1 && repeats >= 15)) { continue; }
                ++k;
                recs.push_back(make_record_of((uint32_t)base, q, (uint32_t)coord, (uint32_t)strand));
                sp.cu[base] += 1;
                sp.qs[base] += q;
                sp.ca[base] += 1;
            }
            std::sort(recs.begin(), recs.end());
            sp.num = sp.dep_uni = (int)recs.size();
            sp.depth = sp.ca[0] + sp.ca[1] + sp.ca[2] + sp.ca[3] + (uint32_t)below(3);
            sp.repeat = sp.depth + (uint32_t)below(3);
            /* the pileup's records: 4 * the group of a repeated key in their
             * low bits, in pileup order, padded */
            std::map<std::pair<int, int>, int> group;
            lean.clear();
            for (uint32_t w : recs) {
                const std::pair<int, int> key{rec_strand(w), rec_coord(w)};
                int id = 0;
                if (keys[key] > 1) {
                    int& g = group[key];
                    if (!g) g = (int)group.size();
                    id = g;
                }
                lean.push_back((w >> 8) << 15 | (uint32_t)id << 2);
            }
            std::shuffle(lean.begin(), lean.end(), rng);
            lean.resize(kLeanG + 4, kLeanPad);
            lean_sort<1>(lean.data(), sp.num, std::min(kLeanG, sp.num + below(17)));
            for (int i = 0; i < sp.num; ++i)
                if (lean_to_record(lean[(size_t)i]) != recs[(size_t)i]) {
                    printf("site %ld: record %d out of order (num %d)\n", site, i, sp.num);
                    return 1;
                }
            LeanPile pile{sp.depth, sp.repeat, 0, sp.num};
            for (int b = 0; b < 4; ++b) {
                const uint64_t extra = (uint64_t)(below(8) == 0 ? below(300) : 0);
                pile.extra4 |= extra << (16 * b);
                sp.ca[b] += (uint32_t)extra;
            }
            LeanSums z;
            lean_walk<1>(a, lean.data(), sp.num, ori & 3, &z);
            double tl64[16] = {0}, main64[10] = {0}, minor64[10] = {0};
            likelihood_fp64<2>(a, recs.data(), seen.data(), 1, sp.num, tl64);
            walk_records<false, 2>(a, recs.data(), seen.data(), 1, sp.num, [&](int, int qa, int coord, int o) {
                for (int k = 0; k < 10; ++k)
                    (o == z.maj ? main64 : minor64)[k] += a.lik64[((size_t)(qa * a.L + coord) * 4 + o) * 10 + k];
            });
            const double u = 0x1p-24;
            for (int j = 0; j < 4; ++j) {
                const double d = fabs((double)z.s4[j] - main64[pair_col(z.maj, j)]);
                if (!(d <= fabs((double)z.s4[j]) * GSNP_FP32_K(sp.num))) {
                    printf("site %ld: main sum %d off by %.3g\n", site, j, d);
                    return 1;
                }
            }
            for (int k = 0; k < 10; ++k) {
                const double d = fabs((double)z.mn[k] - minor64[k]);
                if (!(d <= fabs((double)z.mn[k]) * (z.n_minor + 1) * u)) {
                    printf("site %ld: minor sum %d off by %.3g (%d records)\n", site, k, d, z.n_minor);
                    return 1;
                }
                const int x = col_base(k, 0), y = col_base(k, 1);
                if (x != z.maj && y != z.maj &&
                    main64[k] > std::min(main64[pair_col(z.maj, x)], main64[pair_col(z.maj, y)]) - z.gap * kLeanGapUnit + 1e-12) {
                    printf("site %ld: genotype column %d above its upper bound\n", site, k);
                    return 1;
                }
            }
            for (int b = 0; b < 4; ++b)
                if ((int)((z.cu4 >> (8 * b)) & 0xffu) != sp.cu[b] || (int)((z.qs4 >> (16 * b)) & 0xffffu) != sp.qs[b]) {
                    printf("site %ld: counts of base %d differ\n", site, b);
                    return 1;
                }
            double lp[16];
            load_log_prior(a, -1, ori, lp);
            auto nq = [&](int b) { return (int)((b * 7 + site) % 40); };
            SiteCall want, got;
            site_posterior<false>(a, ori, sp, tl64, nullptr, lp, recs.data(), 1, nq, &want);
            hom += (want.type1 >> 2) == (want.type1 & 3);
            /* the FP64 form: its two sums bit for bit, and its calls */
            {
                std::vector<uint32_t> kept = lean;
                LeanSums y;
                lean_walk<1, true>(a, kept.data(), sp.num, ori & 3, &y);
                for (int x = 0; x < 4; ++x) {
                    double s0, s1;
                    lean_sums64<1>(a, kept.data(), sp.num, y, x, &s0, &s1);
                    if (s0 != tl64[genotype_of(pair_col(y.maj, y.maj))] || s1 != tl64[genotype_of(pair_col(y.maj, x))]) {
                        printf("site %ld: FP64 sums of (%d, %d) differ\n", site, y.maj, x);
                        return 1;
                    }
                }
                CallWords words;
                if (lean_posterior64<1>(a, -1, ori, pile, y, kept.data(), &words)) {
                    ++decided64;
                    memcpy(&got, &words, sizeof got);
                    if (!same_call(got, want)) {
                        printf("site %ld: the FP64 short form gives type %d q %d, FP64 type %d q %d (num %d, ori %d)\n",
                               site, got.type1, got.q_cns, want.type1, want.q_cns, sp.num, ori);
                        return 1;
                    }
                }
                for (int i = 0; i < sp.num; ++i)
                    if (lean_to_record(kept[(size_t)i]) != recs[(size_t)i]) {
                        printf("site %ld: record %d changed\n", site, i);
                        return 1;
                    }
            }
            CallWords words;
            if (!lean_posterior(a, -1, ori, pile, z, &words)) continue;
            memcpy(&got, &words, sizeof got);
            ++decided;
            if (!same_call(got, want)) {
                printf("site %ld: the short form gives type %d q %d, FP64 type %d q %d (num %d, ori %d)\n", site,
                       got.type1, got.q_cns, want.type1, want.q_cns, sp.num, ori);
                return 1;
            }
            /* what the proof may be given: the four sums anywhere in their
             * bounds, the six anywhere at or below their upper bounds */
            for (int v = 0; v < 2; ++v) {
                double t64[16] = {0};
                for (int k = 0; k < 10; ++k) {
                    const int g = genotype_of(k), x = col_base(k, 0), y = col_base(k, 1);
                    const double mn = (double)z.mn[k] * (1.0 + uni(-1.0, 1.0) * z.n_minor * u);
                    if (x == z.maj || y == z.maj) {
                        const double f = z.s4[x == z.maj ? y : x];
                        t64[g] = f + uni(-1.0, 1.0) * 0.999 * fabs(f) * GSNP_FP32_K(sp.num) + mn;
                    } else {
                        const double ub = std::min((double)z.s4[x], (double)z.s4[y]) - (double)z.gap * kLeanGapUnit + mn;
                        t64[g] = v == 0 ? ub : ub - (below(4) == 0 ? 1e6 : uni(0.0, 5.0));
                    }
                }
                ++adversarial;
                site_posterior<false>(a, ori, sp, t64, nullptr, lp, recs.data(), 1, nq, &want);
                if (!same_call(got, want)) {
                    printf("site %ld: adversarial sums %d: type %d q %d against type %d q %d (num %d, ori %d)\n", site, v,
                           got.type1, got.q_cns, want.type1, want.q_cns, sp.num, ori);
                    return 1;
                }
            }
        }
    }
    printf("sites %ld decided %ld of %ld homozygous adversarial %ld decided64 %ld\n", n_sites, decided, hom,
           adversarial, decided64);
    return 0;
}
