/*
 * lean_rules_check.cpp - which tables the short form (lean.cuh) accepts: its
 * bounds are relative to sums of terms that are zero or less, so a matrix with
 * an entry above 1 has to leave it off.  Prints "<kind> lean <0|1>" for a plain
 * matrix, one with an entry of 1.2 and one whose 1.2 no cycle reaches.
 */
#include <stdio.h>

#include <cmath>
#include <string>
#include <vector>

#include "tables.h"

using namespace gsnp;

int main() {
    gsnp_params p{};
    p.read_length = 100;
    p.q_min = 64;
    p.q_max = 64 + 40;
    p.pcr_dependency = log10(0.5);
    p.global_dependency = log10(0.9);
    std::vector<double> prior(128);
    prior_table(p, 1, 0.0010, 0.0005, prior.data());
    for (const char* kind : {"plain", "above", "unreached"}) {
        std::vector<double> pm(256UL * 256UL * 16UL, 1.0);
        for (size_t q = 0; q < 64; ++q)
            for (size_t c = 0; c < 256; ++c)
                for (size_t k = 0; k < 16; ++k) {
                    const double e = std::min(0.75, pow(10.0, -(double)q / 10.0));
                    pm[q << 12 | c << 4 | k] = (k >> 2) == (k & 3) ? 1.0 - e : e / 3.0;
                }
        if (kind[0] != 'p') pm[30UL << 12 | (kind[0] == 'a' ? 50UL : 150UL) << 4 | 5] = 1.2;
        HostTables t;
        std::string err;
        if (build_tables(p, pm.data(), prior.data(), &t, &err) != 0) {
            printf("%s: %s\n", kind, err.c_str());
            return 1;
        }
        printf("%s lean %d\n", kind, (int)t.lean_ok);
    }
    return 0;
}
