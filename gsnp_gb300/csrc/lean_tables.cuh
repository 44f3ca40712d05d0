/*
 * lean_tables.cuh - the tables of the short form (lean.cuh), entry by entry
 * from the general tables; host-compilable.
 *
 *   lean_q  [16][kLeanG][64]        by earlier records of the key, distinct keys
 *                                   before and 64 - q: q_adj * L in bits 15:0,
 *                                   q_adj in bits 23:16, its gap in bits 31:24
 *   lean4   [4][1 + qa_rows * L][4] base o's records: a row of zeros, then the
 *                                   FP32 terms of (o, 0..3)
 *   lean2d  [4][4][qa_rows * L][2]  by [o][x]: the FP64 terms of (o, o), (o, x)
 */
#ifndef GSNP_LEAN_TABLES_CUH
#define GSNP_LEAN_TABLES_CUH

#include "lean.cuh"

namespace gsnp {

constexpr int64_t kLeanQ = (int64_t)16 * kLeanG * 64;
GSNP_HDI int64_t lean4_rows(int qa_rows, int L) { return 4 * ((int64_t)qa_rows * L + 1); }
GSNP_HDI int64_t lean2d_rows(int qa_rows, int L) { return 16 * ((int64_t)qa_rows * L); }

GSNP_HDI uint32_t lean_q_entry(const uint8_t* qadj, int tmax, int gmax, int L, const int8_t* gap, int64_t i) {
    const int q = 64 - (int)(i % 64), g = (int)(i / 64 % kLeanG), tmp = (int)(i / 64 / kLeanG) + 1;
    const int qa = tmp < tmax && g < gmax ? qadj[((int64_t)tmp * gmax + g) * 65 + q] : 1;
    return (uint32_t)(qa * L) | (uint32_t)qa << 16 | (uint32_t)(uint8_t)gap[qa] << 24;
}

GSNP_HDI void lean4_row(const double* lik64, int qa_rows, int L, int64_t i, float* out) {
    const int64_t rows = (int64_t)qa_rows * L + 1;
    const int o = (int)(i / rows);
    const int64_t r = i % rows;
    for (int j = 0; j < 4; ++j)
        out[j] = r == 0 ? 0.f : (float)lik64[((r - 1) * 4 + o) * 10 + (o < j ? col_of(o, j) : col_of(j, o))];
}

GSNP_HDI void lean2d_row(const double* lik64, int qa_rows, int L, int64_t i, double* out) {
    const int64_t rows = (int64_t)qa_rows * L;
    const int x = (int)(i / rows % 4), o = (int)(i / rows / 4);
    const double* r = lik64 + ((i % rows) * 4 + o) * 10;
    out[0] = r[col_of(o, o)];
    out[1] = r[o < x ? col_of(o, x) : col_of(x, o)];
}

}  // namespace gsnp

#endif
