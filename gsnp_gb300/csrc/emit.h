/*
 * emit.h - cns text rows on the device (emit.cu).
 */
#ifndef GSNP_EMIT_H
#define GSNP_EMIT_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "gsnp_device.cuh"

namespace gsnp {

struct EmitArgs {
    const SiteCall* calls;      /* [chr_len] */
    const SiteCounts* counts;   /* [chr_len] or null */
    const uint8_t* codes;       /* [chr_len] */
    const int32_t* host_src;    /* [n_windows] window whose host counts each window shows */
    const char* chr;            /* chromosome name (device) */
    int chr_n;
    int64_t site0, n;           /* rows of sites [site0, site0 + n) */
    uint64_t* off;              /* scratch: byte offset of every kEmitRows-th row */
    char* text;                 /* output of emit_text: one piece's text */
    int* error;                 /* set when a value is outside the formatter's range */
};

constexpr int kEmitRows = 128;                              /* rows of a CTA */
constexpr int64_t kEmitPiece = kWin;                        /* rows of a piece, about 17 MB of text */
constexpr int64_t kPieceBlocks = kEmitPiece / kEmitRows;
static_assert(kEmitPiece % kEmitRows == 0, "a piece is whole blocks");

/* pieces of n rows */
int64_t emit_pieces(int64_t n);

/* device scratch of emit_lengths for n rows */
size_t emit_scratch_bytes(int64_t n);

/* Measure e's rows: byte offsets in scratch (sets e.off). */
cudaError_t emit_lengths(EmitArgs& e, void* scratch, cudaStream_t stream);

/* Copy the first byte of every piece and, last, the total to
 * h_off[0, emit_pieces(e.n)] (after emit_lengths). */
cudaError_t emit_offsets(const EmitArgs& e, uint64_t* h_off, cudaStream_t stream);

/* Write one piece's text to e.text (after emit_lengths). */
cudaError_t emit_text(const EmitArgs& e, int64_t piece, cudaStream_t stream);

}  // namespace gsnp

#endif
