/*
 * emit.cu - cns text rows on the device (cpp/call_genotype.cc:353-411).
 *
 * One row per site:
 *   chr pos ref type q_cns base1 avgQ1 cu1 ca1 base2 avgQ2 cu2 ca2 depth
 *   rank_sum copy_ratio dbsnp
 * tab separated, doubles as %#.6g (fmt_g6.h), and the reference's literal
 * "N ... 1.000 255.000 0" row for sites it does not call.  The row fields
 * come from make_row (rows.h), which reproduces the reference's stale host
 * count arrays in gap windows.
 *
 * The text of a range of sites is built in three steps over blocks of kRows
 * rows.  A first kernel measures the rows and leaves each block's byte count;
 * one CTA scans those into byte offsets (8 bytes per 128 rows instead of 12
 * bytes per row); the write kernel measures again - its rows' values stay in
 * registers - scans the 128 lengths in the CTA, puts the characters into
 * shared memory and stores them as aligned 16-byte words.  A row's call is
 * read twice (64 bytes) against 66 bytes of text written; the link that takes
 * the text to the host is what bounds a program that wants it.
 * 4 M rows of the 10x shape, 264 MB, size and text wanted: 20.1 -> 1.78 ms,
 * 1.37 of it the copy to the host (before: a row per thread formatted in local
 * memory and stored byte by byte, 1.7 ms in the write kernel alone, and a
 * host thread's memcpy out of a pinned buffer).
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "emit.h"
#include "fmt_g6.h"
#include "rows.h"

namespace gsnp {

namespace {

__constant__ char c_abbv[17] = {'A', 'M', 'W', 'R', 'M', 'C', 'Y', 'S', 'W', 'Y', 'T', 'K', 'R', 'S', 'K', 'G', 'N'};
__constant__ char c_actgn[8] = {'A', 'C', 'T', 'G', 'N', 'N', 'N', 'N'};

constexpr int kRows = kEmitRows;      /* rows of a CTA, one per thread */
constexpr int kRowFields = 128;       /* most characters of a row after the name (the fields add up to 111) */
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
__constant__ char c_nlit[] = "\tN\tN\t0\tN\t0\t0\t0\tN\t0\t0\t0\t0\t1.000\t255.000\t0\n";
constexpr int kNLen = (int)sizeof(c_nlit) - 1;

__device__ __forceinline__ int digits(uint32_t v) {
    int n = 1;
    if (v >= 10000) {
        n = 5;
        v /= 10000;
        if (v >= 10000) return 9 + (v >= 100000);
    }
    return n + (v >= 10) + (v >= 100) + (v >= 1000);
}

__device__ __forceinline__ int digits_i(int v) { return v < 0 ? 1 + digits(0u - (uint32_t)v) : digits((uint32_t)v); }

/* v's digits at p, from the back; returns the end */
__device__ __forceinline__ char* put_u(char* p, uint32_t v, int n) {
    for (int i = n - 1; i >= 0; --i) {
        const uint32_t q = v / 10;
        p[i] = (char)('0' + (v - q * 10));
        v = q;
    }
    return p + n;
}

__device__ __forceinline__ char* put_i(char* p, int v) {
    if (v < 0) {
        *p++ = '-';
        v = (int)(0u - (uint32_t)v);
    }
    return put_u(p, (uint32_t)v, digits((uint32_t)v));
}

/* One row: its values and the length of its text, 0 when a double is outside
 * the exact formatter's range. */
struct Row {
    CnsRow r;
    G6 rank, ratio;
    uint32_t pos;       /* 1-based */
    int len;
    bool ok;
};

__device__ __forceinline__ Row measure_row(const EmitArgs& e, int64_t site) {
    Row o;
    const int64_t w = site / kWin, j = site - w * kWin;
    o.r = make_row(e.host_src[w], w, j, e.codes, e.calls, e.counts);
    o.pos = (uint32_t)(site + 1);
    o.ok = true;
    o.len = e.chr_n + 1 + digits(o.pos);
    const CnsRow& r = o.r;
    if (!r.called()) {
        o.len += kNLen;
        return o;
    }
    o.rank = fmt_g6_parse(r.rank_sum);
    o.ratio = fmt_g6_parse(r.depth == 0 ? 255.0 : (double)r.repeat / r.depth);
    /* 15 tabs after the position; ref, type, base1, dbsnp, end of line */
    o.len += 15 + 5 + digits_i(r.q_cns) + digits_i(r.avg1) + digits_i(r.cu1) + digits_i(r.ca1);
    o.len += r.base2 < 4 ? 1 + digits_i(r.avg2) + digits_i(r.cu2) + digits_i(r.ca2) : 4;
    o.len += digits(r.depth) + o.rank.len + o.ratio.len;
    if (o.rank.len == 0 || o.ratio.len == 0) {
        o.ok = false;
        o.len = 0;
    }
    return o;
}

__device__ __forceinline__ void put_row(const EmitArgs& e, const Row& o, const char* name, char* p) {
    const CnsRow& r = o.r;
    for (int i = 0; i < e.chr_n; ++i) *p++ = name[i];
    *p++ = '\t';
    p = put_u(p, o.pos, digits(o.pos));
    if (!r.called()) {
        for (int i = 0; i < kNLen; ++i) p[i] = c_nlit[i];
        return;
    }
    *p++ = '\t';
    *p++ = c_actgn[r.ori & 7];
    *p++ = '\t';
    *p++ = c_abbv[r.type1];
    *p++ = '\t';
    p = put_i(p, r.q_cns);
    /* base, avgQ, unique and all counts of the best and the second base */
    for (int k = 0; k < 2; ++k) {
        const bool any = k == 0 || r.base2 < 4;
        *p++ = '\t';
        *p++ = any ? c_actgn[k == 0 ? r.base1 : r.base2] : 'N';
        *p++ = '\t';
        p = put_i(p, any ? (k == 0 ? r.avg1 : r.avg2) : 0);
        *p++ = '\t';
        p = put_i(p, any ? (k == 0 ? r.cu1 : r.cu2) : 0);
        *p++ = '\t';
        p = put_i(p, any ? (k == 0 ? r.ca1 : r.ca2) : 0);
    }
    *p++ = '\t';
    p = put_u(p, r.depth, digits(r.depth));
    /* the rank sum's p-value, the copy ratio */
    for (int k = 0; k < 2; ++k) {
        const G6 g = k == 0 ? o.rank : o.ratio;
        *p++ = '\t';
        fmt_g6_put(g, p);
        p += g.len;
    }
    *p++ = '\t';
    *p++ = (r.ori & 8) ? '1' : '0';
    *p++ = '\n';
}

/* the bytes of each CTA's rows */
__global__ void __launch_bounds__(kRows) row_len_kernel(EmitArgs e) {
    const int64_t i = (int64_t)blockIdx.x * kRows + threadIdx.x;
    __shared__ uint32_t s_sum[kRows / 32];
    uint32_t len = 0;
    if (i < e.n) {
        const Row o = measure_row(e, e.site0 + i);
        if (!o.ok) atomicExch(e.error, 1);
        len = (uint32_t)o.len;
    }
    len = __reduce_add_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = len;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int k = 0; k < kRows / 32; ++k) t += s_sum[k];
        e.off[blockIdx.x] = t;
    }
}

/* The text of blocks [block0, block0 + gridDim.x) at e.text, which receives
 * block0's first byte.  The characters go to shared memory at the place they
 * have within their 16-byte word of the output, so that whole words can be
 * stored. */
__global__ void __launch_bounds__(kRows) row_write_kernel(EmitArgs e, int64_t block0) {
    extern __shared__ uint4 s_words[];
    __shared__ uint32_t s_sum[kRows / 32];
    __shared__ char s_name[256];
    char* s_text = (char*)s_words;
    const int64_t b = block0 + blockIdx.x, i = b * kRows + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < e.chr_n; k += kRows) s_name[k] = e.chr[k];
    char* dst = e.text + (e.off[b] - e.off[block0]);
    const uint32_t head = (uint32_t)((uintptr_t)dst & 15);
    Row o;
    o.len = 0;
    if (i < e.n) o = measure_row(e, e.site0 + i);
    uint32_t x = (uint32_t)o.len;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int k = 0; k < kRows / 32; ++k) {
        if (k < warp) before += s_sum[k];
        total += s_sum[k];
    }
    if (o.len) put_row(e, o, s_name, s_text + head + before + x - (uint32_t)o.len);
    __syncthreads();
    char* word0 = dst - head;
    const uint32_t end = head + total;
    const uint32_t first = head ? 16 : 0, last = end & ~15u;
    for (uint32_t k = first + threadIdx.x * 16; k < last; k += kRows * 16) *(uint4*)(word0 + k) = s_words[k / 16];
    /* the bytes of the words shared with the neighbouring blocks */
    if (threadIdx.x < 16) {
        const uint32_t k = threadIdx.x;
        if (head && k >= head && k < end) word0[k] = s_text[k];
    } else if (threadIdx.x < 32) {
        const uint32_t k = last + threadIdx.x - 16;
        if (k >= first && k < end) word0[k] = s_text[k];
    }
}

/* exclusive prefix of v over the CTA */
__device__ uint64_t block_exclusive(uint64_t v, uint64_t* total) {
    __shared__ uint64_t warp_sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t x = v;
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint64_t s = lane < kScanThreads / 32 ? warp_sums[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += y;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = s;
    }
    __syncthreads();
    const uint64_t before = (warp ? warp_sums[warp - 1] : 0) + x - v;
    *total = warp_sums[kScanThreads / 32 - 1];
    __syncthreads();
    return before;
}

/* off[0, nb): byte counts to offsets, in place; off[nb, padded): the total */
__global__ void __launch_bounds__(kScanThreads) scan_blocks_kernel(uint64_t* off, int64_t nb, int64_t padded) {
    uint64_t carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += kScanThreads * kScanItems) {
        const int64_t b = b0 + (int64_t)threadIdx.x * kScanItems;
        uint64_t v[kScanItems], t = 0;
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = b + k < nb ? off[b + k] : 0;
            t += v[k];
        }
        uint64_t total;
        uint64_t run = carry + block_exclusive(t, &total);
        for (int k = 0; k < kScanItems; ++k)
            if (b + k < nb) {
                off[b + k] = run;
                run += v[k];
            }
        carry += total;
    }
    for (int64_t b = nb + threadIdx.x; b < padded; b += kScanThreads) off[b] = carry;
}

}  // namespace

int64_t emit_pieces(int64_t n) { return (n + kEmitPiece - 1) / kEmitPiece; }

size_t emit_scratch_bytes(int64_t n) { return (size_t)(emit_pieces(n) * kPieceBlocks + 1) * 8; }

cudaError_t emit_lengths(EmitArgs& e, void* scratch, cudaStream_t stream) {
    e.off = (uint64_t*)scratch;
    const int64_t nb = (e.n + kRows - 1) / kRows;
    if (nb) row_len_kernel<<<(unsigned)nb, kRows, 0, stream>>>(e);
    scan_blocks_kernel<<<1, kScanThreads, 0, stream>>>(e.off, nb, emit_pieces(e.n) * kPieceBlocks + 1);
    return cudaGetLastError();
}

cudaError_t emit_offsets(const EmitArgs& e, uint64_t* h_off, cudaStream_t stream) {
    return cudaMemcpy2DAsync(h_off, 8, e.off, kPieceBlocks * 8, 8, (size_t)emit_pieces(e.n) + 1,
                             cudaMemcpyDeviceToHost, stream);
}

cudaError_t emit_text(const EmitArgs& e, int64_t piece, cudaStream_t stream) {
    const int64_t b0 = piece * kPieceBlocks, b1 = std::min((e.n + kRows - 1) / kRows, b0 + kPieceBlocks);
    if (b1 <= b0) return cudaSuccess;
    const size_t smem = 16 + (size_t)kRows * (size_t)(kRowFields + e.chr_n);
    if (smem > 47 * 1024) {   /* names near 255 bytes; the kernel's static 0.3 KB count too */
        const cudaError_t err =
            cudaFuncSetAttribute(row_write_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 16 + kRows * (kRowFields + 255));   /* the same for every name: threads share it */
        if (err != cudaSuccess) return err;
    }
    row_write_kernel<<<(unsigned)(b1 - b0), kRows, smem, stream>>>(e, b0);
    return cudaGetLastError();
}

}  // namespace gsnp
