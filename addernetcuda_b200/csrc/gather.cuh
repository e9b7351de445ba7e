// Shared part of the gathering kernels (adder_fwd_gather.cu, adder_gx_gather.cu): an adder layer as a
// channels x pixels tile with a streamed reduction, like a matrix product, whose pixel-side operand is gathered
// from an NCHW tensor while it is staged.  Any kernel extent, stride, padding and dilation is one set of
// affine tap offsets, so these kernels take every geometry.
//
// A CTA of 128 threads owns TC channels x TP pixels; pixels run over the whole batch (image, row, column), so
// no plane size leaves a ragged tile behind.  A chunk of the reduction is one shared-memory stage:
//   GATHER_TAP    at most 16 channels of one tap (index order: channel block, tap, channel in the block), so that a
//                 thread computes the address and the bounds test of its pixel once per chunk;
//   GATHER_QUADS  the same for 1x1 layers whose operand is read in order: 16-byte copies;
//   GATHER_NINE   2 channels x the 9 taps of a 3x3 window, in index order (channel, row, column).
// One barrier per chunk; large tiles keep two stages, small ones as many as hide the latency of a load.
#pragma once
#include "common.cuh"

namespace adder {

constexpr int GATHER_CK = 16;
constexpr int GATHER_NINE_CH = 2;        // channels per chunk of GATHER_NINE
constexpr int GATHER_THREADS = 128;
enum GatherMode { GATHER_TAP, GATHER_QUADS, GATHER_NINE };

// Rows of a stage.  1x1 layers take 32 channels at a time where four CTAs still fit an SM: half the barriers (1024->256 on 75,776
// pixels: input gradient 1687 -> 1549 us saturating, 2013 -> 1937 exact, forward 1344 -> 1326; 3x3 layers lose 1-6 %, the weights of
// a chunk being strided).
__host__ __device__ constexpr int gather_rows(int mode, int stages, int tc, int tp, int more_bytes, int ctas) {
    if (mode == GATHER_NINE) return 9 * GATHER_NINE_CH;
    return mode == GATHER_QUADS && ctas <= 4 && stages * 32 * (tp + tc + 4) * 4 + more_bytes <= 56 * 1024 ? 2 * GATHER_CK : GATHER_CK;
}

// What a tile costs, in clocks per reduction step, measured over 30 layers (n 1-256, 3x3 and 1x1) with every tile forced and fitted
// within 3-10 %: `alone` for a CTA that has its SM to itself, `more` for each further one beside it while they hide each other's
// latency, `share` of the SM's throughput.
struct TileCost { float alone, more, share; };
inline double tile_cost(const TileCost& t, long long tiles, int sms) {
    const long long p = (tiles + sms - 1) / sms;
    if (p > 8) return (double)t.share * (double)tiles / sms;        // CTAs come and go: no common waves
    const double a = t.alone + t.more * (double)(p - 1), b = (double)t.share * (double)p;
    return a > b ? a : b;
}

// Where the pixel-side operand of reduction tap (i, j) of pixel (py, px) lives in its source tensor:
// row py*sy + oy0 + i*doy, column px*sx + ox0 + j*dox; out of bounds reads zero.  wt0 + i*dwi + j*dwj is the tap's
// index in the kernel window.
struct GatherMap {
    int PH, PW, P;              // pixel space: rows, columns, N*PH*PW
    int th, tw, ntaps;          // taps of the reduction
    int sy, sx, oy0, doy, ox0, dox;
    int wt0, dwi, dwj;
    FastDiv d_phw, d_pw;
};

// The pixel a thread gathers, decoded once.
struct GatherPixel {
    const float* base;          // source tensor at image n (channel 0)
    int row, col;               // source row / column before the tap offset
    bool ok;
    __device__ __forceinline__ void decode(const GatherMap& m, const float* src, int p, size_t image_stride) {
        ok = p < m.P;
        uint32_t n, r, y, x;
        m.d_phw.divmod(ok ? p : 0, n, r);
        m.d_pw.divmod(r, y, x);
        base = src + n * image_stride;
        row = (int)y * m.sy;
        col = (int)x * m.sx;
    }
};

// The running position in the reduction: chunk -> (channel block, tap).
struct GatherChunk {
    int c0 = 0, i = 0, j = 0;   // first channel of the block, tap row, tap column
    __device__ __forceinline__ void next(const GatherMap& m, int ck) {
        if (++j < m.tw) return;
        j = 0;
        if (++i < m.th) return;
        i = 0;
        c0 += ck;
    }
};

// Copies rows k0, k0 + STEP, ... of one staged column: row k comes from s + k * stride, rows from nch on are zero.
// The common full chunk is straight-line code, an address increment and a copy a row; a column that reads zeros has
// stride 0 and a valid address.
template <int STEP, int PITCH, int CK = GATHER_CK>
__device__ __forceinline__ void copy_rows(float* d, const float* s, int stride, bool ok, int k0, int nch, int ck) {
    d += k0 * PITCH;
    s += k0 * stride;
    if (nch == CK) {
#pragma unroll
        for (int k = 0; k < CK; k += STEP, s += STEP * stride) cp_async4(d + k * PITCH, s, ok);
    } else {
        const float* first = s;
#pragma unroll 2
        for (int k = k0; k < ck; k += STEP, s += STEP * stride, d += STEP * PITCH) cp_async4(d, k < nch ? s : first, ok & (k < nch));
    }
}

// Stages one chunk of the pixel-side operand as [channel][TP pixels].
template <int TP>
__device__ __forceinline__ void gather_pixels(float* dst, const GatherPixel* px, const float* src, const GatherMap& m,
                                              const GatherChunk& c, int nch, int ck, int Hs, int Ws, int tid) {
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;      // pixels per thread
    constexpr int ROWS = TP < GATHER_THREADS ? GATHER_THREADS / TP : 1;      // threads that share a pixel column
    const int plane = Hs * Ws;
#pragma unroll
    for (int q = 0; q < COLS; ++q) {
        const int row = px[q].row + m.oy0 + c.i * m.doy, col = px[q].col + m.ox0 + c.j * m.dox;
        const bool ok = px[q].ok & ((unsigned)row < (unsigned)Hs) & ((unsigned)col < (unsigned)Ws);
        copy_rows<ROWS, TP>(dst + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP), ok ? px[q].base + (c.c0 * plane + row * Ws + col) : src,
                            ok ? plane : 0, ok, tid / TP, nch, ck);
    }
}

// The same for layers whose pixels are the source's own pixels in order (1x1, stride 1, no padding) and whose planes are whole
// quads: 16-byte copies.  px holds the thread's quad (pixel 4 * (tid % (TP/4)) of the tile).
template <int TP, int CK>
__device__ __forceinline__ void gather_quads(float* dst, const float* base, bool ok, const float* src, int c0, int nch, int ck,
                                             int plane, int tid) {
    constexpr int QUADS = TP / 4, ROWS = GATHER_THREADS / QUADS;
    const int k0 = tid / QUADS;
    float* d = dst + k0 * TP + 4 * (tid % QUADS);
    const float* s = ok ? base + (c0 + k0) * plane : src;
    const int step = ok ? ROWS * plane : 0;
    if (nch == CK) {
#pragma unroll
        for (int k = 0; k < CK; k += ROWS, s += step) cp_async16(d + k * TP, s, ok);
    } else {
        for (int k = k0; k < ck; k += ROWS, s += step, d += ROWS * TP) cp_async16(d, k < nch ? s : src, ok & (k < nch));
    }
}

// A bit per tap of the 3x3 window: the tap of this pixel lies inside the plane.
__device__ __forceinline__ unsigned nine_mask(const GatherPixel& px, const GatherMap& m, int Hs, int Ws) {
    unsigned mask = 0;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int row = px.row + m.oy0 + (t / 3) * m.doy, col = px.col + m.ox0 + (t % 3) * m.dox;
        if (px.ok & ((unsigned)row < (unsigned)Hs) & ((unsigned)col < (unsigned)Ws)) mask |= 1u << t;
    }
    return mask;
}

// GATHER_NINE: rows (channel c0 + r/9, tap r%9), r < 18, of the thread's pixels; channels from nch on are zero.
template <int TP>
__device__ __forceinline__ void gather_nine(float* dst, const GatherPixel* px, const unsigned* mask, const GatherMap& m, int c0,
                                            int nch, int Hs, int Ws, int tid) {
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;
    constexpr int ROWS = TP < GATHER_THREADS ? GATHER_THREADS / TP : 1;
    const int plane = Hs * Ws;
#pragma unroll
    for (int q = 0; q < COLS; ++q) {
        const float* s = px[q].base + (c0 * plane + (px[q].row + m.oy0) * Ws + px[q].col + m.ox0);
        float* d = dst + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP);
#pragma unroll
        for (int i = 0; i < (9 * GATHER_NINE_CH + ROWS - 1) / ROWS; ++i) {
            const int r = i * ROWS + (ROWS > 1 ? tid / TP : 0);
            if (ROWS > 1 && (9 * GATHER_NINE_CH) % ROWS != 0 && r >= 9 * GATHER_NINE_CH) break;
            const int c = r / 9, t = r - c * 9;
            // nothing is read where the predicate is false, so the address may lie outside the tensor there
            cp_async4(d + r * TP, s + (c * plane + (t / 3) * m.doy * Ws + (t % 3) * m.dox), (mask[q] >> t & 1) & (c < nch));
        }
    }
}

}  // namespace adder
