// Shared part of the gathering kernels (adder_fwd_gather.cu, adder_gx_gather.cu): an adder layer as a
// channels x pixels tile with a streamed reduction, like a matrix product, whose pixel-side operand is gathered
// from an NCHW tensor while it is staged.  Any kernel extent, stride, padding and dilation is one set of
// affine tap offsets, so these kernels take every geometry.
//
// A CTA of 128 threads owns TC channels x TP pixels; pixels run over the whole batch (image, row, column), so
// no plane size leaves a ragged tile behind.  A chunk of the reduction is one shared-memory stage:
//   GATHER_TAP    16 channels of one tap (index order: channel block, tap, channel in the block), so that a thread computes the
//                 address and the bounds test of its pixel once per chunk (32 of a 1x1 layer in the thin tiles);
//   GATHER_HALVES two blocks of 16 channels and one tap each in one stage of a thin tile;
//   GATHER_QUADS  1x1 layers whose operand is read in order: 16-byte copies, 16 or 32 channels;
//   GATHER_NINE   2 channels (4 in the thin tiles) x the 9 taps of a 3x3 window, in index order (channel, row, column).
//   GATHER_QUADS_ROWS, GATHER_NINE_ROWS (forward, takes_rows) the same with the weights left as they lie, in 16-byte copies;
//   GATHER_TAP_ROWS (input gradient) GATHER_TAP with the weights from a copy by taps, in 16-byte copies.
// One barrier per chunk; large tiles keep two stages, small ones as many as hide the latency of a load.
#pragma once
#include "common.cuh"
#include "../../include/adder_b200.h"

namespace adder {

constexpr int GATHER_CK = 16;
constexpr int GATHER_THREADS = 128;
enum GatherMode { GATHER_TAP, GATHER_QUADS, GATHER_NINE, GATHER_HALVES, GATHER_QUADS_ROWS, GATHER_NINE_ROWS, GATHER_TAP_ROWS };
inline const char* staging_name(int mode) {
    constexpr const char* names[] = {"tap", "quads", "nine", "halves", "quads_rows", "nine_rows", "tap_rows"};
    return names[mode];
}

// Channels of a chunk of GATHER_NINE; thin tiles (a few outputs a thread) spend their time on the instructions around a stage
// rather than on its terms, so their stages are twice as long.
__host__ __device__ constexpr int nine_channels(bool thin) { return thin ? 4 : 2; }

// Rows of a stage.  1x1 layers take 32 channels at a time where four CTAs still fit an SM: half the barriers (1024->256 on 75,776
// pixels: input gradient 1687 -> 1549 us saturating, 2013 -> 1937 exact, forward 1344 -> 1326).  3x3 layers
// lost 1-6 % by it, measured with weights staged as they lie, a tap's words apart; the _ROWS modes were not measured with more rows.
__host__ __device__ constexpr int gather_rows(int mode, int stages, int tc, int tp, int more_bytes, int ctas, bool thin = false) {
    if (mode == GATHER_NINE || mode == GATHER_NINE_ROWS) return 9 * nine_channels(thin);
    if (thin) return 2 * GATHER_CK;
    return (mode == GATHER_QUADS || mode == GATHER_QUADS_ROWS) && ctas <= 4 && stages * 32 * (tp + tc + 4) * 4 + more_bytes <= 56 * 1024 ? 2 * GATHER_CK : GATHER_CK;
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

// Whether a launch of the gathering kernels can be made: the extent of the grid and the shared memory of a CTA.
inline int gather_status(int grid_y, size_t smem) { return grid_y > 65535 || smem > 227 * 1024 ? ADDER_ERR_UNSUPPORTED : ADDER_OK; }

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
template <int TP, int CK = GATHER_CK>
__device__ __forceinline__ void gather_pixels(float* dst, const GatherPixel* px, const float* src, const GatherMap& m,
                                              const GatherChunk& c, int nch, int ck, int Hs, int Ws, int tid) {
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;      // pixels per thread
    constexpr int ROWS = TP < GATHER_THREADS ? GATHER_THREADS / TP : 1;      // threads that share a pixel column
    const int plane = Hs * Ws;
#pragma unroll
    for (int q = 0; q < COLS; ++q) {
        const int row = px[q].row + m.oy0 + c.i * m.doy, col = px[q].col + m.ox0 + c.j * m.dox;
        const bool ok = px[q].ok & ((unsigned)row < (unsigned)Hs) & ((unsigned)col < (unsigned)Ws);
        copy_rows<ROWS, TP, CK>(dst + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP), ok ? px[q].base + (c.c0 * plane + row * Ws + col) : src,
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

// GATHER_NINE: rows (channel c0 + r/9, tap r%9), r < 9 CH, of the thread's pixels; channels from nch on are zero.  Where several
// threads share a pixel (TP < 128: small layers, whose time is this loop's), a thread's rows are not known at compile time: their
// offsets are computed once.
template <int TP, int CH>
struct GatherNine {
    static constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;
    static constexpr int ROWS = TP < GATHER_THREADS ? GATHER_THREADS / TP : 1;
    static constexpr int N = (9 * CH + ROWS - 1) / ROWS;
    unsigned mask[COLS];        // a bit per tap; ROWS > 1: a bit per row of this thread
    int off[ROWS > 1 ? N : 1];

    __device__ __forceinline__ void init(const GatherPixel* px, const GatherMap& m, int Hs, int Ws, int tid) {
#pragma unroll
        for (int q = 0; q < COLS; ++q) mask[q] = nine_mask(px[q], m, Hs, Ws);
        if constexpr (ROWS > 1) {
            const unsigned taps = mask[0];
            mask[0] = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int r = i * ROWS + tid / TP, c = r / 9, t = r - c * 9;
                off[i] = c * Hs * Ws + (t / 3) * m.doy * Ws + (t % 3) * m.dox;
                if (taps >> t & 1) mask[0] |= 1u << i;
            }
        }
    }
    __device__ __forceinline__ void fill(float* dst, const GatherPixel* px, const GatherMap& m, int c0, int nch, int Hs, int Ws,
                                         int tid) const {
        const int plane = Hs * Ws;
        if constexpr (ROWS > 1) {
            const float* s = px[0].base + (c0 * plane + (px[0].row + m.oy0) * Ws + px[0].col + m.ox0);
            const int rows = 9 * CH - tid / TP, full = 9 * nch - tid / TP;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if ((9 * CH) % ROWS != 0 && i == N - 1 && i * ROWS >= rows) break;
                // nothing is read where the predicate is false, so the address may lie outside the tensor there
                cp_async4(dst + tid + i * GATHER_THREADS, s + off[i], (mask[0] >> i & 1) & (i * ROWS < full));
            }
        } else {
#pragma unroll
            for (int q = 0; q < COLS; ++q) {
                const float* s = px[q].base + (c0 * plane + (px[q].row + m.oy0) * Ws + px[q].col + m.ox0);
                float* d = dst + tid + q * GATHER_THREADS;
#pragma unroll
                for (int r = 0; r < 9 * CH; ++r) {
                    const int c = r / 9, t = r - c * 9;
                    cp_async4(d + r * TP, s + (c * plane + (t / 3) * m.doy * Ws + (t % 3) * m.dox), (mask[q] >> t & 1) & (c < nch));
                }
            }
        }
    }
};

}  // namespace adder
