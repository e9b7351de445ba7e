// Input gradient of the adder convolution as a channels x pixels tile with a gathered gradient operand (gather.cuh):
//   gx[n,ci,y,x] = sum over output channels and the taps that read pixel (y, x) of clamp(w - x, -1, 1) * g
// for 1x1 layers and every kernel extent, stride, padding and dilation.  For a stride S the input pixels fall into S*S
// classes (y mod S, x mod S) that are read by different taps; a class is a pixel space of its own (blockIdx.z) whose taps
// are an arithmetic progression, so no thread works on a tap that does not reach its pixel.
//
// A thread keeps 4 input channels x 8 pixels of x and of the sums in registers; a k step is three 128-bit loads for
// 32 terms.  Saturating form: one FFMA.SAT and one FFMA a term, with x' = 1/2 - x/2 in registers:
// clamp(d,-1,1) = 2*sat(d/2 + 1/2) - 1, and the "-1" is the sum of g over the taps, added up once per pixel while the
// stages pass by: in four partial sums, of rows r, r + 4, r + 8 and r + 12 of every 16, whichever threads share the pixel, so that
// the tile - which follows the size of the batch - does not show in the result.  Exact form: min.xorsign.abs is the clamp in one instruction (magnitude min(|d|, 1), sign of d),
// where fminf(fmaxf(d, -1), 1) takes two; differences (large tiles) and sums are packed pairs of pixels.
// With nothing around it the saturating form takes 2.5 lane cycles a term, the register operands that it reads (5 a term, 2 a cycle and
// scheduler); the exact form, a clamp and two halves of packed instructions, is measured at 3.0.  What stands around them is the staging: without it the saturating form of 256->256 14x14 at batch 256
// takes 2.90 lane cycles a term, with it 3.43 from w as it lies and 3.27 from a copy by taps (gx_gather_workspace_bytes).
#include <cstdio>
#include "common.cuh"
#include "gather.cuh"
#include "kernels.h"

namespace adder {

namespace {
constexpr int MAX_CLASSES = 9;
}

struct GxGatherArgs {
    GatherMap m[MAX_CLASSES];
    int ry[MAX_CLASSES], rx[MAX_CLASSES];   // first row and column of the class in the input
    const float* gout;
    const float* x;
    const float* w;          // [Co][Ci][KK]; GATHER_TAP_ROWS: [KK][Co][Ci]
    float* gx;
    int Ci, H, W, Co, Ho, Wo, KK, CK, sh, sw, accumulate;
    int w_quads;             // 1x1: rows of w are whole quads and 16-byte aligned
    int vec_io;              // stride 1, planes are whole quads, x and gx 16-byte aligned
    int fill_block;          // the other pixels of an sh x sw block belong to no class: write zeros there
    int fill_quads;          // ... and four blocks of a row can be written as aligned 128-bit words
    int fill_pairs;          // ... or, rows being even, each block as two aligned 64-bit words
};

// Tiles that may stage their weights from the copy by taps: with 8 and most of those with 16 input channels a row is too short to share
// the 16-byte copies among the threads, and the launch loses up to 11 %, its copy not counted (copy_share).
__host__ __device__ constexpr bool takes_copy(int rc, int rp, int cg) { return rc * cg >= 32 || (rp == 2 && cg == 8); }

// RC channels x RP pixels per thread (RP = 8: two quads half a tile apart), CG channel groups, ST stages, MB CTAs per SM.
// (8 channels x 8 pixels, at 3 CTAs per SM, measured 10-15 % slower than 4 x 8.)
template <int RC_, int RP_, int CG_, int ST_, int MB_>
struct GxTile {
    static constexpr int RC = RC_, RP = RP_, CG = CG_, ST = ST_, MB = MB_;
    static constexpr int PG = GATHER_THREADS / CG, TC = CG * RC, TP = PG * RP, WP = TC + 4;
    static constexpr int PQ = RP == 8 ? 4 : RP;                 // consecutive pixels of a thread
    static constexpr bool TAKES_COPY = takes_copy(RC, RP, CG);
};

template <class T, bool FAST, int MODE>
__global__ void __launch_bounds__(GATHER_THREADS, T::MB) adder_gx_gather_kernel(const __grid_constant__ GxGatherArgs a) {
    constexpr int RC = T::RC, RP = T::RP, CG = T::CG, TC = T::TC, TP = T::TP, WP = T::WP, PQ = T::PQ, ST = T::ST;
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;
    constexpr int ROWS = TP < GATHER_THREADS ? GATHER_THREADS / TP : 1;
    constexpr bool QUADS = MODE == GATHER_QUADS, TAP_ROWS = MODE == GATHER_TAP_ROWS;
    constexpr int CK = gather_rows(MODE, ST, TC, TP, RC * RP * GATHER_THREADS * 4, T::MB);      // rows of a stage
    constexpr int PARTS = 4, MINE = PARTS / ROWS;      // partial sums of g per pixel, and those of one thread
    static_assert(PARTS % ROWS == 0 && (PARTS > ROWS || CK == 16), "whole partial sums per thread, a stage at a time");
    constexpr int FOLD = 64 / CK;                // chunks per partial sum: 64 terms before it is folded into the total
    constexpr bool PACKED = !FAST && RP == 8 && CG >= 8;      // exact form: differences of two pixels at a time
    constexpr int GS = CK * TP, WS = CK * WP;
    extern __shared__ __align__(16) float smem[];
    float* const Gs = smem;
    float* const Ws = smem + ST * GS;
    float4* const Tot = reinterpret_cast<float4*>(Ws + ST * WS) + threadIdx.x;    // [RC * RP / 4][threads]

    const GatherMap& m = a.m[blockIdx.z];
    const int p0 = blockIdx.x * TP, ci0 = blockIdx.y * TC;
    if (p0 >= m.P) return;                       // classes differ by a row and a column
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int cg = (wid % (CG / 4)) * 4 + (lane >> 3), pg = (wid / (CG / 4)) * 8 + (lane & 7);
    const int ry = a.ry[blockIdx.z], rx = a.rx[blockIdx.z];
    const size_t image = (size_t)a.Co * a.Ho * a.Wo;
    const int HW = a.H * a.W;

    GatherPixel px[COLS];
    if (QUADS) {
        px[0].decode(m, a.gout, p0 + 4 * (tid % (TP / 4)), image);
        px[0].base += px[0].row * a.Wo + px[0].col;
    } else {
#pragma unroll
        for (int q = 0; q < COLS; ++q) px[q].decode(m, a.gout, p0 + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP), image);
    }
    GatherChunk fc;
    const int ck4 = round_up(a.CK, 4);
    const int nchunks = ceil_div(a.Co, a.CK) * m.ntaps;
    auto fill = [&](int stage) {
        const int nch = min(a.CK, a.Co - fc.c0);
        if (QUADS) gather_quads<TP, CK>(Gs + stage * GS, px[0].base, px[0].ok, a.gout, fc.c0, nch, ck4, a.Ho * a.Wo, tid);
        else gather_pixels<TP>(Gs + stage * GS, px, a.gout, m, fc, nch, ck4, a.Ho, a.Wo, tid);
        // weights [output channel of the chunk][input channel of the tile]
        float* ws = Ws + stage * WS;
        const float* wsrc;
        if constexpr (TAP_ROWS) wsrc = a.w + (((m.wt0 + fc.i * m.dwi + fc.j * m.dwj) * a.Co + fc.c0) * a.Ci + ci0);
        else wsrc = a.w + ((fc.c0 * a.Ci + ci0) * a.KK + m.wt0 + fc.i * m.dwi + fc.j * m.dwj);
        if (TAP_ROWS || a.w_quads) {
            constexpr int WQ = TC / 4, WROWS = GATHER_THREADS / WQ;
            const int q = 4 * (tid % WQ), k0 = tid / WQ;
            const bool okc = ci0 + q < a.Ci;
            const float* s = okc ? wsrc + (k0 * a.Ci + q) : a.w;
            const int step = okc ? WROWS * a.Ci : 0;
            float* d = ws + k0 * WP + q;
            if (nch == CK && CK % WROWS == 0) {
#pragma unroll
                for (int k = 0; k < CK; k += WROWS, s += step) cp_async16(d + k * WP, s, okc);
            } else {
                for (int k = k0; k < ck4; k += WROWS, s += step, d += WROWS * WP) cp_async16(d, k < nch ? s : a.w, okc & (k < nch));
            }
        } else {
            constexpr int WROWS = GATHER_THREADS / TC;
            const int col = tid % TC;
            const bool okc = ci0 + col < a.Ci;
            copy_rows<WROWS, WP, CK>(ws + col, okc ? wsrc + col * a.KK : a.w, okc ? a.Ci * a.KK : 0, okc, tid / TC, nch, ck4);
        }
        fc.next(m, a.CK);
    };

#pragma unroll 1
    for (int s = 0; s < ST - 1; ++s) {
        if (s < nchunks) fill(s);
        cp_async_commit();
    }

    // x of the thread's pixels
    float xv[RC][RP];
#pragma unroll
    for (int h = 0; h < RP / PQ; ++h) {
        const int p = p0 + h * (TP / 2) + pg * PQ;
        if constexpr (PQ == 4) {
            if (a.vec_io) {
                uint32_t n, r;
                m.d_phw.divmod(p < m.P ? p : 0, n, r);
                const float* xs = a.x + ((size_t)n * a.Ci + ci0 + cg * RC) * HW + r;
#pragma unroll
                for (int c = 0; c < RC; ++c) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p < m.P && ci0 + cg * RC + c < a.Ci) v = __ldg(reinterpret_cast<const float4*>(xs + (size_t)c * HW));
                    xv[c][4 * h] = v.x; xv[c][4 * h + 1] = v.y; xv[c][4 * h + 2] = v.z; xv[c][4 * h + 3] = v.w;
                }
                continue;
            }
        }
#pragma unroll
        for (int j = 0; j < PQ; ++j) {
            uint32_t n, r, y, x;
            m.d_phw.divmod(p + j < m.P ? p + j : 0, n, r);
            m.d_pw.divmod(r, y, x);
            const float* xs = a.x + ((size_t)n * a.Ci + ci0 + cg * RC) * HW + ((int)y * a.sh + ry) * a.W + (int)x * a.sw + rx;
#pragma unroll
            for (int c = 0; c < RC; ++c)
                xv[c][PQ * h + j] = (p + j < m.P && ci0 + cg * RC + c < a.Ci) ? __ldg(xs + (size_t)c * HW) : 0.f;
        }
    }
    float acc[RC][RP];
#pragma unroll
    for (int c = 0; c < RC; ++c)
#pragma unroll
        for (int j = 0; j < RP; ++j) {
            xv[c][j] = FAST ? fmaf(xv[c][j], -0.5f, 0.5f) : -xv[c][j];
            acc[c][j] = 0.f;
        }
    float box[COLS][MINE];
#pragma unroll
    for (int q = 0; q < COLS; ++q)
#pragma unroll
        for (int i = 0; i < MINE; ++i) box[q][i] = 0.f;

    GatherChunk cc;
    int stage = 0, fstage = ST - 1;
    for (int c = 0; c < nchunks; ++c) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (c + ST - 1 < nchunks) fill(fstage);
        cp_async_commit();
        const float* gs = Gs + stage * GS + pg * PQ;
        const float* ws = Ws + stage * WS + cg * RC;
        const int nk = min(ck4, round_up(a.Co - cc.c0, 4));
#pragma unroll 4
        for (int k = 0; k < nk; ++k) {
            float gv[RP], wv[RC];
#pragma unroll
            for (int h = 0; h < RP / PQ; ++h) {
                if constexpr (PQ == 4) {
                    const float4 q = *reinterpret_cast<const float4*>(gs + k * TP + h * (TP / 2));
                    gv[4 * h] = q.x; gv[4 * h + 1] = q.y; gv[4 * h + 2] = q.z; gv[4 * h + 3] = q.w;
                } else {
                    const float2 q = *reinterpret_cast<const float2*>(gs + k * TP);
                    gv[0] = q.x; gv[1] = q.y;
                }
            }
            if constexpr (RC == 4) {
                const float4 q = *reinterpret_cast<const float4*>(ws + k * WP);
                wv[0] = q.x; wv[1] = q.y; wv[2] = q.z; wv[3] = q.w;
            } else {
                const float2 q = *reinterpret_cast<const float2*>(ws + k * WP);
                wv[0] = q.x; wv[1] = q.y;
            }
            if constexpr (FAST) {
#pragma unroll
                for (int r = 0; r < RC; ++r)
#pragma unroll
                    for (int j = 0; j < RP; ++j) acc[r][j] = fmaf(__saturatef(fmaf(wv[r], 0.5f, xv[r][j])), gv[j], acc[r][j]);
            } else if constexpr (PACKED) {
                // both steps of a pair of pixels packed but the clamp: 2.97 lane-clocks a term with nothing around it, 3.31 with a scalar
                // subtraction (1024->256 14x14 at batch 256: 1308 -> 1179 us)
#pragma unroll
                for (int r = 0; r < RC; ++r) {
                    const uint64_t w2 = pack2(wv[r], wv[r]);
#pragma unroll
                    for (int j = 0; j < RP; j += 2) {
                        float d0, d1;
                        unpack2(add2(w2, pack2(xv[r][j], xv[r][j + 1])), d0, d1);
                        const uint64_t s = fma2(pack2(clamp_unit(d0), clamp_unit(d1)), pack2(gv[j], gv[j + 1]), pack2(acc[r][j], acc[r][j + 1]));
                        unpack2(s, acc[r][j], acc[r][j + 1]);
                    }
                }
            } else {                             // (small launches are a chain of latencies: a packed operation is the longer one)
#pragma unroll
                for (int j = 0; j < RP; j += 2)
#pragma unroll
                    for (int r = 0; r < RC; ++r) {
                        const uint64_t s = fma2(pack2(clamp_unit(wv[r] + xv[r][j]), clamp_unit(wv[r] + xv[r][j + 1])),
                                                pack2(gv[j], gv[j + 1]), pack2(acc[r][j], acc[r][j + 1]));
                        unpack2(s, acc[r][j], acc[r][j + 1]);
                    }
            }
        }
        if (FAST) {
            const float* col = Gs + stage * GS + (COLS > 1 ? tid : tid % TP);
            if constexpr (MINE == 1) {               // small tiles: a thread has one of the four
                const float* cq = col + (tid / TP) * TP;
                float s = 0.f;
                if (nk == CK) {
#pragma unroll
                    for (int k = 0; k < CK; k += ROWS) s += cq[k * TP];
                } else {
                    for (int k = 0; k < nk; k += ROWS) s += cq[k * TP];
                }
                box[0][0] += s;
            } else {
#pragma unroll
                for (int q = 0; q < COLS; ++q) {
                    const float* cq = col + (ROWS > 1 ? tid / TP : 0) * TP + q * GATHER_THREADS;
                    if (nk == CK) {
#pragma unroll
                        for (int kb = 0; kb < CK; kb += 16) {
                            float s[MINE];
#pragma unroll
                            for (int k = 0; k < 16 / ROWS; ++k) {
                                const float v = cq[(kb + k * ROWS) * TP];
                                s[k % MINE] = k < MINE ? v : s[k % MINE] + v;
                            }
#pragma unroll
                            for (int i = 0; i < MINE; ++i) box[q][i] += s[i];
                        }
                    } else {
#pragma unroll 1
                        for (int kb = 0; kb < nk; kb += 16) {
                            float s[MINE];
#pragma unroll
                            for (int i = 0; i < MINE; ++i) s[i] = 0.f;
#pragma unroll 1
                            for (int k = kb; k < min(kb + 16, nk); k += PARTS)      // nk is a multiple of 4
#pragma unroll
                                for (int i = 0; i < MINE; ++i) s[i] += cq[(k + i * ROWS) * TP];
#pragma unroll
                            for (int i = 0; i < MINE; ++i) box[q][i] += s[i];
                        }
                    }
                }
            }
        }
        // two-level summation: a long sum over output channels loses far less than one running fp32 accumulator would
        if (c % FOLD == FOLD - 1 && c + 1 < nchunks) {
            float* av = &acc[0][0];
#pragma unroll
            for (int i = 0; i < RC * RP / 4; ++i) {
                float4* t = Tot + i * GATHER_THREADS;
                float4 v = c < FOLD ? make_float4(0.f, 0.f, 0.f, 0.f) : *t;
                v.x += av[4 * i]; v.y += av[4 * i + 1]; v.z += av[4 * i + 2]; v.w += av[4 * i + 3];
                *t = v;
                av[4 * i] = av[4 * i + 1] = av[4 * i + 2] = av[4 * i + 3] = 0.f;
            }
        }
        cc.next(m, a.CK);
        if (++stage == ST) stage = 0;
        if (++fstage == ST) fstage = 0;
    }
    if (nchunks > FOLD) {
        float* av = &acc[0][0];
#pragma unroll
        for (int i = 0; i < RC * RP / 4; ++i) {
            const float4 v = Tot[i * GATHER_THREADS];
            av[4 * i] += v.x; av[4 * i + 1] += v.y; av[4 * i + 2] += v.z; av[4 * i + 3] += v.w;
        }
    }
    if (FAST) {
        __syncthreads();                         // the stages are free
        float* bs = smem;                        // [PARTS][TP]
#pragma unroll
        for (int q = 0; q < COLS; ++q)
#pragma unroll
            for (int i = 0; i < MINE; ++i)
                bs[((ROWS > 1 ? tid / TP : 0) + i * ROWS) * TP + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP)] = box[q][i];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < RP; ++j) {
            const int col = (j / PQ) * (TP / 2) + pg * PQ + (j % PQ);
            float b = bs[col];
#pragma unroll
            for (int r = 1; r < PARTS; ++r) b += bs[r * TP + col];
#pragma unroll
            for (int r = 0; r < RC; ++r) acc[r][j] = fmaf(2.f, acc[r][j], -b);
        }
    }
#pragma unroll
    for (int h = 0; h < RP / PQ; ++h) {
        const int p = p0 + h * (TP / 2) + pg * PQ;
        if constexpr (PQ == 4) {
            if (a.vec_io || a.fill_quads) {
                if (p >= m.P) continue;
                uint32_t n, r, y, x;
                m.d_phw.divmod(p, n, r);
                m.d_pw.divmod(r, y, x);
                float* o = a.gx + ((size_t)n * a.Ci + ci0 + cg * RC) * HW + (a.vec_io ? r : (y * 2) * a.W + x * 2);
#pragma unroll
                for (int c = 0; c < RC; ++c) {
                    if (ci0 + cg * RC + c >= a.Ci) break;
                    float4* o4 = reinterpret_cast<float4*>(o + (size_t)c * HW);
                    float4 v = make_float4(acc[c][4 * h], acc[c][4 * h + 1], acc[c][4 * h + 2], acc[c][4 * h + 3]);
                    if (a.fill_quads) {          // stride 2, pixels of class (0, 0) only: a zero between them and a row of zeros below
                        o4[0] = make_float4(v.x, 0.f, v.y, 0.f);
                        o4[1] = make_float4(v.z, 0.f, v.w, 0.f);
                        o4 = reinterpret_cast<float4*>(o + (size_t)c * HW + a.W);
                        o4[0] = o4[1] = make_float4(0.f, 0.f, 0.f, 0.f);
                        continue;
                    }
                    if (a.accumulate) {
                        const float4 old = *o4;
                        v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
                    }
                    *o4 = v;
                }
                continue;
            }
        }
        if (a.fill_pairs) {                      // stride 2, pixels of class (0, 0) only, rows of an even length
#pragma unroll 1
            for (int j = 0; j < PQ && p + j < m.P; ++j) {
                uint32_t n, r, y, x;
                m.d_phw.divmod(p + j, n, r);
                m.d_pw.divmod(r, y, x);
                float* o = a.gx + ((size_t)n * a.Ci + ci0 + cg * RC) * HW + 2 * y * a.W + 2 * x;
                const bool below = 2 * (int)y + 1 < a.H;
#pragma unroll
                for (int c = 0; c < RC; ++c) {
                    if (ci0 + cg * RC + c >= a.Ci) break;
                    float v = acc[c][PQ * h];
#pragma unroll
                    for (int q = 1; q < PQ; ++q) v = j == q ? acc[c][PQ * h + q] : v;
                    *reinterpret_cast<float2*>(o + (size_t)c * HW) = make_float2(v, 0.f);
                    if (below) *reinterpret_cast<float2*>(o + (size_t)c * HW + a.W) = make_float2(0.f, 0.f);
                }
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < PQ; ++j) {
            if (p + j >= m.P) continue;
            uint32_t n, r, y, x;
            m.d_phw.divmod(p + j, n, r);
            m.d_pw.divmod(r, y, x);
            const int yi = (int)y * a.sh + ry, xi = (int)x * a.sw + rx;
            float* o = a.gx + ((size_t)n * a.Ci + ci0 + cg * RC) * HW + yi * a.W + xi;
#pragma unroll
            for (int c = 0; c < RC; ++c) {
                if (ci0 + cg * RC + c >= a.Ci) break;
                float* oc = o + (size_t)c * HW;
                const float v = acc[c][PQ * h + j];
                if (a.accumulate) { *oc += v; continue; }
                *oc = v;
                // (stride 2 without loops, whose code the packed tiles' register allocation made the slower: 960->24 29x31 at batch 60
                // 340 us scalar, 364 packed, now 302.  The other tiles have the loops: the branch cost some of them 1 to 3 %.)
                if (PACKED && a.fill_block && a.sh == 2 && a.sw == 2) {
                    const bool right = xi + 1 < a.W, below = yi + 1 < a.H;
                    if (right) oc[1] = 0.f;
                    if (below) oc[a.W] = 0.f;
                    if (right & below) oc[a.W + 1] = 0.f;
                } else if (a.fill_block)
                    for (int dy = 0; dy < a.sh && yi + dy < a.H; ++dy)
                        for (int dx = 0; dx < a.sw && xi + dx < a.W; ++dx)
                            if (dy | dx) oc[dy * a.W + dx] = 0.f;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

namespace {

// X(RC, RP, CG, ST, MB, clocks per step: exact form alone, further, throughput; saturating form the same)
#define ADDER_GX_GATHER_TILES(X)                                                                                    \
    X(4, 8, 16, 2, 4, 197, 99, 134, 182, 85, 117) X(4, 8, 8, 2, 4, 196, 112, 134, 182, 85, 118)                     \
    X(4, 8, 4, 2, 4, 219, 122, 142, 213, 112, 132) X(4, 4, 16, 4, 6, 133, 58, 83, 125, 70, 88)                      \
    X(4, 4, 8, 4, 6, 128, 56, 80, 120, 49, 70) X(4, 4, 4, 4, 6, 133, 46, 83, 123, 54, 77)                           \
    X(2, 2, 8, 8, 8, 68, 18, 32, 76, 17, 32) X(2, 2, 4, 8, 8, 70, 18, 33, 80, 18, 33)               \
    X(2, 8, 4, 3, 6, 140, 60, 80, 140, 60, 80)

struct Tile { int rc, rp, cg, st, mb, tc, tp; TileCost exact, fast; };
constexpr Tile kTiles[] = {
#define X(RC, RP, CG, ST, MB, A, M, S, FA, FM, FS) {RC, RP, CG, ST, MB, RC * CG, RP * GATHER_THREADS / CG, {A, M, S}, {FA, FM, FS}},
    ADDER_GX_GATHER_TILES(X)
#undef X
};

long long tile_count(const GxGatherArgs& a, int classes, int Ci, const Tile& t) {
    long long tiles = 0;
    for (int c = 0; c < classes; ++c) tiles += (long long)ceil_div(a.m[c].P, t.tp) * ceil_div(Ci, t.tc);
    return tiles;
}

int choose_tile(const GxGatherArgs& a, int classes, int Ci, bool fast) {
    int best = 0;
    double best_cost = 1e300;
    const int sms = sm_count();
    for (int i = 0; i < (int)(sizeof(kTiles) / sizeof(kTiles[0])); ++i) {
        const Tile& t = kTiles[i];
        const double cost = tile_cost(fast ? t.fast : t.exact, tile_count(a, classes, Ci, t), sms);
        if (cost < best_cost) { best_cost = cost; best = i; }
    }
    return best;
}

int stage_rows(const Tile& t, int mode) {
    return gather_rows(mode, t.st, t.tc, t.tp, t.rc * t.rp * GATHER_THREADS * 4, t.mb);
}

size_t smem_bytes(const Tile& t, int mode) {
    return ((size_t)t.st * stage_rows(t, mode) * (t.tp + t.tc + 4) + (size_t)t.rc * t.rp * GATHER_THREADS) * sizeof(float);
}

// Taps k of one dimension that reach input positions q*S + r: (r + pad - k*dil) % S == 0.  Output position q + o0 + i*d0.
struct ClassTaps { int k0, step, count, o0, d0; };
ClassTaps class_taps(int r, int K, int S, int pad, int dil) {
    ClassTaps t{0, 1, 0, 0, 0};
    for (int k = 0; k < K; ++k) {
        if ((r + pad - k * dil) % S != 0) continue;
        if (t.count == 0) { t.k0 = k; t.o0 = (r + pad - k * dil) / S; }
        else if (t.count == 1) { t.step = k - t.k0; t.d0 = (r + pad - k * dil) / S - t.o0; }
        ++t.count;
    }
    return t;
}

bool fill_classes(const ConvGeom& g, int first, GxGatherArgs& a, int& n, int& total, bool only_first) {
    n = 0; total = 0;
    int at = 0;
    for (int ry = 0; ry < g.sh && ry < g.H; ++ry)
        for (int rx = 0; rx < g.sw && rx < g.W; ++rx) {
            if (only_first && (ry | rx)) continue;
            if (at++ < first || n == MAX_CLASSES) continue;
            const ClassTaps v = class_taps(ry, g.kh, g.sh, g.ph, g.dh), h = class_taps(rx, g.kw, g.sw, g.pw, g.dw);
            GatherMap& m = a.m[n];
            m.PH = ceil_div(g.H - ry, g.sh); m.PW = ceil_div(g.W - rx, g.sw); m.P = g.N * m.PH * m.PW;
            m.th = v.count; m.tw = h.count; m.ntaps = v.count * h.count;
            m.sy = m.sx = 1;
            m.oy0 = v.o0; m.doy = v.d0; m.ox0 = h.o0; m.dox = h.d0;
            m.wt0 = v.k0 * g.kw + h.k0; m.dwi = v.step * g.kw; m.dwj = h.step;
            m.d_phw = FastDiv(m.PH * m.PW); m.d_pw = FastDiv(m.PW);
            a.ry[n] = ry; a.rx[n] = rx;
            ++n;
        }
    total = at;
    return first + n < total;          // classes left for another launch
}

// Every tap reaches class (0, 0) only (1x1 kernels, mostly): the other pixels get zeros, written beside their neighbours.
bool single_class(const ConvGeom& g) {
    if (g.sh == 1 && g.sw == 1) return false;
    for (int r = 1; r < g.sh; ++r) if (class_taps(r, g.kh, g.sh, g.ph, g.dh).count) return false;
    for (int r = 1; r < g.sw; ++r) if (class_taps(r, g.kw, g.sw, g.pw, g.dw).count) return false;
    return true;
}

template <class T, bool FAST, int MODE>
int launch_t(const GxGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kern = adder_gx_gather_kernel<T, FAST, MODE>;
    const int se = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (se != ADDER_OK) return se;
    kern<<<grid, GATHER_THREADS, smem, stream>>>(a);
    return launched();
}

template <bool FAST, int MODE>
int launch_tile(int tile, const GxGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    int i = 0;
#define X(RC, RP, CG, ST, MB, A, M, S, FA, FM, FS) \
    if (tile == i++) {                                                                                        \
        using T = GxTile<RC, RP, CG, ST, MB>;                                                                 \
        if constexpr (MODE != GATHER_TAP_ROWS || T::TAKES_COPY) return launch_t<T, FAST, MODE>(a, grid, smem, stream); \
    }
    ADDER_GX_GATHER_TILES(X)
#undef X
    return ADDER_ERR_INTERNAL;
}

template <bool FAST>
int launch_mode(int mode, int tile, const GxGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    if (mode == GATHER_TAP_ROWS) return launch_tile<FAST, GATHER_TAP_ROWS>(tile, a, grid, smem, stream);
    return mode == GATHER_QUADS ? launch_tile<FAST, GATHER_QUADS>(tile, a, grid, smem, stream) : launch_tile<FAST, GATHER_TAP>(tile, a, grid, smem, stream);
}

int plan(const ConvGeom& g, int first, bool fast, GxGatherArgs& a, dim3& grid, bool& more) {
    const bool single = single_class(g);
    int n, total;
    more = fill_classes(g, first, a, n, total, single);
    a.Ci = g.Ci; a.H = g.H; a.W = g.W; a.Co = g.Co; a.Ho = g.Ho; a.Wo = g.Wo; a.KK = g.kh * g.kw; a.sh = g.sh; a.sw = g.sw;
    const int tile = choose_tile(a, n, g.Ci, fast);
    int most = 0;
    for (int c = 0; c < n; ++c) most = a.m[c].P > most ? a.m[c].P : most;
    grid = dim3((unsigned)ceil_div(most, kTiles[tile].tp), (unsigned)ceil_div(g.Ci, kTiles[tile].tc), (unsigned)n);
    return tile;
}

}  // namespace

// The gradient is read pixel by pixel in order: 1x1 kernels whose class (0, 0) is the output plane.
static bool gx_quads(const ConvGeom& g, const GxGatherArgs& a, const dim3& grid, int first, bool aligned) {
    return g.kh == 1 && g.kw == 1 && g.ph == 0 && g.pw == 0 && a.m[0].PH == g.Ho && a.m[0].PW == g.Wo && grid.z == 1 && first == 0 &&
           (g.Ho * g.Wo) % 4 == 0 && aligned;
}

// w[Co][Ci][KK] -> [KK][Co][Ci]: a block has 64 input channels of one output channel, which are consecutive on both sides.
__global__ void __launch_bounds__(256) by_taps_kernel(const float* __restrict__ w, float* __restrict__ wt, int Co, int Ci, int KK) {
    extern __shared__ float taps[];              // [64][KK]
    const int co = blockIdx.x, ci0 = blockIdx.y * 64, n = min(64, Ci - ci0);
    const float* src = w + ((size_t)co * Ci + ci0) * KK;
    for (int e = threadIdx.x; e < n * KK; e += 256) taps[e] = __ldg(src + e);
    __syncthreads();
    const int c = threadIdx.x & 63;
    if (c < n)
        for (int t = threadIdx.x >> 6; t < KK; t += 4) wt[((size_t)t * Co + co) * Ci + ci0 + c] = taps[c * KK + t];
}

namespace {

// What a launch saves by staging from the copy by taps, as a share of its time and without the copy's own: about the lower quartile of
// 700 layers (2x2 to 7x7 windows, 64-2000 input channels, 25 to 98,000 output positions), measured with and without.  As w lies, a stage's
// weights are 4-byte copies KK words apart: from 9 taps on each fetches a sector of L2 for itself, and the larger w is the less of it
// stays close.  Medians, exact and saturating form: 64 channels x 64 pixels 0.04 and 0.07 at 3x3, 0.17 and 0.24 at 5x5, 0.27 and 0.32 at
// 7x7; 32 x 64 0.05, 0.10; 0.23, 0.29; 0.34, 0.38; 32 x 128 0.01, 0.04; 0.04, 0.10; 0.07, 0.11; 16 x 32 -0.04, 0.01; 0.19, 0.22
// (-0.03 where CTAs have an SM each); 0.25, 0.27.  The other tiles of 8 and 16 channels lose or gain 0.02 at most.
double copy_share(const Tile& t, bool fast, int KK, bool alone) {
    const double nine = t.rp == 8 ? (fast ? 0.04 : 0.025) : alone ? 0.01 : fast ? 0.07 : 0.04;
    const double s = KK < 9 ? 0.015 : KK < 25 ? nine : KK < 49 ? 0.15 : 0.22;
    if (t.rp == 8 && t.tc == 32) return KK < 25 ? (fast ? 0.02 : 0.0) : fast ? 0.09 : 0.035;
    if (t.tc >= 32) return s;
    return takes_copy(t.rc, t.rp, t.tc / t.rc) && KK >= 25 && !alone ? s : 0.0;
}

// Whether the copy pays for itself.  It reads and writes every weight at 2.7 TB/s behind a launch of 4 us, so it takes outputs to share it:
// 2048->2048 7x7 at batch 2 lost 5 % of 1240 us by it, 4096->4096 5x5 at batch 1 20 to 30 %.  256->256 14x14 at batch 256: 2790 -> 2657 us,
// 128->128 56x56 stride 2 at batch 64 783 -> 729, 512->512 14x14 stride 2 771 -> 716, 5x5 256->256 14x14 at batch 16 982 -> 680.  Layers below
// 3e9 terms do without; of 506 measured above that the rule takes 359, none of which loses more than 3 %.  (Classes beyond the first
// launch's, of strides above 3, are not counted.)
bool copy_pays(const ConvGeom& g, const GxGatherArgs& a, int classes, const Tile& t, bool fast) {
    const int sms = sm_count(), KK = g.kh * g.kw;
    const long long tiles = tile_count(a, classes, g.Ci, t);
    int taps = 0;
    for (int c = 0; c < classes; ++c) taps += a.m[c].ntaps;
    const double us = tile_cost(fast ? t.fast : t.exact, tiles, sms) * g.Co * taps / classes / 1965.0;
    return 4.0 + 8.0 * KK * g.Co * g.Ci / 2.7e6 <= copy_share(t, fast, KK, tiles <= sms) * us;
}

}  // namespace

static bool uses_copy(const ConvGeom& g, bool fast) {
    const int KK = g.kh * g.kw;
    const double terms = (double)g.N * g.Ho * g.Wo * g.Co * g.Ci * KK;
    if (KK == 1 || KK > 128 || g.Ci % 4 != 0 || g.Ci > 65535 * 64 || terms < 3e9) return false;
    GxGatherArgs a;
    dim3 grid;
    bool more;
    const int tile = plan(g, 0, fast, a, grid, more);
    return copy_pays(g, a, (int)grid.z, kTiles[tile], fast);
}

// With scratch (staging=tap_rows: the copy by taps is a launch in front).
int describe_gx_gather(const ConvGeom& g, int fast, char* buf, size_t n) {
    GxGatherArgs a;
    dim3 grid;
    bool more;
    const Tile& t = kTiles[plan(g, 0, fast != 0, a, grid, more)];
    const int mode = uses_copy(g, fast != 0) ? GATHER_TAP_ROWS : gx_quads(g, a, grid, 0, true) ? GATHER_QUADS : GATHER_TAP;
    const size_t smem = smem_bytes(t, mode);
    return snprintf(buf, n, "gx gather k=%dx%d fast=%d classes=%u RC=%d RP=%d TC=%d TP=%d staging=%s threads=%d smem=%zu grid=(%u,%u) status=%d",
                    g.kh, g.kw, fast, grid.z, t.rc, t.rp, t.tc, t.tp, staging_name(mode), GATHER_THREADS, smem, grid.x, grid.y,
                    gather_status((int)grid.y, smem));
}

// Bytes of the copy of w by taps; 0 where the layer does without in both forms.
size_t gx_gather_workspace_bytes(const ConvGeom& g) {
    return uses_copy(g, false) || uses_copy(g, true) ? (size_t)g.kh * g.kw * g.Co * g.Ci * sizeof(float) : 0;
}

int launch_gx_gather(const ConvGeom& g, const float* gout, const float* x, const float* w, float* gx, int fast, int accumulate,
                     cudaStream_t stream, void* workspace, size_t workspace_bytes) {
    float* by_taps = nullptr;
    if (workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0 && uses_copy(g, fast != 0) &&
        workspace_bytes >= (size_t)g.kh * g.kw * g.Co * g.Ci * sizeof(float)) {
        by_taps = static_cast<float*>(workspace);
        by_taps_kernel<<<dim3((unsigned)g.Co, (unsigned)ceil_div(g.Ci, 64)), 256, (size_t)64 * g.kh * g.kw * sizeof(float), stream>>>(w, by_taps, g.Co, g.Ci, g.kh * g.kw);
        const int st = launched();
        if (st != ADDER_OK) return st;
    }
    bool more = true;
    for (int first = 0; more; first += MAX_CLASSES) {
        GxGatherArgs a;
        dim3 grid;
        const int tile = plan(g, first, fast != 0, a, grid, more);
        a.gout = gout; a.x = x; a.w = w; a.gx = gx; a.accumulate = accumulate;
        const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gx)) & 15) == 0;
        const bool unit = g.sh == 1 && g.sw == 1;
        a.vec_io = unit && (g.H * g.W) % 4 == 0 && aligned;
        const bool copied = by_taps != nullptr && takes_copy(kTiles[tile].rc, kTiles[tile].rp, kTiles[tile].tc / kTiles[tile].rc);
        if (copied) a.w = by_taps;
        a.w_quads = a.KK == 1 && g.Ci % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
        a.fill_block = single_class(g) && !accumulate;
        a.fill_quads = a.fill_block && g.sh == 2 && g.sw == 2 && g.W == 2 * a.m[0].PW && g.H == 2 * a.m[0].PH && a.m[0].PW % 4 == 0 &&
                       (reinterpret_cast<uintptr_t>(gx) & 15) == 0;
        // (planes of an odd height keep an even number of values, so that every plane starts aligned)
        a.fill_pairs = a.fill_block && !a.fill_quads && g.sh == 2 && g.sw == 2 && g.W % 2 == 0 && (reinterpret_cast<uintptr_t>(gx) & 7) == 0;
        const bool quads = gx_quads(g, a, grid, first, (reinterpret_cast<uintptr_t>(gout) & 15) == 0);
        const int mode = copied ? GATHER_TAP_ROWS : quads ? GATHER_QUADS : GATHER_TAP;
        const int rows = stage_rows(kTiles[tile], mode);
        a.CK = g.Co < rows ? g.Co : rows;      // full blocks have the cheaper staging loops, so one ragged block rather than even ones
        const size_t smem = smem_bytes(kTiles[tile], mode);
        if (gather_status((int)grid.y, smem) != ADDER_OK) return ADDER_ERR_UNSUPPORTED;
        const int st = fast ? launch_mode<true>(mode, tile, a, grid, smem, stream) : launch_mode<false>(mode, tile, a, grid, smem, stream);
        if (st != ADDER_OK) return st;
    }
    return ADDER_OK;
}

}  // namespace adder
