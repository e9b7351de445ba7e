// Forward adder convolution as a channels x pixels tile with a gathered pixel operand (gather.cuh): 1x1 layers, and every
// kernel extent, stride, padding and dilation.
//
// A thread owns RM output channels x 8 pixels (two quads, half a tile apart, so that the 128-bit loads of eight
// neighbouring threads are consecutive); the four channel groups of a warp read the same pixels and its eight pixel groups the
// same weights, so a k step is four 128-bit loads for 64 terms.  The inner loop is that of adder_fwd_kernel: one packed
// subtract per two terms, then two adds of |d|; it is bound by the FP32 pipe (2 slots a term) and runs at 2.2-2.4 lane
// cycles a term.
#include <cstdio>
#include "common.cuh"
#include "gather.cuh"
#include "kernels.h"

namespace adder {

struct FwdGatherArgs {
    GatherMap m;
    const float* x;
    const float* w;
    float* out;
    Epilogue ep;
    int Ci, H, W, Co, KK, CK, nchunks;
    int vec_w;               // rows of w are whole, aligned quads in the order of the reduction
    int vec_store;           // planes are whole quads, `out` and the residual 16-byte aligned
};

// Tiles that may take the weights as they lie (ROWS), where rows of w are whole aligned quads: 16-byte copies instead of four times as many
// that transpose, 5 to 9 % of a tile of 16 x 4 channels (512->512 7x7 3x3 at batch 64: 697 -> 639 us, 512->128 28x28: 250 -> 232).
// Tiles of fewer channels spend their staging on pixels and gain nothing; eight channels a thread have no registers for several steps of
// each at a time and lose 1 to 6 %.
__host__ __device__ constexpr bool takes_rows(int rm, int cg) { return rm == 4 && cg == 16; }

// RM channels x RP pixels per thread (RP = 8: two quads half a tile apart), CG channel groups, ST stages, MB CTAs per SM.
template <int RM_, int RP_, int CG_, int ST_, int MB_>
struct FwdTile {
    static constexpr int RM = RM_, RP = RP_, CG = CG_, ST = ST_, MB = MB_;
    static constexpr int PG = GATHER_THREADS / CG, TC = CG * RM, TP = PG * RP, WP = TC + 4;
    static constexpr int PQ = RP == 8 ? 4 : RP;                 // consecutive pixels of a thread
    static constexpr bool THIN = RM <= 2 && RP <= 2, TAKES_ROWS = takes_rows(RM, CG);
};

// ROWS: weights [channel][step], the floats of a row.  The 18 steps of two channels of a 3x3 window come as the 80 aligned bytes around
// them: they start at the third float for every other pair of channels.
__host__ __device__ constexpr int weight_row(int mode, int rows) { return mode == GATHER_NINE_ROWS ? 20 : rows; }

template <class T, int MODE>
__global__ void __launch_bounds__(GATHER_THREADS, T::MB) adder_fwd_gather_kernel(const __grid_constant__ FwdGatherArgs a) {
    constexpr int RM = T::RM, RP = T::RP, CG = T::CG, TC = T::TC, TP = T::TP, WP = T::WP, PQ = T::PQ, ST = T::ST;
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;
    constexpr int CK = gather_rows(MODE, ST, TC, TP, 0, T::MB, T::THIN);      // rows of a stage
    constexpr bool NINE = MODE == GATHER_NINE || MODE == GATHER_NINE_ROWS, ROWS = MODE == GATHER_QUADS_ROWS || MODE == GATHER_NINE_ROWS;
    constexpr int XS = CK * TP, WK = weight_row(MODE, CK), WS = ROWS ? TC * WK : CK * WP;
    extern __shared__ __align__(16) float smem[];
    float* const Xs = smem;
    float* const Ws = smem + ST * XS;

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int cg = (wid % (CG / 4)) * 4 + (lane >> 3), pg = (wid / (CG / 4)) * 8 + (lane & 7);
    const int p0 = blockIdx.x * TP, co0 = blockIdx.y * TC;
    const size_t image = (size_t)a.Ci * a.H * a.W;

    GatherPixel px[COLS];
    constexpr int CH = nine_channels(T::THIN);
    GatherNine<TP, CH> nine;
    if (MODE == GATHER_QUADS || MODE == GATHER_QUADS_ROWS) {
        px[0].decode(a.m, a.x, p0 + 4 * (tid % (TP / 4)), image);
        px[0].base += px[0].row * a.W + px[0].col;
    } else {
#pragma unroll
        for (int q = 0; q < COLS; ++q) px[q].decode(a.m, a.x, p0 + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP), image);
        if (NINE) nine.init(px, a.m, a.H, a.W, tid);
    }
    GatherChunk fc;              // position of the next chunk to stage
    const int ck4 = round_up(a.CK, 4);
    auto fill = [&](int stage) {
        int nk, rows, wk;        // reduction steps that exist, rows to stage, and the first one's weight index
        int nk2 = 0, wk2 = 0;    // GATHER_HALVES: of the second block
        if constexpr (NINE) {
            const int nch = min(CH, a.Ci - fc.c0);
            nine.fill(Xs + stage * XS, px, a.m, fc.c0, nch, a.H, a.W, tid);
            nk = nch * 9; rows = CK; wk = fc.c0 * 9;
        } else {
            nk = min(a.CK, a.Ci - fc.c0); rows = ck4;
            if (MODE == GATHER_QUADS || MODE == GATHER_QUADS_ROWS) gather_quads<TP, CK>(Xs + stage * XS, px[0].base, px[0].ok, a.x, fc.c0, nk, ck4, a.H * a.W, tid);
            else gather_pixels<TP, MODE == GATHER_HALVES ? GATHER_CK : CK>(Xs + stage * XS, px, a.x, a.m, fc, nk, ck4, a.H, a.W, tid);
            wk = fc.c0 * a.KK + a.m.wt0 + fc.i * a.m.dwi + fc.j * a.m.dwj;
            if constexpr (MODE == GATHER_HALVES) {
                fc.next(a.m, GATHER_CK);
                GatherChunk f2 = fc;
                if (fc.c0 >= a.Ci) f2.c0 = 0;                    // none left: zeros, from an address within the tensor
                else { nk2 = min(GATHER_CK, a.Ci - fc.c0); wk2 = fc.c0 * a.KK + a.m.wt0 + fc.i * a.m.dwi + fc.j * a.m.dwj; }
                gather_pixels<TP>(Xs + stage * XS + GATHER_CK * TP, px, a.x, a.m, f2, nk2, GATHER_CK, a.H, a.W, tid);
            }
        }
        const int kstep = NINE ? 1 : a.KK, row = a.Ci * a.KK;
        if constexpr (ROWS) {
            constexpr int WQ = WK / 4;               // 16-byte words of a row
            const float* wsrc = a.w + (co0 * row + (NINE ? wk - (fc.c0 & 2) : wk));
#pragma unroll
            for (int i0 = 0; i0 < TC * WQ; i0 += GATHER_THREADS) {
                const int c = (i0 + tid) / WQ, k = (i0 + tid) % WQ * 4;
                if ((TC * WQ) % GATHER_THREADS != 0 && c >= TC) break;
                const bool ok = co0 + c < a.Co && (NINE || k < nk);
                cp_async16(Ws + stage * WS + c * WK + k, ok ? wsrc + (c * row + k) : a.w, ok);
            }
        } else if constexpr (T::THIN) {
            // weights [output channel of the tile][reduction step]: a thread copies 4 steps
#pragma unroll
            for (int i0 = 0; i0 < TC * CK / 4; i0 += GATHER_THREADS) {
                const int c = (i0 + tid) / (CK / 4), k = (i0 + tid) % (CK / 4) * 4;
                if ((TC * CK / 4) % GATHER_THREADS != 0 && c >= TC) break;
                float* ws = Ws + stage * WS + c * (CK + 4) + k;
                const bool okc = co0 + c < a.Co;
                const bool second = MODE == GATHER_HALVES && k >= GATHER_CK;
                const int kr = second ? k - GATHER_CK : k, nkr = second ? nk2 : nk;
                const float* wsrc = a.w + (okc ? (co0 + c) * row + (second ? wk2 : wk) : 0);
                if (MODE != GATHER_HALVES && a.vec_w) {
                    const bool ok = okc & (kr < nkr);
                    cp_async16(ws, ok ? wsrc + kr : a.w, ok);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool ok = okc & (kr + i < nkr);
                        cp_async4(ws + i, ok ? wsrc + (kr + i) * kstep : a.w, ok);
                    }
                }
            }
        } else {
            // weights [reduction step][output channel of the tile]: a warp copies 8 steps of 4 outputs
            const int k8 = tid & 7, c4 = tid >> 3;
            float* ws = Ws + stage * WS + k8 * WP + c4;
            const int ncol = a.Co - co0 - c4;
            const float* wsrc = a.w + ((co0 + c4) * row + k8 * kstep + wk);
#pragma unroll
            for (int kb = 0; kb < CK; kb += 8) {
                if (kb + k8 >= rows) break;
                const bool okk = kb + k8 < nk;
#pragma unroll
                for (int c = 0; c < TC; c += GATHER_THREADS / 8) {
                    if (TC % (GATHER_THREADS / 8) != 0 && c + c4 >= TC) break;
                    const bool ok = okk & (c < ncol);
                    cp_async4(ws + kb * WP + c, ok ? wsrc + (c * row + kb * kstep) : a.w, ok);
                }
            }
        }
        if (NINE) fc.c0 += CH;
        else fc.next(a.m, a.CK);
    };

    float acc[RM][RP];
#pragma unroll
    for (int m = 0; m < RM; ++m)
#pragma unroll
        for (int j = 0; j < RP; ++j) acc[m][j] = 0.f;

#pragma unroll 1
    for (int s = 0; s < ST - 1; ++s) {
        if (s < a.nchunks) fill(s);
        cp_async_commit();
    }
    GatherChunk cc;
    int stage = 0, fstage = ST - 1;
#pragma unroll 1
    for (int c = 0; c < a.nchunks; ++c) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (c + ST - 1 < a.nchunks) fill(fstage);
        cp_async_commit();
        const float* xs = Xs + stage * XS + pg * PQ;
        const int nk = NINE || MODE == GATHER_HALVES ? CK : min(ck4, round_up(a.Ci - cc.c0, 4));
        if constexpr (T::THIN) {
            const float* ws = Ws + stage * WS + cg * RM * (CK + 4);
#pragma unroll (RM == 1 ? CK / 4 : 2)
            for (int k = 0; k < CK; k += 4) {
                if (MODE != GATHER_NINE && MODE != GATHER_HALVES && k >= nk) break;
                float4 wq[RM];
                float xv[4][RP];
#pragma unroll
                for (int m = 0; m < RM; ++m) wq[m] = *reinterpret_cast<const float4*>(ws + m * (CK + 4) + k);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if constexpr (RP == 2) {
                        const float2 q = *reinterpret_cast<const float2*>(xs + (k + i) * TP);
                        xv[i][0] = q.x; xv[i][1] = q.y;
                    } else {
                        xv[i][0] = xs[(k + i) * TP];
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int m = 0; m < RM; ++m) {
                        const float wv = i == 0 ? wq[m].x : i == 1 ? wq[m].y : i == 2 ? wq[m].z : wq[m].w;
#pragma unroll
                        for (int j = 0; j < RP; ++j) acc[m][j] += fabsf(wv - xv[i][j]);
                    }
            }
        } else if constexpr (ROWS) {
            // SW steps a load of w; pairs of pixels, as two channels of a step are not neighbours here
            constexpr int SW = NINE ? 2 : 4;
            const float* ws = Ws + stage * WS + cg * RM * WK + (NINE ? 2 * (c & 1) : 0);
#pragma unroll 1
            for (int k = 0; k < nk; k += SW) {
                float wv[RM][SW];
#pragma unroll
                for (int m = 0; m < RM; ++m) {
                    if constexpr (SW == 4) {
                        const float4 q = *reinterpret_cast<const float4*>(ws + m * WK + k);
                        wv[m][0] = q.x; wv[m][1] = q.y; wv[m][2] = q.z; wv[m][3] = q.w;
                    } else {
                        const float2 q = *reinterpret_cast<const float2*>(ws + m * WK + k);
                        wv[m][0] = q.x; wv[m][1] = q.y;
                    }
                }
#pragma unroll
                for (int i = 0; i < SW; ++i) {
                    uint64_t x2[RP / 2];
#pragma unroll
                    for (int h = 0; h < RP / PQ; ++h) {
                        const float4 q = *reinterpret_cast<const float4*>(xs + (k + i) * TP + h * (TP / 2));
                        x2[2 * h] = pack2(q.x, q.y); x2[2 * h + 1] = pack2(q.z, q.w);
                    }
#pragma unroll
                    for (int m = 0; m < RM; ++m) {
                        const uint64_t nw2 = pack2(-wv[m][i], -wv[m][i]);
#pragma unroll
                        for (int j = 0; j < RP / 2; ++j) {
                            float d0, d1;
                            unpack2(add2(x2[j], nw2), d0, d1);
                            acc[m][2 * j] += fabsf(d0);
                            acc[m][2 * j + 1] += fabsf(d1);
                        }
                    }
                }
            }
        } else {
            const float* ws = Ws + stage * WS + cg * RM;
#pragma unroll (RM * RP >= 64 ? 1 : RM * RP >= 32 ? 2 : 4)
            for (int k = 0; k < nk; ++k) {
                float xv[RP], wv[RM];
#pragma unroll
                for (int h = 0; h < RP / PQ; ++h) {
                    const float4 q = *reinterpret_cast<const float4*>(xs + k * TP + h * (TP / 2));
                    xv[4 * h] = q.x; xv[4 * h + 1] = q.y; xv[4 * h + 2] = q.z; xv[4 * h + 3] = q.w;
                }
                if constexpr (RM >= 4) {
#pragma unroll
                    for (int m = 0; m < RM; m += 4) {
                        const float4 q = *reinterpret_cast<const float4*>(ws + k * WP + m);
                        wv[m] = q.x; wv[m + 1] = q.y; wv[m + 2] = q.z; wv[m + 3] = q.w;
                    }
                } else {
                    const float2 q = *reinterpret_cast<const float2*>(ws + k * WP);
                    wv[0] = q.x; wv[1] = q.y;
                }
                uint64_t nx2[RP];
#pragma unroll
                for (int j = 0; j < RP; ++j) nx2[j] = pack2(-xv[j], -xv[j]);
#pragma unroll
                for (int m = 0; m < RM; m += 2) {
                    const uint64_t w2 = pack2(wv[m], wv[m + 1]);
#pragma unroll
                    for (int j = 0; j < RP; ++j) {
                        float d0, d1;
                        unpack2(add2(w2, nx2[j]), d0, d1);
                        acc[m][j] += fabsf(d0);
                        acc[m + 1][j] += fabsf(d1);
                    }
                }
            }
        }
        if (!NINE) cc.next(a.m, a.CK);
        if (++stage == ST) stage = 0;
        if (++fstage == ST) fstage = 0;
    }

    const int PHW = a.m.PH * a.m.PW;
#pragma unroll
    for (int h = 0; h < RP / PQ; ++h) {
        const int p = p0 + h * (TP / 2) + pg * PQ;
        if constexpr (PQ == 4) {
            if (a.vec_store) {
                if (p >= a.m.P) continue;
                uint32_t n, r;
                a.m.d_phw.divmod(p, n, r);
                const int c0 = co0 + cg * RM;
                const size_t at = ((size_t)n * a.Co + c0) * PHW + r;
#pragma unroll
                for (int m = 0; m < RM; ++m) {
                    if (c0 + m >= a.Co) break;
                    const float4 y = make_float4(-acc[m][4 * h], -acc[m][4 * h + 1], -acc[m][4 * h + 2], -acc[m][4 * h + 3]);
                    *reinterpret_cast<float4*>(a.out + at + (size_t)m * PHW) = finish(a.ep, y, c0 + m, at + (size_t)m * PHW);
                }
                continue;
            }
        }
#pragma unroll
        for (int j = 0; j < PQ; ++j) {
            if (p + j >= a.m.P) continue;
            uint32_t n, r;
            a.m.d_phw.divmod(p + j, n, r);
            const int c0 = co0 + cg * RM;
            const size_t at = ((size_t)n * a.Co + c0) * PHW + r;
#pragma unroll
            for (int m = 0; m < RM; ++m) {
                if (c0 + m >= a.Co) break;
                a.out[at + (size_t)m * PHW] = finish(a.ep, -acc[m][PQ * h + j], c0 + m, at + (size_t)m * PHW);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

namespace {

// The tiles: large ones have the fewest loads per term, small ones give a small layer more threads.  The last three (THIN) are
// bound by the instructions around a term in a CTA's chain of stages, few CTAs being resident: they keep their weights as
// [channel][step], which takes 16-byte copies and gives four steps a load, and have stages twice as long.  At batch 1, with the
// 2x2 tiles built like the large ones -> now: 64->64 8x8 14.1 -> 7.5 us, 256->256 14x14 52 -> 43.5, 512->512 7x7 102 -> 63,
// 1024->256 14x14 33 -> 22, 2048->512 7x7 69 -> 41.
// X(RM, RP, CG, ST, MB, clocks per step: alone, each further CTA, throughput)
#define ADDER_FWD_GATHER_TILES(X)                                                                                   \
    X(8, 8, 8, 2, 4, 242, 147, 173) X(8, 8, 16, 2, 4, 241, 74, 186) X(8, 8, 4, 2, 4, 278, 130, 186)                 \
    X(4, 8, 16, 3, 4, 139, 65, 93) X(4, 8, 8, 3, 4, 139, 65, 93) X(4, 8, 4, 2, 4, 174, 76, 109)                     \
    X(4, 4, 16, 4, 6, 92, 30, 54) X(4, 4, 8, 4, 6, 92, 30, 54) X(4, 4, 4, 4, 6, 101, 22, 56)                        \
    X(2, 8, 4, 3, 6, 110, 75, 81) X(2, 2, 8, 4, 8, 35, 10, 20) X(2, 2, 4, 4, 6, 38, 12, 23) X(1, 1, 4, 6, 8, 16, 9, 11)

struct Tile { int rm, rp, cg, st, mb, tc, tp; TileCost cost; };
constexpr Tile kTiles[] = {
#define X(RM, RP, CG, ST, MB, A, M, S) {RM, RP, CG, ST, MB, RM * CG, RP * GATHER_THREADS / CG, {A, M, S}},
    ADDER_FWD_GATHER_TILES(X)
#undef X
};

// `rows`: the layer's weights can be staged as they lie (row_layer), which takes 5 % off what a tile costs that profits: 500 layers whose
// tile, or kernel, that changes gain 3.7 %, 9 of them lose more than 5 %, 12 % at worst (taking nothing off beyond 8 CTAs an SM halves the
// losers and a part of the gains: the same sum).  Without aligned operands nothing is taken off: 944->144 22x22 1x1 at batch 19 then runs
// the other tile, 136 -> 126 us.
int choose_tile(int P, int Co, bool rows) {
    int best = 0;
    double best_cost = 1e300;
    const int sms = sm_count();
    for (int i = 0; i < (int)(sizeof(kTiles) / sizeof(kTiles[0])); ++i) {
        const Tile& t = kTiles[i];
        const double cost = tile_cost(t.cost, (long long)ceil_div(P, t.tp) * ceil_div(Co, t.tc), sms) * (rows && takes_rows(t.rm, t.cg) ? 0.95 : 1.0);
        if (cost < best_cost) { best_cost = cost; best = i; }
    }
    return best;
}

// 16-byte alignment of the operands.
struct Aligned { bool x, w; };

// Layers whose weights can be staged as they lie: 3x3, and 1x1 whose pixels are the input's in order and come in quads.
bool row_layer(const ConvGeom& g, Aligned al) {
    const bool in_order = g.kh * g.kw == 1 && g.sh == 1 && g.sw == 1 && g.ph == 0 && g.pw == 0 && (g.Ho * g.Wo) % 4 == 0 && al.x;
    const int K = g.Ci * g.kh * g.kw;            // (a row of fewer steps is mostly padding of the stage: 4->336 16x16 at batch 11 3.0 -> 3.4 us)
    return al.w && K % 4 == 0 && K >= 32 && (in_order || (g.kh == 3 && g.kw == 3));
}

bool thin(const Tile& t) { return t.rm <= 2 && t.rp <= 2; }
int stage_rows(const Tile& t, int mode) { return gather_rows(mode, t.st, t.tc, t.tp, 0, t.mb, thin(t)); }

size_t smem_bytes(const Tile& t, int mode) {
    const int rows = stage_rows(t, mode);
    return (size_t)t.st * (rows * t.tp + (mode > GATHER_HALVES ? t.tc * weight_row(mode, rows) : rows * (t.tc + 4))) * sizeof(float);
}

GatherMap fwd_map(const ConvGeom& g) {
    GatherMap m;
    m.PH = g.Ho; m.PW = g.Wo; m.P = g.N * g.Ho * g.Wo;
    m.th = g.kh; m.tw = g.kw; m.ntaps = g.kh * g.kw;
    m.sy = g.sh; m.sx = g.sw;
    m.oy0 = -g.ph; m.doy = g.dh; m.ox0 = -g.pw; m.dox = g.dw;
    m.wt0 = 0; m.dwi = g.kw; m.dwj = 1;
    m.d_phw = FastDiv(g.Ho * g.Wo); m.d_pw = FastDiv(g.Wo);
    return m;
}

template <class T, int MODE>
int launch_t(const FwdGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kern = adder_fwd_gather_kernel<T, MODE>;
    const int se = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (se != ADDER_OK) return se;
    kern<<<grid, GATHER_THREADS, smem, stream>>>(a);
    return launched();
}

template <int MODE>
int launch_mode(int tile, const FwdGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    int i = 0;
#define X(RM, RP, CG, ST, MB, A, M, S) \
    if (tile == i++) {                                                                                 \
        using T = FwdTile<RM, RP, CG, ST, MB>;                                                         \
        if constexpr (MODE == GATHER_HALVES ? T::THIN : MODE < GATHER_HALVES || T::TAKES_ROWS) return launch_t<T, MODE>(a, grid, smem, stream); \
    }
    ADDER_FWD_GATHER_TILES(X)
#undef X
    return ADDER_ERR_INTERNAL;
}

}  // namespace

double fwd_gather_clocks(const ConvGeom& g, bool w_aligned) {
    const int P = g.N * g.Ho * g.Wo;
    const bool rows = row_layer(g, {true, w_aligned});
    const Tile& t = kTiles[choose_tile(P, g.Co, rows)];
    return tile_cost(t.cost, (long long)ceil_div(P, t.tp) * ceil_div(g.Co, t.tc), sm_count()) * (rows && takes_rows(t.rm, t.cg) ? 0.95 : 1.0);
}

static int fwd_mode(const ConvGeom& g, const Tile& t, Aligned al) {
    const bool rows = row_layer(g, al) && takes_rows(t.rm, t.cg);
    if (g.kh == 3 && g.kw == 3) return rows ? GATHER_NINE_ROWS : GATHER_NINE;
    const bool in_order = g.kh * g.kw == 1 && g.sh == 1 && g.sw == 1 && g.ph == 0 && g.pw == 0;
    if (!in_order || !al.x || (g.Ho * g.Wo) % 4 != 0) return GATHER_TAP;
    return rows ? GATHER_QUADS_ROWS : GATHER_QUADS;
}

int describe_fwd_gather(const ConvGeom& g, bool aligned, char* buf, size_t n) {
    const int P = g.N * g.Ho * g.Wo;
    const Aligned al{aligned, aligned};
    const Tile& t = kTiles[choose_tile(P, g.Co, row_layer(g, al))];
    const int mode = fwd_mode(g, t, al);
    const size_t smem = smem_bytes(t, mode);
    return snprintf(buf, n, "fwd gather k=%dx%d RM=%d RP=%d TC=%d TP=%d staging=%s threads=%d smem=%zu grid=(%d,%d) status=%d", g.kh, g.kw, t.rm,
                    t.rp, t.tc, t.tp, staging_name(mode), GATHER_THREADS, smem, ceil_div(P, t.tp), ceil_div(g.Co, t.tc), gather_status(ceil_div(g.Co, t.tc), smem));
}

int launch_fwd_gather(const ConvGeom& g, const float* x, const float* w, float* out, cudaStream_t stream, const Epilogue& ep) {
    FwdGatherArgs a;
    a.m = fwd_map(g);
    a.x = x; a.w = w; a.out = out; a.ep = ep;
    a.Ci = g.Ci; a.H = g.H; a.W = g.W; a.Co = g.Co; a.KK = g.kh * g.kw;
    const bool whole_quads = (g.Ho * g.Wo) % 4 == 0;
    const Aligned al{(reinterpret_cast<uintptr_t>(x) & 15) == 0, (reinterpret_cast<uintptr_t>(w) & 15) == 0};
    a.vec_w = (a.KK == 1 || (g.kh == 3 && g.kw == 3)) && (g.Ci * a.KK) % 4 == 0 && al.w;
    a.vec_store = whole_quads && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(ep.residual)) & 15) == 0;
    const int tile = choose_tile(a.m.P, g.Co, row_layer(g, al));
    const Tile& t = kTiles[tile];
    const int mode = fwd_mode(g, t, al);
    const int rows = stage_rows(t, mode);
    // Windows of several taps are added up in the order (block of 16 channels, tap, channel) by every tile: the tile follows the batch,
    // and an image's result must not.  A thin tile, whose stages have 32 rows, takes two such blocks a stage.
    const bool halves = mode == GATHER_TAP && a.KK > 1 && g.Ci > GATHER_CK && rows > GATHER_CK;
    const bool nine = mode == GATHER_NINE || mode == GATHER_NINE_ROWS;
    a.CK = nine ? rows / 9 : halves ? GATHER_CK : g.Ci < rows ? g.Ci : rows;      // full blocks have the cheaper staging loops
    a.nchunks = ceil_div(g.Ci, a.CK) * (nine ? 1 : a.KK);
    if (halves) a.nchunks = ceil_div(a.nchunks, 2);
    const dim3 grid((unsigned)ceil_div(a.m.P, t.tp), (unsigned)ceil_div(g.Co, t.tc));
    const size_t smem = smem_bytes(t, mode);
    if (gather_status((int)grid.y, smem) != ADDER_OK) return ADDER_ERR_UNSUPPORTED;
    if (mode == GATHER_NINE) return launch_mode<GATHER_NINE>(tile, a, grid, smem, stream);
    if (mode == GATHER_NINE_ROWS) return launch_mode<GATHER_NINE_ROWS>(tile, a, grid, smem, stream);
    if (mode == GATHER_QUADS_ROWS) return launch_mode<GATHER_QUADS_ROWS>(tile, a, grid, smem, stream);
    if (halves) return launch_mode<GATHER_HALVES>(tile, a, grid, smem, stream);
    return mode == GATHER_QUADS ? launch_mode<GATHER_QUADS>(tile, a, grid, smem, stream) : launch_mode<GATHER_TAP>(tile, a, grid, smem, stream);
}

}  // namespace adder
