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
    double* stats;           // optional [Co][gridDim.x][2]: per pixel tile, the sum of its outputs and of their squares
    int Ci, H, W, Co, KK, CK, nchunks;
    int vec_store;           // planes are whole quads and `out` is 16-byte aligned
};

template <int RM, int CG, bool QUADS>
__global__ void __launch_bounds__(GATHER_THREADS, 4) adder_fwd_gather_kernel(const __grid_constant__ FwdGatherArgs a) {
    constexpr int PG = GATHER_THREADS / CG, TC = CG * RM, TP = PG * 8, WP = TC + 4;
    constexpr int COLS = TP > GATHER_THREADS ? TP / GATHER_THREADS : 1;
    constexpr int XS = GATHER_CK * TP, WS = GATHER_CK * WP;
    extern __shared__ __align__(16) float smem[];
    float* const Xs = smem;
    float* const Ws = smem + GATHER_STAGES * XS;

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int cg = (wid % (CG / 4)) * 4 + (lane >> 3), pg = (wid / (CG / 4)) * 8 + (lane & 7);
    const int p0 = blockIdx.x * TP, co0 = blockIdx.y * TC;
    const size_t image = (size_t)a.Ci * a.H * a.W;

    GatherPixel px[COLS];
    if (QUADS) {
        px[0].decode(a.m, a.x, p0 + 4 * (tid % (TP / 4)), image);
        px[0].base += px[0].row * a.W + px[0].col;
    } else {
#pragma unroll
        for (int q = 0; q < COLS; ++q) px[q].decode(a.m, a.x, p0 + (COLS > 1 ? tid + q * GATHER_THREADS : tid % TP), image);
    }
    GatherChunk fc;              // position of the next chunk to stage
    const int ck4 = round_up(a.CK, 4);
    auto fill = [&](int stage) {
        const int nch = min(a.CK, a.Ci - fc.c0);
        if (QUADS) gather_quads<TP>(Xs + stage * XS, px[0].base, px[0].ok, a.x, fc.c0, nch, ck4, a.H * a.W, tid);
        else gather_pixels<TP>(Xs + stage * XS, px, a.x, a.m, fc, nch, ck4, a.H, a.W, tid);
        // weights [input channel of the chunk][output channel of the tile]: a warp copies 8 channels of 4 outputs
        const int k8 = tid & 7, c4 = tid >> 3;
        float* ws = Ws + stage * WS + k8 * WP + c4;
        const int row = a.Ci * a.KK, ncol = a.Co - co0 - c4;
        const float* wsrc = a.w + ((co0 + c4) * row + (fc.c0 + k8) * a.KK + a.m.wt0 + fc.i * a.m.dwi + fc.j * a.m.dwj);
#pragma unroll
        for (int kb = 0; kb < GATHER_CK; kb += 8) {
            if (kb + k8 >= ck4) break;
            const bool okk = kb + k8 < nch;
#pragma unroll
            for (int c = 0; c < TC; c += GATHER_THREADS / 8) {
                const bool ok = okk & (c < ncol);
                cp_async4(ws + kb * WP + c, ok ? wsrc + (c * row + kb * a.KK) : a.w, ok);
            }
        }
        fc.next(a.m, a.CK);
    };

    float acc[RM][8];
#pragma unroll
    for (int m = 0; m < RM; ++m)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[m][j] = 0.f;

#pragma unroll
    for (int s = 0; s < GATHER_STAGES - 1; ++s) {
        if (s < a.nchunks) fill(s);
        cp_async_commit();
    }
    GatherChunk cc;
    int stage = 0, fstage = GATHER_STAGES - 1;
    for (int c = 0; c < a.nchunks; ++c) {
        cp_async_wait<GATHER_STAGES - 2>();
        __syncthreads();
        if (c + GATHER_STAGES - 1 < a.nchunks) fill(fstage);
        cp_async_commit();
        const float* xs = Xs + stage * XS + pg * 4;
        const float* ws = Ws + stage * WS + cg * RM;
        const int nk = min(ck4, round_up(a.Ci - cc.c0, 4));
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            float xv[8], wv[RM];
            {
                const float4 q0 = *reinterpret_cast<const float4*>(xs + k * TP);
                const float4 q1 = *reinterpret_cast<const float4*>(xs + k * TP + TP / 2);
                xv[0] = q0.x; xv[1] = q0.y; xv[2] = q0.z; xv[3] = q0.w; xv[4] = q1.x; xv[5] = q1.y; xv[6] = q1.z; xv[7] = q1.w;
            }
#pragma unroll
            for (int m = 0; m < RM; m += 4) {
                const float4 q = *reinterpret_cast<const float4*>(ws + k * WP + m);
                wv[m] = q.x; wv[m + 1] = q.y; wv[m + 2] = q.z; wv[m + 3] = q.w;
            }
            uint64_t nx2[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) nx2[j] = pack2(-xv[j], -xv[j]);
#pragma unroll
            for (int m = 0; m < RM; m += 2) {
                const uint64_t w2 = pack2(wv[m], wv[m + 1]);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float d0, d1;
                    unpack2(add2(w2, nx2[j]), d0, d1);
                    acc[m][j] += fabsf(d0);
                    acc[m + 1][j] += fabsf(d1);
                }
            }
        }
        cc.next(a.m, a.CK);
        if (++stage == GATHER_STAGES) stage = 0;
        if (++fstage == GATHER_STAGES) fstage = 0;
    }

    const int PHW = a.m.PH * a.m.PW;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = p0 + h * (TP / 2) + pg * 4;
        if (a.vec_store) {
            if (p >= a.m.P) continue;
            uint32_t n, r;
            a.m.d_phw.divmod(p, n, r);
            float* o = a.out + ((size_t)n * a.Co + co0 + cg * RM) * PHW + r;
#pragma unroll
            for (int m = 0; m < RM; ++m) {
                if (co0 + cg * RM + m >= a.Co) break;
                *reinterpret_cast<float4*>(o + (size_t)m * PHW) =
                    make_float4(-acc[m][4 * h], -acc[m][4 * h + 1], -acc[m][4 * h + 2], -acc[m][4 * h + 3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (p + j >= a.m.P) continue;
                uint32_t n, r;
                a.m.d_phw.divmod(p + j, n, r);
                float* o = a.out + ((size_t)n * a.Co + co0 + cg * RM) * PHW + r;
#pragma unroll
                for (int m = 0; m < RM; ++m) {
                    if (co0 + cg * RM + m >= a.Co) break;
                    o[(size_t)m * PHW] = -acc[m][4 * h + j];
                }
            }
        }
    }
    if (a.stats == nullptr) return;

    // Batch-norm statistics of this pixel tile, as in adder_fwd_kernel: at most 8 values per thread and channel in fp32, then
    // double in a fixed order.
    __syncthreads();                                        // the stages are free
    float2* st = reinterpret_cast<float2*>(smem);           // [TC][PG + 1]
#pragma unroll
    for (int m = 0; m < RM; ++m) {
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (p0 + (j >> 2) * (TP / 2) + pg * 4 + (j & 3) < a.m.P) { s -= acc[m][j]; q = fmaf(acc[m][j], acc[m][j], q); }
        st[(cg * RM + m) * (PG + 1) + pg] = make_float2(s, q);
    }
    __syncthreads();
    constexpr int TPC = GATHER_THREADS / TC >= 32 ? 32 : (GATHER_THREADS / TC < 1 ? 1 : GATHER_THREADS / TC);   // threads per channel
    const int ch = tid / TPC, l = tid % TPC;
    double ds = 0.0, dq = 0.0;
    if (ch < TC)
        for (int e = l; e < PG; e += TPC) { const float2 v = st[ch * (PG + 1) + e]; ds += (double)v.x; dq += (double)v.y; }
#pragma unroll
    for (int off = TPC >> 1; off > 0; off >>= 1) {
        ds += __shfl_xor_sync(0xffffffffu, ds, off);
        dq += __shfl_xor_sync(0xffffffffu, dq, off);
    }
    if (l == 0 && ch < TC && co0 + ch < a.Co) {
        double* o = a.stats + ((size_t)(co0 + ch) * gridDim.x + blockIdx.x) * 2;
        o[0] = ds; o[1] = dq;
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

namespace {

struct Tile { int rm, cg; };
constexpr Tile kTiles[] = {{8, 8}, {8, 16}, {8, 4}, {4, 16}, {4, 8}, {4, 4}};

// What differs between the tiles is how many of their outputs are past the ends of the layer (channels rounded up to TC, pixels
// to TP), how evenly they fill the SMs, and how much is staged per reduction step (TC + TP values, about 4 lane instructions each
// against 2.2 per term).  An SM runs its CTAs side by side, so its time is its number of tiles; with fewer than four resident
// CTAs (16 warps) it does not reach its full rate.
Tile choose_tile(int P, int Co) {
    static const double rate[4] = {0.5, 0.8, 0.93, 1.0};
    Tile best = kTiles[0];
    double best_cost = 1e300;
    const int sms = sm_count();
    for (const Tile& t : kTiles) {
        const int tc = t.rm * t.cg, tp = GATHER_THREADS / t.cg * 8;
        const long long tiles = (long long)ceil_div(P, tp) * ceil_div(Co, tc);
        const long long per_sm = (tiles + sms - 1) / sms;
        const double cost = per_sm / rate[per_sm < 4 ? per_sm - 1 : 3] * (2.2 * tc * tp + 4.0 * (tc + tp));
        if (cost < best_cost) { best_cost = cost; best = t; }
    }
    return best;
}

size_t smem_bytes(const Tile& t) {
    const int tc = t.rm * t.cg, tp = GATHER_THREADS / t.cg * 8;
    return (size_t)GATHER_STAGES * GATHER_CK * (tp + tc + 4) * sizeof(float);
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

template <int RM, int CG, bool QUADS>
int launch_t(const FwdGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kern = adder_fwd_gather_kernel<RM, CG, QUADS>;
    const int se = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (se != ADDER_OK) return se;
    kern<<<grid, GATHER_THREADS, smem, stream>>>(a);
    return launched();
}

template <bool QUADS>
int launch_q(const Tile& t, const FwdGatherArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    if (t.rm == 8) {
        if (t.cg == 16) return launch_t<8, 16, QUADS>(a, grid, smem, stream);
        if (t.cg == 8) return launch_t<8, 8, QUADS>(a, grid, smem, stream);
        return launch_t<8, 4, QUADS>(a, grid, smem, stream);
    }
    if (t.cg == 16) return launch_t<4, 16, QUADS>(a, grid, smem, stream);
    if (t.cg == 8) return launch_t<4, 8, QUADS>(a, grid, smem, stream);
    return launch_t<4, 4, QUADS>(a, grid, smem, stream);
}

}  // namespace

int fwd_gather_stat_slices(const ConvGeom& g) {
    const int P = g.N * g.Ho * g.Wo;
    return ceil_div(P, GATHER_THREADS / choose_tile(P, g.Co).cg * 8);
}

int describe_fwd_gather(const ConvGeom& g, char* buf, size_t n) {
    const int P = g.N * g.Ho * g.Wo;
    const Tile t = choose_tile(P, g.Co);
    const int tc = t.rm * t.cg, tp = GATHER_THREADS / t.cg * 8;
    return snprintf(buf, n, "fwd gather k=%dx%d RM=%d TC=%d TP=%d threads=%d smem=%zu grid=(%d,%d) status=0", g.kh, g.kw, t.rm, tc, tp,
                    GATHER_THREADS, smem_bytes(t), ceil_div(P, tp), ceil_div(g.Co, tc));
}

int launch_fwd_gather(const ConvGeom& g, const float* x, const float* w, float* out, cudaStream_t stream, double* stats,
                      int stat_slices) {
    FwdGatherArgs a;
    a.m = fwd_map(g);
    a.x = x; a.w = w; a.out = out; a.stats = stats;
    a.Ci = g.Ci; a.H = g.H; a.W = g.W; a.Co = g.Co; a.KK = g.kh * g.kw;
    const int blocks = ceil_div(g.Ci, GATHER_CK);
    a.CK = ceil_div(g.Ci, blocks);              // evenly sized channel blocks
    a.nchunks = ceil_div(g.Ci, a.CK) * a.KK;
    const bool whole_quads = (g.Ho * g.Wo) % 4 == 0;
    a.vec_store = whole_quads && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const bool quads = whole_quads && a.KK == 1 && g.sh == 1 && g.sw == 1 && g.ph == 0 && g.pw == 0 &&
                       (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    const Tile t = choose_tile(a.m.P, g.Co);
    const dim3 grid((unsigned)ceil_div(a.m.P, GATHER_THREADS / t.cg * 8), (unsigned)ceil_div(g.Co, t.rm * t.cg));
    if (grid.y > 65535) return ADDER_ERR_UNSUPPORTED;
    if (stats != nullptr && stat_slices != (int)grid.x) return ADDER_ERR_WORKSPACE;
    return quads ? launch_q<true>(t, a, grid, smem_bytes(t), stream) : launch_q<false>(t, a, grid, smem_bytes(t), stream);
}

}  // namespace adder
