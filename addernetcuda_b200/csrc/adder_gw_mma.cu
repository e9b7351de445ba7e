// Weight gradient on the 5th-generation tensor cores:
//   part[co, ci, tap] = sum over pixels p of g[co, p] * x[ci, p at tap],   gsum[co] = sum of g[co, p]
// (grad_w = part - w * gsum; the finish kernels of adder_bwd_weight.cu add the slices, as for the fp32 kernels).
//
// This is a matrix product whose reduction runs over pixels, so it belongs on the tensor cores, but it must keep fp32
// accuracy.  Every value is split into three bf16 numbers, v = v1 + v2 + v3 (8 bits of significand each, 24 together; exact for
// magnitudes from 2^-110 up to the largest bf16, 3.39e38 - smaller values lose bits of v3, larger ones and infinities become
// NaN).  The split form accumulates the products v_i * u_j with i + j <= 4 in fp32 in tensor memory: what it drops, v2*u3 + v3*u2 +
// v3*u3, is at most 2^-24 of a product, about one fp32 rounding; the stacked form drops nothing.  The tensor core rounds its
// running sums toward zero, which loses about 1.3e-8 of a sum per accumulation (measured), so the leading products v1*u1 have an
// accumulator of their own, and after every 16 accumulations it is moved into fp32 registers (rounded to nearest) and cleared.  The
// others are 2^-8 smaller and stay.  Against float64 the result is as close as the fp32 kernels' (1e-7 to 4e-7).
//
// What bounds it: the loading warps' turn, not a pipe.  On 256->256 14x14 at batch 384 (832 us) the tensor pipe is active 39 % of the
// cycles, issue slots 38 %, the shared-memory pipe 10 %; the warps wait for their loads and for the conversion's chain of
// dependent instructions, 11 of them an SM.  Each value is read and split by every CTA that shares it (x six times there, g twelve).
//
// Operands.  Threads read x and g in fp32 (eight channels of one pixel each; neighbouring lanes take neighbouring pixels), split
// them and store 16-byte rows of 8 channels: shared memory holds [split][channel group of 8][position] rows, the
// "MN-major, no swizzle" operand layout with 16 bytes between reduction steps.  Positions of a chunk are rows of output pixels
// with the pitch of the input patch (g is zero in the pad columns), so a tap of the window is nothing but a start address
// further on by its offset: x is staged once for all taps, no im2col.  A stride S splits x into S x S planes by parity.
//
// Two ways to issue the products:
//   stacked   few channels: the three parts of up to 40 output channels are stacked along M (128 rows), those of the input
//             channels along N, one instruction per tap and 16 pixels forms all nine products, the epilogue adds them;
//   split     many channels: six instructions per tap and 16 pixels, 128 output x up to 192 input channels.
// One CTA per SM: 11 warps load, split and store, a thread of the twelfth issues the products.  Two shared-memory stages; tcgen05.commit releases a stage when the instructions that read it are done.
#include <cstdio>
#include "kernels.h"
#include "tma.cuh"

namespace adder {

namespace {
constexpr int THREADS = 384;         // 12 warps, three per scheduler: 168 registers each
constexpr int LOADERS = THREADS - 32;   // threads that load, split and store; the last warp issues the products
constexpr int TASKS = 4;             // (channel group, position) pairs per thread and chunk
constexpr int WPQ = THREADS / 128;   // warps that share a quarter (32 rows) of the accumulators
constexpr int BLOCKS = 4;            // 16-column blocks of the leading accumulator per warp
constexpr int DRAIN = 16;            // accumulations between two drains
constexpr int MAX_TAPS = 64;         // taps of one CTA
constexpr int ROW0 = 1 << 20;        // added to stored rows, so that rows above the plane differ from "nothing to read"
}

__device__ float zero_word = 0.f;

struct GwMmaArgs {
    const float* x;
    const float* g;
    float* part;
    float* gsum_part;
    unsigned int* ticket;
    int N, Ci, H, W, Co, Ho, Wo, KK;
    int sh, sw, ph, pw;
    int flat;                // 1x1: positions are consecutive output pixels of the batch
    int quads;               // ... 32 to a chunk, in aligned quads (FLAT_QUADS)
    int R, pitch, gpos;      // rows per chunk, positions per row, staged positions of g (a multiple of 16)
    int xrows, xpos, planes, planes_w;       // rows and positions of one plane of x, planes, planes per row of planes
    int chunks, row_blocks, splits;
    int cog, cig;            // channel groups (of 8) per CTA
    int co_tiles, ci_tiles, tap_groups, taps_per_group;
    int xdy;                 // input rows from one tap group to the next (dilation, when the groups are kernel rows)
    int stacked, ncols, n_instr, tmem_cols;  // accumulator columns per tap, N of an instruction
    int small_col;           // split: columns from a leading accumulator to that of its small products
    int drain_chunks;        // chunks between two drains
    int whole;               // both channel counts are multiples of 8
    int tap_off[MAX_TAPS];   // position offset of tap t of a group (plane and shift)
    FastDiv d_pitch, d_xpos, d_gpos, d_planes_w, d_row_blocks, d_howo, d_wo;
};

// Shared-memory operand descriptors: low word = start address / 16 and 128 bytes between groups of 8 reduction steps, high word =
// group_bytes between groups of 8 rows or columns, version 1, no swizzle.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) { return ((addr >> 4) & 0x3fff) | ((128u >> 4) << 16); }
__device__ __forceinline__ uint32_t desc_hi(uint32_t group_bytes) { return ((group_bytes >> 4) & 0x3fff) | (1u << 14); }
// One lane of the issuing warp, chosen in the way the compiler knows: inside `if (elect_one())` it keeps descriptors in the uniform
// registers that the instruction takes them in.  (With `if (lane == 0)` an instruction took 110-170 clocks to issue, whatever its
// size; so chosen, M=128 runs at 45 / 52 / 67 / 97 clocks for N = 32 / 64 / 128 / 192, whatever the operand layout.)
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile("{ .reg .pred p; .reg .b64 da, db; setp.ne.b32 p, %6, 0; mov.b64 da, {%1, %2}; mov.b64 db, {%3, %4};"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p; }"
                 ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_load16(float (&v)[16], uint32_t addr) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_zero16(uint32_t addr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(addr), "r"(0) : "memory");
}

// (a, b) -> bf16 pair (a in the low half), and what is left of both
__device__ __forceinline__ uint32_t take_bf16(float& a, float& b) {
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(b), "f"(a));
    a -= __uint_as_float(p << 16);
    b -= __uint_as_float(p & 0xffff0000u);
    return p;
}

// How positions are read: ROWS of the output with their halo; FLAT, the pixels of the batch in order (1x1 layers); QUADS, the same four
// at a time, which takes half the instructions.
enum { ROWS, FLAT_PIXELS, FLAT_QUADS };

template <int MODE, bool STACKED>
__global__ void __launch_bounds__(THREADS, 1) adder_gw_mma_kernel(const __grid_constant__ GwMmaArgs a, int* error_flag) {
    constexpr bool FLAT = MODE != ROWS;
    extern __shared__ __align__(128) uint4 smem16[];           // rows of 8 channels
    __shared__ __align__(16) uint4 ones[32];                   // 2 groups of 8 columns x 16 steps: column 0 is one
    __shared__ uint64_t full[2], empty[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int gave_up;

    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int xrows_all = a.planes * a.xpos;                   // positions of one channel group of x
    const int gsplit = a.cog * a.gpos, xsplit = a.cig * xrows_all;
    const int stage_rows = 3 * (gsplit + xsplit);

    int tile = blockIdx.y;
    const int tg = tile % a.tap_groups; tile /= a.tap_groups;
    const int ci_tile = tile % a.ci_tiles, co_tile = tile / a.ci_tiles;
    const int ci0 = ci_tile * a.cig * 8, co0 = co_tile * a.cog * 8;
    // the sums of g of a slice's chunks are shared out between the CTAs that read them
    const int sharers = a.tap_groups * a.ci_tiles, share = ci_tile * a.tap_groups + tg;
    const int split = blockIdx.x;
    const int c_begin = (int)((long long)a.chunks * split / a.splits), c_end = (int)((long long)a.chunks * (split + 1) / a.splits);
    const int n_local = c_end - c_begin;

    if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) *a.ticket = 0u;
    if (tid < 32) ones[tid] = tid < 16 ? make_uint4(0x3f80u, 0u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
        gave_up = 0;
        for (int s = 0; s < 2; ++s) { mbar_init(&full[s], LOADERS); mbar_init(&empty[s], 1); }
        mbar_init(&drained, THREADS);
        mbar_fence_init();
    }
    if (wid == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // `ones` is read by the tensor core
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int sum_col = a.taps_per_group * a.ncols;            // accumulator columns of the sums of g
    const uint32_t lane_base = tmem + ((uint32_t)(wid & 3) << 21);      // 32 rows of the warp's quarter, row in bits 16 and up
    if (wid < 4) {
        tmem_zero16(lane_base + sum_col);
        if (!STACKED) tmem_zero16(lane_base + sum_col + a.small_col);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int nb = a.cig >> 1, blocks = a.taps_per_group * nb;          // 16-column blocks of the leading products: per tap, all
    // stacked: the leading products are in the first cog*8 rows only
    const bool drains = !STACKED || (wid & 3) * 32 < a.cog * 8;
    float tot[BLOCKS][16], tot_sum = 0.f;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
        for (int q = 0; q < 16; ++q) tot[b][q] = 0.f;

    // All warps, before the products of chunk i (a multiple of drain_chunks): wait until those of chunk i - 1 are done and move the
    // leading sums into registers.
    auto drain = [&](int i) -> bool {
        if (!mbar_wait(&empty[(i - 1) & 1], ((i - 1) >> 1) & 1)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (drains) {
            float t[16];
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                const int blk = (wid >> 2) + b * WPQ;
                if (blk >= blocks) break;
                const uint32_t at = lane_base + blk / nb * a.ncols + blk % nb * 16;
                tmem_load16(t, at);
                tmem_zero16(at);
#pragma unroll
                for (int q = 0; q < 16; ++q) tot[b][q] += t[q];
            }
            if ((wid >> 2) == 0) {
                tmem_load16(t, lane_base + sum_col);
                tmem_zero16(lane_base + sum_col);
                tot_sum += t[0];
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&drained)) : "memory");
        return true;
    };

    if (wid == LOADERS / 32) {
        // ---- the warp that issues the products
        const uint32_t smem0 = smem_u32(smem16);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((128u >> 4) << 24);
        const uint32_t id_main = idesc | ((uint32_t)(a.n_instr >> 3) << 17), id_sum = idesc | (2u << 17);
        const uint32_t a_hi = desc_hi((uint32_t)a.gpos * 16u), b_hi = desc_hi((uint32_t)xrows_all * 16u);
        const uint32_t ones_lo = desc_lo(smem_u32(ones)), ones_hi = desc_hi(256);
        int i = 0;
        for (; i < n_local; ++i) {
            const int s = i & 1;
            if (!mbar_wait(&full[s], (i >> 1) & 1)) break;
            if (i > 0 && i % a.drain_chunks == 0 && (!drain(i) || !mbar_wait(&drained, (i / a.drain_chunks - 1) & 1))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool sums = (c_begin + i) % sharers == share;
            if (elect_one()) {
                const uint32_t stage = smem0 + (uint32_t)(s * stage_rows) * 16u;
                const uint32_t da0 = desc_lo(stage), db0 = desc_lo(stage + (uint32_t)(3 * gsplit) * 16u);
                for (int k = 0; k < a.gpos; k += 16) {
                    const uint32_t acc = (i | k) != 0, da = da0 + k, db = db0 + k;
                    uint32_t d = tmem;
                    for (int t = 0; t < a.taps_per_group; ++t, d += a.ncols) {
                        const uint32_t bt = db + (uint32_t)a.tap_off[t];
                        if (STACKED) {
                            mma_bf16(d, da, a_hi, bt, b_hi, id_main, acc);
                        } else {
                            const uint32_t ds = d + a.small_col;
                            mma_bf16(ds, da + 2 * gsplit, a_hi, bt, b_hi, id_main, acc);
                            mma_bf16(ds, da, a_hi, bt + 2 * xsplit, b_hi, id_main, 1);
                            mma_bf16(ds, da + gsplit, a_hi, bt + xsplit, b_hi, id_main, 1);
                            mma_bf16(ds, da + gsplit, a_hi, bt, b_hi, id_main, 1);
                            mma_bf16(ds, da, a_hi, bt + xsplit, b_hi, id_main, 1);
                            mma_bf16(d, da, a_hi, bt, b_hi, id_main, acc);
                        }
                    }
                    if (sums) {
                        if (!STACKED) {
                            mma_bf16(d + a.small_col, da + 2 * gsplit, a_hi, ones_lo, ones_hi, id_sum, 1);
                            mma_bf16(d + a.small_col, da + gsplit, a_hi, ones_lo, ones_hi, id_sum, 1);
                        }
                        mma_bf16(d, da, a_hi, ones_lo, ones_hi, id_sum, 1);
                    }
                }
                mma_commit(&empty[s]);
            }
            __syncwarp();
        }
        if (i < n_local) {
            gave_up = 1;
            // what was issued still reads this CTA's shared memory and writes the accumulators that it is about to free
            if (i > 0) mbar_wait(&empty[(i - 1) & 1], ((i - 1) >> 1) & 1);
        }
    } else if constexpr (MODE == FLAT_QUADS) {
        // ---- the warps that load, split and store: a thread has four pixels of eight channels.  The reduction's order is free where no
        // tap shifts it, so pixel 4*l + j of a chunk of 32 is step 8*j + l: eight neighbouring threads store neighbouring rows.
        const int HoWo = a.Ho * a.Wo, grp = tid >> 3, l = tid & 7;
        const bool is_x = grp < a.cig, used = grp < a.cig + a.cog;
        const int C = is_x ? a.Ci : a.Co, ch = is_x ? ci0 + grp * 8 : co0 + (grp - a.cig) * 8, left = used ? C - ch : 0;
        const float* const tensor = is_x ? a.x : a.g;
        const int row = (is_x ? 3 * gsplit + grp * 32 : (grp - a.cig) * 32) + l, split_rows = is_x ? xsplit : gsplit;
        float4 v[8];
        auto load = [&](int chunk) {
            const int p = chunk * 32 + 4 * l;
            const bool in = p < a.N * HoWo;
            uint32_t im, r;
            a.d_howo.divmod(in ? p : 0, im, r);
            if (a.sw == 2 && is_x) {                   // every other pixel of every other row
                uint32_t y, x;
                a.d_wo.divmod(r, y, x);
                const int HW = a.H * a.W;
                const float* src = tensor + ((size_t)im * C + (left > 0 ? ch : 0)) * HW + 2 * y * a.W + 2 * x;
#pragma unroll
                for (int q = 0; q < 8; ++q, src += HW) {
                    const bool ok = in & (q < left);
                    const float4 lo = ok ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float4 hi = ok ? __ldg(reinterpret_cast<const float4*>(src + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[q] = make_float4(lo.x, lo.z, hi.x, hi.z);
                }
                return;
            }
            const float* src = tensor + ((size_t)im * C + (left > 0 ? ch : 0)) * HoWo + r;
#pragma unroll
            for (int q = 0; q < 8; ++q, src += HoWo)
                v[q] = (in & (q < left)) ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        if (n_local > 0) load(c_begin);
        for (int i = 0; i < n_local; ++i) {
            const int s = i & 1;
            if (i >= 2 && !mbar_wait(&empty[s], ((i >> 1) - 1) & 1)) { gave_up = 1; break; }
            if (used) {
                uint4* d = smem16 + s * stage_rows + row;
                auto store = [&](int j, float (&u)[8]) {
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        uint4 p;
                        p.x = take_bf16(u[0], u[1]); p.y = take_bf16(u[2], u[3]);
                        p.z = take_bf16(u[4], u[5]); p.w = take_bf16(u[6], u[7]);
                        d[q * split_rows + j * 8] = p;
                    }
                };
                float u0[8], u1[8], u2[8], u3[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) { u0[q] = v[q].x; u1[q] = v[q].y; u2[q] = v[q].z; u3[q] = v[q].w; }
                store(0, u0); store(1, u1); store(2, u2); store(3, u3);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[s])) : "memory");
            if (i + 1 < n_local) load(c_begin + i + 1);
            if (i > 0 && i % a.drain_chunks == 0 && !drain(i)) { gave_up = 1; break; }
        }
    } else {
        // ---- the warps that load, split and store: each thread has up to TASKS (channel group, position) pairs
        const int xt = a.cig * xrows_all, gt = a.cog * a.gpos;
        const int HW = a.H * a.W, HoWo = a.Ho * a.Wo;
        // per task: offset of its value in its tensor (image 0, first rows), and its row there (FLAT: its position).
        // Packed into `row`: -1 = nothing to read, else the row in the upper bits and the channels left (at most 8) in the lower four.
        int off[TASKS], row[TASKS];
#pragma unroll
        for (int i = 0; i < TASKS; ++i) {
            int t = tid + i * LOADERS;
            off[i] = 0; row[i] = -1;
            int left = 0;
            uint32_t grp, pos, r, c;
            if (t < xt) {
                uint32_t q, plane, pa, pb;
                a.d_xpos.divmod(t, q, pos);
                grp = q / (uint32_t)a.planes; plane = q - grp * a.planes;
                a.d_planes_w.divmod(plane, pa, pb);
                a.d_pitch.divmod(pos, r, c);
                const int ch = ci0 + (int)grp * 8;
                off[i] = ch * HW;
                left = a.Ci - ch;
                if (FLAT) row[i] = (int)pos;
                else {
                    const int x_row = (int)r * a.sh + (int)pa - a.ph + tg * a.xdy, x_col = (int)c * a.sw + (int)pb - a.pw;
                    off[i] += x_row * a.W + x_col;
                    if ((int)r < a.xrows && x_col >= 0 && x_col < a.W) row[i] = x_row + ROW0;
                }
            } else if (t - xt < gt) {
                t -= xt;
                a.d_gpos.divmod(t, grp, pos);
                a.d_pitch.divmod(pos, r, c);
                const int ch = co0 + (int)grp * 8;
                off[i] = ch * HoWo;
                left = a.Co - ch;
                if (FLAT) row[i] = (int)pos;
                else {
                    off[i] += (int)r * a.Wo + (int)c;
                    if ((int)r < a.R && (int)c < a.Wo) row[i] = (int)r + ROW0;
                }
            }
            row[i] = left <= 0 || row[i] < 0 ? -1 : row[i] * 16 + min(left, 8);
        }
        float v[TASKS][8];
        // of the chunk being loaded: offsets of its image and rows.  FLAT: of this thread's position, the same for all of its tasks
        // because gpos divides LOADERS (16 or 32)
        int n_x = 0, n_g = 0, row_x = 0, row_g = 0;
        bool inside = true;
        auto locate = [&](int chunk) {
            if (FLAT) {
                const int p = chunk * a.gpos + (tid & (a.gpos - 1));
                uint32_t im, r;
                inside = p < a.N * HoWo;
                a.d_howo.divmod(inside ? p : 0, im, r);
                n_g = (int)im * a.Co * HoWo + (int)r;
                if (a.sh > 1 || a.sw > 1) {
                    uint32_t y, x;
                    a.d_wo.divmod(r, y, x);
                    r = y * a.sh * a.W + x * a.sw;
                }
                n_x = (int)im * a.Ci * HW + (int)r;
                return;
            }
            uint32_t n, rb;
            a.d_row_blocks.divmod(chunk, n, rb);
            row_g = (int)rb * a.R; row_x = row_g * a.sh;
            n_x = (int)n * a.Ci * HW + row_x * a.W; n_g = (int)n * a.Co * HoWo + row_g * a.Wo;
        };
        auto load = [&](int i) {
            const bool is_x = tid + i * LOADERS < xt;
            const int stride = is_x ? HW : HoWo, at = off[i] + (is_x ? n_x : n_g);
            bool in = row[i] >= 0;
            if (FLAT) in &= inside;
            else in &= (unsigned)((row[i] >> 4) - ROW0 + (is_x ? row_x : row_g)) < (unsigned)(is_x ? a.H : a.Ho);
            // nothing to read: eight times the zero word
            const float* src = in ? (is_x ? a.x : a.g) + at : &zero_word;
            const int step = in ? stride : 0;
            if (a.whole) {
#pragma unroll
                for (int q = 0; q < 8; ++q, src += step) v[i][q] = __ldg(src);
            } else {
                const int left = row[i] & 15;
#pragma unroll
                for (int q = 0; q < 8; ++q, src += step) {
                    if (q == left) src = &zero_word;
                    v[i][q] = __ldg(src);
                    if (q >= left) src -= step;
                }
            }
        };
        if (n_local > 0) {
            locate(c_begin);
#pragma unroll
            for (int j = 0; j < TASKS; ++j)
                if (tid + j * LOADERS < xt + gt) load(j);
        }
        for (int i = 0; i < n_local; ++i) {
            const int s = i & 1;
            if (i >= 2 && !mbar_wait(&empty[s], ((i >> 1) - 1) & 1)) { gave_up = 1; break; }
            uint4* stage = smem16 + s * stage_rows;
#pragma unroll
            for (int j = 0; j < TASKS; ++j) {
                const int t = tid + j * LOADERS;
                if (t >= xt + gt) continue;
                const bool is_x = t < xt;
                uint4* d = stage + (is_x ? 3 * gsplit + t : t - xt);
                const int part = is_x ? xsplit : gsplit;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    uint4 p;
                    p.x = take_bf16(v[j][0], v[j][1]); p.y = take_bf16(v[j][2], v[j][3]);
                    p.z = take_bf16(v[j][4], v[j][5]); p.w = take_bf16(v[j][6], v[j][7]);
                    d[q * part] = p;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[s])) : "memory");
            // (not between the conversions: a conversion would wait for the loads issued just before it as well)
            if (i + 1 < n_local) {
                locate(c_begin + i + 1);
#pragma unroll
                for (int j = 0; j < TASKS; ++j)
                    if (tid + j * LOADERS < xt + gt) load(j);
            }
            if (i > 0 && i % a.drain_chunks == 0) {
                if (!drain(i)) { gave_up = 1; break; }
            }
        }
    }
    if (n_local > 0 && !gave_up && !mbar_wait(&empty[(n_local - 1) & 1], ((n_local - 1) >> 1) & 1)) gave_up = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    const bool ok = gave_up == 0 && n_local > 0;

    // ---- epilogue: sums -> shared memory -> this CTA's slice, in the order of the weights
    float* buf = reinterpret_cast<float*>(smem16);             // [accumulator row][input channel][tap]
    float* part = a.part + (size_t)split * a.Co * a.Ci * a.KK;
    const int taps = a.taps_per_group, cig8 = a.cig * 8, cog8 = a.cog * 8, tap0 = tg * taps;
    const int trow = (wid & 3) * 32 + lane;                    // accumulator row of this thread
    const int cols = taps * cig8, pitch = cols + 1;
    if (gave_up == 0) {
        const int brows = STACKED ? 3 * cog8 : 128;
        {
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                const int blk = (wid >> 2) + b * WPQ;
                if (blk >= blocks) break;
                const int t = blk / nb, c = blk % nb * 16;
                if (ok) {
                    float u[16];
                    if (STACKED) {
                        float u2[16];
                        tmem_load16(u, lane_base + t * a.ncols + 2 * cig8 + c);
                        tmem_load16(u2, lane_base + t * a.ncols + cig8 + c);
#pragma unroll
                        for (int q = 0; q < 16; ++q) u[q] += u2[q];
                    } else {
                        tmem_load16(u, lane_base + t * a.ncols + a.small_col + c);
                    }
                    float m[16];
                    tmem_load16(m, lane_base + t * a.ncols + c);
#pragma unroll
                    for (int q = 0; q < 16; ++q) tot[b][q] += m[q] + u[q];
                }
                if (trow < brows)
#pragma unroll
                    for (int q = 0; q < 16; ++q) buf[trow * pitch + (c + q) * taps + t] = tot[b][q];
            }
        }
        __syncthreads();
        const int orows = min(cog8, a.Co - co0), ocols = min(cig8, a.Ci - ci0) * taps;
        float* out = part + ((size_t)co0 * a.Ci + ci0) * a.KK + tap0;
        for (int e = tid; e < orows * ocols; e += THREADS) {
            const int co = e / ocols, k = e - co * ocols, ci = k / taps, t = k - ci * taps;
            const float* b = buf + co * pitch + k;
            out[((size_t)co * a.Ci + ci) * a.KK + t] = STACKED ? (b[2 * cog8 * pitch] + b[cog8 * pitch]) + b[0] : b[0];
        }
        __syncthreads();
        if (wid < 4) {
            if (ok) {
                float u[16];
                tmem_load16(u, lane_base + sum_col);
                tot_sum += u[0];
                if (!STACKED) {
                    tmem_load16(u, lane_base + sum_col + a.small_col);
                    tot_sum += u[0];
                }
            }
            buf[trow] = tot_sum;
        }
        __syncthreads();
        for (int co = tid; co < orows; co += THREADS)
            a.gsum_part[((size_t)split * sharers + share) * a.Co + co0 + co] =
                STACKED ? (buf[2 * cog8 + co] + buf[cog8 + co]) + buf[co] : buf[co];
    } else if (tid == 0) {
        *error_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols));
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

namespace {

constexpr int TMEM_COLS = 512, SMEM_MAX = 216 * 1024;
// Steps of 16 pixels in one CTA's sum.  The products that are not drained lose 1.3e-8 of their sum per accumulation, times 2^-8
// for their size and five accumulations a step where all of them share an accumulator: 2e-7 of the result at most.
constexpr int MAX_STEPS_SPLIT = 1024, MAX_STEPS_STACKED = 4096;

struct Plan {
    GwMmaArgs a;
    size_t smem;
    double clocks;           // estimated time of the launch in SM clocks
};

// Fills in chunk and launch shape for `rows` rows of output pixels per chunk (flat: 16-pixel steps).  False: does not fit.
bool shape(const ConvGeom& g, GwMmaArgs a, int rows, Plan* p) {
    a.R = rows;
    const int shift_h = a.taps_per_group == a.KK ? (g.kh - 1) * g.dh / g.sh : 0, shift_w = (g.kw - 1) * g.dw / g.sw;
    a.pitch = a.flat ? 1 : g.Wo + shift_w;
    a.gpos = round_up(a.flat ? rows * 16 : rows * a.pitch, 16);
    a.xrows = rows + shift_h;
    a.xpos = a.gpos + shift_h * a.pitch + shift_w;
    const int planes_h = (a.taps_per_group == a.KK && g.kh > 1) ? g.sh : 1;
    a.planes_w = g.kw > 1 ? g.sw : 1;
    a.planes = planes_h * a.planes_w;
    const int tasks = a.cig * a.planes * a.xpos + a.cog * a.gpos, steps = a.gpos / 16;
    if (tasks > TASKS * LOADERS || steps > DRAIN) return false;
    a.drain_chunks = DRAIN / steps;
    a.row_blocks = a.flat ? 1 : ceil_div(g.Ho, rows);
    const long long chunks = a.flat ? ((long long)g.N * g.Ho * g.Wo + a.gpos - 1) / a.gpos : (long long)g.N * a.row_blocks;
    if (chunks > 1 << 24) return false;
    a.chunks = (int)chunks;
    const int gsplit = a.cog * a.gpos, xsplit = a.cig * a.planes * a.xpos, stage_rows = 3 * (gsplit + xsplit);
    // an instruction always reads 16 row groups of g: where fewer exist it reads on into x, whose products land in unused rows
    const int last_read = stage_rows + (a.stacked ? 0 : 2 * gsplit) + 16 * a.gpos;
    const int rows_needed = last_read > 2 * stage_rows ? last_read : 2 * stage_rows;
    const size_t epilogue = (size_t)(a.stacked ? 3 * a.cog * 8 : 128) * (a.taps_per_group * a.cig * 8 + 1) * sizeof(float);
    p->smem = (size_t)rows_needed * 16 > epilogue ? (size_t)rows_needed * 16 : epilogue;
    if (p->smem > (size_t)SMEM_MAX) return false;
    for (int t = 0; t < a.taps_per_group; ++t) {
        const int i = a.taps_per_group == a.KK ? t / g.kw : 0, j = t % g.kw;
        const int dy = i * g.dh, dx = j * g.dw;
        const int plane = (planes_h > 1 ? dy % g.sh : 0) * a.planes_w + (a.planes_w > 1 ? dx % g.sw : 0);
        a.tap_off[t] = plane * a.xpos + (dy / g.sh) * a.pitch + dx / g.sw;
    }
    a.xdy = a.tap_groups > 1 ? g.dh : 0;
    // A chunk takes the longer of its products (measured: max(n/2 + 3, 36 + n/4) clocks for an instruction of 128 x n) with its share of a
    // drain, and the loading warps' turn: the round trip of a load and about 700 clocks for each task (8 values) of a thread.  The
    // slices are written and read again.
    const double instr = a.n_instr / 2 + 3 > 36 + a.n_instr / 4 ? a.n_instr / 2 + 3 : 36 + a.n_instr / 4;
    const double sums = (a.stacked ? 42.0 : 126.0) / (a.ci_tiles * a.tap_groups);
    const double products = steps * ((double)a.taps_per_group * (a.stacked ? 1 : 6) * instr + sums) + 250 + 900.0 / a.drain_chunks;
    const double turn = a.quads ? 1800 : 1000 + 700.0 * tasks / LOADERS;
    const double chunk = products > turn ? products : turn;
    const int tiles = a.co_tiles * a.ci_tiles * a.tap_groups, slots = sm_count();
    const int least = ceil_div(a.chunks, (a.stacked ? MAX_STEPS_STACKED : MAX_STEPS_SPLIT) / steps);
    p->clocks = 1e300;
    for (int waves = 1; waves <= 3; ++waves) {
        int splits = waves * slots / tiles;
        if (splits < least) splits = least;
        if (splits > a.chunks) splits = a.chunks;
        if (splits < 1) splits = 1;                            // an empty batch still writes its (zero) slice
        const double clocks = (double)((tiles * splits + slots - 1) / slots) * (ceil_div(a.chunks, splits) * chunk + 6000) +
                              (double)splits * g.Co * g.Ci * a.KK / 800;
        if (clocks < p->clocks) { p->clocks = clocks; a.splits = splits; }
    }
    p->a = a;
    return true;
}

bool search(const ConvGeom& g, Plan* best) {
    best->clocks = 1e300;
    GwMmaArgs a;
    a.N = g.N; a.Ci = g.Ci; a.H = g.H; a.W = g.W; a.Co = g.Co; a.Ho = g.Ho; a.Wo = g.Wo; a.KK = g.kh * g.kw;
    a.sh = g.sh; a.sw = g.sw; a.ph = g.ph; a.pw = g.pw;
    a.flat = a.KK == 1 && g.ph == 0 && g.pw == 0;
    a.whole = g.Ci % 8 == 0 && g.Co % 8 == 0;
    // whole aligned quads of output pixels, and of the input pixels under them
    a.quads = a.flat && (g.Ho * g.Wo) % 4 == 0 && ((g.sh == 1 && g.sw == 1) || (g.sh == 2 && g.sw == 2 && g.Wo % 4 == 0 && g.W == 2 * g.Wo));
    const int co8 = ceil_div(g.Co, 8), ci8 = round_up(ceil_div(g.Ci, 8), 2);
    for (int form = 0; form < 4; ++form)
        for (int by_rows = 0; by_rows < (g.kh > 1 ? 2 : 1); ++by_rows) {
            const int stacked = form & 1;
            a.stacked = stacked;
            a.taps_per_group = by_rows ? g.kw : a.KK;
            a.tap_groups = by_rows ? g.kh : 1;
            if (a.taps_per_group > MAX_TAPS) continue;
            const int co_max = (stacked ? 5 : 16) / (form < 2 ? 1 : 2);      // half tiles fit longer rows
            a.co_tiles = ceil_div(co8, co_max);
            a.cog = ceil_div(co8, a.co_tiles);
            for (int cig = 2; cig <= (stacked ? 10 : 24); cig += 2) {
                if (cig > ci8) break;
                a.cig = cig;
                a.n_instr = (stacked ? 3 : 1) * cig * 8;
                a.ncols = a.n_instr;
                a.small_col = stacked ? 0 : a.taps_per_group * a.ncols + 16;
                const int cols = (stacked ? 1 : 2) * (a.taps_per_group * a.ncols + 16);
                if (a.n_instr > 256 || cols > TMEM_COLS || a.taps_per_group * cig / 2 > BLOCKS * WPQ) break;
                a.tmem_cols = 32;
                while (a.tmem_cols < cols) a.tmem_cols *= 2;
                a.ci_tiles = ceil_div(ceil_div(g.Ci, 8), cig);
                const int most = a.flat ? 2 : g.Ho;
                for (int rows = a.quads ? 2 : 1; rows <= most; ++rows) {
                    Plan p;
                    if (!shape(g, a, rows, &p)) break;         // more rows only need more
                    if (p.clocks < best->clocks) *best = p;
                }
            }
        }
    if (best->clocks >= 1e300) return false;
    GwMmaArgs& b = best->a;
    if ((long long)b.co_tiles * b.ci_tiles * b.tap_groups > 65535) return false;
    b.d_pitch = FastDiv(b.pitch); b.d_xpos = FastDiv(b.xpos); b.d_gpos = FastDiv(b.gpos); b.d_planes_w = FastDiv(b.planes_w);
    b.d_row_blocks = FastDiv(b.row_blocks); b.d_howo = FastDiv(g.Ho * g.Wo); b.d_wo = FastDiv(g.Wo);
    return true;
}

bool plan(const ConvGeom& g, Plan* p) {
    return cached_plan(g, *p, [&](Plan& q) { return search(g, &q) ? ADDER_OK : ADDER_ERR_UNSUPPORTED; }) == ADDER_OK;
}

}  // namespace

int gw_mma_splits(const ConvGeom& g) {
    Plan p;
    return plan(g, &p) ? p.a.splits : 0;
}

int gw_mma_gsum_splits(const ConvGeom& g) {
    Plan p;
    return plan(g, &p) ? p.a.splits * p.a.tap_groups * p.a.ci_tiles : 0;
}

int describe_gw_mma(const ConvGeom& g, char* buf, size_t n) {
    Plan p;
    if (!plan(g, &p)) return 0;
    const GwMmaArgs& a = p.a;
    return snprintf(buf, n, "gw mma %s co=%d ci=%d taps=%d R=%d K=%d threads=%d smem=%zu cols=%d grid=(%d,%d) splits=%d status=0",
                    a.stacked ? "stacked" : "split", a.cog * 8, a.cig * 8, a.taps_per_group, a.R, a.gpos, THREADS, p.smem, a.tmem_cols,
                    a.splits, a.co_tiles * a.ci_tiles * a.tap_groups, a.splits);
}

int launch_gw_mma(const ConvGeom& g, const float* gout, const float* x, float* part, float* gsum_part, unsigned int* ticket, int splits,
                  cudaStream_t stream) {
    Plan p;
    if (!plan(g, &p) || p.a.splits != splits) return ADDER_ERR_INTERNAL;
    p.a.x = x; p.a.g = gout; p.a.part = part; p.a.gsum_part = gsum_part; p.a.ticket = ticket;
    int* flag = nullptr;
    int st = device_error_flag(&flag);
    if (st != ADDER_OK) return st;
    const bool quads = p.a.quads && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gout)) & 15) == 0;
    auto kern = quads      ? (p.a.stacked ? adder_gw_mma_kernel<FLAT_QUADS, true> : adder_gw_mma_kernel<FLAT_QUADS, false>)
                : p.a.flat ? (p.a.stacked ? adder_gw_mma_kernel<FLAT_PIXELS, true> : adder_gw_mma_kernel<FLAT_PIXELS, false>)
                           : (p.a.stacked ? adder_gw_mma_kernel<ROWS, true> : adder_gw_mma_kernel<ROWS, false>);
    st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), p.smem);
    if (st != ADDER_OK) return st;
    kern<<<dim3((unsigned)splits, (unsigned)(p.a.co_tiles * p.a.ci_tiles * p.a.tap_groups)), THREADS, p.smem, stream>>>(p.a, flag);
    return launched();
}

}  // namespace adder
