// Inverted residual block on small planes as one kernel: QLinearConv 1x1 (expand, ReLU / ReLU6) -> QLinearConv depthwise 3x3 (pads 1,
// stride 1 or 2, ReLU / ReLU6) -> QLinearConv 1x1 (project) [-> QLinearAdd with the block's input], int8 with zero point 0 between them.
//
// The expanded tensor, six times the input, never exists in memory.  A tile is one image (planes 9 to 16 wide, at most 14 high) or two (at most
// 8 x 8).  Per chunk of 128 expanded channels:
//   expand    D1 (TMEM: lane = channel, column = pixel)  =  W1 chunk [128][C]  x  X [C][pixels]            tcgen05, kind::i8
//   epilogue  a thread owns a channel: it requantises the accumulators of (eight columns of) a plane row into packed bytes, keeps three
//             rows of sums in registers, runs the depthwise filter (dp4a on windows cut by byte permutes; no shuffles, no shared memory),
//             requantises and stores the row to shared memory as rows of the next product's operand
//   project   D2 (lane = filter)  +=  W2 [filters][128 channels]  x  Y [128 channels][pixels]
// and after the last chunk the project epilogue requantises D2, adds the block's input from the operand X that is still in shared memory, stages
// the tile and sends it with one bulk copy.  Plane rows lie PITCH = 16 (or 8) columns apart, so that a row is one or half a 16-byte chunk of an
// MN-major operand row and one TMEM load; the columns past the width hold whatever, are masked behind the expansion and never stored.
//
// UNITS.  A wide plane is cut into two halves of its output rows, each with the input rows it reads (one of them twice): two products, two sets
// of barriers, two groups of eight epilogue warps, so that one group issues while the other waits for its accumulators (one set for
// both: 11200 cycles a chunk of 14 x 14, of which a warp computed 5800; with the batched builder, the sender and the paired D2 8700).  Up to 64 filters (`paired`) the halves share the columns of D2: the A
// operand of unit u holds the filters in lanes 64 u .. and zeros elsewhere, and all four lane quarters take part in the project epilogue.
//
// For few images irb_band.cuh deals a block to more CTAs.
//
// What bounds it: instruction issue in the epilogue warps, 31 thousand of the warp instructions of a 14 x 14 x 384 image are the two
// requantisations, the filter and the project epilogue (as separate kernels the depthwise one alone took 31 instructions an output).
//
// Warp roles (640 threads, 96 registers each, one persistent CTA per SM):
//   warp 0 weights (a chunk's W1, W2 and per-channel constants are one bulk copy into a ring)     warp 1 TMEM owner + MMA issuer
//   warps 2-17 epilogue: four per TMEM lane quarter, one for each unit (image) and half of the columns (rows); two per quarter with whole rows
//   had a scheduler issue 43 % of the time
//   warp 18 builder: the input's rows from NCHW into the MN-major operand X (the first tile's: with the epilogue warps)     warp 19 sender of the staged output
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "context.cuh"
#include "fused_cnn.cuh"
#include "geometry.hpp"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"
#include "tc_pw_nchw.cuh"

namespace zb {

// Per expanded channel: kAccBase - bias and multiplier of the expansion, multiplier and (as bits) kAccBase plus bias of the depthwise filter,
// its three rows packed for dp4a.
struct IrbConst { float e_floor, e_mult, d_mult; int32_t d_base; uint32_t k[3], pad; };

struct IrbArgs {
    const uint8_t* x; uint8_t* y; const uint8_t* w;        // w: per chunk [W1 | W2 | constants]
    const float* mult2; const int32_t* bias2;              // project
    int N, C, M, H, W, OH, OW;
    int IB, tiles;                 // images per tile
    int rh;                        // output rows of the first of two units
    int n1, n2;                    // columns of a unit's D1 and of its D2, multiples of 16, at most 128
    int chunks, last_live;         // chunks of 128 expanded channels; channels of the last one
    int kp;                        // C rounded up to K steps of 32
    int mt2;                       // 128-filter tiles of the project product
    int paired;                    // two units, at most 64 filters: one D2, lanes 64 u + filter
    int w2_bytes;                  // W2 of a chunk: [filter tile][8 k16][128][16], or paired [8 k16][64 zero, 64 filter, 64 zero rows][16]
    int d1_bufs;                   // one unit: buffers of D1
    int x_bufs, y_bufs, w_stages;
    int w_bytes, x_bytes, y_bytes; // one stage / buffer
    int off_x, off_y, off_out, off_tail;
    int* status;
};

constexpr int kIrbThreads = 640, kIrbEpiWarps = 16;

// N accumulators of consecutive columns, N at most 9.
template <int N>
__device__ __forceinline__ void irb_tmem_cols(uint32_t taddr, uint32_t (&v)[9]) {
    static_assert(N >= 1 && N <= 9, "");
    ptx::tmem_ld8(taddr, v);
    if constexpr (N == 9) ptx::tmem_ld1(taddr + 8u, v + 8);
}

// (Difference and product two values at a time: 14 x 14 x 384 with the addition, batch 1024, 106 -> 103 us, 64 -> 384 -> 96 95 -> 90, 160 -> 960 -> 160 at
// 7 x 7 92 -> 87.  In the small CNN's kernels, which issue more of other kinds, the same form changed nothing.)
// Requantised expansion of IN consecutive columns: packed bytes, zero where a column does not exist.
template <int IN>
__device__ __forceinline__ void irb_expand(const uint32_t (&v)[9], const uint32_t (&valid)[3], float ef, float em, uint32_t (&A)[(IN + 3) / 4 + 1]) {
    constexpr int NW = (IN + 3) / 4;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        int k4[4];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int x = 4 * w + e;
            auto acc = [&](int i) { return __viaddmax_s32((int)v[i < 9 ? i : 0], kAccBaseBits, __float_as_int(ef)); };
            k4[e] = k4[e + 1] = 0;
            if (x + 1 < IN) sub_mul_rn2(acc(x), acc(x + 1), ef, em, k4[e], k4[e + 1]);
            else if (x < IN) k4[e] = __float2int_rn(__fmul_rn(__fsub_rn(__int_as_float(acc(x)), ef), em));
        }
        A[w] = pack_sat_s8x4(k4[0], k4[1], k4[2], k4[3]) & valid[w];
    }
    A[NW] = 0u;
}
// Requantised sums of up to four outputs.
template <int N>
__device__ __forceinline__ uint32_t irb_filtered(const int* acc, float dm) {
    int k4[4];
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        k4[e] = k4[e + 1] = 0;
        if (e + 1 < N) sub_mul_rn2(max(acc[e], kAccBaseBits), max(acc[e + 1 < N ? e + 1 : 0], kAccBaseBits), kAccBase, dm, k4[e], k4[e + 1]);
        else if (e < N) k4[e] = __float2int_rn(__fmul_rn(__fsub_rn(__int_as_float(max(acc[e < N ? e : 0], kAccBaseBits)), kAccBase), dm));
    }
    return pack_sat_s8x4(k4[0], k4[1], k4[2], k4[3]);
}

// Stride 1: expand epilogue and depthwise filter of one channel's output rows [r0, r1) at OUT consecutive columns.  `src`: TMEM column of the first input
// column at the first input row, max(r0 - 1, 0) (LEFT: the one left of the outputs, else the first output's own, with nothing to its left; RIGHT: one more on the right), rows PITCH apart;
// valid[j]: byte mask of the columns that exist.  put(row, packed codes); drained() once the accumulators have been read.
template <int OUT, bool LEFT, bool RIGHT, int PITCH, typename Put, typename Drained>
__device__ __forceinline__ void irb_rows(uint32_t src, int H, int r0, int r1, const uint32_t (&valid)[3], float ef, float em, float dm, int dbase,
                                         uint32_t k0, uint32_t k1, uint32_t k2, Put put, Drained drained) {
    constexpr int IN = OUT + (LEFT ? 1 : 0) + (RIGHT ? 1 : 0), NW = (IN + 3) / 4;
    const int lo = max(r0 - 1, 0), hi = min(r1, H - 1);                      // input rows
    int acc[3][OUT];
#pragma unroll
    for (int x = 0; x < OUT; ++x) acc[0][x] = acc[1][x] = acc[2][x] = dbase;
    uint32_t v[9];
    irb_tmem_cols<IN>(src, v);
    for (int base = lo; base <= r1; base += 3) {
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int ir = base + u;
            if (ir > r1) break;
            int* up = acc[(u + 2) % 3];                                      // output row ir - 1: this is its filter row 2
            int* at = acc[u];
            int* dn = acc[(u + 1) % 3];
            if (ir <= hi) {
                uint32_t A[NW + 1];
                ptx::tmem_wait_ld();
                irb_expand<IN>(v, valid, ef, em, A);
                src += (uint32_t)PITCH;
                if (ir < hi) irb_tmem_cols<IN>(src, v);
                else drained();
#pragma unroll
                for (int x = 0; x < OUT; ++x) {
                    constexpr int shift = LEFT ? 0 : 3;                      // the window starts at byte x, or at byte x - 1 = 4 * (x / 4 - 1) + x % 4 + 3
                    const int p = x + shift, w = p / 4 - (LEFT ? 0 : 1), o = p % 4;
                    const uint32_t a0 = w < 0 ? 0u : A[w < 0 ? 0 : w], a1 = A[w + 1];
                    const uint32_t win = o == 0 ? a0 : __byte_perm(a0, a1, o == 1 ? 0x4321 : (o == 2 ? 0x5432 : 0x6543));
                    up[x] = dw_dp4a<false>(win, k2, up[x]);
                    at[x] = dw_dp4a<false>(win, k1, at[x]);
                    dn[x] = dw_dp4a<false>(win, k0, dbase);
                }
            }
            if (ir - 1 >= r0) {
                const uint32_t p0 = irb_filtered<(OUT < 4 ? OUT : 4)>(up, dm);
                uint32_t p1 = 0u;
                if constexpr (OUT > 4) p1 = irb_filtered<OUT - 4>(up + 4, dm);
                put(ir - 1, p0, p1);
            }
        }
    }
}

// Stride 2, rows 16 columns apart: output rows [r0, r1) at up to four output columns, input columns 2c - 1 .. (LEFT: from the one left of the first
// output's own, else the first output's own is the leftmost).  `src`: at input row max(2 r0 - 1, 0); an even number of input rows exists.
template <bool LEFT, typename Put, typename Drained>
__device__ __forceinline__ void irb_rows_s2(uint32_t src, int r0, int r1, const uint32_t (&valid)[3], float ef, float em, float dm, int dbase,
                                            uint32_t k0, uint32_t k1, uint32_t k2, Put put, Drained drained) {
    uint32_t v[9], A[3], win[4];
    irb_tmem_cols<8>(src, v);
    auto row = [&](bool last) {
        ptx::tmem_wait_ld();
        irb_expand<8>(v, valid, ef, em, A);
        src += 16u;
        if (last) drained(); else irb_tmem_cols<8>(src, v);
        if (LEFT) { win[0] = A[0]; win[1] = __byte_perm(A[0], A[1], 0x5432); win[2] = A[1]; win[3] = __byte_perm(A[1], 0u, 0x5432); }
        else { win[0] = __byte_perm(0u, A[0], 0x6543); win[1] = __byte_perm(A[0], A[1], 0x4321); win[2] = __byte_perm(A[0], A[1], 0x6543); win[3] = __byte_perm(A[1], 0u, 0x4321); }
    };
    int cur[4], nxt[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) nxt[x] = dbase;
    if (r0 > 0) {
        row(false);
#pragma unroll
        for (int x = 0; x < 4; ++x) nxt[x] = dw_dp4a<false>(win[x], k0, dbase);
    }
    for (int r = r0; r < r1; ++r) {
        row(false);
#pragma unroll
        for (int x = 0; x < 4; ++x) cur[x] = dw_dp4a<false>(win[x], k1, nxt[x]);
        row(r + 1 == r1);
#pragma unroll
        for (int x = 0; x < 4; ++x) { cur[x] = dw_dp4a<false>(win[x], k2, cur[x]); nxt[x] = dw_dp4a<false>(win[x], k0, dbase); }
        put(r, irb_filtered<4>(cur, dm), 0u);
    }
}

// WC: columns computed per row (the width rounded up to an instantiated value).  S: stride.
template <int WC, int S, bool ADD>
__global__ void __launch_bounds__(kIrbThreads, 1) irb_kernel(const __grid_constant__ IrbArgs a, const __grid_constant__ QAddTail add) {
    constexpr int PITCH = WC > 8 ? 16 : 8, OPITCH = S == 1 ? PITCH : 8, U = PITCH == 16 ? 2 : 1;
    static_assert(S == 1 || (PITCH == 16 && !ADD), "");
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* tail = smem + a.off_tail;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 256);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 260);
    const uint32_t smem0 = ptx::smem_u32(smem), bar0 = ptx::smem_u32(bars);
    auto wfull = [&](int s) { return bar0 + 8u * s; };
    auto wempty = [&](int s) { return bar0 + 8u * (2 + s); };
    auto xfull = [&](int b) { return bar0 + 8u * (4 + b); };
    auto xempty = [&](int b) { return bar0 + 8u * (6 + b); };
    auto d1full = [&](int b) { return bar0 + 8u * (8 + b); };            // b: the unit, or the buffer of the one unit
    auto d1empty = [&](int b) { return bar0 + 8u * (10 + b); };
    auto yfull = [&](int u, int b) { return bar0 + 8u * (12 + 2 * u + b); };
    auto yempty = [&](int u, int b) { return bar0 + 8u * (16 + 2 * u + b); };
    const uint32_t d2full = bar0 + 8u * 20, d2empty = bar0 + 8u * 21, out_free = bar0 + 8u * 22, out_full = bar0 + 8u * 23;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slots = U == 2 ? 2 : a.d1_bufs;
    const int d2_cols = (a.paired ? 1 : a.mt2 * U) * a.n2, cols = slots * a.n1 + d2_cols;
    const uint32_t tmem_cols = cols <= 64 ? 64u : (cols <= 128 ? 128u : (cols <= 256 ? 256u : 512u));

    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(wfull(b), 1); ptx::mbar_init(wempty(b), 1 + kIrbEpiWarps);
            ptx::mbar_init(xfull(b), 1); ptx::mbar_init(xempty(b), ADD ? 1 + kIrbEpiWarps : 1);
            ptx::mbar_init(d1full(b), 1); ptx::mbar_init(d1empty(b), kIrbEpiWarps / U);
            for (int u = 0; u < 2; ++u) { ptx::mbar_init(yfull(u, b), kIrbEpiWarps / U); ptx::mbar_init(yempty(u, b), 1); }
        }
        ptx::mbar_init(d2full, 1); ptx::mbar_init(d2empty, kIrbEpiWarps);
        ptx::mbar_init(out_free, 1); ptx::mbar_init(out_full, kIrbEpiWarps);
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(tmem_slot), tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_trigger();
    if (warp != 0) ptx::grid_wait();                     // (weights are constants)
    const int tile0 = (int)blockIdx.x, tile_step = (int)gridDim.x;               // this CTA's tiles: tile0, tile0 + step, ..
    const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0, chunks = a.chunks;
    const int total = my_tiles * chunks;                 // chunks of this CTA, in order
    const uint32_t xblk = (uint32_t)a.kp * 128u;         // a unit's part of X
    constexpr uint32_t yblk = 16384u;

    // X of tile t into buffer xb, by warp `first` of `step`: 16-byte chunk q of channel c, at chunk position q ^ (c % 8) of the
    // channel's 128-byte row of its unit (the form a box with the 128-byte swizzle has).  A lane keeps its chunk position and walks
    // over the channels, four at a time so that their loads are in flight together.  Whole aligned words are read: the input's size is
    // a multiple of four, and words past its end are not.
    auto build = [&](int t, int xb, int first, int step) {
        const int nq = a.n1 >> 4, HW = a.H * a.W;
        const int words = (int)((long long)a.N * a.C * HW / 4);  // (the host admits less than 2^31 bytes)
        const uint32_t* xw = reinterpret_cast<const uint32_t*>(a.x);
        constexpr int RW = PITCH / 4, R = 16 / PITCH, B = 4, Q = U == 2 ? 16 : 8, CS = 32 / Q;     // words of a row, rows of a chunk; lanes per channel
        const int in1 = S == 1 ? a.rh - 1 : 2 * a.rh - 1;        // first input row of the second unit
        const int ql = lane & (Q - 1), uu = U == 2 ? ql >> 3 : 0, q = ql & 7;
        const bool mine = q < nq;
        const uint32_t dst = smem0 + (uint32_t)(a.off_x + xb * a.x_bytes) + (uint32_t)uu * xblk;
        int off[R]; bool on[R];                                  // byte of the chunk's rows at channel 0
#pragma unroll
        for (int h = 0; h < R; ++h) {
            const int rr = q * R + h, img = R == 1 ? 0 : (rr >= a.H ? 1 : 0), r = R == 1 ? rr + (uu ? in1 : 0) : rr - img * a.H, n = t * a.IB + img;
            on[h] = mine && n < a.N && r < a.H;
            off[h] = on[h] ? (n * a.C * a.H + r) * a.W : 0;
        }
        for (int c0 = lane / Q + first * CS * B; c0 < a.C; c0 += step * CS * B) {
            uint32_t v[B][R][RW + 1];
#pragma unroll
            for (int g = 0; g < B; ++g)
#pragma unroll
                for (int h = 0; h < R; ++h) {
                    const int c = c0 + g * CS, w0 = (off[h] + c * HW) >> 2;
#pragma unroll
                    for (int e = 0; e <= RW; ++e) v[g][h][e] = on[h] && c < a.C && w0 + e < words ? __ldg(xw + w0 + e) : 0u;
                }
#pragma unroll
            for (int g = 0; g < B; ++g) {
                const int c = c0 + g * CS;
                uint32_t o[4];
#pragma unroll
                for (int h = 0; h < R; ++h)
#pragma unroll
                    for (int e = 0; e < RW; ++e) o[h * RW + e] = __funnelshift_r(v[g][h][e], v[g][h][e + 1], 8u * ((uint32_t)(off[h] + c * HW) & 3u));
                if (mine && c < a.C) sts_u128(dst + (uint32_t)c * 128u + (((uint32_t)q ^ ((uint32_t)c & 7u)) << 4), o[0], o[1], o[2], o[3]);
            }
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
    };
    if (warp >= 2 && warp <= 18) {
        // the first tile's operand by all warps that have nothing else to do yet
        if (my_tiles > 0) build(tile0, 0, warp - 2, 17);
        ptx::named_barrier_sync(1, 17 * 32);
    }

    if (warp == 0) {
        // ------------------------------------------------------------------ weights
        if (lane == 0) {
            int s = 0, c = 0; uint32_t ph = 0;
            for (int j = 0; j < total; ++j) {
                if (!ptx::mbar_wait_sleeping(wempty(s), ph ^ 1u, abort_flag)) break;
                ptx::mbar_arrive_expect_tx(wfull(s), (uint32_t)a.w_bytes);
                ptx::bulk_g2s(smem0 + (uint32_t)(s * a.w_bytes), a.w + (size_t)c * a.w_bytes, (uint32_t)a.w_bytes, wfull(s));
                if (++c == chunks) c = 0;
                if (++s == a.w_stages) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (the whole warp runs the loop, one lane issues): expand of
        // chunk j, then project of chunk j - 1, so that the epilogue's next accumulators are on their way while it works
        const uint32_t leader = ptx::elect_one() ? 1u : 0u;
        auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag)) != 0; };
        const uint32_t id1 = ptx::idesc_i8(128, a.n1, true, true) | kIdescBMnMajor, id2 = ptx::idesc_i8(128, a.n2, true, true) | kIdescBMnMajor;
        const int rows2 = a.paired ? 192 : 128;                          // rows of a W2 tile
        const uint64_t da1 = ptx::smem_desc_kmajor(0, 128 * 16, 128), da2 = ptx::smem_desc_kmajor(0, (uint32_t)rows2 * 16u, 128);
        const uint32_t a_hi = (uint32_t)(da1 >> 32), w1_bytes = (uint32_t)a.kp * 128u;
        const uint64_t db = ptx::smem_desc_mnmajor_sw128(0, yblk, 1024); // (one block of 128 columns: no leading offset is used)
        const uint32_t b_hi = (uint32_t)(db >> 32);
        const uint32_t d2 = tmem_base + (uint32_t)(slots * a.n1);
        int s = 0, b = 0, c = 0, xb = 0; uint32_t wph = 0, bph = 0, xph = 0;          // of the expand
        int ps = 0, yb = 0, pc = 0; uint32_t yph = 0, d2ph = 0;                       // of the project, a chunk behind
        bool alive = true;
        for (int j = 0; j <= total && alive; ++j) {
            if (j < total) {
                if (!wait(wfull(s), wph) || (c == 0 && !wait(xfull(xb), xph))) break;
                for (int u = 0; u < U && alive; ++u) {
                    const int slot = U == 2 ? u : b;
                    if (!wait(d1empty(slot), bph ^ 1u)) { alive = false; break; }
                    ptx::tc_fence_after();
                    const uint32_t d = tmem_base + (uint32_t)(slot * a.n1);
                    uint32_t al = (uint32_t)da1 + ((smem0 + (uint32_t)(s * a.w_bytes)) >> 4), bl = (uint32_t)db + ((smem0 + (uint32_t)(a.off_x + xb * a.x_bytes) + (uint32_t)u * xblk) >> 4);
                    for (int k = 0; k < a.kp; k += 32, al += 256u, bl += 256u) ptx::mma_i8_if(leader, d, al, a_hi, bl, b_hi, id1, k > 0 ? 1u : 0u);
                    ptx::mma_commit_if(leader, d1full(slot));
                }
                if (!alive) break;
                if (++s == a.w_stages) { s = 0; wph ^= 1u; }
                if (U == 2) bph ^= 1u; else if (++b == a.d1_bufs) { b = 0; bph ^= 1u; }
                if (++c == chunks) {
                    c = 0;
                    ptx::mma_commit_if(leader, xempty(xb));
                    if (++xb == a.x_bufs) { xb = 0; xph ^= 1u; }
                }
            }
            if (j > 0) {
                const int ks = pc == a.chunks - 1 ? (a.last_live + 31) >> 5 : 4;
                const uint32_t w2 = (smem0 + (uint32_t)(ps * a.w_bytes) + w1_bytes) >> 4, y0 = (smem0 + (uint32_t)(a.off_y + yb * a.y_bytes)) >> 4;
                for (int u = 0; u < U && alive; ++u) {
                    if (!wait(yfull(u, yb), yph) || (pc == 0 && u == 0 && !wait(d2empty, d2ph ^ 1u))) { alive = false; break; }
                    ptx::tc_fence_after();
                    for (int m = 0; m < a.mt2; ++m) {
                        // paired: the filters are rows 64 .. 127 of 192, so that a tile that starts at row 64 (0) has them in lanes 0 .. (64 ..)
                        const uint32_t d = d2 + (uint32_t)((a.paired ? 0 : m * U + u) * a.n2);
                        uint32_t al = (uint32_t)da2 + w2 + (a.paired ? (u == 0 ? 64u : 0u) : (uint32_t)m * 1024u), bl = (uint32_t)db + y0 + (uint32_t)u * (yblk >> 4);
                        for (int k = 0; k < ks; ++k, al += (uint32_t)rows2 * 2u, bl += 256u)
                            ptx::mma_i8_if(leader, d, al, a_hi, bl, b_hi, id2, (pc | k) != 0 || (a.paired && u == 1) ? 1u : 0u);
                    }
                    ptx::mma_commit_if(leader, yempty(u, yb));
                }
                if (!alive) break;
                ptx::mma_commit_if(leader, wempty(ps));
                if (++ps == a.w_stages) ps = 0;
                if (++yb == a.y_bufs) { yb = 0; yph ^= 1u; }
                if (++pc == chunks) { pc = 0; ptx::mma_commit_if(leader, d2full); d2ph ^= 1u; }
            }
        }
    } else if (warp == 18) {
        // ------------------------------------------------------------------ builder: the tiles behind the first
        if (my_tiles > 0 && lane == 0) ptx::mbar_arrive(xfull(0));
        int xb = a.x_bufs > 1 ? 1 : 0; uint32_t xph = a.x_bufs > 1 ? 0u : 1u;
        for (int i = 1; i < my_tiles; ++i) {
            int ok = 1;
            if (lane == 0) ok = ptx::mbar_wait_sleeping(xempty(xb), xph ^ 1u, abort_flag) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            build(tile0 + i * tile_step, xb, 0, 1);
            if (lane == 0) ptx::mbar_arrive(xfull(xb));
            if (++xb == a.x_bufs) { xb = 0; xph ^= 1u; }
        }
    } else if (warp == 19) {
        // ------------------------------------------------------------------ sender: a staged tile leaves as one bulk copy
        if (lane == 0) {
            for (int i = 0; i < my_tiles; ++i) {
                const int t = tile0 + i * tile_step;
                if (!ptx::mbar_wait_sleeping(out_full, (uint32_t)i & 1u, abort_flag)) break;
                const int plane = a.M * a.OH * a.OW;
                ptx::bulk_s2g(a.y + (size_t)t * a.IB * plane, smem0 + (uint32_t)a.off_out, (uint32_t)(min(a.IB, a.N - t * a.IB) * plane));
                ptx::bulk_wait_read<0>();
                ptx::mbar_arrive(out_free);
            }
            ptx::bulk_wait_all();
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quarter = warp & 3, part = (warp - 2) >> 2, ch = quarter * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16), d2 = lane_base + (uint32_t)(slots * a.n1);
        const int OHW = a.OH * a.OW;
        // In the chunks: two units - unit part % 2, the left eight input columns or the rest; one unit - image part % 2, half of its rows.
        const int u = U == 2 ? part & 1 : 0, img = U == 2 ? 0 : part & 1, sub = part >> 1;
        const int u0 = u ? a.rh : 0, u1 = U == 2 && u == 0 ? a.rh : a.OH;                     // the unit's output rows
        const int hr = (a.OH + 1) / 2, r0 = U == 2 ? u0 : (sub ? hr : 0), r1 = U == 2 ? u1 : (sub ? a.OH : hr);
        const int in0 = max(S * r0 - 1, 0);                                                   // first input row
        uint32_t valid[3];
        {
            const int n = U == 2 && sub ? a.W - 7 : a.W;             // (the right part's first input column is 7)
#pragma unroll
            for (int j = 0; j < 3; ++j) valid[j] = n >= 4 * j + 4 ? 0xffffffffu : (n <= 4 * j ? 0u : 0xffffffffu >> (8 * (4 * j + 4 - n)));
        }
        // In the project epilogue: filters 128 mt + ch, or paired the lane's one of 64; unit (image) pu, rows p0, p0 + ps, .. below p1, eight columns from pc0.
        const int pu = a.paired ? quarter >> 1 : part & 1, pm = a.paired ? ch & 63 : ch;
        const int pu0 = U == 2 && pu ? a.rh : 0, pu1 = U == 2 && pu == 0 ? a.rh : a.OH;
        const int pc0 = OPITCH == 16 ? (part >> 1) * 8 : 0, pcols = min(8, a.OW - pc0);
        const int ps = OPITCH == 16 ? (a.paired ? 2 : 1) : (a.paired ? 4 : 2);
        const int p0 = pu0 + (OPITCH == 16 ? (a.paired ? part & 1 : 0) : (a.paired ? part : part >> 1));
        auto wait = [&](uint32_t bar, uint32_t parity) {
            int ok = 1;
            if (lane == 0) ok = ptx::mbar_wait_sleeping(bar, parity, abort_flag) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
        };

        // The project epilogue of this CTA's tile number i: behind the next tile's first chunk, so that its last MMAs have had time.
        auto project = [&](int i) -> bool {
            const int t = tile0 + i * tile_step;
            const int n_here = min(a.IB, a.N - t * a.IB);
            if ((i > 0 && !wait(out_free, (uint32_t)(i - 1) & 1u)) || !wait(d2full, (uint32_t)i & 1u)) return false;
            if (ADD && __all_sync(0xffffffffu, ptx::mbar_wait(xfull(i % a.x_bufs), (uint32_t)(i / a.x_bufs) & 1u, abort_flag)) == 0) return false;
            ptx::tc_fence_after();
            uint8_t* out = smem + a.off_out;
            const uint32_t xs = smem0 + (uint32_t)(a.off_x + (i % a.x_bufs) * a.x_bytes);
            for (int mt = 0; mt < a.mt2; ++mt) {
                if (mt * 128 + (a.paired ? (quarter & 1) * 32 : quarter * 32) >= a.M || (U == 1 && pu >= n_here) || p0 >= pu1) break;
                const int m = mt * 128 + pm;
                const bool live = m < a.M;
                const float mlt = live ? __ldg(a.mult2 + m) : 1.0f;
                const int bs = live ? __ldg(a.bias2 + m) : 0;
                uint32_t src = d2 + (uint32_t)((a.paired ? 0 : (U == 2 ? mt * 2 + pu : mt) * a.n2) + (U == 2 ? p0 - pu0 : pu * a.OH + p0) * OPITCH + pc0);
                uint8_t* o = out + ((size_t)(U == 2 ? 0 : pu) * a.M + m) * OHW + p0 * a.OW + pc0;
                uint32_t v[9];
                irb_tmem_cols<8>(src, v);
                for (int r = p0; r < pu1; r += ps, o += ps * a.OW) {
                    ptx::tmem_wait_ld();
                    uint32_t pk[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        pk[j] = pack_sat_s8x4(rq_round((int)v[4 * j] + bs, mlt), rq_round((int)v[4 * j + 1] + bs, mlt), rq_round((int)v[4 * j + 2] + bs, mlt), rq_round((int)v[4 * j + 3] + bs, mlt));
                    src += (uint32_t)(ps * OPITCH);
                    if (r + ps < pu1) irb_tmem_cols<8>(src, v);
                    if constexpr (ADD) {
                        // the block's input at this channel (m < C == M) and row, from the operand
                        const uint32_t rr = (uint32_t)(U == 2 ? r - (pu ? a.rh - 1 : 0) : pu * a.H + r), q = PITCH == 16 ? rr : rr >> 1;
                        const uint32_t ad = xs + (U == 2 ? (uint32_t)pu * xblk : 0u) + (uint32_t)min(m, a.kp - 1) * 128u + (((q & 7u) ^ ((uint32_t)m & 7u)) << 4) + (PITCH == 16 ? (uint32_t)pc0 : (rr & 1u) * 8u);
                        pk[0] = qadd_word<false>(lds_u32<0>(ad), pk[0], add);
                        pk[1] = qadd_word<false>(lds_u32<4>(ad), pk[1], add);
                        __syncwarp();
                    }
                    if (live) {
                        if ((a.OW & 3) == 0) {
                            *reinterpret_cast<uint32_t*>(o) = pk[0];
                            if (pcols > 4) *reinterpret_cast<uint32_t*>(o + 4) = pk[1];
                        } else if ((a.OW & 1) == 0) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) if (2 * k < pcols) *reinterpret_cast<uint16_t*>(o + 2 * k) = (uint16_t)(pk[k / 2] >> (16 * (k % 2)));
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k) if (k < pcols) o[k] = (uint8_t)(pk[k / 4] >> (8 * (k % 4)));
                        }
                    }
                }
            }
            ptx::tc_fence_before();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(d2empty);
                if (ADD) ptx::mbar_arrive(xempty(i % a.x_bufs));
                ptx::mbar_arrive(out_full);
            }
            return true;
        };

        int s = 0, b = 0, yb = 0, c = 0, tile_i = 0; uint32_t wph = 0, bph = 0, yph = 0;
        bool alive = true;
        for (int j = 0; j < total; ++j) {
            const int slot = U == 2 ? u : b;
            // (every lane waits for the weights: each reads its channel's constants)
            alive = __all_sync(0xffffffffu, ptx::mbar_wait_sleeping(wfull(s), wph, abort_flag)) != 0 && wait(yempty(u, yb), yph ^ 1u) && wait(d1full(slot), bph);
            if (!alive) break;
            ptx::tc_fence_after();
            auto drained = [&]() {
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(d1empty(slot));      // this warp has read its accumulators
            };
            if (c < a.chunks - 1 || quarter * 32 < a.last_live) {
                const uint32_t cs = smem0 + (uint32_t)(s * a.w_bytes + a.kp * 128 + a.w2_bytes + ch * 32);
                const uint4 k0 = lds_u128(cs), k1 = lds_u128(cs + 16u);
                const float ef = __uint_as_float(k0.x), em = __uint_as_float(k0.y), dm = __uint_as_float(k0.z);
                // the unit's accumulators start at its first input row, the one unit's at the first image's
                const uint32_t d1 = lane_base + (uint32_t)(slot * a.n1 + (U == 2 ? 0 : (img * a.H + in0) * PITCH)), yrow = smem0 + (uint32_t)(a.off_y + yb * a.y_bytes + ch * 128) + (uint32_t)u * yblk;
                auto put = [&](int r, uint32_t v0, uint32_t v1) {
                    const uint32_t rr = (uint32_t)(U == 2 ? r - u0 : img * a.OH + r), q = OPITCH == 16 ? rr : rr >> 1;
                    const uint32_t ad = yrow + (((q & 7u) ^ ((uint32_t)ch & 7u)) << 4) + (OPITCH == 16 ? 0u : (rr & 1u) * 8u);
                    if (S == 2) asm volatile("st.shared.u32 [%0], %1;" ::"r"(ad + (uint32_t)sub * 4u), "r"(v0) : "memory");
                    else asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(ad + (PITCH == 16 ? (uint32_t)sub * 8u : 0u)), "r"(v0), "r"(v1) : "memory");
                };
                if constexpr (S == 2) {
                    if (sub == 0) irb_rows_s2<false>(d1, r0, r1, valid, ef, em, dm, (int)k0.w, k1.x, k1.y, k1.z, put, drained);
                    else irb_rows_s2<true>(d1 + 7u, r0, r1, valid, ef, em, dm, (int)k0.w, k1.x, k1.y, k1.z, put, drained);
                } else if constexpr (PITCH == 16) {
                    if (sub == 0) irb_rows<8, false, true, 16>(d1, a.H, r0, r1, valid, ef, em, dm, (int)k0.w, k1.x, k1.y, k1.z, put, drained);
                    else irb_rows<WC - 8, true, false, 16>(d1 + 7u, a.H, r0, r1, valid, ef, em, dm, (int)k0.w, k1.x, k1.y, k1.z, put, drained);
                } else {
                    irb_rows<WC, false, false, 8>(d1, a.H, r0, r1, valid, ef, em, dm, (int)k0.w, k1.x, k1.y, k1.z, put, drained);
                }
            } else {
                drained();
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) { ptx::mbar_arrive(yfull(u, yb)); ptx::mbar_arrive(wempty(s)); }
            if (++s == a.w_stages) { s = 0; wph ^= 1u; }
            if (U == 2) bph ^= 1u; else if (++b == a.d1_bufs) { b = 0; bph ^= 1u; }
            if (++yb == a.y_bufs) { yb = 0; yph ^= 1u; }
            if (c == 0 && tile_i > 0) {
                alive = project(tile_i - 1);
                if (!alive) break;
            }
            if (++c == chunks) { c = 0; ++tile_i; }
        }
        if (alive && my_tiles > 0) project(my_tiles - 1);
    }

    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) ptx::tmem_dealloc(tmem_base, tmem_cols);
    if (tid == 0 && *abort_flag) atomicExch(a.status, (int)DEV_ERR_WAIT_TIMEOUT);
}

// =============================================================================================
// Host side
// =============================================================================================
struct IrbPlan {
    IrbArgs a{};
    int wc = 0, E = 0, stride = 1;
    size_t smem_bytes = 0;
};

// Geometry of the three convolutions; false when the kernel does not take them.  With the addition the operand X of a tile is read by the
// project epilogue, behind the next tile's first chunk: it needs a second buffer.
inline bool irb_plan(const ConvGeom& e, const ConvGeom& d, const ConvGeom& p, bool add, IrbPlan& q) {
    auto pointwise = [](const ConvGeom& g) { return g.G == 1 && g.KH == 1 && g.KW == 1 && g.sh == 1 && g.sw == 1 && !g.pt && !g.pl && !g.pb && !g.pr; };
    if (!pointwise(e) || !pointwise(p)) return false;
    if (d.G != d.C || d.M != d.C || d.KH != 3 || d.KW != 3 || d.sh != d.sw || d.sh < 1 || d.sh > 2 || d.dh != 1 || d.dw != 1 || d.pt != 1 || d.pl != 1 || d.pb != 1 || d.pr != 1) return false;
    const bool two = e.W > 8;                                            // units
    if (e.N <= 0 || e.H > (two ? 14 : 8) || e.W > 16 || e.H < 2 || e.W < 3 || e.C > 512 || p.M > 512 || e.M < 128 || e.M > 4096) return false;
    if (d.sh == 2 && (!two || add || e.H % 2 != 0 || e.W % 2 != 0 || e.H < 4 || e.W > 14)) return false;
    if ((long long)e.N * e.C * e.H * e.W % 4 != 0 || (long long)p.M * d.OH * d.OW % 16 != 0 || (long long)e.N * std::max(e.C, p.M) * e.H * e.W > 0x7fffffffLL) return false;
    IrbArgs& a = q.a;
    a = IrbArgs{};
    a.N = e.N; a.C = e.C; a.M = p.M; a.H = e.H; a.W = e.W; a.OH = d.OH; a.OW = d.OW;
    q.E = e.M; q.stride = d.sh;
    q.wc = d.sh == 2 ? 16 : (e.W <= 4 ? 4 : (e.W <= 6 ? 6 : (e.W == 7 ? 7 : (e.W <= 8 ? 8 : (e.W <= 10 ? 10 : (e.W <= 12 ? 12 : (e.W <= 14 ? 14 : 16)))))));
    a.IB = two ? 1 : 2;
    a.tiles = (e.N + a.IB - 1) / a.IB;
    a.rh = (a.OH + 1) / 2;
    if (two) {
        // input rows of a unit: those of its output rows and one (stride 2: as many as are read) beyond the cut
        a.n1 = 16 * (d.sh == 1 ? a.rh + 1 : std::max(2 * a.rh, e.H - 2 * a.rh + 1));
        a.n2 = d.sh == 1 ? 16 * a.rh : (8 * a.rh + 15) / 16 * 16;
    } else {
        a.n1 = a.n2 = 16 * e.H;
    }
    a.chunks = (q.E + 127) / 128; a.last_live = q.E - (a.chunks - 1) * 128;
    a.kp = (e.C + 31) / 32 * 32;
    a.mt2 = (p.M + 127) / 128;
    a.paired = two && p.M <= 64;
    const int d2_cols = (a.paired ? 1 : a.mt2 * (two ? 2 : 1)) * a.n2;
    if ((two ? 2 : 1) * a.n1 + d2_cols > 512 || a.n1 > 128) return false;
    a.d1_bufs = !two && 2 * a.n1 + d2_cols <= 512 ? 2 : 1;
    a.w2_bytes = a.paired ? 8 * 192 * 16 : a.mt2 * 16384;
    a.w_bytes = a.kp * 128 + a.w2_bytes + 128 * (int)sizeof(IrbConst);
    a.x_bytes = (two ? 2 : 1) * a.kp * 128; a.y_bytes = (two ? 2 : 1) * 16384;
    const int out_bytes = (a.IB * a.M * a.OH * a.OW + 127) / 128 * 128;
    // as many buffers as fit: the input's first, then the operand between the products
    for (int n = 0; n < (add ? 2 : 4); ++n) {
        a.w_stages = 2; a.x_bufs = n < 2 ? 2 : 1; a.y_bufs = n % 2 == 0 ? 2 : 1;
        a.off_x = (a.w_stages * a.w_bytes + 1023) / 1024 * 1024;
        a.off_y = a.off_x + a.x_bufs * a.x_bytes;
        a.off_out = a.off_y + a.y_bufs * a.y_bytes;
        a.off_tail = a.off_out + out_bytes;
        q.smem_bytes = (size_t)a.off_tail + 512;
        if (q.smem_bytes <= 227 * 1024) return true;
    }
    return false;
}

// Whether the block is faster as one kernel than as three, or four with the addition.  One kernel takes rounds of the SMs whose time is a
// tile's; the separate ones, a launch each more and the expanded tensor through memory, take a time that grows with the images.  `long_add`: an
// addition whose short form is not proved (15 instructions a value instead of 6.5), which costs the one kernel more.  Measured inside plans, 43 shapes
// of 3 to 14 rows, 16 to 160 channels, 1 to 1500 images; below, us as one kernel / separate, with 14 us of other steps:
//   two units, stride 1, planes of whole words: a tile takes about 6.6 us a chunk less 1.3, at 14 rows, the separate kernels 17.5, or 21.5 where rows
//     are not whole words too, and 3.2 per million expanded values (96 -> 576 at 14 x 14: 8 images 36 / 33, 32 36 / 38, 148 39 / 61, 1024 192 / 282; at
//     12 x 12: 24 images 35 / 30, 64 35 / 36, 148 37 / 50; at 10 x 10: 16 images 30 / 32; 32 -> 192 at 12 x 12: 148 images 26 / 36, 768 86 / 84, 1500
//     150 / 144); with the long addition 2 + 5 us a chunk, at least 13.5, against 16 and 2.25 (96 -> 576 at 14 x 14: 8 images 43 / 34, 48 44 / 42, 148
//     47 / 66; 16 -> 128: 148 images 27 / 37, 768 119 / 86)
//   two units, stride 2 or planes that are not whole words, which the separate kernels put through an im2col pass: always (stride 2, 8 images 30 /
//     33, 1024 132 / 197; 96 -> 576 at 11 x 11: 8 images 45 / 51, 160 84 / 104, 1500 368 / 557; 32 -> 192 at 13 x 13: 34 / 45, 48 / 80, 247 / 357)
//   one unit, seven rows or more, chunks on one CTA: from about three tiles a chunk on (160 -> 960 -> 320 at 7 x 7: 16 tiles 50 / 47, 24 53 / 54, 52
//     54 / 67; 64 -> 384 at 8 x 8: 8 tiles 23 / 27); fewer rows: always (160 -> 960 -> 320 at 6 x 6: 19 tiles 39 / 40, 52 40 / 70; at 4 x 4: 19 29 / 38)
//   planes of less than 16 pixels, a quarter of whose columns exist: while there are few rounds of few chunks (160 -> 960 at 3 x 3: 768 images 77 / 85,
//     1024 95 / 93, 1500 127 / 115; with the long addition 768 90 / 91, 1024 109 / 96)
// Below eight tiles the separate kernels use more of the chip (160 -> 960 at 4 x 4: 4 tiles 19 / 19, 64 -> 384 at 6 x 6: 2 tiles 20 / 19).
inline bool irb_pays(const IrbPlan& q, bool long_add, int sm_count) {
    const IrbArgs& a = q.a;
    if (a.tiles < 8) return false;
    const long long rounds = (a.tiles + sm_count - 1) / sm_count;
    if (a.IB == 1) {
        if (q.stride == 2 || a.H * a.W % 4 != 0) return true;
        const double values = 1e-6 * a.N * q.E * a.H * a.W;
        const double tile = long_add ? std::max(13.5, 2.0 + 5.0 * a.chunks) : std::max(8.0, 6.6 * a.chunks - 1.3);
        return rounds * tile * a.H / 14 <= (long_add ? 16.0 + 2.25 * values : (a.W % 4 != 0 ? 21.5 : 17.5) + 3.2 * values);
    }
    if (a.H >= 7 && a.tiles + 1 < 3 * a.chunks) return false;
    return a.H * a.W >= 16 || rounds * a.chunks <= (long_add ? 16 : 30);
}

// Weights and constants per chunk; false when an accumulator could leave the range of kAccBase.  eb, db: biases with -x_zp * sum(w) folded in.
inline bool irb_prepare(const IrbPlan& q, const int8_t* we, const float* em, const int32_t* eb, const int8_t* wd, const float* dm, const int32_t* db,
                        const int8_t* wp, std::vector<uint8_t>& out) {
    const IrbArgs& a = q.a;
    out.assign((size_t)a.chunks * a.w_bytes, 0);
    for (int e = 0; e < q.E; ++e) {
        uint8_t* stage = out.data() + (size_t)(e / 128) * a.w_bytes;
        const int r = e % 128;
        const int8_t* w = we + (size_t)e * a.C;
        int s1 = 0, s2 = 0;
        for (int c = 0; c < a.C; ++c) s1 += std::abs((int)w[c]);
        for (int c = 0; c < a.C; c += 16) std::memcpy(stage + ((size_t)(c / 16) * 128 + r) * 16, w + c, std::min(16, a.C - c));
        IrbConst k{};
        for (int i = 0; i < 9; ++i) { k.k[i / 3] |= (uint32_t)(uint8_t)wd[e * 9 + i] << (8 * (i % 3)); s2 += std::abs((int)wd[e * 9 + i]); }
        if (!acc_base_ok(eb[e]) || !acc_base_ok(db[e]) || s1 * 128 + std::abs(eb[e]) >= (1 << 22) || s2 * 128 + std::abs(db[e]) >= (1 << 22)) return false;
        k.e_floor = kAccBase - (float)eb[e]; k.e_mult = em[e]; k.d_mult = dm[e]; k.d_base = kAccBaseBits + db[e];
        std::memcpy(stage + (size_t)a.kp * 128 + (size_t)a.w2_bytes + (size_t)r * sizeof(IrbConst), &k, sizeof k);
    }
    for (int m = 0; m < a.M; ++m)
        for (int e = 0; e < q.E; e += 16) {
            const int k16 = e % 128 / 16;
            const size_t at = a.paired ? ((size_t)k16 * 192 + 64 + m) * 16 : (size_t)(m / 128) * 16384 + ((size_t)k16 * 128 + m % 128) * 16;
            std::memcpy(out.data() + (size_t)(e / 128) * a.w_bytes + (size_t)a.kp * 128 + at, wp + (size_t)m * q.E + e, std::min(16, q.E - e));
        }
    return true;
}

// x: 4-byte aligned, y: 16-byte aligned.
inline int32_t irb_run(zant_ctx* ctx, const IrbPlan& q, const void* x, const uint8_t* w, const float* mult2, const int32_t* bias2, void* y, const QAddTail* add) {
    IrbArgs a = q.a;
    a.x = (const uint8_t*)x; a.y = (uint8_t*)y; a.w = w; a.mult2 = mult2; a.bias2 = bias2; a.status = ctx->status_word;
    const int grid = std::min(a.tiles, ctx->sm_count);
    auto go = [&](auto wc, auto stride, auto with) -> int32_t {
        constexpr int WC = decltype(wc)::value, S = decltype(stride)::value;
        constexpr bool ADD = decltype(with)::value;
        ZB_SMEM_ATTR(ctx, (irb_kernel<WC, S, ADD>), 227 * 1024);
        launch_const(ctx, irb_kernel<WC, S, ADD>, grid, kIrbThreads, q.smem_bytes, a, add ? *add : QAddTail{});
        return check_launch(ctx, "irb_kernel");
    };
    using one = std::integral_constant<int, 1>;
    if (q.stride == 2) return go(std::integral_constant<int, 16>{}, std::integral_constant<int, 2>{}, std::false_type{});
    auto pick = [&](auto wc) -> int32_t { return add ? go(wc, one{}, std::true_type{}) : go(wc, one{}, std::false_type{}); };
    switch (q.wc) {
        case 4: return pick(std::integral_constant<int, 4>{});
        case 6: return pick(std::integral_constant<int, 6>{});
        case 7: return pick(std::integral_constant<int, 7>{});
        case 8: return pick(std::integral_constant<int, 8>{});
        case 10: return pick(std::integral_constant<int, 10>{});
        case 12: return pick(std::integral_constant<int, 12>{});
        case 14: return pick(std::integral_constant<int, 14>{});
        default: return pick(std::integral_constant<int, 16>{});
    }
}

}  // namespace zb
