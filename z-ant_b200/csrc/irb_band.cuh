// Inverted residual block for few images or wide planes as one kernel: QLinearConv 1x1 (expand, ReLU / ReLU6) -> QLinearConv depthwise 3x3
// (pads 1, stride 1 or 2, ReLU / ReLU6) -> QLinearConv 1x1 (project) [-> QLinearAdd with the block's input], int8 with zero point 0 between
// them.  irb_q8.cuh is the form for many images on small planes.
//
// A block of a network run on a few images is 10^5 to 10^7 multiplications: as three or four launches it is three or four load latencies, and a
// kernel that gives an SM a whole image leaves most of the SMs idle.  Here a tile is a band of output rows of one image, all columns, with the
// input rows that its filter reads (those at its edge are expanded by two bands), and the 16-channel tiles of the expanded tensor are dealt to a
// cluster of up to eight CTAs.  How many rows and CTAs is decided by measured times (irb_band_plan).  A CTA, per chunk of its channels:
//   expand     E [channel][pixel] = requantised W1 X on warp-level MMAs (m16n8k32): the input's rows lie in shared memory as in memory (a channel's
//              pixels contiguous, rows P bytes apart), and ldmatrix transposes 16 x 16 bytes of them into an MMA's B operand
//   depthwise  a thread owns four columns of a channel and walks over the rows (dp4a on windows cut by byte permutes)      -> D [channel][pixel]
//   project    D's sums for all filters, the same way; kept in shared memory between chunks
// At the end each CTA of a cluster sends its sums, 16 filters x 8 pixels a block, to the CTA of the cluster that adds this block up and requantises it
// (32-bit integers, exact in any order): writes into the other's shared memory, one cluster barrier, no global traffic.
//
// What bounds it: latency.  A launch on one image of 14 x 14 x 384 takes 4.6 us: 1.3 of launch, 0.5 for the input, 0.4 expand, 0.4 filter, 0.6
// project and sending, 0.6 barrier, 0.5 adding up (clock counts of one CTA); as separate launches the block was 12.8 us, 17 with the addition.
// MobileNetV2-style plans: one image of 224 x 224 246 -> 121 us, 37 of 160 x 160 373 -> 250, 8 of 128 x 128 269 -> 119.  With the SMs full (512
// images) it is bound by issue, at half the rate of irb_q8.cuh.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "context.cuh"
#include "dwconv_q8.cuh"
#include "fused_cnn.cuh"
#include "geometry.hpp"
#include "irb_q8.cuh"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"

namespace zb {

struct IrbBandArgs {
    const uint8_t* x; uint8_t* y; const uint8_t* w;        // w: per chunk [W1 | W2 | IrbConst of its channels | (multiplier, bias) of the filters]
    int N, C, M, H, W, OH, OW;
    int rb, bands;                 // output rows of a band, bands of an image
    int cs, chunks;                // CTAs of a cluster, chunks of a CTA
    int ct;                        // 16-channel tiles of a chunk
    int P, OP;                     // bytes between rows of X and E, of D: multiples of four
    int xp, ep, dp;                // bytes between channels of X, E, D: odd multiples of 16 (ldmatrix and the stores then spread over the banks)
    int in_rows, dpx;              // most input rows of a band; pixels of D rounded up to 32
    int ks1, ks2, mt2;             // K steps of 32 of the two products (the second's per chunk), 16-filter tiles
    int nm1, nm2;                  // 16-row tiles of an item of the products: 1 or 2
    int segs, seg_rows;            // depthwise: parts of the band's rows, for different threads
    uint32_t per_magic, pw_magic, op_magic, opw_magic, ch_magic, cs_magic;       // divisions by in_rows * P / 4, P / 4, OP, OP / 4, 16 ct, cs
    int chunk_bytes, w_stages;
    int off_x, off_e, off_d, off_sum, off_recv, off_w, off_tail;
    int give_up;                   // self test: a CTA whose first wait counts as run out (-1: none)
    int* status;
};

constexpr int kIrbBandThreads = 384;                        // at most; 256 where that is the faster

// floor(i / d) for i * d < 2^32 (magic = floor(2^32 / d) + 1, 0 for d == 1)
__device__ __forceinline__ uint32_t div_magic(uint32_t i, uint32_t magic) { return magic ? __umulhi(i, magic) : i; }
inline uint32_t magic_of(uint32_t d) { return d == 1 ? 0u : (uint32_t)(0x100000000ull / d + 1); }

// Two 16 x 16 byte blocks, rows (K) 0..15 and 16..31 at the lanes' addresses, transposed: r[0], r[2] are the two B registers of the left eight
// columns, r[1], r[3] of the right.
__device__ __forceinline__ void ldmatrix_b_32x16(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_m16n8k32_s8(int (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory"); return v; }
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

// NM 16-row tiles of A (fragment order, `second` bytes apart) times 32 (wide) or 16 columns of B (K rows `pitch32` / 32 bytes apart).
template <int NM>
__device__ __forceinline__ void irb_band_gemm(int (&acc)[2][4][4], uint32_t b, uint32_t pitch32, uint32_t wa, uint32_t second, int steps, bool wide) {
#pragma unroll 2
    for (int ks = 0; ks < steps; ++ks, b += pitch32, wa += 512u) {
        uint32_t b0[4], b1[4];
        ldmatrix_b_32x16(b, b0);
        if (wide) ldmatrix_b_32x16(b + 16u, b1);
#pragma unroll
        for (int i = 0; i < NM; ++i) {
            const uint4 w = lds_u128(wa + (i ? second : 0u));
            mma_m16n8k32_s8(acc[i][0], w, b0[0], b0[2]); mma_m16n8k32_s8(acc[i][1], w, b0[1], b0[3]);
            if (wide) { mma_m16n8k32_s8(acc[i][2], w, b1[0], b1[2]); mma_m16n8k32_s8(acc[i][3], w, b1[1], b1[3]); }
        }
    }
}

// S: stride.  CLUSTER: more than one CTA a tile.
template <int S, bool ADD, bool CLUSTER>
__global__ void __launch_bounds__(kIrbBandThreads, 2) irb_band_kernel(const __grid_constant__ IrbBandArgs a, const __grid_constant__ QAddTail add) {
    static_assert(!ADD || S == 1, "");
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t s0 = ptx::smem_u32(smem);
    const int tid = threadIdx.x, threads = (int)blockDim.x, warps = threads >> 5, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const uint32_t bar = s0 + (uint32_t)a.off_tail, zero = bar + 32u;            // two barriers, the abort flag, a word of zeros
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + a.off_tail + 16);
    const int cs = CLUSTER ? a.cs : 1, rank = CLUSTER ? (int)blockIdx.x % cs : 0, tile = (int)blockIdx.x / cs;
    const int n = tile / a.bands, o0 = (tile - n * a.bands) * a.rb, o1 = min(o0 + a.rb, a.OH);       // output rows
    const int in0 = max(S * o0 - 1, 0), in1 = min(S * (o1 - 1) + 2, a.H);                            // input rows
    const uint8_t* wsrc = a.w + (size_t)rank * a.chunks * a.chunk_bytes;
    if (tid == 0) {
        ptx::mbar_init(bar, 1); ptx::mbar_init(bar + 8u, 1);
        *abort_flag = 0;
        ptx::mbar_fence_init();
        for (int i = 0; i < a.w_stages; ++i) {
            ptx::mbar_arrive_expect_tx(bar + 8u * i, (uint32_t)a.chunk_bytes);
            ptx::bulk_g2s(s0 + (uint32_t)(a.off_w + i * a.chunk_bytes), wsrc + (size_t)i * a.chunk_bytes, (uint32_t)a.chunk_bytes, bar + 8u * i);
        }
        sts_u32(zero, 0u);
    }
    __syncthreads();                                                             // (the barriers are set up before any thread waits on one)
    if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // this CTA's shared memory may be written to
    ptx::grid_trigger();
    ptx::grid_wait();
    // The band's input rows, P bytes apart, channels xp apart; whole aligned words are read, none past the input's end.  (Columns from W on are
    // whatever follows.)
    {
        const int PW = a.P >> 2, per = a.in_rows * PW, total = a.C * per, rows = in1 - in0, HW = a.H * a.W, words = (int)((long long)a.N * a.C * HW >> 2);
        const uint32_t* xw = reinterpret_cast<const uint32_t*>(a.x);
        const int base = (n * a.C * a.H + in0) * a.W;
        for (int i0 = tid; i0 < total; i0 += threads * 4) {
            uint32_t v[4][2], dst[4]; int off[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * threads, c = (int)div_magic(i, a.per_magic), r = i - c * per, row = (int)div_magic(r, a.pw_magic), j = r - row * PW;
                const bool on = i < total && row < rows;
                off[k] = base + c * HW + row * a.W + 4 * j;
                dst[k] = on ? s0 + (uint32_t)(a.off_x + c * a.xp + row * a.P + 4 * j) : 0u;
                const int w0 = off[k] >> 2;
                v[k][0] = on ? __ldg(xw + w0) : 0u;
                v[k][1] = on && (off[k] & 3) && w0 + 1 < words ? __ldg(xw + w0 + 1) : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (dst[k]) sts_u32(dst[k], __funnelshift_r(v[k][0], v[k][1], 8u * ((uint32_t)off[k] & 3u)));
        }
    }
    ptx::mbar_wait(bar, 0u, abort_flag);                                         // the first chunk's weights
    if ((int)blockIdx.x == a.give_up) *abort_flag = 1;
    __syncthreads();
    const int px_in = (in1 - in0) * a.P, px_out = (o1 - o0) * a.OP, CH = a.ct * 16;
    const int g1 = (px_in + 31) >> 5, g2 = (px_out + 31) >> 5, mp1 = (a.ct + a.nm1 - 1) / a.nm1, mp2 = (a.mt2 + a.nm2 - 1) / a.nm2;
    uint32_t pc = 0;                                                             // the chunk's (multiplier, bias) of the filters
    // Four finished sums: filter m, pixels px .. of D's rows.
    auto emit = [&](const int (&v)[4], int m, int px) {
        const int row = (int)div_magic(px, a.op_magic), col = px - row * a.OP, o = o0 + row;
        if (o >= o1 || col >= a.OW || m >= a.M) return;
        const uint2 c = lds_u64(pc + (uint32_t)m * 8u);
        const float mlt = __uint_as_float(c.x); const int bs = (int)c.y;
        uint32_t pk = pack_sat_s8x4(rq_round(v[0] + bs, mlt), rq_round(v[1] + bs, mlt), rq_round(v[2] + bs, mlt), rq_round(v[3] + bs, mlt));
        if constexpr (ADD) pk = qadd_word<false>(lds_u32<0>(s0 + (uint32_t)(a.off_x + m * a.xp + (o - in0) * a.P + col)), pk, add);
        uint8_t* y = a.y + ((size_t)(n * a.M + m) * a.OH + o) * a.OW + col;
        if ((a.OW & 3) == 0) *reinterpret_cast<uint32_t*>(y) = pk;
        else if ((a.OW & 1) == 0) { *reinterpret_cast<uint16_t*>(y) = (uint16_t)pk; if (col + 2 < a.OW) *reinterpret_cast<uint16_t*>(y + 2) = (uint16_t)(pk >> 16); }
        else {
#pragma unroll
            for (int k = 0; k < 4; ++k) if (col + k < a.OW) y[k] = (uint8_t)(pk >> (8 * k));
        }
    };
    const int er = g + 8 * (q & 1), ep = 4 * (q >> 1);                           // row and first pixel that this lane has of a finished 16 x 8 block
    for (int ck = 0; ck < a.chunks; ++ck) {
        const int ws = a.w_stages == 1 ? 0 : ck & 1;
        if (ck > 0) { ptx::mbar_wait(bar + 8u * ws, (uint32_t)(ck >> 1) & 1u, abort_flag); __syncwarp(); }
        const uint32_t w1 = s0 + (uint32_t)(a.off_w + ws * a.chunk_bytes), w2 = w1 + (uint32_t)(a.ct * a.ks1 * 512), kc = w2 + (uint32_t)(a.mt2 * a.ks2 * 512);
        pc = kc + (uint32_t)a.ct * 512u;
        // ------------------------------------------------------------ expand: items of 32 pixels and one or two 16-channel tiles
        auto expand = [&](auto tiles_of_item) {
            constexpr int NM = decltype(tiles_of_item)::value;
            for (int it = warp; it < g1 * mp1; it += warps) {
                const int mp = it / g1, px0 = (it - mp * g1) * 32;
                const bool wide = px0 + 16 < px_in;
                int acc[2][4][4];
#pragma unroll
                for (int i = 0; i < NM; ++i)
#pragma unroll
                    for (int t = 0; t < 4; ++t)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[i][t][e] = kAccBaseBits;
                irb_band_gemm<NM>(acc, s0 + (uint32_t)(a.off_x + lane * a.xp + px0), 32u * a.xp, w1 + (uint32_t)(mp * NM * a.ks1 * 512 + lane * 16),
                                  NM * mp + 1 < a.ct ? (uint32_t)(a.ks1 * 512) : 0u, a.ks1, wide);
#pragma unroll
                for (int i = 0; i < NM; ++i) {
                    if (i && NM * mp + i >= a.ct) break;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int ch = (NM * mp + i) * 16 + g + 8 * h;
                        const uint2 c = lds_u64(kc + (uint32_t)ch * 32u);
                        const float ef = __uint_as_float(c.x), em = __uint_as_float(c.y);
                        const uint32_t dst = s0 + (uint32_t)(a.off_e + ch * a.ep + px0 + 2 * q);
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            if (t == 2 && !wide) break;
                            int r0, r1;
                            sub_mul_rn2(max(acc[i][t][2 * h], (int)c.x), max(acc[i][t][2 * h + 1], (int)c.x), ef, em, r0, r1);
                            asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + 8u * t), "h"((uint16_t)pack_sat_s8x2(r0, r1)) : "memory");
                        }
                    }
                }
            }
        };
        if (a.nm1 == 2) expand(std::integral_constant<int, 2>{}); else expand(std::integral_constant<int, 1>{});
        __syncthreads();
        // ------------------------------------------------------------ depthwise: a task is four columns of a channel over a part of the rows
        const int OPW = a.OP >> 2, PW = a.P >> 2, tasks = OPW * CH * a.segs;
        for (int i = tid; i < tasks; i += threads) {
            const int cj = (int)div_magic(i, a.opw_magic), j = i - cj * OPW, sg = (int)div_magic(cj, a.ch_magic), c = cj - sg * CH;
            const int r0 = o0 + sg * a.seg_rows, r1 = min(r0 + a.seg_rows, o1);
            if (r0 >= r1) break;
            const uint32_t cst = kc + (uint32_t)c * 32u;
            const uint4 kk = lds_u128(cst + 16u);                                // x, y, z: the filter's rows
            const uint2 c2 = lds_u64(cst + 8u);
            const float dm = __uint_as_float(c2.x);
            const int db = (int)c2.y;
            uint32_t d = s0 + (uint32_t)(a.off_d + c * a.dp + (r0 - o0) * a.OP + 4 * j);
            // three words of an input row: the one left of the first output's own, that one, the next; zero where a word or column does not exist
            const int lo = max(S * r0 - 1, 0), hi = min(S * (r1 - 1) + 1, a.H - 1), fw = S * j, left = a.W - 4 * fw;
            uint32_t pm = s0 + (uint32_t)(a.off_e + c * a.ep + (lo - in0) * a.P + 4 * fw), pl = j > 0 ? pm - 4u : zero, pr = fw + 1 < PW ? pm + 4u : zero;
            const uint32_t im = (uint32_t)a.P, il = j > 0 ? im : 0u, ir_ = fw + 1 < PW ? im : 0u;
            const uint32_t mask_m = left >= 4 ? 0xffffffffu : 0xffffffffu >> (8 * (4 - left));
            const uint32_t mask_r = S == 1 || left >= 8 ? 0xffffffffu : (left <= 4 ? 0u : 0xffffffffu >> (8 * (8 - left)));   // (stride 1 uses one byte of it, which exists)
            struct Row { uint32_t l, m, r; };
            auto fetch = [&](Row& w) { w.l = lds_u32<0>(pl); w.m = lds_u32<0>(pm) & mask_m; w.r = lds_u32<0>(pr) & mask_r; pl += il; pm += im; pr += ir_; };
            auto windows = [&](const Row& w, uint32_t (&win)[4]) {
                win[0] = __byte_perm(w.l, w.m, 0x6543);
                if (S == 1) { win[1] = w.m; win[2] = __byte_perm(w.m, w.r, 0x4321); win[3] = __byte_perm(w.m, w.r, 0x5432); }
                else { win[1] = w.m >> 8; win[2] = __byte_perm(w.m, w.r, 0x6543); win[3] = w.r >> 8; }
            };
            auto put = [&](const int (&s)[4]) { sts_u32(d, irb_filtered<4>(s, dm)); d += (uint32_t)a.OP; };
            if (a.seg_rows == 1) {
                Row w[3] = {{0u, 0u, 0u}, {0u, 0u, 0u}, {0u, 0u, 0u}};           // (all nine loads in flight together)
                if (S * r0 > 0) fetch(w[0]);
                fetch(w[1]);
                if (S * r0 + 1 < a.H) fetch(w[2]);
                int acc[4] = {db, db, db, db};
                const uint32_t rows[3] = {kk.x, kk.y, kk.z};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    uint32_t win[4];
                    windows(w[k], win);
#pragma unroll
                    for (int x = 0; x < 4; ++x) acc[x] = dw_dp4a<false>(win[x], rows[k], acc[x]);
                }
                put(acc);
            } else if constexpr (S == 1) {
                int acc[3][4];
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[0][x] = acc[1][x] = acc[2][x] = db;
                Row w;
                fetch(w);
                for (int base = lo; base <= r1; base += 3) {
#pragma unroll
                    for (int u = 0; u < 3; ++u) {
                        const int ir = base + u;
                        if (ir > r1) break;
                        int (&up)[4] = acc[(u + 2) % 3]; int (&at)[4] = acc[u]; int (&dn)[4] = acc[(u + 1) % 3];     // output rows ir - 1, ir, ir + 1
                        if (ir <= hi) {
                            uint32_t win[4];
                            windows(w, win);
                            if (ir < hi) fetch(w);
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                up[x] = dw_dp4a<false>(win[x], kk.z, up[x]);
                                at[x] = dw_dp4a<false>(win[x], kk.y, at[x]);
                                dn[x] = dw_dp4a<false>(win[x], kk.x, db);
                            }
                        }
                        if (ir - 1 >= r0) put(up);
                    }
                }
            } else {
                Row w, w2;
                uint32_t win[4];
                int nxt[4] = {db, db, db, db}, cur[4];
                fetch(w);
                if (r0 > 0) {
                    windows(w, win);
                    fetch(w);
#pragma unroll
                    for (int x = 0; x < 4; ++x) nxt[x] = dw_dp4a<false>(win[x], kk.x, db);
                }
                for (int r = r0; r < r1; ++r) {
                    const bool below = 2 * r + 1 < a.H;
                    if (below) fetch(w2);
                    windows(w, win);
#pragma unroll
                    for (int x = 0; x < 4; ++x) cur[x] = dw_dp4a<false>(win[x], kk.y, nxt[x]);
                    if (r + 1 < r1) fetch(w);
                    if (below) {
                        windows(w2, win);
#pragma unroll
                        for (int x = 0; x < 4; ++x) { cur[x] = dw_dp4a<false>(win[x], kk.z, cur[x]); nxt[x] = dw_dp4a<false>(win[x], kk.x, db); }
                    }
                    put(cur);
                }
            }
        }
        __syncthreads();
        // ------------------------------------------------------------ project: items of 32 pixels and one or two 16-filter tiles
        const bool last = ck + 1 == a.chunks;
        if (CLUSTER && last) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // the other CTAs have started
        auto project = [&](auto tiles_of_item) {
            constexpr int NM = decltype(tiles_of_item)::value;
            for (int it = warp; it < g2 * mp2; it += warps) {
                const int mp = it / g2, px0 = (it - mp * g2) * 32;
                const bool wide = px0 + 16 < px_out;
                int acc[2][4][4];
                const uint32_t sum = s0 + (uint32_t)(a.off_sum + it * (NM * 2048) + lane * 16);
#pragma unroll
                for (int i = 0; i < NM; ++i)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        uint4 v = make_uint4(0u, 0u, 0u, 0u);
                        if (ck > 0) v = lds_u128(sum + (uint32_t)(i * 4 + t) * 512u);
                        acc[i][t][0] = (int)v.x; acc[i][t][1] = (int)v.y; acc[i][t][2] = (int)v.z; acc[i][t][3] = (int)v.w;
                    }
                irb_band_gemm<NM>(acc, s0 + (uint32_t)(a.off_d + lane * a.dp + px0), 32u * a.dp, w2 + (uint32_t)(mp * NM * a.ks2 * 512 + lane * 16),
                                  NM * mp + 1 < a.mt2 ? (uint32_t)(a.ks2 * 512) : 0u, a.ks2, wide);
#pragma unroll
                for (int i = 0; i < NM; ++i) {
                    const int mt = NM * mp + i;
                    if (i && mt >= a.mt2) break;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int (&c)[4] = acc[i][t];
                        if (!last) { sts_u128(sum + (uint32_t)(i * 4 + t) * 512u, (uint32_t)c[0], (uint32_t)c[1], (uint32_t)c[2], (uint32_t)c[3]); continue; }
                        const int px = px0 + 8 * t;
                        if (px >= px_out) break;
                        // {row g: pixels 2q, 2q + 1; row g + 8: the same} of two neighbouring lanes -> four consecutive pixels of a row each
                        const bool odd = q & 1;
                        const int r0 = __shfl_xor_sync(0xffffffffu, odd ? c[0] : c[2], 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? c[1] : c[3], 1);
                        const int v[4] = {odd ? r0 : c[0], odd ? r1 : c[1], odd ? c[2] : r0, odd ? c[3] : r1};
                        if constexpr (CLUSTER) {
                            // to the CTA that adds this block up; blocks are dealt in turn
                            const uint32_t blk = (uint32_t)(mt * (a.dpx >> 3) + (px >> 3)), slot = div_magic(blk, a.cs_magic), owner = blk - slot * (uint32_t)cs;
                            uint32_t at;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(s0 + (uint32_t)a.off_recv + (slot * (uint32_t)cs + (uint32_t)rank) * 512u + (uint32_t)lane * 16u), "r"(owner));
                            asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
                        } else {
                            emit(v, mt * 16 + er, px + ep);
                            __syncwarp();
                        }
                    }
                }
            }
        };
        if (a.nm2 == 2) project(std::integral_constant<int, 2>{}); else project(std::integral_constant<int, 1>{});
        if (ck + 2 < a.chunks) {
            __syncthreads();                                                     // this chunk's weights have been read
            if (tid == 0 && !*abort_flag) {
                ptx::mbar_arrive_expect_tx(bar + 8u * ws, (uint32_t)a.chunk_bytes);
                ptx::bulk_g2s(s0 + (uint32_t)(a.off_w + ws * a.chunk_bytes), wsrc + (size_t)(ck + 2) * a.chunk_bytes, (uint32_t)a.chunk_bytes, bar + 8u * ws);
            }
            __syncwarp();
        }
    }
    if constexpr (CLUSTER) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int per_mt = a.dpx >> 3, blocks = a.mt2 * per_mt;
        for (int slot = warp; slot * cs + rank < blocks; slot += warps) {
            const int blk = slot * cs + rank, mt = blk / per_mt, px = (blk - mt * per_mt) * 8;
            if (px >= px_out) continue;
            int v[4] = {0, 0, 0, 0};
            const uint32_t at = s0 + (uint32_t)a.off_recv + (uint32_t)(slot * cs) * 512u + (uint32_t)lane * 16u;
#pragma unroll 4
            for (int r = 0; r < cs; ++r) {
                const uint4 w = lds_u128(at + (uint32_t)r * 512u);
                v[0] += (int)w.x; v[1] += (int)w.y; v[2] += (int)w.z; v[3] += (int)w.w;
            }
            emit(v, mt * 16 + er, px + ep);
        }
    }
    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);                         // (copies still in flight land before the CTA's memory goes away)
    }
    if (tid == 0 && *abort_flag) atomicExch(a.status, (int)DEV_ERR_WAIT_TIMEOUT);
}

// =============================================================================================
// Host side
// =============================================================================================
struct IrbBandPlan {
    IrbBandArgs a{};
    int E = 0, stride = 1, threads = 256;
    size_t smem_bytes = 0;
    double us = 0.0;               // expected time of a launch
};

// Clusters of n CTAs that an SM's share of shared memory and registers lets run at once, one to three CTAs an SM (the occupancy calculator's
// answers on a device of 148 SMs: clusters do not straddle its groups of SMs; scaled for another count).  Expected
// times are all that they decide.
inline int irb_band_resident(int per_sm, int n, int sm_count) {
    static const int clusters[3][9] = {{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 296, 148, 93, 71, 56, 45, 37, 33}, {0, 444, 222, 142, 104, 82, 71, 56, 48}};
    return std::max(1, (int)((long long)clusters[per_sm - 1][n] * sm_count / 148));
}

// One split of a block: rb output rows a band, cs CTAs a cluster, ct tiles a chunk.  False when it does not fit, or takes `limit` us at least.
inline bool irb_band_split(const ConvGeom& d, int C, int M, int rb, int cs, int ct, int threads, int sm_count, double limit, IrbBandPlan& q) {
    IrbBandArgs& a = q.a;
    a = IrbBandArgs{};
    const int S = d.sh, E = d.C, warps = threads / 32;
    q.E = E; q.stride = S; q.threads = threads;
    auto up = [](int v, int m) { return (v + m - 1) / m; };
    a.N = d.N; a.C = C; a.M = M; a.H = d.H; a.W = d.W; a.OH = d.OH; a.OW = d.OW;
    a.rb = rb; a.bands = up(a.OH, rb); a.cs = cs; a.ct = ct; a.chunks = up(up(E, 16), cs * ct);
    a.P = up(a.W, 4) * 4; a.OP = up(a.OW, 4) * 4;
    a.in_rows = std::min(S * (rb - 1) + 3, a.H);
    const int g1 = up(a.in_rows * a.P, 32), g2 = up(rb * a.OP, 32);
    auto pitch = [&](int px) { return 16 * (up(px, 16) | 1); };
    a.xp = a.ep = pitch(32 * g1); a.dp = pitch(32 * g2); a.dpx = 32 * g2;
    a.ks1 = up(C, 32); a.ks2 = up(ct, 2); a.mt2 = up(M, 16);
    // two tiles an item where that takes the warps less time (a second tile shares the columns' fragments: 1.6 times the time of one)
    auto tiles_of_item = [&](int groups, int tiles) { return up(groups * up(tiles, 2), warps) * 16 <= up(groups * tiles, warps) * 10 ? 2 : 1; };
    a.nm1 = tiles_of_item(g1, ct); a.nm2 = tiles_of_item(g2, a.mt2);
    a.chunk_bytes = ct * a.ks1 * 512 + a.mt2 * a.ks2 * 512 + ct * 16 * (int)sizeof(IrbConst) + a.mt2 * 128;
    a.w_stages = a.chunks > 1 ? 2 : 1;
    const int items2 = g2 * up(a.mt2, a.nm2), blocks = a.mt2 * (a.dpx / 8);
    a.off_x = 0;
    a.off_e = a.ks1 * 32 * a.xp;
    a.off_d = a.off_e + ct * 16 * a.ep;
    const long long off_sum = (long long)a.off_d + (long long)a.ks2 * 32 * a.dp, off_recv = off_sum + (a.chunks > 1 ? (long long)items2 * a.nm2 * 2048 : 0),
                    off_w = off_recv + (cs > 1 ? (long long)up(blocks, cs) * cs * 512 : 0), off_tail = off_w + (long long)a.w_stages * a.chunk_bytes;
    if (off_tail + 64 > 227 * 1024) return false;
    a.off_sum = (int)off_sum; a.off_recv = (int)off_recv; a.off_w = (int)off_w; a.off_tail = (int)off_tail;
    // A grid that starts while its predecessor drains piles up on the SMs that are free first: so much shared memory that no SM takes more than
    // its share (112 CTAs, several to an SM: 9.5 us instead of 6.9).
    const long long ctas = (long long)a.N * a.bands * cs, share = (ctas + sm_count - 1) / sm_count;
    q.smem_bytes = std::max<size_t>((size_t)off_tail + 64, share == 1 ? 116 * 1024 : (share == 2 ? 78 * 1024 : 0));
    // Expected time, fitted to 7843 launches (eleven kinds of blocks at 96 to 224 pixels, 1 to 128 images, splits at random):
    // 6 % rms, and the split it chooses 1.2 % slower than the best of those measured.  What a CTA alone takes counts once a round of the SMs, what it
    // issues once for every CTA that an SM runs.
    const int per_sm = std::max(1, std::min({(int)(227 * 1024 / (q.smem_bytes + 1024)), 65536 / (80 * threads), 3})), resident = irb_band_resident(per_sm, cs, sm_count);
    const long long tiles = (long long)a.N * a.bands, rounds = (tiles + resident - 1) / resident, rest = tiles - (rounds - 1) * resident;
    const double on_sm = (double)((rounds - 1) * per_sm + (rest * per_sm + resident - 1) / resident);
    const int words = C * a.in_rows * a.P / 4, it1 = g1 * up(ct, a.nm1);
    auto time = [&](int dw, int rows) {
        const double alone = 1.41 + 0.088 * up(words, 4 * threads) + a.chunks * (0.0145 * up(it1, warps) * a.nm1 * a.ks1 + 0.1445 * up(dw, threads) * rows + up(items2, warps) * a.nm2 * (0.048 * a.ks2 + 0.15)) +
                             0.54 * (a.chunks - 1) + (cs > 1 ? 0.53 : 0.0);
        const double issue = 0.242e-3 * words + a.chunks * (0.0055 * it1 * a.nm1 * a.ks1 + 0.3636e-3 * dw * rows + items2 * a.nm2 * (0.0031 * a.ks2 + 0.012)) + blocks * (cs > 1 ? 0.0099 : 0.005);
        return 0.93 + rounds * alone + on_sm * issue;
    };
    if (time(0, 0) >= limit) return false;
    // the rows of a band in as many parts as give the threads the fewest rows
    long long fewest = 1LL << 60;
    for (int s = 1; s <= rb; ++s) {
        const int rows = up(rb, s), segs = up(rb, rows);
        const long long cost = (long long)up(a.OP / 4 * ct * 16 * segs, threads) * (S * rows + 2);
        if (cost < fewest) { fewest = cost; a.segs = segs; a.seg_rows = rows; }
    }
    a.per_magic = magic_of(a.in_rows * a.P / 4); a.pw_magic = magic_of(a.P / 4); a.op_magic = magic_of(a.OP); a.opw_magic = magic_of(a.OP / 4);
    a.ch_magic = magic_of(16 * ct); a.cs_magic = magic_of(cs);
    q.us = time(a.OP / 4 * ct * 16 * a.segs, S * a.seg_rows + 2);
    return true;
}

// The block's fastest split by expected time; false when the kernel does not take it or has no chance (irb_form).
inline bool irb_band_plan(const ConvGeom& e, const ConvGeom& d, const ConvGeom& p, bool add, int sm_count, IrbBandPlan& best) {
    auto pointwise = [](const ConvGeom& g) { return g.G == 1 && g.KH == 1 && g.KW == 1 && g.sh == 1 && g.sw == 1 && !g.pt && !g.pl && !g.pb && !g.pr; };
    if (!pointwise(e) || !pointwise(p)) return false;
    if (d.G != d.C || d.M != d.C || d.KH != 3 || d.KW != 3 || d.sh != d.sw || d.sh < 1 || d.sh > 2 || d.dh != 1 || d.dw != 1 || d.pt != 1 || d.pl != 1 || d.pb != 1 || d.pr != 1) return false;
    const int C = e.C, M = p.M, S = d.sh;
    if (d.OH != (d.H - 1) / S + 1 || d.OW != (d.W - 1) / S + 1) return false;
    if (d.N <= 0 || d.H < 2 || d.W < 3 || d.H > 512 || d.W > 512 || C > 512 || M > 512 || d.C > 4096 || (add && (S != 1 || C != M)) || (double)d.N * d.C * d.H * d.W > 6.4e7) return false;
    if ((long long)d.N * C * d.H * d.W % 4 != 0 || (long long)d.N * std::max(C, M) * d.H * d.W > 0x7fffffffLL) return false;
    const int tiles = (d.C + 15) / 16;
    best.us = 1e300;
    IrbBandPlan q;
    for (int k = 1, last_rb = 0; k <= d.OH; ++k) {
        const int rb = (d.OH + k - 1) / k;
        if (rb == last_rb) continue;
        last_rb = rb;
        for (int cs = 1; cs <= 8 && cs <= tiles; ++cs) {
            const int per = (tiles + cs - 1) / cs;
            if (per * (cs - 1) >= tiles) continue;                               // (a CTA without channels)
            if ((long long)d.N * k * cs > 16LL * sm_count && (k > 1 || cs > 1)) continue;
            for (int div = 1, last_ct = 0; div <= per && div <= 12; ++div) {
                const int ct = (per + div - 1) / div;
                if (ct == last_ct) continue;
                last_ct = ct;
                for (int threads : {256, 384})
                    if (irb_band_split(d, C, M, rb, cs, ct, threads, sm_count, best.us, q) && q.us < best.us) best = q;
            }
        }
    }
    return best.us < 1e300;
}

// Weights and constants per chunk, the products' in fragment order (lane (g, q) of a 16 x 32 block: rows g, g + 8, K 4q .. and 16 + 4q ..); false
// when an accumulator could leave the range of kAccBase.  eb, db: biases with -x_zp * sum(w) folded in.
inline bool irb_band_prepare(const IrbBandPlan& q, const int8_t* we, const float* em, const int32_t* eb, const int8_t* wd, const float* dm, const int32_t* db,
                             const int8_t* wp, const float* pm, const int32_t* pb, std::vector<uint8_t>& out) {
    const IrbBandArgs& a = q.a;
    const int stages = a.cs * a.chunks, CH = a.ct * 16;
    out.assign((size_t)stages * a.chunk_bytes, 0);
    // Row r of a product: a K step is eight words, which with those of row r ^ 8 are 64 bytes of the block.  (A byte at a time the sixteen blocks of
    // a MobileNetV2-style plan took 3.3 ms of host time instead of 0.4; finalizing it for one image: 6.1 -> 3.6 ms.)
    auto row = [](uint8_t* blocks, int r, int ksteps, const int8_t* v, int n) {
        uint8_t* to = blocks + (size_t)(r >> 4) * ksteps * 512 + (r & 7) * 64 + ((r >> 3) & 1) * 4;
        for (; n > 0; n -= 32, v += 32, to += 512) {
            uint32_t w[8] = {};
            if (n >= 32) std::memcpy(w, v, 32); else std::memcpy(w, v, (size_t)n);
            for (int i = 0; i < 4; ++i) { std::memcpy(to + 16 * i, w + i, 4); std::memcpy(to + 16 * i + 8, w + 4 + i, 4); }
        }
    };
    const size_t w1_bytes = (size_t)a.ct * a.ks1 * 512, w12_bytes = w1_bytes + (size_t)a.mt2 * a.ks2 * 512;
    for (int e = 0; e < q.E; ++e) {
        uint8_t* stage = out.data() + (size_t)(e / CH) * a.chunk_bytes;
        const int8_t* w = we + (size_t)e * a.C;
        const int r = e % CH;
        IrbConst k{};
        int s1 = 0, s2 = 0;
        for (int c = 0; c < a.C; ++c) s1 += std::abs((int)w[c]);
        row(stage, r, a.ks1, w, a.C);
        for (int i = 0; i < 9; ++i) { k.k[i / 3] |= (uint32_t)(uint8_t)wd[e * 9 + i] << (8 * (i % 3)); s2 += std::abs((int)wd[e * 9 + i]); }
        if (!acc_base_ok(eb[e]) || !acc_base_ok(db[e]) || s1 * 128 + std::abs(eb[e]) >= (1 << 22) || s2 * 128 + std::abs(db[e]) >= (1 << 22)) return false;
        k.e_floor = kAccBase - (float)eb[e]; k.e_mult = em[e]; k.d_mult = dm[e]; k.d_base = kAccBaseBits + db[e];
        std::memcpy(stage + w12_bytes + (size_t)r * sizeof(IrbConst), &k, sizeof k);
    }
    for (int j = 0; j < stages; ++j) {
        uint8_t* stage = out.data() + (size_t)j * a.chunk_bytes;
        const int e0 = j * CH, live = std::min(CH, q.E - e0);
        for (int m = 0; m < a.M; ++m) {
            row(stage + w1_bytes, m, a.ks2, wp + (size_t)m * q.E + e0, live);
            uint8_t* tail = stage + a.chunk_bytes - (size_t)a.mt2 * 128 + (size_t)m * 8;
            std::memcpy(tail, pm + m, 4); std::memcpy(tail + 4, pb + m, 4);
        }
    }
    return true;
}

// Which form a block takes: this kernel, irb_q8.cuh's (`one`; null: it does not take the block) or the separate ones.  By expected times, from plans of
// eleven kinds of blocks at 96 to 224 pixels and 1 to 200 images with one kind of block at a time in another form (us this kernel / separate /
// irb_q8.cuh; the rule's mistakes cost up to 3 us):
//   separate kernels, planes that irb_q8.cuh does not take: a launch each and the expanded tensor through memory, 12 and 1.2 per million expanded values,
//     with stride 2 9 and 0.87 (24 -> 144 at 56 x 56: 1 image 6 / 10, 16 20 / 25, 24 27 / 26, 64 78 / 48, 200 223 / 135; at 40 x 40: 37 images 21 / 28, 64 35 / 33;
//     32 -> 192 at 28 x 28: 16 images 9 / 17, 148 43 / 41; 16 -> 96 at 112 x 112, stride 2: 8 images 16 / 20, 24 38 / 34, 200 289 / 181)
//   irb_q8.cuh: rounds of the SMs of a tile's time, which grows with its chunks (64 -> 384 at 14 x 14: 24 images 9 / 22 / 15, 64 17 / 26 / 17, 148 29 / 33 / 15;
//     96 -> 576 at 10 x 10: 37 images 13 / 26 / 20, 100 30 / 36 / 21; stride 2: 37 images 10 / 30 / 9; 160 -> 960 at 7 x 7: 8 images 7 / 23 / 19, 37 13 / 31 / 21, 64
//     22 / 37 / 28, 100 30 / 44 / 24; -> 320: 24 images 12 / 24 / 31, 64 31 / 32 / 25)
//   irb_q8.cuh without an addition: blocks of any widths, fitted to 1413 of them in both kernels (rms 6 %).  A launch of irb_q8.cuh takes 2.7 us more
//     than one of this kernel beside the rounds, a chunk K steps of the input and filters besides its rows; this kernel's results go out a word, two or one
//     bytes at a time, which counts where filters are many beside the expanded channels and rows are not whole words (2169 x 12 x 13 x 13, 144 -> 64 filters
//     199 / - / 112, 281 x 8 x 11 x 11, 160 -> 96 35 / - / 23).  Of 756 blocks of MobileNetV2 widths, 298 of them not among the fitted, six are slower than in
//     irb_q8.cuh by 4 to 16 % of a plan that holds little else, and all lose 0.1 % against the better kernel of each; of 1278 random ones 25 and 0.5 %
//     (by rounds of whole tiles as above: 17 and 0.3 %, 166 and 2.1 %)
enum class IrbForm { kSeparate, kOne, kBand };
inline IrbForm irb_form(const IrbPlan* one, const IrbBandPlan* band, const ConvGeom& d, bool add, bool long_add, int sm_count) {
    const bool one_pays = one && irb_pays(*one, long_add, sm_count);
    if (band) {
        const double values = 1e-6 * d.N * d.C * d.H * d.W;
        double mine = band->us, other = d.sh == 2 ? 9.0 + 0.87 * values : 12.0 + 1.2 * values;
        if (one_pays) {
            const IrbArgs& a = one->a;
            const double rounds = (a.tiles + sm_count - 1) / sm_count;
            if (add) {
                other = rounds * (a.IB > 1 ? 2.0 + a.chunks * (1.2 + 0.25 * a.H) : (long_add ? std::max(13.5, 2.0 + 5.0 * a.chunks) : 2.0 + 4.1 * a.chunks) * (0.7 + 0.3 * a.H / 14.0));
            } else {
                const IrbBandArgs& b = band->a;
                const double h = a.H / 14.0, k = (b.C + 31) / 32, m = (b.M + 63) / 64;
                const double tile = a.IB > 1 ? 1.3 + a.chunks * (3.2 * h + 0.1 * k + 0.12 * m) : (d.sh == 2 ? 1.75 + a.chunks * (0.9 * h + 0.25 * k + 0.16 * m) : 1.85 + a.chunks * (2.2 * h + 0.23 * k + 0.24 * m));
                other = 2.7 + rounds * tile;
                mine = 0.93 * mine + 1e-3 * d.N * b.M * d.OH * d.OW / sm_count * (d.OW % 4 == 0 ? 0.026 : (d.OW % 2 == 0 ? 0.1 : 0.245));
            }
        }
        if (mine < other) return IrbForm::kBand;
    }
    return one_pays ? IrbForm::kOne : IrbForm::kSeparate;
}

template <int S, bool ADD, bool CLUSTER>
inline int32_t irb_band_launch(zant_ctx* ctx, const IrbBandPlan& q, const IrbBandArgs& a, const QAddTail& add) {
    auto kernel = irb_band_kernel<S, ADD, CLUSTER>;
    ZB_SMEM_ATTR(ctx, kernel, 227 * 1024);
    launch_cluster(ctx, kernel, (unsigned)(a.N * a.bands * a.cs), (unsigned)q.threads, q.smem_bytes, CLUSTER ? (unsigned)a.cs : 1u, a, add);
    return check_launch(ctx, "irb_band_kernel");
}

// A step of a plan (weights are read before the kernel in front is complete).  x: 4-byte aligned, and so is y where OW is a multiple of four.
inline int32_t irb_band_run(zant_ctx* ctx, const IrbBandPlan& q, const void* x, const uint8_t* w, void* y, const QAddTail* add) {
    IrbBandArgs a = q.a;
    a.x = (const uint8_t*)x; a.y = (uint8_t*)y; a.w = w; a.status = ctx->status_word;
    a.give_up = ctx->give_up_cta < 0 ? -1 : ctx->give_up_cta % (a.N * a.bands * a.cs);
    ctx->give_up_cta = -1;
    auto go = [&](auto stride, auto with) -> int32_t {
        constexpr int S = decltype(stride)::value;
        constexpr bool ADD = decltype(with)::value;
        return a.cs > 1 ? irb_band_launch<S, ADD, true>(ctx, q, a, add ? *add : QAddTail{}) : irb_band_launch<S, ADD, false>(ctx, q, a, add ? *add : QAddTail{});
    };
    if (q.stride == 2) return go(std::integral_constant<int, 2>{}, std::false_type{});
    return add ? go(std::integral_constant<int, 1>{}, std::true_type{}) : go(std::integral_constant<int, 1>{}, std::false_type{});
}

}  // namespace zb
