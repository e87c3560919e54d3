// Convolutions between channels-last activations inside a plan: int8 (QLinearConv) and TF32 (Conv in TF32 mode) on tcgen05.
//
// The plan keeps the activations between convolutions as [N][H][W][C], because then a tiled TMA box (KC bytes of channels x
// PW x PH pixels, 32/64/128-byte swizzle) IS the K-major operand of an MMA: tap (kh, kw) is the same shared memory
// (kh * dh * PW + kw * dw) rows further on, any image size works (no row of H * W bytes has to be a multiple of anything), and
// nothing like an im2col matrix exists in memory.  (im2col + GEMM, which this replaces for such layers, wrote and re-read taps x
// the input: 29 MB for 512 x 13 x 13 at batch 32, 100 MB in fp32 at batch 8.)
//
// Fused pool: a 3x3 / stride 1 / pad 1 convolution followed by MaxPool 2x2 / 2.  MMA row = pooled pixel; the four members of its
// window are four accumulators, and member (dy, dx), tap (kh, kw) reads the view (ry, rx) = (dy + kh, dx + kw): parity plane
// (ry & 1, rx & 1) of the input shifted by (ry >> 1, rx >> 1) - four boxes per stage, one per parity, over four tensor maps whose
// strides skip every other row and column.  The maximum is taken on the accumulators, so a quarter of the values is
// requantised, none is stored unpooled and no thread needs another's data.  A view serves several members, so their filters are
// put side by side in one wider MMA (narrow ones are bound by operand fetch and issue):
//   NH_POOL_VIEWS (up to 32 filters)  one MMA of 4 NT columns per view, 16 in all, zero weights where a member has no such tap
//   NH_POOL_PAIRS (64-filter tiles)   per filter row and member row: the two middle views with both members' filters (2 NT columns),
//                                     the outer ones with one member's - 24 MMAs, no zeros
//                                     (MMAs of 2 NT and of NT columns write TMEM columns that overlap, in the order of issue; that order is
//                                     documented for equal shapes only and otherwise what every run has shown, with the sums compared bit
//                                     for bit in the channels-last tests.  One shape would need zeros, and zero times an infinite input is a NaN)
//
// Stride 2 reads the four parity planes as well, with one accumulator: tap (kh, kw) is plane ((kh - pt) & 1, (kw - pl) & 1) shifted by
// ((kh - pt) >> 1, (kw - pl) >> 1).  (A 1x1 filter with stride 2 reads one plane, as an image of its own.)
//
// At most 16 channel bytes (KC = 16: first layers, 16-channel int8 layers) would leave half of every 32-byte K step empty: there a
// pixel is one 16-byte row without swizzle, and a K step takes TWO views, whose distance in shared memory is the descriptor's
// leading-dimension offset: 8 MMAs instead of 16.
//
// Weights stay resident when one filter tile covers M and they fit; else they stream through a ring of their own, a few taps of one
// channel stage at a time.  The issuing warp runs converged with one lane's MMAs predicated on, so that descriptors are built in
// uniform registers, which the instruction wants: a single-thread loop needs ~80 clocks per MMA, more than most take to execute.
//
// Output: channels-last with any pixel pitch and channel offset (a Concat's operands are written in place), optionally every pixel
// to a 2x2 block (a nearest-neighbour Resize by two behind the convolution), or NCHW, optionally dequantised (graph outputs).
// TF32: what a later convolution reads is rounded to TF32 (nearest) when it is written; split form: hi and lo halves of C channels
// each, three MMAs per K step (A_hi W_hi + A_lo W_hi + A_hi W_lo).
//
// Roles (608 threads, one persistent CTA per SM): warp 0 activations, warp 1 TMEM owner + MMA issuer, warps 2-17 epilogue,
// warp 18 weights.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <vector>

#include "context.cuh"
#include "geometry.hpp"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"
#include "fused_cnn.cuh"
#include "tc_conv_nhwc.cuh"
#include "tc_gemm_tf32.cuh"

namespace zb {

enum NhPool { NH_POOL_NONE = 0, NH_POOL_VIEWS = 1, NH_POOL_PAIRS = 2, NH_STRIDE2 = 3 };
enum NhKind { NH_I8 = 0, NH_U8 = 1, NH_TF32 = 2, NH_TF32X3 = 3 };      // type of the activations read

struct NhConvArgs {
    int N, M, KH, KW, dh, dw, pt, pl;
    int imgs, IB;                 // images; images per tile, where whole patches of them fit one row block (N: groups of IB)
    int GH, GW;                   // rows of the product: output pixels, or pooled ones
    int BW, PW, BH, RB, PH;       // a row block is BH x BW pixels at pitch PW; RB blocks per tile; patch rows
    int hseg, wseg, n_tiles;
    int KC, c_stages;             // channel bytes per stage and operand row; stages that cover the channels
    int parts;                    // 2: hi and lo operands (split TF32)
    int lo_off;                   // channel offset (elements) of the lo half
    int NT;                       // filters per tile
    int w_resident, off_w, off_const, const_n;
    int T, w_chunk;               // tap iterations (taps, views, or pairs of them) per channel stage, bytes of one's weights
    int w_group, w_stages;        // tap iterations that are issued (and streamed) as one (divides T), ring depth of streamed weights
    int tmem_cols;
    int stages, stage_bytes, plane_bytes;     // a stage = the patch of every part (and parity plane)
    const uint8_t* w; const float* mult; const int32_t* bias; const float* fbias; const uint8_t* lut;
    uint8_t* y; long long y_img, y_row, y_pix;           // byte strides of the output (channels-last)
    int nchw;                     // 1: y is [N][M][GH][GW] codes or floats, 2: dequantised floats
    int up2;                      // channels-last: every pixel goes to a 2x2 block
    int act, six;                 // int8: zant_qact; TF32: FAct
    int wide;                     // the epilogue stores 32 channels of a pixel at a time (int8, channels-last, no pool)
    float slope, dq_scale; int dq_zp;
    int lo_out;                   // split form: channel offset of the lo half in the output
    int round_out;                // TF32: the output feeds convolutions: rounded, split form: hi and lo
    int* status;
    // operand A of iteration t: descriptor low half relative to the patch (offset, and leading-dimension offset of a pair of views);
    // NH_POOL_PAIRS: of its MMAs at [4 * t ..]
    alignas(16) uint32_t aoff[64];
};

constexpr int kNhThreads = 608;
constexpr int kNhMaxStages = 8, kNhMaxW = 12;
constexpr int kNhOrderN = 8;                             // batch whose best tiling fixes the order of float sums
constexpr int kNhTail = 48 * 8 + 256 + 64;               // barriers, TMEM slot, flag, activation table

struct NhMaps { CUtensorMap m[4]; };

// K-major swizzled operand: rows of 32, 64 or 128 bytes
__device__ __forceinline__ uint64_t nh_desc(uint32_t addr, uint32_t row_bytes) {
    uint64_t d = smem_desc_kmajor_swizzled(addr, row_bytes);
    if (row_bytes == 32) { d &= ~((uint64_t)7 << 61); d |= (uint64_t)6 << 61; }       // layout type: 32-byte swizzle
    return d;
}

// One lane's (`leader`) MMA of a converged warp.
template <int KIND>
__device__ __forceinline__ void nh_mma(uint32_t leader, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    if (KIND <= NH_U8) {
        ptx::mma_i8_if(leader, d_tmem, a_lo, a_hi, b_lo, b_hi, idesc, accumulate);
    } else {
        const uint32_t zero = 0u;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %8, 0;\n\t"
            "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, {%7, %7, %7, %7}, p;\n\t}\n"
            ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(zero), "r"(leader) : "memory");
    }
}

__host__ __device__ __forceinline__ int nh_shift(int d) { return d >= 0 ? d / 2 : -((1 - d) / 2); }

// The tiles of a CTA, grid-size apart, as a mixed-radix counter: divisions at the start only (a tile's four cost its 19 warps
// more issue slots than a first layer's epilogue has to spare).
struct NhTile { int nt, ws, hs, img, d_nt, d_ws, d_hs, d_img; };
__device__ __forceinline__ NhTile nh_first(const NhConvArgs& a) {
    NhTile c;
    int t = (int)blockIdx.x, d = (int)gridDim.x;
    c.nt = t % a.n_tiles; t /= a.n_tiles; c.ws = t % a.wseg; t /= a.wseg; c.hs = t % a.hseg; c.img = t / a.hseg;
    c.d_nt = d % a.n_tiles; d /= a.n_tiles; c.d_ws = d % a.wseg; d /= a.wseg; c.d_hs = d % a.hseg; c.d_img = d / a.hseg;
    return c;
}
__device__ __forceinline__ void nh_next(const NhConvArgs& a, NhTile& c) {
    int k;
    c.nt += c.d_nt; k = c.nt >= a.n_tiles; c.nt -= k ? a.n_tiles : 0;
    c.ws += c.d_ws + k; k = c.ws >= a.wseg; c.ws -= k ? a.wseg : 0;
    c.hs += c.d_hs + k; k = c.hs >= a.hseg; c.hs -= k ? a.hseg : 0;
    c.img += c.d_img + k;
}

// WIDE: the epilogue can store 32 channels of a pixel at a time (nh_launch_k).
template <int KIND, int POOL, bool WIDE>
__global__ void __launch_bounds__(kNhThreads, 1) tc_nhwc_net_kernel(const __grid_constant__ NhConvArgs a, const __grid_constant__ NhMaps maps) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr bool I8 = KIND <= NH_U8;
    constexpr bool POOLED = POOL == NH_POOL_VIEWS || POOL == NH_POOL_PAIRS;
    constexpr int PLANES = POOL ? 4 : 1, SETS = POOLED ? 4 : 1;    // parity planes per stage, accumulators per row block
    static_assert(!WIDE || (I8 && !POOLED), "");
    float* sMult = reinterpret_cast<float*>(smem + a.off_const);
    int* sBias = reinterpret_cast<int*>(sMult + a.const_n);         // TF32: the float bias' bits
    uint64_t* bars = reinterpret_cast<uint64_t*>(sBias + a.const_n);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 46);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint8_t* sLut = reinterpret_cast<uint8_t*>(bars + 48);
    const uint32_t bar0 = ptx::smem_u32(bars);
    const int S = a.stages;
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kNhMaxStages + s); };
    auto tfull = [&](int b) { return bar0 + 8u * (2 * kNhMaxStages + b); };
    auto tempty = [&](int b) { return bar0 + 8u * (2 * kNhMaxStages + 2 + b); };
    auto wfull = [&](int s) { return bar0 + 8u * (2 * kNhMaxStages + 4 + s); };
    auto wempty = [&](int s) { return bar0 + 8u * (2 * kNhMaxStages + 4 + kNhMaxW + s); };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = a.N * a.hseg * a.wseg * a.n_tiles;
    const uint32_t w_stage = (uint32_t)(a.w_chunk * a.w_group);
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols;
    const int NT = a.NT;

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { ptx::mbar_init(full(s), 1); ptx::mbar_init(empty(s), 1); }
        for (int s = 0; s < kNhMaxW; ++s) { ptx::mbar_init(wfull(s), 1); ptx::mbar_init(wempty(s), 1); }
        for (int b = 0; b < 2; ++b) { ptx::mbar_init(tfull(b), 1); ptx::mbar_init(tempty(b), 16); }
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    for (int i = tid; i < a.const_n; i += kNhThreads) {
        if (I8) { sMult[i] = __ldg(a.mult + i); sBias[i] = __ldg(a.bias + i); }
        else sBias[i] = __float_as_int(__ldg(a.fbias + i));
    }
    if (I8 && a.lut && tid < 256) sLut[tid] = __ldg(a.lut + tid);
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(tmem_slot), tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_trigger();
    if (warp != 18) ptx::grid_wait();                    // (weights are constants)

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t box = (uint32_t)(a.KC * a.PW * a.PH * a.IB), esz = I8 ? 1u : 4u;
            const int chans = a.KC / (int)esz;
            int s = 0; uint32_t ph = 0;
            bool alive = true;
            NhTile T = nh_first(a);
            for (int t = blockIdx.x; t < tiles && alive; t += gridDim.x, nh_next(a, T)) {
                const int w0 = T.ws * a.BW, h0 = T.hs * (a.BH * a.RB);
                for (int cs = 0; cs < a.c_stages; ++cs) {
                    if (!ptx::mbar_wait(empty(s), ph ^ 1u, abort_flag)) { alive = false; break; }
                    const uint32_t stage0 = ptx::smem_u32(smem + (size_t)s * a.stage_bytes);
                    ptx::mbar_arrive_expect_tx(full(s), box * (uint32_t)(PLANES * a.parts));
                    uint32_t dst = stage0;
                    for (int part = 0; part < a.parts; ++part) {
                        const int c0 = cs * chans + part * a.lo_off;
                        if (POOLED) {
                            // parity plane (pr, pc) of the zero-bordered image: rows 2 * i + pr - 1; the odd image rows (pr = 0) start one higher
#pragma unroll
                            for (int pp = 0; pp < 4; ++pp, dst += (uint32_t)a.plane_bytes)
                                ptx::tma_load_4d(dst, &maps.m[pp], c0, w0 - ((pp & 1) ? 0 : 1), h0 - ((pp & 2) ? 0 : 1), T.img, full(s));
                        } else if (POOL == NH_STRIDE2) {
#pragma unroll
                            for (int pp = 0; pp < 4; ++pp, dst += (uint32_t)a.plane_bytes)
                                ptx::tma_load_4d(dst, &maps.m[pp], c0, w0 + nh_shift(-a.pl), h0 + nh_shift(-a.pt), T.img * a.IB, full(s));
                        } else {
                            ptx::tma_load_4d(dst, &maps.m[0], c0, w0 - a.pl, h0 - a.pt, T.img * a.IB, full(s));
                            dst += (uint32_t)a.plane_bytes;
                        }
                    }
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 18) {
        if (lane == 0) {
            if (a.w_resident) {
                const uint32_t all = (uint32_t)(a.c_stages * a.T * a.w_chunk);
                ptx::mbar_arrive_expect_tx(wfull(0), all);
                ptx::bulk_g2s(ptx::smem_u32(smem + a.off_w), a.w, all, wfull(0));
            } else {
                int s = 0; uint32_t ph = 0;
                bool alive = true;
                const int n = a.c_stages * (a.T / a.w_group);
                for (int t = blockIdx.x; t < tiles && alive; t += gridDim.x) {
                    const uint8_t* src = a.w + (size_t)(t % a.n_tiles) * n * w_stage;
                    for (int i = 0; i < n; ++i, src += w_stage) {
                        if (!ptx::mbar_wait(wempty(s), ph ^ 1u, abort_flag)) { alive = false; break; }
                        ptx::mbar_arrive_expect_tx(wfull(s), w_stage);
                        ptx::bulk_g2s(ptx::smem_u32(smem + a.off_w) + (uint32_t)s * w_stage, src, w_stage, wfull(s));
                        if (++s == a.w_stages) { s = 0; ph ^= 1u; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // the whole warp runs the loop; `leader` issues
        const uint32_t leader = ptx::elect_one() ? 1u : 0u;
        const int NB = POOL == NH_POOL_VIEWS ? 4 * NT : (POOL == NH_POOL_PAIRS ? 2 * NT : NT);        // rows of a weight chunk
        const uint32_t idesc = I8 ? ptx::idesc_i8(128, NB, KIND == NH_I8, true) : idesc_tf32(128, NB);
        const uint32_t idesc1 = I8 ? ptx::idesc_i8(128, NT, KIND == NH_I8, true) : idesc_tf32(128, NT);
        const int ksteps = max(1, a.KC / 32);
        const uint32_t part_u = ((uint32_t)a.plane_bytes >> 4) * PLANES;
        const uint32_t blk_u = (uint32_t)(a.BH * a.PW) * ((uint32_t)a.KC >> 4), wpart_u = (uint32_t)(NB * max(a.KC, 32)) >> 4;
        const uint32_t wsingle_u = (uint32_t)(NT * a.KC) >> 4;                     // NH_POOL_PAIRS: second half of a chunk of singles
        // K-major operands: swizzled rows, or (KC = 16) rows of 16 bytes whose second K chunk the leading-dimension offset finds
        const uint64_t da = a.KC == 16 ? ptx::smem_desc_kmajor(0, 0, 128) : nh_desc(0, (uint32_t)a.KC);
        const uint64_t db = a.KC == 16 ? ptx::smem_desc_kmajor(0, (uint32_t)NB * 16, 128) : nh_desc(0, (uint32_t)a.KC);
        const uint32_t a_hi = (uint32_t)(da >> 32), b_hi = (uint32_t)(db >> 32), w0 = (uint32_t)db + (ptx::smem_u32(smem + a.off_w) >> 4);
        const uint32_t p0 = (uint32_t)da + (ptx::smem_u32(smem) >> 4), stage_u = (uint32_t)a.stage_bytes >> 4, chunk_u = (uint32_t)a.w_chunk >> 4, wstage_u = w_stage >> 4;
        auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag)) != 0; };
        // one A operand against one B block, every part
        auto mma = [&](uint32_t d, uint32_t ak, uint32_t bk, uint32_t id, uint32_t acc) {
            nh_mma<KIND>(leader, d, ak, a_hi, bk, b_hi, id, acc);
            if (KIND == NH_TF32X3) {
                nh_mma<KIND>(leader, d, ak + part_u, a_hi, bk, b_hi, id, 1u);
                nh_mma<KIND>(leader, d, ak, a_hi, bk + wpart_u, b_hi, id, 1u);
            }
        };
        uint32_t a0 = 0u, d0 = 0u, acc = 0u;
        // G tap iterations from `it0` on, weights from `bl`: unrolled, their offsets fetched together (one at a time, an iteration
        // cost ~240 clocks of latency on top of its MMAs)
        auto group = [&](auto gc, int it0, uint32_t bl) {
            constexpr int G = decltype(gc)::value;
            if constexpr (POOL == NH_POOL_PAIRS) {
                uint4 off[G];
#pragma unroll
                for (int j = 0; j < G; ++j) off[j] = *reinterpret_cast<const uint4*>(&a.aoff[4 * (it0 + j)]);
#pragma unroll
                for (int j = 0; j < G; ++j, bl += chunk_u) {
                    const bool singles = G == 1 ? it0 % 3 == 2 : j % 3 == 2;
#pragma unroll 1
                    for (int kk = 0; kk < ksteps; ++kk) {
                        const uint32_t bk = bl + 2u * kk, ab = a0 + 2u * kk;
                        if (!singles) {
                            mma(d0, ab + off[j].x, bk, idesc, acc);                          // member row 0, both columns
                            mma(d0 + 2 * NT, ab + off[j].y, bk, idesc, acc);                 // member row 1
                            acc = 1u;
                        } else {
                            mma(d0, ab + off[j].x, bk, idesc1, 1u);                          // (0,0): rx = 0
                            mma(d0 + 2 * NT, ab + off[j].y, bk, idesc1, 1u);                 // (1,0)
                            mma(d0 + NT, ab + off[j].z, bk + wsingle_u, idesc1, 1u);         // (0,1): rx = 3
                            mma(d0 + 3 * NT, ab + off[j].w, bk + wsingle_u, idesc1, 1u);     // (1,1)
                        }
                    }
                }
            } else {
                uint32_t off[G];
#pragma unroll
                for (int j = 0; j < G; ++j) off[j] = a.aoff[it0 + j];
#pragma unroll
                for (int j = 0; j < G; ++j, bl += chunk_u) {
#pragma unroll 1
                    for (int kk = 0; kk < ksteps; ++kk) {
                        const uint32_t bk = bl + 2u * kk;
                        uint32_t ak = a0 + 2u * kk + off[j];
                        mma(d0, ak, bk, idesc, acc);
                        if (a.RB > 1) mma(d0 + NB, ak + blk_u, bk, idesc, acc);
                        if (a.RB > 2) {
                            mma(d0 + 2 * NB, ak + 2 * blk_u, bk, idesc, acc);
                            if (a.RB > 3) mma(d0 + 3 * NB, ak + 3 * blk_u, bk, idesc, acc);
                        }
                        acc = 1u;
                    }
                }
            }
        };
        int s = 0, ws = 0; uint32_t ph = 0, wph = 0;
        int tile_it = 0;
        bool alive = !a.w_resident || wait(wfull(0), 0);
        for (int t = blockIdx.x; t < tiles && alive; t += gridDim.x, ++tile_it) {
            const int b = tile_it & 1;
            const uint32_t bph = (uint32_t)(tile_it >> 1) & 1u;
            if (!wait(tempty(b), bph ^ 1u)) break;
            d0 = tmem_base + (uint32_t)(b * SETS * a.RB * NT);
            acc = 0u;
            uint32_t bl = w0;
            for (int cs = 0; cs < a.c_stages && alive; ++cs) {
                if (!wait(full(s), ph)) { alive = false; break; }
                ptx::tc_fence_after();
                a0 = p0 + (uint32_t)s * stage_u;
                for (int it0 = 0; it0 < a.T; it0 += a.w_group, bl += wstage_u) {
                    if (!a.w_resident) {
                        if (!wait(wfull(ws), wph)) { alive = false; break; }
                        ptx::tc_fence_after();
                        bl = w0 + (uint32_t)ws * wstage_u;
                    }
                    if constexpr (POOL == NH_POOL_VIEWS) {
                        if (a.w_group == 16) group(std::integral_constant<int, 16>{}, it0, bl);
                        else if (a.w_group == 8) group(std::integral_constant<int, 8>{}, it0, bl);
                        else group(std::integral_constant<int, 4>{}, it0, bl);
                    } else {
                        if (a.w_group == 9) group(std::integral_constant<int, 9>{}, it0, bl);
                        else if (a.w_group == 3) group(std::integral_constant<int, 3>{}, it0, bl);
                        else group(std::integral_constant<int, 1>{}, it0, bl);
                    }
                    if (!a.w_resident) {
                        ptx::mma_commit_if(leader, wempty(ws));
                        if (++ws == a.w_stages) { ws = 0; wph ^= 1u; }
                    }
                }
                if (!alive) break;
                ptx::mma_commit_if(leader, empty(s));
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!alive) break;
            ptx::mma_commit_if(leader, tfull(b));
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue: four warps per TMEM lane quarter that take the
        // tile's chunks - 16 filters of one row block - in turn; a thread is one pixel of the row block
        const int quarter = warp & 3, part = (warp - 2) >> 2;      // (warp 18 is the weights')
        constexpr int CH = 16;
        const int row = quarter * 32 + lane;
        const int img_l = a.IB > 1 ? row / (a.PH * a.PW) : 0, row_i = row - img_l * (a.PH * a.PW);
        const int oh_l = row_i / a.PW, ow_l = row_i - oh_l * a.PW;
        const bool row_live = oh_l < a.BH && ow_l < a.BW && img_l < a.IB;
        const uint32_t hi4 = a.act == ZANT_QACT_RELU6 ? 0x01010101u * (uint32_t)(a.six & 255) : 0x7f7f7f7fu;
        // int8 without a pool: two chunks of 16 filters at a time, one store of 32 bytes a pixel, where the four warps of a quarter still have as much to do
        // each and the stores are aligned.  A lane's pixel is a line of its own, so a store takes the load-store unit 32 clocks at either width: for the
        // chunks of sixteen warps 1545 clocks with two stores and 1233 with one
        const int halves = WIDE && a.wide ? 2 : 1;
        const int per_blk = NT / CH / halves, chunks = a.RB * per_blk;
        int tile_it = 0;
        NhTile T = nh_first(a);
        const int rb0 = part / per_blk, hc0 = part - rb0 * per_blk;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++tile_it, nh_next(a, T)) {
            const int b = tile_it & 1;
            const uint32_t bph = (uint32_t)(tile_it >> 1) & 1u;
            int ok = 1;
            if (lane == 0) ok = ptx::mbar_wait(tfull(b), bph, abort_flag) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            ptx::tc_fence_after();
            const int gw = T.ws * a.BW + ow_l, h0 = T.hs * (a.BH * a.RB);
            int rb = rb0, h = hc0;
            for (int ch = part; ch < chunks; ch += 4) {
                const int g0 = h0 + rb * a.BH, gh = g0 + oh_l;
                const int img = POOLED ? T.img : T.img * a.IB + img_l;
                const bool live = row_live && gh < a.GH && gw < a.GW && (POOLED || img < a.imgs);
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((b * a.RB + rb) * SETS * NT + h * halves * CH);
                const int c0 = T.nt * NT + h * halves * CH;
                h += 4;
                while (h >= per_blk) { h -= per_blk; ++rb; }
                if (c0 < a.M && g0 < a.GH) {              // (filter padding, row blocks below the image)
                    __syncwarp();                                          // (the lanes without a pixel skip the stores below)
                    uint32_t v[SETS][CH];
                    if (!I8) {
#pragma unroll
                        for (int m = 0; m < SETS; ++m) ptx::tmem_ld16(taddr + (uint32_t)(m * NT), v[m]);
                        ptx::tmem_wait_ld();
                    }
                    uint8_t* yp = a.nchw ? a.y : a.y + (long long)img * a.y_img + (long long)gh * (a.up2 ? 2 : 1) * a.y_row + (long long)gw * (a.up2 ? 2 : 1) * a.y_pix;
                    if constexpr (I8) {
                        uint32_t wd[(WIDE ? 2 : 1) * CH / 4];
#pragma unroll
                        for (int hf = 0; hf < (WIDE ? 2 : 1); ++hf) {
                            if (hf == halves) break;
#pragma unroll
                            for (int m = 0; m < SETS; ++m) ptx::tmem_ld16(taddr + (uint32_t)(m * NT + hf * CH), v[m]);
                            ptx::tmem_wait_ld();
#pragma unroll
                            for (int j4 = 0; j4 < CH / 4; ++j4) {
                                const float4 m4 = *reinterpret_cast<const float4*>(sMult + c0 + hf * CH + j4 * 4);
                                const int4 b4 = *reinterpret_cast<const int4*>(sBias + c0 + hf * CH + j4 * 4);
                                int s[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    s[j] = (int)v[0][j4 * 4 + j];
                                    if (POOLED) s[j] = max(__vimax3_s32(s[j], (int)v[SETS > 1 ? 1 : 0][j4 * 4 + j], (int)v[SETS > 2 ? 2 : 0][j4 * 4 + j]), (int)v[SETS > 3 ? 3 : 0][j4 * 4 + j]);
                                }
                                uint32_t pk = pack_act_s8x4(rq_round(s[0] + b4.x, m4.x), rq_round(s[1] + b4.y, m4.y), rq_round(s[2] + b4.z, m4.z), rq_round(s[3] + b4.w, m4.w),
                                                            a.act != ZANT_QACT_NONE, hi4);
                                if (a.lut) pk = lut4_smem(sLut, pk);
                                wd[hf * (CH / 4) + j4] = pk;
                            }
                        }
                        if (!live) continue;
                        if (a.nchw) {
                            const size_t plane = (size_t)a.GH * a.GW, at = ((size_t)img * a.M + c0) * plane + (size_t)gh * a.GW + gw;
#pragma unroll
                            for (int j = 0; j < CH; ++j) {
                                if (c0 + j >= a.M) break;
                                const int q = (int)(int8_t)(wd[j >> 2] >> (8 * (j & 3)));
                                if (a.nchw == 2) reinterpret_cast<float*>(a.y)[at + j * plane] = __fmul_rn(__int2float_rn(q - a.dq_zp), a.dq_scale);
                                else a.y[at + j * plane] = (uint8_t)q;
                            }
                        } else {
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (u && !a.up2) break;
                                uint8_t* yc = yp + (u >> 1) * a.y_row + (u & 1) * a.y_pix + c0;
                                if constexpr (WIDE) if (halves == 2) { ptx::st_global_v8(yc, wd); continue; }
                                *reinterpret_cast<uint4*>(yc) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
                            }
                        }
                    } else {
                        float r[CH];
#pragma unroll
                        for (int j = 0; j < CH; ++j) {
                            const float bs = __int_as_float(sBias[c0 + j]);
                            float best = -INFINITY;                        // (the comparison chain of lean_onnx_maxpool: NaNs are skipped)
#pragma unroll
                            for (int m = 0; m < SETS; ++m) {
                                float q = __fadd_rn(__uint_as_float(v[m][j]), bs);
                                if (a.act == FACT_RELU) q = q > 0.0f ? q : 0.0f;
                                else if (a.act == FACT_LEAKY) q = q <= 0.0f ? __fmul_rn(a.slope, q) : q;
                                best = !POOLED ? q : (q > best ? q : best);
                            }
                            r[j] = best;
                        }
                        if (!live) continue;
                        if (a.nchw) {
                            const size_t plane = (size_t)a.GH * a.GW, at = ((size_t)img * a.M + c0) * plane + (size_t)gh * a.GW + gw;
#pragma unroll
                            for (int j = 0; j < CH; ++j) {
                                if (c0 + j >= a.M) break;
                                reinterpret_cast<float*>(a.y)[at + j * plane] = r[j];
                            }
                        } else {
                            float lo[CH];
                            if (a.round_out) {
#pragma unroll
                                for (int j = 0; j < CH; ++j) {
                                    const float hi = round_tf32(r[j]);
                                    lo[j] = round_tf32(__fadd_rn(r[j], -hi));
                                    r[j] = hi;
                                }
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (u && !a.up2) break;
                                uint8_t* yc = yp + (u >> 1) * a.y_row + (u & 1) * a.y_pix + (long long)c0 * 4;
#pragma unroll
                                for (int j = 0; j < CH; j += 8) {
                                    ptx::st_global_v8(yc + j * 4, r + j);
                                    if (KIND == NH_TF32X3 && a.round_out) ptx::st_global_v8(yc + (long long)a.lo_out * 4 + j * 4, lo + j);
                                }
                            }
                        }
                    }
                }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(tempty(b));
        }
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
struct NhConvPlan {
    NhConvArgs a{};
    int kind = NH_I8, NT = 0;
    int pool = 0;                 // NhPool
    bool half = false;            // 1x1, stride 2: every second row and column of the input is the image
    int cin = 0, w_cin = 0;       // channels a pixel of the input holds, channels of the weights (fewer: zero weights behind them)
    size_t smem_bytes = 0, w_bytes = 0;
};

// Taps of pair `it` (KC = 16) without a pool; the second one lies behind the first in shared memory.  -1: none (zero weights).
__host__ __device__ inline int nh_pair(int it, int which, int taps) {
    const int t = 2 * it + which;
    return t < taps ? t : -1;
}
// NH_POOL_VIEWS: view of pair `it`: two rows apart, i.e. in the same parity plane.
__host__ __device__ inline int nh_view_pair(int it, int which) { return (it >> 2) * 4 + (it & 3) + which * 8; }

// Stride 2: row (or column) d of the image relative to 2 * i lies in parity plane d & 1, row i + nh_shift(d).
// Operand offsets, in 16-byte units.
inline void nh_offsets(NhConvArgs& a, int mode) {
    const int unit = a.KC / 16, taps = a.KH * a.KW;
    auto tap_at = [&](int tap) { return (uint32_t)((tap / a.KW * a.dh * a.PW + tap % a.KW * a.dw) * unit); };
    auto view_at = [&](int ry, int rx) { return (uint32_t)(((ry & 1) * 2 + (rx & 1)) * (a.plane_bytes / 16) + ((ry >> 1) * a.PW + (rx >> 1)) * unit); };
    for (int it = 0; it < a.T; ++it) {
        if (mode == NH_POOL_PAIRS) {
            const int kh = it / 3, j = it % 3;                // j: views rx = 1, rx = 2, the outer ones
            for (int dy = 0; dy < 2; ++dy) {
                a.aoff[4 * it + dy] = view_at(dy + kh, j == 0 ? 1 : (j == 1 ? 2 : 0));
                a.aoff[4 * it + 2 + dy] = view_at(dy + kh, 3);
            }
        } else if (a.KC == 16) {
            uint32_t o0, o1;
            if (mode == NH_POOL_VIEWS) { const int v0 = nh_view_pair(it, 0), v1 = nh_view_pair(it, 1); o0 = view_at(v0 / 4, v0 % 4); o1 = view_at(v1 / 4, v1 % 4); }
            else { const int t1 = nh_pair(it, 1, taps); o0 = tap_at(nh_pair(it, 0, taps)); o1 = t1 >= 0 ? tap_at(t1) : o0; }
            a.aoff[it] = o0 | ((o1 - o0) << 16);
        } else if (mode == NH_STRIDE2) {
            const int dh = it / a.KW - a.pt, dw = it % a.KW - a.pl;
            a.aoff[it] = (uint32_t)(((dh & 1) * 2 + (dw & 1)) * (a.plane_bytes / 16) + ((nh_shift(dh) - nh_shift(-a.pt)) * a.PW + nh_shift(dw) - nh_shift(-a.pl)) * unit);
        } else a.aoff[it] = mode == NH_POOL_VIEWS ? view_at(it / 4, it % 4) : tap_at(it);
    }
}

// Clocks of a candidate tiling: the waves of tiles over the SMs times the slowest of a tile's parts.
inline double nh_cost(const NhConvArgs& a, int kind, int mode, long long tiles, int sm_count, int planes, bool resident, long long w_all) {
    const int NT = a.NT, per = kind == NH_TF32X3 ? 3 : 1, ksteps = std::max(1, a.KC / 32);
    const int NB = NT * (mode == NH_POOL_VIEWS ? 4 : (mode == NH_POOL_PAIRS ? 2 : 1));
    // an MMA of 128 x n x 32 bytes: n / 2 of math, or its operands out of shared memory, or the issue of the next one
    auto clocks = [](int n) { return std::max(std::max(n / 2.0, 32.0 + n / 4.0), 46.0); };
    const double iters = (double)a.c_stages * a.T;
    const double mma = iters * ksteps * per * a.RB * (mode == NH_POOL_PAIRS ? (4 * clocks(NB) + 4 * clocks(NT)) / 3.0 : clocks(NB));
    const double issue = iters * (40.0 + 20.0 * ksteps) + iters / a.w_group * 150.0 + a.c_stages * 150.0;
    const double bytes = (double)a.c_stages * planes * a.parts * a.PH * a.PW * a.IB * a.KC + (resident ? 0.0 : (double)w_all);
    const double epi = (double)a.RB * NT / 64.0 * (mode == NH_POOL_VIEWS || mode == NH_POOL_PAIRS ? 700.0 : 450.0);
    const double tile = std::max(std::max(mma + issue, bytes / 40.0), epi) + 300.0;
    return std::ceil((double)tiles / sm_count) * tile + epi;
}

// `g`: the convolution on NCHW shapes.  False when the kernel does not take it.  `same`: only tilings that add an output's products up in
// the order of that one (channel stages, and the way the views of a pool are taken).
inline bool nh_conv_search(const ConvGeom& g, int kind, bool pool, int sm_count, NhConvPlan& p, const NhConvPlan* same) {
    const bool i8 = kind <= NH_U8;
    const int esz = i8 ? 1 : 4, parts = kind == NH_TF32X3 ? 2 : 1;
    const bool s2 = g.sh == 2 && (g.KH > 1 || g.KW > 1), planed = pool || s2;
    if (g.sh == 2 && !s2 && (g.pt || g.pl)) return false;
    if (g.G != 1 || g.sh != g.sw || (g.sh != 1 && g.sh != 2) || (g.sh == 2 && (pool || !i8 || g.dh != 1 || g.dw != 1 || g.H < 2 || g.W < 2)) || g.N <= 0 || g.OH <= 0 || g.OW <= 0 || g.M > 4096) return false;
    if (pool && (g.KH != 3 || g.KW != 3 || g.dh != 1 || g.dw != 1 || g.pt != 1 || g.pl != 1 || g.pb != 1 || g.pr != 1 || g.H % 2 || g.W % 2)) return false;
    const int halo_w = pool ? 1 : (s2 ? nh_shift(g.KW - 1 - g.pl) - nh_shift(-g.pl) : (g.KW - 1) * g.dw), halo_h = pool ? 1 : (s2 ? nh_shift(g.KH - 1 - g.pt) - nh_shift(-g.pt) : (g.KH - 1) * g.dh);
    if (halo_w > 32 || halo_h > 32 || (s2 ? g.pt >= g.KH || g.pl >= g.KW : g.pt > halo_h + 1 || g.pl > halo_w + 1)) return false;
    NhConvArgs base{};
    base.N = g.N; base.M = g.M; base.KH = g.KH; base.KW = g.KW; base.dh = g.dh; base.dw = g.dw; base.pt = g.pt; base.pl = g.pl;
    base.GH = pool ? g.OH / 2 : g.OH; base.GW = pool ? g.OW / 2 : g.OW;
    base.wseg = (base.GW + 127 - halo_w) / (128 - halo_w);
    base.BW = (base.GW + base.wseg - 1) / base.wseg;
    base.PW = base.BW + halo_w;
    base.BH = std::max(1, std::min(base.GH, 128 / base.PW));
    // images whose whole patch is at most half a row block share one (7 x 7 outputs with stride 2: two, of 64 rows each)
    base.imgs = g.N; base.IB = 1;
    if (!pool && base.wseg == 1 && base.BH == base.GH) base.IB = std::max(1, std::min(i8 ? g.N : std::min(g.N, kNhOrderN), 128 / ((base.GH + halo_h) * base.PW)));
    base.N = (g.N + base.IB - 1) / base.IB;
    base.parts = parts;
    const int cin = parts > 1 ? (g.C + 7) / 8 * 8 : g.C;             // (a stage of the hi half must not run into the lo half)
    base.lo_off = cin;
    const int cbytes = cin * esz, planes = planed ? 4 : 1, sets = pool ? 4 : 1, taps = g.KH * g.KW;
    p.kind = kind; p.cin = cin; p.w_cin = g.C; p.half = g.sh == 2 && !s2;
    if (taps > 64) return false;
    double best = 1e300;
    for (int NT = pool ? 16 : 32; NT <= (pool ? 64 : 256); NT *= 2)
        for (int KC = 16; KC <= 128; KC *= 2)
            for (int rb = 1; rb <= 4; ++rb) {
                const int mode = s2 ? NH_STRIDE2 : !pool ? NH_POOL_NONE : (NT <= 32 ? NH_POOL_VIEWS : NH_POOL_PAIRS);
                const int NB = NT * (mode == NH_POOL_VIEWS ? 4 : (mode == NH_POOL_PAIRS ? 2 : 1));
                if (2 * sets * rb * NT > 512 || (NT > 32 && NT / 2 >= g.M) || (mode == NH_POOL_PAIRS && KC == 16)) continue;
                if (KC > (s2 ? 32 : 16) && KC / 2 >= cbytes) continue;               // (channels past C arrive as zeros)
                if (KC == 16 && (cbytes > 16 || parts > 1 || s2)) continue;
                if (same && (KC != same->a.KC || mode != same->pool)) continue;
                NhConvArgs a = base;
                a.n_tiles = (g.M + NT - 1) / NT;
                a.KC = KC; a.c_stages = (cbytes + KC - 1) / KC;
                a.T = mode == NH_POOL_VIEWS ? (KC == 16 ? 8 : 16) : (KC == 16 ? (taps + 1) / 2 : taps);
                a.w_chunk = NB * std::max(KC, 32) * parts;
                a.RB = rb; a.PH = rb * a.BH + halo_h;
                if (a.PH > 256 || (rb > 1 && (rb - 1) * a.BH >= a.GH)) continue;
                if (parts > 1 && cin % (KC / 4) != 0) continue;
                a.hseg = (a.GH + rb * a.BH - 1) / (rb * a.BH);
                const int rows = std::max(a.PH * a.PW * a.IB, (rb - 1) * a.BH * a.PW + 128 + halo_h * a.PW + halo_w);
                a.plane_bytes = (rows * KC + 1023) / 1024 * 1024;
                a.const_n = (a.n_tiles * NT + 15) / 16 * 16;
                const int tail = a.const_n * 8 + kNhTail;
                a.stage_bytes = planes * parts * a.plane_bytes;
                const long long w_all = (long long)a.w_chunk * a.T * a.c_stages;
                const long long tiles = (long long)a.N * a.hseg * a.wseg * a.n_tiles;
                if (tiles > 0x7fffffffLL) continue;
                a.NT = NT;
                for (int resident = 1; resident >= 0; --resident) {
                    if (resident && (a.n_tiles != 1 || w_all > 100 * 1024)) continue;
                    for (int G : {16, 9, 8, 4, 3, 1}) {
                        const bool views = mode == NH_POOL_VIEWS;
                        if (a.T % G || (views ? (G != 16 && G != 8 && G != 4) : (G != 9 && G != 3 && G != 1)) || (resident && G != a.T && G != 1 && !(views && G == 4 && a.T < 8))) continue;
                        a.w_group = G;
                        const int w_stage = a.w_chunk * G;
                        long long room = 232448 - 1024 - tail;
                        // streamed weights: as many stages as fit beside the patches
                        a.w_stages = resident ? 0 : (int)std::min<long long>(kNhMaxW, std::max<long long>(0, (room - 2LL * a.stage_bytes) / w_stage));
                        if (!resident && a.w_stages < 2) continue;
                        room -= resident ? w_all : (long long)a.w_stages * w_stage;
                        const int stages = (int)std::min<long long>(kNhMaxStages, room / a.stage_bytes);
                        if (stages < 2) continue;
                        const double cost = nh_cost(a, kind, mode, tiles, sm_count, planes, resident != 0, w_all);
                        if (cost >= best) continue;
                        best = cost;
                        for (a.tmem_cols = 32; a.tmem_cols < 2 * sets * rb * NT; a.tmem_cols *= 2) {}
                        a.w_resident = resident; a.stages = stages;
                        a.off_w = stages * a.stage_bytes;
                        a.off_const = (a.off_w + (resident ? (int)w_all : a.w_stages * w_stage) + 127) / 128 * 128;
                        nh_offsets(a, mode);
                        p.pool = mode;
                        p.a = a; p.NT = NT;
                        p.smem_bytes = (size_t)a.off_const + tail;
                        p.w_bytes = (size_t)a.n_tiles * w_all;
                    }
                }
            }
    return best < 1e300;
}

// Float sums depend on their order: the one that suits 8 images is kept for every batch, so that an image's result does not depend on how
// many others it is run with (a sharded batch equals the whole one).  int8 sums are exact and take the best tiling of each batch.
inline bool nh_conv_plan(const ConvGeom& g, int kind, bool pool, int sm_count, NhConvPlan& p) {
    if (kind <= NH_U8) return nh_conv_search(g, kind, pool, sm_count, p, nullptr);
    ConvGeom few = g;
    few.N = kNhOrderN;
    NhConvPlan order;
    return nh_conv_search(few, kind, pool, sm_count, order, nullptr) && nh_conv_search(g, kind, pool, sm_count, p, &order);
}

// Weights [M][C][KH][KW] -> [filter tile][channel stage][iteration][part][NB rows of KC bytes], rows swizzled as the tensor core reads
// them (16-byte chunk c of row j at c ^ (j % 8), c ^ (j / 2 % 4), c ^ (j / 4 % 2) for rows of 128, 64, 32 bytes); KC = 16: [filter
// tile][pair][2][NB rows of 16 bytes].  Rows of an iteration: the tile's filters (no pool), those of the four members for the
// iteration's view (NH_POOL_VIEWS), those of two members for a middle view, or of one member for each outer view (NH_POOL_PAIRS).
// Done on the device when a plan is finalized, a thread per 16-byte chunk (the byte shuffle of a 1024 x 512 x 3 x 3 tensor took the
// host 30 ms).  T: int8_t, or float (rounded to TF32, part 1 the remainder).
struct NhWeightArgs { const void* w; uint8_t* out; int M, C, taps, NT, NB, KC, T, c_stages, parts, pool; long long chunks; };
template <typename T>
__device__ __forceinline__ void nh_weight_chunks(const NhWeightArgs& a, long long first, long long step) {
    constexpr int PER = 16 / (int)sizeof(T);
    const int per_row = a.KC / 16;
    for (long long i = first; i < a.chunks; i += step) {
        long long t = i;
        int slot = (int)(t % per_row); t /= per_row;
        const int row = (int)(t % a.NB); t /= a.NB;
        int half = 0, part = 0;
        if (a.KC == 16) { half = (int)(t & 1); t >>= 1; } else { part = (int)(t % a.parts); t /= a.parts; }
        const int it = (int)(t % a.T); t /= a.T;
        const int cs = (int)(t % a.c_stages), nt = (int)(t / a.c_stages);
        slot ^= a.KC == 128 ? (row & 7) : (a.KC == 64 ? (row >> 1) & 3 : (a.KC == 32 ? (row >> 2) & 1 : 0));      // the chunk that is stored here
        const int blk = row / a.NT, m = nt * a.NT + row - blk * a.NT, c0 = (cs * per_row + slot) * PER;
        int tap = -1;
        if (a.pool == NH_POOL_VIEWS) {
            const int view = a.KC == 16 ? nh_view_pair(it, half) : it, kh = view / 4 - (blk >> 1), kw = view % 4 - (blk & 1);
            if (kh >= 0 && kh < 3 && kw >= 0 && kw < 3) tap = kh * 3 + kw;
        } else if (a.pool == NH_POOL_PAIRS) {
            const int kh = it / 3, j = it - 3 * kh;            // rx = 1: kw = 1, 0; rx = 2: kw = 2, 1; rx = 0: kw = 0 and rx = 3: kw = 2
            tap = kh * 3 + (j == 2 ? 2 * blk : j + 1 - blk);
        } else {
            tap = a.KC == 16 ? nh_pair(it, half, a.taps) : it;
        }
        union { T v[PER]; uint4 q; } u;
        u.q = make_uint4(0u, 0u, 0u, 0u);
        if (m < a.M && tap >= 0) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (c0 + k >= a.C) break;
                const T v = __ldg((const T*)a.w + ((size_t)m * a.C + c0 + k) * a.taps + tap);
                if constexpr (sizeof(T) == 4) { const float hi = round_tf32(v); u.v[k] = part == 0 ? hi : round_tf32(__fadd_rn(v, -hi)); }
                else u.v[k] = v;
            }
        }
        reinterpret_cast<uint4*>(a.out)[i] = u.q;
    }
}
template <typename T>
__global__ void __launch_bounds__(256) nh_weights_k(const __grid_constant__ NhWeightArgs a) {
    ptx::grid_start();
    nh_weight_chunks<T>(a, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}
inline NhWeightArgs nh_weight_args(const NhConvPlan& p, const void* w, void* out) {
    NhWeightArgs a{};
    a.w = w; a.out = (uint8_t*)out; a.M = p.a.M; a.C = p.w_cin; a.taps = p.a.KH * p.a.KW; a.NT = p.a.NT; a.KC = p.a.KC; a.T = p.a.T; a.c_stages = p.a.c_stages;
    a.NB = p.a.NT * (p.pool == NH_POOL_VIEWS ? 4 : (p.pool == NH_POOL_PAIRS ? 2 : 1));
    a.parts = p.a.parts; a.pool = p.pool; a.chunks = (long long)p.w_bytes / 16;
    return a;
}
inline int32_t run_nh_weights(zant_ctx* ctx, const NhConvPlan& p, const void* w, void* out) {
    const NhWeightArgs a = nh_weight_args(p, w, out);
    const int grid = grid_for((size_t)a.chunks, 256, ctx->sm_count);
    if (p.kind <= NH_U8) launch(ctx, nh_weights_k<int8_t>, grid, 256, 0, a);
    else launch(ctx, nh_weights_k<float>, grid, 256, 0, a);
    return check_launch(ctx, "nh_weights_k");
}

// A single call's plan: the search visits some hundred tilings (1 to 2 us of the 30 a small call takes), so a thread keeps the plans of
// the last 16 shapes it used.  (60 different shapes in a cycle: 32 us a call, as with 8.)
inline bool nh_conv_plan_kept(const ConvGeom& g, int kind, int sm_count, NhConvPlan& p) {
    struct Entry { ConvGeom g; int kind = -1, sm = 0; bool ok = false; NhConvPlan p; };
    constexpr int kEntries = 16;
    static thread_local std::vector<Entry> kept;
    static thread_local int next = 0;
    static_assert(std::is_trivially_copyable<ConvGeom>::value && sizeof(ConvGeom) % sizeof(int) == 0, "compared as bytes");
    for (const Entry& e : kept) if (e.kind == kind && e.sm == sm_count && std::memcmp(&e.g, &g, sizeof(g)) == 0) { p = e.p; return e.ok; }
    Entry e;
    e.g = g; e.kind = kind; e.sm = sm_count;
    e.ok = nh_conv_plan(g, kind, false, sm_count, e.p);
    p = e.p;
    const bool ok = e.ok;
    if ((int)kept.size() < kEntries) kept.push_back(e);
    else { kept[next] = e; next = (next + 1) % kEntries; }
    return ok;
}

// A channels-last buffer: `ptr` = channel 0 of pixel (0, 0), pixels `pix` bytes apart; lo: split form, channel offset of the lo half.
struct NhView { void* ptr; long long pix; int H, W; int lo; };

inline int32_t nh_encode_map(int N, int box_n, const NhView& x, int chan_elems, int esz, int KC, int box_w, int box_h, bool parity, int pr, int pc, CUtensorMap* map) {
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static std::atomic<EncodeFn> encode{nullptr};
    if (!encode.load()) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) { cudaGetLastError(); return fail(ZANT_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver"); }
        encode.store(reinterpret_cast<EncodeFn>(fn));
    }
    const cuuint64_t row = (cuuint64_t)x.pix * x.W, img = row * x.H;
    cuuint64_t dims[4] = {(cuuint64_t)chan_elems, (cuuint64_t)x.W, (cuuint64_t)x.H, (cuuint64_t)N}, strides[3] = {(cuuint64_t)x.pix, row, img};
    char* base = (char*)x.ptr;
    if (parity) {
        // plane (pr, pc) of the zero-bordered image: pr = 0 are the odd image rows, pr = 1 the even ones, columns likewise
        base += (pr ? 0 : (long long)row) + (pc ? 0 : x.pix);
        dims[1] = (x.W + pc) / 2; dims[2] = (x.H + pr) / 2; strides[0] = 2 * (cuuint64_t)x.pix; strides[1] = 2 * row;
    }
    const cuuint32_t box[4] = {(cuuint32_t)(KC / esz), (cuuint32_t)box_w, (cuuint32_t)box_h, (cuuint32_t)box_n}, estr[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle sw = KC == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (KC == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : (KC == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE));
    const CUresult r = encode.load()(map, esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ZANT_E_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return ZANT_OK;
}

template <int KIND, int POOL, bool WIDE = false>
inline int32_t nh_launch_t(zant_ctx* ctx, const NhConvPlan& p, const NhConvArgs& a, const NhMaps& maps) {
    ZB_SMEM_ATTR(ctx, (tc_nhwc_net_kernel<KIND, POOL, WIDE>), 232448);
    const long long tiles = (long long)a.N * a.hseg * a.wseg * a.n_tiles;
    launch_const(ctx, tc_nhwc_net_kernel<KIND, POOL, WIDE>, (unsigned)std::min<long long>(tiles, ctx->sm_count), kNhThreads, p.smem_bytes, a, maps);
    return check_launch(ctx, "tc_nhwc_net_kernel");
}
// int8 without a pool: the kernel that can store 32 channels at a time takes 96 registers a thread, the other 78, beside which the CTAs of a next kernel
// of another kind start early (28 x 32 x 5 x 5 -> 192 filters, depthwise, 64 filters 25.0 us, 31.8 when all took the larger one; 43 x 160 x 6 x 6 -> 960,
// depthwise with stride 2, 160 39.4 and 45.7; with 80 registers for both 384 -> 256 filters on 32 x 26 x 26 went from 31.2 to 32.4).  So the larger
// one runs where it does store 32 channels, and for dequantised values of layers like the ones whose results it stores (256 -> 255 18.1 -> 17.6); not
// wherever it could: a chain that alternates between the two loads either's instructions each time, 2 us.
template <int KIND>
inline int32_t nh_launch_k(zant_ctx* ctx, const NhConvPlan& p, const NhConvArgs& a, const NhMaps& maps) {
    if (p.pool == NH_POOL_VIEWS) return nh_launch_t<KIND, NH_POOL_VIEWS>(ctx, p, a, maps);
    if (p.pool == NH_POOL_PAIRS) return nh_launch_t<KIND, NH_POOL_PAIRS>(ctx, p, a, maps);
    if constexpr (KIND <= NH_U8) {
        if (p.pool == NH_STRIDE2) return a.wide ? nh_launch_t<KIND, NH_STRIDE2, true>(ctx, p, a, maps) : nh_launch_t<KIND, NH_STRIDE2>(ctx, p, a, maps);
        if (a.wide || (a.nchw == 2 && p.cin % 32 == 0 && a.RB * a.NT % 128 == 0)) return nh_launch_t<KIND, NH_POOL_NONE, true>(ctx, p, a, maps);
    }
    return nh_launch_t<KIND, NH_POOL_NONE>(ctx, p, a, maps);
}

// `a`: p.a with the device pointers, the output and the epilogue filled in.
inline int32_t nh_conv_run(zant_ctx* ctx, const NhConvPlan& p, NhConvArgs a, const NhView& x) {
    const int esz = p.kind <= NH_U8 ? 1 : 4;
    a.status = ctx->status_word;
    a.lo_off = x.lo;
    NhMaps maps;
    for (int pp = 0; pp < (p.pool ? 4 : 1); ++pp) {
        // (the pooled form numbers the planes of the bordered image, whose odd rows are the image's even ones)
        const int pr = p.pool == NH_STRIDE2 || p.half ? 1 - (pp >> 1) : pp >> 1, pc = p.pool == NH_STRIDE2 || p.half ? 1 - (pp & 1) : pp & 1;
        ZB_TRY(nh_encode_map(a.imgs, a.IB, x, a.parts > 1 ? x.lo + p.cin : p.cin, esz, a.KC, a.PW, a.PH, p.pool != 0 || p.half, pr, pc, &maps.m[pp]));
    }
    a.wide = !a.nchw && a.M % 32 == 0 && a.NT % 32 == 0 && a.RB * a.NT % 128 == 0 && ((uintptr_t)a.y & 31) == 0 && a.y_pix % 32 == 0 && a.y_row % 32 == 0 && a.y_img % 32 == 0 ? 1 : 0;
    switch (p.kind) {
        case NH_I8: return nh_launch_k<NH_I8>(ctx, p, a, maps);
        case NH_U8: return nh_launch_k<NH_U8>(ctx, p, a, maps);
        case NH_TF32: return nh_launch_k<NH_TF32>(ctx, p, a, maps);
        default: return nh_launch_k<NH_TF32X3>(ctx, p, a, maps);
    }
}

// ---------------------------------------------------------------------------------------------
// The operators between those convolutions, channels-last.
// ---------------------------------------------------------------------------------------------
// First layers: an NCHW tensor of at most four channels -> pixels of 16 bytes.  MODE 0: float, quantised (QuantizeLinear);
// 1: 8-bit codes as they are; 2: float, rounded to TF32 (pixels of 4 floats); 3: hi and lo halves of 8 floats each.
// A CTA takes 1024 pixels, a lane every 32nd of its warp's 128: loads and 16-byte pixel stores are contiguous over the warp
// whatever the plane's alignment.  (Four neighbouring pixels a thread stored 16 bytes of every 64: 32 images of 3 x 416 x 416 took 43 us,
// 155 MB.)  PACKED, planes of at most 512 pixels: as many whole images as 1024 pixels hold, a pixel's image is a division (one image a
// CTA: 4096 of 3 x 8 x 8 14.7 us, packed 7.2); larger planes: 1024 pixels of one image.
struct ToNhwcArgs { const void* x; uint8_t* y; int C, N, imgs; long long HW, blocks_per_image; QuantFast qf; QuantSteps qs; int zp; };
template <int MODE, bool PACKED>
__global__ void __launch_bounds__(256) to_nhwc_small_k(const __grid_constant__ ToNhwcArgs a) {
    ptx::grid_start();
    const int t = (int)(threadIdx.x >> 5) * 128 + (int)(threadIdx.x & 31);
    long long px0, off[4];                   // the first pixel, in the whole run; element of channel 0
    bool on[4];
    if (PACKED) {
        const int hw = (int)a.HW, n0 = (int)blockIdx.x * a.imgs, here = min(a.imgs, a.N - n0) * hw;
        px0 = (long long)n0 * hw + t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = t + 32 * j, dn = (int)((unsigned)r / (unsigned)hw);
            off[j] = (long long)n0 * a.C * hw + dn * a.C * hw + (r - dn * hw); on[j] = r < here;
        }
    } else {
        const long long n = (long long)blockIdx.x / a.blocks_per_image, p0 = ((long long)blockIdx.x - n * a.blocks_per_image) * 1024 + t;
        px0 = n * a.HW + p0;
#pragma unroll
        for (int j = 0; j < 4; ++j) { off[j] = n * a.C * a.HW + p0 + 32 * j; on[j] = p0 + 32 * j < a.HW; }
    }
    float f[4][4] = {};
    uint32_t q[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (c >= a.C) break;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!on[j]) continue;
            const long long at = off[j] + c * a.HW;
            if (MODE == 1) q[j] |= (uint32_t)__ldg((const uint8_t*)a.x + at) << (8 * c);
            else f[j][c] = __ldg((const float*)a.x + at);
        }
    }
    if (MODE == 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c >= a.C) break;
            if (a.qs.rl != 0.0f) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    q[j] |= (uint32_t)((__float2int_rn(fminf(fmaxf(quant_quotient(f[j][c], a.qs.rh, a.qs.rl), a.qf.lo), a.qf.hi)) + a.zp) & 255) << (8 * c);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] |= (uint32_t)((quantize_fast(f[j][c], a.qf) + a.zp) & 255) << (8 * c);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (!on[j]) break;
        const long long px = px0 + 32 * j;
        if (MODE <= 1) {
            *reinterpret_cast<uint4*>(a.y + px * 16) = make_uint4(q[j], 0u, 0u, 0u);
        } else {
            float4* d = reinterpret_cast<float4*>(a.y + px * (MODE == 3 ? 64 : 16));
            float hi[4], lo[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) { hi[c] = round_tf32(f[j][c]); lo[c] = round_tf32(__fadd_rn(f[j][c], -hi[c])); }
            d[0] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            if (MODE == 3) { d[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f); d[2] = make_float4(lo[0], lo[1], lo[2], lo[3]); d[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
        }
    }
}
// `steps`: the quantisation's quotient without a division, where the caller has it (quant_steps).
inline int32_t run_to_nhwc(zant_ctx* ctx, int mode, const void* x, void* y, int N, int C, long long HW, float scale, int zp, bool u8, const QuantSteps& steps = QuantSteps{0.0f, 0.0f}) {
    ToNhwcArgs a{};
    const bool packed = HW <= 512;
    const long long imgs = packed && HW > 0 ? 1024 / HW : 1, per = (HW + 1023) / 1024, grid = (N + imgs - 1) / imgs * per;
    if (grid > 0x7fffffffLL) return fail(ZANT_E_TOO_LARGE, "too many pixels for the channels-last conversion");
    if (grid == 0) return ZANT_OK;
    a.x = x; a.y = (uint8_t*)y; a.C = C; a.N = N; a.imgs = (int)imgs; a.HW = HW; a.blocks_per_image = per; a.zp = zp; a.qs = steps;
    if (mode == 0) a.qf = quant_fast(scale, (float)((u8 ? 0 : -128) - zp), (float)((u8 ? 255 : 127) - zp));
    auto go = [&](auto m) {
        if (packed) launch(ctx, to_nhwc_small_k<decltype(m)::value, true>, (unsigned)grid, 256, 0, a);
        else launch(ctx, to_nhwc_small_k<decltype(m)::value, false>, (unsigned)grid, 256, 0, a);
    };
    switch (mode) {
        case 0: go(std::integral_constant<int, 0>{}); break;
        case 1: go(std::integral_constant<int, 1>{}); break;
        case 2: go(std::integral_constant<int, 2>{}); break;
        default: go(std::integral_constant<int, 3>{}); break;
    }
    return check_launch(ctx, "to_nhwc_small_k");
}

// What a single call prepares on the device, one launch, blocks by kind: the input channels-last, the weights in their blocks, the bias.
//   input  8-bit NCHW -> pixels of `pix` bytes (channels rounded up to 16, zeros behind the last): a block takes 64 channels x 128 pixels of one image
//          through shared memory; rows of a channel plane start at any byte, so a word is cut out of two aligned ones.  A thread then has four pixels of
//          16 channels as sixteen words, transposes them by byte permutes (instead of 64 byte loads from shared memory) and four lanes write 64
//          contiguous bytes of a pixel.  Words of a row are stored at w ^ 8 (channel / 16), so that the four lanes' channels lie in different banks.
//   bias   bias - x_zp * (sum of the filter's weights), zeros behind the last filter: a warp per entry
// The kinds do not depend on each other: as launches one after the other, latency chains both, 7.4 + 14.4 us for 256 x 256 x 14 x 14 and 512 filters of
// 3 x 3 and 6.4 + 6.1 for 33 x 45 x 27 x 27 and 85, together 15.1 and 6.9; the calls 95.8 -> 93.6 (the weights' upload is most of it) and 38.2 -> 32.6.
struct NhPrepArgs {
    const uint8_t* x; uint8_t* y; int C, HW, pix; long long bytes;
    int px_tiles, ch_tiles;
    unsigned x_blocks, w_blocks;
    NhWeightArgs w;
    const int8_t* bw; const int32_t* bias; int32_t* bias_out; int M, K, bias_n, x_zp;      // bias_n 0: the bias is ready
};
constexpr int kNhPrepThreads = 128;
__global__ void __launch_bounds__(kNhPrepThreads) nh_prep_k(const __grid_constant__ NhPrepArgs a) {
    ptx::grid_start();
    __shared__ uint32_t tile[64 * 32];
    unsigned b = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (b < a.x_blocks) {
        const int per = a.px_tiles * a.ch_tiles;
        const long long n = b / per;
        const int r = (int)(b - n * per), c0 = r / a.px_tiles * 64, p0 = (r - r / a.px_tiles * a.px_tiles) * 128;
        for (int i0 = 0; i0 < 16; i0 += 8) {
            uint32_t lo[8], hi[8], sh[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int c = c0 + warp + 4 * (i0 + i), p = p0 + 4 * lane;
                lo[i] = hi[i] = sh[i] = 0u;
                if (c < a.C && p < a.HW) {
                    const long long at = (n * a.C + c) * (long long)a.HW + p, al = at & ~3LL;
                    if (al + 8 <= a.bytes) {
                        const uint32_t* s = reinterpret_cast<const uint32_t*>(a.x + al);
                        sh[i] = (uint32_t)(at & 3) * 8u;
                        lo[i] = __ldg(s);
                        if (sh[i]) hi[i] = __ldg(s + 1);
                    } else {
                        for (int k = 0; k < 4; ++k) if (at + k < a.bytes) lo[i] |= (uint32_t)__ldg(a.x + at + k) << (8 * k);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int c = warp + 4 * (i0 + i);
                tile[c * 32 + (lane ^ (8 * (c >> 4)))] = __funnelshift_r(lo[i], hi[i], sh[i]);
            }
        }
        __syncthreads();
        const int j = lane & 3, word = warp * 8 + (lane >> 2), p = p0 + 4 * word, c = c0 + 16 * j;
        if (p >= a.HW || c >= a.pix) return;
        uint32_t o[4][4];                                                        // [pixel][four channels]
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t* t = tile + (16 * j + 4 * q) * 32 + (word ^ (8 * j));
            const uint32_t v0 = t[0], v1 = t[32], v2 = t[64], v3 = t[96];
            const uint32_t a0 = __byte_perm(v0, v1, 0x5140), a1 = __byte_perm(v2, v3, 0x5140), a2 = __byte_perm(v0, v1, 0x7362), a3 = __byte_perm(v2, v3, 0x7362);
            o[0][q] = __byte_perm(a0, a1, 0x5410); o[1][q] = __byte_perm(a0, a1, 0x7632);
            o[2][q] = __byte_perm(a2, a3, 0x5410); o[3][q] = __byte_perm(a2, a3, 0x7632);
        }
        uint8_t* y = a.y + (n * a.HW + p) * (long long)a.pix + c;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (p + k < a.HW) *reinterpret_cast<uint4*>(y + (long long)k * a.pix) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
        return;
    }
    b -= a.x_blocks;
    if (b < a.w_blocks) { nh_weight_chunks<int8_t>(a.w, (long long)b * kNhPrepThreads + tid, (long long)a.w_blocks * kNhPrepThreads); return; }
    b -= a.w_blocks;
    const int m = (int)b * (kNhPrepThreads / 32) + warp;
    if (m >= a.bias_n) return;
    int s = 0;
    if (m < a.M && a.x_zp != 0) for (int k = lane; k < a.K; k += 32) s += __ldg(a.bw + (size_t)m * a.K + k);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) a.bias_out[m] = m < a.M ? (a.bias ? __ldg(a.bias + m) : 0) - a.x_zp * s : 0;
}
inline NhPrepArgs nh_prep_input(const void* x, void* y, int N, int C, int HW, int pix) {
    NhPrepArgs a{};
    a.x = (const uint8_t*)x; a.y = (uint8_t*)y; a.C = C; a.HW = HW; a.pix = pix; a.bytes = (long long)N * C * HW;
    a.px_tiles = (HW + 127) / 128; a.ch_tiles = (pix + 63) / 64;
    a.x_blocks = (unsigned)((long long)N * a.px_tiles * a.ch_tiles);
    return a;
}
inline void nh_prep_weights(zant_ctx* ctx, NhPrepArgs& a, const NhConvPlan& p, const void* w, void* out) {
    a.w = nh_weight_args(p, w, out);
    a.w_blocks = (unsigned)grid_for((size_t)a.w.chunks, kNhPrepThreads, ctx->sm_count, 16);
}
inline int32_t run_nh_prep(zant_ctx* ctx, const NhPrepArgs& a) {
    const unsigned blocks = a.x_blocks + a.w_blocks + (unsigned)((a.bias_n + kNhPrepThreads / 32 - 1) / (kNhPrepThreads / 32));
    if (blocks == 0) return ZANT_OK;
    launch(ctx, nh_prep_k, blocks, kNhPrepThreads, 0, a);
    return check_launch(ctx, "nh_prep_k");
}

// A channels-last tensor in the graph's order, for a caller that asked for its address; split form: hi + lo.
struct FromNhwcArgs { const uint8_t* x; uint8_t* y; long long pix, hw, total; int C, lo; };
template <typename T>
__global__ void __launch_bounds__(256) from_nhwc_k(const __grid_constant__ FromNhwcArgs a) {
    ptx::grid_start();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.total; i += (long long)gridDim.x * blockDim.x) {
        const long long t = i / a.hw, p = i - t * a.hw, n = t / a.C, c = t - n * a.C;
        const T* s = reinterpret_cast<const T*>(a.x + (n * a.hw + p) * a.pix) + c;
        T v = *s;
        if constexpr (sizeof(T) == 4) { if (a.lo) v = __fadd_rn(v, s[a.lo]); }
        reinterpret_cast<T*>(a.y)[i] = v;
    }
}
inline int32_t run_from_nhwc(zant_ctx* ctx, const NhView& x, void* y, size_t N, size_t C, size_t esz) {
    FromNhwcArgs a{};
    a.x = (const uint8_t*)x.ptr; a.y = (uint8_t*)y; a.pix = x.pix; a.hw = (long long)x.H * x.W; a.C = (int)C; a.lo = x.lo;
    a.total = (long long)(N * C) * a.hw;
    const int grid = grid_for((size_t)a.total, 256, ctx->sm_count);
    if (esz == 1) launch(ctx, from_nhwc_k<uint8_t>, grid, 256, 0, a);
    else launch(ctx, from_nhwc_k<float>, grid, 256, 0, a);
    return check_launch(ctx, "from_nhwc_k");
}

// MaxPool: a thread owns 16 bytes of one output pixel's channels.  KIND as above; split form: the larger hi + lo.
struct NhPoolArgs { const uint8_t* x; uint8_t* y; long long x_pix, y_pix, total; int chunks, H, W, OH, OW, KH, KW, sh, sw, dh, dw, pt, pl; int lo_in, lo_out; };
template <int KIND>
__global__ void __launch_bounds__(256) nh_maxpool_k(const __grid_constant__ NhPoolArgs a) {
    ptx::grid_start();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.total; i += (long long)gridDim.x * blockDim.x) {
        const int ch = (int)(i % a.chunks); long long t = i / a.chunks;
        const long long px = t;
        const int ow = (int)(t % a.OW); t /= a.OW;
        const int oh = (int)(t % a.OH); const long long n = t / a.OH;
        const uint8_t* x = a.x + n * a.H * a.W * a.x_pix + ch * 16;
        const uint32_t m = KIND == NH_U8 ? 0u : 0x80808080u;
        uint32_t q[4] = {m, m, m, m};
        float best[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, lo[4] = {0.0f, 0.0f, 0.0f, 0.0f}, sum[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        for (int kh = 0; kh < a.KH; ++kh) {
            const int ih = oh * a.sh - a.pt + kh * a.dh;
            if (ih < 0 || ih >= a.H) continue;
            for (int kw = 0; kw < a.KW; ++kw) {
                const int iw = ow * a.sw - a.pl + kw * a.dw;
                if (iw < 0 || iw >= a.W) continue;
                const uint8_t* s = x + ((long long)ih * a.W + iw) * a.x_pix;
                const uint4 v = *reinterpret_cast<const uint4*>(s);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                if (KIND == NH_I8 || KIND == NH_U8) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[j] = KIND == NH_I8 ? __vmaxs4(q[j], w[j]) : __vmaxu4(q[j], w[j]);
                } else if (KIND == NH_TF32) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { const float f = __uint_as_float(w[j]); best[j] = f > best[j] ? f : best[j]; }
                } else {
                    const float4 l4 = *reinterpret_cast<const float4*>(s + (long long)a.lo_in * 4);
                    const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float f = __fadd_rn(__uint_as_float(w[j]), l[j]);
                        if (f > sum[j]) { sum[j] = f; best[j] = __uint_as_float(w[j]); lo[j] = l[j]; }
                    }
                }
            }
        }
        uint8_t* y = a.y + px * a.y_pix + ch * 16;
        if (KIND <= NH_U8) *reinterpret_cast<uint4*>(y) = make_uint4(q[0], q[1], q[2], q[3]);
        else {
            *reinterpret_cast<float4*>(y) = make_float4(best[0], best[1], best[2], best[3]);
            if (KIND == NH_TF32X3) *reinterpret_cast<float4*>(y + (long long)a.lo_out * 4) = make_float4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
}
inline int32_t run_nh_maxpool(zant_ctx* ctx, int kind, const PoolGeom& g, int N, int C, const NhView& x, const NhView& y) {
    NhPoolArgs a{};
    a.x = (const uint8_t*)x.ptr; a.y = (uint8_t*)y.ptr; a.x_pix = x.pix; a.y_pix = y.pix; a.H = g.H; a.W = g.W; a.OH = g.OH; a.OW = g.OW;
    a.KH = g.KH; a.KW = g.KW; a.sh = g.sh; a.sw = g.sw; a.dh = g.dh; a.dw = g.dw; a.pt = g.pt; a.pl = g.pl; a.lo_in = x.lo; a.lo_out = y.lo;
    a.chunks = C * (kind <= NH_U8 ? 1 : 4) / 16;
    a.total = (long long)N * g.OH * g.OW * a.chunks;
    const int grid = grid_for((size_t)a.total, 256, ctx->sm_count);
    switch (kind) {
        case NH_I8: launch(ctx, nh_maxpool_k<NH_I8>, grid, 256, 0, a); break;
        case NH_U8: launch(ctx, nh_maxpool_k<NH_U8>, grid, 256, 0, a); break;
        case NH_TF32: launch(ctx, nh_maxpool_k<NH_TF32>, grid, 256, 0, a); break;
        default: launch(ctx, nh_maxpool_k<NH_TF32X3>, grid, 256, 0, a); break;
    }
    return check_launch(ctx, "nh_maxpool_k");
}

}  // namespace zb
