// QuantizeLinear + QLinearConv 3x3 (at most four channels) + activation + MaxPool 2x2/2 in one launch: float NCHW -> int8 channels-last.
//
// A CTA takes a band of pooled rows of one image.  It quantises the rows that the band reads, halo included, into shared memory, planes of bytes, and
// contracts them with warp MMAs: a unit is 16 pooled pixels of a row, the rows of an MMA (row g is pixel 2g, row g + 8 pixel 2g + 1); K is the 4 x 4
// patch of a pooled pixel in every channel, byte 16 * channel + 4 * row + column, so that a lane's register `channel` is one word of patch row lane % 4.
// The four members of the pool window are four MMAs with the filter shifted inside the patch, so a thread ends up with all four of an
// output: the pool is three maxima, before the requantisation as elsewhere (it does not decrease).  Filters are permuted (column n of group j is filter
// 4 (n / 2) + 2 j + n % 2 of its 16), so that a lane's four outputs of a pixel are one word.
// The tcgen05 form reads 16-byte pixels, twelve of them zeros, which a conversion writes first: four bytes stored and four loaded for one that counts,
// and K rows of zeros.  32 x 3 x 416 x 416 -> 16 filters: 30 us of conversion and 48 of convolution there, 46 here (each kernel's own time; as steps of a plan, between
// events, 88.0 and 51.5; 88 MB are 14 us at the rate of a copy).  What
// bounds it is the chain of a unit - loads, sixteen MMAs of eight clocks each, maxima, conversions, table - at 24 warps an SM: 57 % of the issue slots, no
// pipe above 40 %.  Four CTAs of 64 registers an SM 48 us, five of 48 (spills) 59; rounding by an addition of 1.5 * 2^23 instead of the conversion
// instruction 51.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "context.cuh"
#include "geometry.hpp"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"

namespace zb {

struct FirstQ8Args {
    const float* x; uint8_t* y;
    const uint32_t* wfrag;           // [M / 16][4 members][2 groups][C][32 lanes]
    const float* mult; const int32_t* bias;      // per filter
    const uint8_t* lut;              // of the codes, or none: an activation that is not a ReLU
    int M, H, W, GH, GW;             // GH, GW: pooled rows and columns
    int PR, rows, pitch, units;      // pooled rows of a band, its input rows, words of a row, units of a pooled row
    int bands;
    long long y_img, y_row, y_pix;
    QuantFast qf; QuantSteps qs; int zp;
    int vec;                         // rows can be read as float4
    int floor;                       // of the sums: 0 for a ReLU (positive multipliers, zero point 0: the same as one behind the requantisation), else INT_MIN
};

constexpr int kFirstQ8Threads = 256;

template <bool XU8>
__device__ __forceinline__ void first_q8_mma32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const int (&c)[4]) {
    if (XU8)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
template <bool XU8>
__device__ __forceinline__ void first_q8_mma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const int (&c)[4]) {
    if (XU8)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

// Four floats quantised, packed (little endian).  MODE 0: uint8 with zero point 0 - the conversion gives 0 for a NaN, the lower bound, and the pack
// saturates; 1: clamped in front of the conversion; 2: no two-step quotient for this scale.
template <int MODE, bool XU8>
__device__ __forceinline__ uint32_t first_q8_word(const float4& v, const FirstQ8Args& a) {
    const float f[4] = {v.x, v.y, v.z, v.w};
    int k[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (MODE == 0) k[e] = __float2int_rn(quant_quotient(f[e], a.qs.rh, a.qs.rl));
        else if (MODE == 1) k[e] = __float2int_rn(fminf(fmaxf(quant_quotient(f[e], a.qs.rh, a.qs.rl), a.qf.lo), a.qf.hi)) + a.zp;
        else k[e] = quantize_fast(f[e], a.qf) + a.zp;
    }
    return XU8 ? pack_sat_u8x4(k[0], k[1], k[2], k[3]) : pack_sat_s8x4(k[0], k[1], k[2], k[3]);
}

// The band's rows, quantised: word k of a row holds columns 4 (k - 1) .. 4 (k - 1) + 3, what lies outside the image is 0.
template <int MODE, int C, bool XU8>
__device__ __forceinline__ void first_q8_rows(const FirstQ8Args& a, uint32_t* s_in, int n, int h0, int warp, int lane) {
    for (int r = warp; r < C * a.rows; r += kFirstQ8Threads / 32) {
        const int c = r / a.rows, h = h0 + (r - c * a.rows);
        uint32_t* const wr = s_in + r * a.pitch;
        if (h < 0 || h >= a.H) {
            for (int k = lane; k < a.pitch; k += 32) wr[k] = 0u;
            continue;
        }
        const float* xr = a.x + (((long long)n * C + c) * a.H + h) * a.W;
        if (a.vec) {
            const int words = a.W >> 2;
            if (lane == 0) wr[0] = 0u;
            for (int k = words + 1 + lane; k < a.pitch; k += 32) wr[k] = 0u;
            for (int k0 = lane; k0 < words; k0 += 128) {
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) if (k0 + 32 * u < words) v[u] = __ldg(reinterpret_cast<const float4*>(xr) + k0 + 32 * u);
#pragma unroll
                for (int u = 0; u < 4; ++u) if (k0 + 32 * u < words) wr[k0 + 32 * u + 1] = first_q8_word<MODE, XU8>(v[u], a);
            }
        } else {
            for (int k = lane; k < a.pitch; k += 32) {
                const int col = 4 * (k - 1);
                auto at = [&](int e) { return col >= 0 && col + e < a.W ? __ldg(xr + col + e) : 0.0f; };
                uint32_t w = first_q8_word<MODE, XU8>(make_float4(at(0), at(1), at(2), at(3)), a);
                if (col < 0 || col >= a.W) w = 0u;
                else if (col + 4 > a.W) w &= 0xffffffffu >> (8 * (col + 4 - a.W));
                wr[k] = w;
            }
        }
    }
}

template <int C, bool XU8>
__global__ void __launch_bounds__(kFirstQ8Threads, 3) first_layer_q8_kernel(const __grid_constant__ FirstQ8Args a) {
    extern __shared__ __align__(16) uint32_t first_q8_smem[];           // the activation's table, [C][rows][pitch]
    ptx::grid_start();
    uint8_t* const s_lut = reinterpret_cast<uint8_t*>(first_q8_smem);
    uint32_t* const s_in = first_q8_smem + 64;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int n = (int)blockIdx.x / a.bands, py0 = ((int)blockIdx.x - n * a.bands) * a.PR;
    if (a.lut) s_lut[threadIdx.x] = a.lut[threadIdx.x];
    if (XU8 && a.qs.rl != 0.0f && a.zp == 0) first_q8_rows<0, C, XU8>(a, s_in, n, 2 * py0 - 1, warp, lane);
    else if (a.qs.rl != 0.0f) first_q8_rows<1, C, XU8>(a, s_in, n, 2 * py0 - 1, warp, lane);
    else first_q8_rows<2, C, XU8>(a, s_in, n, 2 * py0 - 1, warp, lane);
    __syncthreads();
    // ------------------------------------------------------------------ units
    const int plane = a.rows * a.pitch, n_rows = min(a.PR, a.GH - py0), y_pix = (int)a.y_pix;
    uint8_t* const y_band = a.y + n * a.y_img + py0 * a.y_row + 4 * q;
    for (int fb = 0; fb < a.M; fb += 16) {
        uint32_t wf[4][2][C];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c) wf[m][j][c] = __ldg(a.wfrag + (((size_t)(fb / 16 * 4 + m) * 2 + j) * C + c) * 32 + lane);
        const float4 ml = __ldg(reinterpret_cast<const float4*>(a.mult + fb + 4 * q));
        const int4 bs = __ldg(reinterpret_cast<const int4*>(a.bias + fb + 4 * q));
        const int cb[2][4] = {{bs.x, bs.y, bs.x, bs.y}, {bs.z, bs.w, bs.z, bs.w}};          // the bias is what the sums start with
        const float mf[2][2] = {{ml.x, ml.y}, {ml.z, ml.w}};
        int py = 0, ux = warp;
        for (;; ux += kFirstQ8Threads / 32) {
            while (ux >= a.units) { ux -= a.units; ++py; }
            if (py >= n_rows) break;
            const uint32_t* row = s_in + (2 * py + q) * a.pitch + ux * 8 + g;
            uint32_t ev[C], od[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t w0 = row[c * plane], w1 = row[c * plane + 1], w2 = row[c * plane + 2];
                ev[c] = __byte_perm(w0, w1, 0x6543u); od[c] = __byte_perm(w1, w2, 0x4321u);      // from column 2 * pixel - 1
            }
            int r[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                int d[4][4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    if (C & 1) first_q8_mma16<XU8>(d[m], ev[C - 1], od[C - 1], wf[m][j][C - 1], cb[j]);
#pragma unroll
                    for (int c = 0; c + 1 < C; c += 2) {
                        if (c == 0 && C % 2 == 0) first_q8_mma32<XU8>(d[m], ev[c], od[c], ev[c + 1], od[c + 1], wf[m][j][c], wf[m][j][c + 1], cb[j]);
                        else first_q8_mma32<XU8>(d[m], ev[c], od[c], ev[c + 1], od[c + 1], wf[m][j][c], wf[m][j][c + 1], d[m]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) r[j][e] = rq_round(__vimax3_s32(__vimax3_s32(d[0][e], d[1][e], d[2][e]), d[3][e], a.floor), mf[j][e & 1]);
            }
            const int px = ux * 16 + 2 * g;
            uint8_t* y = y_band + py * a.y_row + px * y_pix + fb;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t pk = pack_sat_s8x4(r[0][2 * h], r[0][2 * h + 1], r[1][2 * h], r[1][2 * h + 1]);
                if (a.lut) pk = lut4_smem(s_lut, pk);
                if (px + h < a.GW) *reinterpret_cast<uint32_t*>(y + h * y_pix) = pk;
            }
        }
    }
}

// Shared memory of a band of `pr` pooled rows; a word per four columns, one in front and what the last unit reads, a pitch at which the four patch rows of
// a unit lie in different banks.
inline int first_q8_pitch(const ConvGeom& g) {
    const int units = (g.OW / 2 + 15) / 16, need = std::max(units * 8 + 2, (g.W + 3) / 4 + 1);
    return (need + 7) / 16 * 16 + 8;
}
constexpr size_t kFirstQ8Smem = 48 * 1024;                     // of a launch; the table is part of it (as static memory it was rounded up to 1024 bytes)
inline size_t first_q8_smem_bytes(const ConvGeom& g, int pr) { return 256 + (size_t)g.C * (2 * pr + 2) * first_q8_pitch(g) * 4; }

// `g`: a layer that the channels-last kernel takes with its pool (3x3, stride 1, a border of one pixel, an even image).
// Rows of at least four units, or so few rows that all CTAs are resident at once and the launch that is saved counts.  Two launches (conversion, tcgen05
// form) and one, us between events: 32 x 3 x 416 x 416, 16 filters, 88.0 and 51.5; 224 x 224, 16 / 64 filters 39.3 / 66.7 and 30.4 / 57.2; 1 x 3 x 224 x 224, 64 filters
// 23.5 and 13.5.  Narrow rows leave a warp one unit or none a band, against the filters' fragments that it loads: 500 x 3 x 64 x 64, 16 / 64 filters
// 46.4 / 91.9 and 49.7 / 84.2, 2000 x 3 x 32 x 32, 16 filters 49.2 and 79.5.  Rows that are not whole float4s are read float by float:
// 300 x 3 x 130 x 130, 16 filters 101.9 and 105.2 (128 x 128 97.9 and 73.2).
inline bool first_q8_takes(const ConvGeom& g, int sm_count) {
    if (g.OW / 2 < (g.W % 4 == 0 ? 64 : 128) && (long long)g.N * (g.OH / 2) > 3LL * sm_count) return false;
    return g.C >= 1 && g.C <= 4 && g.M % 16 == 0 && g.M <= 64 && first_q8_smem_bytes(g, 1) <= kFirstQ8Smem && (long long)g.N * (g.OH / 2) < 0x7fffffffLL;
}

// Weights [M][C][3][3] in fragment order.
inline void first_q8_weights(const ConvGeom& g, const int8_t* w, std::vector<uint32_t>& out) {
    out.assign((size_t)g.M / 16 * 8 * g.C * 32, 0u);
    size_t at = 0;
    for (int fb = 0; fb < g.M; fb += 16)
        for (int m = 0; m < 4; ++m)
            for (int j = 0; j < 2; ++j)
                for (int c = 0; c < g.C; ++c)
                    for (int lane = 0; lane < 32; ++lane, ++at) {
                        const int col = lane >> 2, kh = (lane & 3) - (m >> 1), f = fb + 4 * (col >> 1) + 2 * j + (col & 1);
                        for (int s = 0; s < 4; ++s) {
                            const int kw = s - (m & 1);
                            if (kh < 0 || kh > 2 || kw < 0 || kw > 2) continue;
                            out[at] |= (uint32_t)(uint8_t)w[(((size_t)f * g.C + c) * 3 + kh) * 3 + kw] << (8 * s);
                        }
                    }
}

// `a`: pointers, output strides, quantisation and activation filled in.
inline int32_t first_q8_run(zant_ctx* ctx, const ConvGeom& g, bool u8, FirstQ8Args a) {
    a.M = g.M; a.H = g.H; a.W = g.W; a.GH = g.OH / 2; a.GW = g.OW / 2;
    a.pitch = first_q8_pitch(g); a.units = (a.GW + 15) / 16;
    // rows of a band: as many as leave two CTAs an SM (of the three that fit).  3 x 416 x 416, 16 filters, 2 / 4 / 8 / 16 images, bands of 1, 2, 4, 8 rows, us:
    // 10.2 12.2 14.3 18.4 / 15.3 12.3 14.4 18.4 / 24.5 19.5 18.4 22.4 / 40.9 32.7 28.6 26.6
    a.PR = 8;
    while (a.PR > 1 && (first_q8_smem_bytes(g, a.PR) > kFirstQ8Smem || (long long)g.N * ((a.GH + a.PR - 1) / a.PR) < 2LL * ctx->sm_count)) a.PR /= 2;
    a.rows = 2 * a.PR + 2; a.bands = (a.GH + a.PR - 1) / a.PR;
    a.vec = g.W % 4 == 0 && ((uintptr_t)a.x & 15) == 0;
    const size_t smem = first_q8_smem_bytes(g, a.PR);
    const unsigned grid = (unsigned)(g.N * (long long)a.bands);
    auto go = [&](auto c, auto xu8) { launch(ctx, first_layer_q8_kernel<decltype(c)::value, decltype(xu8)::value>, grid, kFirstQ8Threads, smem, a); };
    auto with = [&](auto c) { if (u8) go(c, std::true_type{}); else go(c, std::false_type{}); };
    switch (g.C) {
        case 1: with(std::integral_constant<int, 1>{}); break;
        case 2: with(std::integral_constant<int, 2>{}); break;
        case 3: with(std::integral_constant<int, 3>{}); break;
        default: with(std::integral_constant<int, 4>{}); break;
    }
    return check_launch(ctx, "first_layer_q8_kernel");
}

}  // namespace zb
