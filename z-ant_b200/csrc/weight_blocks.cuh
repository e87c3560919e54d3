// Weights of a single QLinearConv / QLinearMatMul call, from the tensor's own order into the blocked form a tensor-core
// kernel reads, on the device.
//
// A call brings its weights along every time, so re-blocking them is part of the call: on the host the byte shuffle of a
// 512 x 256 x 3 x 3 tensor took 1.1 of 1.5 ms (the convolution itself takes 0.05), here the raw tensor is uploaded as it is
// and one launch of a few microseconds shuffles it.  One block per (padded) filter row; a thread moves 16-byte chunks of K
// and the block adds the row up for the bias (bias - x_zp * sum).  A plan blocks its weights once, when it is finalized: those of the
// channels-last and few-position kernels on the device, the others on the host.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "context.cuh"
#include "tc_conv_generic.cuh"
#include "tc_conv_nchw.cuh"
#include "tc_conv_nhwc.cuh"
#include "tc_pw_nchw.cuh"

namespace zb {

struct WBlockArgs {
    const int8_t* w; uint4* dst; const int32_t* bias; int32_t* bias_out;
    size_t sm, sc, st;          // element strides of filter, channel, tap in w
    int M, C, taps, x_zp;
    int rows;                   // padded rows of dst
    int q_total, NT;            // 16-byte chunks per row; rows per tile: chunk q of row r is dst[((r / NT) * q_total + q) * NT + r % NT]
    int order;                  // 0: K = (channel, tap); 1: K = (tap, channel); 2: (channel stage of CB chunks, tap, chunk); 3: as 2, one swizzled row of CB chunks per (stage, tap)
    int CB;
    int G, m_pad, group_q;      // block-diagonal form (tc_pw_nchw.cuh): row g * m_pad + m holds filter m in the chunks of group g
};

__global__ void __launch_bounds__(128) weight_blocks_kernel(const WBlockArgs a) {
    __shared__ int part[4];
    const int r = blockIdx.x, grp = a.G > 1 ? r / a.m_pad : 0, m = a.G > 1 ? r - grp * a.m_pad : r;
    const int K = a.C * a.taps;
    int sum = 0;
    for (int q = threadIdx.x; q < a.q_total; q += blockDim.x) {
        uint32_t v[4] = {0u, 0u, 0u, 0u};
        const int qq = a.G > 1 ? q - grp * a.group_q : q;       // chunk of the filter's own K
        if (m < a.M && qq >= 0 && (a.G == 1 || qq < a.group_q)) {
            const int8_t* row = a.w + (size_t)m * a.sm;
            int tap = 0, c = 0;
            if (a.order == 1) { const int per = a.C / 16; tap = qq / per; c = (qq - tap * per) * 16; }
            else if (a.order >= 2) { const int t = qq / a.CB, cs = t / a.taps; tap = t - cs * a.taps; c = (cs * a.CB + (qq - t * a.CB)) * 16; }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                int8_t b = 0;
                if (a.order == 0) {
                    const int k = qq * 16 + i;
                    if (k < K) { const int ch = a.taps == 1 ? k : k / a.taps; b = __ldg(row + (size_t)ch * a.sc + (size_t)(k - ch * a.taps) * a.st); }
                } else if (tap < a.taps && c + i < a.C) {
                    b = __ldg(row + (size_t)(c + i) * a.sc + (size_t)tap * a.st);
                }
                sum += b;
                v[i >> 2] |= (uint32_t)(uint8_t)b << (8 * (i & 3));
            }
        }
        size_t at;
        const int rt = r / a.NT, j = r - rt * a.NT;
        if (a.order == 3) {
            const int x = a.CB == 8 ? (j & 7) : ((j >> 1) & 3), t = q / a.CB, blk = q - t * a.CB;
            at = (((size_t)rt * (a.q_total / a.CB) + t) * a.NT + j) * a.CB + (blk ^ x);
        } else {
            at = ((size_t)rt * a.q_total + q) * a.NT + j;
        }
        a.dst[at] = make_uint4(v[0], v[1], v[2], v[3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0 && grp == 0) {
        const int s = part[0] + part[1] + part[2] + part[3];
        if (a.G == 1 || m < a.M) a.bias_out[m] = m < a.M ? (a.bias ? __ldg(a.bias + m) : 0) - a.x_zp * s : 0;
    }
}

inline WBlockArgs weight_blocks_conv(int M, int C, int taps, int x_zp) {
    WBlockArgs a{};
    a.M = M; a.C = C; a.taps = taps; a.x_zp = x_zp; a.G = 1; a.CB = 1;
    a.sm = (size_t)C * taps; a.sc = (size_t)taps; a.st = 1;
    return a;
}
// im2col + GEMM (QGemmPrep with its sizes set)
inline WBlockArgs weight_blocks_of(const QGemmPrep& p, int M, int C, int taps, int x_zp) {
    WBlockArgs a = weight_blocks_conv(M, C, taps, x_zp);
    a.rows = p.N_pad; a.q_total = p.K16; a.NT = p.NT; a.order = p.tap_major ? 1 : 0;
    return a;
}
// implicit GEMM from NCHW, or channels-last
inline WBlockArgs weight_blocks_of(const TcConvPlan& p, int x_zp, bool nhwc) {
    const TcConvArgs& c = p.a;
    WBlockArgs a = weight_blocks_conv(c.M, c.C, c.KH * c.KW, x_zp);
    a.rows = c.m_pad; a.q_total = c.c_stages * a.taps * c.CB; a.NT = p.NT; a.order = nhwc ? 3 : 2; a.CB = c.CB;
    return a;
}
// filters on the lanes; a stem's K is (channel, tap), which the weight tensor holds contiguously
inline WBlockArgs weight_blocks_of(const PwConvPlan& p, int x_zp) {
    WBlockArgs a = weight_blocks_conv(p.a.M, p.a.C, 1, x_zp);
    a.rows = p.m_tiles * 128; a.q_total = p.a.a_steps * 2; a.NT = 128; a.order = 0;
    a.G = p.a.G; a.m_pad = p.a.m_pad; a.group_q = a.q_total / a.G;
    return a;
}
// bytes of the blocked weights, entries of the folded bias
inline size_t weight_blocks_bytes(const WBlockArgs& a) { return (size_t)a.rows * a.q_total * 16; }
inline size_t weight_blocks_bias(const WBlockArgs& a) { return (size_t)(a.G > 1 ? a.M : a.rows); }

inline int32_t run_weight_blocks(zant_ctx* ctx, WBlockArgs a, const int8_t* w, const int32_t* bias, int8_t* dst, int32_t* bias_out) {
    a.w = w; a.bias = bias; a.dst = reinterpret_cast<uint4*>(dst); a.bias_out = bias_out;
    weight_blocks_kernel<<<a.rows, 128, 0, ctx->stream>>>(a);
    // (not an operator launch: zant_b200_ctx_launch_count counts those)
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ZANT_OK : fail(ZANT_E_CUDA, "launch of weight_blocks_kernel failed: %s", cudaGetErrorString(e));
}

// |accumulator * multiplier| <= this over the M filters, for tc_conv_run / tc_conv_nhwc_run (tc_conv_max_product without the folded
// bias, which only the device knows): |x - x_zp| <= 255 for every activation and |x_zp| <= 255 for the folded zero point.  `mult` may
// be padded behind the filters; `bias_host` is the caller's array of M values.
inline double weight_blocks_max_product(const std::vector<float>& mult, const int32_t* bias_host, bool bias_known, int M, long long K) {
    double worst = 0.0;
    for (int m = 0; m < M; ++m) {
        if (!std::isfinite(mult[m])) return INFINITY;
        const double b = bias_host ? std::fabs((double)bias_host[m]) : (bias_known ? 0.0 : 2147483648.0);
        worst = std::max(worst, (2.0 * 255.0 * 128.0 * (double)K + b) * std::fabs((double)mult[m]));
    }
    return worst;
}

}  // namespace zb
