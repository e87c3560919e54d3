// QLinearConv (group 1) and QLinearMatMul with FEW output positions on warp-level MMAs: the deep layers of a network run on
// one image, the classifier of a small batch.
//
// With fewer than 256 output positions a 128-row tcgen05 tile is mostly padding and a launch has a handful of tiles; what
// such a layer needs is its weights once (tens to hundreds of KB, out of L2 or HBM) spread over as many SMs as possible, i.e.
// it is bound by load latency.  So: filters are the MMA rows (mma.sync.m16n8k32, weights stored in fragment order: one
// coalesced 16-byte load per lane and 16 x 32 block, no shared memory), 32 output positions the columns, a CTA owns 16 or 32
// filters x 32 positions and its warps SPLIT THE K RANGE between them, so that a 960-deep sum is eight chains of four steps
// whose loads are all in flight at once; the partial sums (exact int32) meet in shared memory, and the requantisation runs once.
// Column c of MMA j is position 4 * c + j: a lane then needs the SAME four channels of FOUR neighbouring positions - four
// word loads of an NCHW plane and a 4x4 byte transpose give its B registers of all four MMAs.
//
// Three ways to load the activations (PATH):
//   0  one position per image (matrix product, 1x1 planes): K is contiguous, 16-byte loads
//   1  1x1 filter, stride 1, planes of whole words: word loads
//   2  anything else: byte loads, taps outside the image hold the input zero point
// Measured against the one-thread-per-output kernels (MobileNetV2-style network, one image): 1x1 384 -> 64 on 14 x 14 planes
// 160 us, 960 -> 160 on 7 x 7 384 us, the 1280 -> 1000 classifier 66 us (139 us for 37 rows) there.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "context.cuh"
#include "geometry.hpp"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"

namespace zb {

struct SmallGemmArgs {
    const uint8_t* x; const uint4* w; void* y;
    const float* mult; const int32_t* bias;      // bias has -x_zp * sum(w) folded in; null: zeros
    ConvGeom g;
    int P, OHW;            // output positions in all, per image
    int c_steps;           // K steps of 32 channels per tap
    int k_steps;           // K steps in all (padded to a multiple of two on PATH 0)
    int vec;               // PATH 0: rows are whole 16-byte units; PATH 1, 2: output planes are whole words
    uint32_t pad;          // input zero point as a byte
    Requant rq;
    QAddTail add;          // res != nullptr: a QLinearAdd behind it (int8)
};

constexpr int kSmallWarps = 8;

template <bool XU8>
__device__ __forceinline__ void mma_s8_16832(int (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    if (XU8)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// bytes k of four words (one per channel) -> word k (one per position)
__device__ __forceinline__ void transpose4x4(const uint32_t (&v)[4], uint32_t (&o)[4]) {
    const uint32_t t0 = __byte_perm(v[0], v[1], 0x5140), t1 = __byte_perm(v[2], v[3], 0x5140);
    const uint32_t t2 = __byte_perm(v[0], v[1], 0x7362), t3 = __byte_perm(v[2], v[3], 0x7362);
    o[0] = __byte_perm(t0, t1, 0x5410); o[1] = __byte_perm(t0, t1, 0x7632);
    o[2] = __byte_perm(t2, t3, 0x5410); o[3] = __byte_perm(t2, t3, 0x7632);
}

template <bool XU8, bool YU8, int PATH, int MT>
__global__ void __launch_bounds__(kSmallWarps * 32) small_gemm_q8_kernel(const SmallGemmArgs a) {
    constexpr int LD = 36;                                     // row pitch of the partial sums: 16-byte rows, banks spread
    extern __shared__ int red[];                               // [warps][MT * 16][LD]
    ptx::grid_start();
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = lane >> 2, tq = lane & 3;
    const int m0 = blockIdx.x * (MT * 16), p0 = blockIdx.y * 32;
    const ConvGeom& g = a.g;
    const int HW = g.H * g.W;

    // this lane's four positions p0 + 4 * gq + j
    const int pl = p0 + 4 * gq;
    long long base[4]; int ih0[4], iw0[4];
    if (PATH == 1) {
        const int n = pl / HW, pix = pl - n * HW;              // four positions of one image (HW % 4 == 0)
        base[0] = (long long)n * g.C * HW + pix;
    } else if (PATH == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = min(pl + j, a.P - 1);
            const int n = p / a.OHW, pos = p - n * a.OHW, oh = pos / g.OW, ow = pos - oh * g.OW;
            ih0[j] = oh * g.sh - g.pt; iw0[j] = ow * g.sw - g.pl;
            base[j] = (long long)n * g.C * HW + (long long)ih0[j] * g.W + iw0[j];
        }
    }

    int acc[MT][4][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0;

    const uint4* wl = a.w + (size_t)blockIdx.x * MT * a.k_steps * 32 + lane;
    if (PATH == 0) {
        // two K steps per block of 64: a lane's 16 bytes are its B registers of both steps
        for (int kb = warp; kb < a.k_steps / 2; kb += warps) {
            uint4 wv[MT][2];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                wv[i][0] = __ldg(wl + ((size_t)i * a.k_steps + 2 * kb) * 32);
                wv[i][1] = __ldg(wl + ((size_t)i * a.k_steps + 2 * kb + 1) * 32);
            }
            const int k = kb * 64 + tq * 16;
            uint4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                b[j] = make_uint4(0u, 0u, 0u, 0u);
                const int p = pl + j;
                if (p < a.P && k < g.C) {
                    const uint8_t* src = a.x + (size_t)p * g.C + k;
                    if (a.vec) b[j] = __ldg(reinterpret_cast<const uint4*>(src));
                    else {
                        uint32_t t[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                        for (int q = 0; q < 16; ++q)
                            if (k + q < g.C) t[q >> 2] |= (uint32_t)__ldg(src + q) << (8 * (q & 3));
                        b[j] = make_uint4(t[0], t[1], t[2], t[3]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mma_s8_16832<XU8>(acc[i][j], wv[i][0], b[j].x, b[j].y);
                    mma_s8_16832<XU8>(acc[i][j], wv[i][1], b[j].z, b[j].w);
                }
        }
    } else {
#pragma unroll 2
        for (int s = warp; s < a.k_steps; s += warps) {
            uint4 wv[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) wv[i] = __ldg(wl + ((size_t)i * a.k_steps + s) * 32);
            uint32_t b[2][4];                                  // [K half][position]
            if (PATH == 1) {
                const bool ok = pl < a.P;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int c = s * 32 + h * 16 + tq * 4 + i;
                        v[i] = (ok && c < g.C) ? __ldg(reinterpret_cast<const uint32_t*>(a.x + base[0] + (long long)c * HW)) : 0u;
                    }
                    transpose4x4(v, b[h]);
                }
            } else {
                const int tap = s / a.c_steps, c0 = (s - tap * a.c_steps) * 32;
                const int kh = tap / g.KW, kw = tap - kh * g.KW;
                const int dy = kh * g.dh, dx = kw * g.dw;
                const long long toff = (long long)dy * g.W + dx;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool in = (unsigned)(ih0[j] + dy) < (unsigned)g.H && (unsigned)(iw0[j] + dx) < (unsigned)g.W;
                    const uint8_t* src = a.x + base[j] + toff;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t w4 = 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int c = c0 + h * 16 + tq * 4 + i;
                            const uint32_t v = (in && c < g.C) ? (uint32_t)__ldg(src + (long long)c * HW) : a.pad;
                            w4 |= v << (8 * i);
                        }
                        b[h][j] = w4;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_s8_16832<XU8>(acc[i][j], wv[i], b[0][j], b[1][j]);
        }
    }

    // partial sums of this warp: row = filter, column = position
    int* mine = red + warp * (MT * 16 * LD);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q)                            // accumulator q: row gq (+ 8 for q >= 2), MMA column 2 * tq + (q & 1)
            *reinterpret_cast<int4*>(mine + (i * 16 + gq + (q >> 1) * 8) * LD + (2 * tq + (q & 1)) * 4) =
                make_int4(acc[i][0][q], acc[i][1][q], acc[i][2][q], acc[i][3][q]);
    __syncthreads();
    for (int u = threadIdx.x; u < MT * 16 * 8; u += blockDim.x) {
        if (PATH == 0) {
            // four filters of one position: contiguous in the output
            const int col = u / (MT * 4), r0 = (u - col * (MT * 4)) * 4;
            const int p = p0 + col;
            if (p >= a.P) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = m0 + r0 + j;
                if (m >= g.M) break;
                int s = a.bias ? __ldg(a.bias + m) : 0;
                for (int w = 0; w < warps; ++w) s += red[w * (MT * 16 * LD) + (r0 + j) * LD + col];
                int q = requant_one<YU8>(s, __ldg(a.mult + m), a.rq);
                if (!YU8 && a.add.res) q = (int)(int8_t)qadd_word<false>((uint32_t)__ldg(a.add.res + (size_t)p * g.M + m), (uint32_t)(q & 255), a.add);
                store_q<YU8>(a.y, (size_t)p * g.M + m, q);
            }
        } else {
            // four positions of one filter
            const int row = u >> 3, c4 = (u & 7) * 4, m = m0 + row, p = p0 + c4;
            if (m >= g.M || p >= a.P) continue;
            const int bs = a.bias ? __ldg(a.bias + m) : 0;
            const float mu = __ldg(a.mult + m);
            int s[4] = {bs, bs, bs, bs};
            for (int w = 0; w < warps; ++w) {
                const int4 v = *reinterpret_cast<const int4*>(red + w * (MT * 16 * LD) + row * LD + c4);
                s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
            }
            int n = p / a.OHW, pos = p - n * a.OHW;
            if (a.vec) {
                uint32_t pk = 0;
                const size_t at = ((size_t)n * g.M + m) * a.OHW + pos;
#pragma unroll
                for (int j = 0; j < 4; ++j) pk |= (uint32_t)(requant_one<YU8>(s[j], mu, a.rq) & 255) << (8 * j);
                if (!YU8 && a.add.res) pk = qadd_word<false>(__ldg(reinterpret_cast<const uint32_t*>(a.add.res + at)), pk, a.add);
                *reinterpret_cast<uint32_t*>((uint8_t*)a.y + at) = pk;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (p + j >= a.P) break;
                    const size_t at = ((size_t)n * g.M + m) * a.OHW + pos;
                    int q = requant_one<YU8>(s[j], mu, a.rq);
                    if (!YU8 && a.add.res) q = (int)(int8_t)qadd_word<false>((uint32_t)__ldg(a.add.res + at), (uint32_t)(q & 255), a.add);
                    store_q<YU8>(a.y, at, q);
                    if (++pos == a.OHW) { pos = 0; ++n; }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------- weights
// Fragment order, on the device: [16-filter tile][K step][32 lanes][4 words], a thread per lane and step.  The weight of (filter, channel,
// tap) is w[m * sm + c * sc + tap * st] (a convolution's [M][C][KH][KW], or a matrix [K][N]).  A call brings its weights along every time:
// shuffled by the host, a 4096 x 4096 matrix took 13 of the call's 13.2 ms.
struct SmallWeightArgs { const int8_t* w; uint4* out; size_t sm, sc, st; int M, C, contiguous, c_steps, k_steps; long long units; };
__global__ void __launch_bounds__(256) small_gemm_weights_k(const __grid_constant__ SmallWeightArgs a) {
    ptx::grid_start();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.units; i += (long long)gridDim.x * blockDim.x) {
        const int lane = (int)(i & 31), gq = lane >> 2, tq = lane & 3;
        const long long t = i >> 5;
        const int s = (int)(t % a.k_steps), tile = (int)(t / a.k_steps);
        const int tap = a.contiguous ? 0 : s / a.c_steps;
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                          // register j: filter gq + 8 * (j & 1), half j >> 1 of the step
            const int m = tile * 16 + gq + (j & 1) * 8, h = j >> 1;
            const int c0 = 4 * (a.contiguous ? (s >> 1) * 16 + tq * 4 + (s & 1) * 2 + h : (s - tap * a.c_steps) * 8 + h * 4 + tq);
            v[j] = 0u;
            if (m < a.M) {
                const int8_t* src = a.w + (size_t)m * a.sm + (size_t)tap * a.st;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c0 + k < a.C) v[j] |= (uint32_t)(uint8_t)__ldg(src + (size_t)(c0 + k) * a.sc) << (8 * k);
            }
        }
        a.out[i] = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// bias - x_zp * (sum of the filter's weights), element k of filter m at w[m * sm + k * sk]: 32 filters a block, 8 threads a filter that
// walk K (sm == 1: the filters are the contiguous side), or a warp a filter.
__global__ void __launch_bounds__(256) small_gemm_bias_k(const int8_t* __restrict__ w, const int32_t* __restrict__ bias, int32_t* __restrict__ out, int M, int K, size_t sm, size_t sk, int x_zp) {
    ptx::grid_start();
    __shared__ int part[256];
    const int tid = threadIdx.x;
    if (sm == 1) {
        const int m = blockIdx.x * 32 + (tid & 31);
        int s = 0;
        if (m < M) for (int k = tid >> 5; k < K; k += 8) s += __ldg(w + (size_t)k * sk + m);
        part[tid] = s;
        __syncthreads();
        if (tid < 32 && m < M) {
            s = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) s += part[j * 32 + tid];
            out[m] = (bias ? __ldg(bias + m) : 0) - x_zp * s;
        }
    } else {
        for (int m = blockIdx.x * 32 + (tid >> 5); m < min(M, (int)blockIdx.x * 32 + 32); m += 8) {
            int s = 0;
            for (int k = tid & 31; k < K; k += 32) s += __ldg(w + (size_t)m * sm + (size_t)k * sk);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((tid & 31) == 0) out[m] = (bias ? __ldg(bias + m) : 0) - x_zp * s;
        }
    }
}

// ---------------------------------------------------------------------------- host side
struct SmallGemmPlan {
    int path = 2, MT = 1, c_steps = 0, k_steps = 0, warps = 1;
    size_t w_bytes = 0;               // weights in fragment order
};

inline bool small_gemm_eligible(const ConvGeom& g, bool w_zp_all_zero) {
    const long long P = (long long)g.N * g.OH * g.OW;
    return g.G == 1 && w_zp_all_zero && P > 0 && P < 256 && (long long)g.Cg * g.KH * g.KW <= (1 << 20) && g.M <= (1 << 20);
}

inline SmallGemmPlan small_gemm_plan(const ConvGeom& g, int sm_count) {
    SmallGemmPlan p;
    const int taps = g.KH * g.KW;
    const bool pointwise = taps == 1 && g.sh == 1 && g.sw == 1 && g.pt == 0 && g.pl == 0 && g.pb == 0 && g.pr == 0;
    p.path = pointwise && g.H * g.W == 1 ? 0 : (pointwise && (g.H * g.W) % 4 == 0 ? 1 : 2);
    p.c_steps = (g.Cg + 31) / 32;
    p.k_steps = p.path == 0 ? (g.Cg + 63) / 64 * 2 : taps * p.c_steps;
    // 32 filters per CTA halve the activation loads; taken when 16 would leave more CTAs than the SMs hold at once anyway
    const long long P = (long long)g.N * g.OH * g.OW, cols = (P + 31) / 32;
    p.MT = (long long)((g.M + 15) / 16) * cols > 2LL * sm_count ? 2 : 1;
    p.warps = std::max(1, std::min(kSmallWarps, p.path == 0 ? p.k_steps / 2 : p.k_steps));
    const int tiles = (g.M + 16 * p.MT - 1) / (16 * p.MT) * p.MT;
    p.w_bytes = (size_t)tiles * p.k_steps * 512;
    return p;
}

// `matrix`: w is [K][N] (g.Cg rows, g.M columns).  With a zero point `bias_out` (g.M values) receives the folded bias; without one it
// is not written and the tensor's own bias goes to run_small_gemm.
inline int32_t run_small_gemm_weights(zant_ctx* ctx, const ConvGeom& g, const SmallGemmPlan& p, bool matrix, const int8_t* w, const int32_t* bias, int x_zp, void* out, int32_t* bias_out) {
    const size_t taps = (size_t)g.KH * g.KW;
    SmallWeightArgs a{};
    a.w = w; a.out = (uint4*)out; a.M = g.M; a.C = g.Cg; a.contiguous = p.path == 0 ? 1 : 0; a.c_steps = p.c_steps; a.k_steps = p.k_steps;
    a.sm = matrix ? 1 : (size_t)g.Cg * taps; a.sc = matrix ? (size_t)g.M : taps; a.st = 1;
    a.units = (long long)(p.w_bytes / 16);
    launch(ctx, small_gemm_weights_k, grid_for((size_t)a.units, 256, ctx->sm_count), 256, 0, a);
    ZB_TRY(check_launch(ctx, "small_gemm_weights_k"));
    if (x_zp == 0) return ZANT_OK;
    launch(ctx, small_gemm_bias_k, (unsigned)((g.M + 31) / 32), 256, 0, w, bias, bias_out, g.M, g.Cg * (int)taps, a.sm, matrix ? (size_t)g.M : (size_t)1, x_zp);
    return check_launch(ctx, "small_gemm_bias_k");
}

// `w_dev`, `bias_dev`: as run_small_gemm_weights leaves them; `bias_dev` may be null.
inline int32_t run_small_gemm(zant_ctx* ctx, const ConvGeom& g, const SmallGemmPlan& p, const void* x, bool x_u8, int x_zp, const void* w_dev, const float* mult_dev,
                              const int32_t* bias_dev, void* y, bool y_u8, const Requant& rq, const QAddTail* add = nullptr) {
    SmallGemmArgs a{};
    if (add) a.add = *add;
    a.x = (const uint8_t*)x; a.w = (const uint4*)w_dev; a.y = y; a.mult = mult_dev; a.bias = bias_dev; a.g = g;
    a.OHW = g.OH * g.OW; a.P = g.N * a.OHW; a.c_steps = p.c_steps; a.k_steps = p.k_steps; a.pad = (uint32_t)(x_zp & 255); a.rq = rq;
    // a word path needs word-aligned rows on the side it vectorises; x that is not falls back to byte loads
    const uintptr_t xa = reinterpret_cast<uintptr_t>(x), ya = reinterpret_cast<uintptr_t>(y);
    int path = p.path;
    if (path == 1 && (xa & 3u)) path = 2;
    a.vec = path == 0 ? (g.C % 16 == 0 && (xa & 15u) == 0) : (a.OHW % 4 == 0 && (ya & 3u) == 0);
    const dim3 grid((unsigned)((g.M + 16 * p.MT - 1) / (16 * p.MT)), (unsigned)((a.P + 31) / 32));
    auto go = [&](auto path_c, auto mt_c) -> int32_t {
        constexpr int PATH = decltype(path_c)::value, MT = decltype(mt_c)::value;
        const size_t smem = (size_t)p.warps * MT * 16 * 36 * 4;          // 36 KB at most
        const int threads = p.warps * 32;
        if (x_u8 && y_u8) launch(ctx, small_gemm_q8_kernel<true, true, PATH, MT>, grid, threads, smem, a);
        else if (x_u8) launch(ctx, small_gemm_q8_kernel<true, false, PATH, MT>, grid, threads, smem, a);
        else if (y_u8) launch(ctx, small_gemm_q8_kernel<false, true, PATH, MT>, grid, threads, smem, a);
        else launch(ctx, small_gemm_q8_kernel<false, false, PATH, MT>, grid, threads, smem, a);
        return check_launch(ctx, "small_gemm_q8_kernel");
    };
    auto with_mt = [&](auto path_c) -> int32_t {
        return p.MT == 2 ? go(path_c, std::integral_constant<int, 2>{}) : go(path_c, std::integral_constant<int, 1>{});
    };
    if (path == 0) return with_mt(std::integral_constant<int, 0>{});
    if (path == 1) return with_mt(std::integral_constant<int, 1>{});
    return with_mt(std::integral_constant<int, 2>{});
}

}  // namespace zb
