// The example CNN (QuantizeLinear -> [QLinearConv 3x3 -> Relu -> MaxPool] x 2 -> QLinearMatMul -> Relu -> QLinearMatMul -> DequantizeLinear on 28 x 28
// images) as one kernel for few images.  The four kernels of fused_cnn.cuh and tc_gemm.cuh are four dependent launches of 3.5 to 4.5 us each, and
// with one image most of the SMs idle in all of them.
//
// A cluster of eight CTAs takes 1, 2, 4, 8 or 16 images: 8, 4, 2 or 1 CTAs an image, or two images a CTA one after the other.  Every CTA quantizes its image and computes the whole first stage (its CTAs
// repeat that: 0.2 M multiplications), then its share of the 25 pool windows of the second, whose codes it writes into the shared memory of all eight
// CTAs; after a cluster barrier each CTA has the images' 1600 activations and multiplies them with 64 of fc1's 512 columns, then with its 64 rows of
// fc2; the sums of fc2 go to the first CTA, which adds them up and dequantises.  All products are warp-level MMAs.  A CTA's weights (102 KB of fc1, 18 of
// conv2) are in fragment order and on their way from the start, before the kernel in front is complete.
//
// What bounds it: latency, about 2 us of launch and 4 of load, two cluster barriers and the chains of MMAs.  Whole network, four kernels -> this one: 1 image 15.9 -> 4.8 us, 30
// 16.6 -> 5.7, 60 17.0 -> 6.2, 120 18.0 -> 7.0, 240 18.8 -> 10.4, 480 20.3 -> 19.8 (two rounds of 15 clusters).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "context.cuh"
#include "fused_cnn.cuh"
#include "irb_band.cuh"
#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"

namespace zb {

struct CnnFewArgs {
    const float* x; float* y;
    int n_images, imgs;                      // imgs: images of a cluster
    float x_scale; int x_zp; float q_rh, q_rl;                              // as in Conv1MmaArgs
    const uint32_t* wfrag; const float* floor1; const float* mult1;
    const uint8_t* w;                        // cnn_few_weights
    const float* floor2; const float* mult2; // [64]: kAccBase - bias, multiplier
    const float* mult3; const int32_t* bias3;
    const float* mult4; const int32_t* bias4;
    int ncls; float y_scale; int y_zp; float dq_scale; int dq_zp;
    int* status;
};

struct CnnFewCfg {
    static constexpr int CTAS = 8, THREADS = 256;
    static constexpr int W3 = 64 * 1600, W2 = 9 * 8 * 256, W4 = 16 * 64;    // a CTA's weights: fc1 [8-column tile][K step][lane][8], conv2 [tap][8-filter tile][lane][8], fc2 [class][64]
    static constexpr int W_CTA = W3 + W4, W_BYTES = CTAS * W_CTA + W2;
    static constexpr int P1 = 36, ROW = 1616;                               // bytes between pixels of the first stage's result, between images' activations
    static constexpr int OFF_W2 = W_CTA, IMGS = 16, OFF_ACT = OFF_W2 + W2, OFF_P1 = OFF_ACT + IMGS * ROW, OFF_IMG = OFF_P1 + 144 * P1, OFF_FC1 = OFF_IMG + 28 * 32 + 32, OFF_SUM = OFF_FC1 + IMGS * 80,
                         OFF_BAR = OFF_SUM + CTAS * IMGS * 16 * 4, SMEM_BYTES = OFF_BAR + 32;
};
static_assert(CnnFewCfg::OFF_P1 % 16 == 0 && CnnFewCfg::OFF_IMG % 16 == 0 && CnnFewCfg::OFF_FC1 % 16 == 0 && CnnFewCfg::OFF_SUM % 16 == 0 && CnnFewCfg::OFF_BAR % 16 == 0 && CnnFewCfg::SMEM_BYTES <= 227 * 1024, "");

// TWO: sixteen images a cluster, two a CTA.
template <bool TWO>
__global__ void __launch_bounds__(CnnFewCfg::THREADS, 1) cnn_few_kernel(const __grid_constant__ CnnFewArgs a) {
    using Cfg = CnnFewCfg;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t s0 = ptx::smem_u32(smem), bar = s0 + Cfg::OFF_BAR;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::OFF_BAR + 16);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int rank = (int)blockIdx.x % Cfg::CTAS, first = (int)blockIdx.x / Cfg::CTAS * a.imgs;
    const int per_img = TWO ? 1 : Cfg::CTAS / a.imgs, per_cta = TWO ? 2 : 1, slot0 = rank * per_cta / per_img, part = per_img > 1 ? rank - slot0 * per_img : 0;
    const int w0 = 25 * part / per_img, w1 = 25 * (part + 1) / per_img;             // this CTA's pool windows of the second stage
    if (tid == 0) {
        ptx::mbar_init(bar, 1); ptx::mbar_init(bar + 8u, 1);
        *abort_flag = 0;
        ptx::mbar_fence_init();
        ptx::mbar_arrive_expect_tx(bar, (uint32_t)Cfg::W2);
        ptx::bulk_g2s(s0 + Cfg::OFF_W2, a.w + (size_t)Cfg::CTAS * Cfg::W_CTA, (uint32_t)Cfg::W2, bar);
        ptx::mbar_arrive_expect_tx(bar + 8u, (uint32_t)Cfg::W_CTA);
        ptx::bulk_g2s(s0, a.w + (size_t)rank * Cfg::W_CTA, (uint32_t)Cfg::W_CTA, bar + 8u);
    }
    // windows in groups of eight, a group's eight 8-filter tiles over 8 / groups warps
    const int groups = w1 - w0 <= 8 ? 1 : (w1 - w0 <= 16 ? 2 : 4), group = warp / (8 / groups), nt0 = (warp - group * (8 / groups)) * groups;
    float2 fl2[4], ml2[4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
        if (n < groups) {
            fl2[n] = __ldg(reinterpret_cast<const float2*>(a.floor2 + (nt0 + n) * 8 + 2 * q)); ml2[n] = __ldg(reinterpret_cast<const float2*>(a.mult2 + (nt0 + n) * 8 + 2 * q));
        }
    const int col = rank * 64 + warp * 8 + 2 * q;                                   // fc1
    const float2 m3 = __ldg(reinterpret_cast<const float2*>(a.mult3 + col));
    const int2 b3 = __ldg(reinterpret_cast<const int2*>(a.bias3 + col));
    __syncthreads();                                                                // (the barriers are set up before any thread waits on one)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");           // this CTA's shared memory may be written to
    ptx::grid_trigger();
    ptx::grid_wait();
    // ---------------------------------------------------------------- QuantizeLinear: rows 0..25 (the pools read no others), 32 bytes apart
    uint32_t* img = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_IMG);
#pragma unroll 1
    for (int slot = slot0; slot < slot0 + per_cta; ++slot) {
        const int image = first + slot;
        if (tid < 182 && image < a.n_images) {
            float4 v = __ldg(reinterpret_cast<const float4*>(a.x + (size_t)image * 784) + tid);
            if (a.q_rl != 0.0f) {
                v.x = quant_quotient(v.x, a.q_rh, a.q_rl); v.y = quant_quotient(v.y, a.q_rh, a.q_rl); v.z = quant_quotient(v.z, a.q_rh, a.q_rl); v.w = quant_quotient(v.w, a.q_rh, a.q_rl);
            } else {
                v.x = __fdiv_rn(v.x, a.x_scale); v.y = __fdiv_rn(v.y, a.x_scale); v.z = __fdiv_rn(v.z, a.x_scale); v.w = __fdiv_rn(v.w, a.x_scale);
            }
            // (conv1_mma_relu_pool_kernel's clamp: integer bounds, a NaN becomes the lower one; with zero point 0 a NaN becomes 0, which is it)
            const float lo = (float)(-a.x_zp), hi = (float)(255 - a.x_zp);
            const uint32_t q0 = (uint32_t)(__float2int_rn(fminf(fmaxf(v.x, lo), hi)) + a.x_zp), q1 = (uint32_t)(__float2int_rn(fminf(fmaxf(v.y, lo), hi)) + a.x_zp);
            const uint32_t q2 = (uint32_t)(__float2int_rn(fminf(fmaxf(v.z, lo), hi)) + a.x_zp), q3 = (uint32_t)(__float2int_rn(fminf(fmaxf(v.w, lo), hi)) + a.x_zp);
            img[tid / 7 * 8 + tid % 7] = q0 | (q1 << 8) | (q2 << 16) | (q3 << 24);
        }
        __syncthreads();
        // ---------------------------------------------------------------- stage 1: 12 x 12 pooled pixels, 16 a unit, half of the channel groups an item (see
        // conv1_mma_relu_pool_kernel)
        int base_q[4] = {kAccBaseBits, kAccBaseBits, kAccBaseBits, kAccBaseBits};
        for (int it = warp; it < 18; it += 8) {
            const int u = it >> 1, jp = it & 1, pa = u * 16 + g, pb = pa + 8;
            auto patch = [&](int p) {
                const int py = p / 12, px = p - py * 12;
                const uint32_t* r = img + (2 * py + q) * 8 + (px >> 1);
                return __byte_perm(r[0], r[1], (px & 1) ? 0x5432u : 0x3210u);
            };
            const uint32_t a0 = patch(pa), a1 = patch(pb);
            int r[2][4];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
                const int j = jp * 2 + jj;
                int d[4][4];
#pragma unroll
                for (int m = 0; m < 4; ++m) mma_m16n8k16_u8s8(d[m], a0, a1, __ldg(a.wfrag + (m * 4 + j) * 32 + lane), base_q);
                const float2 f = __ldg(reinterpret_cast<const float2*>(a.floor1) + j * 32 + lane), ml = __ldg(reinterpret_cast<const float2*>(a.mult1) + j * 32 + lane);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float fk = (k & 1) ? f.y : f.x;
                    const int mx = __vimax3_s32(__vimax3_s32(d[0][k], d[1][k], d[2][k]), d[3][k], __float_as_int(fk));
                    r[jj][k] = __float2int_rn(__fmul_rn(__fsub_rn(__int_as_float(mx), fk), (k & 1) ? ml.y : ml.x));
                }
            }
            sts_u32(s0 + (uint32_t)(Cfg::OFF_P1 + pa * Cfg::P1 + 8 * q + 4 * jp), pack_sat_s8x4(r[0][0], r[0][1], r[1][0], r[1][1]));
            sts_u32(s0 + (uint32_t)(Cfg::OFF_P1 + pb * Cfg::P1 + 8 * q + 4 * jp), pack_sat_s8x4(r[0][2], r[0][3], r[1][2], r[1][3]));
        }
        if (slot == slot0) ptx::mbar_wait(bar, 0u, abort_flag);
        __syncthreads();
        // ---------------------------------------------------------------- stage 2: rows g and g + 8 of two MMAs are the four members of window g of the group
        {
            const int win = w0 + group * 8 + g, wc = min(win, w1 - 1), wy = wc / 5, wx = wc - wy * 5;
            uint32_t v[4][4][2];                                                        // view (ry, rx) of the window, both K halves
#pragma unroll
            for (int ry = 0; ry < 4; ++ry)
#pragma unroll
                for (int rx = 0; rx < 4; ++rx) {
                    const uint32_t ad = s0 + (uint32_t)(Cfg::OFF_P1 + ((2 * wy + ry) * 12 + 2 * wx + rx) * Cfg::P1 + 4 * q);
                    v[ry][rx][0] = lds_u32<0>(ad); v[ry][rx][1] = lds_u32<16>(ad);
                }
            if (slot == slot0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // the other CTAs have started
            uint32_t to[Cfg::CTAS];
#pragma unroll
            for (int r = 0; r < Cfg::CTAS; ++r)
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to[r]) : "r"(s0 + (uint32_t)(Cfg::OFF_ACT + slot * Cfg::ROW + wc * 64 + nt0 * 8 + 2 * q)), "r"(r));
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                if (n >= groups) break;
                int da[4] = {kAccBaseBits, kAccBaseBits, kAccBaseBits, kAccBaseBits}, db[4] = {kAccBaseBits, kAccBaseBits, kAccBaseBits, kAccBaseBits};
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int kh = t / 3, kw = t - kh * 3;
                    const uint2 b = lds_u64(s0 + (uint32_t)(Cfg::OFF_W2 + ((t * 8 + nt0 + n) * 32 + lane) * 8));
                    mma_m16n8k32_s8(da, make_uint4(v[kh][kw][0], v[kh][kw + 1][0], v[kh][kw][1], v[kh][kw + 1][1]), b.x, b.y);
                    mma_m16n8k32_s8(db, make_uint4(v[kh + 1][kw][0], v[kh + 1][kw + 1][0], v[kh + 1][kw][1], v[kh + 1][kw + 1][1]), b.x, b.y);
                }
                int k[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float f = c ? fl2[n].y : fl2[n].x;
                    const int mx = __vimax3_s32(__vimax3_s32(da[c], da[2 + c], db[c]), db[2 + c], __float_as_int(f));
                    k[c] = __float2int_rn(__fmul_rn(__fsub_rn(__int_as_float(mx), f), c ? ml2[n].y : ml2[n].x));
                }
                const uint16_t code = (uint16_t)pack_sat_s8x2(k[0], k[1]);
                if (win < w1) {
#pragma unroll
                    for (int r = 0; r < Cfg::CTAS; ++r) asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(to[r] + 8u * (uint32_t)n), "h"(code) : "memory");
                }
            }
        }
    }
    ptx::mbar_wait(bar + 8u, 0u, abort_flag);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // ---------------------------------------------------------------- fc1: eight columns a warp, images on the rows; four chains of MMAs
    {
        int acc[4][4] = {};
        const uint32_t ra = s0 + (uint32_t)(Cfg::OFF_ACT + g * Cfg::ROW + 4 * q), rb = s0 + (uint32_t)((warp * 50 * 32 + lane) * 8);
#pragma unroll
        for (int ks = 0; ks < 50; ++ks) {
            const uint2 b = lds_u64(rb + (uint32_t)ks * 256u);
            const uint32_t ak = ra + (uint32_t)ks * 32u;
            uint4 f = make_uint4(lds_u32<0>(ak), 0u, lds_u32<16>(ak), 0u);
            if (TWO) { f.y = lds_u32<0>(ak + 8u * Cfg::ROW); f.w = lds_u32<16>(ak + 8u * Cfg::ROW); }
            mma_m16n8k32_s8(acc[ks & 3], f, b.x, b.y);
        }
#pragma unroll
        for (int h = 0; h < per_cta; ++h) {
            const int k0 = max(rq_round(acc[0][2 * h] + acc[1][2 * h] + acc[2][2 * h] + acc[3][2 * h] + b3.x, m3.x), 0);
            const int k1 = max(rq_round(acc[0][2 * h + 1] + acc[1][2 * h + 1] + acc[2][2 * h + 1] + acc[3][2 * h + 1] + b3.y, m3.y), 0);
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(s0 + (uint32_t)(Cfg::OFF_FC1 + (g + 8 * h) * 80 + warp * 8 + 2 * q)), "h"((uint16_t)pack_sat_s8x2(k0, k1)) : "memory");
        }
    }
    __syncthreads();
    // ---------------------------------------------------------------- fc2: this CTA's 64 rows, a thread an image and class, the sums to the first CTA
    if (tid < a.imgs * 16) {
        const int i = tid >> 4, c = tid & 15;
        int s = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint4 x = lds_u128(s0 + (uint32_t)(Cfg::OFF_FC1 + i * 80 + 16 * k)), w = lds_u128(s0 + (uint32_t)(Cfg::W3 + c * 64 + 16 * k));
            s = __dp4a((int)x.x, (int)w.x, s); s = __dp4a((int)x.y, (int)w.y, s); s = __dp4a((int)x.z, (int)w.z, s); s = __dp4a((int)x.w, (int)w.w, s);
        }
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(s0 + (uint32_t)(Cfg::OFF_SUM + (rank * 256 + tid) * 4)), "r"(0));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(s) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 0 && tid < a.imgs * 16) {
        const int i = first + (tid >> 4), c = tid & 15;
        if (i < a.n_images && c < a.ncls) {
            int s = __ldg(a.bias4 + c);
#pragma unroll
            for (int r = 0; r < Cfg::CTAS; ++r) s += (int)lds_u32<0>(s0 + (uint32_t)(Cfg::OFF_SUM + (r * 256 + tid) * 4));
            const int k = requant_one<false>(s, __ldg(a.mult4 + c), Requant{a.y_scale, a.y_zp, ZANT_QACT_NONE});
            a.y[(size_t)i * a.ncls + c] = __fmul_rn(__int2float_rn(k - a.dq_zp), a.dq_scale);
        }
    }
    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);                            // (copies still in flight land before the CTA's memory goes away)
    }
    if (tid == 0 && *abort_flag) atomicExch(a.status, (int)DEV_ERR_WAIT_TIMEOUT);
}

// w2 [64][32][3][3], w3 [1600][512] with rows (c, h, w), w4 [512][ncls] -> CnnFewArgs::w.  (K of fc1 is (h, w, c), the order in which the second stage's
// codes are written.)
inline void cnn_few_weights(const int8_t* w2, const int8_t* w3, const int8_t* w4, int ncls, std::vector<uint8_t>& out) {
    using Cfg = CnnFewCfg;
    out.assign(Cfg::W_BYTES, 0);
    for (int hw = 0; hw < 25; ++hw)
        for (int c = 0; c < 64; c += 4) {
            const int8_t *r0 = w3 + (size_t)(c * 25 + hw) * 512, *r1 = r0 + 25 * 512, *r2 = r1 + 25 * 512, *r3 = r2 + 25 * 512;
            const int ks = hw * 2 + (c >> 5), half = (c & 31) >> 4, q = (c & 15) >> 2;
            for (int n = 0; n < 512; ++n) {
                const uint32_t v = (uint32_t)(uint8_t)r0[n] | (uint32_t)(uint8_t)r1[n] << 8 | (uint32_t)(uint8_t)r2[n] << 16 | (uint32_t)(uint8_t)r3[n] << 24;
                std::memcpy(out.data() + (size_t)(n >> 6) * Cfg::W_CTA + ((size_t)(((n >> 3) & 7) * 50 + ks) * 32 + (n & 7) * 4 + q) * 8 + half * 4, &v, 4);
            }
        }
    for (int n = 0; n < 512; ++n)
        for (int c = 0; c < ncls; ++c) out[(size_t)(n >> 6) * Cfg::W_CTA + Cfg::W3 + c * 64 + (n & 63)] = (uint8_t)w4[n * ncls + c];
    uint8_t* b = out.data() + (size_t)Cfg::CTAS * Cfg::W_CTA;
    for (int f = 0; f < 64; ++f)
        for (int ch = 0; ch < 32; ++ch)
            for (int t = 0; t < 9; ++t) b[((size_t)(t * 8 + f / 8) * 32 + (f % 8) * 4 + ((ch & 15) >> 2)) * 8 + (ch >> 4) * 4 + (ch & 3)] = (uint8_t)w2[(f * 32 + ch) * 9 + t];
}

}  // namespace zb
