// Fused kernels for quantized 3x3 convolution stages followed by ReLU and a 2x2/2 MaxPool.
//
// Internal activation layout between the two stages, "image blocks": [N / 128][12 x 12 pixels][2 chunks of 16 channels][128 images][16]
// (a batch below 128: one block of as many images, whose MMA rows beyond them read the bytes behind and are not stored), so that the 128 rows of an MMA are the same pixel of 128 images.  With that layout the A operand of an implicit-GEMM convolution
// FOLLOWED BY a 2x2/2 pool needs no im2col and computes nothing twice: the view (ry, rx) of a pool window - input pixel (2py + ry, 2px + rx),
// ry = dy + kh, rx = dx + kw - is one 4 KB block (K-major, no swizzle: 8 rows = 8 consecutive 16-byte chunks), and every one of the
// 25 windows of an image is a tile row that is kept.
//
// MaxPool is applied to the int32 accumulators BEFORE requantisation.  That is exact because the
// requantisation y = sat(rne(float(acc + bias) * M) + zp) is non-decreasing in acc whenever M > 0
// (checked on the host), so max and requantise commute; the bias is the same for the four members of a
// window, so it is added after the max.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "kernels_q8.cuh"
#include "ptx_sm100.cuh"

namespace zb {

enum DeviceError : int {
    DEV_OK = 0,
    DEV_ERR_WAIT_TIMEOUT = 1,   // a bounded mbarrier wait gave up
};

// =============================================================================================
// Stage 1: QuantizeLinear(uint8) + QLinearConv(1 -> 32, 3x3, stride 1, no pad) + ReLU + MaxPool 2x2/2
//          float [N,1,28,28]  ->  int8 image blocks (c2_block_bytes)
// Host-side description of the stage (the plan fills it from the graph; the kernel below takes its
// own argument block derived from it).
// =============================================================================================
struct Conv1Args {
    const float* x;
    int8_t* y;
    int n_images;
    float x_scale; int x_zp;            // QuantizeLinear of the input (uint8)
    uint32_t wpack[32][3][2];           // [m][kh][dx]: dx=0 -> bytes (w0,w1,w2,0); dx=1 -> (0,w0,w1,w2)
    float mult[32];                     // (x_scale * w_scale[m]) / y_scale
    int32_t bias[32];                   // bias[m] - x_zp * sum(w[m])   (no padding: all 9 taps always valid)
    float y_scale; int y_zp; int act;
};

// =============================================================================================
// Stage 1 kernel.  The contraction is only 9 deep and the input has one channel, so the 128-row
// tcgen05 shape has nothing to contract over; the 3x3 contraction runs on warp-level int8 MMAs (mma.sync m16n8k16, u8 x s8 -> s32):
//   rows    = 16 pooled pixels (two per thread-row group g and g+8),
//   K (16)  = the 4x4 input patch of a pooled pixel, byte (r,s) at k = 4r + s, so a thread's A
//             register is simply patch row r = lane%4 as one packed word,
//   columns = 8 output channels; the four members (dy,dx) of the 2x2 pool window are four
//             MMAs with the filter shifted inside the patch (zero where it falls outside).
// All four members of one pooled pixel and channel land in the same thread and register slot,
// so the pool is three max instructions without any data exchange.  Channels are permuted
// (group j, column n <-> channel 8*(n/2) + 2j + n%2) so that a thread ends up with eight
// consecutive channels of its two pixels and stores them as one 8-byte word each.
// =============================================================================================
struct Conv1MmaArgs {
    const float* x;
    int8_t* y;
    int n_images, ib;
    float x_scale; int x_zp;
    float q_rh, q_rl;        // the quotient of the quantisation in two instructions (quant_steps); q_rl == 0: by division
    const uint32_t* wfrag;   // [4 members][4 groups][32 lanes] B-fragment words
    const float* floorfrag;  // [4 groups][32 lanes][2]  kAccBase - (bias - x_zp * sum(w)) of the lane's two columns (or the bits of the bias)
    const float* multfrag;   // [4 groups][32 lanes][2]
    int* status;             // device status word: DEV_ERR_WAIT_TIMEOUT when a bounded wait gave up
    // Output layout: image blocks for tc_conv3x3_pool_kernel; pooled row and column 12 are neither computed nor stored (the next
    // stage's pool never reads them).
};

__device__ __forceinline__ void mma_m16n8k16_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const int (&c)[4]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

// Accumulators that start at the bit pattern of 1.5 * 2^23 are, read as floats, 1.5 * 2^23 + acc exactly (|acc| < 2^22), and order as
// integers the way the sums do.  With floor = 1.5 * 2^23 - bias, max(acc', floor) as integers is the ReLU and one subtraction of floats
// then gives float(max(acc + bias, 0)): no register moves of the bias into the MMAs' C operand (one quad serves all of
// them) and no integer -> float conversion, which shares the half-rate ALU pipe with the maxima.
constexpr int kAccBaseBits = 0x4b400000;
constexpr float kAccBase = 12582912.0f;
// biases that keep floor and the sums of nine products of 255 x 128 inside [2^23, 2^24)
inline bool acc_base_ok(int32_t bias) { return bias > -3800000 && bias < 3800000; }

inline float int_bits_as_float(int32_t v) { float f; std::memcpy(&f, &v, 4); return f; }

// Image blocks between the stages: ib = min(128, N) images, a pixel is both their 16-channel chunks, 144 pixels are a block.
__host__ __device__ constexpr int c2_pixel_bytes(int ib) { return 2 * ib * 16; }
__host__ __device__ constexpr int c2_block_bytes(int ib) { return 144 * c2_pixel_bytes(ib); }

// Images per CTA iteration: 4 x 144 pooled pixels = 36 units of 16.
constexpr int C1M_G = 4;
constexpr int C1M_THREADS = 384;
// words of a quantized image in shared memory: the four images of a unit's rows lie in different banks
constexpr int C1M_IMG_WORDS = 28 * 8 + 2;

constexpr int C1M_IMG_FLOATS = 28 * 28;
constexpr int C1M_GROUP_BYTES = C1M_G * C1M_IMG_FLOATS * 4;   // 9408: a multiple of 16, as the bulk copy wants

// The float images of a group arrive by one bulk async copy into a two-deep shared-memory ring: the copy
// of group i+1 is issued when the MMA phase of group i starts, so no thread waits on global loads.  The
// quantized bytes are double-buffered too, which leaves one __syncthreads per group.
// A group is 36 units of 16 rows: four neighbouring pixels of a pooled row times its four images.  Twelve warps take three units each, the same
// third of every fourth row, and a thread's rows are one image's pixels of one column parity, so that everything about a unit but
// constant offsets is known before the loop (a table of pixels and eight warps, 4.5 units each, cost 870 of 1880 warp instructions an image).
// Two CTAs per SM (80 registers per thread).
// BASE false: biases that do not qualify (acc_base_ok); the accumulators start at 0 and are converted.
template <bool BASE>
__global__ void __launch_bounds__(C1M_THREADS, 2) conv1_mma_relu_pool_kernel(const Conv1MmaArgs a) {
    ptx::grid_start();
    __shared__ __align__(128) float stage[2][C1M_G * C1M_IMG_FLOATS];
    __shared__ uint32_t img2[2][C1M_G * C1M_IMG_WORDS];   // quantized uint8 rows of 32 bytes (28 pixels + 4 pad)
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int stride = gridDim.x * C1M_G;
    const uint32_t bar0 = ptx::smem_u32(&bars[0]);
    if (tid == 0) {
        abort_flag = 0;
        ptx::mbar_init(bar0, 1); ptx::mbar_init(bar0 + 8, 1);
        ptx::mbar_fence_init();
        const int base = blockIdx.x * C1M_G;
        if (base < a.n_images) {
            const uint32_t bytes = (uint32_t)min(C1M_G, a.n_images - base) * (C1M_IMG_FLOATS * 4);
            ptx::mbar_arrive_expect_tx(bar0, bytes);
            ptx::bulk_g2s(ptx::smem_u32(&stage[0][0]), a.x + (size_t)base * C1M_IMG_FLOATS, bytes, bar0);
        }
    }
    uint32_t wf[4][4]; float flr[4][2]; float mult[4][2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) wf[m][j] = __ldg(a.wfrag + (m * 4 + j) * 32 + lane);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int b = 0; b < 2; ++b) { flr[j][b] = __ldg(a.floorfrag + (j * 32 + lane) * 2 + b); mult[j][b] = __ldg(a.multfrag + (j * 32 + lane) * 2 + b); }
    int base_q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) asm volatile("mov.b32 %0, %1;" : "=r"(base_q[k]) : "n"(BASE ? kAccBaseBits : 0));   // (opaque: kept in a register quad)
    __syncthreads();                               // barriers and the abort flag are set up

    const float q_lo = (float)(-a.x_zp), q_hi = (float)(255 - a.x_zp);
    // Only the 12 x 12 pooled pixels that the next stage reads are computed.  Rows g and g + 8 of unit k of this warp: image g % 4, pooled row
    // warp / 3 + 4k, columns 4 (warp % 3) + g / 4 and the one two further; patch row t.  This thread's 8 channels: chunk t >> 1, half t & 1.
    const int my_img = g & 3, odd = g >> 2;
    const uint32_t sel = odd ? 0x5432u : 0x3210u;
    const int word0 = my_img * C1M_IMG_WORDS + (warp / 3) * 16 + t * 8 + (warp % 3) * 2;
    const int pixel = c2_pixel_bytes(a.ib);
    int8_t* const y_thread = a.y + ((warp / 3) * 12 + (warp % 3) * 4 + odd) * pixel + (t >> 1) * (pixel >> 1) + my_img * 16 + (t & 1) * 8;
    // The float4s that this thread quantizes: pooled rows and columns 0..11 read input rows 0..25 (26 rows of 7 float4)
    constexpr int n_f4 = C1M_G * 182, F4 = (n_f4 + C1M_THREADS - 1) / C1M_THREADS;
    int f_src[F4], f_dst[F4], f_img[F4];
#pragma unroll
    for (int k = 0; k < F4; ++k) {
        const int i = tid + k * C1M_THREADS, gi = i / 182, p4 = i - gi * 182, r = p4 / 7;
        f_src[k] = gi * 196 + p4; f_dst[k] = gi * C1M_IMG_WORDS + r * 8 + (p4 - r * 7); f_img[k] = i < n_f4 ? gi : C1M_G;
    }
    int it = 0;
    for (int base = blockIdx.x * C1M_G; base < a.n_images; base += stride, ++it) {
        const int s = it & 1;
        // ---- the group's floats have landed (bounded wait; after a time-out the results are void and the
        //      status word says so)
        ptx::mbar_wait(bar0 + 8 * s, (uint32_t)(it >> 1) & 1u, &abort_flag);
        // ---- quantize C1M_G images: float4 in, four uint8 out
        uint32_t* img = img2[s];
        const int n_here = min(C1M_G, a.n_images - base);
#pragma unroll
        for (int k = 0; k < F4; ++k) {
            if (f_img[k] < n_here) {
                uint32_t word;
                float4 v = reinterpret_cast<const float4*>(stage[s])[f_src[k]];
                if (a.q_rl != 0.0f) {
                    v.x = quant_quotient(v.x, a.q_rh, a.q_rl); v.y = quant_quotient(v.y, a.q_rh, a.q_rl);
                    v.z = quant_quotient(v.z, a.q_rh, a.q_rl); v.w = quant_quotient(v.w, a.q_rh, a.q_rl);
                } else {
                    v.x = __fdiv_rn(v.x, a.x_scale); v.y = __fdiv_rn(v.y, a.x_scale); v.z = __fdiv_rn(v.z, a.x_scale); v.w = __fdiv_rn(v.w, a.x_scale);
                }
                if (a.x_zp == 0) {
                    // zero point 0: sat_u8(rne(clamp(t, -512, 511))) is the float -> int32 conversion (rne, a NaN gives 0) followed
                    // by the pack instruction's own saturation to [0, 255]; no clamps, no adds (the ALU pipe bounds this kernel)
                    word = pack_sat_u8x4(__float2int_rn(v.x), __float2int_rn(v.y), __float2int_rn(v.z), __float2int_rn(v.w));
                } else {
                    // sat_u8(rne(clamp(t, -512, 511)) + zp) == rne(clamp(t, -zp, 255 - zp)) + zp: the bounds are integers
                    // inside [-512, 511] and rounding is monotonic; a NaN becomes the lower bound either way.
                    const int q0 = __float2int_rn(fminf(fmaxf(v.x, q_lo), q_hi)) + a.x_zp, q1 = __float2int_rn(fminf(fmaxf(v.y, q_lo), q_hi)) + a.x_zp;
                    const int q2 = __float2int_rn(fminf(fmaxf(v.z, q_lo), q_hi)) + a.x_zp, q3 = __float2int_rn(fminf(fmaxf(v.w, q_lo), q_hi)) + a.x_zp;
                    word = (uint32_t)q0 | ((uint32_t)q1 << 8) | ((uint32_t)q2 << 16) | ((uint32_t)q3 << 24);
                }
                img[f_dst[k]] = word;
            }
        }
        __syncthreads();
        // ---- every thread is done with the other ring slot (it was read one group ago): refill it
        if (tid == 0 && base + stride < a.n_images) {
            const int nb = base + stride;
            const uint32_t bytes = (uint32_t)min(C1M_G, a.n_images - nb) * (C1M_IMG_FLOATS * 4);
            const uint32_t bar = bar0 + 8 * (s ^ 1);
            ptx::mbar_arrive_expect_tx(bar, bytes);
            ptx::bulk_g2s(ptx::smem_u32(&stage[s ^ 1][0]), a.x + (size_t)nb * C1M_IMG_FLOATS, bytes, bar);
        }
        // ---- 16 pooled pixels per warp iteration (a group does not straddle blocks of 128 images)
        int8_t* const y_group = y_thread + (size_t)(base >> 7) * (144 * 4096) + (base & 127) * 16;
        const bool ok = base + my_img < a.n_images;
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {
            const uint32_t* row = img + word0 + k * 64;
            const uint32_t x0 = row[0], x1 = row[1], x2 = row[2];
            const uint32_t afrag[2] = {__byte_perm(x0, x1, sel), __byte_perm(x1, x2, sel)};
            uint32_t outw[2][2];
#pragma unroll
            for (int jp = 0; jp < 2; ++jp) {          // two channel groups at a time -> one packed word per pixel
                int r[2][4];                          // [j in pair][row g: ch0, ch1 ; row g+8: ch0, ch1]
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    const int j = jp * 2 + jj;
                    int d0[4], d1[4], d2[4], d3[4];
                    mma_m16n8k16_u8s8(d0, afrag[0], afrag[1], wf[0][j], base_q);
                    mma_m16n8k16_u8s8(d1, afrag[0], afrag[1], wf[1][j], base_q);
                    mma_m16n8k16_u8s8(d2, afrag[0], afrag[1], wf[2][j], base_q);
                    mma_m16n8k16_u8s8(d3, afrag[0], afrag[1], wf[3][j], base_q);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int mx = __vimax3_s32(d0[k], d1[k], d2[k]);
                        const float f = flr[j][k & 1];                 // BASE: kAccBase - bias, else the bits of the bias
                        const float v = BASE ? __fsub_rn(__int_as_float(__vimax3_s32(mx, d3[k], __float_as_int(f))), f)
                                             : __int2float_rn(max(max(mx, d3[k]) + __float_as_int(f), 0));
                        r[jj][k] = __float2int_rn(__fmul_rn(v, mult[j][k & 1]));
                    }
                }
                outw[0][jp] = pack_sat_s8x4(r[0][0], r[0][1], r[1][0], r[1][1]);   // row g   : ch 8t+4jp .. +3
                outw[1][jp] = pack_sat_s8x4(r[0][2], r[0][3], r[1][2], r[1][3]);   // row g+8
            }
            if (ok) {
                int8_t* yo = y_group + k * (48 * pixel);
                *reinterpret_cast<uint2*>(yo) = make_uint2(outw[0][0], outw[0][1]);
                *reinterpret_cast<uint2*>(yo + 2 * pixel) = make_uint2(outw[1][0], outw[1][1]);
            }
        }
    }
    if (tid == 0 && abort_flag) atomicExch(a.status, (int)DEV_ERR_WAIT_TIMEOUT);
}

// =============================================================================================
// Stage 2: QLinearConv(32 -> 64, 3x3, no pad) + ReLU + MaxPool 2x2/2 on the image blocks that stage 1 writes.
//
// A tile is one pool window (py, px) of 128 images: MMA row r is image 128 * block + r.  The members (dy, dx) of the window are four accumulators
// of 64 columns; the two of a row dy are one MMA accumulator of 128: filter row kh of member row dy reads the views (dy + kh, rx), rx 0..3, and
// the block (kh, rx) of the weights holds tap (kh, rx) for dx = 0 and tap (kh, rx - 1) for dx = 1, zeros where that tap does not exist: 24 MMAs of
// 128x128x32 a tile.  MMAs write TMEM in the order of issue only when they have the same accumulator and the same shape; hence two accumulators
// that do not overlap and one shape.  (18 MMAs of 64, 128 and 256 columns, all of them useful, accumulated into columns that overlap: 102 us at
// batch 65536, 117 with this form; one 128x256x32 MMA for each of the 16 views 130.)
//
// An item is a row of five windows (block, py), or one window where that takes the rounds of the SMs less time (the plan's rule).  Its input is
// six (two) column pairs of 4 x 2 pixels, 32 KB each, of which a window reads two: a ring of five stages, each read by two windows.
//   warp 0 producer, warp 1 MMA issuer (the whole warp runs the loop, one lane issues; TMEM: two sets of 4 x 64 columns, so the epilogue of a
//   tile overlaps the MMAs of the next), warps 2-17 epilogue: a thread holds all four members of its window for 16 filters - max, bias, ReLU
//   and requantisation in registers, one 16-byte store into the GEMM-blocked layout [N/128][1600/16][ib images][16], 512 contiguous bytes a warp.
// =============================================================================================
struct TcConvPoolArgs {
    const int8_t* x;
    const int8_t* w;                    // tc_conv_pool_weights
    float mult[64], bias[64];           // per filter, constant-bank operands; bias - x_zp * sum(w) as kAccBase - bias (BASE), else its bits
    int8_t* y;
    int n_images, ib, items, wins;      // images per block, items, windows per item (5 or 1)
    int* status;
};

struct TcConvPoolCfg {
    static constexpr int STAGES = 5, STAGE_BYTES = 8 * c2_pixel_bytes(128);      // [ry][column of the pair][chunk][128][16]
    static constexpr int W_BLOCK_BYTES = 2 * 128 * 16, W_BYTES = 12 * W_BLOCK_BYTES;     // [kh][rx][chunk][dx][64][16]
    static constexpr int OFF_A = W_BYTES, OFF_BAR = OFF_A + STAGES * STAGE_BYTES, SMEM_BYTES = OFF_BAR + 256;
    static constexpr int TMEM_COLS = 512, THREADS = 576;
};
static_assert(TcConvPoolCfg::OFF_A % 128 == 0 && TcConvPoolCfg::SMEM_BYTES <= 227 * 1024, "");

// w: [64][32][3][3]
inline void tc_conv_pool_weights(const int8_t* w, int8_t* out) {
    std::memset(out, 0, TcConvPoolCfg::W_BYTES);
    for (int kh = 0; kh < 3; ++kh)
        for (int rx = 0; rx < 4; ++rx)
            for (int dx = 0; dx < 2; ++dx) {
                const int kw = rx - dx;
                if (kw < 0 || kw > 2) continue;
                for (int ch = 0; ch < 32; ++ch)
                    for (int m = 0; m < 64; ++m)
                        out[(kh * 4 + rx) * TcConvPoolCfg::W_BLOCK_BYTES + (ch / 16 * 128 + dx * 64 + m) * 16 + ch % 16] = w[(m * 32 + ch) * 9 + kh * 3 + kw];
            }
}

template <bool BASE>
__global__ void __launch_bounds__(576, 1) tc_conv3x3_pool_kernel(const __grid_constant__ TcConvPoolArgs a) {
    using Cfg = TcConvPoolCfg;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sW = smem;
    uint8_t* sA = smem + Cfg::OFF_A;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_BAR + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::OFF_BAR + 132);
    const uint32_t bar0 = ptx::smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (Cfg::STAGES + s); };
    auto tfull = [&](int b) { return bar0 + 8u * (2 * Cfg::STAGES + b); };
    auto tempty = [&](int b) { return bar0 + 8u * (2 * Cfg::STAGES + 2 + b); };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) { ptx::mbar_init(full(s), 1); ptx::mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; ++b) { ptx::mbar_init(tfull(b), 1); ptx::mbar_init(tempty(b), 16); }
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    for (int i = tid; i < Cfg::W_BYTES / 16; i += Cfg::THREADS)
        reinterpret_cast<uint4*>(sW)[i] = __ldg(reinterpret_cast<const uint4*>(a.w) + i);
    ptx::fence_proxy_async_smem();
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(tmem_slot), Cfg::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_trigger();
    ptx::grid_wait();

    const int pixel = c2_pixel_bytes(a.ib);
    if (warp == 0) {
        // ------------------------------------------------------------------ producer: the column pairs of the items
        if (ptx::elect_one()) {
            int s = 0; uint32_t ph = 0;
            bool alive = true;
            for (int item = blockIdx.x; item < a.items && alive; item += gridDim.x) {
                const int win = item * a.wins, nb = win / 25, py = (win - nb * 25) / 5, px0 = win % 5;
                const int8_t* src = a.x + (size_t)nb * (144 * pixel) + (size_t)((2 * py) * 12 + 2 * px0) * pixel;
                for (int cp = 0; cp <= a.wins; ++cp, src += 2 * pixel) {
                    if (!ptx::mbar_wait(empty(s), ph ^ 1u, abort_flag)) { alive = false; break; }
                    const uint32_t dst = ptx::smem_u32(sA + s * Cfg::STAGE_BYTES);
                    // (a last block's images that do not exist: whatever is there)
                    ptx::mbar_arrive_expect_tx(full(s), (uint32_t)(8 * pixel));
#pragma unroll
                    for (int ry = 0; ry < 4; ++ry)
                        ptx::bulk_g2s(dst + (uint32_t)(ry * 2 * pixel), src + (size_t)(ry * 12) * pixel, (uint32_t)(2 * pixel), full(s));
                    if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t leader = ptx::elect_one() ? 1u : 0u;
        auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag)) != 0; };
        const uint64_t da = ptx::smem_desc_kmajor(0, (uint32_t)pixel >> 1, 128);
        const uint32_t pixel_u = (uint32_t)pixel >> 4;
        const uint32_t hi = (uint32_t)(da >> 32), a_lo0 = (uint32_t)da + (ptx::smem_u32(sA) >> 4), w_lo0 = (uint32_t)ptx::smem_desc_kmajor(ptx::smem_u32(sW), 2048, 128);
        int s = 0, it = 0; uint32_t ph = 0;                       // stage of the window's left column pair
        bool alive = true;
        for (int item = blockIdx.x; item < a.items && alive; item += gridDim.x) {
            for (int px = 0; px < a.wins; ++px, ++it) {
                const int b = it & 1;
                const int s1 = s + 1 == Cfg::STAGES ? 0 : s + 1;
                const uint32_t ph1 = s1 == 0 ? ph ^ 1u : ph;
                alive = wait(tempty(b), ((uint32_t)(it >> 1) & 1u) ^ 1u) && (px > 0 || wait(full(s), ph)) && wait(full(s1), ph1);
                if (!alive) break;
                ptx::tc_fence_after();
                const uint32_t left = a_lo0 + (uint32_t)(s * (Cfg::STAGE_BYTES / 16)), right = a_lo0 + (uint32_t)(s1 * (Cfg::STAGE_BYTES / 16));
                const uint32_t d = tmem_base + (uint32_t)(b * 256);
#pragma unroll
                for (int i = 0; i < 12; ++i) {                    // block (kh, rx) of the weights
                    const int kh = i >> 2, rx = i & 3;
                    const uint32_t al = (rx < 2 ? left : right) + (uint32_t)(kh * 2 + (rx & 1)) * pixel_u, bl = w_lo0 + (uint32_t)(i * (Cfg::W_BLOCK_BYTES >> 4));
#pragma unroll
                    for (int dy = 0; dy < 2; ++dy)
                        ptx::mma_i8_if(leader, d + (uint32_t)(dy * 128), al + (uint32_t)(dy * 2) * pixel_u, hi, bl, hi, ptx::idesc_i8(128, 128, true, true), i > 0 ? 1u : 0u);
                }
                ptx::mma_commit_if(leader, empty(s));
                if (px == a.wins - 1) ptx::mma_commit_if(leader, empty(s1));
                ptx::mma_commit_if(leader, tfull(b));
                s = s1; ph = ph1;
            }
            if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }          // the next item starts behind the last pair
        }
    } else {
        // ------------------------------------------------------------------ epilogue: 16 warps, four per TMEM lane
        // quarter; each takes 16 of the 64 filters of its quarter's 32 images, in every tile (a single warp per
        // quarter and tile would be latency-bound and slower than the MMAs of the next tile).
        const int quarter = warp & 3;               // TMEM lane quarter this warp may access
        const int cg = (warp - 2) >> 2;             // 16-filter group of this warp
        const int row = quarter * 32 + lane;        // MMA row = image within the block
        float mult[16], flr[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) { mult[j] = a.mult[cg * 16 + j]; flr[j] = a.bias[cg * 16 + j]; }
        int it = 0;
        bool alive = true;
        for (int item = blockIdx.x; item < a.items && alive; item += gridDim.x) {
            const int win = item * a.wins, nb = win / 25;
            const bool live = nb * 128 + row < a.n_images;
            int8_t* yw = a.y + ((size_t)nb * 100 + (win - nb * 25) * 4 + cg) * (size_t)(a.ib * 16) + (size_t)row * 16;
            for (int px = 0; px < a.wins; ++px, ++it, yw += 4 * a.ib * 16) {
                const int b = it & 1;
                int ok = 1;
                if (lane == 0) ok = ptx::mbar_wait(tfull(b), (uint32_t)(it >> 1) & 1u, abort_flag) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) { alive = false; break; }
                ptx::tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 256 + cg * 16);
                uint32_t v[4][16];
#pragma unroll
                for (int m = 0; m < 4; ++m) ptx::tmem_ld16(taddr + (uint32_t)(m * 64), v[m]);
                ptx::tmem_wait_ld();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(tempty(b));   // this warp has its values: the set may be overwritten once all 16 arrived
                uint32_t pk[4];
#pragma unroll
                for (int j4 = 0; j4 < 4; ++j4) {
                    int r[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c = j4 * 4 + j;
                        const int mx = max(__vimax3_s32((int)v[0][c], (int)v[1][c], (int)v[2][c]), (int)v[3][c]);
                        // bias and ReLU (kAccBase: one instruction, and a subtraction gives the float)
                        const float f = BASE ? __fsub_rn(__int_as_float(__viaddmax_s32(mx, kAccBaseBits, __float_as_int(flr[c]))), flr[c])
                                             : __int2float_rn(max(mx + __float_as_int(flr[c]), 0));
                        r[j] = __float2int_rn(__fmul_rn(f, mult[c]));
                    }
                    pk[j4] = pack_sat_s8x4(r[0], r[1], r[2], r[3]);
                }
                if (live) *reinterpret_cast<uint4*>(yw) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
        }
    }

    // ---------------------------------------------------------------------- teardown
    if (*abort_flag) {
        // give copies and MMAs that are still in flight time to land before the CTA's memory goes away
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) ptx::tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    if (tid == 0 && *abort_flag) atomicExch(a.status, (int)DEV_ERR_WAIT_TIMEOUT);
}

}  // namespace zb
