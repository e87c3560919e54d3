// Device-level operator launchers: resolved geometry + device pointers -> kernel launches on
// the context's stream.  Shared by the single-operator C entry points and by the plan.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>
#include "context.cuh"
#include "geometry.hpp"
#include "contract_f32.cuh"
#include "kernels_f32.cuh"
#include "kernels_q8.cuh"

namespace zb {

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---------------------------------------------------------------------------- fp32
// What a fused step applies to a contraction's finished sums.
struct ContractFusion { int act = CT_ACT_NONE; float slope = 0.0f; const float* bias = nullptr; bool pool = false; };

// Up to three tiles per SM: so much shared memory that no SM takes more than its share.  A grid that starts while its predecessor
// drains would otherwise pile up on the SMs that are free first (128 tiles, two to an SM: 290 -> 540 us).
inline size_t contract_share(zant_ctx* ctx, const dim3& grid, size_t smem) {
    const long long share = ((long long)grid.x * grid.y + ctx->sm_count - 1) / ctx->sm_count;
    return std::max<size_t>(smem, share == 1 ? 122880 : (share == 2 ? 81920 : (share == 3 ? 61440 : 0)));
}

template <bool CONV, bool POOL, int BM, int BN, int TM, int TN>
inline int32_t launch_contract_tile(zant_ctx* ctx, const ContractArgs& p) {
    ZB_SMEM_ATTR(ctx, (contract_f32_tile<CONV, POOL, BM, BN, TM, TN>), 122880);
    const dim3 grid(((unsigned)p.M + BM - 1) / BM, ((unsigned)p.N + BN - 1) / BN);
    const size_t smem = contract_share(ctx, grid, contract_smem<BM, BN>());
    launch(ctx, contract_f32_tile<CONV, POOL, BM, BN, TM, TN>, grid, (BM / TM) * (BN / TN), smem, p);
    return check_launch(ctx, "contract_f32_tile");
}

// Tile by time: what n tiles of a shape cost an SM for each k, in ns, and 25 k's worth per tile for its results.  Up to three tiles get an SM's
// shared memory in equal shares and overlap (lone + n * per); more queue (base + n * slope).  The numbers are medians over 220 convolutions, as
// calls and as plans (whose weights are in slab order), and 200 products of 5 us to 2 ms with every shape forced: the choice is 1.5 % slower
// than the best shape in the mean.  By waves and the rate of a full SM alone, which knows no latency, it was 4 to 15 %, and up to 20 %
// slower than 64 x 64 tiles where a few narrow tiles met a long k (convolution 2312 x 155 x 800: 115 us there, 125, now 75).
struct ContractTime { double lone, per, base, slope; };
inline double contract_cost(const ContractTime& t, double tiles_per_sm, double k) {
    const double ns = tiles_per_sm <= 3.0 ? t.lone + t.per * tiles_per_sm : t.base + t.slope * tiles_per_sm;
    return ns * k + 25.0 * t.slope * tiles_per_sm;
}
// A first layer with its pool in contract_f32.cuh's kernel for it: at any size (1 image of 28 x 28 6.3 -> 4.2 us).  All filters in a thread, or as few as
// it takes for three CTAs an SM (256 images: 32 filters a thread 10.4 us, 16 8.3; 16 images: 32 6.3, 8 4.4).
inline bool conv_lowc_takes(const ContractArgs& p) {
    const ConvGeom& g = p.g;
    return g.KH == 3 && g.KW == 3 && g.sh == 1 && g.sw == 1 && g.dh == 1 && g.dw == 1 && g.C <= 3 && p.N <= kLowCMaxFilters && (long long)g.C * g.H * g.W < 0x7fffffffLL;
}
inline int32_t launch_conv_lowc(zant_ctx* ctx, const ContractArgs& p) {
    const unsigned gx = ((unsigned)(p.M / 4) + kLowCThreads - 1) / kLowCThreads;
    int per = (p.N + 7) / 8 * 8;
    while (per > 8 && (long long)gx * ((p.N + per - 1) / per) < 3LL * ctx->sm_count) per = (per / 2 + 7) / 8 * 8;
    const dim3 grid(gx, (unsigned)((p.N + per - 1) / per));
    const size_t smem = (size_t)(p.g.C * 9 + 1) * per * 4;
    switch (p.g.C) {
        case 1: launch(ctx, conv3x3_pool_f32_lowc<1>, grid, kLowCThreads, smem, p, per); break;
        case 2: launch(ctx, conv3x3_pool_f32_lowc<2>, grid, kLowCThreads, smem, p, per); break;
        default: launch(ctx, conv3x3_pool_f32_lowc<3>, grid, kLowCThreads, smem, p, per); break;
    }
    return check_launch(ctx, "conv3x3_pool_f32_lowc");
}

template <bool CONV, bool POOL>
inline int32_t launch_contract(zant_ctx* ctx, ContractArgs& p) {
    p.neg_zero = 0x8000000080000000ull;
    if constexpr (CONV && POOL) if (conv_lowc_takes(p)) return launch_conv_lowc(ctx, p);
    static const int shapes[6][2] = {{128, 128}, {128, 64}, {128, 32}, {128, 16}, {32, 32}, {CF_BM, CF_BN}};
    static const ContractTime times[3][6] = {
        {{0, 204, 50, 195}, {45, 87, 40, 92}, {95, 36, 130, 46}, {72, 23, 90, 31}, {52, 9, 55, 17.5}, {0, 33, 30, 26}},        // B runs along k (a convolution's weights as the tensor has them, a transposed matrix)
        {{0, 186, 30, 180}, {32, 81, 30, 83}, {78, 35, 115, 42}, {62, 23, 85, 28.5}, {38, 8, 45, 14.5}, {0, 14.5, 12, 10.2}},  // convolution, weights in slab order
        {{0, 167, 0, 165}, {12, 83, 10, 83}, {22, 48, 25, 49}, {55, 16.5, 65, 32}, {19, 9, 42, 11}, {1, 9, 12, 8}},            // product with B in rows
    };
    const ContractTime* t = times[!p.b_vec && p.sbk == 1 ? 0 : (CONV ? 1 : 2)];
    int best = -1; double cost = 1e300;
    for (int i = 0; i < 6; ++i) {
        const double row_tiles = std::ceil((double)p.M / shapes[i][0]), col_tiles = std::ceil((double)p.N / shapes[i][1]);
        if (col_tiles > 65535.0 || row_tiles * shapes[i][0] > 2147483648.0) continue;        // (grid.y; a tile's rows are ints)
        const double c = contract_cost(t[i], std::ceil(row_tiles * col_tiles / ctx->sm_count), p.K);
        if (c < cost) { cost = c; best = i; }
    }
    if (best < 0) return fail(ZANT_E_TOO_LARGE, "too many output columns");
    switch (best) {
        case 0: return launch_contract_tile<CONV, POOL, 128, 128, 8, 8>(ctx, p);
        case 1: return launch_contract_tile<CONV, POOL, 128, 64, 8, 4>(ctx, p);
        case 2: return launch_contract_tile<CONV, POOL, 128, 32, 8, 4>(ctx, p);
        case 3: return launch_contract_tile<CONV, POOL, 128, 16, 4, 4>(ctx, p);
        case 4: return launch_contract_tile<CONV, POOL, 32, 32, 4, 2>(ctx, p);
        default: break;
    }
    ZB_SMEM_ATTR(ctx, (contract_f32_few<CONV, POOL>), 122880);
    const dim3 grid(((unsigned)p.M + CF_BM - 1) / CF_BM, ((unsigned)p.N + CF_BN - 1) / CF_BN);
    launch(ctx, contract_f32_few<CONV, POOL>, grid, 256, contract_share(ctx, grid, contract_few_smem()), p);
    return check_launch(ctx, "contract_f32_few");
}

inline int32_t run_transpose_pad_f32(zant_ctx* ctx, const float* w, float* wt, int M, int K, int N4) {
    const dim3 grid((unsigned)((N4 + 31) / 32), (unsigned)((K + 31) / 32));
    if (grid.y > 65535) return fail(ZANT_E_TOO_LARGE, "too many taps");
    launch(ctx, transpose_pad_f32, grid, 256, 0, w, wt, M, K, N4);
    return check_launch(ctx, "transpose_pad_f32");
}

// `w_kn`: the weights as [K][N rounded up to 4] (a plan transposes them once), else null and `w` is [M][C][KH][KW].
inline int32_t run_conv_f32(zant_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y,
                            const ContractFusion& fu = ContractFusion{}, const float* w_kn = nullptr) {
    ContractArgs p{};
    p.a = x; p.b = w; p.d = y; p.bias = bias; p.g = g; p.act = fu.act; p.slope = fu.slope;
    p.PH = g.OH / 2; p.PW = g.OW / 2;
    const long long M = (long long)g.N * (fu.pool ? 4LL * p.PH * p.PW : (long long)g.OH * g.OW);
    if (M > 0x7fffffffLL) return fail(ZANT_E_TOO_LARGE, "Conv output pixels exceed int range");
    p.M = (int)M; p.N = g.M; p.K = g.C * g.KH * g.KW;
    p.padded = g.pt > 0 || g.pl > 0 || (g.OH - 1) * g.sh - g.pt + (g.KH - 1) * g.dh >= g.H || (g.OW - 1) * g.sw - g.pl + (g.KW - 1) * g.dw >= g.W;
    p.y_vec = (g.OH * g.OW) % 4 == 0 && aligned16(y);
    if (w_kn) { p.b = w_kn; p.sbk = (g.M + 3) / 4 * 4; p.sbj = 1; p.b_vec = 1; }
    else { p.sbk = 1; p.sbj = p.K; }
    return fu.pool ? launch_contract<true, true>(ctx, p) : launch_contract<true, false>(ctx, p);
}

inline int32_t run_contract_f32(zant_ctx* ctx, ContractArgs& p) {
    p.a_vec = p.sak == 1 && p.sam % 4 == 0 && p.K % 4 == 0 && aligned16(p.a);
    p.b_vec = p.sbj == 1 && p.sbk % 4 == 0 && p.N % 4 == 0 && aligned16(p.b);
    return launch_contract<false, false>(ctx, p);
}

inline int32_t run_matmul_f32(zant_ctx* ctx, const MatGeom& g, const float* a, const float* b, float* y, const ContractFusion& fu = ContractFusion{}) {
    if (g.M > 0x7fffffffULL || g.N > 0x7fffffffULL || g.K > 0x7fffffffULL) return fail(ZANT_E_TOO_LARGE, "MatMul dims exceed int range");
    ContractArgs p{};
    p.a = a; p.b = b; p.d = y; p.M = (int)g.M; p.N = (int)g.N; p.K = (int)g.K;
    p.sam = (long long)g.K; p.sak = 1; p.sbk = (long long)g.N; p.sbj = 1;
    p.bias = fu.bias; p.act = fu.act; p.slope = fu.slope;
    return run_contract_f32(ctx, p);
}

inline int32_t run_gemm_f32(zant_ctx* ctx, const GemmGeom& g, const float* a, const float* b, const float* c,
                            float alpha, float beta, bool ta, bool tb, float* y) {
    if (g.rows > 0x7fffffffULL || g.cols > 0x7fffffffULL || g.K > 0x7fffffffULL) return fail(ZANT_E_TOO_LARGE, "Gemm dims exceed int range");
    ContractArgs p{};
    p.a = a; p.b = b; p.d = y; p.M = (int)g.rows; p.N = (int)g.cols; p.K = (int)g.K;
    // A' = A^T when transA: A is [K, rows] row-major; B' = B^T when transB: B is [cols, K].
    p.sam = ta ? 1 : (long long)g.K; p.sak = ta ? (long long)g.rows : 1;
    p.sbk = tb ? 1 : (long long)g.cols; p.sbj = tb ? (long long)g.K : 1;
    p.gemm = 1; p.alpha = alpha; p.beta = beta; p.c = c; p.c_mode = g.c_mode;
    if (g.c_mode == 1) { p.c_rs = (long long)g.cols; p.c_cs = 1; }
    else if (g.c_mode == 2) { p.c_rs = g.c_rows == 1 ? 0 : (long long)g.c_cols; p.c_cs = g.c_cols == 1 ? 0 : 1; }
    int32_t st = run_contract_f32(ctx, p);
    if (st != ZANT_OK) return st;
    const size_t first = g.rows * g.cols, total = g.batch * first;
    if (total > first) {
        launch(ctx, gemm_tail_f32, grid_for(total - first, 256, ctx->sm_count), 256, 0, 
            y, first, total, alpha, c, g.c_mode, beta, g.rows, g.cols, g.c_rows, g.c_cols, 0, g.c_ch);
        st = check_launch(ctx, "gemm_tail_f32");
    }
    return st;
}

template <typename T>
inline int32_t run_maxpool(zant_ctx* ctx, const PoolGeom& g, const T* x, T* y) {
    const size_t total = (size_t)g.NC * g.OH * g.OW;
    if (total == 0) return ZANT_OK;
    if constexpr (sizeof(T) == 1) {
        const bool fast = g.KH == 2 && g.KW == 2 && g.sh == 2 && g.sw == 2 && g.dh == 1 && g.dw == 1 && g.pt == 0 && g.pl == 0 &&
                          g.W % 8 == 0 && g.H == 2 * g.OH && g.W == 2 * g.OW &&
                          (reinterpret_cast<uintptr_t>(x) & 7u) == 0 && (reinterpret_cast<uintptr_t>(y) & 3u) == 0;
        if (fast) {
            const size_t words = total / 4;
            const int grid = grid_for(words, 256, ctx->sm_count, 16);
            if (std::is_signed<T>::value)
                launch(ctx, maxpool2x2s2_q8<true>, grid, 256, 0, (const uint2*)x, (uint32_t*)y, (size_t)g.NC * g.OH, g.OW / 4, g.W / 8);
            else
                launch(ctx, maxpool2x2s2_q8<false>, grid, 256, 0, (const uint2*)x, (uint32_t*)y, (size_t)g.NC * g.OH, g.OW / 4, g.W / 8);
            return check_launch(ctx, "maxpool2x2s2_q8");
        }
    }
    if constexpr (std::is_same<T, float>::value) {
        const bool fast = g.KH == 2 && g.KW == 2 && g.sh == 2 && g.sw == 2 && g.dh == 1 && g.dw == 1 && g.pt == 0 && g.pl == 0 &&
                          g.W % 4 == 0 && g.H == 2 * g.OH && g.W == 2 * g.OW &&
                          (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(y) & 7u) == 0;
        if (fast) {
            const size_t pairs = total / 2;
            launch(ctx, maxpool2x2s2_f32, grid_for(pairs, 256, ctx->sm_count, 16), 256, 0, (const float4*)x, (float2*)y, (size_t)g.NC * g.OH, g.OW / 2, g.W / 4);
            return check_launch(ctx, "maxpool2x2s2_f32");
        }
    }
    launch(ctx, maxpool_nchw<T>, grid_for(total, 256, ctx->sm_count), 256, 0, x, y, g);
    return check_launch(ctx, "maxpool_nchw");
}

template <typename F>
inline int32_t run_unary_f32(zant_ctx* ctx, const float* x, float* y, size_t n, F f, const char* name) {
    if (n == 0) return ZANT_OK;
    const bool vec = aligned16(x) && aligned16(y);
    launch(ctx, unary_f32<F>, grid_for(vec ? (n + 3) / 4 : n, 256, ctx->sm_count), 256, 0, x, y, n, vec, f);
    return check_launch(ctx, name);
}

inline int32_t run_binary_same_f32(zant_ctx* ctx, const float* a, const float* b, float* y, size_t n, bool divide) {
    if (n == 0) return ZANT_OK;
    const int grid = grid_for(n, 256, ctx->sm_count);
    if (divide) launch(ctx, binary_same_f32<true>, grid, 256, 0, a, b, y, n);
    else launch(ctx, binary_same_f32<false>, grid, 256, 0, a, b, y, n);
    return check_launch(ctx, divide ? "div_f32" : "mul_f32");
}

inline int32_t run_softmax_f32(zant_ctx* ctx, const float* x, float* y, size_t rows, size_t cols) {
    if (rows == 0 || cols == 0) return ZANT_OK;
    launch(ctx, softmax_rows_f32, grid_for(rows, 128, ctx->sm_count), 128, 0, x, y, rows, cols);
    return check_launch(ctx, "softmax_rows_f32");
}

inline int32_t run_add_f32(zant_ctx* ctx, const BcastGeom& g, const float* a, const float* b, float* y) {
    if (g.total == 0) return ZANT_OK;
    if (g.same_size) {
        const bool vec = aligned16(a) && aligned16(b) && aligned16(y);
        launch(ctx, add_same_f32, grid_for(vec ? (g.total + 3) / 4 : g.total, 256, ctx->sm_count), 256, 0, a, b, y, g.total, vec);
        return check_launch(ctx, "add_same_f32");
    }
    BcastArgs k{};
    k.rank = g.rank; k.total = g.total;
    for (int d = 0; d < g.rank; ++d) { k.out_shape[d] = g.out_shape[d]; k.a_stride[d] = g.a_stride[d]; k.b_stride[d] = g.b_stride[d]; }
    launch(ctx, add_bcast_f32, grid_for(g.total, 256, ctx->sm_count), 256, 0, a, b, y, k);
    return check_launch(ctx, "add_bcast_f32");
}

inline int32_t run_sum_list_f32(zant_ctx* ctx, const float* const* ts, size_t nt, float* y, size_t n) {
    if (n == 0) return ZANT_OK;
    size_t done = 0;
    while (done < nt) {
        SumListArgs l{};
        l.n = (int)std::min<size_t>(8, nt - done);
        for (int i = 0; i < l.n; ++i) l.t[i] = ts[done + i];
        launch(ctx, sum_list_f32, grid_for(n, 256, ctx->sm_count), 256, 0, l, y, n, done != 0);
        int32_t st = check_launch(ctx, "sum_list_f32");
        if (st != ZANT_OK) return st;
        done += l.n;
    }
    return ZANT_OK;
}

inline int32_t run_copy2d(zant_ctx* ctx, const void* src, size_t sp, void* dst, size_t dp, size_t row_bytes, size_t rows) {
    if (row_bytes == 0 || rows == 0) return ZANT_OK;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) | sp | dp | row_bytes;
    const char* s = static_cast<const char*>(src);
    char* d = static_cast<char*>(dst);
    if ((bits & 15) == 0) {
        launch(ctx, copy2d<uint4>, grid_for(row_bytes / 16 * rows, 256, ctx->sm_count), 256, 0, s, sp, d, dp, row_bytes / 16, rows);
    } else if ((bits & 3) == 0) {
        launch(ctx, copy2d<uint32_t>, grid_for(row_bytes / 4 * rows, 256, ctx->sm_count), 256, 0, s, sp, d, dp, row_bytes / 4, rows);
    } else {
        launch(ctx, copy2d<uint8_t>, grid_for(row_bytes * rows, 256, ctx->sm_count), 256, 0, s, sp, d, dp, row_bytes, rows);
    }
    return check_launch(ctx, "copy2d");
}

// One strided copy per input tensor: slice s of tensor t lands at out[s*out_row + off_t].
inline int32_t run_concat(zant_ctx* ctx, const ConcatGeom& g, size_t esz, const void* const* ts, void* y) {
    const size_t out_row = g.out_axis_dim * g.slice * esz;
    size_t off = 0;
    for (size_t t = 0; t < g.axis_dim.size(); ++t) {
        const size_t row = g.axis_dim[t] * g.slice * esz;
        int32_t st = run_copy2d(ctx, ts[t], row, static_cast<char*>(y) + off, out_row, row, g.num_slices);
        if (st != ZANT_OK) return st;
        off += row;
    }
    return ZANT_OK;
}

inline int32_t run_resize(zant_ctx* ctx, size_t esz, const void* x, void* y, const int32_t* table_dev,
                          const size_t* xs, const size_t* os, size_t r, const std::vector<int32_t>& axis_offset) {
    ResizeArgs k{};
    k.rank = (int)r; k.total = 1;
    size_t s = 1;
    for (size_t d = r; d-- > 0;) { k.in_stride[d] = s; s *= xs[d]; k.out_shape[d] = os[d]; k.total *= os[d]; k.axis_offset[d] = axis_offset[d]; }
    if (k.total == 0) return ZANT_OK;
    const int grid = grid_for(k.total, 256, ctx->sm_count);
    const bool small = k.total < 0x7fffffffull && s < 0x7fffffffull;      // s: elements of the input
    if (esz == 4) {
        if (small) launch(ctx, resize_gather<uint32_t, uint32_t>, grid, 256, 0, (const uint32_t*)x, (uint32_t*)y, table_dev, k);
        else launch(ctx, resize_gather<uint32_t, size_t>, grid, 256, 0, (const uint32_t*)x, (uint32_t*)y, table_dev, k);
    } else {
        if (small) launch(ctx, resize_gather<uint8_t, uint32_t>, grid, 256, 0, (const uint8_t*)x, (uint8_t*)y, table_dev, k);
        else launch(ctx, resize_gather<uint8_t, size_t>, grid, 256, 0, (const uint8_t*)x, (uint8_t*)y, table_dev, k);
    }
    return check_launch(ctx, "resize_gather");
}

inline int32_t run_reduce_mean_f32(zant_ctx* ctx, const ReduceGeom& g, const float* x, float* y) {
    if (g.mode == 0) {
        ZB_CUDA(cudaMemcpyAsync(y, x, g.total * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
        return ZANT_OK;
    }
    if (g.mode == 1) {
        launch(ctx, reduce_all_mean_f32, 1, 32, 0, x, y, g.total);
        return check_launch(ctx, "reduce_all_mean_f32");
    }
    ReduceArgs k{};
    k.out_total = g.out_total; k.count = g.count; k.n_keep = g.n_keep; k.n_red = g.n_red;
    for (int i = 0; i < 8; ++i) { k.keep_ostride[i] = g.keep_ostride[i]; k.keep_istride[i] = g.keep_istride[i]; k.red_size[i] = g.red_size[i]; k.red_istride[i] = g.red_istride[i]; }
    if (g.out_total == 0) return ZANT_OK;
    launch(ctx, reduce_mean_f32, grid_for(g.out_total, 128, ctx->sm_count), 128, 0, x, y, k);
    return check_launch(ctx, "reduce_mean_f32");
}

// ---------------------------------------------------------------------------- quantized
inline int32_t run_quantize(zant_ctx* ctx, const float* x, void* y, size_t n, float scale, int zp, int32_t out_dtype) {
    if (n == 0) return ZANT_OK;
    const bool vec = aligned16(x) && ((reinterpret_cast<uintptr_t>(y) & 3) == 0);
    const int grid = grid_for(vec ? (n + 3) / 4 : n, 256, ctx->sm_count);
    if (out_dtype == ZANT_U8) launch(ctx, quantize_linear_k<true>, grid, 256, 0, x, y, n, scale, zp, vec);
    else launch(ctx, quantize_linear_k<false>, grid, 256, 0, x, y, n, scale, zp, vec);
    return check_launch(ctx, "quantize_linear_k");
}

inline int32_t run_dequantize(zant_ctx* ctx, int32_t in_dtype, const void* q, float* y, size_t n, float scale, int zp) {
    if (n == 0) return ZANT_OK;
    const int grid = grid_for(n, 256, ctx->sm_count);
    if (in_dtype == ZANT_U8) launch(ctx, dequantize_linear_k<uint8_t>, grid, 256, 0, (const uint8_t*)q, y, n, scale, zp);
    else if (in_dtype == ZANT_I8) launch(ctx, dequantize_linear_k<int8_t>, grid, 256, 0, (const int8_t*)q, y, n, scale, zp);
    else launch(ctx, dequantize_linear_k<int32_t>, grid, 256, 0, (const int32_t*)q, y, n, scale, zp);
    return check_launch(ctx, "dequantize_linear_k");
}

inline int32_t run_qconv_generic(zant_ctx* ctx, const QConvArgs& p, int32_t x_dtype, int32_t y_dtype) {
    const size_t total = (size_t)p.g.N * p.g.M * p.g.OH * p.g.OW;
    if (total == 0) return ZANT_OK;
    const int grid = grid_for(total, 128, ctx->sm_count, 32);
    const bool xu = x_dtype == ZANT_U8, yu = y_dtype == ZANT_U8;
    if (xu && yu) launch(ctx, qconv_nchw_generic<true, true>, grid, 128, 0, p);
    else if (xu) launch(ctx, qconv_nchw_generic<true, false>, grid, 128, 0, p);
    else if (yu) launch(ctx, qconv_nchw_generic<false, true>, grid, 128, 0, p);
    else launch(ctx, qconv_nchw_generic<false, false>, grid, 128, 0, p);
    return check_launch(ctx, "qconv_nchw_generic");
}

inline int32_t run_qmatmul_generic(zant_ctx* ctx, const QMatArgs& p, int32_t a_dtype, int32_t y_dtype) {
    const size_t total = (size_t)p.M * p.N;
    if (total == 0) return ZANT_OK;
    const int grid = grid_for(total, 128, ctx->sm_count, 32);
    const bool au = a_dtype == ZANT_U8, yu = y_dtype == ZANT_U8;
    if (au && yu) launch(ctx, qmatmul_generic<true, true>, grid, 128, 0, p);
    else if (au) launch(ctx, qmatmul_generic<true, false>, grid, 128, 0, p);
    else if (yu) launch(ctx, qmatmul_generic<false, true>, grid, 128, 0, p);
    else launch(ctx, qmatmul_generic<false, false>, grid, 128, 0, p);
    return check_launch(ctx, "qmatmul_generic");
}

inline int32_t run_qadd(zant_ctx* ctx, int32_t dtype, const void* a, float a_s, int a_zp, const void* b, float b_s, int b_zp,
                        float y_s, int y_zp, int act, void* y, size_t n) {
    if (n == 0) return ZANT_OK;
    const bool u8 = dtype == ZANT_U8;
    const bool zp_ok = u8 ? (y_zp >= 0 && y_zp <= 255) : (y_zp >= -128 && y_zp <= 127);
    size_t done = 0;
    if (zp_ok && n >= 16 && aligned16(a) && aligned16(b) && aligned16(y)) {
        const size_t n16 = n / 16;
        const int grid = grid_for(n16, 256, ctx->sm_count);
        if (u8) launch(ctx, qadd_vec_k<true>, grid, 256, 0, (const uint4*)a, (const uint4*)b, (uint4*)y, n16, qadd_tail<true>(a_s, a_zp, b_s, b_zp, y_s, y_zp, act));
        else launch(ctx, qadd_vec_k<false>, grid, 256, 0, (const uint4*)a, (const uint4*)b, (uint4*)y, n16, qadd_tail<false>(a_s, a_zp, b_s, b_zp, y_s, y_zp, act));
        ZB_TRY(check_launch(ctx, "qadd_vec_k"));
        done = n16 * 16;
        if (done == n) return ZANT_OK;
    }
    const char* pa = (const char*)a + done; const char* pb = (const char*)b + done; char* py = (char*)y + done;
    const size_t rest = n - done;
    const int grid = grid_for(rest, 256, ctx->sm_count);
    if (u8) launch(ctx, qadd_k<true>, grid, 256, 0, pa, a_s, a_zp, pb, b_s, b_zp, y_s, y_zp, act, py, rest);
    else launch(ctx, qadd_k<false>, grid, 256, 0, pa, a_s, a_zp, pb, b_s, b_zp, y_s, y_zp, act, py, rest);
    return check_launch(ctx, "qadd_k");
}

inline int32_t run_qgap(zant_ctx* ctx, int32_t dtype, const void* x, void* y, size_t planes, int hw,
                        float x_s, int x_zp, float y_s, int y_zp) {
    if (planes == 0) return ZANT_OK;
    if (hw <= 256 && planes >= 4096 && (reinterpret_cast<uintptr_t>(x) & 3u) == 0) {
        // many small planes: a thread per plane
        const int grid = grid_for(planes, 128, ctx->sm_count);
        if (dtype == ZANT_U8) launch(ctx, qgap_small_k<true>, grid, 128, 0, (const uint8_t*)x, y, planes, hw, x_s, x_zp, y_s, y_zp);
        else launch(ctx, qgap_small_k<false>, grid, 128, 0, (const uint8_t*)x, y, planes, hw, x_s, x_zp, y_s, y_zp);
        return check_launch(ctx, "qgap_small_k");
    }
    const int grid = grid_for(planes * 32, 256, ctx->sm_count);
    if (dtype == ZANT_U8) launch(ctx, qgap_k<true>, grid, 256, 0, x, y, planes, hw, x_s, x_zp, y_s, y_zp);
    else launch(ctx, qgap_k<false>, grid, 256, 0, x, y, planes, hw, x_s, x_zp, y_s, y_zp);
    return check_launch(ctx, "qgap_k");
}

inline int32_t run_lut(zant_ctx* ctx, const void* x, void* y, size_t n, const uint8_t* lut_dev) {
    if (n == 0) return ZANT_OK;
    const bool vec = aligned16(x) && aligned16(y);
    launch(ctx, lut_q8_k, grid_for(vec ? (n + 15) / 16 : n, 256, ctx->sm_count), 256, 0, (const uint8_t*)x, (uint8_t*)y, n, lut_dev, vec);
    return check_launch(ctx, "lut_q8_k");
}

// Per-output-channel requantisation multipliers M[m] = (x_scale * w_scale[m]) / y_scale:
// one fp32 multiply then one fp32 divide, computed on the host once.
inline void requant_multipliers(float x_scale, const float* w_scale, size_t nws, float y_scale, size_t M, std::vector<float>& out) {
    out.resize(M);
    for (size_t m = 0; m < M; ++m) {
        volatile float xw = x_scale * w_scale[nws == 1 ? 0 : m];
        out[m] = xw / y_scale;
    }
}

inline int32_t run_strided_copy(zant_ctx* ctx, size_t esz, const void* x, void* y, const StridedMap& m) {
    if (m.total == 0) return ZANT_OK;
    StridedMapDev d{};
    d.rank = m.rank; d.base = m.base; d.total = m.total;
    for (int i = 0; i < 8; ++i) { d.out_dims[i] = m.out_dims[i]; d.in_stride[i] = m.in_stride[i]; }
    const int grid = grid_for(m.total, 256, ctx->sm_count);
    if (esz == 4) launch(ctx, strided_copy_k<uint32_t>, grid, 256, 0, (const uint32_t*)x, (uint32_t*)y, d);
    else launch(ctx, strided_copy_k<uint8_t>, grid, 256, 0, (const uint8_t*)x, (uint8_t*)y, d);
    return check_launch(ctx, "strided_copy_k");
}

inline int32_t run_gather(zant_ctx* ctx, size_t esz, const void* x, const int32_t* idx_dev, void* y, const GatherGeom& g) {
    const size_t total = g.outer * g.n_idx * g.inner;
    if (total == 0) return ZANT_OK;
    const int grid = grid_for(total, 256, ctx->sm_count);
    if (esz == 4) launch(ctx, gather_axis_k<uint32_t>, grid, 256, 0, (const uint32_t*)x, idx_dev, (uint32_t*)y, g.outer, g.n_idx, g.inner, g.axis_dim);
    else launch(ctx, gather_axis_k<uint8_t>, grid, 256, 0, (const uint8_t*)x, idx_dev, (uint8_t*)y, g.outer, g.n_idx, g.inner, g.axis_dim);
    return check_launch(ctx, "gather_axis_k");
}

}  // namespace zb
