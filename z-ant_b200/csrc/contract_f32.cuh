// FP32 contractions with the reference's arithmetic: every dot product is accumulated by ONE thread in ascending k with a
// separately rounded multiply and add, so results are bit-identical to the reference's CPU loops
// (op_convolution.zig:316-328, op_mat_mul.zig:92-172, op_gemm.zig:128-178).
//
//   D[m,j] = sum_k A(m,k) * B(k,j)
//   CONV = true : A is gathered on the fly from an NCHW input (implicit im2col, k = (c,kh,kw) exactly as lean_im2col orders
//                 it), D scattered to NCHW with the bias added after the sum, then the activation, then (POOL) a 2x2 / 2 maximum.
//   CONV = false: A(m,k) = a[m*sam + k*sak] (MatMul, the transposed operands of Gemm), then  v*alpha  and  + c*beta  as two
//                 separately rounded steps, or the bias row of an Add behind the product and a Relu behind that.
//   B(k,j) = b[k*sbk + j*sbj].
//
// What bounds it: without fused multiply-adds a MAC is two FP32 operations, 64 a clock and SM.  Packed pairs
// (fma / add.rn.f32x2: two exactly rounded operations per instruction) halve the issue slots, so that address arithmetic and
// shared-memory loads fit beside the math; a thread keeps 8 x 8 (8 x 4, ...) sums in registers, slabs of 16 k arrive by
// cp.async three deep, out-of-image taps as zero fills.  The (c,kh,kw) of a slab's k is worked out by 16 threads one slab
// ahead instead of once per element.
// Few outputs (contract_f32_few): one output per thread, the k-ascending chain of additions is the floor (about 4 clocks a
// step), so slabs of 64 k, four deep, keep it fed: MatMul 1 x 1600 x 512 took 88 us on 64 x 64 tiles.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "geometry.hpp"
#include "ptx_sm100.cuh"

namespace zb {

enum { CT_ACT_NONE = 0, CT_ACT_RELU = 1, CT_ACT_LEAKY = 2 };

struct ContractArgs {
    const float* a; const float* b; float* d;
    int M, N, K;
    long long sam, sak, sbk, sbj;     // plain-matrix strides (elements); sbk, sbj also for a convolution's weights
    int a_vec, b_vec;                 // rows of A / B are whole, aligned 16-byte units along k / j
    ConvGeom g;
    int padded;                       // some tap of some output lies outside the image
    int PH, PW;                       // POOL: pooled output; rows are (image, pooled pixel, window member)
    int y_vec;                        // CONV: output planes are whole, aligned 16-byte units
    const float* bias;                // per column, nullable
    int act; float slope;
    int gemm;                         // matrix form: alpha, optional C
    float alpha, beta;
    const float* c; int c_mode; long long c_rs, c_cs;   // c index = m*c_rs + j*c_cs
    uint64_t neg_zero;                // two times -0.0f: see ct::mul2
};

namespace ct {

__device__ __forceinline__ void cp4(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two products, two sums, each rounded on its own.  The assembler contracts mul.rn.f32x2 + add.rn.f32x2 into one fused operation
// (measured: the pair returns the fused result), so the product is a fused multiply-add of -0 that it cannot see through:
// `neg_zero` comes in as a kernel argument.  a * b + (-0) is the rounded product, signed zeros included.
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t neg_zero) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg_zero)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t dup2(float v) { uint64_t r; asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v)); return r; }
__device__ __forceinline__ void split2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

__device__ __forceinline__ float activate(float v, int act, float slope) {
    if (act == CT_ACT_RELU) return v > 0.0f ? v : 0.0f;
    if (act == CT_ACT_LEAKY) return v <= 0.0f ? __fmul_rn(slope, v) : v;
    return v;
}

// offset of k in the input and its tap displacement; k >= K: a tap that is outside every image
struct __align__(16) Tap { long long off; int dy, dx; };
__device__ __forceinline__ Tap tap_of(const ContractArgs& p, int k) {
    const ConvGeom& g = p.g;
    if (k >= p.K) return Tap{0, 0x7fffffff, 0};
    const int khw = g.KH * g.KW, c = k / khw, r = k - c * khw, kh = r / g.KW, kw = r - kh * g.KW;
    const int dy = kh * g.dh, dx = kw * g.dw;
    return Tap{((long long)c * g.H + dy) * g.W + dx, dy, dx};
}

// origin of a row's window: element offset of tap (0,0) of channel 0, and its image coordinates
struct Row { const float* src; int ih0, iw0; bool ok; };
template <bool POOL>
__device__ __forceinline__ Row row_of(const ContractArgs& p, int m) {
    const ConvGeom& g = p.g;
    Row r{p.a, 0, 0, m < p.M};
    if (!r.ok) return r;
    int n, oh, ow;
    if (POOL) {
        const int pp = m >> 2, hw = p.PH * p.PW;
        n = pp / hw;
        const int q = pp - n * hw, ph = q / p.PW;
        oh = 2 * ph + ((m >> 1) & 1); ow = 2 * (q - ph * p.PW) + (m & 1);
    } else {
        const int t = m / g.OW;
        ow = m - t * g.OW; n = t / g.OH; oh = t - n * g.OH;
    }
    r.ih0 = oh * g.sh - g.pt; r.iw0 = ow * g.sw - g.pl;
    r.src = p.a + (long long)n * g.C * g.H * g.W + (long long)r.ih0 * g.W + r.iw0;
    return r;
}
__device__ __forceinline__ bool inside(const ContractArgs& p, const Row& r, const Tap& t) {
    if (!p.padded) return r.ok && t.dy != 0x7fffffff;
    return r.ok && t.dy != 0x7fffffff && (unsigned)(r.ih0 + t.dy) < (unsigned)p.g.H && (unsigned)(r.iw0 + t.dx) < (unsigned)p.g.W;
}

}  // namespace ct

constexpr int CT_BK = 16, CT_NS = 3;

template <int BM, int BN>
constexpr int contract_smem() { return CT_NS * CT_BK * (BM + 4 + BN + 4) * 4 + 3 * CT_BK * 16; }

template <bool CONV, bool POOL, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) contract_f32_tile(const __grid_constant__ ContractArgs p) {
    ptx::grid_start();
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN, LDA = BM + 4, LDB = BN + 4;
    extern __shared__ __align__(16) float ct_smem[];
    float* As = ct_smem;                                   // [stage][k][row]
    float* Bs = ct_smem + CT_NS * CT_BK * LDA;             // [stage][k][column]
    ct::Tap* taps = reinterpret_cast<ct::Tap*>(Bs + CT_NS * CT_BK * LDB);   // [3][k]
    const uint32_t as0 = (uint32_t)__cvta_generic_to_shared(As), bs0 = (uint32_t)__cvta_generic_to_shared(Bs);
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.x * BM, j0 = blockIdx.y * BN;
    const int slabs = (p.K + CT_BK - 1) / CT_BK;
    const uint64_t neg_zero = p.neg_zero;

    ct::Row row{};
    if (CONV) row = ct::row_of<POOL>(p, m0 + tid % BM);

    auto load = [&](int slab) {
        const int st = slab % CT_NS, k0 = slab * CT_BK;
        const uint32_t ad = as0 + (uint32_t)(st * CT_BK * LDA * 4), bd = bs0 + (uint32_t)(st * CT_BK * LDB * 4);
        if (CONV) {
            static_assert(THREADS >= BM, "one row per thread");
#pragma unroll
            for (int i = 0; i < CT_BK * BM / THREADS; ++i) {
                const int kk = tid / BM + i * (THREADS / BM);
                const ct::Tap t = taps[slab % 3 * CT_BK + kk];
                const bool ok = ct::inside(p, row, t);
                ct::cp4(ad + (uint32_t)((kk * LDA + tid % BM) * 4), ok ? row.src + t.off : p.a, ok);
            }
        } else if (p.sak == 1) {
            // rows are contiguous along k: 16 threads a row
#pragma unroll
            for (int i = 0; i < CT_BK * BM / THREADS; ++i) {
                const int r = tid / CT_BK + i * (THREADS / CT_BK), kk = tid % CT_BK;
                const bool ok = m0 + r < p.M && k0 + kk < p.K;
                ct::cp4(ad + (uint32_t)((kk * LDA + r) * 4), ok ? p.a + (long long)(m0 + r) * p.sam + (k0 + kk) : p.a, ok);
            }
        } else {
#pragma unroll
            for (int i = 0; i < CT_BK * BM / THREADS; ++i) {
                const int e = tid + i * THREADS, kk = e / BM, r = e % BM;
                const bool ok = m0 + r < p.M && k0 + kk < p.K;
                ct::cp4(ad + (uint32_t)((kk * LDA + r) * 4), ok ? p.a + (long long)(m0 + r) * p.sam + (long long)(k0 + kk) * p.sak : p.a, ok);
            }
        }
        if (p.b_vec) {
            for (int e = tid; e < CT_BK * BN / 4; e += THREADS) {
                const int kk = e / (BN / 4), j = e % (BN / 4) * 4;
                const bool ok = k0 + kk < p.K && j0 + j < p.N;
                ct::cp16(bd + (uint32_t)((kk * LDB + j) * 4), ok ? p.b + (long long)(k0 + kk) * p.sbk + (j0 + j) : p.b, ok);
            }
        } else {
            const bool kfast = p.sbk == 1;
            for (int e = tid; e < CT_BK * BN; e += THREADS) {
                const int kk = kfast ? e % CT_BK : e / BN, j = kfast ? e / CT_BK : e % BN;
                const bool ok = k0 + kk < p.K && j0 + j < p.N;
                ct::cp4(bd + (uint32_t)((kk * LDB + j) * 4), ok ? p.b + (long long)(k0 + kk) * p.sbk + (long long)(j0 + j) * p.sbj : p.b, ok);
            }
        }
        ct::commit();
    };

    uint64_t acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    if (CONV && tid < 3 * CT_BK) taps[tid] = ct::tap_of(p, tid);
    if (CONV) __syncthreads();
#pragma unroll
    for (int s = 0; s < CT_NS - 1; ++s) {
        if (s < slabs) load(s); else ct::commit();
    }
    for (int it = 0; it < slabs; ++it) {
        ct::wait<CT_NS - 2>();
        __syncthreads();
        // the taps of slab it + 3 replace those of slab it, which was loaded two barriers ago
        if (CONV && tid < CT_BK) taps[it % 3 * CT_BK + tid] = ct::tap_of(p, (it + 3) * CT_BK + tid);
        if (it + CT_NS - 1 < slabs) load(it + CT_NS - 1); else ct::commit();
        const float* A = As + (it % CT_NS) * CT_BK * LDA + ty * TM;
        const float* B = Bs + (it % CT_NS) * CT_BK * LDB;
        auto step = [&](int kk) {
            float av[TM];
            uint64_t bv[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(A + kk * LDA + i);
                av[i] = v.x; av[i + 1] = v.y; av[i + 2] = v.z; av[i + 3] = v.w;
            }
            if (TN == 2) {
                bv[0] = *reinterpret_cast<const uint64_t*>(B + kk * LDB + tx * 2);
            } else {
                // columns tx * 4 + (0..3) of each group of BN * 4 / TN: 16-byte reads without bank conflicts
#pragma unroll
                for (int j = 0; j < TN / 4; ++j) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(B + kk * LDB + j * (TX * 4) + tx * 4);
                    bv[2 * j] = v.x; bv[2 * j + 1] = v.y;
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const uint64_t a2 = ct::dup2(av[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = ct::add2(acc[i][j], ct::mul2(a2, bv[j], neg_zero));
            }
        };
        const int left = p.K - it * CT_BK;
        if (left >= CT_BK) {
#pragma unroll
            for (int kk = 0; kk < CT_BK; ++kk) step(kk);
        } else {
            // (K = 9 of a first layer: a full slab would be half padding)
#pragma unroll 1
            for (int kk = 0; kk + 3 <= left; kk += 3) { step(kk); step(kk + 1); step(kk + 2); }
            for (int kk = left / 3 * 3; kk < left; ++kk) step(kk);
        }
    }

    // column of pair j, element e
    auto col_of = [&](int j, int e) { return j0 + (TN == 2 ? tx * 2 + e : (j >> 1) * (TX * 4) + tx * 4 + (j & 1) * 2 + e); };
    const int mr = m0 + ty * TM;
    if (CONV) {
        const int ohw = POOL ? p.PH * p.PW : p.g.OH * p.g.OW;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int f = col_of(j >> 1, j & 1);
            if (f >= p.N) continue;
            const float bv = p.bias ? __ldg(p.bias + f) : 0.0f;
            float v[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float lo, hi;
                ct::split2(acc[i][j >> 1], lo, hi);
                v[i] = ct::activate(__fadd_rn((j & 1) ? hi : lo, bv), p.act, p.slope);
            }
            if (POOL) {
#pragma unroll
                for (int i = 0; i < TM; i += 4) {
                    const int pp = (mr + i) >> 2;
                    if (mr + i >= p.M) break;
                    // the reference's comparison chain (lean_onnx_maxpool): NaNs are skipped
                    float mx = -INFINITY;
#pragma unroll
                    for (int q = 0; q < 4; ++q) mx = v[i + q] > mx ? v[i + q] : mx;
                    const int n = pp / ohw;
                    p.d[((long long)n * p.N + f) * ohw + (pp - n * ohw)] = mx;
                }
            } else {
#pragma unroll
                for (int i = 0; i < TM; i += 4) {
                    int m = mr + i, n = m / ohw, pos = m - n * ohw;
                    if (m >= p.M) break;
                    if (p.y_vec) {
                        *reinterpret_cast<float4*>(p.d + ((long long)n * p.N + f) * ohw + pos) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if (m + q >= p.M) break;
                            p.d[((long long)n * p.N + f) * ohw + pos] = v[i + q];
                            if (++pos == ohw) { pos = 0; ++n; }
                        }
                    }
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = mr + i;
            if (m >= p.M) break;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int col = col_of(j >> 1, j & 1);
                if (col >= p.N) continue;
                float lo, hi;
                ct::split2(acc[i][j >> 1], lo, hi);
                float v = (j & 1) ? hi : lo;
                if (p.gemm) {
                    v = __fmul_rn(v, p.alpha);
                    if (p.c_mode) v = __fadd_rn(v, __fmul_rn(__ldg(p.c + (long long)m * p.c_rs + (long long)col * p.c_cs), p.beta));
                }
                if (p.bias) v = __fadd_rn(v, __ldg(p.bias + col));
                p.d[(long long)m * p.N + col] = ct::activate(v, p.act, p.slope);
            }
        }
    }
}

// Few outputs: 8 rows x 32 columns per CTA, one output per thread (a warp is one row), slabs of 64 k.
constexpr int CF_BM = 8, CF_BN = 32, CF_BK = 64, CF_NS = 4;
constexpr int contract_few_smem() { return CF_NS * (CF_BM * (CF_BK + 4) + CF_BK * CF_BN) * 4 + 4 * CF_BK * 16; }

template <bool CONV, bool POOL>
__global__ void __launch_bounds__(256) contract_f32_few(const __grid_constant__ ContractArgs p) {
    ptx::grid_start();
    constexpr int LDA = CF_BK + 4;
    extern __shared__ __align__(16) float ct_smem[];
    float* As = ct_smem;                                   // [stage][row][k]
    float* Bs = ct_smem + CF_NS * CF_BM * LDA;             // [stage][k][column]
    ct::Tap* taps = reinterpret_cast<ct::Tap*>(Bs + CF_NS * CF_BK * CF_BN);   // [4][k]
    const uint32_t as0 = (uint32_t)__cvta_generic_to_shared(As), bs0 = (uint32_t)__cvta_generic_to_shared(Bs);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * CF_BM, j0 = blockIdx.y * CF_BN;
    const int slabs = (p.K + CF_BK - 1) / CF_BK;
    ct::Row row{};
    if (CONV) row = ct::row_of<POOL>(p, m0 + warp);

    auto load = [&](int slab) {
        const int st = slab % CF_NS, k0 = slab * CF_BK;
        const uint32_t ad = as0 + (uint32_t)(st * CF_BM * LDA * 4), bd = bs0 + (uint32_t)(st * CF_BK * CF_BN * 4);
        if (CONV) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kk = lane + 32 * i;
                const ct::Tap t = taps[slab % 4 * CF_BK + kk];
                const bool ok = ct::inside(p, row, t);
                ct::cp4(ad + (uint32_t)((warp * LDA + kk) * 4), ok ? row.src + t.off : p.a, ok);
            }
        } else if (p.a_vec) {
            if (tid < CF_BM * CF_BK / 4) {
                const int r = tid / (CF_BK / 4), kk = tid % (CF_BK / 4) * 4;
                const bool ok = m0 + r < p.M && k0 + kk < p.K;
                ct::cp16(ad + (uint32_t)((r * LDA + kk) * 4), ok ? p.a + (long long)(m0 + r) * p.sam + (k0 + kk) : p.a, ok);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kk = lane + 32 * i;
                const bool ok = m0 + warp < p.M && k0 + kk < p.K;
                ct::cp4(ad + (uint32_t)((warp * LDA + kk) * 4), ok ? p.a + (long long)(m0 + warp) * p.sam + (long long)(k0 + kk) * p.sak : p.a, ok);
            }
        }
        if (p.b_vec) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int e = tid + 256 * i, kk = e >> 3, j = (e & 7) * 4;
                const bool ok = k0 + kk < p.K && j0 + j < p.N;
                ct::cp16(bd + (uint32_t)((kk * CF_BN + j) * 4), ok ? p.b + (long long)(k0 + kk) * p.sbk + (j0 + j) : p.b, ok);
            }
        } else {
            const bool kfast = p.sbk == 1;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = tid + 256 * i, kk = kfast ? e % CF_BK : e / CF_BN, j = kfast ? e / CF_BK : e % CF_BN;
                const bool ok = k0 + kk < p.K && j0 + j < p.N;
                ct::cp4(bd + (uint32_t)((kk * CF_BN + j) * 4), ok ? p.b + (long long)(k0 + kk) * p.sbk + (long long)(j0 + j) * p.sbj : p.b, ok);
            }
        }
        ct::commit();
    };

    if (CONV) { taps[tid] = ct::tap_of(p, tid); __syncthreads(); }
#pragma unroll
    for (int s = 0; s < CF_NS - 1; ++s) {
        if (s < slabs) load(s); else ct::commit();
    }
    float acc = 0.0f;
    const bool live = m0 + warp < p.M;
    for (int it = 0; it < slabs; ++it) {
        ct::wait<CF_NS - 2>();
        __syncthreads();
        // the taps of slab it + 4 replace those of slab it
        if (CONV && tid < CF_BK) taps[it % 4 * CF_BK + tid] = ct::tap_of(p, (it + 4) * CF_BK + tid);
        if (it + CF_NS - 1 < slabs) load(it + CF_NS - 1); else ct::commit();
        if (live) {
            const float* A = As + (it % CF_NS) * CF_BM * LDA + warp * LDA;
            const float* B = Bs + (it % CF_NS) * CF_BK * CF_BN + lane;
#pragma unroll
            for (int kk = 0; kk < CF_BK; kk += 4) {
                const float4 a = *reinterpret_cast<const float4*>(A + kk);
                acc = __fadd_rn(acc, __fmul_rn(a.x, B[kk * CF_BN]));
                acc = __fadd_rn(acc, __fmul_rn(a.y, B[(kk + 1) * CF_BN]));
                acc = __fadd_rn(acc, __fmul_rn(a.z, B[(kk + 2) * CF_BN]));
                acc = __fadd_rn(acc, __fmul_rn(a.w, B[(kk + 3) * CF_BN]));
            }
        }
    }
    const int m = m0 + warp, col = j0 + lane;
    if (CONV) {
        float v = acc;
        if (col < p.N) v = ct::activate(__fadd_rn(v, p.bias ? __ldg(p.bias + col) : 0.0f), p.act, p.slope);
        if (POOL) {
            // the four members of a window are four warps of the CTA
            __shared__ float win[CF_BM][CF_BN];
            win[warp][lane] = v;
            __syncthreads();
            if ((warp & 3) == 0 && live && col < p.N) {
                const int pp = m >> 2, ohw = p.PH * p.PW, n = pp / ohw;
                float mx = -INFINITY;
#pragma unroll
                for (int q = 0; q < 4; ++q) { const float t = win[warp + q][lane]; mx = t > mx ? t : mx; }
                p.d[((long long)n * p.N + col) * ohw + (pp - n * ohw)] = mx;
            }
        } else if (live && col < p.N) {
            const int ohw = p.g.OH * p.g.OW, n = m / ohw;
            p.d[((long long)n * p.N + col) * ohw + (m - n * ohw)] = v;
        }
    } else if (live && col < p.N) {
        float v = acc;
        if (p.gemm) {
            v = __fmul_rn(v, p.alpha);
            if (p.c_mode) v = __fadd_rn(v, __fmul_rn(__ldg(p.c + (long long)m * p.c_rs + (long long)col * p.c_cs), p.beta));
        }
        if (p.bias) v = __fadd_rn(v, __ldg(p.bias + col));
        p.d[(long long)m * p.N + col] = ct::activate(v, p.act, p.slope);
    }
}

// First layers: 3x3, stride 1, up to three channels, 2x2 / 2 pool behind.  K is 9 to 27, a slab or two, and what a tile of contract_f32_tile costs
// beside its math (taps, asynchronous copies and their wait, the CTA itself, 36 gathered values a window) is twice the math.  Here a thread takes a
// pooled pixel: the 4 x 4 patch of its window is in registers for all filters, each value as a pair; eight filters at a time are four pairs x four
// members of sums, and a tap's two weight loads from shared memory (the same address in all lanes) feed 32 packed operations.  Products and sums in the
// order of the other kernels: (c, kh, kw) ascending from 0, taps outside the image as zeros.
// 32 filters of one channel, 28 x 28 images with the pool: 4096 images 143 -> 66 us (45 of packed operations), 1024 41 -> 21, 256 14.5 -> 8.3, 1 6.3 -> 4.2.
// (Also measured here: weights as pairs of equal values instead, which doubles the bytes out of shared memory, 142 us.)
constexpr int kLowCThreads = 128, kLowCMaxFilters = 256;
template <int C>
__global__ void __launch_bounds__(kLowCThreads) conv3x3_pool_f32_lowc(const __grid_constant__ ContractArgs p, int per_cta) {
    ptx::grid_start();
    extern __shared__ __align__(16) float ct_smem[];                             // [k][filter], then the biases
    const ConvGeom& g = p.g;
    const int f0 = (int)blockIdx.y * per_cta, nf = min(per_cta, (p.N + 7) / 8 * 8 - f0);             // filters of this CTA, a multiple of eight
    for (int i = threadIdx.x; i < (C * 9 + 1) * nf; i += kLowCThreads) {
        const int k = i / nf, f = f0 + i - k * nf;
        ct_smem[i] = f >= p.N ? 0.0f : (k < C * 9 ? __ldg(p.b + (long long)k * p.sbk + (long long)f * p.sbj) : (p.bias ? __ldg(p.bias + f) : 0.0f));
    }
    const int u = (int)(blockIdx.x * kLowCThreads + threadIdx.x), hw = p.PH * p.PW;      // pooled pixel (the host admits less than 2^29)
    const bool live = u < p.M >> 2;
    const int n = live ? u / hw : 0, pos = live ? u - n * hw : 0, ph = pos / p.PW, pw = pos - ph * p.PW, ih0 = 2 * ph - g.pt, iw0 = 2 * pw - g.pl;
    uint64_t v[C][4][4];
    {
        bool in_h[4], in_w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { in_h[i] = live && (unsigned)(ih0 + i) < (unsigned)g.H; in_w[i] = (unsigned)(iw0 + i) < (unsigned)g.W; }
        const float* src = p.a + (long long)n * C * g.H * g.W + (long long)ih0 * g.W + iw0;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[c][i][j] = ct::dup2(in_h[i] && in_w[j] ? __ldg(src + (c * g.H + i) * g.W + j) : 0.0f);
    }
    __syncthreads();
    if (!live) return;
    const uint64_t neg_zero = p.neg_zero;
    float* d = p.d + ((long long)n * p.N + f0) * hw + pos;
    for (int f = 0; f < nf; f += 8) {
        uint64_t acc[4][4];                                                      // [filter pair][member]
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[q][m] = 0ull;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const ulonglong2* w = reinterpret_cast<const ulonglong2*>(ct_smem + (c * 9 + t) * nf + f);
                const ulonglong2 wa = w[0], wb = w[1];
                const uint64_t wq[4] = {wa.x, wa.y, wb.x, wb.y};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint64_t x = v[c][t / 3 + (m >> 1)][t % 3 + (m & 1)];
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[q][m] = ct::add2(acc[q][m], ct::mul2(x, wq[q], neg_zero));
                }
            }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t bias = *reinterpret_cast<const uint64_t*>(ct_smem + C * 9 * nf + f + 2 * q);
            float lo[4], hi[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) ct::split2(ct::add2(acc[q][m], bias), lo[m], hi[m]);
            auto pooled = [&](const float (&x)[4]) {
                // ReLU (a NaN becomes 0) and the maximum: none of the values is a NaN or below 0, so the order of the comparisons does not matter
                if (p.act == CT_ACT_RELU) return fmaxf(fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])), 0.0f);
                // the reference's comparison chain (lean_onnx_maxpool): NaNs are skipped
                float mx = -INFINITY;
#pragma unroll
                for (int m = 0; m < 4; ++m) { const float y = ct::activate(x[m], p.act, p.slope); mx = y > mx ? y : mx; }
                return mx;
            };
            if (f0 + f + 2 * q < p.N) d[0] = pooled(lo);
            if (f0 + f + 2 * q + 1 < p.N) d[hw] = pooled(hi);
            d += 2 * (long long)hw;
        }
    }
}

// A convolution's weights [M][K] -> [K][N4], the order of the slabs (columns M .. N4 - 1 are zero).
__global__ void __launch_bounds__(256) transpose_pad_f32(const float* __restrict__ w, float* __restrict__ wt, int M, int K, int N4) {
    ptx::grid_start();
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, k0 = blockIdx.y * 32, m0 = blockIdx.x * 32;
    for (int r = ty; r < 32; r += 8) tile[r][tx] = (m0 + r < M && k0 + tx < K) ? __ldg(w + (size_t)(m0 + r) * K + k0 + tx) : 0.0f;
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
        if (k0 + r < K && m0 + tx < N4) wt[(size_t)(k0 + r) * N4 + m0 + tx] = tile[tx][r];
}

}  // namespace zb
