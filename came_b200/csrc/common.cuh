// Shared device helpers of the CAME step kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "came_b200.h"

namespace came {

constexpr int QBLOCK = 256;   // elements per absmax of the flat codec (blockwise_quantization.py)
constexpr int TILE = 16;      // edge of an exp_avg tile in CAME_MODE_TILE8 (came_kernels.cu:19)
constexpr float QMAX_I8 = 127.0f;
constexpr float QMAX_U8 = 255.0f;

// reduction tile of the gradient passes (rows x cols handled by one CTA)
constexpr int K_TR = 128;
constexpr int K_TC = 512;
constexpr int THREADS = 256;
// tile of the shared-memory staged (tile-layout) momentum / apply passes
constexpr int W_TR = 128;
constexpr int W_TC = 1024;
constexpr int W_THREADS = 512;

// Per-tensor scratch, laid out in the caller's workspace by the plan.  All pointers are device
// pointers to fp32.
struct Scratch {
    float* vr;        // [rows]  fresh second-moment row vector (fp32, before requantisation)
    float* vc;        // [cols]
    float* Rr;        // [rows]  fresh residual row vector
    float* Rc;        // [cols]
    float* rowblk;    // [nbR]   sum of vr over each block of 256 rows
    float* rowblk2;   // [nbR]   same for Rr
    float* scal;      // [4]     {S = sum (g r c)^2, clip, -, -}
    float* rowpart;   // [max(tiles_c, ptiles_c) * rows]  per-CTA row partial sums
    float* colpart;   // [tiles_r * cols]                 per-CTA column partial sums
    float* spart;     // [tiles_r * tiles_c] partials of S; 1-D tensors: [nbR] block partials of sum u^2
    float* fac;       // flat layout on generic.cu: row factors r_i times the gradient scale [rows], else nullptr
    float* tpart;     // fused first pass only: [tiles_r * cols] per-strip column sums of g^2 / v_row
    int32_t tiles_r, tiles_c;     // K_TR x K_TC grid
    int32_t ptiles_r, ptiles_c;   // W_TR x W_TC grid of the staged passes
    int32_t nbR, nbC;             // ceil(rows/256), ceil(cols/256)
    int32_t fused_a;              // 1: the fused first pass runs (complete row sums, v_row and tpart come from it)
    int32_t fa_rb;                // fused first pass: rows per staged batch
    float* mfac;                  // staged momentum pass: row factors r_i / clip [R]
    float* mfac_c;                // staged passes: column factors [C], 16-byte aligned (c_j; after the residual finalize C'_j)
    float* mfac_c2;               // flat layout on the staged path: C'_j (c_j stays in mfac_c for the apply items), else nullptr
    int32_t g_v, g_nb;            // generic.cu: elements per access (8 or 1), bands of 16 rows per item
    int32_t* counters;            // generic.cu: items through with a phase (zero between launches)
    int32_t sq_col_parts;         // column partial sets the first pass leaves (strips, or strips x 2 warp groups)
    int32_t res_eps_deferred;     // 1: the residual partials hold sums of (u-m)^2 only; eps1 is added per row / column
                                  //    by the finalize kernel (cols * eps1, rows * eps1)
};

struct Work {
    int32_t tensor;
    int32_t tile;
};

// ------------------------------------------------------------------------------------------
// element conversion
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// round to T and back (the value a T-typed parameter holds after a store)
template <typename T> __device__ __forceinline__ float round_to(float x) { return to_f32(from_f32<T>(x)); }

// ------------------------------------------------------------------------------------------
// N contiguous elements -> fp32 registers and back, by 16-byte accesses (the caller guarantees the alignment)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void unpack_bf16x8(const uint4& r, float* v) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ void unpack_f16x8(const uint4& r, float* v) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

template <int N>
__device__ __forceinline__ void load_run(const float* p, float* v) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
        const float4 f = reinterpret_cast<const float4*>(p)[i];
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
    }
}
template <int N>
__device__ __forceinline__ void load_run(const __nv_bfloat16* p, float* v) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) unpack_bf16x8(reinterpret_cast<const uint4*>(p)[i], v + 8 * i);
}
template <int N>
__device__ __forceinline__ void load_run(const __half* p, float* v) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) unpack_f16x8(reinterpret_cast<const uint4*>(p)[i], v + 8 * i);
}

template <int N>
__device__ __forceinline__ void store_run(float* p, const float* v) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) reinterpret_cast<float4*>(p)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}
template <int N>
__device__ __forceinline__ void store_run(__nv_bfloat16* p, const float* v) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * i + 2 * k], v[8 * i + 2 * k + 1]);
            w[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
        reinterpret_cast<uint4*>(p)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
template <int N>
__device__ __forceinline__ void store_run(__half* p, const float* v) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const __half2 h = __floats2half2_rn(v[8 * i + 2 * k], v[8 * i + 2 * k + 1]);
            w[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
        reinterpret_cast<uint4*>(p)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// ------------------------------------------------------------------------------------------
// reductions (fixed order -> run-to-run identical results)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// all THREADS threads call; result valid in every thread.  `red` is a shared float[33].
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        red[32] = t;
    }
    __syncthreads();
    return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
    v = warp_max(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = red[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = fmaxf(t, red[w]);
        red[32] = t;
    }
    __syncthreads();
    return red[32];
}
// sum of x[0..n) by the whole block
__device__ __forceinline__ float block_vector_sum(const float* x, int n, float* red) {
    float t = 0.0f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) t += x[i];
    return block_sum(t, red);
}

// ------------------------------------------------------------------------------------------
// codec arithmetic.  Quantisation is rint((x / absmax) * qmax) with an IEEE quotient, as
// blockwise_quantization.py:73-80 computes it.  div_by() forms the quotient from a precomputed reciprocal with one
// residual correction (P. Markstein, IBM J. Res. Dev. 34, 1990: correctly rounded when the reciprocal is and nothing
// under- or overflows), which is cheaper than a division per element.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float fix_absmax(float a) { return a > 0.0f ? a : 1.0f; }

__device__ __forceinline__ float div_by(float x, float d, float inv_d) {
    const float q0 = x * inv_d;
    const float r = fmaf(-q0, d, x);
    return fmaf(r, inv_d, q0);
}
__device__ __forceinline__ int quant_i8_div(float x, float absmax) {
    const float q = rintf((x / absmax) * QMAX_I8);
    return (int)fminf(QMAX_I8, fmaxf(-QMAX_I8, q));
}
__device__ __forceinline__ int quant_u8_div(float x, float absmax) {
    const float q = rintf((x / absmax) * QMAX_U8);
    return (int)fminf(QMAX_U8, fmaxf(0.0f, q));
}
// The reciprocal trick needs 1/absmax and the residual to stay normal; outside this range take the
// plain division (uniform per block, so no divergence inside a warp's block).
__device__ __forceinline__ bool recip_safe(float absmax) { return absmax > 1e-30f && absmax < 1e30f; }

template <bool SIGNED>
__device__ __forceinline__ uint32_t quant_code(float x, float a) {
    return SIGNED ? (uint32_t)quant_i8_div(x, a) & 0xffu : (uint32_t)quant_u8_div(x, a);
}
// Four codes.  code = rint(RN(x / a) * qmax) is what the reference computes; a division per element makes the encoders
// issue-bound (66 us for a 4096 x 11008 matrix, tile layout).  t = x * RN(qmax / a) differs from RN(x / a) * qmax by
// at most four roundings, 4 * 2^-24 * 255 < 6.1e-5, so both round to the same integer unless t lies within that
// distance of a half-integer: only then (one element in ten thousand; also NaN, or an absmax outside the range in which
// qmax / a is safe) are the four divided.  The sum t + 1.5 * 2^23 rounds t to the nearest integer, ties to even, and
// carries the code in its low byte.
constexpr float QUANT_SURE = 0.5f - 6.5e-5f;
template <bool SIGNED>
__device__ __forceinline__ uint32_t quant_pack4(const float4& v, float a, float scale) {
    const float magic = 12582912.0f;
    const float x[4] = {v.x, v.y, v.z, v.w};
    uint32_t y[4];
    bool sure = true;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float t = __fmul_rn(SIGNED ? x[e] : fmaxf(x[e], 0.0f), scale);
        const float r = __fadd_rn(t, magic);
        sure = sure && fabsf(__fsub_rn(t, __fsub_rn(r, magic))) <= QUANT_SURE;
        y[e] = __float_as_uint(r);
    }
    if (!sure)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = quant_code<SIGNED>(x[e], a);
    return __byte_perm(__byte_perm(y[0], y[1], 0x0040u), __byte_perm(y[2], y[3], 0x0040u), 0x5410u);
}
// NaN where the multiplication is not safe: every comparison above then fails
template <bool SIGNED>
__device__ __forceinline__ float quant_scale(float a) {
    return recip_safe(a) ? (SIGNED ? QMAX_I8 : QMAX_U8) / a : __int_as_float(0x7fffffff);
}

// ------------------------------------------------------------------------------------------
// exponential moving average of a row / column statistic, with every rounding pinned (no contraction into
// fused multiply-adds): two kernels that finalize the same vector then agree bit for bit, and the value is the one
// the reference's separate multiply and add produce (came_kernels.cu:91, 546)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float ema_update(float old, float beta, float om, float x) {
    return __fadd_rn(__fmul_rn(old, beta), __fmul_rn(om, x));
}
// (sum + n * eps) / n
__device__ __forceinline__ float mean_plus_eps(float sum, float n, float eps) {
    return __fdiv_rn(__fadd_rn(sum, __fmul_rn(n, eps)), n);
}

// ------------------------------------------------------------------------------------------
// factor guards (one per reference code path, selected by CAME_F_* flags)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float guard_mean(float mean, bool fix, bool clamp) {
    if (clamp) return fmaxf(mean, 1e-30f);
    if (fix) return mean > 0.0f ? mean : 1.0f;
    return mean;
}
__device__ __forceinline__ float row_factor(float v, float mean, bool clamp) {
    float ratio = v / mean;
    if (clamp) ratio = fmaxf(ratio, 1e-30f);
    return 1.0f / sqrtf(ratio);
}
__device__ __forceinline__ float col_factor(float v, bool clamp) {
    if (clamp) v = fmaxf(v, 1e-30f);
    return 1.0f / sqrtf(v);
}

// 1 / sqrt(x) by one Newton step y (3 - x y^2) / 2 from the hardware's approximation, in a fifth of the instructions of a
// rounded division of a rounded square root.  Against 64 bits, every mantissa of two binades: at most 1.00 units in the last
// place off, 0.33 in the mean square, 13 % of the values not the nearest (division of a root: 1.49, 0.43, 26 %).  Outside
// the range in which no term under- or overflows: division and root.
static __device__ __noinline__ float inv_sqrt_plain(float x) { return 1.0f / sqrtf(x); }      // (out of line: rare, and long)
__device__ __forceinline__ float inv_sqrt(float x) {
    if (!(x > 1e-30f && x < 1e30f)) return inv_sqrt_plain(x);
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));      // (x is normal: no scaling of denormals around it)
    return fmaf(0.5f * y, fmaf(-x * y, y, 1.0f), y);
}

// ------------------------------------------------------------------------------------------
// weight decay + update of one parameter value, in the three forms the reference uses (wd_form: 0 no decay, 1 one
// rounding, 2 multiply form with a rounding to the parameter's type, 3 subtract form with one); every fused multiply-add
// is written out, so that all kernels agree bit for bit
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int wd_form(const CameHyper& h, uint32_t flags) {
    return h.weight_decay == 0.0f ? 0 : ((flags & CAME_F_WD_MUL2) ? 2 : ((flags & CAME_F_WD_ADD2) ? 3 : 1));
}
// (selects, no branches: wd is uniform, but a branch per element would serialise the elements of a thread)
template <typename RND>
__device__ __forceinline__ float apply_step(float pv, float upd, float lr, float wd_lr, float decay_mul, int wd, RND round) {
    const float x = wd == 2 ? __fmul_rn(pv, decay_mul) : wd == 0 ? pv : fmaf(-wd_lr, pv, pv);
    return fmaf(-lr, upd, wd >= 2 ? round(x) : x);
}

// ------------------------------------------------------------------------------------------
// 1-D tensors: second moment, update before the clip, momentum (came_kernels.cu:1035-1042, 1489-1601)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float nf_second_moment(float old, float g, const CameHyper& h) {
    return fmaf(old, h.beta2, __fmul_rn(h.om_beta2, fmaf(g, g, h.eps0)));
}
__device__ __forceinline__ float nf_update(float v, float g, uint32_t flags) {
    return __fmul_rn(inv_sqrt((flags & CAME_F_RSQRT_CLAMP) ? fmaxf(v, 1e-30f) : v), g);
}
__device__ __forceinline__ float nf_clip(float S, int64_t n, const CameHyper& h) {
    return fmaxf(1.0f, sqrtf(S / (float)n) / h.clip_threshold);
}
// (clip >= 1: the quotient by div_by is the correctly rounded one unless it is close to underflow; an infinite divisor or
// dividend has no remainder to correct by)
static __device__ __noinline__ float nf_plain_quotient(float u, float clip) { return u / clip; }      // (out of line: rare, and long)
__device__ __forceinline__ float nf_momentum(float m_old, float u, float clip, float inv_clip, uint32_t flags, const CameHyper& h) {
    if (flags & CAME_F_UPDATE_F16) u = __half2float(__float2half_rn(u));
    if (clip != 1.0f) u = clip < 1e30f && fabsf(u) < 1e30f ? div_by(u, clip, inv_clip) : nf_plain_quotient(u, clip);
    return fmaf(m_old, h.beta1, __fmul_rn(h.om_beta1, u));
}

// ------------------------------------------------------------------------------------------
// sums of per-item partials in a fixed order: groups of 64 consecutive ones, then the groups (one warp each)
// ------------------------------------------------------------------------------------------
constexpr int PARTIAL_GROUP = 64;
__device__ __forceinline__ float partial_group_sum(const float* part, int g, int n, int lane) {
    const int i = g * PARTIAL_GROUP + lane;
    const float x = i < n ? __ldcg(part + i) : 0.0f, y = i + 32 < n ? __ldcg(part + i + 32) : 0.0f;
    return warp_sum(x + y);
}
__device__ __forceinline__ float partial_total(const float* groups, int ng, int lane) {
    float t = 0.0f;
    for (int i = lane; i < ng; i += 32) t += __ldcg(groups + i);
    return warp_sum(t);
}

}  // namespace came
