// CAME step for tensors made of 3 x 3 or 1 x 1 matrices (convolution kernels): the small-matrix passes of nd.cu with the
// shape known at compile time.  Same two passes, same arithmetic, same chunk partials:
//
//   sumsq   g, old second moment      -> chunk partials of S = sum (g r c)^2
//   step    g, m, p, states           -> all states, m, p
//
// What bounds them: instruction issue, then latency; DRAM is far from busy.  3 x 3: everything of a matrix stays in its
// thread's registers.  A chunk of 256 matrices (2304 elements, 768 entries of each vector: whole blocks of 256) comes
// to shared memory as the raw bytes it has in global memory, by 16-byte asynchronous copies, the next chunk's under way
// while one is computed; a thread picks its 9 (3) entries out, and writes codes and parameters back over the bytes it read,
// from where they leave in 16-byte stores.  An fp32 copy of the chunk (38 KB instead of 15 KB) would cost a conversion pass
// in, one out, and a third of the resident warps.  The absmax of a block that several warps share is a maximum of
// non-negative floats in shared memory, compared as integers.  1 x 1: elementwise; a warp owns a block of 256
// elements, a lane 8 consecutive ones, and nothing goes through shared memory.
//
// 52 M elements of 3 x 3 and 1 x 1 kernels (fp16, flat layout): 640 us a step; with an fp32 copy of every chunk in shared
// memory and no copies ahead 983 us.
#include "common.cuh"
#include "launch.h"
#include "pipeline.cuh"

#include <type_traits>

namespace came {

namespace {

constexpr int F3_MATS = 256;                 // matrices of a 3 x 3 chunk, one per thread
constexpr int F3_ROWS = 3 * F3_MATS;         // entries of a vector of the chunk
constexpr int F1_MATS = 8 * QBLOCK;          // elements of a 1 x 1 chunk, a block per warp


// `bytes` consecutive bytes global -> shared.  A base on a 16-byte boundary: asynchronous 16-byte copies, of the last one
// only the array's bytes; any other: byte by byte.
__device__ __forceinline__ void copy_in(char* dst, const char* src, int bytes) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        for (int j = 16 * threadIdx.x; j < bytes; j += 16 * THREADS) cp16(dst + j, src + j, min(16, bytes - j));
    } else {
        for (int j = threadIdx.x; j < bytes; j += THREADS) dst[j] = src[j];
    }
}
__device__ __forceinline__ void copy_out(char* dst, const char* src, int bytes) {
    const int whole = (reinterpret_cast<uintptr_t>(dst) & 15) == 0 ? bytes & ~15 : 0;
    for (int j = 16 * threadIdx.x; j < whole; j += 16 * THREADS) *reinterpret_cast<uint4*>(dst + j) = *reinterpret_cast<const uint4*>(src + j);
    for (int j = whole + threadIdx.x; j < bytes; j += THREADS) dst[j] = src[j];
}

// element types are uniform over a launch: f(tag) with a value of the type
template <typename F> __device__ __forceinline__ void with_type(int dt, F f) {
    if (dt == CAME_DT_F32) f(float{});
    else if (dt == CAME_DT_F16) f(__half{});
    else f(__nv_bfloat16{});
}
// byte of a code -> fp32: 2^23 + byte, minus 2^23 (the sign bit of a signed one turned first)
__device__ __forceinline__ float code_value(uint32_t byte, bool is_signed) {
    return __uint_as_float(0x4b000000u | (is_signed ? byte ^ 0x80u : byte)) - (is_signed ? 8388736.0f : 8388608.0f);
}

// mean of three terms: the quotient without a division or a branch (an infinite sum has no remainder)
__device__ __forceinline__ float third(float sum) {
    return sum < 1e38f ? div_by(sum, 3.0f, 1.0f / 3.0f) : sum * (1.0f / 3.0f);
}
// (out of line: rare, and long)
static __device__ __noinline__ float plain_ratio(float x, float d) { return x / d; }

// Fresh row and column entries of a 3 x 3 matrix from its terms x (EMA with the old ones), and its factors.
__device__ __forceinline__ void matrix3(const float (&x)[9], float (&row)[3], float (&col)[3], float (&r)[3], float (&c)[3], float beta,
                                        float om, bool fix, bool clamp_row, bool clamp_col) {
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        row[i] = ema_update(row[i], beta, om, third(x[3 * i] + x[3 * i + 1] + x[3 * i + 2]));
        total += row[i];
    }
    const float mean = guard_mean(third(total), fix, clamp_row), inv = 1.0f / mean;
    const bool easy = mean > 1e-30f && mean < 1e30f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float ratio = easy ? div_by(row[i], mean, inv) : plain_ratio(row[i], mean);
        if (clamp_row) ratio = fmaxf(ratio, 1e-30f);
        r[i] = inv_sqrt(ratio);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        col[j] = ema_update(col[j], beta, om, third(x[j] + x[3 + j] + x[6 + j]));
        c[j] = inv_sqrt(clamp_col ? fmaxf(col[j], 1e-30f) : col[j]);
    }
}
// The same of a 1 x 1 matrix: its mean is its only entry, so that the row factor is 1 unless a guard or the range of the
// quotient says otherwise.
__device__ __forceinline__ void matrix1(float x, float& row, float& col, float& r, float& c, float beta, float om, bool fix,
                                        bool clamp_row, bool clamp_col) {
    row = ema_update(row, beta, om, x);
    col = ema_update(col, beta, om, x);
    r = 1.0f;
    if (!(row > 1e-30f && row < 1e30f)) r = row_factor(row, guard_mean(row, fix, clamp_row), clamp_row);
    c = inv_sqrt(clamp_col ? fmaxf(col, 1e-30f) : col);
}

// Byte offsets of a 3 x 3 chunk in a stage: gradients, second moment, (step:) parameters, momentum, residual vectors, absmax
// of the vectors (3 blocks each, in the order below) and of the momentum (9)
struct Lay3 {
    int g, row, col, ax, p, m, rrow, rcol, bytes;
    __host__ __device__ Lay3(bool quant, bool step, int gsz, int psz) {
        const int vec = F3_ROWS * (quant ? 1 : 4);
        g = 0;
        row = 9 * F3_MATS * gsz; col = row + vec; ax = col + vec;
        p = ax + 24 * 4;
        m = p + 9 * F3_MATS * psz; rrow = m + 9 * F3_MATS * (quant ? 1 : 4); rcol = rrow + vec;
        bytes = step ? rcol + vec : p;
    }
};
constexpr int AX_ROW = 0, AX_COL = 3, AX_RROW = 6, AX_RCOL = 9, AX_M = 12, AX_N = 21;

template <int N> __device__ __forceinline__ void load_elems(const char* src, int dt, int at, float scale, float (&v)[N]) {
    with_type(dt, [&](auto tag) {
        const auto* s = reinterpret_cast<const decltype(tag)*>(src) + at;
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = to_f32(s[e]) * scale;
    });
}
// N entries from `at` of codes (or fp32 values) in a stage; dq: their blocks' absmax over the codec's range
template <int N, bool QUANT, bool SIGNED>
__device__ __forceinline__ void load_state(const char* src, const float* dq, int at, float (&v)[N]) {
    if constexpr (!QUANT) {
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = reinterpret_cast<const float*>(src)[at + e];
    } else {
        const int b = at >> 8, split = ((b + 1) << 8) - at;
        const float s0 = dq[b], s1 = dq[(at + N - 1) >> 8];
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = code_value(reinterpret_cast<const uint8_t*>(src)[at + e], SIGNED) * (e < split ? s0 : s1);
    }
}
// Leaves the maximum of N non-negative values per thread, thread t's from entry N * t on, in its blocks' words.  (A warp's
// 32 N entries lie in at most 2 blocks for N = 3, 3 for N = 9.)
template <int N> __device__ __forceinline__ void leave_max(const float (&v)[N], uint32_t* dst) {
    const int at = N * threadIdx.x, b = at >> 8, split = ((b + 1) << 8) - at, first = (N * (threadIdx.x & ~31)) >> 8;
    float lo = 0.0f, hi = 0.0f;      // (fmaxf drops a NaN)
#pragma unroll
    for (int e = 0; e < N; ++e) {
        lo = fmaxf(lo, e < split ? fabsf(v[e]) : 0.0f);
        hi = fmaxf(hi, e < split ? 0.0f : fabsf(v[e]));
    }
#pragma unroll
    for (int k = 0; k < (N == 9 ? 3 : 2); ++k) {
        const float x = b == first + k ? lo : b + 1 == first + k ? hi : 0.0f;
        const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(x));
        if ((threadIdx.x & 31) == 0 && first + k < N) atomicMax(dst + first + k, w);
    }
}
// N entries back over the bytes they came from: codes by their blocks' absmax `a` and scale `s`, or the fp32 values
template <int N, bool QUANT, bool SIGNED>
__device__ __forceinline__ void store_state(char* dst, const float* a, const float* s, int at, const float (&v)[N]) {
    if constexpr (!QUANT) {
#pragma unroll
        for (int e = 0; e < N; ++e) reinterpret_cast<float*>(dst)[at + e] = v[e];
    } else {
        const int b = at >> 8, b1 = (at + N - 1) >> 8, split = ((b + 1) << 8) - at;
        const float s0 = s[b], s1 = s[b1];
        uint32_t y[N];
        bool sure = true;      // as in quant_pack4
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const float t = __fmul_rn(SIGNED ? v[e] : fmaxf(v[e], 0.0f), e < split ? s0 : s1), r = __fadd_rn(t, 12582912.0f);
            sure = sure && fabsf(__fsub_rn(t, __fsub_rn(r, 12582912.0f))) <= QUANT_SURE;
            y[e] = __float_as_uint(r);
        }
        if (!sure)
#pragma unroll
            for (int e = 0; e < N; ++e) y[e] = quant_code<SIGNED>(v[e], e < split ? a[b] : a[b1]);
#pragma unroll
        for (int e = 0; e < N; ++e) reinterpret_cast<uint8_t*>(dst)[at + e] = (uint8_t)y[e];
    }
}

struct Chunk3 {
    int tensor, tile, nm;
    int64_t mat0;
    __device__ __forceinline__ Chunk3(const StepArgs& a, const Work& w) : tensor(w.tensor), tile(w.tile) {
        mat0 = (int64_t)w.tile * F3_MATS;
        nm = (int)min((int64_t)F3_MATS, (int64_t)a.descs[w.tensor].batch - mat0);
    }
};

template <bool QUANT, bool STEP>
__device__ __forceinline__ void issue3(const StepArgs& a, const Chunk3& k, const Lay3& L, char* st, int gsz, int psz) {
    const CameTensorDesc& d = a.descs[k.tensor];
    const int ne = 9 * k.nm, nv = 3 * k.nm, vsz = QUANT ? 1 : 4;
    const int64_t e0 = 9 * k.mat0, v0 = 3 * k.mat0;
    auto at = [](const void* base, int64_t bytes) { return reinterpret_cast<const char*>(base) + bytes; };
    copy_in(st + L.g, at(d.g, e0 * gsz), ne * gsz);
    copy_in(st + L.row, at(d.sq_row, v0 * vsz), nv * vsz);
    copy_in(st + L.col, at(d.sq_col, v0 * vsz), nv * vsz);
    if (STEP) {
        copy_in(st + L.p, at(d.p, e0 * psz), ne * psz);
        copy_in(st + L.m, at(d.m, e0 * vsz), ne * vsz);
        copy_in(st + L.rrow, at(d.res_row, v0 * vsz), nv * vsz);
        copy_in(st + L.rcol, at(d.res_col, v0 * vsz), nv * vsz);
    }
    if (QUANT && threadIdx.x < (STEP ? AX_N : AX_RROW)) {
        const int t = threadIdx.x, b = t < AX_M ? t % 3 : t - AX_M;
        const float* src = t < AX_COL ? d.sq_row_absmax : t < AX_RROW ? d.sq_col_absmax : t < AX_RCOL ? d.res_row_absmax
                         : t < AX_M ? d.res_col_absmax : d.m_absmax;
        if (b * QBLOCK < (t < AX_M ? nv : ne)) cp4(st + L.ax + 4 * t, src + ((t < AX_M ? v0 : e0) >> 8) + b);
    }
}

// One persistent launch per pass; two stages, a chunk computed while the next one's copies run.
template <bool QUANT, bool STEP>
__global__ void __launch_bounds__(THREADS, 3) k_nd33(StepArgs a, const Work* __restrict__ work, int n, int gdt, int pdt) {
    extern __shared__ __align__(16) char f3_smem[];
    __shared__ float red[33], s_dq[AX_N], s_a[AX_N], s_s[AX_N];
    __shared__ uint32_t s_max[AX_N];
    const int gsz = gdt == CAME_DT_F32 ? 4 : 2, psz = pdt == CAME_DT_F32 ? 4 : 2, t = threadIdx.x, stride = gridDim.x;
    const Lay3 L(QUANT, STEP, gsz, psz);
    int i = blockIdx.x, buf = 0;
    if (i >= n) return;
    Chunk3 next(a, work[i]);
    issue3<QUANT, STEP>(a, next, L, f3_smem, gsz, psz);
    cp_commit();
    for (; i < n; i += stride, buf ^= 1) {
        const Chunk3 k = next;
        if (i + stride < n) {
            next = Chunk3(a, work[i + stride]);
            issue3<QUANT, STEP>(a, next, L, f3_smem + (buf ^ 1) * L.bytes, gsz, psz);
        }
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        char* const st = f3_smem + buf * L.bytes;
        if (QUANT) {
            if (t < AX_N) {
                s_dq[t] = (STEP || t < AX_RROW) ? reinterpret_cast<const float*>(st + L.ax)[t] / (t < AX_M ? QMAX_U8 : QMAX_I8) : 0.0f;
                s_max[t] = 0;
            }
            __syncthreads();
        }
        const CameTensorDesc& d = a.descs[k.tensor];
        const Scratch& s = a.scr[k.tensor];
        const CameHyper& h = a.hyp[d.group];
        const uint32_t flags = d.flags;
        const bool mine = t < k.nm, sq_clamp = flags & CAME_F_SQ_CLAMP;
        float g[9], row[3], col[3], r[3], c[3];
        if (mine) {
            load_elems<9>(st + L.g, gdt, 9 * t, h.grad_scale, g);
            load_state<3, QUANT, false>(st + L.row, s_dq + AX_ROW, 3 * t, row);
            load_state<3, QUANT, false>(st + L.col, s_dq + AX_COL, 3 * t, col);
            float x[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) x[e] = fmaf(g[e], g[e], h.eps0);
            matrix3(x, row, col, r, c, h.beta2, h.om_beta2, flags & CAME_F_SQ_FIX, sq_clamp, sq_clamp);
        } else {
#pragma unroll
            for (int e = 0; e < 9; ++e) g[e] = 0.0f;
#pragma unroll
            for (int e = 0; e < 3; ++e) { row[e] = 0.0f; col[e] = 0.0f; r[e] = 0.0f; c[e] = 0.0f; }
        }
        if constexpr (!STEP) {
            float acc = 0.0f;
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                const float u = (g[e] * r[e / 3]) * c[e % 3];
                acc = fmaf(u, u, acc);
            }
            const float sum = block_sum(acc, red);      // (syncs: the stage is free again)
            if (t == 0) s.spart[k.tile] = sum;
        } else {
            float m[9], rrow[3] = {0.0f, 0.0f, 0.0f}, rcol[3] = {0.0f, 0.0f, 0.0f};
            if (mine) {
                const float inv_clip = 1.0f / s.scal[1];
                load_state<9, QUANT, true>(st + L.m, s_dq + AX_M, 9 * t, m);
                load_state<3, QUANT, false>(st + L.rrow, s_dq + AX_RROW, 3 * t, rrow);
                load_state<3, QUANT, false>(st + L.rcol, s_dq + AX_RCOL, 3 * t, rcol);
                float x[9], rr[3], rc[3];
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    const float u = ((g[e] * r[e / 3]) * c[e % 3]) * inv_clip;
                    m[e] = m[e] * h.beta1 + h.om_beta1 * u;
                    const float df = u - m[e];
                    x[e] = fmaf(df, df, h.eps1);
                }
                matrix3(x, rrow, rcol, rr, rc, h.beta3, h.om_beta3, flags & CAME_F_RESROW_FIX, flags & CAME_F_RESROW_CLAMP,
                        flags & CAME_F_RESCOL_CLAMP);
                const float lr = h.lr, wd_lr = h.wd_lr, decay_mul = h.decay_mul;
                const int wd = wd_form(h, flags);
                with_type(pdt, [&](auto tag) {
                    using TP = decltype(tag);
                    TP* p = reinterpret_cast<TP*>(st + L.p) + 9 * t;
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        p[e] = from_f32<TP>(apply_step(to_f32(p[e]), (m[e] * rr[e / 3]) * rc[e % 3], lr, wd_lr, decay_mul, wd,
                                                       [](float v) { return round_to<TP>(v); }));
                });
            } else {
#pragma unroll
                for (int e = 0; e < 9; ++e) m[e] = 0.0f;
            }
            if (QUANT) {
                leave_max<3>(row, s_max + AX_ROW);
                leave_max<3>(col, s_max + AX_COL);
                leave_max<3>(rrow, s_max + AX_RROW);
                leave_max<3>(rcol, s_max + AX_RCOL);
                leave_max<9>(m, s_max + AX_M);
                __syncthreads();
                if (t < AX_N) {
                    const float A = fix_absmax(__uint_as_float(s_max[t]));
                    s_a[t] = A;
                    s_s[t] = t < AX_M ? quant_scale<false>(A) : quant_scale<true>(A);
                    const int b = t < AX_M ? t % 3 : t - AX_M;
                    float* dst = t < AX_COL ? d.sq_row_absmax : t < AX_RROW ? d.sq_col_absmax : t < AX_RCOL ? d.res_row_absmax
                               : t < AX_M ? d.res_col_absmax : d.m_absmax;
                    if (b * QBLOCK < (t < AX_M ? 3 : 9) * k.nm) dst[(((t < AX_M ? 3 : 9) * k.mat0) >> 8) + b] = A;
                }
                __syncthreads();
            }
            if (mine) {
                store_state<3, QUANT, false>(st + L.row, s_a + AX_ROW, s_s + AX_ROW, 3 * t, row);
                store_state<3, QUANT, false>(st + L.col, s_a + AX_COL, s_s + AX_COL, 3 * t, col);
                store_state<3, QUANT, false>(st + L.rrow, s_a + AX_RROW, s_s + AX_RROW, 3 * t, rrow);
                store_state<3, QUANT, false>(st + L.rcol, s_a + AX_RCOL, s_s + AX_RCOL, 3 * t, rcol);
                store_state<9, QUANT, true>(st + L.m, s_a + AX_M, s_s + AX_M, 9 * t, m);
            }
            __syncthreads();
            const int ne = 9 * k.nm, nv = 3 * k.nm, vsz = QUANT ? 1 : 4;
            const int64_t e0 = 9 * k.mat0, v0 = 3 * k.mat0;
            auto at = [](void* base, int64_t bytes) { return reinterpret_cast<char*>(base) + bytes; };
            copy_out(at(d.p, e0 * psz), st + L.p, ne * psz);
            copy_out(at(d.m, e0 * vsz), st + L.m, ne * vsz);
            copy_out(at(d.sq_row, v0 * vsz), st + L.row, nv * vsz);
            copy_out(at(d.sq_col, v0 * vsz), st + L.col, nv * vsz);
            copy_out(at(d.res_row, v0 * vsz), st + L.rrow, nv * vsz);
            copy_out(at(d.res_col, v0 * vsz), st + L.rcol, nv * vsz);
            __syncthreads();      // the stage is free again
        }
    }
    cp_wait<0>();
}

// ---- 1 x 1 ------------------------------------------------------------------------------------------------------
// 8 consecutive values from index i (a multiple of 8) of an array of n; past the end: 0
__device__ __forceinline__ void load8(const void* base, int dt, int64_t i, int64_t n, float scale, float (&v)[8]) {
    with_type(dt, [&](auto tag) {
        const auto* p = reinterpret_cast<const decltype(tag)*>(base);
        if (i + 8 <= n && (reinterpret_cast<uintptr_t>(base) & 15) == 0) load_run<8>(p + i, v);
        else
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = i + e < n ? to_f32(p[i + e]) : 0.0f;
    });
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= scale;
}
__device__ __forceinline__ void store8(void* base, int dt, int64_t i, int64_t n, const float (&v)[8]) {
    with_type(dt, [&](auto tag) {
        using T = decltype(tag);
        T* p = reinterpret_cast<T*>(base);
        if (i + 8 <= n && (reinterpret_cast<uintptr_t>(base) & 15) == 0) store_run<8>(p + i, v);
        else
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (i + e < n) p[i + e] = from_f32<T>(v[e]);
    });
}
// the same for a state array; a warp's 256 values are one block of codes
template <bool QUANT, bool SIGNED>
__device__ __forceinline__ void load8_state(const void* base, const float* absmax, int64_t i, int64_t n, float (&v)[8]) {
    if constexpr (!QUANT) {
        load8(base, CAME_DT_F32, i, n, 1.0f, v);
    } else {
        const uint8_t* q = reinterpret_cast<const uint8_t*>(base);
        const float dq = (i & ~(int64_t)(QBLOCK - 1)) < n ? absmax[i >> 8] / (SIGNED ? QMAX_I8 : QMAX_U8) : 0.0f;
        uint32_t w[2] = {0, 0};
        if (i + 8 <= n && (reinterpret_cast<uintptr_t>(q) & 7) == 0) {
            const uint2 x = *reinterpret_cast<const uint2*>(q + i);
            w[0] = x.x; w[1] = x.y;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e >> 2] |= (i + e < n ? (uint32_t)q[i + e] : 0u) << (8 * (e & 3));
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = code_value((w[e >> 2] >> (8 * (e & 3))) & 0xffu, SIGNED) * dq;
    }
}
template <bool QUANT, bool SIGNED>
__device__ __forceinline__ void store8_state(void* base, float* absmax, int64_t i, int64_t n, const float (&v)[8]) {
    if constexpr (!QUANT) {
        store8(base, CAME_DT_F32, i, n, v);
    } else {
        float mx = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) mx = fmaxf(mx, i + e < n ? fabsf(v[e]) : 0.0f);
        const float A = fix_absmax(warp_max(mx)), sc = quant_scale<SIGNED>(A);
        if (i >= n) return;
        if ((threadIdx.x & 31) == 0) absmax[i >> 8] = A;
        const uint32_t lo = quant_pack4<SIGNED>(make_float4(v[0], v[1], v[2], v[3]), A, sc);
        const uint32_t hi = quant_pack4<SIGNED>(make_float4(v[4], v[5], v[6], v[7]), A, sc);
        uint8_t* q = reinterpret_cast<uint8_t*>(base);
        if (i + 8 <= n && (reinterpret_cast<uintptr_t>(q) & 7) == 0) *reinterpret_cast<uint2*>(q + i) = make_uint2(lo, hi);
        else
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (i + e < n) q[i + e] = (uint8_t)((e < 4 ? lo : hi) >> (8 * (e & 3)));
    }
}

template <bool QUANT, bool STEP>
__global__ void __launch_bounds__(THREADS) k_nd11(StepArgs a, const Work* __restrict__ work, int gdt, int pdt) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = a.hyp[d.group];
    const uint32_t flags = d.flags;
    const bool sq_clamp = flags & CAME_F_SQ_CLAMP;
    const int64_t n = d.batch, i = (int64_t)w.tile * F1_MATS + 8 * threadIdx.x;
    float g[8], row[8], col[8], r[8], c[8];
    load8(d.g, gdt, i, n, h.grad_scale, g);
    load8_state<QUANT, false>(d.sq_row, d.sq_row_absmax, i, n, row);
    load8_state<QUANT, false>(d.sq_col, d.sq_col_absmax, i, n, col);
    if constexpr (!STEP) {
        float acc = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            matrix1(fmaf(g[e], g[e], h.eps0), row[e], col[e], r[e], c[e], h.beta2, h.om_beta2, flags & CAME_F_SQ_FIX, sq_clamp, sq_clamp);
            const float u = (g[e] * r[e]) * c[e];
            acc = i + e < n ? fmaf(u, u, acc) : acc;
        }
        const float sum = block_sum(acc, red);
        if (threadIdx.x == 0) s.spart[w.tile] = sum;
    } else {
        float m[8], rrow[8], rcol[8], p[8];
        load8_state<QUANT, true>(d.m, d.m_absmax, i, n, m);
        load8_state<QUANT, false>(d.res_row, d.res_row_absmax, i, n, rrow);
        load8_state<QUANT, false>(d.res_col, d.res_col_absmax, i, n, rcol);
        load8(d.p, pdt, i, n, 1.0f, p);
        const float inv_clip = 1.0f / s.scal[1], lr = h.lr, wd_lr = h.wd_lr, decay_mul = h.decay_mul;
        const int wd = wd_form(h, flags);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            matrix1(fmaf(g[e], g[e], h.eps0), row[e], col[e], r[e], c[e], h.beta2, h.om_beta2, flags & CAME_F_SQ_FIX, sq_clamp, sq_clamp);
            const float u = ((g[e] * r[e]) * c[e]) * inv_clip;
            m[e] = m[e] * h.beta1 + h.om_beta1 * u;
            const float df = u - m[e];
            matrix1(fmaf(df, df, h.eps1), rrow[e], rcol[e], r[e], c[e], h.beta3, h.om_beta3, flags & CAME_F_RESROW_FIX,
                    flags & CAME_F_RESROW_CLAMP, flags & CAME_F_RESCOL_CLAMP);
        }
        with_type(pdt, [&](auto tag) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                p[e] = apply_step(p[e], (m[e] * r[e]) * c[e], lr, wd_lr, decay_mul, wd, [](float v) { return round_to<decltype(tag)>(v); });
        });
        __syncwarp();      // every old absmax of the warp's blocks has been read
        store8(d.p, pdt, i, n, p);
        store8_state<QUANT, true>(d.m, d.m_absmax, i, n, m);
        store8_state<QUANT, false>(d.sq_row, d.sq_row_absmax, i, n, row);
        store8_state<QUANT, false>(d.sq_col, d.sq_col_absmax, i, n, col);
        store8_state<QUANT, false>(d.res_row, d.res_row_absmax, i, n, rrow);
        store8_state<QUANT, false>(d.res_col, d.res_col_absmax, i, n, rcol);
    }
}

template <bool QUANT, bool STEP>
cudaError_t launch33(const KernelKey& key, const StepArgs& a, const Work* work, int n, cudaStream_t st) {
    const int gsz = key.g_dtype == CAME_DT_F32 ? 4 : 2, psz = key.p_dtype == CAME_DT_F32 ? 4 : 2;
    const int smem = 2 * Lay3(QUANT, STEP, gsz, psz).bytes;
    const auto fn = k_nd33<QUANT, STEP>;
    int per_sm = 0;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * Lay3(QUANT, STEP, 4, 4).bytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, THREADS, smem);
    if (e != cudaSuccess) return e;
    fn<<<min(n, max(1, per_sm) * persistent_grid_limit()), THREADS, smem, st>>>(a, work, n, key.g_dtype, key.p_dtype);
    return cudaGetLastError();
}

}  // namespace

int nd_fixed_batch(int64_t rows, int64_t cols) { return rows == 3 && cols == 3 ? F3_MATS : rows == 1 && cols == 1 ? F1_MATS : 0; }

cudaError_t launch_nd_fixed(int kernel, const KernelKey& key, const StepArgs& a, const Work* work, int n, cudaStream_t st) {
    const bool quant = key.mode & 1, step = kernel == KID_ND_APPLY;
    if (!step && kernel != KID_ND_SUMSQ) return cudaErrorInvalidValue;
    if (key.mode & 2) {      // 3 x 3
        if (quant) return step ? launch33<true, true>(key, a, work, n, st) : launch33<true, false>(key, a, work, n, st);
        return step ? launch33<false, true>(key, a, work, n, st) : launch33<false, false>(key, a, work, n, st);
    }
    const auto fn = quant ? (step ? k_nd11<true, true> : k_nd11<true, false>) : (step ? k_nd11<false, true> : k_nd11<false, false>);
    fn<<<n, THREADS, 0, st>>>(a, work, key.g_dtype, key.p_dtype);
    return cudaGetLastError();
}

}  // namespace came
