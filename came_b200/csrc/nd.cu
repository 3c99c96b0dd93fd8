// CAME step for tensors of more than two dimensions: a batch of B contiguous [R, C] matrices (B = product of the
// leading dimensions) that share ONE RMS clip over the whole tensor, with row / column state vectors of B*R / B*C
// entries that are quantised in blocks of 256 over their flattened entries (a block may straddle matrices) and a
// momentum quantised in blocks of 256 flat elements.  This is what the reference's classes compute for such tensors on
// their generic paths (came_pytorch/CAME.py:117-172, CAMECUDA.py:275-326, CAME8bitFull.py:1006-1075: reductions over
// dim -1 / -2, `_rms` over the whole update, `quantize_blockwise` over the flattened state); its batched CUDA variants
// (came_kernels.cu:5707-6184, global RMS at :5880-5884) follow the same algebra.
//
// Two sets of kernels, chosen per tensor by the size of one matrix.
//
// Small matrices (nd_small_batch() > 0: convolution kernels, 3 x 3 or 1 x 1, by the hundred thousand): everything but the
// clip is local to a matrix, and 256 matrices are whole blocks of every quantised vector.  A CTA takes a chunk of a
// multiple of 256 matrices into shared memory, a thread owns a matrix, and a step is two passes over the elements:
//   nd_sumsq (small)   g, old second moment      -> chunk partials of S = sum (g r c)^2; nothing else is written
//   nd_s               partials                  -> S, clip
//   nd_apply (small)   g, m, p, states           -> all states, m, p (the second moment is formed again from g and the
//                                                  old state: cheaper than 4 bytes per vector entry written and read)
// 3 x 3 and 1 x 1 have kernels of their own (nd_fixed.cu), the other shapes up to 64 elements run below.  Bound by
// instruction issue and latency, not by DRAM: ~240 thread instructions per element, most of them divisions and square
// roots of the factors and the codec.
//
// Any other shape: one thread owns one entry of a state vector and walks its row (column); the element-wise passes own
// one flat block of 256 elements per CTA.
// Every reduction has a fixed order (bit-reproducible).  Launch sequence per step, each over all N-D tensors:
//
//   nd_sq     g              -> fresh v_row / v_col (EMA with the dequantised old state), requantised states
//   nd_mean   v_row          -> mean of v_row per matrix (guarded)
//   nd_sumsq  g              -> block partials of S = sum (g r c)^2
//   nd_s      partials       -> S, clip
//   nd_res    g, m           -> fresh residual row / column vectors, requantised states
//   nd_mean   Rr             -> mean per matrix
//   nd_apply  g, m, p        -> m (requantised per flat block), p
#include "common.cuh"
#include "launch.h"

namespace came {

namespace {

__device__ __forceinline__ float nd_load(const void* base, int dtype, int64_t i) {
    if (dtype == CAME_DT_F32) return reinterpret_cast<const float*>(base)[i];
    if (dtype == CAME_DT_F16) return __half2float(reinterpret_cast<const __half*>(base)[i]);
    return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[i]);
}
__device__ __forceinline__ float nd_round(float x, int dtype) {
    if (dtype == CAME_DT_F32) return x;
    if (dtype == CAME_DT_F16) return __half2float(__float2half_rn(x));
    return __bfloat162float(__float2bfloat16_rn(x));
}
__device__ __forceinline__ void nd_store(void* base, int dtype, int64_t i, float x) {
    if (dtype == CAME_DT_F32) reinterpret_cast<float*>(base)[i] = x;
    else if (dtype == CAME_DT_F16) reinterpret_cast<__half*>(base)[i] = __float2half_rn(x);
    else reinterpret_cast<__nv_bfloat16*>(base)[i] = __float2bfloat16_rn(x);
}

// four consecutive values at an aligned address
__device__ __forceinline__ void nd_load4(const void* base, int dtype, int64_t i, float* v) {
    if (dtype == CAME_DT_F32) {
        const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + i);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        return;
    }
    const uint2 x = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(base) + i);
    const uint32_t w[2] = {x.x, x.y};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        if (dtype == CAME_DT_F16) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
            v[2 * e] = f.x; v[2 * e + 1] = f.y;
        } else {
            v[2 * e] = __uint_as_float(w[e] << 16); v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
        }
    }
}
__device__ __forceinline__ void nd_store4(void* base, int dtype, int64_t i, const float* v) {
    if (dtype == CAME_DT_F32) store_run<4>(reinterpret_cast<float*>(base) + i, v);
    else {
        uint32_t w[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (dtype == CAME_DT_F16) {
                const __half2 x = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t*>(&x);
            } else {
                const __nv_bfloat162 x = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t*>(&x);
            }
        }
        *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + i) = make_uint2(w[0], w[1]);
    }
}

struct NdShape {
    int64_t B, R, C, NR, NC, n;
};
__device__ __forceinline__ NdShape nd_shape(const CameTensorDesc& d) {
    NdShape s;
    s.B = d.batch; s.R = d.rows; s.C = d.cols;
    s.NR = s.B * s.R; s.NC = s.B * s.C; s.n = s.NR * s.C;
    return s;
}

// old value of entry e of a state vector (fp32 or uint8 with one absmax per 256 flat entries)
__device__ __forceinline__ float nd_old_vec(const void* state, const float* absmax, bool quant, int64_t e) {
    return quant ? (float)reinterpret_cast<const uint8_t*>(state)[e] * (absmax[e >> 8] / QMAX_U8)
                 : reinterpret_cast<const float*>(state)[e];
}

// fresh copy, requantisation of one block of 256 entries of a state vector (all 256 threads call)
__device__ __forceinline__ void nd_store_vec(void* state, float* absmax, float* fresh, bool quant, int64_t e, int blk, bool valid,
                                             float v, float* red) {
    if (valid) fresh[e] = v;
    if (quant) {
        const float bmax = fix_absmax(block_max(valid ? v : 0.0f, red));      // syncs: every old absmax read is done
        if (threadIdx.x == 0) absmax[blk] = bmax;
        if (valid) reinterpret_cast<uint8_t*>(state)[e] = (uint8_t)quant_u8_div(v, bmax);
    } else if (valid) {
        reinterpret_cast<float*>(state)[e] = v;
    }
}

// u0 = (g r_i) c_j and, from it, the new momentum value of element (b, i, j) at flat index f
struct NdElem {
    float u, m;
};
__device__ __forceinline__ float nd_u0(const CameTensorDesc& d, const Scratch& s, const NdShape& sh, int64_t b, int64_t i, int64_t j,
                                       int64_t f, float gscale) {
    const bool clamp = d.flags & CAME_F_SQ_CLAMP;
    const float r = row_factor(s.vr[b * sh.R + i], s.rowblk[b], clamp);
    const float c = col_factor(s.vc[b * sh.C + j], clamp);
    return ((nd_load(d.g, d.g_dtype, f) * gscale) * r) * c;
}
__device__ __forceinline__ NdElem nd_moment(const CameTensorDesc& d, const Scratch& s, const CameHyper& h, const NdShape& sh,
                                            int64_t b, int64_t i, int64_t j, int64_t f, float inv_clip) {
    NdElem o;
    o.u = nd_u0(d, s, sh, b, i, j, f, h.grad_scale) * inv_clip;
    const float m_old = d.mode == CAME_MODE_FP32 ? reinterpret_cast<const float*>(d.m)[f]
                                                 : (float)reinterpret_cast<const int8_t*>(d.m)[f] * (d.m_absmax[f >> 8] / QMAX_I8);
    o.m = m_old * h.beta1 + h.om_beta1 * o.u;
    return o;
}

}  // namespace

// RES = false: second moment of g (beta2, eps0); RES = true: residual (beta3, eps1).  Work item: one block of 256
// entries, the row vector's blocks first.
template <bool RES>
__global__ void __launch_bounds__(THREADS) k_nd_vec(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = a.hyp[d.group];
    const NdShape sh = nd_shape(d);
    const int nbr = (int)((sh.NR + QBLOCK - 1) / QBLOCK);
    const bool is_col = w.tile >= nbr;
    const int blk = is_col ? w.tile - nbr : w.tile;
    const int64_t e = (int64_t)blk * QBLOCK + threadIdx.x;
    const bool valid = e < (is_col ? sh.NC : sh.NR);
    const bool quant = d.mode != CAME_MODE_FP32;
    const float inv_clip = RES ? 1.0f / s.scal[1] : 1.0f;
    const float eps = RES ? h.eps1 : h.eps0;
    float v = 0.0f;
    if (valid) {
        const int64_t len = is_col ? sh.R : sh.C;                  // entries the mean runs over
        const int64_t b = e / (is_col ? sh.C : sh.R), k = e - b * (is_col ? sh.C : sh.R);
        float acc = 0.0f;
        for (int64_t t = 0; t < len; ++t) {
            const int64_t i = is_col ? t : k, j = is_col ? k : t;
            const int64_t f = (b * sh.R + i) * sh.C + j;
            float x;
            if (RES) {
                const NdElem o = nd_moment(d, s, h, sh, b, i, j, f, inv_clip);
                const float df = o.u - o.m;
                x = fmaf(df, df, eps);
            } else {
                const float g = nd_load(d.g, d.g_dtype, f) * h.grad_scale;
                x = fmaf(g, g, eps);
            }
            acc += x;
        }
        const float mean = acc / (float)len;
        const void* state = RES ? (is_col ? d.res_col : d.res_row) : (is_col ? d.sq_col : d.sq_row);
        const float* absmax = RES ? (is_col ? d.res_col_absmax : d.res_row_absmax) : (is_col ? d.sq_col_absmax : d.sq_row_absmax);
        v = ema_update(nd_old_vec(state, absmax, quant, e), RES ? h.beta3 : h.beta2, RES ? h.om_beta3 : h.om_beta2, mean);
    }
    void* state = RES ? (is_col ? d.res_col : d.res_row) : (is_col ? d.sq_col : d.sq_row);
    float* absmax = RES ? (is_col ? d.res_col_absmax : d.res_row_absmax) : (is_col ? d.sq_col_absmax : d.sq_row_absmax);
    float* fresh = RES ? (is_col ? s.Rc : s.Rr) : (is_col ? s.vc : s.vr);
    nd_store_vec(state, absmax, fresh, quant, e, blk, valid, v, red);
}

// guarded mean of the fresh row vector of one matrix (work item: matrix index)
template <bool RES>
__global__ void __launch_bounds__(THREADS) k_nd_mean(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const int R = (int)d.rows;
    const float* v = (RES ? s.Rr : s.vr) + (int64_t)w.tile * R;
    float mean = block_vector_sum(v, R, red) / (float)R;
    mean = RES ? guard_mean(mean, d.flags & CAME_F_RESROW_FIX, d.flags & CAME_F_RESROW_CLAMP)
               : guard_mean(mean, d.flags & CAME_F_SQ_FIX, d.flags & CAME_F_SQ_CLAMP);
    if (threadIdx.x == 0) (RES ? s.rowblk2 : s.rowblk)[w.tile] = mean;
}

// block partials of S = sum (g r c)^2 (work item: flat block of 256 elements)
__global__ void __launch_bounds__(THREADS) k_nd_sumsq(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const NdShape sh = nd_shape(d);
    const int64_t f = (int64_t)w.tile * QBLOCK + threadIdx.x;
    float u = 0.0f;
    if (f < sh.n) {
        const int64_t b = f / (sh.R * sh.C), rem = f - b * sh.R * sh.C, i = rem / sh.C, j = rem - i * sh.C;
        u = nd_u0(d, s, sh, b, i, j, f, a.hyp[d.group].grad_scale);
    }
    const float t = block_sum(u * u, red);
    if (threadIdx.x == 0) s.spart[w.tile] = t;
}

// S and the clip divisor of one tensor (clip = max(1, sqrt(S/n)/clip_threshold), came_kernels.cu:2619-2620)
__global__ void __launch_bounds__(THREADS) k_nd_s(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const NdShape sh = nd_shape(d);
    const float S = block_vector_sum(s.spart, s.tiles_r, red);      // blocks, or chunks of small matrices
    if (threadIdx.x == 0) {
        s.scal[0] = S;
        s.scal[1] = fmaxf(1.0f, sqrtf(S / (float)sh.n) / a.hyp[d.group].clip_threshold);
    }
}

// momentum (requantised per flat block of 256) and parameter update (work item: flat block)
__global__ void __launch_bounds__(THREADS) k_nd_apply(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = a.hyp[d.group];
    const NdShape sh = nd_shape(d);
    const int64_t f = (int64_t)w.tile * QBLOCK + threadIdx.x;
    const bool valid = f < sh.n;
    float m = 0.0f;
    if (valid) {
        const int64_t b = f / (sh.R * sh.C), rem = f - b * sh.R * sh.C, i = rem / sh.C, j = rem - i * sh.C;
        m = nd_moment(d, s, h, sh, b, i, j, f, 1.0f / s.scal[1]).m;
        const float rr = row_factor(s.Rr[b * sh.R + i], s.rowblk2[b], d.flags & CAME_F_RESROW_CLAMP);
        const float rc = col_factor(s.Rc[b * sh.C + j], d.flags & CAME_F_RESCOL_CLAMP);
        const float upd = (m * rr) * rc;
        nd_store(d.p, d.p_dtype, f, apply_step(nd_load(d.p, d.p_dtype, f), upd, h.lr, h.wd_lr, h.decay_mul, wd_form(h, d.flags),
                                               [&](float x) { return nd_round(x, d.p_dtype); }));
    }
    if (d.mode == CAME_MODE_FP32) {
        if (valid) reinterpret_cast<float*>(d.m)[f] = m;
    } else {
        const float bmax = fix_absmax(block_max(valid ? fabsf(m) : 0.0f, red));   // syncs: every old absmax read is done
        if (threadIdx.x == 0) d.m_absmax[w.tile] = bmax;
        if (valid) reinterpret_cast<int8_t*>(d.m)[f] = (int8_t)quant_i8_div(m, bmax);
    }
}


// ------------------------------------------------------------------------------------------
// small matrices
// ------------------------------------------------------------------------------------------
constexpr int NDS_SMEM_MAX = 200 * 1024;

// Shared-memory position of entry i.  Threads own matrices, i.e. strides of R * C, R or C words: an odd stride is free of
// bank conflicts; one word of padding every 32 spreads the even ones.
__host__ __device__ __forceinline__ int nds_pos(int i) { return i + (i >> 5); }

// shared floats of a chunk of `nm` matrices: elements (g, then u, then the update), momentum, the four vectors (old,
// then fresh values) and two vectors of factors
static size_t nds_floats(int nm, int64_t R, int64_t C) {
    auto up = [](int n) { return (size_t)((n + (n >> 5) + 4) & ~3); };
    return 2 * up((int)(nm * R * C)) + 3 * (up((int)(nm * R)) + up((int)(nm * C)));
}

// matrices of a chunk (a multiple of 256, about 2048 elements at least), 0: not a small matrix
int nd_small_batch(int64_t rows, int64_t cols) {
    if (rows * cols > 64) return 0;
    if (const int fixed = nd_fixed_batch(rows, cols)) return fixed;
    const int nm = QBLOCK * (int)(rows * cols >= 8 ? 1 : 8 / (rows * cols));
    return nds_floats(nm, rows, cols) * sizeof(float) <= (size_t)NDS_SMEM_MAX ? nm : 0;
}
// KB of shared memory of a launch
int nd_small_kb(int64_t rows, int64_t cols) {
    return (int)((nds_floats(nd_small_batch(rows, cols), rows, cols) * sizeof(float) + 1023) / 1024);
}

struct NdsChunk {
    int nm, R, C, RC;          // matrices of this chunk (the last one may be short), shape
    int64_t e0, r0, c0;        // first element, row entry, column entry
    float *el, *m, *row, *col, *rrow, *rcol, *frow, *fcol;
};
__device__ __forceinline__ NdsChunk nds_chunk(const CameTensorDesc& d, const Scratch& s, int tile, float* smem) {
    NdsChunk k;
    const int full = s.tiles_c;
    k.R = (int)d.rows; k.C = (int)d.cols; k.RC = k.R * k.C;
    const int64_t mat0 = (int64_t)tile * full;
    k.nm = (int)min((int64_t)full, (int64_t)d.batch - mat0);
    k.e0 = mat0 * k.RC; k.r0 = mat0 * k.R; k.c0 = mat0 * k.C;
    auto up = [](int n) { return (n + (n >> 5) + 4) & ~3; };
    const int ne = up(full * k.RC), nr = up(full * k.R), nc = up(full * k.C);
    k.el = smem; k.row = k.el + ne; k.col = k.row + nr; k.frow = k.col + nc; k.fcol = k.frow + nr;
    k.m = k.fcol + nc; k.rrow = k.m + ne; k.rcol = k.rrow + nr;
    return k;
}

// Four consecutive values of a chunk in shared memory, i a multiple of 4
__device__ __forceinline__ void nds_put4(float* dst, int i, const float4& v) {
    float* p = dst + nds_pos(i);      // four entries never straddle a padding word
    p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
}
__device__ __forceinline__ float4 nds_get4(const float* src, int i) {
    const float* p = src + nds_pos(i);
    return make_float4(p[0], p[1], p[2], p[3]);
}

// n values from element index `base` (a multiple of 256) of an array -> shared memory.  A group of 4 consecutive values
// per thread; the last, short group and arrays off the alignment of four values go one by one.
__device__ __forceinline__ void nds_stage(const void* src, int dtype, int64_t base, int n, float scale, float* dst) {
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    for (int i = 4 * threadIdx.x; i < n; i += 4 * THREADS) {
        float v[4];
        if (vec && i + 4 <= n) nd_load4(src, dtype, base + i, v);
        else
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = i + e < n ? nd_load(src, dtype, base + i + e) : 0.0f;
        nds_put4(dst, i, make_float4(v[0] * scale, v[1] * scale, v[2] * scale, v[3] * scale));
    }
}
// the same for 8-bit codes with one absmax per 256 entries (a warp's 4 x 32 entries lie in one block)
template <bool SIGNED>
__device__ __forceinline__ void nds_stage_codes(const void* codes, const float* absmax, int64_t base, int n, float* dst) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(codes);
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 3) == 0;
    for (int i = 4 * threadIdx.x; i < n; i += 4 * THREADS) {
        const float sc = absmax[(base + i) >> 8] / (SIGNED ? QMAX_I8 : QMAX_U8);
        uint32_t w = 0;
        if (vec && i + 4 <= n) w = *reinterpret_cast<const uint32_t*>(src + base + i);
        else
#pragma unroll
            for (int e = 0; e < 4; ++e) w |= (i + e < n ? (uint32_t)src[base + i + e] : 0u) << (8 * e);
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t b = (w >> (8 * e)) & 0xffu;
            v[e] = (SIGNED ? (float)(int8_t)b : (float)b) * sc;
        }
        nds_put4(dst, i, make_float4(v[0], v[1], v[2], v[3]));
    }
}
__device__ __forceinline__ void nds_stage_vec(const void* state, const float* absmax, bool quant, int64_t base, int n, float* dst) {
    if (quant) nds_stage_codes<false>(state, absmax, base, n, dst);
    else nds_stage(state, CAME_DT_F32, base, n, 1.0f, dst);
}
// fresh values back into a state vector: a warp owns a block of 256 entries, a lane entries 4 lane .. + 3 of each half
__device__ __forceinline__ void nds_store_vec(void* state, float* absmax, bool quant, int64_t base, int n, const float* src) {
    const int lane = threadIdx.x & 31;
    uint8_t* q = reinterpret_cast<uint8_t*>(state);
    const bool vec = (reinterpret_cast<uintptr_t>(state) & (quant ? 3 : 15)) == 0;
    for (int b = threadIdx.x >> 5; b * QBLOCK < n; b += THREADS / 32) {
        const int i0 = b * QBLOCK + 4 * lane;
        float4 v[2];
        float m = 0.0f;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = i0 + 128 * t;
            v[t] = nds_get4(src, i);      // (entries past the end lie in the arrays' own shared memory)
            if (i >= n) v[t].x = 0.0f;
            if (i + 1 >= n) v[t].y = 0.0f;
            if (i + 2 >= n) v[t].z = 0.0f;
            if (i + 3 >= n) v[t].w = 0.0f;
            m = fmaxf(m, fmaxf(fmaxf(v[t].x, v[t].y), fmaxf(v[t].z, v[t].w)));
        }
        const float a = fix_absmax(warp_max(m)), sc = quant_scale<false>(a);
        if (quant && lane == 0) absmax[(base >> 8) + b] = a;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = i0 + 128 * t;
            const float x[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
            const uint32_t w = quant ? quant_pack4<false>(v[t], a, sc) : 0u;
            if (vec && i + 4 <= n) {
                if (quant) *reinterpret_cast<uint32_t*>(q + base + i) = w;
                else *reinterpret_cast<float4*>(reinterpret_cast<float*>(state) + base + i) = v[t];
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i + e < n) {
                        if (quant) q[base + i + e] = (uint8_t)(w >> (8 * e));
                        else reinterpret_cast<float*>(state)[base + i + e] = x[e];
                    }
            }
        }
    }
}

// Row and column vectors of matrix `mat` from the terms x(e): EMA with the old values in row / col (replaced by the
// fresh ones), then out(e, r_i, c_j) for every element e.
template <typename X, typename OUT>
__device__ __forceinline__ void nds_matrix(const NdsChunk& k, int mat, float* row, float* col, X x, OUT out, float beta, float om,
                                           bool fix, bool clamp_row, bool clamp_col) {
    const int e0 = mat * k.RC, r0 = mat * k.R, c0 = mat * k.C;
    float total = 0.0f;
    for (int i = 0; i < k.R; ++i) {
        float acc = 0.0f;
        for (int j = 0; j < k.C; ++j) acc += x(e0 + i * k.C + j);
        const float v = ema_update(row[nds_pos(r0 + i)], beta, om, acc / (float)k.C);
        row[nds_pos(r0 + i)] = v;
        total += v;
    }
    const float mean = guard_mean(total / (float)k.R, fix, clamp_row);
    for (int i = 0; i < k.R; ++i) k.frow[nds_pos(r0 + i)] = row_factor(row[nds_pos(r0 + i)], mean, clamp_row);
    for (int j = 0; j < k.C; ++j) {
        float acc = 0.0f;
        for (int i = 0; i < k.R; ++i) acc += x(e0 + i * k.C + j);
        const float v = ema_update(col[nds_pos(c0 + j)], beta, om, acc / (float)k.R);
        col[nds_pos(c0 + j)] = v;
        k.fcol[nds_pos(c0 + j)] = col_factor(v, clamp_col);
    }
    for (int i = 0; i < k.R; ++i) {
        const float r = k.frow[nds_pos(r0 + i)];
        for (int j = 0; j < k.C; ++j) out(e0 + i * k.C + j, r, k.fcol[nds_pos(c0 + j)]);
    }
}
template <typename OUT>
__device__ __forceinline__ void nds_second_moment(const NdsChunk& k, int mat, const CameTensorDesc& d, const CameHyper& h, OUT out) {
    const bool clamp = d.flags & CAME_F_SQ_CLAMP;
    nds_matrix(k, mat, k.row, k.col, [&](int e) { const float g = k.el[nds_pos(e)]; return fmaf(g, g, h.eps0); },
                       out, h.beta2, h.om_beta2, d.flags & CAME_F_SQ_FIX, clamp, clamp);
}

__global__ void __launch_bounds__(THREADS) k_nds_sumsq(StepArgs a, const Work* __restrict__ work) {
    extern __shared__ __align__(16) float nds_smem[];
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = a.hyp[d.group];
    const NdsChunk k = nds_chunk(d, s, w.tile, nds_smem);
    const bool quant = d.mode != CAME_MODE_FP32;
    nds_stage(d.g, d.g_dtype, k.e0, k.nm * k.RC, h.grad_scale, k.el);
    nds_stage_vec(d.sq_row, d.sq_row_absmax, quant, k.r0, k.nm * k.R, k.row);
    nds_stage_vec(d.sq_col, d.sq_col_absmax, quant, k.c0, k.nm * k.C, k.col);
    __syncthreads();
    float acc = 0.0f;
    for (int mat = threadIdx.x; mat < k.nm; mat += THREADS)
        nds_second_moment(k, mat, d, h, [&](int e, float r, float c) {
            const float u = (k.el[nds_pos(e)] * r) * c;
            acc = fmaf(u, u, acc);
        });
    const float t = block_sum(acc, red);
    if (threadIdx.x == 0) s.spart[w.tile] = t;
}

__global__ void __launch_bounds__(THREADS) k_nds_step(StepArgs a, const Work* __restrict__ work) {
    extern __shared__ __align__(16) float nds_smem[];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper h = a.hyp[d.group];
    const uint32_t flags = d.flags;
    const NdsChunk k = nds_chunk(d, s, w.tile, nds_smem);
    const bool quant = d.mode != CAME_MODE_FP32;
    const int ne = k.nm * k.RC, nr = k.nm * k.R, nc = k.nm * k.C, lane = threadIdx.x & 31, wd = wd_form(h, flags);
    const float inv_clip = 1.0f / s.scal[1];
    nds_stage(d.g, d.g_dtype, k.e0, ne, h.grad_scale, k.el);
    if (quant) nds_stage_codes<true>(d.m, d.m_absmax, k.e0, ne, k.m);
    else nds_stage(d.m, CAME_DT_F32, k.e0, ne, 1.0f, k.m);
    nds_stage_vec(d.sq_row, d.sq_row_absmax, quant, k.r0, nr, k.row);
    nds_stage_vec(d.sq_col, d.sq_col_absmax, quant, k.c0, nc, k.col);
    nds_stage_vec(d.res_row, d.res_row_absmax, quant, k.r0, nr, k.rrow);
    nds_stage_vec(d.res_col, d.res_col_absmax, quant, k.c0, nc, k.rcol);
    __syncthreads();
    for (int mat = threadIdx.x; mat < k.nm; mat += THREADS) {
        // u in place of g, the new momentum in place of the old
        nds_second_moment(k, mat, d, h, [&](int e, float r, float c) {
            const int at = nds_pos(e);
            const float u = ((k.el[at] * r) * c) * inv_clip;
            k.el[at] = u;
            k.m[at] = k.m[at] * h.beta1 + h.om_beta1 * u;
        });
        // the update in place of u
        nds_matrix(k, mat, k.rrow, k.rcol,
            [&](int e) { const int at = nds_pos(e); const float df = k.el[at] - k.m[at]; return fmaf(df, df, h.eps1); },
            [&](int e, float r, float c) { const int at = nds_pos(e); k.el[at] = (k.m[at] * r) * c; },
            h.beta3, h.om_beta3, flags & CAME_F_RESROW_FIX, flags & CAME_F_RESROW_CLAMP, flags & CAME_F_RESCOL_CLAMP);
    }
    __syncthreads();
    nds_store_vec(d.sq_row, d.sq_row_absmax, quant, k.r0, nr, k.row);
    nds_store_vec(d.sq_col, d.sq_col_absmax, quant, k.c0, nc, k.col);
    nds_store_vec(d.res_row, d.res_row_absmax, quant, k.r0, nr, k.rrow);
    nds_store_vec(d.res_col, d.res_col_absmax, quant, k.c0, nc, k.rcol);
    // momentum and parameter, a warp per flat block of 256 elements
    const bool vec = (reinterpret_cast<uintptr_t>(d.p) & 15) == 0 && (reinterpret_cast<uintptr_t>(d.m) & 15) == 0;
    for (int b = threadIdx.x >> 5; b * QBLOCK < ne; b += THREADS / 32) {
        const int i0 = b * QBLOCK + 4 * lane;
        float pv[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = i0 + 128 * t;
            if (vec && i + 4 <= ne) nd_load4(d.p, d.p_dtype, k.e0 + i, pv[t]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) pv[t][e] = i + e < ne ? nd_load(d.p, d.p_dtype, k.e0 + i + e) : 0.0f;
        }
        float4 m[2];
        float mx = 0.0f;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = i0 + 128 * t;
            m[t] = nds_get4(k.m, i);
            if (i >= ne) m[t].x = 0.0f;
            if (i + 1 >= ne) m[t].y = 0.0f;
            if (i + 2 >= ne) m[t].z = 0.0f;
            if (i + 3 >= ne) m[t].w = 0.0f;
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(m[t].x), fabsf(m[t].y)), fmaxf(fabsf(m[t].z), fabsf(m[t].w))));
        }
        const float A = fix_absmax(warp_max(mx)), sc = quant_scale<true>(A);
        if (quant && lane == 0) d.m_absmax[(k.e0 >> 8) + b] = A;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = i0 + 128 * t;
            const int64_t f = k.e0 + i;
            const float4 u4 = nds_get4(k.el, i);
            const float upd[4] = {u4.x, u4.y, u4.z, u4.w}, mv[4] = {m[t].x, m[t].y, m[t].z, m[t].w};
            const uint32_t codes = quant ? quant_pack4<true>(m[t], A, sc) : 0u;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                pv[t][e] = apply_step(pv[t][e], upd[e], h.lr, h.wd_lr, h.decay_mul, wd, [&](float x) { return nd_round(x, d.p_dtype); });
            if (vec && i + 4 <= ne) {
                nd_store4(d.p, d.p_dtype, f, pv[t]);
                if (quant) *reinterpret_cast<uint32_t*>(reinterpret_cast<int8_t*>(d.m) + f) = codes;
                else *reinterpret_cast<float4*>(reinterpret_cast<float*>(d.m) + f) = m[t];
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i + e < ne) {
                        nd_store(d.p, d.p_dtype, f + e, pv[t][e]);
                        if (quant) reinterpret_cast<int8_t*>(d.m)[f + e] = (int8_t)(codes >> (8 * e));
                        else reinterpret_cast<float*>(d.m)[f + e] = mv[e];
                    }
            }
        }
    }
}

static cudaError_t launch_nds(int kernel, const StepArgs& a, const Work* work, int n, int smem, cudaStream_t st) {
    if (kernel != KID_ND_SUMSQ && kernel != KID_ND_APPLY) return cudaErrorInvalidValue;
    auto fn = kernel == KID_ND_SUMSQ ? k_nds_sumsq : k_nds_step;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, NDS_SMEM_MAX);
    if (e != cudaSuccess) return e;
    fn<<<n, THREADS, smem, st>>>(a, work);
    return cudaGetLastError();
}

cudaError_t launch_nd(int kernel, const KernelKey& key, const StepArgs& a, const Work* work, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (key.variant == 3) return launch_nd_fixed(kernel, key, a, work, n, st);
    if (key.variant == 2) return launch_nds(kernel, a, work, n, key.mode * 1024, st);      // small matrices of any shape
    switch (kernel) {
        case KID_ND_SQ: k_nd_vec<false><<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_MEAN: k_nd_mean<false><<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_SUMSQ: k_nd_sumsq<<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_S: k_nd_s<<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_RES: k_nd_vec<true><<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_RESMEAN: k_nd_mean<true><<<n, THREADS, 0, st>>>(a, work); break;
        case KID_ND_APPLY: k_nd_apply<<<n, THREADS, 0, st>>>(a, work); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace came
