// Small kernels around the staged passes over the matrices (fused_sq.cu, fused_ma.cu, fast_tile8.cu, fp_wide.cu), each
// one launch over all tensors of a kind:
//   sq_partials  : g          -> per-CTA row/col partial sums of g^2 + eps0     (rows too wide for fused_sq.cu)
//   vec_finalize : partials   -> exp_avg_{sq,res}_row/col (EMA, requantised), fresh fp32 copies
//   sumsq        : g          -> per-CTA partials of S = sum (g r c)^2          (same rows; or a clamp binds)
//   s_finalize   : partials   -> S, clip, factor vectors of the momentum pass
// All reductions are two-level with a fixed order, so a step is bit-reproducible run to run.
#include "common.cuh"
#include "launch.h"

namespace came {

// ------------------------------------------------------------------------------------------
// shared: stage the row / column factors of one CTA tile into shared memory
// ------------------------------------------------------------------------------------------
template <int TR, int TC>
__device__ __forceinline__ void stage_factors(const float* __restrict__ vrow, const float* __restrict__ vcol,
                                              const float* __restrict__ rowblk, int nbR, int R, int C, int row0,
                                              int col0, bool fix, bool clamp_row, bool clamp_col, float* s_r,
                                              float* s_c, float* red) {
    float mean = block_vector_sum(rowblk, nbR, red) / (float)R;
    mean = guard_mean(mean, fix, clamp_row);
    for (int i = threadIdx.x; i < TR; i += THREADS) {
        const int row = row0 + i;
        s_r[i] = row < R ? row_factor(vrow[row], mean, clamp_row) : 0.0f;
    }
    for (int i = threadIdx.x; i < TC; i += THREADS) {
        const int col = col0 + i;
        s_c[i] = col < C ? col_factor(vcol[col], clamp_col) : 0.0f;
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// pass 1: row / column partial sums of g^2 + eps0 over a K_TR x K_TC tile
// (reference: kUpdateSqRowQuantized came_kernels.cu:61-96 and the column walk of :198-243)
// ------------------------------------------------------------------------------------------
template <typename TG>
__global__ void __launch_bounds__(THREADS) k_sq_partials(StepArgs a, const Work* __restrict__ work) {
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const int R = (int)d.rows, C = (int)d.cols;
    const int tr = w.tile / s.tiles_c, tc = w.tile - tr * s.tiles_c;
    const int row0 = tr * K_TR, col0 = tc * K_TC;
    const float eps0 = a.hyp[d.group].eps0, gscale = a.hyp[d.group].grad_scale;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TG* __restrict__ g = reinterpret_cast<const TG*>(d.g);

    __shared__ float s_col[THREADS / 32][K_TC];
    float colacc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) colacc[e] = 0.0f;

    for (int k = 0; k < K_TR / 8; ++k) {
        const int row = row0 + warp + 8 * k;
        if (row >= R) break;   // uniform per warp
        float racc = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = col0 + h * 256 + lane * 8;
            if (col < C) {
                float v[8];
                load_run<8>(g + (int64_t)row * C + col, v);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    v[e] *= gscale;
                    float q = fmaf(v[e], v[e], eps0);
                    racc += q;
                    colacc[h * 8 + e] += q;
                }
            }
        }
        racc = warp_sum(racc);
        if (lane == 0) s.rowpart[(int64_t)tc * R + row] = racc;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) s_col[warp][h * 256 + lane * 8 + e] = colacc[h * 8 + e];
    __syncthreads();
    for (int cc = threadIdx.x; cc < K_TC; cc += THREADS) {
        const int col = col0 + cc;
        if (col < C) {
            float t = 0.0f;
#pragma unroll
            for (int ww = 0; ww < THREADS / 32; ++ww) t += s_col[ww][cc];
            s.colpart[(int64_t)tr * C + col] = t;
        }
    }
}

// ------------------------------------------------------------------------------------------
// finalize one block of 256 entries of a row or column vector: EMA with the dequantised old state,
// fresh fp32 copy for the following passes, requantisation (uint8, absmax = block max, 0 -> 1).
// RES=false: second moment (beta2, partials of pass 1); RES=true: residual (beta3, partials of moment).
// (reference: came_kernels.cu:77-93, 215-242, 298-333, 2685-2706, 2742-2779, 524-593, 1436-1487)
// ------------------------------------------------------------------------------------------
// Sum of the `parts` rows of a [parts x n] matrix of column partials for the 256 columns of block b; the result
// for column b * 256 + threadIdx.x.  Warp w adds the rows w, w + 8, ... (a lane holds 8 columns: two 16-byte loads
// per row), then the eight per-warp sums are added in a fixed order: the chain of dependent loads is parts / 8
// long instead of parts, and the order of the additions does not depend on timing.
__device__ __forceinline__ float column_partial_sum(const float* __restrict__ part, int parts, int n, int b,
                                                    float (*s_acc)[QBLOCK]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = b * QBLOCK + lane * 8;
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const bool vec = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(part) & 15) == 0 && c0 + 8 <= n;
    if (vec) {
#pragma unroll 8
        for (int t = warp; t < parts; t += THREADS / 32) {
            const float4* p = reinterpret_cast<const float4*>(part + (int64_t)t * n + c0);
            const float4 x = p[0], y = p[1];
            acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
            acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
        }
    } else {
        for (int t = warp; t < parts; t += THREADS / 32)
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (c0 + e < n) acc[e] += part[(int64_t)t * n + c0 + e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s_acc[warp][lane * 8 + e] = acc[e];
    __syncthreads();
    float r = 0.0f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) r += s_acc[w][threadIdx.x];
    __syncthreads();      // the buffer may be reused right away
    return r;
}

template <bool RES>
__global__ void __launch_bounds__(THREADS) k_vec_finalize(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    __shared__ float s_acc[THREADS / 32][QBLOCK];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = a.hyp[d.group];
    const int R = (int)d.rows, C = (int)d.cols;
    const bool is_col = w.tile >= s.nbR;
    const int b = is_col ? w.tile - s.nbR : w.tile;
    const int n = is_col ? C : R;
    const int idx = b * QBLOCK + threadIdx.x;
    const bool valid = idx < n;
    const bool quant = d.mode != CAME_MODE_FP32;
    const float beta = RES ? h.beta3 : h.beta2;
    const float om = RES ? h.om_beta3 : h.om_beta2;

    void* state = RES ? (is_col ? d.res_col : d.res_row) : (is_col ? d.sq_col : d.sq_row);
    float* absmax = RES ? (is_col ? d.res_col_absmax : d.res_row_absmax) : (is_col ? d.sq_col_absmax : d.sq_row_absmax);
    float* fresh = RES ? (is_col ? s.Rc : s.Rr) : (is_col ? s.vc : s.vr);

    // the fused first pass delivers finished v_row values, column sums without eps0, and tpart
    const bool fused = !RES && s.fused_a;
    float v = 0.0f, tsum = 0.0f;
    // column partials: summed by the whole block together (every thread takes part, also beyond the last column)
    float colsum = 0.0f;
    if (is_col) {
        const int parts = RES ? s.ptiles_r : s.sq_col_parts;
        colsum = column_partial_sum(s.colpart, parts, C, b, s_acc);
        if (fused) {      // the fused first pass sums the raw gradient: the gradient scale enters here, squared
            const float gs2 = h.grad_scale * h.grad_scale;
            tsum = column_partial_sum(s.tpart, parts, C, b, s_acc) * gs2;
            colsum *= gs2;
        }
    }
    if (valid) {
        if (fused && !is_col) {
            v = s.vr[idx];
        } else {
            float acc = 0.0f;
            if (!is_col) {
                const int parts = RES ? s.ptiles_c : s.tiles_c;
                for (int t = 0; t < parts; ++t) acc += s.rowpart[(int64_t)t * R + idx];
                acc = (RES && s.res_eps_deferred) ? mean_plus_eps(acc, (float)C, h.eps1) : __fdiv_rn(acc, (float)C);
            } else {
                acc = colsum;
                if (fused) acc = __fadd_rn(acc, __fmul_rn((float)R, h.eps0));
                acc = (RES && s.res_eps_deferred) ? mean_plus_eps(acc, (float)R, h.eps1) : __fdiv_rn(acc, (float)R);
            }
            float old;
            if (quant) {
                old = (float)reinterpret_cast<const uint8_t*>(state)[idx] * (absmax[b] / QMAX_U8);
            } else {
                old = reinterpret_cast<const float*>(state)[idx];
            }
            v = ema_update(old, beta, om, acc);
            fresh[idx] = v;
        }
    }
    // The fused first pass gets the clip sum from a closed form that assumes r_i^2 = mean / v_row_i and c_j^2 = 1 / v_col_j,
    // i.e. that none of the 1e-30 clamps binds.  Far outside this range one could: the two-pass sum then runs instead.
    if (fused && (d.flags & CAME_F_SQ_CLAMP) && valid && !(v >= 1e-20f && v <= 1e8f)) s.scal[3] = 1.0f;
    if (quant) {
        const float bmax = fix_absmax(block_max(valid ? v : 0.0f, red));   // syncs: every old absmax read is done
        if (threadIdx.x == 0) absmax[b] = bmax;
        if (valid) reinterpret_cast<uint8_t*>(state)[idx] = (uint8_t)quant_u8_div(v, bmax);
    } else if (valid) {
        reinterpret_cast<float*>(state)[idx] = v;
    }
    if (!is_col) {
        const float bs = block_sum(valid ? v : 0.0f, red);
        if (threadIdx.x == 0) (RES ? s.rowblk2 : s.rowblk)[b] = bs;
    } else if (fused) {
        // this block's share of sum_j T_j / v_col_j  (S = mean(v_row) * that sum, see fused_sq.cu)
        const float bs = block_sum((valid && v > 0.0f) ? tsum / v : 0.0f, red);
        if (threadIdx.x == 0) s.spart[b] = bs;
    }
}

// ------------------------------------------------------------------------------------------
// pass 2: partials of S = sum (g * r_i * c_j)^2   (reference: kSumUpdateSq came_kernels.cu:596-619)
// ------------------------------------------------------------------------------------------
template <typename TG>
__global__ void __launch_bounds__(THREADS) k_sumsq(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    __shared__ float s_r[K_TR];
    __shared__ float s_c[K_TC];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    if (s.fused_a && s.scal[3] == 0.0f) return;      // the fused first pass's closed form stands: nothing to do
    const int R = (int)d.rows, C = (int)d.cols;
    const int tr = w.tile / s.tiles_c, tc = w.tile - tr * s.tiles_c;
    const int row0 = tr * K_TR, col0 = tc * K_TC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TG* __restrict__ g = reinterpret_cast<const TG*>(d.g);
    const bool clamp = d.flags & CAME_F_SQ_CLAMP;
    const float gscale = a.hyp[d.group].grad_scale;
    stage_factors<K_TR, K_TC>(s.vr, s.vc, s.rowblk, s.nbR, R, C, row0, col0, d.flags & CAME_F_SQ_FIX, clamp, clamp,
                              s_r, s_c, red);
    float cf[16];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int e = 0; e < 8; ++e) cf[hh * 8 + e] = s_c[hh * 256 + lane * 8 + e];

    float acc = 0.0f;
    for (int k = 0; k < K_TR / 8; ++k) {
        const int rl = warp + 8 * k;
        const int row = row0 + rl;
        if (row >= R) break;
        const float r = s_r[rl];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int col = col0 + hh * 256 + lane * 8;
            if (col < C) {
                float v[8];
                load_run<8>(g + (int64_t)row * C + col, v);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float u = ((v[e] * gscale) * r) * cf[hh * 8 + e];   // masked elements: v = 0, cf = 0
                    acc = fmaf(u, u, acc);
                }
            }
        }
    }
    const float t = block_sum(acc, red);
    if (threadIdx.x == 0) s.spart[w.tile] = t;
}

// S and the clip divisor of one tensor (reference: kReducePartialSum came_kernels.cu:763-779 and
// clip = max(1, sqrt(S/n)/clip_threshold), came_kernels.cu:2619-2620)
__global__ void __launch_bounds__(THREADS) k_s_finalize(StepArgs a, const Work* __restrict__ work) {
    __shared__ float red[33];
    const Work w = work[blockIdx.x];
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    float S;
    if (s.fused_a && s.scal[3] == 0.0f) {
        float mean = block_vector_sum(s.rowblk, s.nbR, red) / (float)d.rows;
        mean = guard_mean(mean, d.flags & CAME_F_SQ_FIX, d.flags & CAME_F_SQ_CLAMP);
        S = mean * block_vector_sum(s.spart, s.nbC, red);
    } else {
        S = block_vector_sum(s.spart, s.tiles_r * s.tiles_c, red);
    }
    const float n = (float)((int64_t)d.rows * d.cols);
    const float clip = fmaxf(1.0f, sqrtf(S / n) / a.hyp[d.group].clip_threshold);   // S is the same in every thread
    if (threadIdx.x == 0 && w.tile == 0) {
        s.scal[0] = S;
        s.scal[1] = clip;
    }
    if (s.mfac) {
        // factor vectors of the momentum pass, once per tensor instead of once per tile: r_i / clip, then c_j
        const bool clamp = d.flags & CAME_F_SQ_CLAMP;
        float mean = block_vector_sum(s.rowblk, s.nbR, red) / (float)d.rows;
        mean = guard_mean(mean, d.flags & CAME_F_SQ_FIX, clamp);
        const float inv_clip = 1.0f / clip;
        const int R = (int)d.rows, C = (int)d.cols;
        const int hi = min(R + C, (w.tile + 1) * S_FIN_CHUNK);      // this CTA's chunk of the R + C entries
        for (int i = w.tile * S_FIN_CHUNK + threadIdx.x; i < hi; i += THREADS)
            if (i < R) s.mfac[i] = row_factor(s.vr[i], mean, clamp) * inv_clip * a.hyp[d.group].grad_scale;   // g enters u through it
            else s.mfac_c[i - R] = col_factor(s.vc[i - R], clamp);
    }
}

// ------------------------------------------------------------------------------------------
// host-side launchers
// ------------------------------------------------------------------------------------------
template <typename F>
static cudaError_t go(F kernel, const StepArgs& a, const Work* work, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    kernel<<<n, THREADS, 0, st>>>(a, work);
    return cudaGetLastError();
}

using KernelFn = void (*)(StepArgs, const Work*);

static KernelFn pick_sq_partials(int g) {
    switch (g) {
        case CAME_DT_F32: return k_sq_partials<float>;
        case CAME_DT_F16: return k_sq_partials<__half>;
        default: return k_sq_partials<__nv_bfloat16>;
    }
}
static KernelFn pick_sumsq(int g) {
    switch (g) {
        case CAME_DT_F32: return k_sumsq<float>;
        case CAME_DT_F16: return k_sumsq<__half>;
        default: return k_sumsq<__nv_bfloat16>;
    }
}

cudaError_t launch_factored(int kernel, const KernelKey& key, const StepArgs& a, const Work* work, int n,
                            cudaStream_t st) {
    switch (kernel) {
        case KID_SQ_PARTIALS: return go(pick_sq_partials(key.g_dtype), a, work, n, st);
        case KID_SQ_FINALIZE: return go(k_vec_finalize<false>, a, work, n, st);
        case KID_SUMSQ: return go(pick_sumsq(key.g_dtype), a, work, n, st);
        case KID_S_FINALIZE: return go(k_s_finalize, a, work, n, st);
        case KID_RES_FINALIZE: return go(k_vec_finalize<true>, a, work, n, st);
        case KID_MOMENT:
        case KID_APPLY:
            if (key.mode == CAME_MODE_FP32) return launch_fp32_wide(kernel, key, a, work, n, st);
            return launch_fast_tile8(kernel, key, a, work, n, st);
        case KID_APPLY_FLAT: return launch_fast_tile8(kernel, key, a, work, n, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace came
