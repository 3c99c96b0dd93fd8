// Stand-alone blockwise codec kernels (not on the step's hot path, where the codec is fused into the
// step kernels).  Bit-exact with came_pytorch/blockwise_quantization.py:66-124: IEEE division,
// round-half-even, zero padding of the last block.
//
// All four are bound by DRAM (5 bytes per element).  Flat layout: a warp owns a block of 256 elements, so the absmax is
// a warp reduction and nothing waits at a CTA barrier; a lane holds elements [4 lane, 4 lane + 4) and the same 128 further
// on: 512-byte loads and 128-byte code stores per warp.  Tile layout: a warp owns 16 rows x 128 columns (eight tiles), a
// lane 4 columns of every row, so a tile is four lanes, the sixteen loads of a lane are in flight together.  The form with
// one element per lane serves rows and buffers whose alignment does not allow 16-byte accesses.
#include "common.cuh"
#include "launch.h"

namespace came {

constexpr int CODEC_THREADS = 256;
constexpr int CODEC_WARPS = CODEC_THREADS / 32;

template <bool SIGNED>
__device__ __forceinline__ float4 codec_unpack4(uint32_t w, float s) {
    if (SIGNED)
        return make_float4((float)(int8_t)(w & 0xffu) * s, (float)(int8_t)((w >> 8) & 0xffu) * s,
                           (float)(int8_t)((w >> 16) & 0xffu) * s, (float)(int8_t)(w >> 24) * s);
    return make_float4((float)(w & 0xffu) * s, (float)((w >> 8) & 0xffu) * s, (float)((w >> 16) & 0xffu) * s, (float)(w >> 24) * s);
}
__device__ __forceinline__ float absmax4(const float4& v) {
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}
__device__ __forceinline__ float max4(const float4& v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }

// signed: max |x|; unsigned: max x over the zero-padded block (blockwise_quantization.py:73-79)
template <bool SIGNED, bool VEC>
__global__ void __launch_bounds__(CODEC_THREADS) k_quant_flat(const float* __restrict__ src, uint8_t* __restrict__ q,
                                                              float* __restrict__ absmax, int64_t n, int64_t nblk) {
    const int lane = threadIdx.x & 31;
    const int64_t blk = (int64_t)blockIdx.x * CODEC_WARPS + (threadIdx.x >> 5);
    if (blk >= nblk) return;
    const int64_t base = blk * QBLOCK;
    if (VEC && base + QBLOCK <= n) {
        const float4* s4 = reinterpret_cast<const float4*>(src + base);
        const float4 v0 = __ldcs(s4 + lane), v1 = __ldcs(s4 + 32 + lane);
        const float a = fix_absmax(warp_max(SIGNED ? fmaxf(absmax4(v0), absmax4(v1)) : fmaxf(max4(v0), max4(v1))));
        uint32_t* dst = reinterpret_cast<uint32_t*>(q + base);
        const float sc = quant_scale<SIGNED>(a);
        dst[lane] = quant_pack4<SIGNED>(v0, a, sc);
        dst[32 + lane] = quant_pack4<SIGNED>(v1, a, sc);
        if (lane == 0) absmax[blk] = a;
        return;
    }
    float v[QBLOCK / 32], m = 0.0f;
#pragma unroll
    for (int i = 0; i < QBLOCK / 32; ++i) {
        const int64_t idx = base + 32 * i + lane;
        v[i] = idx < n ? src[idx] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < QBLOCK / 32; ++i) {
        const float x = SIGNED ? fabsf(v[i]) : v[i];
        m = i ? fmaxf(m, x) : x;
    }
    const float a = fix_absmax(warp_max(m));
#pragma unroll
    for (int i = 0; i < QBLOCK / 32; ++i) {
        const int64_t idx = base + 32 * i + lane;
        if (idx < n) q[idx] = (uint8_t)quant_code<SIGNED>(v[i], a);
    }
    if (lane == 0) absmax[blk] = a;
}

template <bool SIGNED, bool VEC>
__global__ void __launch_bounds__(CODEC_THREADS) k_dequant_flat(const uint8_t* __restrict__ q, const float* __restrict__ absmax,
                                                                float* __restrict__ dst, int64_t n, int64_t nblk) {
    const int lane = threadIdx.x & 31;
    const int64_t blk = (int64_t)blockIdx.x * CODEC_WARPS + (threadIdx.x >> 5);
    if (blk >= nblk) return;
    const int64_t base = blk * QBLOCK;
    const float s = absmax[blk] / (SIGNED ? QMAX_I8 : QMAX_U8);
    if (VEC && base + QBLOCK <= n) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(q + base);
        const uint32_t w0 = w[lane], w1 = w[32 + lane];
        float4* d4 = reinterpret_cast<float4*>(dst + base);
        __stcs(d4 + lane, codec_unpack4<SIGNED>(w0, s));
        __stcs(d4 + 32 + lane, codec_unpack4<SIGNED>(w1, s));
        return;
    }
#pragma unroll
    for (int i = 0; i < QBLOCK / 32; ++i) {
        const int64_t idx = base + 32 * i + lane;
        if (idx < n) dst[idx] = (SIGNED ? (float)(int8_t)q[idx] : (float)q[idx]) * s;
    }
}

// W columns per lane: 4 (16-byte accesses, column count a multiple of 4) or 1.  A tile's columns are 16 / W lanes.
template <int W>
__global__ void __launch_bounds__(CODEC_THREADS) k_quant_tile(const float* __restrict__ src, int8_t* __restrict__ q,
                                                              float* __restrict__ absmax, int rows, int cols, int tile_cols,
                                                              int strips, int64_t n_items) {
    const int lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * CODEC_WARPS + (threadIdx.x >> 5);
    if (item >= n_items) return;
    const int ty = (int)(item / strips), col = ((int)(item - (int64_t)ty * strips) * 32 + lane) * W;
    const int nrows = min(TILE, rows - ty * TILE);
    const bool in = col < cols;
    const int64_t off = (int64_t)ty * TILE * cols + col;
    float m = 0.0f;
    if (W == 4) {
        float4 v[TILE];
#pragma unroll
        for (int r = 0; r < TILE; ++r)
            v[r] = (in && r < nrows) ? __ldcs(reinterpret_cast<const float4*>(src + off + (int64_t)r * cols)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < TILE; ++r) m = fmaxf(m, absmax4(v[r]));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        const float a = fix_absmax(m), sc = quant_scale<true>(a);
#pragma unroll
        for (int r = 0; r < TILE; ++r)
            if (in && r < nrows) *reinterpret_cast<uint32_t*>(q + off + (int64_t)r * cols) = quant_pack4<true>(v[r], a, sc);
        if (in && (lane & 3) == 0) absmax[(int64_t)ty * tile_cols + (col >> 4)] = a;
    } else {
        float v[TILE];
#pragma unroll
        for (int r = 0; r < TILE; ++r) v[r] = (in && r < nrows) ? __ldcs(src + off + (int64_t)r * cols) : 0.0f;
#pragma unroll
        for (int r = 0; r < TILE; ++r) m = fmaxf(m, fabsf(v[r]));
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float a = fix_absmax(m);
#pragma unroll
        for (int r = 0; r < TILE; ++r)
            if (in && r < nrows) q[off + (int64_t)r * cols] = (int8_t)quant_i8_div(v[r], a);
        if (in && (lane & 15) == 0) absmax[(int64_t)ty * tile_cols + (col >> 4)] = a;
    }
}

template <int W>
__global__ void __launch_bounds__(CODEC_THREADS) k_dequant_tile(const int8_t* __restrict__ q, const float* __restrict__ absmax,
                                                                float* __restrict__ dst, int rows, int cols, int tile_cols,
                                                                int strips, int64_t n_items) {
    const int lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * CODEC_WARPS + (threadIdx.x >> 5);
    if (item >= n_items) return;
    const int ty = (int)(item / strips), col = ((int)(item - (int64_t)ty * strips) * 32 + lane) * W;
    const int nrows = min(TILE, rows - ty * TILE);
    if (col >= cols) return;
    const int64_t off = (int64_t)ty * TILE * cols + col;
    const float a = absmax[(int64_t)ty * tile_cols + (col >> 4)];
    const float s = a > 0.0f ? a / QMAX_I8 : 0.0f;
    uint32_t w[TILE];
#pragma unroll
    for (int r = 0; r < TILE; ++r)
        w[r] = r < nrows ? (W == 4 ? *reinterpret_cast<const uint32_t*>(q + off + (int64_t)r * cols)
                                   : (uint32_t)(uint8_t)q[off + (int64_t)r * cols]) : 0u;
#pragma unroll
    for (int r = 0; r < TILE; ++r) {
        if (r >= nrows) break;
        float* d = dst + off + (int64_t)r * cols;
        // (an absmax of zero decodes to zero even where the scale times a code would be -0)
        if (W == 4) __stcs(reinterpret_cast<float4*>(d), a > 0.0f ? codec_unpack4<true>(w[r], s) : make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        else __stcs(d, a > 0.0f ? (float)(int8_t)w[r] * s : 0.0f);
    }
}

static inline int64_t nblocks(int64_t n) { return n <= 0 ? 1 : (n + QBLOCK - 1) / QBLOCK; }
static inline bool aligned(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }
static inline unsigned codec_grid(int64_t warps) { return (unsigned)((warps + CODEC_WARPS - 1) / CODEC_WARPS); }

cudaError_t launch_quantize_blockwise(const float* src, void* q, float* absmax, int64_t n, bool is_signed,
                                      cudaStream_t st) {
    const int64_t nblk = nblocks(n);
    const unsigned grid = codec_grid(nblk);
    uint8_t* qb = static_cast<uint8_t*>(q);
    const bool vec = aligned(src, 16) && aligned(q, 4);
    if (is_signed && vec) k_quant_flat<true, true><<<grid, CODEC_THREADS, 0, st>>>(src, qb, absmax, n, nblk);
    else if (is_signed) k_quant_flat<true, false><<<grid, CODEC_THREADS, 0, st>>>(src, qb, absmax, n, nblk);
    else if (vec) k_quant_flat<false, true><<<grid, CODEC_THREADS, 0, st>>>(src, qb, absmax, n, nblk);
    else k_quant_flat<false, false><<<grid, CODEC_THREADS, 0, st>>>(src, qb, absmax, n, nblk);
    return cudaGetLastError();
}

cudaError_t launch_dequantize_blockwise(const void* q, const float* absmax, float* dst, int64_t n, bool is_signed,
                                        cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int64_t nblk = nblocks(n);
    const unsigned grid = codec_grid(nblk);
    const uint8_t* qb = static_cast<const uint8_t*>(q);
    const bool vec = aligned(dst, 16) && aligned(q, 4);
    if (is_signed && vec) k_dequant_flat<true, true><<<grid, CODEC_THREADS, 0, st>>>(qb, absmax, dst, n, nblk);
    else if (is_signed) k_dequant_flat<true, false><<<grid, CODEC_THREADS, 0, st>>>(qb, absmax, dst, n, nblk);
    else if (vec) k_dequant_flat<false, true><<<grid, CODEC_THREADS, 0, st>>>(qb, absmax, dst, n, nblk);
    else k_dequant_flat<false, false><<<grid, CODEC_THREADS, 0, st>>>(qb, absmax, dst, n, nblk);
    return cudaGetLastError();
}

cudaError_t launch_quantize_tile16(const float* src, int8_t* q, float* absmax, int64_t rows, int64_t cols,
                                   cudaStream_t st) {
    const int tr = (int)((rows + TILE - 1) / TILE), tc = (int)((cols + TILE - 1) / TILE);
    const bool vec = cols % 4 == 0 && aligned(src, 16) && aligned(q, 4);
    const int strips = (int)((cols + (vec ? 127 : 31)) / (vec ? 128 : 32));
    const int64_t items = (int64_t)tr * strips;
    if (vec) k_quant_tile<4><<<codec_grid(items), CODEC_THREADS, 0, st>>>(src, q, absmax, (int)rows, (int)cols, tc, strips, items);
    else k_quant_tile<1><<<codec_grid(items), CODEC_THREADS, 0, st>>>(src, q, absmax, (int)rows, (int)cols, tc, strips, items);
    return cudaGetLastError();
}

cudaError_t launch_dequantize_tile16(const int8_t* q, const float* absmax, float* dst, int64_t rows, int64_t cols,
                                     cudaStream_t st) {
    const int tr = (int)((rows + TILE - 1) / TILE), tc = (int)((cols + TILE - 1) / TILE);
    const bool vec = cols % 4 == 0 && aligned(dst, 16) && aligned(q, 4);
    const int strips = (int)((cols + (vec ? 127 : 31)) / (vec ? 128 : 32));
    const int64_t items = (int64_t)tr * strips;
    if (vec) k_dequant_tile<4><<<codec_grid(items), CODEC_THREADS, 0, st>>>(q, absmax, dst, (int)rows, (int)cols, tc, strips, items);
    else k_dequant_tile<1><<<codec_grid(items), CODEC_THREADS, 0, st>>>(q, absmax, dst, (int)rows, (int)cols, tc, strips, items);
    return cudaGetLastError();
}

}  // namespace came
