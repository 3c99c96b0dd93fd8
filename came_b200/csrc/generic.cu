// The whole step of any set of matrices and vectors as ONE cooperative kernel: every shape and alignment, and the sets
// that are too small for the staged kernels.
//
// The staged kernels (fused_sq.cu, fused_ma.cu, fp_wide.cu) move 128 x 1024 tiles through one CTA per SM and need columns
// in multiples of 64.  Two kinds of work do not fit them.  Small sets: eight such tiles leave 140 SMs idle, and the seven
// launches of a step, each 2-5 us with its gap, are most of its time.  Odd widths, unaligned buffers and thin matrices:
// no bulk copies.  Here a step is six phases of one kernel, separated by grid-wide barriers:
//
//   S1  g                 -> row / column partial sums of g^2          1-D tensors: partials of sum u^2, their sum
//   F1  partials          -> v_row, c_j, requantised states, mean      1-D tensors: v, m, p
//   S2  g                 -> partials of S = sum (g r c)^2; the tensor's last item leaves S and the clip
//   M   g, m              -> m, row / column partials of (u - m)^2     (flat layout: m is not written yet)
//   F2  partials          -> residual vectors, C'_j, mean
//   A   m, p (flat: g too) -> p (flat: m too)
//
// What bounds it: latency in small sets (a phase is a chain of dependent loads, and its code is fetched cold), bytes in
// flight and instruction issue in large ones.  So the unit of work on a matrix is a warp, not a CTA: bands of 16 rows x 64
// columns, which hold whole 16 x 16 tiles of the momentum; nothing meets at a CTA barrier.  A band and everything it needs
// (vector slices, absmax) comes to the warp's own shared memory by 16-byte asynchronous copies of the aligned chunks that
// cover its rows, whatever the rows' alignment, and (16-bit types) the next band is under way while one is computed.  V =
// 8: rows on 16-byte boundaries, a lane owns 8 consecutive columns of 4 rows; V = 1: any alignment, a lane owns columns
// lane and lane + 32 of 16 rows.  Items are dealt out across the SMs first.  All reductions have a fixed order: of the items
// that share a result the last to finish (a counter) adds the partials in index order.
#include "common.cuh"
#include "launch.h"
#include "pipeline.cuh"

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

namespace came {

namespace {

constexpr int G_WARPS = THREADS / 32;
constexpr uint32_t G_POLL_LIMIT = 1u << 22;      // polls of the grid barrier (seconds) before a CTA gives up

// ---- element buffers: one type, or (g and p of different types) a type read at run time --------------------------
template <typename T> struct Buf {
    T* p;
    __device__ __forceinline__ Buf(const void* q, int) : p(reinterpret_cast<T*>(const_cast<void*>(q))) {}
    __device__ __forceinline__ float get(int64_t i) const { return to_f32(p[i]); }
    __device__ __forceinline__ void get8(int64_t i, float* v) const { load_run<8>(p + i, v); }
    __device__ __forceinline__ float round(float x) const { return round_to<T>(x); }
    __device__ __forceinline__ void put(int64_t i, float x, int64_t delta = 0) const {
        *reinterpret_cast<T*>(reinterpret_cast<char*>(p + i) + delta) = from_f32<T>(x);
    }
    __device__ __forceinline__ void put8(int64_t i, const float* v, int64_t delta = 0) const {
        store_run<8>(reinterpret_cast<T*>(reinterpret_cast<char*>(p + i) + delta), v);
    }
};
struct Any {};
template <> struct Buf<Any> {
    void* p;
    int dt;
    __device__ __forceinline__ Buf(const void* q, int t) : p(const_cast<void*>(q)), dt(t) {}
    template <typename F> __device__ __forceinline__ void with(F f) const {
        if (dt == CAME_DT_F32) f(Buf<float>(p, 0));
        else if (dt == CAME_DT_F16) f(Buf<__half>(p, 0));
        else f(Buf<__nv_bfloat16>(p, 0));
    }
    __device__ __forceinline__ float get(int64_t i) const { float x; with([&](auto b) { x = b.get(i); }); return x; }
    __device__ __forceinline__ void get8(int64_t i, float* v) const { with([&](auto b) { b.get8(i, v); }); }
    __device__ __forceinline__ float round(float x) const { float y; with([&](auto b) { y = b.round(x); }); return y; }
    __device__ __forceinline__ void put(int64_t i, float x, int64_t delta = 0) const { with([&](auto b) { b.put(i, x, delta); }); }
    __device__ __forceinline__ void put8(int64_t i, const float* v, int64_t delta = 0) const { with([&](auto b) { b.put8(i, v, delta); }); }
};

struct GShared {
    float red[33];
    int last;
    float col[G_WARPS][QBLOCK];
};

// (acquire-release instead of __threadfence(), which is sequentially consistent and waits longer)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ int atom_add_acq_rel(int* p, int x) {
    int old;
    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(x) : "memory");
    return old;
}

__device__ __forceinline__ uint32_t ld_acquire_gpu_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier of a cooperative launch.  One word: arrivals in its low 16 bits, zero again once all have come, the
// generation above.  False when the others did not arrive within the limit: the status word is set, the arrival is taken
// back (unless the generation has moved on after all) and the CTA leaves, so that a later launch finds a clean word.
constexpr uint32_t G_ARRIVALS = 0xffffu;
__device__ __forceinline__ bool grid_barrier(uint32_t* bar, int* status, uint32_t limit = G_POLL_LIMIT) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_ok = 1;
        fence_gpu();      // (the whole CTA's writes: they happened before the barrier above)
        const uint32_t before = (uint32_t)atom_add_acq_rel(reinterpret_cast<int*>(bar), 1), gen = before & ~G_ARRIVALS;
        if ((before & G_ARRIVALS) == gridDim.x - 1) {
            atom_add_acq_rel(reinterpret_cast<int*>(bar), (int)(G_ARRIVALS + 1 - gridDim.x));
        } else {
            uint32_t now = ld_acquire_gpu_u32(bar), polls = 0;
            while ((now & ~G_ARRIVALS) == gen) {
                if (++polls > limit) {
                    const uint32_t seen = atomicCAS(bar, now, now - 1);
                    if (seen == now) { atomicExch(status, STATUS_MBAR_TIMEOUT); s_ok = 0; break; }
                    now = seen;      // (another arrival, or the release: look again)
                } else {
                    now = ld_acquire_gpu_u32(bar);
                }
            }
        }
        fence_gpu();
    }
    __syncthreads();
    return s_ok != 0;
}

// True in every thread of the CTA that is the last of `total` to come here (the counter is then back at zero); the
// other CTAs' writes are visible to it.
__device__ __forceinline__ bool last_cta(int* counter, int total, GShared& sh) {
    __syncthreads();
    if (threadIdx.x == 0) {
        fence_gpu();      // (the whole CTA's writes: they happened before the barrier)
        const int before = atom_add_acq_rel(counter, 1);
        sh.last = before == total - 1;
        if (sh.last) *counter = 0;
        fence_gpu();
    }
    __syncthreads();
    return sh.last;
}
__device__ __forceinline__ float block_vector_sum_cg(const float* x, int n, float* red) {
    float t = 0.0f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) t += __ldcg(x + i);
    return block_sum(t, red);
}

// True (in every lane) when this warp is the last of `total` to come here; the counter is then back at zero and the
// other warps' writes are visible.
__device__ __forceinline__ bool last_warp(int* counter, int total, int lane) {
    __syncwarp();
    int before = 0;
    if (lane == 0) {
        fence_gpu();
        before = atom_add_acq_rel(counter, 1);
        if (before == total - 1) *counter = 0;
        fence_gpu();
    }
    before = __shfl_sync(0xffffffffu, before, 0);
    __syncwarp();      // (a shuffle orders no memory: what lane 0 has acquired the other lanes may read from here on)
    return before == total - 1;
}
// Sum of n partials, one per item, in index order: the last of every 64 items adds their partials (leave_partial); up to
// 32 such groups the readers add themselves (read_sum: one load per lane, cheaper than one more chain of a fence, an atomic
// and a load before the grid barrier), more the last group adds.
// part: n partials, the groups' sums, the total; counters: one for the groups, then one per group.
__device__ __forceinline__ void leave_partial(float* part, int* counters, int i, int n, float x, int lane) {
    const int ng = (n + PARTIAL_GROUP - 1) / PARTIAL_GROUP, g = i / PARTIAL_GROUP;
    if (lane == 0) part[i] = x;
    if (!last_warp(counters + 1 + g, min(PARTIAL_GROUP, n - g * PARTIAL_GROUP), lane)) return;
    const float t = partial_group_sum(part, g, n, lane);
    if (lane == 0) part[n + g] = t;
    if (ng <= 32 || !last_warp(counters, ng, lane)) return;
    const float sum = partial_total(part + n, ng, lane);
    if (lane == 0) part[n + ng] = sum;
}
__device__ __forceinline__ float read_sum(const float* part, int n, int lane) {
    const int ng = (n + PARTIAL_GROUP - 1) / PARTIAL_GROUP;
    if (ng > 32) return __ldcg(part + n + ng);
    return warp_sum(lane < ng ? __ldcg(part + n + lane) : 0.0f);
}
// mean of a vector from the sums of its blocks of 256 entries, guarded
__device__ __forceinline__ float read_mean(const float* blk, int nb, int n, bool fix, bool clamp, int lane) {
    float t = 0.0f;
    for (int i = lane; i < nb; i += 32) t += __ldcg(blk + i);
    return guard_mean(warp_sum(t) / (float)n, fix, clamp);
}

// ---- a warp's item of a matrix ---------------------------------------------------------------------------------
constexpr int G_CW = 64;      // columns of an item

template <typename T> struct Size { static constexpr int BYTES = sizeof(T), FIXED = sizeof(T); };
template <> struct Size<Any> { static constexpr int BYTES = 4, FIXED = 0; };      // the largest; not known
template <typename T> __device__ __forceinline__ int size_of(int dt) {
    if constexpr (std::is_same<T, Any>::value) return dt == CAME_DT_F32 ? 4 : 2;
    else return (int)sizeof(T);
}

// One band (16 rows x 64 columns) in a warp's shared memory: rows of operand A (g or p) and of the momentum, each from the
// 16-byte boundary at or before its first byte; the band's 16 row values, 64 column factors, and absmax values.
template <typename T, int MODE> struct Stage {
    static constexpr int PA = G_CW * Size<T>::BYTES + 16;
    static constexpr int PM = G_CW * (MODE == CAME_MODE_FP32 ? 4 : 1) + 16;
    static constexpr int OFF_M = 16 * PA, OFF_V = OFF_M + 16 * PM, OFF_C = OFF_V + 16 * 4, OFF_X = OFF_C + G_CW * 4, BYTES = OFF_X + 32 * 4;
    // two stages where a third CTA per SM still fits beside them
    static constexpr int COUNT = 2 * G_WARPS * BYTES <= 72 * 1024 ? 2 : 1;
};


struct Item {
    int tensor, tile, R, C, tr, tc, brow, col0, k, nb;      // brow: first row of band k of nb
    bool v8;
    __device__ __forceinline__ void decode(const StepArgs& a, const Work& w) {
        const CameTensorDesc& d = a.descs[w.tensor];
        const Scratch& s = a.scr[w.tensor];
        tensor = w.tensor; tile = w.tile;
        R = (int)d.rows; C = (int)d.cols;
        tr = w.tile / s.tiles_c; tc = w.tile - tr * s.tiles_c;
        brow = tr * s.g_nb * 16; col0 = tc * G_CW; k = 0;
        nb = min(s.g_nb, ((R - brow - 1) >> 4) + 1);
        v8 = s.g_v == 8;
    }
};

// The band's rows of an array of R x C elements of `esz` bytes (ESZ: the same, or 0 for a size known at run time).  Rows
// past the end are zero-filled; the columns past the end of a row are the next row's (the reader masks them).  A chunk may
// begin before the array or end behind it only inside the same 16 bytes, and of the last one only the array's bytes are
// read.  Whole bands away from the array's end need none of those tests, and rows on 16-byte boundaries no ninth chunk and
// no division (bf16: about 20 instructions a lane instead of 110, of the 250 to 900 that a band takes in a phase).
template <int ESZ>
__device__ __forceinline__ void stage_rows(char* dst, int pitch, const void* base, int esz, const Item& it, int lane) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(base);
    const uintptr_t first = b + (uintptr_t)(((int64_t)it.brow * it.C + it.col0) * esz);
    if constexpr (ESZ > 0) {
        constexpr int NCH = G_CW * ESZ / 16;
        if (it.R - it.brow >= 16 && it.C - it.col0 >= G_CW && it.C < (1 << 29)) {
            const int pitch_g = it.C * ESZ;      // (below 2^31: one multiplication to 64 bits per address)
            if (((first | (uintptr_t)pitch_g) & 15) == 0) {
                const int r = lane / NCH, ch = lane % NCH;
                const char* src = reinterpret_cast<const char*>(first) + (int64_t)r * pitch_g + 16 * ch;
                char* to = dst + r * pitch + 16 * ch;
#pragma unroll
                for (int k = 0; k < NCH / 2; ++k, src += (int64_t)(32 / NCH) * pitch_g, to += 32 / NCH * pitch) cp16(to, src, 16);
                return;
            }
            if (it.R - it.brow > 16) {      // (a row follows: the last chunk stays inside the array)
#pragma unroll
                for (int k = 0; k < (16 * (NCH + 1) + 31) / 32; ++k) {
                    const int j = lane + 32 * k, r = j / (NCH + 1), ch = j - r * (NCH + 1);
                    const uintptr_t src = ((first + (uintptr_t)((int64_t)r * pitch_g)) & ~(uintptr_t)15) + 16 * ch;
                    if (j < 16 * (NCH + 1)) cp16(dst + r * pitch + 16 * ch, reinterpret_cast<const void*>(src), 16);
                }
                return;
            }
        }
    }
    const int nch = G_CW / 16 * esz + 1, rows = min(16, it.R - it.brow), width = min(G_CW, it.C - it.col0) * esz;
    const uintptr_t end = b + (uintptr_t)((int64_t)it.R * it.C * esz);
    for (int j = lane; j < 16 * nch; j += 32) {
        const int r = j / nch, ch = j - r * nch;
        const uintptr_t row = first + (uintptr_t)((int64_t)r * it.C * esz), src = (row & ~(uintptr_t)15) + 16 * ch;
        const bool want = r < rows && src < row + width;
        cp16(dst + r * pitch + 16 * ch, reinterpret_cast<const void*>(want ? src : b & ~(uintptr_t)15),
             want ? (int)min((uintptr_t)16, end - src) : 0);
    }
}
// 16 row values from `v`, 64 column values from `c` (arrays of the workspace: 16-byte aligned, padded to 4 values)
__device__ __forceinline__ void stage_vectors(char* st, int off_v, int off_c, const float* v, const float* c, const Item& it, int lane) {
    if (lane < 16) {
        const int col = it.col0 + 4 * lane;
        cp16(st + off_c + 16 * lane, c + (col < it.C ? col : 0), col < it.C ? 16 : 0);
    } else if (lane < 20) {
        const int row = it.brow + 4 * (lane - 16);
        cp16(st + off_v + 16 * (lane - 16), v + (row < it.R ? row : 0), row < it.R ? 16 : 0);
    }
}
// tile layout: the absmax of the band's four tiles; flat layout: of the two flat blocks a row's columns may lie in
template <int MODE>
__device__ __forceinline__ void stage_absmax(char* x, const float* absmax, const Item& it, int lane) {
    if (MODE == CAME_MODE_TILE8) {
        const int tile_cols = ((it.C - 1) / TILE + 1), t = (it.col0 >> 4) + lane;
        if (lane < 4 && t < tile_cols) cp4(x + 4 * lane, absmax + (int64_t)(it.brow >> 4) * tile_cols + t);
    } else if (MODE == CAME_MODE_FLAT8) {
        const int row = min(it.brow + (lane >> 1), it.R - 1);
        const int64_t last = ((int64_t)it.R * it.C - 1) >> 8, blk = (((int64_t)row * it.C + it.col0) >> 8) + (lane & 1);
        cp4(x + 4 * lane, absmax + min(blk, last));
    }
}

// Walks a warp's items band by band: issue(item, stage) starts the copies of a band, proc(item, stage) computes it.
template <int STAGES, typename ISSUE, typename PROC>
__device__ __forceinline__ void stream(const StepArgs& a, const Work* list, int n, int first, int stride, ISSUE issue, PROC proc) {
    if (first >= n) return;
    Item it;
    it.decode(a, list[first]);
    issue(it, 0);
    cp_commit();
    Work ahead = list[min(first + stride, n - 1)];
    int st = 0;
    for (int i = first;;) {
        Item nx = it;
        bool more = true;
        if (++nx.k < it.nb) {
            nx.brow += 16;
        } else {
            i += stride;
            more = i < n;
            if (more) {
                nx.decode(a, ahead);
                ahead = list[min(i + stride, n - 1)];
            }
        }
        if (STAGES == 2) {
            if (more) issue(nx, st ^ 1);
            cp_commit();
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncwarp();
        proc(it, st);
        __syncwarp();      // the stage is read before it is filled again
        if (STAGES == 1 && more) { issue(nx, 0); cp_commit(); }
        if (!more) break;
        it = nx;
        if (STAGES == 2) st ^= 1;
    }
    cp_wait<0>();
}

// How a lane reads its part of a band.  V = 8: columns 8 (lane & 7) .. + 7 of rows (lane >> 3) + 4 i; V = 1: columns lane
// and lane + 32 of row i.
template <int V> struct Lane {
    static constexpr int NR = V == 8 ? 4 : 16, E = V == 8 ? 8 : 2;
    static __device__ __forceinline__ int row(int lane, int i) { return V == 8 ? (lane >> 3) + 4 * i : i; }
    static __device__ __forceinline__ int col(int lane, int e) { return V == 8 ? 8 * (lane & 7) + e : lane + 32 * e; }
};
// Elements of row r of a staged array; `low`: byte offset of the row's first element from a 16-byte boundary
template <int V, typename T>
__device__ __forceinline__ void read_row(const char* rows, int pitch, int dt, int low, int r, int lane, float* x) {
    const Buf<T> b(rows + r * pitch + (V == 8 ? 0 : low), dt);
    if constexpr (V == 8) b.get8(8 * (lane & 7), x);
    else { x[0] = b.get(lane); x[1] = b.get(lane + 32); }
}
template <int V>
__device__ __forceinline__ void read_codes(const char* rows, int pitch, int low, int r, int lane, float* x) {
    if constexpr (V == 8) {
        const uint2 q = *reinterpret_cast<const uint2*>(rows + r * pitch + low + 8 * (lane & 7));
        const uint32_t w[2] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u};
#pragma unroll
        for (int e = 0; e < 8; e += 2) { const u64 f = codes_to_f2(w[e >> 2], e & 3); x[e] = f.x; x[e + 1] = f.y; }
    } else {
        const signed char* p = reinterpret_cast<const signed char*>(rows + r * pitch + low);
        x[0] = (float)p[lane]; x[1] = (float)p[lane + 32];
    }
}
// offset of a band's first row from a 16-byte boundary, and what the offset grows by per row, modulo 16
__device__ __forceinline__ int low_bits(const void* base, const Item& it, int esz) {
    return (int)((reinterpret_cast<uintptr_t>(base) + (uintptr_t)(((int64_t)it.brow * it.C + it.col0) * esz)) & 15);
}

__device__ __forceinline__ int low_step(const Item& it, int esz) { return (int)(((uint32_t)it.C * (uint32_t)esz) & 15u); }

// Squares of a pair added to a row's sum: V = 8 two chains, V = 1 (one pair a row) one chain in .x
template <int V> __device__ __forceinline__ u64 add_squares(const u64& y, const u64& sum) {
    if (V == 8) return fma2(y, y, sum);
    return pk(fmaf(y.y, y.y, fmaf(y.x, y.x, sum.x)), 0.0f);
}
// Sums over a row's lanes of the NR row values a lane holds -> the band's row partials.  Halving butterfly: each step
// exchanges half of the rows.
template <int V>
__device__ __forceinline__ void band_row_sums(const Item& it, float* rowpart, float* rs, int lane) {
    int o = V == 8 ? 4 : 16;
#pragma unroll
    for (int h = Lane<V>::NR / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float send = up ? rs[k] : rs[k + h], keep = up ? rs[k + h] : rs[k];
            rs[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    const float v = rs[0] + __shfl_xor_sync(0xffffffffu, rs[0], 1);
    const int row = it.brow + (V == 8 ? (lane >> 3) + 4 * ((lane >> 1) & 3) : lane >> 1);
    if ((lane & 1) == 0 && row < it.R) rowpart[(int64_t)it.tc * it.R + row] = v;
}
template <int V>
__device__ __forceinline__ void tile_col_sums(const Item& it, float* colpart, const u64* pairs, int lane) {
    float* dst = colpart + (int64_t)it.tr * it.C + it.col0;
    float acc[Lane<V>::E];
#pragma unroll
    for (int e = 0; e < Lane<V>::E / 2; ++e) upk(pairs[e], acc[2 * e], acc[2 * e + 1]);
    if constexpr (V == 8) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 8);
            acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
        }
        if (lane < 8 && it.col0 + 8 * lane < it.C) store_run<8>(dst + 8 * lane, acc);
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (it.col0 + lane + 32 * e < it.C) dst[lane + 32 * e] = acc[e];
    }
}
// Row factors 1 / sqrt(v_i / mean) times `mul` of a band: lane l < 16 has the one of row l (0 past the end).
__device__ __forceinline__ float band_row_factor(const Item& it, const float* v, float mean, bool clamp, float mul, int lane) {
    if (it.brow + (lane & 15) >= it.R) return 0.0f;
    const float x = v[lane & 15];
    float ratio = mean > 1e-30f && mean < 1e30f ? div_by(x, mean, 1.0f / mean) : x / mean;
    if (clamp) ratio = fmaxf(ratio, 1e-30f);
    return inv_sqrt(ratio) * mul;
}
// column factors of a lane (0 past the end: those columns then take no part in anything)
template <int V>
__device__ __forceinline__ void band_col_factors(const Item& it, const float* c, int lane, u64* cf) {
#pragma unroll
    for (int e = 0; e < Lane<V>::E; e += 2) {
        const int c0 = Lane<V>::col(lane, e), c1 = Lane<V>::col(lane, e + 1);
        cf[e / 2] = pk(it.col0 + c0 < it.C ? c[c0] : 0.0f, it.col0 + c1 < it.C ? c[c1] : 0.0f);
    }
}

// ---- S1 -------------------------------------------------------------------------------------------------------
template <typename TG, int V>
__device__ __forceinline__ void band_sq(const StepArgs& a, const CameHyper* hyp, const Item& it, const char* st, int pitch, u64* colacc, float& gs) {
    constexpr int NR = Lane<V>::NR, E = Lane<V>::E;
    const CameTensorDesc& d = a.descs[it.tensor];
    const int lane = threadIdx.x & 31, esz = size_of<TG>(d.g_dtype), dt = d.g_dtype;
    const int low = low_bits(d.g, it, esz), grow = low_step(it, esz);
    if (it.k == 0) gs = hyp[d.group].grad_scale;
    const u64 scale = splat(gs);      // (before the square: unscaled gradients may be too large or too small for one)
    float rs[NR];
    if (it.k == 0)
#pragma unroll
        for (int e = 0; e < E / 2; ++e) colacc[e] = F2ZERO;
    // What lies past the end of a row: zeros from the staging, except that for V = 1 its last 16 bytes may hold elements of
    // the next row, which a band that ends there masks.
    auto rows = [&](auto ends_here) {
        bool in[2] = {true, true};
        if constexpr (decltype(ends_here)::value) { in[0] = it.col0 + lane < it.C; in[1] = it.col0 + lane + 32 < it.C; }
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = Lane<V>::row(lane, i);
            float x[E];
            read_row<V, TG>(st, pitch, dt, (low + r * grow) & 15, r, lane, x);
            u64 sum = F2ZERO;
#pragma unroll
            for (int e = 0; e < E; e += 2) {
                const u64 y = mul2(pk(in[0] ? x[e] : 0.0f, in[1] ? x[e + 1] : 0.0f), scale);
                sum = add_squares<V>(y, sum);
                colacc[e / 2] = fma2(y, y, colacc[e / 2]);
            }
            rs[i] = V == 8 ? sum.x + sum.y : sum.x;
        }
    };
    if (V == 8 || it.C - it.col0 >= G_CW) rows(std::false_type{});
    else rows(std::true_type{});
    const Scratch& s = a.scr[it.tensor];
    float* colpart = s.colpart;
    band_row_sums<V>(it, s.rowpart, rs, lane);
    if (it.k == it.nb - 1) tile_col_sums<V>(it, colpart, colacc, lane);
}

// ---- S2 -------------------------------------------------------------------------------------------------------
template <typename TG, typename S, int V>
__device__ __forceinline__ void band_clip(const StepArgs& a, const CameHyper* hyp, const Item& it, const char* st, float& acc, float& mean, float& gs) {
    constexpr int NR = Lane<V>::NR, E = Lane<V>::E;
    const CameTensorDesc& d = a.descs[it.tensor];
    const Scratch& s = a.scr[it.tensor];
    const int lane = threadIdx.x & 31, esz = size_of<TG>(d.g_dtype), dt = d.g_dtype;
    const int low = low_bits(d.g, it, esz), grow = low_step(it, esz);
    if (it.k == 0) {
        acc = 0.0f;
        gs = hyp[d.group].grad_scale;
        mean = read_mean(s.rowblk, s.nbR, it.R, d.flags & CAME_F_SQ_FIX, d.flags & CAME_F_SQ_CLAMP, lane);
    }
    // (the gradient scale rides on the row factors)
    const float f = band_row_factor(it, reinterpret_cast<const float*>(st + S::OFF_V), mean, d.flags & CAME_F_SQ_CLAMP, gs, lane);
    u64 cf[E / 2], sum = F2ZERO;
    band_col_factors<V>(it, reinterpret_cast<const float*>(st + S::OFF_C), lane, cf);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int r = Lane<V>::row(lane, i);
        const u64 rf = splat(__shfl_sync(0xffffffffu, f, r));
        float x[E];
        read_row<V, TG>(st, S::PA, dt, (low + r * grow) & 15, r, lane, x);
#pragma unroll
        for (int e = 0; e < E; e += 2) {
            const u64 u = mul2(mul2(pk(x[e], x[e + 1]), rf), cf[e / 2]);
            sum = fma2(u, u, sum);
        }
    }
    acc += sum.x + sum.y;
    if (s.fac && it.tc == 0 && lane < 16 && it.brow + lane < it.R) s.fac[it.brow + lane] = f;      // for the flat apply phase
    if (it.k == it.nb - 1) leave_partial(s.spart, s.counters, it.tile, s.tiles_r * s.tiles_c, warp_sum(acc), lane);
}
// 1 / clip divisor, clip = max(1, sqrt(S/n)/clip_threshold) (came_kernels.cu:2619-2620)
__device__ __forceinline__ float read_inv_clip(const Scratch& s, const CameHyper& h, int64_t n, int lane) {
    return 1.0f / fmaxf(1.0f, sqrtf(read_sum(s.spart, s.tiles_r * s.tiles_c, lane) / (float)n) / h.clip_threshold);
}

// ---- M --------------------------------------------------------------------------------------------------------
// u = g r c / clip, m = beta1 m + (1 - beta1) u, sums of (u - m)^2 (eps1 is added when the partials are finalised).
// tile layout (came_kernels.cu:2584-2683): m re-quantised per 16 x 16 tile; fp32 (came_kernels.cu:2307-2342): m written;
// flat layout: nothing written, the apply phase forms m again (came_kernels.cu:2246-2305 keeps it in fp32 scratch)
template <typename TG, int MODE, int V>
__device__ __forceinline__ void band_moment(const StepArgs& a, const CameHyper* hyp, const Item& it, const char* st, u64* colacc, float& mean,
                                            float& inv_clip, float& gs) {
    using S = Stage<TG, MODE>;
    constexpr int NR = Lane<V>::NR, E = Lane<V>::E;
    const CameTensorDesc& d = a.descs[it.tensor];
    const Scratch& s = a.scr[it.tensor];
    const int lane = threadIdx.x & 31, esz = size_of<TG>(d.g_dtype), dt = d.g_dtype, msz = MODE == CAME_MODE_FP32 ? 4 : 1;
    const int low = low_bits(d.g, it, esz), grow = low_step(it, esz), mlow = low_bits(d.m, it, msz), mgrow = low_step(it, msz);
    const float beta1 = hyp[d.group].beta1, om1 = hyp[d.group].om_beta1;
    if (it.k == 0) {
        mean = read_mean(s.rowblk, s.nbR, it.R, d.flags & CAME_F_SQ_FIX, d.flags & CAME_F_SQ_CLAMP, lane);
        inv_clip = read_inv_clip(s, hyp[d.group], (int64_t)it.R * it.C, lane);
        gs = hyp[d.group].grad_scale;
    }
    const float f = band_row_factor(it, reinterpret_cast<const float*>(st + S::OFF_V), mean, d.flags & CAME_F_SQ_CLAMP, gs, lane);
    const float* xs = reinterpret_cast<const float*>(st + S::OFF_X);
    char* const m_base = reinterpret_cast<char*>(d.m);
    float* const absmax = d.m_absmax;
    float* const rowpart = s.rowpart;
    float* const colpart = s.colpart;
    u64 cf[E / 2];
    float m[NR][E], rs[NR], amax[V == 8 ? 1 : 2], sc[V == 8 ? 1 : 2];
    bool in[V == 8 ? 1 : 2];
    band_col_factors<V>(it, reinterpret_cast<const float*>(st + S::OFF_C), lane, cf);
#pragma unroll
    for (int q = 0; q < (V == 8 ? 1 : 2); ++q) in[q] = it.col0 + Lane<V>::col(lane, q) < it.C;
    if (it.k == 0)
#pragma unroll
        for (int e = 0; e < E / 2; ++e) colacc[e] = F2ZERO;
    const u64 b2 = splat(beta1), o2 = splat(om1), clip2 = splat(inv_clip);
    const float dq = MODE == CAME_MODE_FLAT8 ? xs[lane] / QMAX_I8 : 0.0f;      // of the two blocks of row lane / 2
#pragma unroll
    for (int q = 0; q < (V == 8 ? 1 : 2); ++q) {
        amax[q] = 0.0f;
        if (MODE == CAME_MODE_TILE8) {
            const float A = in[q] ? xs[V == 8 ? (lane & 7) >> 1 : (lane >> 4) + 2 * q] : 0.0f;
            sc[q] = A > 0.0f ? A / QMAX_I8 : 0.0f;
        }
    }
    // (past the end of the matrix g is masked by its factors, m by a zero scale: u = m = 0, nothing enters the sums)
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int r = Lane<V>::row(lane, i);
        const u64 rf = splat(__shfl_sync(0xffffffffu, f, r));
        float x[E];
        read_row<V, TG>(st, S::PA, dt, (low + r * grow) & 15, r, lane, x);
        if constexpr (MODE == CAME_MODE_FP32) read_row<V, float>(st + S::OFF_M, S::PM, 0, (mlow + r * mgrow) & 15, r, lane, m[i]);
        else read_codes<V>(st + S::OFF_M, S::PM, (mlow + r * mgrow) & 15, r, lane, m[i]);
        float fs[2];
        if (MODE == CAME_MODE_FLAT8) { fs[0] = __shfl_sync(0xffffffffu, dq, 2 * r); fs[1] = __shfl_sync(0xffffffffu, dq, 2 * r + 1); }
        const uint32_t o8 = MODE == CAME_MODE_FLAT8 ? (uint32_t)(((uint32_t)(it.brow + r) * (uint32_t)it.C + (uint32_t)it.col0) & 255u) : 0u;
        u64 sum = F2ZERO;
#pragma unroll
        for (int e = 0; e < E; e += 2) {
            const u64 u = mul2(mul2(mul2(pk(x[e], x[e + 1]), rf), cf[e / 2]), clip2);
            u64 mo = pk(m[i][e], m[i][e + 1]);
            constexpr int Q1 = V == 8 ? 0 : 1;      // the second of a pair: V = 1 another tile, 32 columns on
            if (MODE == CAME_MODE_TILE8) mo = mul2(mo, pk(sc[0], sc[Q1]));
            else if (MODE == CAME_MODE_FLAT8) {      // V = 8: a lane's columns lie in one block
                const uint32_t c0 = Lane<V>::col(lane, V == 8 ? 0 : e), c1 = Lane<V>::col(lane, V == 8 ? 0 : e + 1);
                mo = mul2(mo, pk(!in[0] ? 0.0f : o8 + c0 < 256u ? fs[0] : fs[1], !in[Q1] ? 0.0f : o8 + c1 < 256u ? fs[0] : fs[1]));
            }
            else { if (!in[0]) mo.x = 0.0f; if (!in[Q1]) mo.y = 0.0f; }
            const u64 mn = fma2(mo, b2, mul2(o2, u)), df = sub2(u, mn);      // the reference's order
            sum = add_squares<V>(df, sum);
            colacc[e / 2] = fma2(df, df, colacc[e / 2]);
            m[i][e] = mn.x; m[i][e + 1] = mn.y;
            if (MODE == CAME_MODE_TILE8) { amax[0] = fmaxf(amax[0], fabsf(mn.x)); amax[Q1] = fmaxf(amax[Q1], fabsf(mn.y)); }
        }
        rs[i] = V == 8 ? sum.x + sum.y : sum.x;
    }
    const int64_t at = ((int64_t)it.brow * it.C + it.col0);
    const int live = it.R - it.brow;
    if (MODE == CAME_MODE_TILE8) {
        float q127[V == 8 ? 1 : 2];
        const int tile_cols = ((it.C - 1) / TILE + 1);
#pragma unroll
        for (int q = 0; q < (V == 8 ? 1 : 2); ++q) {
            float A = amax[q];
            if (V == 8) {
                A = fmaxf(A, __shfl_xor_sync(0xffffffffu, A, 1));
                A = fmaxf(A, __shfl_xor_sync(0xffffffffu, A, 8));
                A = fmaxf(A, __shfl_xor_sync(0xffffffffu, A, 16));
            } else {
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) A = fmaxf(A, __shfl_xor_sync(0xffffffffu, A, o));
            }
            A = fix_absmax(A);
            // one lane per tile: the one that holds its first row and column
            if (in[q] && (V == 8 ? (lane & 0x19) == 0 : (lane & 15) == 0))
                absmax[(int64_t)(it.brow >> 4) * tile_cols + (it.col0 >> 4) + (V == 8 ? (lane & 7) >> 1 : (lane >> 4) + 2 * q)] = A;
            // 127 / A overflows below 4e-37: there m and A are first scaled by 2^64 (exact)
            q127[q] = QMAX_I8 / A;
            if (__any_sync(0xffffffffu, A < 4e-37f)) {
                const float up = A < 4e-37f ? 18446744073709551616.0f : 1.0f;
                q127[q] = QMAX_I8 / (A * up);
#pragma unroll
                for (int i = 0; i < NR; ++i)
#pragma unroll
                    for (int e = 0; e < E; ++e)
                        if (V == 8 || e == q) m[i][e] *= up;
            }
        }
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = Lane<V>::row(lane, i);
            int8_t* dst = reinterpret_cast<int8_t*>(m_base) + at + (int64_t)r * it.C + Lane<V>::col(lane, 0);
            // The low byte of m * (127 / A) + 1.5 * 2^23 is the code (see fast_tile8.cu).  Of 26 M random values 20 do not get
            // the code nearest to the 64-bit quotient (rounded quotient times 127: 38).
            uint32_t y[E];
#pragma unroll
            for (int e = 0; e < E; e += 2) {
                const u64 t = fma2(pk(m[i][e], m[i][e + 1]), pk(q127[0], q127[V == 8 ? 0 : 1]), splat(ROUND_MAGIC));
                y[e] = __float_as_uint(t.x); y[e + 1] = __float_as_uint(t.y);
            }
            if constexpr (V == 8) {
                if (r < live && in[0])
                    *reinterpret_cast<uint2*>(dst) = make_uint2(__byte_perm(__byte_perm(y[0], y[1], 0x0040u), __byte_perm(y[2], y[3], 0x0040u), 0x5410u),
                                                                __byte_perm(__byte_perm(y[4], y[5], 0x0040u), __byte_perm(y[6], y[7], 0x0040u), 0x5410u));
            } else {
                if (r < live && in[0]) dst[0] = (int8_t)y[0];
                if (r < live && in[1]) dst[32] = (int8_t)y[1];
            }
        }
    } else if (MODE == CAME_MODE_FP32) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = Lane<V>::row(lane, i);
            float* dst = reinterpret_cast<float*>(m_base) + at + (int64_t)r * it.C + Lane<V>::col(lane, 0);
            if constexpr (V == 8) {
                if (r < live && in[0]) store_run<8>(dst, m[i]);
            } else {
                if (r < live && in[0]) dst[0] = m[i][0];
                if (r < live && in[1]) dst[32] = m[i][1];
            }
        }
    }
    band_row_sums<V>(it, rowpart, rs, lane);
    if (it.k == it.nb - 1) tile_col_sums<V>(it, colpart, colacc, lane);
}

// ---- A --------------------------------------------------------------------------------------------------------
template <typename TP>
__device__ __forceinline__ float g_apply_one(const Buf<TP>& b, float pv, float upd, const CameHyper& h, int wd) {
    return apply_step(pv, upd, h.lr, h.wd_lr, h.decay_mul, wd, [&](float x) { return b.round(x); });
}

// peers that receive a tensor's new values (push mode)
__device__ __forceinline__ int peers_of(const StepArgs& a, const CameTensorDesc& d, int esz) {
    if (a.n_push == 0) return 0;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(d.p);
    return lo >= a.push_lo && lo + (uintptr_t)(d.rows * d.cols * esz) <= a.push_hi ? a.n_push : 0;
}

// p -= lr m R'_i C'_j with m read back from the state (came_kernels.cu:3332-3366, 2487-2511)
template <typename TP, int MODE, int V>
__device__ __forceinline__ void band_apply(const StepArgs& a, const CameHyper* hyp, const Item& it, const char* st, float& mean) {
    using S = Stage<TP, MODE>;
    constexpr int NR = Lane<V>::NR, E = Lane<V>::E;
    const CameTensorDesc& d = a.descs[it.tensor];
    const Scratch& s = a.scr[it.tensor];
    const CameHyper h = hyp[d.group];      // (a copy: the stores below could alias the table)
    const int lane = threadIdx.x & 31, esz = size_of<TP>(d.p_dtype), dt = d.p_dtype, msz = MODE == CAME_MODE_FP32 ? 4 : 1;
    const int low = low_bits(d.p, it, esz), grow = low_step(it, esz), mlow = low_bits(d.m, it, msz), mgrow = low_step(it, msz);
    const int wd = wd_form(h, d.flags);
    if (it.k == 0) mean = read_mean(s.rowblk2, s.nbR, it.R, d.flags & CAME_F_RESROW_FIX, d.flags & CAME_F_RESROW_CLAMP, lane);
    const float f = band_row_factor(it, reinterpret_cast<const float*>(st + S::OFF_V), mean, d.flags & CAME_F_RESROW_CLAMP, 1.0f, lane);
    const float* xs = reinterpret_cast<const float*>(st + S::OFF_X);
    u64 cf[E / 2];
    float sc[V == 8 ? 1 : 2];
    bool in[V == 8 ? 1 : 2];
    band_col_factors<V>(it, reinterpret_cast<const float*>(st + S::OFF_C), lane, cf);
#pragma unroll
    for (int q = 0; q < (V == 8 ? 1 : 2); ++q) {
        in[q] = it.col0 + Lane<V>::col(lane, q) < it.C;
        sc[q] = 1.0f;
        if (MODE == CAME_MODE_TILE8) {
            const float A = in[q] ? xs[V == 8 ? (lane & 7) >> 1 : (lane >> 4) + 2 * q] : 0.0f;
            sc[q] = A > 0.0f ? A / QMAX_I8 : 0.0f;
        }
    }
    // decay as one packed operation k p + base (apply_step's forms: 0 and 2 multiply, 1 and 3 subtract; x + -0 is x)
    const bool subtract = wd & 1;
    const u64 k2 = splat(subtract ? -h.wd_lr : wd == 2 ? h.decay_mul : 1.0f), lr2 = splat(-h.lr);
    const Buf<TP> p(d.p, dt);
    const int64_t at = (int64_t)it.brow * it.C + it.col0 + Lane<V>::col(lane, 0);
    const int live = it.R - it.brow, n_push = peers_of(a, d, esz);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int r = Lane<V>::row(lane, i);
        const float rf = __shfl_sync(0xffffffffu, f, r);
        float x[E], m[E];
        read_row<V, TP>(st, S::PA, dt, (low + r * grow) & 15, r, lane, x);
        if constexpr (MODE == CAME_MODE_FP32) read_row<V, float>(st + S::OFF_M, S::PM, 0, (mlow + r * mgrow) & 15, r, lane, m);
        else read_codes<V>(st + S::OFF_M, S::PM, (mlow + r * mgrow) & 15, r, lane, m);
#pragma unroll
        for (int e = 0; e < E; e += 2) {
            const u64 pv = pk(x[e], x[e + 1]);
            const u64 t = fma2(k2, pv, subtract ? pv : splat(-0.0f));
            x[e] = t.x; x[e + 1] = t.y;
        }
        if (wd >= 2)
#pragma unroll
            for (int e = 0; e < E; ++e) x[e] = p.round(x[e]);
#pragma unroll
        for (int e = 0; e < E; e += 2) {
            const u64 upd = mul2(mul2(pk(m[e], m[e + 1]), pk(rf * sc[0], rf * sc[V == 8 ? 0 : 1])), cf[e / 2]);
            const u64 t = fma2(lr2, upd, pk(x[e], x[e + 1]));
            x[e] = t.x; x[e + 1] = t.y;
        }
        const int64_t o = at + (int64_t)r * it.C;
        if (r < live) {
            if constexpr (V == 8) {
                if (in[0]) p.put8(o, x);
                if (n_push && in[0])
                    for (int q = 0; q < n_push; ++q) p.put8(o, x, a.push_delta[q]);
            } else {
                if (in[0]) p.put(o, x[0]);
                if (in[1]) p.put(o + 32, x[1]);
                if (n_push)
                    for (int q = 0; q < n_push; ++q) {
                        if (in[0]) p.put(o, x[0], a.push_delta[q]);
                        if (in[1]) p.put(o + 32, x[1], a.push_delta[q]);
                    }
            }
        }
    }
}

// flat layout: a warp owns a block of 256 consecutive elements, whatever rows they belong to (the un-quantised momentum
// feeds the update: came_kernels.cu:2246-2305, 2487-2511).  The blocks of g, p and the codes come to the warp's shared
// memory, in the room its bands had, some blocks ahead; buffers off the 16-byte boundary are read where they are.
template <typename T, int MODE> struct FlatSlot {
    static constexpr int ESZ = Size<T>::BYTES, OFF_P = QBLOCK * ESZ, OFF_M = 2 * OFF_P, OFF_X = OFF_M + QBLOCK, BYTES = OFF_X + 16;
    static constexpr int ROOM = Stage<T, MODE>::COUNT * Stage<T, MODE>::BYTES / BYTES, COUNT = ROOM < 4 ? ROOM : 4;
    static_assert(COUNT >= 2, "a block is computed while the next is on its way");
};
__device__ __forceinline__ bool flat_staged(const CameTensorDesc& d) {
    return ((reinterpret_cast<uintptr_t>(d.g) | reinterpret_cast<uintptr_t>(d.p) | reinterpret_cast<uintptr_t>(d.m)) & 15) == 0;
}
template <typename TG, typename TP, typename S>
__device__ __forceinline__ void issue_flat(const StepArgs& a, const Work& w, char* slot, int lane) {
    const CameTensorDesc& d = a.descs[w.tensor];
    if (!flat_staged(d)) return;
    const int64_t i0 = (int64_t)w.tile * QBLOCK;
    const int cnt = (int)min((int64_t)QBLOCK, d.rows * d.cols - i0);
    auto rows = [&](char* dst, const void* base, int esz) {
        const char* src = reinterpret_cast<const char*>(base) + i0 * esz;
        for (int j = 16 * lane; j < cnt * esz; j += 512) cp16(dst + j, src + j, min(16, cnt * esz - j));
    };
    rows(slot, d.g, size_of<TG>(d.g_dtype));
    rows(slot + S::OFF_P, d.p, size_of<TP>(d.p_dtype));
    rows(slot + S::OFF_M, d.m, 1);
    if (lane == 0) cp4(slot + S::OFF_X, d.m_absmax + w.tile);
}
struct FlatTensor {      // what a warp's blocks of one tensor share: formed once, not per block of 8 elements per lane
    int tensor = -1, n_push;
    float inv_clip, mean, inv;
    __device__ __forceinline__ void use(const StepArgs& a, const CameHyper* hyp, int t, int p_size, int lane) {
        if (t == tensor) return;
        tensor = t;
        const CameTensorDesc& d = a.descs[t];
        const Scratch& s = a.scr[t];
        inv_clip = read_inv_clip(s, hyp[d.group], d.rows * d.cols, lane);
        mean = read_mean(s.rowblk2, s.nbR, (int)d.rows, d.flags & CAME_F_RESROW_FIX, d.flags & CAME_F_RESROW_CLAMP, lane);
        inv = 1.0f / mean;
        n_push = peers_of(a, d, p_size);
    }
};
template <typename TG, typename TP, typename S, int V>
__device__ __forceinline__ void phase_apply_flat(const StepArgs& a, const CameHyper* hyp, const Work& w, const FlatTensor& ft, const char* slot) {
    const CameTensorDesc d = a.descs[w.tensor];
    const Scratch s = a.scr[w.tensor];
    const CameHyper h = hyp[d.group];
    const int lane = threadIdx.x & 31, C = (int)d.cols, blk = w.tile;
    const int64_t n = d.rows * d.cols, b0 = (int64_t)blk * QBLOCK;
    const int wd = wd_form(h, d.flags);
    const float inv_clip = ft.inv_clip, mean = ft.mean, inv = ft.inv;
    const bool clamp = d.flags & CAME_F_RESROW_CLAMP, easy = mean > 1e-30f && mean < 1e30f;
    int8_t* mq = reinterpret_cast<int8_t*>(d.m);
    const Buf<TP> p(d.p, d.p_dtype);
    // the block's elements: in the slot, or where they lie (V = 8: always in the slot)
    const bool staged = V == 8 || flat_staged(d);
    const Buf<TG> gs(staged ? slot : reinterpret_cast<const char*>(d.g) + b0 * size_of<TG>(d.g_dtype), d.g_dtype);
    const Buf<TP> ps(staged ? slot + S::OFF_P : reinterpret_cast<const char*>(d.p) + b0 * size_of<TP>(d.p_dtype), d.p_dtype);
    const int8_t* ms = staged ? reinterpret_cast<const int8_t*>(slot + S::OFF_M) : mq + b0;
    const int j0 = V == 8 ? 8 * lane : lane;
    const int64_t i0 = b0 + j0;
    float x[8], m[8], pv[8];
    int cnt;      // elements of this lane (they end where the tensor does)
    if (V == 8) {
        cnt = i0 >= n ? 0 : 8;      // n is a multiple of 8
        if (cnt) {
            gs.get8(j0, x);
            ps.get8(j0, pv);
            const uint2 r = *reinterpret_cast<const uint2*>(ms + j0);
            const uint32_t y[2] = {r.x ^ 0x80808080u, r.y ^ 0x80808080u};
#pragma unroll
            for (int e = 0; e < 8; e += 2) { const u64 f = codes_to_f2(y[e >> 2], e & 3); m[e] = f.x; m[e + 1] = f.y; }
        }
    } else {
        cnt = i0 >= n ? 0 : (int)min((int64_t)8, (n - i0 + 31) >> 5);
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e < cnt) { x[e] = gs.get(j0 + 32 * e); pv[e] = ps.get(j0 + 32 * e); m[e] = (float)ms[j0 + 32 * e]; }
    }
    const float sc = (staged ? *reinterpret_cast<const float*>(slot + S::OFF_X) : __ldcg(d.m_absmax + blk)) / QMAX_I8;
    // (plain loads of the factors: the grid barriers order them behind other SMs' stores, and lines are used many times)
    float upd[8], amax = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        upd[e] = 0.0f;
        if (e >= cnt) { x[e] = 0.0f; m[e] = 0.0f; pv[e] = 0.0f; }
    }
    auto row_factors = [&](int row, float& r, float& rr) {
        r = s.fac[row];
        const float y = s.Rr[row];
        float ratio = easy ? div_by(y, mean, inv) : y / mean;
        if (clamp) ratio = fmaxf(ratio, 1e-30f);
        rr = inv_sqrt(ratio);
    };
    // elements e and e + 1 (past the tensor's end g = m = 0 and the factors are 0: no part in anything)
    const u64 clip2 = splat(inv_clip), sc2 = splat(sc), b2 = splat(h.beta1), o2 = splat(h.om_beta1);
    auto pair = [&](int e, u64 r, u64 rr, u64 c, u64 rc) {
        const u64 u = mul2(mul2(mul2(pk(x[e], x[e + 1]), r), c), clip2);
        const u64 mn = fma2(mul2(pk(m[e], m[e + 1]), sc2), b2, mul2(o2, u));
        const u64 up = mul2(mul2(mn, rr), rc);
        amax = fmaxf(amax, fmaxf(fabsf(mn.x), fabsf(mn.y)));
        m[e] = mn.x; m[e + 1] = mn.y; upd[e] = up.x; upd[e + 1] = up.y;
    };
    // row and column of an element (most tensors: a 32-bit division)
    auto locate = [&](int64_t i, int& row, int& col) {
        if (n < 0x7fffffff) { row = (int)((uint32_t)i / (uint32_t)C); col = (int)i - row * C; }
        else { row = (int)(i / C); col = (int)(i - (int64_t)row * C); }
    };
    int row, col;
    if (V == 8) {      // the columns are a multiple of 8: a lane's elements lie in one row
        if (cnt) {
            float r, rr, c[8], rc[8];
            locate(i0, row, col);
            row_factors(row, r, rr);
            load_run<8>(s.vc + col, c);
            load_run<8>(s.Rc + col, rc);
#pragma unroll
            for (int e = 0; e < 8; e += 2) pair(e, splat(r), splat(rr), pk(c[e], c[e + 1]), pk(rc[e], rc[e + 1]));
        }
    } else {
        float r[8], rr[8], c[8], rc[8];
        if (C >= 32) {
            // The block lies in at most nine rows: lane l forms the factors of the l-th of them, the elements get them by
            // shuffles, and no column factor's load waits for a test for a new row.
            locate(b0, row, col);
            float fr, frr;
            row_factors(row + min(lane, (int)d.rows - 1 - row), fr, frr);
            uint32_t at = (uint32_t)col + (uint32_t)lane, k = at / (uint32_t)C;
            at -= k * (uint32_t)C;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                r[e] = __shfl_sync(0xffffffffu, fr, k);
                rr[e] = __shfl_sync(0xffffffffu, frr, k);
                c[e] = e < cnt ? s.vc[at] : 0.0f;
                rc[e] = e < cnt ? s.Rc[at] : 0.0f;
                at += 32;
                if (at >= (uint32_t)C) { at -= (uint32_t)C; ++k; }
            }
        } else {
            int have = -1;      // row the factors r, rr belong to
            locate(i0, row, col);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                r[e] = rr[e] = c[e] = rc[e] = 0.0f;
                if (e < cnt) {
                    if (row != have) { have = row; row_factors(row, r[e], rr[e]); }
                    else { r[e] = r[e ? e - 1 : 0]; rr[e] = rr[e ? e - 1 : 0]; }
                    c[e] = s.vc[col];
                    rc[e] = s.Rc[col];
                    col += 32;
                    while (col >= C) { col -= C; ++row; }
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) pair(e, pk(r[e], r[e + 1]), pk(rr[e], rr[e + 1]), pk(c[e], c[e + 1]), pk(rc[e], rc[e + 1]));
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e >= cnt) m[e] = 0.0f;
    }
    const float A = fix_absmax(warp_max(amax));
    if (lane == 0) d.m_absmax[blk] = A;      // (every lane has read the old value: the reduction is behind them)
    uint32_t lo, hi;
    if (recip_safe(A)) {      // the low byte of m * (127 / A) + 1.5 * 2^23 is the code (as in the fused kernel)
        const u64 s127 = splat(QMAX_I8 / A), magic = splat(ROUND_MAGIC);
        u64 y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = fma2(pk(m[2 * e], m[2 * e + 1]), s127, magic);
        lo = pack_codes4(y[0], y[1]);
        hi = pack_codes4(y[2], y[3]);
    } else {
        const float scale = quant_scale<true>(A);
        lo = quant_pack4<true>(make_float4(m[0], m[1], m[2], m[3]), A, scale);
        hi = quant_pack4<true>(make_float4(m[4], m[5], m[6], m[7]), A, scale);
    }
    // decay as in band_apply
    const bool subtract = wd & 1;
    const u64 k2 = splat(subtract ? -h.wd_lr : wd == 2 ? h.decay_mul : 1.0f), lr2 = splat(-h.lr);
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        const u64 q = pk(pv[e], pv[e + 1]), t = fma2(k2, q, subtract ? q : splat(-0.0f));
        pv[e] = t.x; pv[e + 1] = t.y;
    }
    if (wd >= 2)
#pragma unroll
        for (int e = 0; e < 8; ++e) pv[e] = p.round(pv[e]);
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        const u64 t = fma2(lr2, pk(upd[e], upd[e + 1]), pk(pv[e], pv[e + 1]));
        pv[e] = t.x; pv[e + 1] = t.y;
    }
    if (V == 8) {
        if (cnt) {
            *reinterpret_cast<uint2*>(mq + i0) = make_uint2(lo, hi);
            p.put8(i0, pv);
            for (int k = 0; k < ft.n_push; ++k) p.put8(i0, pv, a.push_delta[k]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e < cnt) {
                mq[i0 + 32 * e] = (int8_t)((e < 4 ? lo : hi) >> (8 * (e & 3)));
                p.put(i0 + 32 * e, pv[e]);
                for (int k = 0; k < ft.n_push; ++k) p.put(i0 + 32 * e, pv[e], a.push_delta[k]);
            }
    }
}

// ---- F1 / F2 ------------------------------------------------------------------------------------------------------
// One block of 256 entries of a row or column vector, by a CTA: partials -> EMA with the dequantised old state ->
// requantised state, fresh fp32 row values / column factors, the sum of a row block
// (came_kernels.cu:77-93, 215-242, 298-333, 2685-2706, 2742-2779).  Warp w adds the partials w, w + 8, ... of all 256
// entries, then thread t has entry t: one entry per thread keeps the code short, and cold code is what takes the time
// (8 entries per lane of one warp: 5 us a block, like this 2 us).
template <bool RES>
__device__ __forceinline__ void phase_finalize(const StepArgs& a, const CameHyper* hyp, const Work& w, GShared& sh) {
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    const CameHyper& h = hyp[d.group];
    const int R = (int)d.rows, C = (int)d.cols, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool is_col = w.tile >= s.nbR, quant = d.mode != CAME_MODE_FP32;
    const int b = is_col ? w.tile - s.nbR : w.tile, n = is_col ? C : R, idx = b * QBLOCK + threadIdx.x;
    const int parts = is_col ? s.tiles_r : s.tiles_c;
    const float* part = (is_col ? s.colpart : s.rowpart) + b * QBLOCK + lane;
    void* state = RES ? (is_col ? d.res_col : d.res_row) : (is_col ? d.sq_col : d.sq_row);
    float* absmax = RES ? (is_col ? d.res_col_absmax : d.res_row_absmax) : (is_col ? d.sq_col_absmax : d.sq_row_absmax);
    float old = 0.0f;
    if (idx < n) old = quant ? (float)reinterpret_cast<const uint8_t*>(state)[idx] * (absmax[b] / QMAX_U8) : reinterpret_cast<const float*>(state)[idx];
    const int left = n - b * QBLOCK - lane;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.0f;
    // (32 loads in flight: the 785 partials of a column of a 50257-row matrix are 98 steps for the one CTA that adds them,
    // while the other CTAs wait at the next barrier)
#pragma unroll 4
    for (int t = warp; t < parts; t += G_WARPS)
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (32 * e < left) acc[e] += __ldcg(part + (int64_t)t * n + 32 * e);
#pragma unroll
    for (int e = 0; e < 8; ++e) sh.col[warp][32 * e + lane] = acc[e];
    __syncthreads();
    float v = 0.0f, sum = 0.0f;
#pragma unroll
    for (int k = 0; k < G_WARPS; ++k) sum += sh.col[k][threadIdx.x];
    if (idx < n) {
        v = ema_update(old, RES ? h.beta3 : h.beta2, RES ? h.om_beta3 : h.om_beta2, mean_plus_eps(sum, (float)(is_col ? R : C), RES ? h.eps1 : h.eps0));
        const bool clamp = d.flags & (RES ? CAME_F_RESCOL_CLAMP : CAME_F_SQ_CLAMP);
        if (is_col) (RES ? s.Rc : s.vc)[idx] = inv_sqrt(clamp ? fmaxf(v, 1e-30f) : v);
        else (RES ? s.Rr : s.vr)[idx] = v;
    }
    if (quant) {
        const float bmax = fix_absmax(block_max(v, sh.red));      // syncs: every old absmax read is done
        if (threadIdx.x == 0) absmax[b] = bmax;
        if (idx < n) reinterpret_cast<uint8_t*>(state)[idx] = (uint8_t)quant_u8_div(v, bmax);
    } else if (idx < n) {
        reinterpret_cast<float*>(state)[idx] = v;
    }
    if (!is_col) {
        float* blk = RES ? s.rowblk2 : s.rowblk;
        const float bs = block_sum(v, sh.red);
        if (threadIdx.x == 0) blk[b] = bs;
    }
    // The counters of the next phase.  They are back at zero after every phase that ran to its end; after one that some
    // CTAs left at a barrier they are not.
    if (!RES && w.tile == 0)
        for (int i = threadIdx.x, nc = 1 + (s.tiles_r * s.tiles_c + PARTIAL_GROUP - 1) / PARTIAL_GROUP; i < nc; i += THREADS) s.counters[i] = 0;
    __syncthreads();      // (the shared arrays are free for the next item)
}

// ---- 1-D tensors --------------------------------------------------------------------------------------------------
// (reference: kCameNonfactoredSqUpdateAndQuant[TypedUpdate] came_kernels.cu:1013-1122,
// kCameNonfactoredExpAvgParamUpdate[TypedUpdate] came_kernels.cu:1489-1601; CAMECUDA.py:247-273; no confidence term,
// CAME.py:163-164).  A CTA owns a block of 256 elements.
template <typename TG>
__device__ __forceinline__ void vector_element(const CameTensorDesc& d, const CameHyper& h, int b, int64_t idx, float& v, float& u) {
    v = 0.0f; u = 0.0f;
    if (idx >= d.rows) return;
    const float g = Buf<TG>(d.g, d.g_dtype).get(idx) * h.grad_scale;
    const float old = d.mode != CAME_MODE_FP32 ? (float)reinterpret_cast<const uint8_t*>(d.sq_row)[idx] * (d.sq_row_absmax[b] / QMAX_U8)
                                               : reinterpret_cast<const float*>(d.sq_row)[idx];
    v = nf_second_moment(old, g, h);
    u = nf_update(v, g, d.flags);
}
constexpr int VECTOR_DIRECT = 512;      // block partials that every reader adds by itself (beyond: the last block does)
template <typename TG>
__device__ __forceinline__ void phase_vector_sq(const StepArgs& a, const CameHyper* hyp, const Work& w, GShared& sh) {
    const CameTensorDesc& d = a.descs[w.tensor];
    const Scratch& s = a.scr[w.tensor];
    float v, u;
    vector_element<TG>(d, hyp[d.group], w.tile, (int64_t)w.tile * QBLOCK + threadIdx.x, v, u);
    const float t = block_sum(u * u, sh.red);
    if (threadIdx.x == 0) s.spart[w.tile] = t;
    if (s.nbR > VECTOR_DIRECT && last_cta(s.counters, s.nbR, sh)) {
        const float S = block_vector_sum_cg(s.spart, s.nbR, sh.red);
        if (threadIdx.x == 0) s.scal[0] = S;
    }
    __syncthreads();
}
template <typename TG, typename TP>
__device__ __forceinline__ void phase_vector_apply(const StepArgs& a, const CameHyper* hyp, const Work& w, GShared& sh) {
    const CameTensorDesc& d = a.descs[w.tensor];
    const CameHyper& h = hyp[d.group];
    const int b = w.tile;
    const int64_t idx = (int64_t)b * QBLOCK + threadIdx.x;
    const bool in = idx < d.rows, quant = d.mode != CAME_MODE_FP32;
    const Buf<TP> p(d.p, d.p_dtype);
    float v, u, m = 0.0f;
    vector_element<TG>(d, h, b, idx, v, u);
    if (in) m = quant ? (float)reinterpret_cast<const int8_t*>(d.m)[idx] * (d.m_absmax[b] / QMAX_I8) : reinterpret_cast<const float*>(d.m)[idx];
    const float pv = in ? p.get(idx) : 0.0f;
    const Scratch& s = a.scr[w.tensor];
    const float S = s.nbR > VECTOR_DIRECT ? __ldcg(s.scal) : block_vector_sum_cg(s.spart, s.nbR, sh.red);
    const float clip = nf_clip(S, d.rows, h);
    m = in ? nf_momentum(m, u, clip, 1.0f / clip, d.flags, h) : 0.0f;
    if (in) p.put(idx, g_apply_one(p, pv, m, h, wd_form(h, d.flags)));
    if (quant) {
        const float vmax = fix_absmax(block_max(v, sh.red)), mmax = fix_absmax(block_max(fabsf(m), sh.red));      // (syncs)
        if (threadIdx.x == 0) { d.sq_row_absmax[b] = vmax; d.m_absmax[b] = mmax; }
        if (in) {
            reinterpret_cast<uint8_t*>(d.sq_row)[idx] = (uint8_t)quant_u8_div(v, vmax);
            reinterpret_cast<int8_t*>(d.m)[idx] = (int8_t)quant_i8_div(m, mmax);
        }
    } else if (in) {
        reinterpret_cast<float*>(d.sq_row)[idx] = v;
        reinterpret_cast<float*>(d.m)[idx] = m;
    }
}

// ---- the kernel ---------------------------------------------------------------------------------------------------
struct GenericArgs {
    StepArgs a;
    GenericLists l;
    int n_hyp;                        // records in `hyp`: the step's hyper-parameters; 0: a.hyp holds them
    CameHyper hyp[GENERIC_MAX_HYP];
};

template <typename TG, typename TP, int MODE, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) k_step_generic(const __grid_constant__ GenericArgs ga) {
    using S = Stage<TG, MODE>;
    extern __shared__ __align__(128) char g_smem[];
    __shared__ GShared sh;
    const StepArgs& a = ga.a;
    const GenericLists& l = ga.l;
    const CameHyper* hyp = ga.n_hyp ? ga.hyp : a.hyp;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    char* const stages = g_smem + warp * (S::COUNT * S::BYTES);
    auto stage = [&](int k) { return stages + k * S::BYTES; };
    // warp items: across the SMs first, then over the warps; CTA items of 1-D tensors: from the last CTA on, which comes
    // last in the deal of the others
    const int first = warp * gridDim.x + blockIdx.x, stride = G_WARPS * gridDim.x, back = gridDim.x - 1 - blockIdx.x;
    u64 colacc[4];
    float acc = 0.0f, mean = 1.0f, inv_clip = 1.0f, gs = 1.0f;      // of the item in work

    for (int i = back; i < l.n_ones; i += gridDim.x) phase_vector_sq<TG>(a, hyp, l.ones[i], sh);
    stream<S::COUNT>(a, l.tiles, l.n_tiles, first, stride,
        [&](const Item& it, int k) {
            const CameTensorDesc& d = a.descs[it.tensor];
            stage_rows<Size<TG>::FIXED>(stage(k), S::PA, d.g, size_of<TG>(d.g_dtype), it, lane);
        },
        [&](const Item& it, int k) {
            if (it.v8) band_sq<TG, 8>(a, hyp, it, stage(k), S::PA, colacc, gs);
            else band_sq<TG, 1>(a, hyp, it, stage(k), S::PA, colacc, gs);
        });
    if (!grid_barrier(l.bar, a.status)) return;

    for (int i = back; i < l.n_ones; i += gridDim.x) phase_vector_apply<TG, TP>(a, hyp, l.ones[i], sh);
    if (l.n_tiles == 0) return;
    for (int i = blockIdx.x; i < l.n_vecs; i += gridDim.x) phase_finalize<false>(a, hyp, l.vecs[i], sh);
    if (!grid_barrier(l.bar, a.status)) return;

    stream<S::COUNT>(a, l.tiles, l.n_tiles, first, stride,
        [&](const Item& it, int k) {
            const CameTensorDesc& d = a.descs[it.tensor];
            const Scratch& s = a.scr[it.tensor];
            stage_vectors(stage(k), S::OFF_V, S::OFF_C, s.vr, s.vc, it, lane);
            stage_rows<Size<TG>::FIXED>(stage(k), S::PA, d.g, size_of<TG>(d.g_dtype), it, lane);
        },
        [&](const Item& it, int k) {
            if (it.v8) band_clip<TG, S, 8>(a, hyp, it, stage(k), acc, mean, gs);
            else band_clip<TG, S, 1>(a, hyp, it, stage(k), acc, mean, gs);
        });
    if (!grid_barrier(l.bar, a.status)) return;

    stream<S::COUNT>(a, l.tiles, l.n_tiles, first, stride,
        [&](const Item& it, int k) {
            const CameTensorDesc& d = a.descs[it.tensor];
            const Scratch& s = a.scr[it.tensor];
            stage_vectors(stage(k), S::OFF_V, S::OFF_C, s.vr, s.vc, it, lane);
            stage_absmax<MODE>(stage(k) + S::OFF_X, d.m_absmax, it, lane);
            stage_rows<Size<TG>::FIXED>(stage(k), S::PA, d.g, size_of<TG>(d.g_dtype), it, lane);
            stage_rows<(MODE == CAME_MODE_FP32 ? 4 : 1)>(stage(k) + S::OFF_M, S::PM, d.m, MODE == CAME_MODE_FP32 ? 4 : 1, it, lane);
        },
        [&](const Item& it, int k) {
            if (it.v8) band_moment<TG, MODE, 8>(a, hyp, it, stage(k), colacc, mean, inv_clip, gs);
            else band_moment<TG, MODE, 1>(a, hyp, it, stage(k), colacc, mean, inv_clip, gs);
        });
    if (!grid_barrier(l.bar, a.status)) return;

    for (int i = blockIdx.x; i < l.n_vecs; i += gridDim.x) phase_finalize<true>(a, hyp, l.vecs[i], sh);
    if (!grid_barrier(l.bar, a.status)) return;

    if constexpr (MODE == CAME_MODE_FLAT8) {
        using F = FlatSlot<TG, MODE>;
        FlatTensor ft;
        Work ahead[F::COUNT];      // the blocks under way, the next to compute first
#pragma unroll
        for (int k = 0; k < F::COUNT - 1; ++k) {
            const int i = first + k * stride;
            if (i < l.n_flats) {
                ahead[k] = l.flats[i];
                issue_flat<TG, TP, F>(a, ahead[k], stages + k * F::BYTES, lane);
            }
            cp_commit();
        }
        for (int i = first, slot = 0; i < l.n_flats; i += stride) {
            const int j = i + (F::COUNT - 1) * stride, free = slot == 0 ? F::COUNT - 1 : slot - 1;      // (of the block before)
            if (j < l.n_flats) {
                ahead[F::COUNT - 1] = l.flats[j];
                issue_flat<TG, TP, F>(a, ahead[F::COUNT - 1], stages + free * F::BYTES, lane);
            }
            cp_commit();
            const Work w = ahead[0];
            ft.use(a, hyp, w.tensor, size_of<TP>(a.descs[w.tensor].p_dtype), lane);
            cp_wait<F::COUNT - 1>();
            __syncwarp();
            if (a.scr[w.tensor].g_v == 8) phase_apply_flat<TG, TP, F, 8>(a, hyp, w, ft, stages + slot * F::BYTES);
            else phase_apply_flat<TG, TP, F, 1>(a, hyp, w, ft, stages + slot * F::BYTES);
            __syncwarp();      // the slot is read before it is filled again
#pragma unroll
            for (int k = 0; k < F::COUNT - 1; ++k) ahead[k] = ahead[k + 1];
            if (++slot == F::COUNT) slot = 0;
        }
        cp_wait<0>();
    } else {
        stream<S::COUNT>(a, l.tiles, l.n_tiles, first, stride,
            [&](const Item& it, int k) {
                const CameTensorDesc& d = a.descs[it.tensor];
                const Scratch& s = a.scr[it.tensor];
                stage_vectors(stage(k), S::OFF_V, S::OFF_C, s.Rr, s.Rc, it, lane);
                stage_absmax<MODE>(stage(k) + S::OFF_X, d.m_absmax, it, lane);
                stage_rows<Size<TP>::FIXED>(stage(k), S::PA, d.p, size_of<TP>(d.p_dtype), it, lane);
                stage_rows<(MODE == CAME_MODE_FP32 ? 4 : 1)>(stage(k) + S::OFF_M, S::PM, d.m, MODE == CAME_MODE_FP32 ? 4 : 1, it, lane);
            },
            [&](const Item& it, int k) {
                if (it.v8) band_apply<TP, MODE, 8>(a, hyp, it, stage(k), mean);
                else band_apply<TP, MODE, 1>(a, hyp, it, stage(k), mean);
            });
    }
}

struct GenericKernel {
    void (*fn)(const GenericArgs);
    int smem;
};
template <typename TG, typename TP, int MODE> GenericKernel generic_kernel(int ctas) {
    return {ctas == 2 ? k_step_generic<TG, TP, MODE, 2> : k_step_generic<TG, TP, MODE, 3>, G_WARPS * Stage<TG, MODE>::COUNT * Stage<TG, MODE>::BYTES};
}
template <typename TG, typename TP> GenericKernel pick_mode(int mode, int ctas) {
    switch (mode) {
        case CAME_MODE_FP32: return generic_kernel<TG, TP, CAME_MODE_FP32>(ctas);
        case CAME_MODE_TILE8: return generic_kernel<TG, TP, CAME_MODE_TILE8>(ctas);
        default: return generic_kernel<TG, TP, CAME_MODE_FLAT8>(ctas);
    }
}
GenericKernel pick_generic(int g, int p, int mode, int ctas) {
    if (g != p) return pick_mode<Any, Any>(mode, ctas);
    if (g == CAME_DT_F32) return pick_mode<float, float>(mode, ctas);
    if (g == CAME_DT_F16) return pick_mode<__half, __half>(mode, ctas);
    return pick_mode<__nv_bfloat16, __nv_bfloat16>(mode, ctas);
}

}  // namespace

int generic_tile_cols() { return G_CW; }

// Self-test of the grid barrier: CTAs below `absent` leave without arriving, the others wait and record what they got.
__global__ void k_selftest_grid_barrier(uint32_t* bar, int* status, int absent, uint32_t limit, int* observed) {
    if ((int)blockIdx.x < absent) return;
    const bool ok = grid_barrier(bar, status, limit);
    if (threadIdx.x == 0) observed[blockIdx.x] = ok ? 1 : 0;
}
// One CTA of four stays away, then all four come: words = {status, barrier, observed[4], observed[4]}
cudaError_t launch_selftest_grid_barrier(int* words, cudaStream_t st) {
    for (int k = 0; k < 2; ++k) {
        uint32_t* bar = reinterpret_cast<uint32_t*>(words + 1);
        int *status = words, absent = k == 0, *observed = words + 2 + 4 * k;
        uint32_t limit = k == 0 ? 4096u : G_POLL_LIMIT;
        void* params[] = {&bar, &status, &absent, &limit, &observed};
        const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_selftest_grid_barrier), dim3(4), dim3(64), params, 0, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_generic(const KernelKey& key, const StepArgs& a, const CameHyper* host_hyp, int n_hyp, const GenericLists& l,
                           cudaStream_t st) {
    const GenericKernel kernel = pick_generic(key.g_dtype, key.p_dtype, key.mode, key.variant);
    const void* fn = reinterpret_cast<const void*>(kernel.fn);
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> cache;      // CTAs an SM holds, per device and kernel
    int dev = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find({dev, fn});
        if (it == cache.end()) {
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kernel.smem);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, THREADS, kernel.smem);
            if (e != cudaSuccess) return e;
            cache[{dev, fn}] = per_sm;
        } else {
            per_sm = it->second;
        }
    }
    const int most = std::max({l.n_tiles + l.n_ones, l.n_vecs + l.n_ones, l.n_flats});
    const int grid = std::min(most, std::max(1, per_sm) * persistent_grid_limit());
    GenericArgs ga{};
    ga.a = a;
    ga.l = l;
    if (host_hyp && n_hyp <= GENERIC_MAX_HYP) {
        ga.n_hyp = n_hyp;
        for (int i = 0; i < n_hyp; ++i) ga.hyp[i] = host_hyp[i];
    }
    void* params[] = {&ga};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(THREADS), params, (size_t)kernel.smem, st);
}

}  // namespace came
