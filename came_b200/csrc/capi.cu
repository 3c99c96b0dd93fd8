// C ABI of libcame_b200: descriptor validation, workspace layout, work lists, step scheduling.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <tuple>
#include <vector>

#include "came_b200.h"
#include "launch.h"

using namespace came;

namespace {

constexpr int MAX_GROUPS = 64;
constexpr size_t ALIGN = 256;

thread_local char g_err[512] = "";
// CAME_B200_DISABLE_FAST=1 in the environment routes every matrix through the whole-step kernel (used by the
// tests to compare the two implementations of a pass against each other).  Read whenever a plan is sized or created,
// so that it must not change between came_b200_workspace_bytes and came_b200_plan_create of one plan.
inline bool disable_fast() { const char* e = getenv("CAME_B200_DISABLE_FAST"); return e && e[0] == '1'; }

// CAME_B200_WAVE_MB=n: run the momentum / apply passes in waves of tensors holding at most n MB of momentum state
const size_t g_wave_bytes = [] { const char* e = getenv("CAME_B200_WAVE_MB"); return e ? (size_t)atol(e) << 20 : (size_t)0; }();

// The fused momentum / apply kernel (fused_ma.cu).  CAME_B200_FUSED_MA=0 runs the three passes as separate launches.
// CAME_B200_MA_LAG: momentum items of later tensors placed between a tensor's last momentum item and its apply items
// (default: 5 per CTA; measured on Llama-7B shapes: 2 per CTA leaves the apply items waiting for the residual
// finalize, from 5 on the kernel runs at the DRAM limit).
// Read when a plan is created.
bool fused_ma_enabled() { const char* e = getenv("CAME_B200_FUSED_MA"); return !(e && e[0] == '0'); }
int env_int(const char* name, int dflt) { const char* e = getenv(name); return e ? atoi(e) : dflt; }

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

inline size_t align_up(size_t x, size_t a = ALIGN) { return (x + a - 1) / a * a; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

struct LaunchItem {
    int kernel;
    KernelKey key;
    size_t work_off;   // in Work units from the start of the work region
    int n;
    size_t work2_off;  // fused momentum / apply kernel: its F items; whole-step kernel: vector blocks
    int n2;
    size_t work3_off, work4_off;      // whole-step kernel: flat blocks, 1-D blocks
    int n3, n4, bar;
};

inline int elem_bytes(int dt) { return dt == CAME_DT_F32 ? 4 : 2; }
inline bool is_nd(const CameTensorDesc& d) { return d.cols != 0 && d.batch > 1; }
inline int nd_chunk(const CameTensorDesc& d) { return is_nd(d) && !disable_fast() ? nd_small_batch(d.rows, d.cols) : 0; }

// Which kernels take the passes of a matrix.
struct VecFlags {
    int k;      // gradient sums of the staged path: 2 = one pass (fused_sq.cu), 1 = two passes (rows too wide for it)
    int wide;   // staged momentum / apply passes
    int v;      // elements per access of the whole-step kernel (generic.cu): 8, or 1 for any shape and alignment
    bool operator==(const VecFlags& o) const { return k == o.k && wide == o.wide && v == o.v; }
};

VecFlags vec_flags(const CameTensorDesc& d, bool fast) {
    VecFlags f{0, 0, 0};
    if (d.cols == 0 || is_nd(d)) return f;      // 1-D and N-D tensors have kernels of their own
    const bool aligned = aligned16(d.g) && aligned16(d.m) && aligned16(d.p);
    f.v = aligned && d.cols % 8 == 0 ? 8 : 1;
    f.wide = fast && aligned &&
             ((d.mode != CAME_MODE_FLAT8 && d.cols % 64 == 0) ||
              (d.mode == CAME_MODE_FLAT8 && d.cols % 256 == 0 && d.g_dtype == d.p_dtype));
    // (tensors with the 1e-30 clamps take the fused first pass too: its closed form for the clip sum holds whenever no
    // clamp binds, which the finalize checks; if one does, the two-pass sum runs for that tensor)
    if (f.wide) f.k = fused_sq_eligible(d.cols, elem_bytes(d.g_dtype)) ? 2 : 1;
    return f;
}

VecFlags vec_flags(const CameTensorDesc& d) { return vec_flags(d, !disable_fast()); }

// Small sets: every matrix of a set with fewer elements than this on the staged path takes the whole-step kernel; the flat
// layout counts 4/3, as the whole-step kernel reads its gradients once more than the others'.  us a step, staged / whole-step
// (p and g in bf16, fp32 for the last; one n x n matrix, or decoders of l layers of width h):
//                            tile              flat              fp32
//   n = 1024                  98 /  43         112 /  45         104 /  42
//   n = 2048                 105 /  55         119 /  65         119 /  61
//   n = 3072                 118 /  77         131 /  99         137 /  97
//   n = 3840 (14 Mi)         125 / 105         138 / 138         151 / 132
//   l = 4, h = 512 (13.5 Mi) 134 / 106         155 / 159         154 / 133
//   l = 8, h = 512 (26.5 Mi) 161 / 184         193 / 304         230 / 255
// CAME_B200_SMALL_SET_ELEMS overrides the line (0: none; read whenever a plan is sized or created).
constexpr long long SMALL_SET_ELEMS = 16 << 20;

// What a plan decides about the set as a whole.
struct Context {
    bool small;      // the whole-step kernel takes every matrix
    int bands;       // its bands of 16 rows per warp
    bool generic(const CameTensorDesc& d) const { return d.cols != 0 && !is_nd(d) && (small || !vec_flags(d).wide); }
};

int64_t generic_tiles(const CameTensorDesc& d, int bands) {
    return cdiv(d.rows, (int64_t)bands * 16) * cdiv(d.cols, generic_tile_cols());
}
// partials, groups of them and counters of a reduction over n items (leave_partial in generic.cu)
size_t partial_floats(int64_t n) { return (size_t)(n + cdiv(n, PARTIAL_GROUP) + 1); }
size_t partial_counters(int64_t n) { return (size_t)(1 + cdiv(n, PARTIAL_GROUP)); }

Context context(const CameTensorDesc* descs, int n) {
    const char* e = getenv("CAME_B200_SMALL_SET_ELEMS");
    const double line = e ? atof(e) : (double)SMALL_SET_ELEMS;
    double staged = 0.0;
    for (int i = 0; i < n; ++i)
        if (vec_flags(descs[i]).wide)
            staged += (double)descs[i].rows * (double)descs[i].cols * (descs[i].mode == CAME_MODE_FLAT8 ? 4.0 / 3.0 : 1.0);
    Context c{staged < line, 16};
    auto items = [&](int bands) {
        int64_t tiles = 0;
        for (int i = 0; i < n; ++i)
            if (c.generic(descs[i])) tiles += generic_tiles(descs[i], bands);
        return tiles;
    };
    // Where it takes 8 bands or fewer: the fewest that leave no resident warp (16 per SM) a second item.  Fewer bands make
    // more column partials, which the finalize phases add in one chain per column while the other CTAs wait at a barrier:
    // one bf16 matrix of 3840 x 3840 takes 154 / 130 / 115 / 105 us at 1 / 2 / 4 / 8 bands, 16384 x 768 178 / 130 / 117 / 104,
    // 1024 x 1024 43 / 48 / 58 / 67.
    for (int b = 1; b <= 8; b *= 2)
        if (items(b) <= 16 * 148) {
            c.bands = b;
            return c;
        }
    // Larger sets: as few bands per item as it takes to give every resident warp of the GPU (24 per SM) two items; more than 4, which
    // only saves column partials and their summation, where every warp (16 per SM) still has eight to even the load out.
    for (; c.bands > 1; c.bands /= 2)
        if (items(c.bands) >= (c.bands > 4 ? 8 * 16 : 2 * 24) * 148) break;
    return c;
}

struct Geometry {
    int64_t R, C;
    int tiles_r, tiles_c, ptiles_r, ptiles_c, nbR, nbC;
    int64_t flat_chunks;
};

Geometry geometry(const CameTensorDesc& d, const Context& ctx) {
    Geometry g{};
    g.R = d.rows;
    g.C = d.cols;
    g.nbR = (int)cdiv(g.R, QBLOCK);
    if (d.cols == 0) return g;
    if (is_nd(d)) {      // nbR / nbC: blocks of the flattened row / column vectors; flat_chunks: flat blocks of 256 elements
        g.nbR = (int)cdiv((int64_t)d.batch * g.R, QBLOCK);
        g.nbC = (int)cdiv((int64_t)d.batch * g.C, QBLOCK);
        const int nm = nd_chunk(d);      // small matrices: flat_chunks counts chunks of them, and nothing else is launched
        g.flat_chunks = nm ? cdiv((int64_t)d.batch, nm) : cdiv((int64_t)d.batch * g.R * g.C, QBLOCK);
        return g;
    }
    g.nbC = (int)cdiv(g.C, QBLOCK);
    if (ctx.generic(d)) {
        g.tiles_r = (int)cdiv(g.R, (int64_t)ctx.bands * 16);
        g.tiles_c = (int)cdiv(g.C, generic_tile_cols());
        if (d.mode == CAME_MODE_FLAT8) g.flat_chunks = cdiv(g.R * g.C, QBLOCK);
        return g;
    }
    g.tiles_r = (int)cdiv(g.R, K_TR);
    g.tiles_c = (int)cdiv(g.C, K_TC);
    g.ptiles_r = (int)cdiv(g.R, W_TR);
    g.ptiles_c = (int)cdiv(g.C, W_TC);
    return g;
}

// carve the per-tensor float scratch; base == nullptr computes sizes only
size_t carve(const CameTensorDesc& d, const Geometry& g, const Context& ctx, float* base, Scratch* out) {
    size_t off = 0;
    auto take = [&](size_t n) -> float* {
        float* p = base ? base + off : nullptr;
        off += align_up(n, 4);
        return p;
    };
    Scratch s{};
    s.nbR = g.nbR;
    if (d.cols == 0) {
        s.spart = take((size_t)g.nbR);      // block partials of sum u^2
        s.scal = take(4);
        s.counters = reinterpret_cast<int32_t*>(take(4));
    } else if (is_nd(d)) {
        const size_t B = d.batch;
        s.nbC = g.nbC;
        s.tiles_r = (int)g.flat_chunks;      // partials of S
        s.tiles_c = nd_chunk(d);
        if (s.tiles_c) {
            s.scal = take(4);
            s.spart = take((size_t)g.flat_chunks);
            if (out) *out = s;
            return off;
        }
        s.vr = take(B * (size_t)g.R); s.vc = take(B * (size_t)g.C);
        s.Rr = take(B * (size_t)g.R); s.Rc = take(B * (size_t)g.C);
        s.rowblk = take(B); s.rowblk2 = take(B);      // per matrix: guarded mean of the fresh row vectors
        s.scal = take(4);
        s.spart = take((size_t)g.flat_chunks);
    } else if (ctx.generic(d)) {
        s.nbC = g.nbC;
        s.tiles_r = g.tiles_r; s.tiles_c = g.tiles_c;
        s.g_v = vec_flags(d).v;
        s.g_nb = ctx.bands;
        s.vr = take((size_t)g.R); s.vc = take((size_t)g.C);      // v_row, column factors c_j
        s.Rr = take((size_t)g.R); s.Rc = take((size_t)g.C);      // residual row vector, C'_j
        s.rowblk = take((size_t)g.nbR); s.rowblk2 = take((size_t)g.nbR);
        s.scal = take(4);
        s.rowpart = take((size_t)g.tiles_c * (size_t)g.R);
        s.colpart = take((size_t)g.tiles_r * (size_t)g.C);
        const int64_t items = (int64_t)g.tiles_r * g.tiles_c;
        s.spart = take(partial_floats(items));
        s.fac = d.mode == CAME_MODE_FLAT8 ? take((size_t)g.R) : nullptr;
        s.counters = reinterpret_cast<int32_t*>(take(partial_counters(items)));
    } else {
        s.nbC = g.nbC;
        s.tiles_r = g.tiles_r; s.tiles_c = g.tiles_c;
        s.ptiles_r = g.ptiles_r; s.ptiles_c = g.ptiles_c;
        s.vr = take((size_t)g.R); s.vc = take((size_t)g.C);
        s.Rr = take((size_t)g.R); s.Rc = take((size_t)g.C);
        s.rowblk = take((size_t)g.nbR); s.rowblk2 = take((size_t)g.nbR);
        s.scal = take(4);
        s.rowpart = take((size_t)std::max(g.tiles_c, g.ptiles_c) * (size_t)g.R);
        s.sq_col_parts = g.tiles_r;
        int fa_groups = 1, fa_ng = 1, fa_rb = 1, fa_slot_kb = 64;
        if (vec_flags(d).k == 2) {
            fused_sq_geometry(g.C, elem_bytes(d.g_dtype), &fa_groups, &fa_ng, &fa_rb, &fa_slot_kb);
            s.sq_col_parts = g.tiles_r * fa_groups;
        }
        s.colpart = take((size_t)std::max(s.sq_col_parts, g.ptiles_r) * (size_t)g.C);
        s.spart = take(std::max((size_t)g.tiles_r * (size_t)g.tiles_c, (size_t)g.nbC));
        s.res_eps_deferred = 1;
        s.mfac = take((size_t)g.R);
        s.mfac_c = take((size_t)g.C);
        s.mfac_c2 = d.mode == CAME_MODE_FLAT8 ? take((size_t)g.C) : nullptr;
        if (vec_flags(d).k == 2) {
            s.fused_a = 1;
            s.fa_rb = fa_rb;
            s.tpart = take((size_t)s.sq_col_parts * (size_t)g.C);
        }
    }
    if (out) *out = s;
    return off;
}

int validate(const CameTensorDesc& d, int i) {
    if (!d.p || !d.g || !d.m) return fail(CAME_E_INVALID, "tensor %d: p, g and m must be non-null", i);
    if (d.rows <= 0 || d.cols < 0) return fail(CAME_E_INVALID, "tensor %d: bad shape [%lld, %lld]", i, (long long)d.rows, (long long)d.cols);
    if (d.rows > 0x7fffffffLL || d.cols > 0x7fffffffLL) return fail(CAME_E_UNSUPPORTED, "tensor %d: dimension above 2^31-1", i);
    if (d.mode < CAME_MODE_FP32 || d.mode > CAME_MODE_FLAT8) return fail(CAME_E_INVALID, "tensor %d: bad mode %d", i, d.mode);
    if (d.p_dtype < CAME_DT_F32 || d.p_dtype > CAME_DT_BF16 || d.g_dtype < CAME_DT_F32 || d.g_dtype > CAME_DT_BF16)
        return fail(CAME_E_INVALID, "tensor %d: bad dtype", i);
    if (d.group < 0 || d.group >= MAX_GROUPS) return fail(CAME_E_INVALID, "tensor %d: group %d outside [0, %d)", i, d.group, MAX_GROUPS);
    const bool quant = d.mode != CAME_MODE_FP32;
    if (quant && !d.m_absmax) return fail(CAME_E_INVALID, "tensor %d: 8-bit exp_avg needs m_absmax", i);
    if (!d.sq_row || (quant && !d.sq_row_absmax)) return fail(CAME_E_INVALID, "tensor %d: missing exp_avg_sq state", i);
    if (d.cols == 0) {
        if (d.mode == CAME_MODE_TILE8) return fail(CAME_E_INVALID, "tensor %d: 1-D tensors use CAME_MODE_FLAT8 or CAME_MODE_FP32", i);
        return CAME_OK;
    }
    if (!d.sq_col || !d.res_row || !d.res_col) return fail(CAME_E_INVALID, "tensor %d: missing factored state", i);
    if (d.batch > 1) {
        if (d.mode == CAME_MODE_TILE8) return fail(CAME_E_INVALID, "tensor %d: the tile layout holds single matrices (batch %u)", i, d.batch);
        if ((double)d.batch * (double)d.rows * (double)d.cols > 9.0e18) return fail(CAME_E_UNSUPPORTED, "tensor %d: too many elements", i);
        if (cdiv((int64_t)d.batch * d.rows * d.cols, QBLOCK) > 0x7fffffffLL) return fail(CAME_E_UNSUPPORTED, "tensor %d: too many elements", i);
    }
    if (quant && (!d.sq_col_absmax || !d.res_row_absmax || !d.res_col_absmax))
        return fail(CAME_E_INVALID, "tensor %d: missing factored absmax", i);
    return CAME_OK;
}

struct Layout {
    size_t off_descs, off_scr, off_hyp, off_status, off_bar, off_sync, off_work, off_float, total;
    size_t n_work;
};

size_t count_work(const CameTensorDesc* descs, int n, const Context& ctx) {
    size_t w = 0;
    for (int i = 0; i < n; ++i) {
        const Geometry g = geometry(descs[i], ctx);
        if (descs[i].cols == 0) {
            w += (size_t)g.nbR;
            continue;
        }
        if (ctx.generic(descs[i])) {
            w += (size_t)g.tiles_r * g.tiles_c + (size_t)(g.nbR + g.nbC) + (size_t)g.flat_chunks;
            continue;
        }
        if (is_nd(descs[i])) {      // two vector passes, two mean passes (one item per matrix), S, two element passes
            w += 2 * (size_t)(g.nbR + g.nbC) + 2 * (size_t)descs[i].batch + 1 + 2 * (size_t)g.flat_chunks;
            continue;
        }
        w += 2 * (size_t)g.tiles_r * g.tiles_c;      // sq_partials, sumsq
        w += 2 * (size_t)(g.nbR + g.nbC);            // two vector finalizes
        w += (size_t)std::max<int64_t>(1, cdiv(g.R + g.C, S_FIN_CHUNK));      // clip finalize
        w += 2 * (size_t)g.ptiles_r * g.ptiles_c;    // moment, apply
    }
    return w;
}

constexpr int MAX_GENERIC_LAUNCHES = 32;      // (gradient type, parameter type, layout) combinations: 27

Layout layout(const CameTensorDesc* descs, int n, const Context& ctx) {
    Layout L{};
    size_t off = 0;
    L.off_descs = off; off = align_up(off + (size_t)n * sizeof(CameTensorDesc));
    L.off_scr = off;   off = align_up(off + (size_t)n * sizeof(Scratch));
    L.off_hyp = off;   off = align_up(off + (size_t)MAX_GROUPS * sizeof(CameHyper));
    L.off_status = off; off = align_up(off + sizeof(int));
    L.off_sync = off;  off = align_up(off + (2 * (size_t)n + 12) * sizeof(int));   // fused kernel: per-tensor item counters, list cursors
    L.off_bar = off;   off = align_up(off + MAX_GENERIC_LAUNCHES * sizeof(uint32_t));      // grid barriers of the whole-step kernel
    L.n_work = count_work(descs, n, ctx);
    L.off_work = off;  off = align_up(off + L.n_work * sizeof(Work));
    L.off_float = off;
    size_t fl = 0;
    for (int i = 0; i < n; ++i) fl += align_up(carve(descs[i], geometry(descs[i], ctx), ctx, nullptr, nullptr), 64);
    off = align_up(off + fl * sizeof(float));
    L.total = off;
    return L;
}

}  // namespace

namespace came {
// lets other translation units leave a message for came_b200_last_error()
void set_last_error(const char* msg) { snprintf(g_err, sizeof(g_err), "%s", msg); }
int persistent_grid_limit() {
    static int limit = 0;
    if (limit == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
        int reserved = 0;
        if (const char* e = getenv("CAME_B200_RESERVED_SMS")) reserved = atoi(e);
        if (reserved < 0) reserved = 0;
        if (reserved > sms - 1) reserved = sms - 1;
        limit = sms - reserved;
    }
    return limit;
}
}  // namespace came

struct came_plan {
    int n_tensors = 0;
    std::vector<CameTensorDesc> descs;
    std::vector<VecFlags> vflags;
    char* ws = nullptr;
    Layout L{};
    std::vector<LaunchItem> launches;
    int last_launches = 0;
    bool has_fused_ma = false;
    std::vector<char> fused;       // per tensor: stepped by the fused momentum / apply kernel
    std::vector<char> pushable;    // ... or by the whole-step kernel, which serves the push mode too
    std::vector<char> push_must;   // pushable whatever the size of the set: has to lie in the local buffer (else it is not pushed)
    bool needs_hyp = false;        // some kernel reads the hyper-parameters from the workspace
    int n_push = 0;                // push mode: peers that receive every parameter the fused kernel updates
    long long push_delta[MAX_PUSH_PEERS] = {};
    uintptr_t push_lo = 0, push_hi = 0;      // the local buffer the pushed parameters must lie in
    bool timing = false;
    struct Timed { int kernel; cudaEvent_t t0, t1; };
    std::vector<Timed> timed;
    // page-locked copy of the hyper-parameter records: the source of the upload when a step is captured into a
    // CUDA graph (the graph's copy node reads it again at every replay)
    CameHyper* graph_hyp = nullptr;
    int graph_groups = 0;
    ~came_plan() {
        for (auto& t : timed) { cudaEventDestroy(t.t0); cudaEventDestroy(t.t1); }
        if (graph_hyp) cudaFreeHost(graph_hyp);
    }
};

static int check_hypers(const char* who, const came_plan* plan, const CameHyper* hypers, int n_groups) {
    if (!plan || !hypers) return fail(CAME_E_INVALID, "%s: null argument", who);
    if (n_groups <= 0 || n_groups > MAX_GROUPS) return fail(CAME_E_INVALID, "%s: n_groups %d outside [1, %d]", who, n_groups, MAX_GROUPS);
    for (const auto& d : plan->descs)
        if (d.group >= n_groups) return fail(CAME_E_INVALID, "%s: a tensor refers to group %d, %d given", who, d.group, n_groups);
    for (int i = 0; i < n_groups; ++i) {
        if (!(hypers[i].clip_threshold > 0.0f)) return fail(CAME_E_INVALID, "%s: group %d: clip_threshold must be > 0", who, i);
    }
    return CAME_OK;
}

// (the buffer is allocated when the plan is created: page-locking memory is not allowed while a stream is captured)
// grad_scale == 0 (a zero-initialised record) means "no scaling"
static void normalise_hypers(CameHyper* h, int n_groups) {
    for (int i = 0; i < n_groups; ++i)
        if (h[i].grad_scale == 0.0f) h[i].grad_scale = 1.0f;
}

static int stage_graph_hypers(const char* who, came_plan* plan, const CameHyper* hypers, int n_groups) {
    if (!plan->graph_hyp) return fail(CAME_E_CUDA, "%s: the plan has no page-locked hyper-parameter buffer", who);
    std::memcpy(plan->graph_hyp, hypers, (size_t)n_groups * sizeof(CameHyper));
    normalise_hypers(plan->graph_hyp, n_groups);
    plan->graph_groups = n_groups;
    return CAME_OK;
}

extern "C" {

int came_b200_version(void) { return CAME_B200_VERSION; }
const char* came_b200_last_error(void) { return g_err; }

int came_b200_quantize_blockwise(const float* src, void* q, float* absmax, int64_t n, int is_signed, came_stream_t stream) {
    if (!q || !absmax || n < 0 || (n > 0 && !src)) return fail(CAME_E_INVALID, "quantize_blockwise: null pointer or negative size");
    const cudaError_t e = launch_quantize_blockwise(src, q, absmax, n, is_signed != 0, (cudaStream_t)stream);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "quantize_blockwise: %s", cudaGetErrorString(e));
}

int came_b200_dequantize_blockwise(const void* q, const float* absmax, float* dst, int64_t n, int is_signed, came_stream_t stream) {
    if (n < 0 || (n > 0 && (!q || !absmax || !dst))) return fail(CAME_E_INVALID, "dequantize_blockwise: null pointer or negative size");
    const cudaError_t e = launch_dequantize_blockwise(q, absmax, dst, n, is_signed != 0, (cudaStream_t)stream);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "dequantize_blockwise: %s", cudaGetErrorString(e));
}

int came_b200_quantize_tile16(const float* src, int8_t* q, float* absmax, int64_t rows, int64_t cols, came_stream_t stream) {
    if (!src || !q || !absmax || rows <= 0 || cols <= 0) return fail(CAME_E_INVALID, "quantize_tile16: bad argument");
    const cudaError_t e = launch_quantize_tile16(src, q, absmax, rows, cols, (cudaStream_t)stream);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "quantize_tile16: %s", cudaGetErrorString(e));
}

int came_b200_dequantize_tile16(const int8_t* q, const float* absmax, float* dst, int64_t rows, int64_t cols, came_stream_t stream) {
    if (!dst || !q || !absmax || rows <= 0 || cols <= 0) return fail(CAME_E_INVALID, "dequantize_tile16: bad argument");
    const cudaError_t e = launch_dequantize_tile16(q, absmax, dst, rows, cols, (cudaStream_t)stream);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "dequantize_tile16: %s", cudaGetErrorString(e));
}

size_t came_b200_workspace_bytes(const CameTensorDesc* descs, int n_tensors) {
    if (!descs || n_tensors <= 0) return 0;
    for (int i = 0; i < n_tensors; ++i)
        if (validate(descs[i], i) != CAME_OK) return 0;
    return layout(descs, n_tensors, context(descs, n_tensors)).total;
}

int came_b200_plan_create(const CameTensorDesc* descs, int n_tensors, void* workspace, size_t workspace_bytes,
                          came_stream_t stream, came_plan_t** out) {
    if (!out) return fail(CAME_E_INVALID, "plan_create: out is null");
    *out = nullptr;
    if (!descs || n_tensors <= 0) return fail(CAME_E_INVALID, "plan_create: no tensors");
    for (int i = 0; i < n_tensors; ++i) {
        const int rc = validate(descs[i], i);
        if (rc != CAME_OK) return rc;
    }
    const Context ctx = context(descs, n_tensors);
    const Layout L = layout(descs, n_tensors, ctx);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) % ALIGN) != 0)
        return fail(CAME_E_WORKSPACE, "plan_create: workspace must be non-null and %zu-byte aligned", ALIGN);
    if (workspace_bytes < L.total)
        return fail(CAME_E_WORKSPACE, "plan_create: workspace of %zu bytes, %zu needed", workspace_bytes, L.total);

    came_plan* plan = new (std::nothrow) came_plan();
    if (!plan) return fail(CAME_E_INVALID, "plan_create: out of host memory");
    plan->n_tensors = n_tensors;
    plan->descs.assign(descs, descs + n_tensors);
    plan->ws = static_cast<char*>(workspace);
    plan->L = L;
    plan->vflags.resize(n_tensors);

    std::vector<Scratch> scr(n_tensors);
    std::vector<Geometry> geo(n_tensors);
    float* fbase = reinterpret_cast<float*>(plan->ws + L.off_float);
    size_t foff = 0;
    for (int i = 0; i < n_tensors; ++i) {
        geo[i] = geometry(descs[i], ctx);
        plan->vflags[i] = vec_flags(descs[i]);
        foff += align_up(carve(descs[i], geo[i], ctx, fbase + foff, &scr[i]), 64);
    }

    // work lists, one per (kernel, template key), in execution order
    std::vector<Work> work;
    work.reserve(L.n_work);
    using Key = std::tuple<int, int, int, int>;   // g, p, mode, vec
    auto build = [&](int kernel, auto select, auto keyof, auto count) {
        std::map<Key, std::vector<int>> groups;
        for (int i = 0; i < n_tensors; ++i)
            if (select(i)) groups[keyof(i)].push_back(i);
        for (auto& kv : groups) {
            LaunchItem it{};
            it.kernel = kernel;
            it.key = KernelKey{std::get<0>(kv.first), std::get<1>(kv.first), std::get<2>(kv.first), std::get<3>(kv.first)};
            it.work_off = work.size();
            for (int i : kv.second) {
                const int64_t c = count(i);
                for (int64_t t = 0; t < c; ++t) work.push_back(Work{i, (int32_t)t});
            }
            it.n = (int)(work.size() - it.work_off);
            if (it.n > 0) plan->launches.push_back(it);
        }
    };
    const CameTensorDesc* D = descs;
    auto is1d = [&](int i) { return D[i].cols == 0; };
    auto isgen = [&](int i) { return ctx.generic(D[i]); };
    auto is2d = [&](int i) { return D[i].cols != 0 && !is_nd(D[i]) && !isgen(i); };      // staged
    auto isnd = [&](int i) { return is_nd(D[i]); };
    auto nokey = [&](int) { return Key{0, 0, 0, 0}; };
    const auto& vf = plan->vflags;

    // Whole-step kernel: one launch per (gradient type, parameter type, layout) of its matrices; the vectors of the
    // same types ride along with the first of them, or get a launch of their own.
    {
        using GKey = std::tuple<int, int, int>;
        std::map<GKey, std::pair<std::vector<int>, std::vector<int>>> groups;      // matrices, vectors
        for (int i = 0; i < n_tensors; ++i)
            if (isgen(i)) groups[GKey{D[i].g_dtype, D[i].p_dtype, D[i].mode}].first.push_back(i);
        for (int i = 0; i < n_tensors; ++i)
            if (is1d(i)) {
                auto it = groups.lower_bound(GKey{D[i].g_dtype, D[i].p_dtype, 0});
                if (it == groups.end() || std::get<0>(it->first) != D[i].g_dtype || std::get<1>(it->first) != D[i].p_dtype)
                    it = groups.emplace(GKey{D[i].g_dtype, D[i].p_dtype, CAME_MODE_FP32}, std::pair<std::vector<int>, std::vector<int>>{}).first;
                it->second.second.push_back(i);
            }
        for (auto& kv : groups) {
            LaunchItem it{};
            it.kernel = KID_GENERIC;
            // Two CTAs per SM with 128 registers a thread, or three with 80 (and spills).  More registers win (a bf16 set of
            // widths 770 / 3083 / 50257: 589 against about 700 us) unless bands are mostly empty: where matrices are narrower than
            // 64 columns a band is little work behind the same latency, and warps count (rank-16 factors: 196 against 225 us).
            double elems = 0.0, room = 0.0;
            for (int i : kv.second.first) {
                elems += (double)D[i].rows * (double)D[i].cols;
                room += (double)cdiv(D[i].rows, 16) * (double)cdiv(D[i].cols, generic_tile_cols()) * (16.0 * generic_tile_cols());
            }
            it.key = KernelKey{std::get<0>(kv.first), std::get<1>(kv.first), std::get<2>(kv.first), elems < 0.5 * room ? 3 : 2};
            it.bar = (int)plan->launches.size();
            auto list = [&](const std::vector<int>& ids, auto count) {
                const size_t off = work.size();
                for (int i : ids)
                    for (int64_t t = 0, c = count(i); t < c; ++t) work.push_back(Work{i, (int32_t)t});
                return std::pair<size_t, int>{off, (int)(work.size() - off)};
            };
            const auto& mats = kv.second.first;
            std::tie(it.work_off, it.n) = list(mats, [&](int i) { return (int64_t)geo[i].tiles_r * geo[i].tiles_c; });
            std::tie(it.work2_off, it.n2) = list(mats, [&](int i) { return (int64_t)geo[i].nbR + geo[i].nbC; });
            std::tie(it.work3_off, it.n3) = list(mats, [&](int i) { return geo[i].flat_chunks; });
            std::tie(it.work4_off, it.n4) = list(kv.second.second, [&](int i) { return (int64_t)geo[i].nbR; });
            plan->launches.push_back(it);
        }
    }
    // tensors of more than two dimensions
    auto nvec = [&](int i) { return (int64_t)geo[i].nbR + geo[i].nbC; };
    auto nmat = [&](int i) { return (int64_t)D[i].batch; };
    auto nblk = [&](int i) { return geo[i].flat_chunks; };
    auto ndlarge = [&](int i) { return isnd(i) && !nd_chunk(D[i]); };
    auto ndkey = [&](int i) {
        if (!nd_chunk(D[i])) return Key{0, 0, 0, 0};
        if (!nd_fixed_batch(D[i].rows, D[i].cols)) return Key{0, 0, nd_small_kb(D[i].rows, D[i].cols), 2};
        return Key{D[i].g_dtype, D[i].p_dtype, (D[i].mode != CAME_MODE_FP32 ? 1 : 0) | (D[i].rows == 3 ? 2 : 0), 3};
    };
    build(KID_ND_SQ, ndlarge, nokey, nvec);
    build(KID_ND_MEAN, ndlarge, nokey, nmat);
    build(KID_ND_SUMSQ, isnd, ndkey, nblk);
    build(KID_ND_S, isnd, nokey, [&](int) { return (int64_t)1; });
    build(KID_ND_RES, ndlarge, nokey, nvec);
    build(KID_ND_RESMEAN, ndlarge, nokey, nmat);
    build(KID_ND_APPLY, isnd, ndkey, nblk);
    auto fusedA = [&](int i) { return is2d(i) && vf[i].k == 2; };
    auto twopass = [&](int i) { return is2d(i) && vf[i].k != 2; };
    auto fused_code = [&](int i) {      // column groups per thread | row sets << 4 | ring slot KB << 8
        int groups, ng, rb, slot_kb;
        fused_sq_geometry(D[i].cols, elem_bytes(D[i].g_dtype), &groups, &ng, &rb, &slot_kb);
        return ng | (groups << 4) | (slot_kb << 8);
    };
    build(KID_SQ_PARTIALS, fusedA, [&](int i) { return Key{D[i].g_dtype, 0, fused_code(i), 2}; },
          [&](int i) { return (int64_t)geo[i].tiles_r; });
    build(KID_SQ_PARTIALS, twopass, [&](int i) { return Key{D[i].g_dtype, 0, 0, 1}; },
          [&](int i) { return (int64_t)geo[i].tiles_r * geo[i].tiles_c; });
    build(KID_SQ_FINALIZE, is2d, nokey, [&](int i) { return (int64_t)geo[i].nbR + geo[i].nbC; });
    // (also for fused-first-pass tensors that carry the clamps: those CTAs return at once unless a clamp binds)
    auto needs_sumsq = [&](int i) { return twopass(i) || (fusedA(i) && (D[i].flags & CAME_F_SQ_CLAMP)); };
    build(KID_SUMSQ, needs_sumsq, [&](int i) { return Key{D[i].g_dtype, 0, 0, 1}; },
          [&](int i) { return (int64_t)geo[i].tiles_r * geo[i].tiles_c; });
    // one CTA per S_FIN_CHUNK entries of a tensor's factor vectors (each CTA repeats the cheap scalar part)
    build(KID_S_FINALIZE, is2d, nokey, [&](int i) { return std::max<int64_t>(1, cdiv(D[i].rows + D[i].cols, S_FIN_CHUNK)); });
    // Tensors of the tile layout on the staged path (same element type for g and p) take the fused kernel: their M, F
    // and A items form one list, a tensor's F and A items delayed by `lag` momentum items of later tensors.
    std::vector<char> fused(n_tensors, 0);
    if (!disable_fast() && fused_ma_enabled()) {
        for (int i = 0; i < n_tensors; ++i)
            fused[i] = is2d(i) && D[i].g_dtype == D[i].p_dtype && D[i].mode != CAME_MODE_FP32;
    }
    {
        const int grid = persistent_grid_limit();
        const size_t lag_a = (size_t)std::max(0, env_int("CAME_B200_MA_LAG", 5 * grid));
        const bool reverse_a = env_int("CAME_B200_MA_REVERSE", 1) != 0;
        const bool interleave = env_int("CAME_B200_MA_INTERLEAVE", 1) != 0;
        for (int dm = 0; dm < 6; ++dm) {
            const int dt = CAME_DT_F32 + dm % 3, md = dm < 3 ? CAME_MODE_TILE8 : CAME_MODE_FLAT8;
            LaunchItem it{};
            it.kernel = KID_MOMENT_APPLY;
            it.key = KernelKey{dt, dt, md, 2};
            it.work_off = work.size();
            struct Burst { size_t release; int tensor; };
            std::vector<Burst> pend;      // apply bursts waiting for their place in the list
            size_t next = 0, emitted = 0;
            auto burst = [&](const Burst& b) {
                const int64_t c = (int64_t)geo[b.tensor].ptiles_r * geo[b.tensor].ptiles_c;
                // the tiles written last are the likeliest to be still in L2: the apply items of a tensor run through its
                // tiles in the reverse order (CAME_B200_MA_REVERSE=0: same order as the momentum items)
                for (int64_t k = 0; k < c; ++k)
                    work.push_back(Work{b.tensor, (int32_t)(((uint32_t)MA_KIND_A << 28) | (uint32_t)(reverse_a ? c - 1 - k : k))});
            };
            // A released burst is dealt out one apply item per momentum item instead of all at once (CAME_B200_MA_INTERLEAVE=0:
            // all at once): DRAM-bound apply items and issue-bound momentum items then share the GPU at all times
            std::vector<Work> trickle;
            size_t tnext = 0;
            auto release = [&](const Burst& b) {
                if (!interleave) { burst(b); return; }
                const size_t before = work.size();
                burst(b);
                trickle.insert(trickle.end(), work.begin() + before, work.end());
                work.resize(before);
            };
            for (int i = 0; i < n_tensors; ++i) {
                if (!fused[i] || D[i].g_dtype != dt || D[i].mode != md) continue;
                const int64_t c = (int64_t)geo[i].ptiles_r * geo[i].ptiles_c;
                for (int64_t k = 0; k < c; ++k) {
                    work.push_back(Work{i, (int32_t)(((uint32_t)MA_KIND_M << 28) | (uint32_t)k)});
                    ++emitted;
                    while (next < pend.size() && pend[next].release <= emitted) release(pend[next++]);
                    if (tnext < trickle.size()) work.push_back(trickle[tnext++]);
                }
                pend.push_back(Burst{emitted + lag_a, i});
            }
            while (next < pend.size()) release(pend[next++]);
            while (tnext < trickle.size()) work.push_back(trickle[tnext++]);
            it.n = (int)(work.size() - it.work_off);
            it.work2_off = work.size();
            for (int i = 0; i < n_tensors; ++i) {
                if (!fused[i] || D[i].g_dtype != dt || D[i].mode != md) continue;
                for (int k = 0; k < geo[i].nbR + geo[i].nbC; ++k) work.push_back(Work{i, k});
            }
            it.n2 = (int)(work.size() - it.work2_off);
            if (it.n > 0) { plan->launches.push_back(it); plan->has_fused_ma = true; }
        }
    }
    plan->fused = fused;
    plan->pushable = plan->push_must = fused;
    for (int i = 0; i < n_tensors; ++i) {
        plan->pushable[i] = fused[i] || isgen(i);
        plan->push_must[i] = fused[i] || (isgen(i) && vf[i].wide && fused_ma_enabled() && D[i].g_dtype == D[i].p_dtype && D[i].mode != CAME_MODE_FP32);
    }
    // The momentum pass, the residual finalize and the apply pass run wave by wave: a wave is a run of consecutive
    // tensors whose momentum state together stays below `wave_bytes`, so that the codes the momentum pass writes are
    // still in L2 when the apply pass reads them back (0: one wave, every pass covers all tensors).
    std::vector<int> wave(n_tensors, 0);
    int n_waves = 1;
    if (g_wave_bytes > 0) {
        size_t acc = 0;
        int w = 0;
        for (int i = 0; i < n_tensors; ++i) {
            if (D[i].cols == 0) { wave[i] = 0; continue; }
            const size_t mb = (size_t)D[i].rows * (size_t)D[i].cols * (D[i].mode == CAME_MODE_FP32 ? 4 : 1);
            if (acc > 0 && acc + mb > g_wave_bytes) { ++w; acc = 0; }
            wave[i] = w;
            acc += mb;
        }
        n_waves = w + 1;
    }
    for (int w = 0; w < n_waves; ++w) {
        auto in2d = [&](int i) { return is2d(i) && wave[i] == w && !fused[i]; };
        auto in_notflat = [&](int i) { return in2d(i) && D[i].mode != CAME_MODE_FLAT8; };
        auto in_flat = [&](int i) { return in2d(i) && D[i].mode == CAME_MODE_FLAT8; };
        auto tiles = [&](int i) { return (int64_t)geo[i].ptiles_r * geo[i].ptiles_c; };
        build(KID_MOMENT, in2d, [&](int i) { return Key{D[i].g_dtype, 0, D[i].mode, 2}; }, tiles);
        build(KID_RES_FINALIZE, in2d, nokey, [&](int i) { return (int64_t)geo[i].nbR + geo[i].nbC; });
        build(KID_APPLY, in_notflat, [&](int i) { return Key{0, D[i].p_dtype, D[i].mode, 2}; }, tiles);
        build(KID_APPLY_FLAT, in_flat, [&](int i) { return Key{D[i].g_dtype, D[i].p_dtype, 0, 2}; }, tiles);
    }

    if (work.size() > L.n_work) {
        delete plan;
        return fail(CAME_E_INVALID, "plan_create: internal work-list overflow (%zu > %zu)", work.size(), L.n_work);
    }

    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemcpyAsync(plan->ws + L.off_descs, plan->descs.data(), (size_t)n_tensors * sizeof(CameTensorDesc),
                                    cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(plan->ws + L.off_scr, scr.data(), (size_t)n_tensors * sizeof(Scratch), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(plan->ws + L.off_status, 0, L.off_work - L.off_status, st);      // status word, barriers, counters
    // the scratch starts at zero once (flags in it are reset by the kernels that use them)
    if (e == cudaSuccess) e = cudaMemsetAsync(plan->ws + L.off_float, 0, L.total - L.off_float, st);
    if (e == cudaSuccess && !work.empty())
        e = cudaMemcpyAsync(plan->ws + L.off_work, work.data(), work.size() * sizeof(Work), cudaMemcpyHostToDevice, st);
    // the host vectors above die at return: wait for the copies
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess)
        e = cudaHostAlloc(reinterpret_cast<void**>(&plan->graph_hyp), (size_t)MAX_GROUPS * sizeof(CameHyper), cudaHostAllocDefault);
    if (e != cudaSuccess) {
        delete plan;
        return fail(CAME_E_CUDA, "plan_create: %s", cudaGetErrorString(e));
    }
    for (const LaunchItem& it : plan->launches) plan->needs_hyp = plan->needs_hyp || it.kernel != KID_GENERIC;
    *out = plan;
    return CAME_OK;
}

void came_b200_plan_destroy(came_plan_t* plan) { delete plan; }

// push mode: the whole parameter must lie inside the local buffer the peers mirror
static bool param_in_range(uintptr_t buf_lo, uintptr_t buf_hi, const CameTensorDesc& d) {
    const uintptr_t lo = reinterpret_cast<uintptr_t>(d.p);
    const uintptr_t bytes = (uintptr_t)d.rows * (uintptr_t)(d.cols ? d.cols : 1) * (uintptr_t)(d.batch > 1 ? d.batch : 1) *
                            (uintptr_t)elem_bytes(d.p_dtype);
    return lo >= buf_lo && lo + bytes <= buf_hi;
}
static bool pushed_param_in_range(const came_plan& plan, const CameTensorDesc& d) {
    return param_in_range(plan.push_lo, plan.push_hi, d);
}

int came_b200_plan_set_push(came_plan_t* plan, const void* local_base, size_t local_bytes, void* const* peer_bases, int n_peers) {
    if (!plan) return fail(CAME_E_INVALID, "plan_set_push: plan is null");
    if (n_peers == 0) { plan->n_push = 0; return CAME_OK; }
    if (n_peers < 0 || n_peers > MAX_PUSH_PEERS) return fail(CAME_E_INVALID, "plan_set_push: %d peers outside [0, %d]", n_peers, MAX_PUSH_PEERS);
    if (!local_base || !peer_bases || local_bytes == 0) return fail(CAME_E_INVALID, "plan_set_push: null argument");
    const uintptr_t buf_lo = reinterpret_cast<uintptr_t>(local_base), buf_hi = buf_lo + local_bytes;
    if (buf_lo % 16 != 0) return fail(CAME_E_INVALID, "plan_set_push: the local buffer is not 16-byte aligned");
    for (int i = 0; i < plan->n_tensors; ++i)
        if (plan->push_must[i] && !param_in_range(buf_lo, buf_hi, plan->descs[i]))
            return fail(CAME_E_INVALID, "plan_set_push: tensor %d does not lie inside the local buffer", i);
    long long delta[MAX_PUSH_PEERS];
    for (int k = 0; k < n_peers; ++k) {
        const uintptr_t pb = reinterpret_cast<uintptr_t>(peer_bases[k]);
        if (!pb || pb % 16 != 0) return fail(CAME_E_INVALID, "plan_set_push: peer buffer %d is null or not 16-byte aligned", k);
        if (pb < buf_hi && pb + local_bytes > buf_lo) return fail(CAME_E_INVALID, "plan_set_push: peer buffer %d overlaps the local one", k);
        delta[k] = (long long)(pb - buf_lo);      // modular: the kernel adds it to a local address
    }
    plan->push_lo = buf_lo; plan->push_hi = buf_hi;
    for (int k = 0; k < n_peers; ++k) plan->push_delta[k] = delta[k];
    plan->n_push = n_peers;
    return CAME_OK;
}

int came_b200_plan_pushed(const came_plan_t* plan, int* flags, int n_tensors) {
    if (!plan || !flags) return fail(CAME_E_INVALID, "plan_pushed: null argument");
    if (n_tensors != plan->n_tensors) return fail(CAME_E_INVALID, "plan_pushed: %d tensors given, plan has %d", n_tensors, plan->n_tensors);
    for (int i = 0; i < n_tensors; ++i)
        flags[i] = plan->pushable[i] && (plan->n_push == 0 || pushed_param_in_range(*plan, plan->descs[i])) ? 1 : 0;
    return CAME_OK;
}

int came_b200_plan_set_pointers(came_plan_t* plan, const void* const* g, void* const* p, int n_tensors, came_stream_t stream) {
    if (!plan) return fail(CAME_E_INVALID, "set_pointers: plan is null");
    if (n_tensors != plan->n_tensors) return fail(CAME_E_INVALID, "set_pointers: %d tensors given, plan has %d", n_tensors, plan->n_tensors);
    if (!g && !p) return CAME_OK;
    // (only the addresses change: nothing is copied back when one of them is refused)
    const bool fast = !disable_fast();
    for (int i = 0; i < n_tensors; ++i) {
        CameTensorDesc next = plan->descs[i];
        if (g) next.g = g[i];
        if (p) next.p = p[i];
        if (!next.g || !next.p) return fail(CAME_E_INVALID, "set_pointers: tensor %d: null pointer", i);
        if (!(vec_flags(next, fast) == plan->vflags[i]))
            return fail(CAME_E_INVALID, "set_pointers: tensor %d changes 16-byte alignment class; create a new plan", i);
        if (plan->n_push > 0 && plan->pushable[i] && pushed_param_in_range(*plan, plan->descs[i]) && !pushed_param_in_range(*plan, next))
            return fail(CAME_E_INVALID, "set_pointers: tensor %d leaves the buffer the push mode was set up for", i);
    }
    for (int i = 0; i < n_tensors; ++i) {
        if (g) plan->descs[i].g = g[i];
        if (p) plan->descs[i].p = p[i];
    }
    // pageable copies up to 64 KB return as soon as they are staged; longer ones wait for the stream
    const size_t total = (size_t)n_tensors * sizeof(CameTensorDesc), piece = 48 * 1024;
    const char* src = reinterpret_cast<const char*>(plan->descs.data());
    for (size_t at = 0; at < total; at += piece) {
        const cudaError_t e = cudaMemcpyAsync(plan->ws + plan->L.off_descs + at, src + at, std::min(piece, total - at),
                                              cudaMemcpyHostToDevice, (cudaStream_t)stream);
        if (e != cudaSuccess) return fail(CAME_E_CUDA, "set_pointers: %s", cudaGetErrorString(e));
    }
    return CAME_OK;
}

int came_b200_plan_set_hyper(came_plan_t* plan, const CameHyper* hypers, int n_groups) {
    int rc = check_hypers("plan_set_hyper", plan, hypers, n_groups);
    if (rc != CAME_OK) return rc;
    if (plan->graph_groups && n_groups != plan->graph_groups)
        return fail(CAME_E_INVALID, "plan_set_hyper: %d groups given, the captured step has %d", n_groups, plan->graph_groups);
    return stage_graph_hypers("plan_set_hyper", plan, hypers, n_groups);
}

int came_b200_step(came_plan_t* plan, const CameHyper* hypers, int n_groups, came_stream_t stream) {
    int rc = check_hypers("step", plan, hypers, n_groups);
    if (rc != CAME_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    // While the stream is being captured into a CUDA graph the upload must read memory that outlives the call:
    // the plan's page-locked copy, which came_b200_plan_set_hyper rewrites between replays.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) { cap = cudaStreamCaptureStatusNone; cudaGetLastError(); }
    const bool capturing = cap == cudaStreamCaptureStatusActive;
    CameHyper norm[MAX_GROUPS];      // pageable source: read before the copy call returns
    std::memcpy(norm, hypers, (size_t)n_groups * sizeof(CameHyper));
    normalise_hypers(norm, n_groups);
    const CameHyper* src = norm;
    if (capturing) {
        rc = stage_graph_hypers("step", plan, hypers, n_groups);
        if (rc != CAME_OK) return rc;
        src = plan->graph_hyp;
    }
    // The whole-step kernel takes a few records as kernel arguments; a captured step reads them from memory, so that a
    // replay sees new values.
    const bool by_value = !capturing && n_groups <= GENERIC_MAX_HYP;
    cudaError_t e = cudaSuccess;
    if (plan->needs_hyp || !by_value) {
        e = cudaMemcpyAsync(plan->ws + plan->L.off_hyp, src, (size_t)n_groups * sizeof(CameHyper), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return fail(CAME_E_CUDA, "step: hyper-parameter upload: %s", cudaGetErrorString(e));
    }
    const bool timing = plan->timing && !capturing;      // events are not recorded into a graph
    StepArgs a{reinterpret_cast<const CameTensorDesc*>(plan->ws + plan->L.off_descs),
               reinterpret_cast<const Scratch*>(plan->ws + plan->L.off_scr),
               reinterpret_cast<const CameHyper*>(plan->ws + plan->L.off_hyp),
               reinterpret_cast<int*>(plan->ws + plan->L.off_status), plan->n_push, 0, {}, plan->push_lo, plan->push_hi};
    for (int k = 0; k < plan->n_push; ++k) a.push_delta[k] = plan->push_delta[k];
    const Work* wbase = reinterpret_cast<const Work*>(plan->ws + plan->L.off_work);
    int* sync = reinterpret_cast<int*>(plan->ws + plan->L.off_sync);
    if (plan->has_fused_ma) {      // the per-tensor item counters start every step at zero
        e = cudaMemsetAsync(sync, 0, (2 * (size_t)plan->n_tensors + 12) * sizeof(int), st);
        if (e != cudaSuccess) return fail(CAME_E_CUDA, "step: counter reset: %s", cudaGetErrorString(e));
    }
    int launches = 0, fused_launches = 0;
    for (const LaunchItem& it : plan->launches) {
        came_plan::Timed tm{it.kernel, nullptr, nullptr};
        if (timing) {
            if (cudaEventCreate(&tm.t0) != cudaSuccess || cudaEventCreate(&tm.t1) != cudaSuccess)
                return fail(CAME_E_CUDA, "step: cudaEventCreate failed");
            cudaEventRecord(tm.t0, st);
        }
        if (it.kernel == KID_GENERIC) {
            const GenericLists l{wbase + it.work_off, wbase + it.work2_off, wbase + it.work3_off, wbase + it.work4_off,
                                 it.n, it.n2, it.n3, it.n4, reinterpret_cast<uint32_t*>(plan->ws + plan->L.off_bar) + it.bar};
            e = launch_generic(it.key, a, by_value ? norm : nullptr, n_groups, l, st);
        }
        else if (it.kernel == KID_SQ_PARTIALS && it.key.variant == 2)
            e = launch_fused_sq(it.key, a, wbase + it.work_off, it.n, st);
        else if (it.kernel >= KID_ND_SQ && it.kernel <= KID_ND_APPLY)
            e = launch_nd(it.kernel, it.key, a, wbase + it.work_off, it.n, st);
        else if (it.kernel == KID_MOMENT_APPLY)
            e = launch_fused_ma(it.key, a, wbase + it.work_off, it.n, wbase + it.work2_off, it.n2, sync, sync + plan->n_tensors,
                                sync + 2 * plan->n_tensors + 2 * (fused_launches++ % 6), st);      // two list cursors per launch (at most 6)
        else
            e = launch_factored(it.kernel, it.key, a, wbase + it.work_off, it.n, st);
        if (timing) {
            cudaEventRecord(tm.t1, st);
            plan->timed.push_back(tm);
        }
        if (e != cudaSuccess) return fail(CAME_E_CUDA, "step: kernel %d: %s", it.kernel, cudaGetErrorString(e));
        ++launches;
    }
    plan->last_launches = launches;
    return CAME_OK;
}

int came_b200_peer_copy_async(void* dst, const void* src, size_t bytes, int src_device, came_stream_t stream) {
    if (!dst || !src) return fail(CAME_E_INVALID, "peer_copy_async: null pointer");
    if (bytes == 0) return CAME_OK;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(CAME_E_CUDA, "peer_copy_async: %s", cudaGetErrorString(e));
    if (src_device >= 0 && src_device != dev) {
        e = cudaDeviceEnablePeerAccess(src_device, 0);
        if (e == cudaErrorPeerAccessAlreadyEnabled) { cudaGetLastError(); e = cudaSuccess; }
        if (e != cudaSuccess) return fail(CAME_E_CUDA, "peer_copy_async: enabling access to GPU %d: %s", src_device, cudaGetErrorString(e));
    }
    e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "peer_copy_async: %s", cudaGetErrorString(e));
}

int came_b200_ipc_export(const void* ptr, unsigned char handle[CAME_B200_IPC_HANDLE_BYTES], uint64_t* offset) {
    static_assert(sizeof(cudaIpcMemHandle_t) == CAME_B200_IPC_HANDLE_BYTES, "IPC handle size");
    if (!ptr || !handle || !offset) return fail(CAME_E_INVALID, "ipc_export: null argument");
    // base of the allocation that contains ptr (driver entry point: the runtime has no such query)
    typedef int (*range_fn)(unsigned long long*, size_t*, unsigned long long);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || !fn) return fail(CAME_E_CUDA, "ipc_export: cuMemGetAddressRange is not available");
    unsigned long long base = 0;
    size_t size = 0;
    if (reinterpret_cast<range_fn>(fn)(&base, &size, (unsigned long long)(uintptr_t)ptr) != 0)
        return fail(CAME_E_CUDA, "ipc_export: the pointer is not inside a device allocation");
    cudaIpcMemHandle_t h;
    e = cudaIpcGetMemHandle(&h, reinterpret_cast<void*>((uintptr_t)base));
    if (e != cudaSuccess) return fail(CAME_E_CUDA, "ipc_export: %s", cudaGetErrorString(e));
    std::memcpy(handle, &h, sizeof(h));
    *offset = (uint64_t)((uintptr_t)ptr - (uintptr_t)base);
    return CAME_OK;
}

int came_b200_ipc_open(const unsigned char handle[CAME_B200_IPC_HANDLE_BYTES], void** base) {
    if (!handle || !base) return fail(CAME_E_INVALID, "ipc_open: null argument");
    cudaIpcMemHandle_t h;
    std::memcpy(&h, handle, sizeof(h));
    const cudaError_t e = cudaIpcOpenMemHandle(base, h, cudaIpcMemLazyEnablePeerAccess);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "ipc_open: %s", cudaGetErrorString(e));
}

int came_b200_ipc_close(void* base) {
    if (!base) return CAME_OK;
    const cudaError_t e = cudaIpcCloseMemHandle(base);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "ipc_close: %s", cudaGetErrorString(e));
}

int came_b200_selftest_bounded_wait(int* device_words, came_stream_t stream) {
    if (!device_words) return fail(CAME_E_INVALID, "selftest_bounded_wait: device_words is null");
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(device_words, 0xff, 3 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(device_words, 0, sizeof(int), st);
    if (e == cudaSuccess) e = launch_selftest_bounded_wait(device_words, device_words + 1, st);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "selftest_bounded_wait: %s", cudaGetErrorString(e));
}

int came_b200_selftest_grid_barrier(int* device_words, came_stream_t stream) {
    if (!device_words) return fail(CAME_E_INVALID, "selftest_grid_barrier: device_words is null");
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(device_words, 0xff, 10 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(device_words, 0, 2 * sizeof(int), st);
    if (e == cudaSuccess) e = launch_selftest_grid_barrier(device_words, st);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "selftest_grid_barrier: %s", cudaGetErrorString(e));
}

int came_b200_plan_last_launches(const came_plan_t* plan) { return plan ? plan->last_launches : 0; }

int came_b200_plan_status(came_plan_t* plan, came_stream_t stream, int* status) {
    if (!plan || !status) return fail(CAME_E_INVALID, "plan_status: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemcpyAsync(status, plan->ws + plan->L.off_status, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? CAME_OK : fail(CAME_E_CUDA, "plan_status: %s", cudaGetErrorString(e));
}

int came_b200_plan_set_timing(came_plan_t* plan, int enable) {
    if (!plan) return fail(CAME_E_INVALID, "set_timing: plan is null");
    plan->timing = enable != 0;
    return CAME_OK;
}

int came_b200_plan_read_timing(came_plan_t* plan, float* ms, int* launches) {
    if (!plan || !ms || !launches) return fail(CAME_E_INVALID, "read_timing: null argument");
    static_assert(CAME_KERNEL_COUNT == KID_COUNT, "header and kernel table out of sync");
    for (int k = 0; k < CAME_KERNEL_COUNT; ++k) { ms[k] = 0.0f; launches[k] = 0; }
    int rc = CAME_OK;
    for (auto& t : plan->timed) {
        float dt = 0.0f;
        cudaError_t e = cudaEventSynchronize(t.t1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&dt, t.t0, t.t1);
        if (e == cudaSuccess) { ms[t.kernel] += dt; launches[t.kernel] += 1; }
        else rc = fail(CAME_E_CUDA, "read_timing: %s", cudaGetErrorString(e));
        cudaEventDestroy(t.t0);
        cudaEventDestroy(t.t1);
    }
    plan->timed.clear();
    return rc;
}

const char* came_b200_kernel_name(int kernel) {
    static const char* names[CAME_KERNEL_COUNT] = {
        "sq_partials", "sq_finalize", "sumsq", "s_finalize", "moment", "res_finalize",
        "apply", "generic", "apply_flat", "?", "?", "?", "nd_sq", "nd_mean", "nd_sumsq", "nd_s", "nd_res",
        "nd_resmean", "nd_apply", "moment_apply"};
    return (kernel >= 0 && kernel < CAME_KERNEL_COUNT) ? names[kernel] : "?";
}

}  // extern "C"
