// Shared internals of libantipodal_gb300: error reporting, the context (stream, scratch arena, options,
// timing), host/device pointer handling and small device helpers.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/antipodal_gb300.h"
#include "intfp.cuh"

namespace agwn
{
// ---- errors --------------------------------------------------------------------------------------------------
void set_message(const char* fmt, ...);
int fail(int status, const char* fmt, ...);
void clear_message();

#define AGWN_TRY_CUDA(expr)                                                                                        \
    do                                                                                                             \
    {                                                                                                              \
        cudaError_t agwn_e_ = (expr);                                                                              \
        if (agwn_e_ != cudaSuccess)                                                                                \
            return ::agwn::fail(agwn_e_ == cudaErrorMemoryAllocation ? AGWN_ERR_NOMEM : AGWN_ERR_CUDA,             \
                                "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(agwn_e_), __FILE__, __LINE__); \
    } while (0)

#define AGWN_TRY(expr)                                                                                             \
    do                                                                                                             \
    {                                                                                                              \
        int agwn_s_ = (expr);                                                                                      \
        if (agwn_s_ != AGWN_OK)                                                                                    \
            return agwn_s_;                                                                                        \
    } while (0)

#define AGWN_CHECK_ARG(cond, ...)                                                                                  \
    do                                                                                                             \
    {                                                                                                              \
        if (!(cond))                                                                                               \
            return ::agwn::fail(AGWN_ERR_INVALID, __VA_ARGS__);                                                    \
    } while (0)

// Device-side error flags, one word each, set with atomicOr by kernels and read by the host at synchronisation.
constexpr int kCounters = 12; // device statistics counters of a context

enum flag_slot
{
    FLAG_STACK = 0,   // traversal stack exhausted
    FLAG_TIMEOUT = 1, // bounded wait ran out
    FLAG_COUNT = 8
};

// ---- device scratch ----------------------------------------------------------------------------------------
// A grow-only device buffer.  Slots are reused across calls of one context.
struct DevBuf
{
    void* ptr = nullptr;
    size_t cap = 0;
    // Room for `bytes`, with a quarter more while that stays within `most` and there is memory for it.
    int reserve(size_t bytes, size_t most = SIZE_MAX);
    void release();
};

// Build temporaries of one context, taken and given back in stack order on the context's stream: cudaMalloc and
// cudaFree cost more than most of the kernels between them (and a free waits for the device).  The memory stays for
// the context's next build, up to kKeep bytes.
struct Arena
{
    static constexpr size_t kKeep = size_t(1) << 30;
    struct Chunk
    {
        char* ptr;
        size_t cap, used;
    };
    std::vector<Chunk> chunks;
    int depth = 0;
    size_t limit = SIZE_MAX; // of all chunks together
    int take(size_t bytes, void** out);
    void release();
};

enum scratch_slot
{
    S_QUERIES = 0,
    S_OUT = 1,
    S_COUNTS = 2,
    S_SEGS = 3,
    S_SEGS_RAW = 4,
    S_FRAME = 5,
    S_MISC0 = 6,
    S_MISC1 = 7,
    S_MISC2 = 8,
    S_MISC3 = 9,
    S_PARTIAL = 10, // the split exact kernels' terms; the parametric integrator's pair counter
    S_ORDER0 = 11,  // the spatial order of the queries: sort keys, indices, digit counters (order.cu)
    S_ORDER1 = 12,  // the queries in that order and their outputs
    S_COUNT = 13
};

// A hierarchy over triangles in the frame of one ray direction (built by build_hier, lbvh.cu): internal nodes,
// the triangles in leaf order, their projected (u, v) corners, the frame and the depth.
struct Hier
{
    DevBuf nodes;
    DevBuf tri;
    DevBuf leaf_uv;
    int32_t depth = 0;
    int64_t n_tri = 0;
    float frame[9] = {};
    double scale = 1.0; // largest |coordinate| of the triangles
    float ext[4] = {};  // min u, min v, max u, max v of the leaves' float corners (min above max: none finite)
    void release()
    {
        nodes.release();
        tri.release();
        leaf_uv.release();
    }
};

// A uniform grid over the (u, v) plane of a ray-frame hierarchy: per cell (CSR), the leaves whose (u, v) box,
// widened by `margin`, overlaps the cell (lbvh.cu).
struct CellGrid
{
    DevBuf offsets; // n_cells + 1 unsigned
    DevBuf list;    // leaf indices
    int gu = 0, gv = 0;
    float umin = 0, vmin = 0, umax = 0, vmax = 0, inv_u = 0, inv_v = 0;
    float margin = 0;  // the widening of every leaf's box
    float tol_max = 0; // queries whose own tolerance exceeds this take the hierarchy walk
    int64_t entries = 0;
    int per_leaf = 0;   // cells per leaf it was built with
    int64_t calls = 0;  // calls prepared for on this hierarchy so far
    bool pinned = false; // a captured call reads it: no finer grid takes its place while this hierarchy is cached
    bool valid = false;
    void release()
    {
        offsets.release();
        list.release();
        valid = false;
    }
};

// The hierarchy of one intersector along one direction, cached per context.  Keyed by the intersector's
// generation number and the direction's bits.
struct RayCache
{
    unsigned long long generation = 0;
    double dir[3] = {0, 0, 0};
    int scalar_bytes = 0;
    Hier h;
    CellGrid cells; // built on first use, invalid whenever h is rebuilt
};

struct Context
{
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int* d_flags = nullptr;        // FLAG_COUNT ints
    int* h_flags = nullptr;        // pinned mirror
    long long* d_counters = nullptr; // kCounters: [0] fp64 pairs, [1] pairs, [2] parametric skips, [3] certified pairs, [4..7] integer, [8..11] patches
                                     // term: queries, cell-list entries, candidate leaves, exact tests
    DevBuf scratch[S_COUNT];
    // Buffers that a captured call was given: a graph holds their addresses, so one that has to grow is set aside, not
    // freed, until the context ends or is trimmed.
    bool scratch_captured[S_COUNT] = {};
    std::vector<void*> set_aside;
    Arena arena;
    static constexpr int kArrivals = 2048;
    int* d_arrivals = nullptr; // kArrivals zeroed counters, left zeroed by each kernel that uses them
    int sm_count = 0;
    RayCache ray_cache;
    DevBuf bernstein; // the exact parametric integrator's node bases (param.cu), filled on first use
    bool bernstein_filled = false;
    // host-array pipeline (mesh batch): upload and download streams and their events, created on first use
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    cudaStream_t compute2 = nullptr; // the host-array pipeline runs alternate chunks' kernels here
    cudaEvent_t pipe_ev[8] = {};
    int ensure_pipeline();

    // options
    int frac_mode = AGWN_FRAC_EXACT;
    double mixed_tau = 4.0;
    double mixed_term_err = 6e-8;
    int robust_mode = AGWN_ROBUST_EXACT;
    double robust_term_err = 1e-7;
    int param_mode = AGWN_PARAM_EXACT;
    const agwn_mlp* panel_mlp = nullptr; // the per-panel network of the double-float integrator (or none)
    float panel_beta = 0.02f;
    int integer_cells = 1;
    double mixed_min_pairs = double(1 << 14);
    bool mixed_certify = true;
    // the spatial order of the queries (order.cu): the last decision and its key, and whether an evaluation on an
    // ordered copy is running (no second ordering inside it)
    const void* order_ptr = nullptr;
    int64_t order_n = 0;
    double order_dir[3] = {0, 0, 0};
    bool order_incoherent = false;
    float order_lo[2] = {0.f, 0.f};
    float order_scale = 1.f;
    bool ordering = false;
    int queries_per_thread = 2;
    int frac_block = 0; // 0: chosen per launch (frac.cu)
    int seg_tile = 512;
    int timing = 0;
    size_t scratch_limit = SIZE_MAX; // the largest scratch buffer of a call

    // statistics
    double kernel_ms[AGWN_K_COUNT] = {};
    long long launches[AGWN_K_COUNT] = {};
    static constexpr int kMaxPending = 64;
    cudaEvent_t ev_begin[kMaxPending] = {};
    cudaEvent_t ev_end[kMaxPending] = {};
    int pending_class[kMaxPending] = {};
    int n_pending = 0;

    // Whether a mixed-mode call of `pairs` (query, segment) pairs over a boundary of n_seg segments runs the mixed
    // kernels: at least mixed_min_pairs pairs over at least kMixedMinSegments segments, or always with the minimum 0.
    // The mixed kernel has a fixed part (the boundary's preparation) and, over long segments, many pairs within the near
    // distance that go to FP64 anyway.  The line was drawn where the two met when the exact kernels took 8 us a segment:
    // faster below 32 segments at every query count tried (2,000 to 200,000 random queries).  They take less now (257
    // queries x 24 segments 55 us, 261,632 x 102 2.1 ms), but the two forms' values differ by up to 6e-8 a term, so the
    // line stays where calls expect it.
    static constexpr int64_t kMixedMinSegments = 32;
    bool use_mixed(double pairs, int64_t n_seg) const
    {
        return mixed_min_pairs == 0.0 || (pairs >= mixed_min_pairs && n_seg >= kMixedMinSegments);
    }

    int scratch_reserve(int slot, size_t bytes, void** out);
    void scratch_drop(int slot); // frees a slot's buffer (nothing queued reads it), or sets it aside
    // scratch_reserve of fixed + unit * *units bytes; *units is halved, down to 1, while there is no memory for them
    int scratch_reserve_units(int slot, size_t fixed, size_t unit, int64_t* units, void** out);
    // Brackets a launch with timing events when AGWN_OPT_TIMING is on; always counts the launch.
    int launch_begin(int kclass);
    int launch_end(int kclass);
    int drain_timing(); // folds finished events into kernel_ms (synchronises the stream)
    int check_flags();  // synchronises and reports device flags
};

// The temporaries taken between its construction and its destruction.
class ArenaScope
{
public:
    explicit ArenaScope(Context& ctx);
    ~ArenaScope();
    ArenaScope(ArenaScope const&) = delete;
    ArenaScope& operator=(ArenaScope const&) = delete;

private:
    Context& ctx_;
    size_t chunk_, used_;
};
// One temporary of the enclosing ArenaScope.
struct Tmp
{
    Context& ctx;
    void* p = nullptr;
    explicit Tmp(Context& c) : ctx(c) {}
    int alloc(size_t bytes) { return ctx.arena.take(bytes, &p); }
    template <class U>
    U* as() const
    {
        return static_cast<U*>(p);
    }
};

// ---- host/device pointers ----------------------------------------------------------------------------------
bool is_device_pointer(const void* p);

// Makes `count` elements of `src` readable by the device: returns src itself for device memory, else copies
// it into scratch `slot` on the context's stream.
int stage_in(Context& ctx, const void* src, size_t bytes, int slot, const void** dev);
// Output staging: returns `dst` for device memory, else scratch `slot`; `*host` tells whether a copy back is due.
int stage_out(Context& ctx, void* dst, size_t bytes, int slot, void** dev, bool* host);

// ---- parametric path (param.cu, mlp.cu) ----------------------------------------------------------------------
// Device-side runners behind the parametric entry points; all pointers are device memory of the context's GPU.
int param_run(Context& ctx, const double* d_pos, int64_t n, double* d_out, const double* x0, const double* d_curves,
              int64_t n_curves, int min_depth, int max_depth, double tol, const uint8_t* d_start, uint32_t* d_stats,
              int32_t* d_nodes, uint32_t* d_panel_log = nullptr, unsigned long long* d_log_count = nullptr,
              long long log_cap = 0);
// The device copies of a network's weights (BF16 layouts) and FP32 parameters.
void mlp_device_weights(const agwn_mlp* mlp, const void** bf16_weights, const float** params);
int mlp_propose_run(Context& ctx, const agwn_mlp* mlp, const double* d_pos, int64_t n, const double* x0,
                    const double* d_curves, int64_t n_curves, int n_classes, int min_depth, int max_depth, double tol,
                    float alpha, uint8_t* d_start, float* d_logits);

// ---- launch geometry ---------------------------------------------------------------------------------------
inline int div_up(int64_t a, int64_t b)
{
    return int((a + b - 1) / b);
}
} // namespace agwn

struct agwn_context : agwn::Context
{
};

// ---- device helpers ----------------------------------------------------------------------------------------
namespace agwn
{
// Unfused IEEE arithmetic.  Each operation rounds once, like the reference's default (FMA-free) CPU build, so a
// formula written with these reproduces the CPU's values exactly.  The intrinsics are never contracted.  Division
// and square root of doubles run on the integer pipe (intfp.cuh), with the same bits.
struct rd
{
    double v;
    rd() = default;
    __host__ __device__ __forceinline__ constexpr rd(double x) : v(x) {}
    __device__ __forceinline__ friend rd operator+(rd a, rd b) { return rd(__dadd_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rd operator-(rd a, rd b) { return rd(__dsub_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rd operator*(rd a, rd b) { return rd(__dmul_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rd operator/(rd a, rd b) { return rd(div_rn_int(a.v, b.v)); }
    __device__ __forceinline__ friend rd operator-(rd a) { return rd(-a.v); }
};
// The same values with the products on the integer pipe too (mul_rn_int), for kernels with warps enough to hide its
// longer chain: sums and products then issue side by side.
struct rdi
{
    double v;
    rdi() = default;
    __host__ __device__ __forceinline__ constexpr rdi(double x) : v(x) {}
    __device__ __forceinline__ friend rdi operator+(rdi a, rdi b) { return rdi(__dadd_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rdi operator-(rdi a, rdi b) { return rdi(__dsub_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rdi operator*(rdi a, rdi b) { return rdi(mul_rn_int(a.v, b.v)); }
    __device__ __forceinline__ friend rdi operator/(rdi a, rdi b) { return rdi(div_rn_int(a.v, b.v)); }
    __device__ __forceinline__ friend rdi operator-(rdi a) { return rdi(-a.v); }
};
struct rf
{
    float v;
    rf() = default;
    __device__ __forceinline__ constexpr rf(float x) : v(x) {}
    __device__ __forceinline__ friend rf operator+(rf a, rf b) { return rf(__fadd_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rf operator-(rf a, rf b) { return rf(__fsub_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rf operator*(rf a, rf b) { return rf(__fmul_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rf operator/(rf a, rf b) { return rf(__fdiv_rn(a.v, b.v)); }
    __device__ __forceinline__ friend rf operator-(rf a) { return rf(-a.v); }
};
template <class T>
struct exact_of;
template <>
struct exact_of<double>
{
    using type = rd;
};
template <>
struct exact_of<float>
{
    using type = rf;
};

template <class T>
struct exact_int_of
{
    using type = rf;
};
template <>
struct exact_int_of<double>
{
    using type = rdi;
};

__device__ __forceinline__ rd ex_sqrt(rd a)
{
    return rd(sqrt_rn_int(a.v));
}
__device__ __forceinline__ rdi ex_sqrt(rdi a)
{
    return rdi(sqrt_rn_int(a.v));
}
__device__ __forceinline__ rf ex_sqrt(rf a)
{
    return rf(__fsqrt_rn(a.v));
}
__device__ __forceinline__ double ex_atan2(rd y, rd x)
{
    return atan2_int(y.v, x.v);
}
__device__ __forceinline__ double ex_atan2(rdi y, rdi x)
{
    return atan2_int(y.v, x.v);
}
__device__ __forceinline__ float ex_atan2(rf y, rf x)
{
    return atan2f(y.v, x.v);
}

template <class S>
struct ev3
{
    S x, y, z;
};
template <class S>
__device__ __forceinline__ ev3<S> operator-(ev3<S> a, ev3<S> b)
{
    return {a.x - b.x, a.y - b.y, a.z - b.z};
}
template <class S>
__device__ __forceinline__ S edot(ev3<S> a, ev3<S> b)
{
    return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <class S>
__device__ __forceinline__ ev3<S> ecross(ev3<S> a, ev3<S> b)
{
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// Bounded spin limits: every device-side wait gives up after this many polls and raises FLAG_TIMEOUT.
constexpr long long kSpinLimit = 1ll << 22;
} // namespace agwn
