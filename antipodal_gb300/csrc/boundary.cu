// Open boundary of a triangle mesh on the device: build_boundary_segments (src/antipodal/math/common.hh:123-174).
// Every triangle edge u -> v adds +1 (u < v) or -1 (u >= v) to its undirected edge {min, max}; edges whose net count
// is not zero are emitted as weighted segments, directed lo -> hi when the count is positive and hi -> lo otherwise,
// with weight |count|.  The reference accumulates in a hash map and emits in the map's order; here the output is in
// ascending (lo, hi) order, deterministically.
//
// The edges are binned by their lower vertex (a counting sort); each edge then scans its bin -- a vertex's few edges --
// for its net count and for the emitted edges before it.  Eleven launches over the edges, against some 35 for a radix
// sort of 64-bit keys: 229,488 edges take 42 us of kernels instead of 186.  A bin longer than kBinMax (a vertex with hundreds of
// edges) would make the scans quadratic, so such a mesh takes the radix sort; so does one whose vertex array is far larger
// than its triangles use, where the counters would outweigh the edges.

#include "agwn_internal.cuh"
#include "radix.cuh"

#include <algorithm>

namespace agwn
{
namespace
{
constexpr int kScanBlock = 1024;

__global__ void k_edge_keys(const int32_t* __restrict__ idx, int64_t n_tri, int64_t nv,
                            unsigned long long* __restrict__ keys, int* __restrict__ vals, int* flags)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < 3 * n_tri;
         i += int64_t(gridDim.x) * blockDim.x)
    {
        int64_t const t = i / 3;
        int const e = int(i - 3 * t);
        int32_t const u = idx[3 * t + e], v = idx[3 * t + (e + 1) % 3];
        if (u < 0 || v < 0 || u >= nv || v >= nv)
        {
            atomicOr(flags + FLAG_COUNT - 1, 1); // the invalid-index slot, as in the hierarchy build
            keys[i] = 0ull;
            vals[i] = 0;
            continue;
        }
        unsigned long long const lo = unsigned(min(u, v)), hi = unsigned(max(u, v));
        keys[i] = (lo << 32) | hi;
        vals[i] = u < v ? 1 : -1;
    }
}

constexpr unsigned kBinMax = 512;

// state[0]: an out-of-range index; state[1]: a bin above kBinMax.
// rank[i]: edge i's place in its lower vertex's bin (0xffffffff for an invalid edge).
__global__ void k_edge_count(const int32_t* __restrict__ idx, int64_t n_tri, int64_t nv, unsigned* __restrict__ bins,
                             unsigned* __restrict__ rank, unsigned* __restrict__ state)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < 3 * n_tri;
         i += int64_t(gridDim.x) * blockDim.x)
    {
        int64_t const t = i / 3;
        int const e = int(i - 3 * t);
        int32_t const u = idx[3 * t + e], v = idx[3 * t + (e + 1) % 3];
        unsigned r = 0xffffffffu;
        if (u < 0 || v < 0 || u >= nv || v >= nv)
            state[0] = 1u;
        else
        {
            r = atomicAdd(bins + min(u, v), 1u);
            if (r >= kBinMax)
                state[1] = 1u;
        }
        rank[i] = r;
    }
}

// Edges into their bins: the lower vertex, and the upper one with the direction (bit 0: u < v).
__global__ void k_edge_place(const int32_t* __restrict__ idx, int64_t n_tri, const unsigned* __restrict__ bins,
                             const unsigned* __restrict__ rank, int* __restrict__ lo, unsigned* __restrict__ hi)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < 3 * n_tri;
         i += int64_t(gridDim.x) * blockDim.x)
    {
        int64_t const t = i / 3;
        int const e = int(i - 3 * t);
        if (rank[i] == 0xffffffffu)
            continue;
        int32_t const u = idx[3 * t + e], v = idx[3 * t + (e + 1) % 3];
        unsigned const slot = bins[min(u, v)] + rank[i];
        lo[slot] = min(u, v);
        hi[slot] = (unsigned(max(u, v)) << 1) | (u < v ? 1u : 0u);
    }
}

// net[i]: the net count of slot i's edge at its first slot in the bin, 0 at the others; emitted edges per lower vertex.
__global__ void k_edge_net(const int* __restrict__ lo, const unsigned* __restrict__ hi, int64_t m,
                           const unsigned* __restrict__ bins, const unsigned* __restrict__ state, int* __restrict__ net,
                           unsigned* __restrict__ emitted)
{
    if (state[0] || state[1])
        return;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
    {
        int const v = lo[i];
        unsigned const h = hi[i] >> 1, e = bins[v + 1];
        int sum = 0;
        bool first = true;
        for (unsigned j = bins[v]; j < e; ++j)
            if ((hi[j] >> 1) == h)
            {
                sum += (hi[j] & 1u) ? 1 : -1;
                first = first && j >= i;
            }
        net[i] = first ? sum : 0;
        if (first && sum != 0)
            atomicAdd(emitted + v, 1u);
    }
}

template <class T>
__global__ void k_edge_rows(const int* __restrict__ lo, const unsigned* __restrict__ hi, int64_t m,
                            const unsigned* __restrict__ bins, const int* __restrict__ net,
                            const unsigned* __restrict__ emitted, const T* __restrict__ verts, int64_t capacity,
                            T* __restrict__ out)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
    {
        int const s = net[i];
        if (s == 0)
            continue;
        int const v = lo[i];
        unsigned const h = hi[i] >> 1, e = bins[v + 1];
        int64_t row = emitted[v];
        for (unsigned j = bins[v]; j < e; ++j)
            row += net[j] != 0 && (hi[j] >> 1) < h ? 1 : 0;
        if (row >= capacity)
            continue;
        int64_t const a = s > 0 ? v : int64_t(h), b = s > 0 ? int64_t(h) : v;
        T* const o = out + 7 * row;
        for (int k = 0; k < 3; ++k)
        {
            o[k] = verts[3 * a + k];
            o[3 + k] = verts[3 * b + k];
        }
        o[6] = T(s > 0 ? s : -s);
    }
}

// Net count of each run of equal keys, at the run's first element (0 elsewhere), and whether it is emitted.
__global__ void k_edge_reduce(const unsigned long long* __restrict__ keys, const int* __restrict__ vals, int64_t m,
                              int* __restrict__ net, unsigned* __restrict__ emit)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
    {
        bool const head = i == 0 || keys[i] != keys[i - 1];
        int s = 0;
        if (head)
            for (int64_t j = i; j < m && keys[j] == keys[i]; ++j)
                s += vals[j];
        net[i] = s;
        emit[i] = head && s != 0 ? 1u : 0u;
    }
}

// Exclusive scan, phase 1: each block of kScanBlock flags -> its sum.
__global__ void __launch_bounds__(kScanBlock) k_scan_sums(const unsigned* __restrict__ f, int64_t m,
                                                          unsigned* __restrict__ sums)
{
    __shared__ unsigned part[kScanBlock / 32];
    int64_t const i = int64_t(blockIdx.x) * kScanBlock + threadIdx.x;
    unsigned v = i < m ? f[i] : 0u;
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        unsigned w = part[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1)
            w += __shfl_down_sync(0xffffffffu, w, o);
        if (threadIdx.x == 0)
            sums[blockIdx.x] = w;
    }
}

// Phase 3: positions = block offset (phase 2 scanned the sums) + exclusive scan within the block.
__global__ void __launch_bounds__(kScanBlock) k_scan_apply(const unsigned* __restrict__ f, int64_t m,
                                                           const unsigned* __restrict__ offs, unsigned* __restrict__ pos)
{
    __shared__ unsigned wsum[kScanBlock / 32];
    int64_t const i = int64_t(blockIdx.x) * kScanBlock + threadIdx.x;
    unsigned const v = i < m ? f[i] : 0u;
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v; // inclusive within the warp
    for (int o = 1; o < 32; o <<= 1)
    {
        unsigned const y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        wsum[warp] = x;
    __syncthreads();
    if (warp == 0)
    {
        unsigned w = wsum[lane];
        for (int o = 1; o < 32; o <<= 1)
        {
            unsigned const y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
                w += y;
        }
        wsum[lane] = w; // inclusive over warps
    }
    __syncthreads();
    unsigned const before = warp ? wsum[warp - 1] : 0u;
    if (i < m)
        pos[i] = offs[blockIdx.x] + before + x - v;
}

template <class T>
__global__ void k_edge_emit(const unsigned long long* __restrict__ keys, const int* __restrict__ net,
                            const unsigned* __restrict__ emit, const unsigned* __restrict__ pos, int64_t m,
                            int64_t capacity, const T* __restrict__ verts, T* __restrict__ out)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
    {
        if (!emit[i] || int64_t(pos[i]) >= capacity)
            continue;
        int64_t const lo = int64_t(keys[i] >> 32), hi = int64_t(keys[i] & 0xffffffffull);
        int const s = net[i];
        int64_t const a = s > 0 ? lo : hi, b = s > 0 ? hi : lo;
        T* const o = out + 7 * int64_t(pos[i]);
        for (int k = 0; k < 3; ++k)
        {
            o[k] = verts[3 * a + k];
            o[3 + k] = verts[3 * b + k];
        }
        o[6] = T(s > 0 ? s : -s);
    }
}

// Where the rows go: given their number by prepare, the first `rows` of them into the device array `dev`, then (finish)
// to `host` if that is the output.  out_for(number, &out, &rows) is the caller's choice of array and rows.
template <class T>
struct RowsOut
{
    T* dev = nullptr;
    T* host = nullptr;
    int64_t rows = 0;

    template <class OutFor>
    int prepare(Context& ctx, OutFor out_for, int64_t number)
    {
        T* out = nullptr;
        AGWN_TRY(out_for(number, &out, &rows));
        if (rows == 0)
            return AGWN_OK;
        dev = out;
        if (!is_device_pointer(out))
        {
            host = out;
            AGWN_TRY(ctx.scratch_reserve(S_MISC2, sizeof(T) * 7 * size_t(rows), reinterpret_cast<void**>(&dev)));
        }
        return AGWN_OK;
    }
    int finish(Context& ctx) const
    {
        if (rows == 0)
            return AGWN_OK;
        if (host)
            AGWN_TRY_CUDA(cudaMemcpyAsync(host, dev, sizeof(T) * 7 * size_t(rows), cudaMemcpyDeviceToHost, ctx.stream));
        return ctx.check_flags();
    }
};

// The extraction by radix sort (bins above kBinMax).
template <class T, class OutFor>
int boundary_radix(Context& ctx, const T* dv, int64_t nv, const int32_t* di, int64_t m, OutFor out_for, RowsOut<T>& o,
                   int64_t* n_segments)
{
    cudaStream_t const st = ctx.stream;
    ArenaScope scope(ctx);
    int const n_rs_blocks = int((m + kRsTile - 1) / kRsTile);
    int64_t const n_sb = (m + kScanBlock - 1) / kScanBlock;
    Tmp ka(ctx), kb(ctx), va(ctx), vb(ctx), hist(ctx), net(ctx), emit(ctx), pos(ctx), sums(ctx);
    AGWN_TRY(ka.alloc(sizeof(unsigned long long) * m));
    AGWN_TRY(kb.alloc(sizeof(unsigned long long) * m));
    AGWN_TRY(va.alloc(sizeof(int) * m));
    AGWN_TRY(vb.alloc(sizeof(int) * m));
    AGWN_TRY(hist.alloc(sizeof(unsigned) * 256 * size_t(n_rs_blocks)));
    Tmp hsum(ctx);
    AGWN_TRY(hsum.alloc(sizeof(unsigned) * size_t(scan_sums_count(int64_t(256) * n_rs_blocks))));
    AGWN_TRY(net.alloc(sizeof(int) * m));
    AGWN_TRY(emit.alloc(sizeof(unsigned) * m));
    AGWN_TRY(pos.alloc(sizeof(unsigned) * m));
    AGWN_TRY(sums.alloc(sizeof(unsigned) * size_t(n_sb)));
    int const grid = int(std::min<int64_t>(div_up(m, 256), 8 * ctx.sm_count));
    AGWN_TRY_CUDA(cudaMemsetAsync(ctx.d_flags + FLAG_COUNT - 1, 0, sizeof(int), st));
    AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
    k_edge_keys<<<grid, 256, 0, st>>>(di, m / 3, nv, ka.as<unsigned long long>(),
                                      va.as<int>(), ctx.d_flags);
    // radix passes over the bits that can be set: the low `bits` of each 32-bit half
    int bits = 1;
    while ((int64_t(1) << bits) < nv)
        ++bits;
    unsigned long long *kin = ka.as<unsigned long long>(), *kout = kb.as<unsigned long long>();
    int *vin = va.as<int>(), *vout = vb.as<int>();
    for (int half = 0; half < 2; ++half)
        for (int sh = 0; sh < bits; sh += 8)
        {
            int const shift = 32 * half + sh;
            k_rs_hist<unsigned long long><<<n_rs_blocks, kRsBlock, 0, st>>>(kin, m, shift, hist.as<unsigned>(),
                                                                            n_rs_blocks);
            scan_counters(st, hist.as<unsigned>(), int64_t(256) * n_rs_blocks, hsum.as<unsigned>());
            k_rs_scatter<unsigned long long, int><<<n_rs_blocks, kRsBlock, 0, st>>>(
                kin, vin, m, shift, hist.as<unsigned>(), n_rs_blocks, kout, vout);
            std::swap(kin, kout);
            std::swap(vin, vout);
        }
    k_edge_reduce<<<grid, 256, 0, st>>>(kin, vin, m, net.as<int>(), emit.as<unsigned>());
    k_scan_sums<<<int(n_sb), kScanBlock, 0, st>>>(emit.as<unsigned>(), m, sums.as<unsigned>());
    // the block sums become block offsets; keep the total in a copy of the last sum
    unsigned last_sum = 0, last_off = 0;
    AGWN_TRY_CUDA(cudaMemcpyAsync(&last_sum, sums.as<unsigned>() + n_sb - 1, sizeof(unsigned), cudaMemcpyDeviceToHost,
                                  st));
    k_rs_scan<<<1, 1024, 0, st>>>(sums.as<unsigned>(), n_sb);
    AGWN_TRY_CUDA(cudaMemcpyAsync(&last_off, sums.as<unsigned>() + n_sb - 1, sizeof(unsigned), cudaMemcpyDeviceToHost,
                                  st));
    k_scan_apply<<<int(n_sb), kScanBlock, 0, st>>>(emit.as<unsigned>(), m, sums.as<unsigned>(), pos.as<unsigned>());
    AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
    int bad = 0;
    AGWN_TRY_CUDA(cudaMemcpyAsync(&bad, ctx.d_flags + FLAG_COUNT - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    AGWN_TRY_CUDA(cudaStreamSynchronize(st));
    if (bad)
    {
        AGWN_TRY_CUDA(cudaMemsetAsync(ctx.d_flags + FLAG_COUNT - 1, 0, sizeof(int), st));
        return fail(AGWN_ERR_INVALID, "triangle index out of range [0, %lld)", (long long)nv);
    }
    int64_t const count = int64_t(last_off) + int64_t(last_sum);
    *n_segments = count;
    AGWN_TRY(o.prepare(ctx, out_for, count));
    if (o.rows == 0)
        return AGWN_OK;
    AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
    k_edge_emit<T><<<grid, 256, 0, st>>>(kin, net.as<int>(), emit.as<unsigned>(), pos.as<unsigned>(), m, o.rows, dv,
                                         o.dev);
    return ctx.launch_end(AGWN_K_OTHER);
}

// The extraction by bins, or *radix and nothing else where a bin is above kBinMax.  Its buffers are given back before the
// radix sort takes its own.
template <class T, class OutFor>
int boundary_bins(Context& ctx, const T* dv, int64_t nv, const int32_t* di, int64_t m, OutFor out_for, RowsOut<T>& o,
                  int64_t* n_segments, bool* radix)
{
    cudaStream_t const st = ctx.stream;
    ArenaScope scope(ctx);
    Tmp bins(ctx), sums(ctx), rank(ctx), lo(ctx), hi(ctx), net(ctx);
    // one counter per vertex and its end for the bins, the same for the emitted edges, and the state
    size_t const n_cnt = size_t(nv) + 1;
    AGWN_TRY(bins.alloc(sizeof(unsigned) * (2 * n_cnt + 2)));
    AGWN_TRY(sums.alloc(sizeof(unsigned) * size_t(scan_sums_count(int64_t(n_cnt)))));
    AGWN_TRY(rank.alloc(sizeof(unsigned) * m));
    AGWN_TRY(lo.alloc(sizeof(int) * m));
    AGWN_TRY(hi.alloc(sizeof(unsigned) * m));
    AGWN_TRY(net.alloc(sizeof(int) * m));
    unsigned* const bin = bins.as<unsigned>();
    unsigned* const emitted = bin + n_cnt;
    unsigned* const state = emitted + n_cnt;
    int const grid = int(std::min<int64_t>(div_up(m, 256), 8 * ctx.sm_count));
    AGWN_TRY_CUDA(cudaMemsetAsync(bin, 0, sizeof(unsigned) * (2 * n_cnt + 2), st));
    AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
    k_edge_count<<<grid, 256, 0, st>>>(di, m / 3, nv, bin, rank.as<unsigned>(), state);
    scan_counters(st, bin, int64_t(n_cnt), sums.as<unsigned>());
    k_edge_place<<<grid, 256, 0, st>>>(di, m / 3, bin, rank.as<unsigned>(), lo.as<int>(), hi.as<unsigned>());
    k_edge_net<<<grid, 256, 0, st>>>(lo.as<int>(), hi.as<unsigned>(), m, bin, state, net.as<int>(), emitted);
    scan_counters(st, emitted, int64_t(n_cnt), sums.as<unsigned>()); // its last counter: all emitted edges
    AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
    unsigned back[3] = {}; // the last counter and the state
    AGWN_TRY_CUDA(cudaMemcpyAsync(back, emitted + nv, sizeof(back), cudaMemcpyDeviceToHost, st));
    AGWN_TRY_CUDA(cudaStreamSynchronize(st));
    if (back[1])
        return fail(AGWN_ERR_INVALID, "triangle index out of range [0, %lld)", (long long)nv);
    *radix = back[2] != 0;
    if (*radix)
        return AGWN_OK;
    *n_segments = back[0];
    AGWN_TRY(o.prepare(ctx, out_for, int64_t(back[0])));
    if (o.rows == 0)
        return AGWN_OK;
    AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
    k_edge_rows<T><<<grid, 256, 0, st>>>(lo.as<int>(), hi.as<unsigned>(), m, bin, net.as<int>(), emitted, dv, o.rows,
                                         o.dev);
    return ctx.launch_end(AGWN_K_OTHER);
}

template <class T, class OutFor>
int boundary_build(agwn_context* ctx, const T* vertices, int64_t nv, const int32_t* indices, int64_t n_idx, OutFor out_for,
                   int64_t* n_segments)
{
    AGWN_CHECK_ARG(ctx && n_segments, "null context/count");
    AGWN_CHECK_ARG(nv >= 0 && n_idx >= 0 && n_idx % 3 == 0, "bad sizes");
    AGWN_CHECK_ARG(n_idx == 0 || (vertices && indices), "null geometry");
    AGWN_CHECK_ARG(nv <= (int64_t(1) << 31) && n_idx / 3 < (int64_t(1) << 31), "mesh too large");
    clear_message();
    AGWN_TRY_CUDA(cudaSetDevice(ctx->device));
    *n_segments = 0;
    int64_t const m = n_idx; // one entry per triangle edge
    RowsOut<T> o;
    if (m == 0)
        return o.prepare(*ctx, out_for, 0);
    const void *dv = nullptr, *di = nullptr;
    AGWN_TRY(stage_in(*ctx, vertices, sizeof(T) * 3 * nv, S_MISC0, &dv));
    AGWN_TRY(stage_in(*ctx, indices, sizeof(int32_t) * n_idx, S_MISC1, &di));
    const T* const verts = static_cast<const T*>(dv);
    const int32_t* const ip = static_cast<const int32_t*>(di);
    bool radix = nv > 16 * m + 65536;
    if (!radix)
        AGWN_TRY(boundary_bins<T>(*ctx, verts, nv, ip, m, out_for, o, n_segments, &radix));
    if (radix)
        AGWN_TRY(boundary_radix<T>(*ctx, verts, nv, ip, m, out_for, o, n_segments));
    return o.finish(*ctx);
}

// The rows into a given array, up to its capacity (out may be null: the count alone).
template <class T>
int boundary_into(agwn_context* ctx, const T* vertices, int64_t nv, const int32_t* indices, int64_t n_idx, T* out,
                  int64_t capacity, int64_t* n_segments)
{
    AGWN_CHECK_ARG(capacity >= 0, "bad sizes");
    return boundary_build<T>(ctx, vertices, nv, indices, n_idx,
                             [&](int64_t number, T** dst, int64_t* rows) -> int
                             {
                                 *dst = out;
                                 *rows = out ? std::min(capacity, number) : 0;
                                 return AGWN_OK;
                             },
                             n_segments);
}

// All rows into the array that alloc gives for their number.
template <class T>
int boundary_alloc(agwn_context* ctx, const T* vertices, int64_t nv, const int32_t* indices, int64_t n_idx,
                   agwn_alloc_rows alloc, void* user, int64_t* n_segments)
{
    AGWN_CHECK_ARG(alloc, "null alloc");
    return boundary_build<T>(ctx, vertices, nv, indices, n_idx,
                             [&](int64_t number, T** dst, int64_t* rows) -> int
                             {
                                 *dst = static_cast<T*>(alloc(user, number));
                                 *rows = number;
                                 return *dst || number == 0 ? int(AGWN_OK)
                                                            : fail(AGWN_ERR_NOMEM, "no array for %lld boundary rows",
                                                                   (long long)number);
                             },
                             n_segments);
}
} // namespace
} // namespace agwn

using namespace agwn;

extern "C" int agwn_build_boundary_segments_f64(agwn_context* ctx, const double* vertices, int64_t n_vertices,
                                                const int32_t* indices, int64_t n_indices, double* out,
                                                int64_t capacity, int64_t* n_segments)
{
    return boundary_into<double>(ctx, vertices, n_vertices, indices, n_indices, out, capacity, n_segments);
}
extern "C" int agwn_build_boundary_segments_f32(agwn_context* ctx, const float* vertices, int64_t n_vertices,
                                                const int32_t* indices, int64_t n_indices, float* out,
                                                int64_t capacity, int64_t* n_segments)
{
    return boundary_into<float>(ctx, vertices, n_vertices, indices, n_indices, out, capacity, n_segments);
}
extern "C" int agwn_build_boundary_segments_alloc_f64(agwn_context* ctx, const double* vertices, int64_t n_vertices,
                                                      const int32_t* indices, int64_t n_indices, agwn_alloc_rows alloc,
                                                      void* user, int64_t* n_segments)
{
    return boundary_alloc<double>(ctx, vertices, n_vertices, indices, n_indices, alloc, user, n_segments);
}
extern "C" int agwn_build_boundary_segments_alloc_f32(agwn_context* ctx, const float* vertices, int64_t n_vertices,
                                                      const int32_t* indices, int64_t n_indices, agwn_alloc_rows alloc,
                                                      void* user, int64_t* n_segments)
{
    return boundary_alloc<float>(ctx, vertices, n_vertices, indices, n_indices, alloc, user, n_segments);
}
