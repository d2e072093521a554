// Kernels of the Visual Mesh hot path for sm_100a.
//
// A chunk is a run of frames of one batch processed by one set of launches. Grids are two-dimensional:
// blockIdx.y is the frame within the chunk, blockIdx.x walks that frame's candidates (or rows). Blocks past the end of
// their frame exit at once, so no launch needs a count that only the device knows and the host never waits in the
// middle of a chunk. No kernel waits on another block: compaction is count -> scatter in two launches.
//
// Row spaces: points of frame f start at offsets[f] in the batch-wide result arrays; rows (points + one off-screen
// row per frame) start at offsets[f] + f. Feature buffers are chunk-local: rows start at
// offsets[f] - offsets[f0] + (f - f0) where f0 is the chunk's first frame.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "conv_args.hpp"
#include "device_math.cuh"
#include "tile_plan.cuh"

namespace vm {

constexpr int SELECT_THREADS = 256;
constexpr int ROW_THREADS    = 256;
constexpr int SCATTER_UNITS  = 4;    // runs of SELECT_THREADS candidates per block of k_scatter
constexpr int GROUP_BLOCKS   = 64;   // blocks of k_select whose counts are also summed as a group (a multiple of SCATTER_UNITS)
constexpr int EXPORT_THREADS = 512;
constexpr int FETCH_THREADS  = 256;

// Where a chunk's results go when they are wanted on the host: pinned memory that the device writes directly. It heads the
// chunk's staging block, so that a recorded graph of the chunk's kernels serves results buffers that change from call to call.
struct alignas(16) ChunkHeader {
    float2* px;
    int32_t* gi;
    int32_t* nb;
    float* cls;
    int32_t* offsets;  // every chunk: the batch's offsets array in pinned memory
};
constexpr int SAMPLE_ROWS    = 2;    // points per thread of k_sample

// ---- staging block of a chunk, read by the device --------------------------------------------------------------------
// For chunks whose images travel on the copy stream. A copy of these few kilobytes waits in the copy engine behind every image that is
// on its way, this chunk's and the next one's, and with it the projection and its results' way back: in a batch of chunks of four
// 5 MB frames the second projection ended 1.1 ms after the first. Read by a kernel instead (64 such frames, results on the host):
// one engine 7.46 -> 6.83 ms, two engines with half of them each 7.52 -> 6.78, where the bare copies take 6.67; 32 frames on one engine
// 3.90 -> 3.50. `n` pieces of 16 bytes, read past the L1 cache because the host rewrites them between launches.
__global__ void __launch_bounds__(FETCH_THREADS) k_fetch(const uint4* __restrict__ from, uint4* __restrict__ to, int32_t n) {
    for (int i = blockIdx.x * FETCH_THREADS + threadIdx.x; i < n; i += gridDim.x * FETCH_THREADS) to[i] = __ldcv(from + i);
}

enum : uint8_t { BSP_DESCEND = 0, BSP_INSIDE = 1, BSP_OUTSIDE = 2 };

// ---- device-side Mesh::lookup, part 1: classify every BSP element ----------------------------------------------
// cpp/visualmesh/mesh.hpp:521-539 (field-of-view cone test) and :362-406 (check_on_screen), evaluated for every
// element independently of its ancestors; the descent in k_select applies them top-down.
__global__ void __launch_bounds__(SELECT_THREADS) k_bsp_state(const FrameParams* __restrict__ frames, uint8_t* __restrict__ state) {
    const FrameParams& p = frames[blockIdx.y];
    const int e          = blockIdx.x * SELECT_THREADS + threadIdx.x;
    if (p.ranges != nullptr || e >= p.n_bsp) return;
    const float4 a  = __ldg(p.bsp_cones_a + e);
    const float sn  = __ldg(p.bsp_cones_s + e);
    const float cs  = a.w;
    const float delta = dot3(p.Rco[0], p.Rco[1], p.Rco[2], a.x, a.y, a.z);
    bool outside = delta < __fsub_rn(__fmul_rn(p.cos_fov, cs), __fmul_rn(p.sin_fov, sn));
    bool inside  = delta > __fadd_rn(__fmul_rn(p.cos_fov, cs), __fmul_rn(p.sin_fov, sn));
    if (!outside && inside) {
        float cx, cy, cz;
        rotate(p, a.x, a.y, a.z, cx, cy, cz);
        const bool axis_on_screen = on_screen_loose(project(cx, cy, cz, p), p);
        float angles[4];
        bool contains = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            angles[i] = dot3(a.x, a.y, a.z, p.edges[i][0], p.edges[i][1], p.edges[i][2]);
            contains |= angles[i] > __fadd_rn(__fmul_rn(p.edges[i][3], cs), __fmul_rn(p.edges[i][4], sn));
        }
        if (!axis_on_screen && contains) {
            inside  = false;
            outside = true;
        }
        else {
            bool intersects = true;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                intersects &= angles[i] < __fsub_rn(__fmul_rn(p.edges[i][3], cs), __fmul_rn(p.edges[i][4], sn));
            }
            inside  = axis_on_screen && intersects;
            outside = false;
        }
    }
    state[p.bsp_off + e] = inside ? BSP_INSIDE : (outside ? BSP_OUTSIDE : BSP_DESCEND);
}

// ---- select + project + count -----------------------------------------------------------------------------------
// One thread per candidate. With host ranges (cpp/visualmesh/engine/cpu/engine.hpp:110-122) a candidate is the c-th
// node of the concatenated ranges. With device lookup every node is a candidate and the thread first walks the BSP
// from the root: an INSIDE ancestor selects the node, an OUTSIDE one drops it, a leaf tests the node itself
// (cpp/visualmesh/mesh.hpp:559-583: inside the field of view and loosely on screen). Selected nodes then take the
// engine's strict on-screen test. Writes the pixel and node id (-1 = dropped) per candidate, the number kept per block and,
// added up in group_counts (which starts at zero), per group of GROUP_BLOCKS blocks.
__global__ void __launch_bounds__(SELECT_THREADS) k_select(const FrameParams* __restrict__ frames,
                                                           const uint8_t* __restrict__ state,
                                                           float2* __restrict__ cand_px,
                                                           int32_t* __restrict__ cand_node,
                                                           int32_t* __restrict__ block_counts,
                                                           int32_t* __restrict__ group_counts,
                                                           int32_t n_groups,
                                                           int32_t* __restrict__ abort_flags) {
    const FrameParams& p = frames[blockIdx.y];
    const int c          = blockIdx.x * SELECT_THREADS + threadIdx.x;
    bool keep            = false;
    if (c < p.n_candidates) {
        int g          = c;
        bool selected  = true;
        bool test_fov  = false;
        if (p.ranges != nullptr) {
            // binary search for the last range whose start is <= c
            int lo = 0, hi = p.n_ranges - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (__ldg(p.range_starts + mid) <= c) { lo = mid; }
                else {
                    hi = mid - 1;
                }
            }
            g = __ldg(p.ranges + lo).x + (c - __ldg(p.range_starts + lo));
        }
        else {
            int e = 0;
            int steps = 0;
            for (; steps < 128; ++steps) {
                // both loads of a step are issued together: the walk is a chain of dependent loads, and the element's
                // topology is in bounds whatever its state turns out to be
                const uint8_t s = state[p.bsp_off + e];
                const int4 t    = __ldg(p.bsp_topology + e);
                if (s == BSP_INSIDE) break;
                if (s == BSP_OUTSIDE) {
                    selected = false;
                    break;
                }
                if (t.x < 0) {
                    test_fov = true;
                    break;
                }
                e = (g < t.z) ? t.x : t.y;
            }
            if (steps == 128) {
                // a tree deeper than any the builder makes: give up on this node and report it
                raise_flag(abort_flags, ABORT_BSP_DEPTH);
                selected = false;
            }
        }
        float2 px = make_float2(0.0f, 0.0f);
        if (selected) {
            const float4 r = __ldg(p.rays + g);
            float cx, cy, cz;
            rotate(p, r.x, r.y, r.z, cx, cy, cz);
            px   = project(cx, cy, cz, p);
            keep = on_screen_strict(px, p) && (!test_fov || cx > p.cos_fov);
        }
        if (keep) cand_px[p.cand_off + c] = px;  // the scatter reads the pixels of kept candidates only
        cand_node[p.cand_off + c] = keep ? g : -1;
    }
    const int n = __syncthreads_count(keep);
    if (threadIdx.x == 0) {
        block_counts[blockIdx.y * gridDim.x + blockIdx.x] = n;
        if (n > 0) atomicAdd(group_counts + blockIdx.y * n_groups + blockIdx.x / GROUP_BLOCKS, n);
    }
}

// ---- scatter: stable compaction ----------------------------------------------------------------------------------
// Kept candidates, in candidate order, become the frame's points: global_indices ascending
// (cpp/visualmesh/engine/cpu/engine.hpp:110-120). Also fills the node -> local index table that k_remap reads in
// place of the reference's r_lookup (engine.hpp:128-131); with device lookup every entry is written, with host
// ranges only the candidates' (k_remap then checks what it reads).
// A block adds up what comes before it itself: the groups of the frames before, the groups of its own frame, the blocks
// of its own group. That is a few hundred counts that sit in L2 (64 frames x 8 groups for a mesh of 121 k nodes, 8 x 106
// for 1.7 M), read side by side, where a scan kernel of one block cost a launch and 6 to 9 us of every call.
// The batch-wide offsets array continues from offsets[f0], which the chunk before has written (0 for the first chunk).
template <int UNITS>
__global__ void __launch_bounds__(SELECT_THREADS) k_scatter(const FrameParams* __restrict__ frames,
                                                            const ChunkHeader* __restrict__ header,
                                                            const float2* __restrict__ cand_px,
                                                            const int32_t* __restrict__ cand_node,
                                                            const int32_t* __restrict__ block_counts,
                                                            const int32_t* __restrict__ group_counts,
                                                            int32_t blocks_per_frame,
                                                            int32_t n_groups,
                                                            int32_t* offsets,
                                                            int32_t f0,
                                                            float2* __restrict__ out_px,
                                                            int32_t* __restrict__ out_gi,
                                                            int32_t* __restrict__ node_rank) {
    static_assert(GROUP_BLOCKS % UNITS == 0, "a block's runs lie in one group");
    constexpr int WARPS = SELECT_THREADS / 32;
    // a block compacts UNITS runs of SELECT_THREADS candidates (the unit k_select counted); their loads are issued together
    __shared__ int32_t warp_counts[UNITS][WARPS];
    __shared__ int32_t sums[3][WARPS];
    const FrameParams& p = frames[blockIdx.y];
    const int lane       = threadIdx.x & 31;
    const int warp       = threadIdx.x >> 5;
    const int frame      = f0 + blockIdx.y;
    const int unit0      = blockIdx.x * UNITS;
    int c[UNITS], g[UNITS];
    unsigned mask[UNITS];
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        c[u] = (unit0 + u) * SELECT_THREADS + threadIdx.x;
        g[u] = (c[u] < p.n_candidates) ? cand_node[p.cand_off + c[u]] : -1;
    }
    // points of the frames before, points of this frame before this block, and (first block only) points of this frame
    int before_frame = 0, before_block = 0, of_frame = 0;
    const int own_first = blockIdx.y * n_groups;
    for (int i = threadIdx.x; i < own_first; i += SELECT_THREADS) before_frame += group_counts[i];
    const int group = unit0 / GROUP_BLOCKS;
    for (int i = threadIdx.x; i < group; i += SELECT_THREADS) before_block += group_counts[own_first + i];
    if (static_cast<int>(threadIdx.x) < unit0 - group * GROUP_BLOCKS) {
        before_block += block_counts[blockIdx.y * blocks_per_frame + group * GROUP_BLOCKS + threadIdx.x];
    }
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < n_groups; i += SELECT_THREADS) of_frame += group_counts[own_first + i];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        before_frame += __shfl_xor_sync(0xffffffffu, before_frame, d);
        before_block += __shfl_xor_sync(0xffffffffu, before_block, d);
        of_frame += __shfl_xor_sync(0xffffffffu, of_frame, d);
    }
    if (lane == 0) {
        sums[0][warp] = before_frame;
        sums[1][warp] = before_block;
        sums[2][warp] = of_frame;
    }
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        mask[u] = __ballot_sync(0xffffffffu, g[u] >= 0);
        if (lane == 0) warp_counts[u][warp] = __popc(mask[u]);
    }
    const int chunk_base = (f0 == 0) ? 0 : *static_cast<volatile int32_t*>(offsets + f0);
    __syncthreads();
    int frame_base = chunk_base, in_frame = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
        frame_base += sums[0][w];
        in_frame += sums[1][w];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int total = frame_base;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) total += sums[2][w];
        offsets[frame + 1]         = total;
        header->offsets[frame + 1] = total;
        if (frame == 0) {
            offsets[0]         = 0;
            header->offsets[0] = 0;
        }
    }
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        if (unit0 + u >= blocks_per_frame) break;
        int before = in_frame, of_unit = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            if (w < warp) before += warp_counts[u][w];
            of_unit += warp_counts[u][w];
        }
        if (g[u] >= 0) {
            const int k  = before + __popc(mask[u] & ((1u << lane) - 1u));
            const int o  = frame_base + k;
            out_px[o]    = cand_px[p.cand_off + c[u]];
            out_gi[o]    = g[u];
            node_rank[p.node_off + g[u]] = k;
        }
        else if (c[u] < p.n_candidates && p.ranges == nullptr) {
            node_rank[p.node_off + c[u]] = -1;
        }
        in_frame += of_unit;
    }
}

// ---- neighbour remap ---------------------------------------------------------------------------------------------
// cpp/visualmesh/engine/cpu/engine.hpp:134-143: neighbours into the frame's compact index space; a neighbour that is
// off the mesh or not on screen becomes n (the off-screen row); row n is all n.
// With PLAN the block - which owns 256 consecutive rows, exactly one super-tile of the staged layer kernels - also makes
// that super-tile's part of the tile plan (tile_plan.cuh) from the indices it has just computed.
// Rows of neighbour indices are read and written in pieces of 16 bytes (six neighbours: 8), because rows lie one after another: index by
// index a warp touched all of their lines N times, and the load/store path was what bound the kernel. 7.4 M rows of eight neighbours, plan
// included, 330 -> 275 us; 4.5 M of six 113 -> 109; 571 k of eight 35 -> 27. (The layers' own reads of a row, one index per slot, gained
// nothing from it: 8 -> 8 105 us either way.)
template <int N>
__device__ __forceinline__ void load_neighbours(const int32_t* __restrict__ row, int (&v)[N]) {
    static_assert(N % 2 == 0, "whole pieces");
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N / 4; ++k) {
            const int4 p = __ldg(reinterpret_cast<const int4*>(row) + k);
            v[4 * k]     = p.x;
            v[4 * k + 1] = p.y;
            v[4 * k + 2] = p.z;
            v[4 * k + 3] = p.w;
        }
    }
    else {
#pragma unroll
        for (int k = 0; k < N / 2; ++k) {
            const int2 p = __ldg(reinterpret_cast<const int2*>(row) + k);
            v[2 * k]     = p.x;
            v[2 * k + 1] = p.y;
        }
    }
}
// whole: the array begins on a 16-byte boundary
template <int N>
__device__ __forceinline__ void store_neighbours(int32_t* row, const int (&v)[N], bool whole) {
    if (!whole) {
#pragma unroll
        for (int j = 0; j < N; ++j) row[j] = v[j];
    }
    else if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N / 4; ++k) reinterpret_cast<int4*>(row)[k] = make_int4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
    else {
#pragma unroll
        for (int k = 0; k < N / 2; ++k) reinterpret_cast<int2*>(row)[k] = make_int2(v[2 * k], v[2 * k + 1]);
    }
}
template <int N, bool PLAN>
__global__ void __launch_bounds__(ROW_THREADS) k_remap(const FrameParams* __restrict__ frames,
                                                       const int32_t* __restrict__ offsets,
                                                       int32_t f0,
                                                       const int32_t* __restrict__ out_gi,
                                                       const int32_t* __restrict__ node_rank,
                                                       int32_t* __restrict__ out_nb,
                                                       const st::PlanOut plan) {
    static_assert(!PLAN || ROW_THREADS == st::ST, "a block of the remap is a super-tile of the plan");
    const FrameParams& p = frames[blockIdx.y];
    const int frame      = f0 + blockIdx.y;
    const int start      = offsets[frame];
    const int n          = offsets[frame + 1] - start;
    const int t0         = blockIdx.x * ROW_THREADS;
    if (t0 > n) return;  // the whole block is past the frame's n + 1 rows
    const int i      = t0 + threadIdx.x;
    const bool valid = i <= n;
    int v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = n;
    if (valid) {
        int32_t* row = out_nb + static_cast<size_t>(start + frame + i) * N;
        if (i < n) {
            const int g         = out_gi[start + i];
            int nbrs[N];
            load_neighbours<N>(p.neighbours + static_cast<size_t>(g) * N, nbrs);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int t = nbrs[j];
                if (t >= 0 && t < p.n_nodes) {
                    const int k = node_rank[p.node_off + t];
                    bool known  = k >= 0;
                    // with host ranges the table holds what earlier frames left for the nodes that were no candidates now: an
                    // entry counts only if its point is this node
                    if (p.ranges != nullptr) known = known && k < n && out_gi[start + k] == t;
                    v[j] = known ? k : n;
                }
            }
        }
        // the engine's own array does, a caller's (vm_project_static) may begin anywhere
        store_neighbours<N>(row, v, (reinterpret_cast<uintptr_t>(out_nb) & 15) == 0);
    }
    if (PLAN) st::plan_super_tile<N>(v, valid, t0, static_cast<int>(blockIdx.y), offsets, f0, plan);
}

// ---- image sampling ----------------------------------------------------------------------------------------------
// cpp/visualmesh/engine/cpu/engine.hpp:198-206: bilinear sample at every point, four -1 for the off-screen row.
// PACKED4: every frame of the launch is RGBA or BGRA. The general sampler carries the 5x5 Bayer patch in its register
// count (66), which holds it to three blocks per SM although it waits on memory; the packed one fills the SM.
template <bool PACKED4>
__global__ void __launch_bounds__(ROW_THREADS) k_sample(const FrameParams* __restrict__ frames,
                                                        const int32_t* __restrict__ offsets,
                                                        int32_t f0,
                                                        const float2* __restrict__ out_px,
                                                        float4* __restrict__ features) {
    // a thread samples SAMPLE_ROWS points, ROW_THREADS apart: the pixel coordinates of all of them are loaded before
    // the first texel, so that many independent chains of two dependent loads are in flight per thread
    const FrameParams& p = frames[blockIdx.y];
    const int frame      = f0 + blockIdx.y;
    const int start      = offsets[frame];
    const int n          = offsets[frame + 1] - start;
    const int first      = blockIdx.x * (ROW_THREADS * SAMPLE_ROWS) + threadIdx.x;
    if (first > n) return;
    const int row0 = start - offsets[f0] + blockIdx.y;
    float2 px[SAMPLE_ROWS];
#pragma unroll
    for (int q = 0; q < SAMPLE_ROWS; ++q) {
        const int i = first + q * ROW_THREADS;
        px[q]       = (i < n) ? out_px[start + i] : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int q = 0; q < SAMPLE_ROWS; ++q) {
        const int i = first + q * ROW_THREADS;
        if (i > n) break;
        float4 v = make_float4(-1.0f, -1.0f, -1.0f, -1.0f);
        if (i < n) {
            if (PACKED4) { v = interpolate_packed4(px[q], p.image, p.dims[0], p.dims[1], p.format == fcc('B', 'G', 'R', 'A')); }
            else {
                v = interpolate(px[q], p.image, p.dims[0], p.dims[1], format_class(p.format));
            }
        }
        features[row0 + i] = v;
    }
}

// ---- results to the host -----------------------------------------------------------------------------------------
// Writes a chunk's results into pinned host memory. The device knows how many there are, so the copy needs no count on the host
// and no wait for one in the middle of a call; the bus takes 64 KB in 3 us more than a copy engine would and 5 MB in 10 us more
// (112 us against 102). WHICH: 0 = pixel coordinates, node indices and (rows given) neighbourhood, 1 = classifications, 2 = neighbourhood.
__device__ __forceinline__ void export_words(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, size_t begin, size_t end) {
    // 16-byte pieces between the first and the last whole one (both arrays start on 256-byte boundaries), words at the ends
    const size_t first = (begin + 3) / 4, last = end / 4;
    const size_t t = static_cast<size_t>(blockIdx.x) * EXPORT_THREADS + threadIdx.x, step = static_cast<size_t>(gridDim.x) * EXPORT_THREADS;
    if (first >= last) {
        if (t < end - begin) dst[begin + t] = src[begin + t];
        return;
    }
    if (t < first * 4 - begin) dst[begin + t] = src[begin + t];
    if (t < end - last * 4) dst[last * 4 + t] = src[last * 4 + t];
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4       = reinterpret_cast<uint4*>(dst);
    size_t i        = first + t;
    for (; i + 3 * step < last; i += 4 * step) {
        const uint4 a = s4[i], b = s4[i + step], c = s4[i + 2 * step], d = s4[i + 3 * step];
        d4[i]            = a;
        d4[i + step]     = b;
        d4[i + 2 * step] = c;
        d4[i + 3 * step] = d;
    }
    for (; i < last; i += step) d4[i] = s4[i];
}
template <int WHICH>
__global__ void __launch_bounds__(EXPORT_THREADS) k_export(const ChunkHeader* __restrict__ header,
                                                           const int32_t* __restrict__ offsets,
                                                           int32_t f0,
                                                           int32_t f1,
                                                           int32_t width,  // neighbours or classes
                                                           const float2* __restrict__ px,
                                                           const int32_t* __restrict__ gi,
                                                           const void* __restrict__ rows) {
    const size_t p0 = offsets[f0], p1 = offsets[f1];
    if (WHICH == 0) {
        export_words(reinterpret_cast<uint32_t*>(header->px), reinterpret_cast<const uint32_t*>(px), 2 * p0, 2 * p1);
        export_words(reinterpret_cast<uint32_t*>(header->gi), reinterpret_cast<const uint32_t*>(gi), p0, p1);
        if (rows == nullptr) return;
    }
    uint32_t* dst = WHICH == 1 ? reinterpret_cast<uint32_t*>(header->cls) : reinterpret_cast<uint32_t*>(header->nb);
    export_words(dst, static_cast<const uint32_t*>(rows), (p0 + f0) * width, (p1 + f1) * width);
}

// The same sampler on a flat list of pixel coordinates (stand-alone stage for unit parity tests).
__global__ void __launch_bounds__(ROW_THREADS) k_sample_flat(const float2* __restrict__ px,
                                                             int32_t n,
                                                             const uint8_t* __restrict__ image,
                                                             int32_t W,
                                                             int32_t H,
                                                             int32_t cls,
                                                             float4* __restrict__ out) {
    const int i = blockIdx.x * ROW_THREADS + threadIdx.x;
    if (i < n) out[i] = interpolate(px[i], image, W, H, cls);
}

}  // namespace vm
