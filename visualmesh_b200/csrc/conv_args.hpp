// Arguments of one graph-convolution layer launch, shared by every layer kernel and by the host code that fills them.
#pragma once

#include <cstdint>

namespace vm {

// ---- fused graph convolution layer -------------------------------------------------------------------------------
// gather (cpp/visualmesh/engine/cpu/engine.hpp:216-235) + dense with the accumulator started at the bias and k
// ascending (engine.hpp:250-256) + activation (engine.hpp:259), one launch per dense layer, nothing materialised.
// Feature layout between layers. A width that is a multiple of 4 is stored "chunk-planar": float4 chunk c of row r at
// float4 index c * stride + r, so that the 32 threads of a warp, which own 32 consecutive rows, read and write
// consecutive 16-byte pieces (one 512-byte request per instruction instead of 32 pieces scattered over 16 cache
// lines). Other widths, and the final classifications, are row-major [row][width].
struct ConvArgs {
    const float* in;        // chunk-local features (planar when CIN % 4 == 0, else row-major)
    float* out;             // chunk-local features, or the batch-wide row-major classifications when out_global
    const int32_t* nb;      // batch-wide neighbourhood rows (frame-local indices)
    const int32_t* offsets; // batch-wide point offsets
    const float* weights;   // [n_slots * CIN][COUTP] row-major, COUTP = COUT rounded up to 4, zero padded
    const float* biases;    // [COUTP]
    int32_t n_slots;        // N + 1 for the first layer of a group, 1 for the layers that follow it
    int32_t n_neighbours;   // N
    int32_t activation;
    int32_t f0;
    int32_t out_global;
    int32_t in_stride;      // rows per planar chunk of `in`
    int32_t out_stride;     // rows per planar chunk of `out`
    int32_t out_planar;     // write `out` chunk-planar (needs COUT % 4 == 0 and !out_global)
    int32_t out_split;      // write `out` as fp16 hi/lo parts for a tensor-core consumer: SPLIT_PLANES (COUT % 8 == 0), SPLIT_ROWS or SPLIT_QUADS
    float* const* out_host; // where the batch-wide classifications go instead of `out`: the device address of a pointer to pinned memory
    int32_t* range_flag;    // the engine's abort flags: ABORT_RANGE is raised when a value is too large for the fp16 split
    int32_t early;          // for the launch: may start while the layer before finishes (launch_kernel)
};

// ConvArgs::out_split. Planes of 16-byte chunks; whole rows for the window kernel (its 32 input channels: COUT == 32), pieces of
// two hi, two lo, two hi and two lo parts, odd rows with their second half first; whole rows for the staged kernel (its 16 input channels: COUT == 16), pieces of four hi and four lo parts.
enum SplitLayout { SPLIT_NONE = 0, SPLIT_PLANES = 1, SPLIT_ROWS = 2, SPLIT_QUADS = 3 };

constexpr int CONV_THREADS = 128;

// Why a call had to be given up: one flag per reason, in pinned host memory. A kernel raises one with a plain store, so a healthy
// call neither clears nor copies anything.
enum AbortReason { ABORT_BSP_DEPTH = 1, ABORT_TC_TIMEOUT = 2, ABORT_TC_RANGE = 3, ABORT_FLAGS = 4 };
#ifdef __CUDACC__
// A layer that launch_kernel starts early begins before the one in front of it has ended. Before it reads what that one writes, or
// writes what that one reads, it waits for it here: everything of the layer in front is then done and visible. The pointer goes through
// the wait, so that no load from it is scheduled in front of it. Launched the ordinary way a kernel passes at once. All warps make this
// wait, also those that only read what others of their block bring: their bounded waits (vm_set_wait_limit) then count polls of this
// layer's work alone, and the issue slots stay with the layer in front. Features are never read by way of the read-only path (__ldg,
// ld.global.nc): that is for what nobody writes while the kernel runs, and the layer in front still writes them when this one starts.
// Ordinary loads may keep them in the L1 cache, __ldcg measured 3 % slower where most halos are too large for their window.
template <typename T>
__device__ __forceinline__ T* wait_previous(T* p) {
    asm volatile("griddepcontrol.wait;" : "+l"(p)::"memory");
    return p;
}
// The same, and the next layer may start in turn. Not sooner: a layer must not run beside the one two in front of it, which reads the
// buffer that the layer between them writes and could leave its old lines in an L1 cache that was cleaned when the layer behind started.
// At least one block of every launch must call; blocks without work may leave before.
template <typename T>
__device__ __forceinline__ T* after_previous(T* p) {
    p = wait_previous(p);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return p;
}
__device__ __forceinline__ void raise_flag(int32_t* flags, int reason) {
    *static_cast<volatile int32_t*>(flags + reason) = 1;
}
#endif

}  // namespace vm
