// Host-side interface between the engine (engine.cu) and the translation units that hold the graph-convolution layer
// kernels with their launchers (conv_ffma.cu, conv_tc.cu, conv_staged.cu). Splitting them keeps every kernel family in
// a translation unit of its own, compiled in parallel.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "conv_args.hpp"

namespace vm {

struct CudaFailure {
    cudaError_t code;
    const char* what;
};
#define VM_CUDA(expr)                                        \
    do {                                                     \
        cudaError_t vm_e_ = (expr);                          \
        if (vm_e_ != cudaSuccess) throw CudaFailure{vm_e_, #expr}; \
    } while (0)

struct DenseLayer {
    float* d_weights = nullptr;  // [n_slots * cin][coutp] then [coutp] biases
    int cin = 0, cout = 0, coutp = 0, n_slots = 1, activation = 0;
    std::string stage;  // name under which this layer's kernel is timed, e.g. "graph_conv_16x16"
    std::vector<float> host_packed;  // [K][coutp] weights then biases, as on the device (for parameter-space kernels)
    // tensor-core path (conv_tc.cuh): weights split into TF32 hi/lo parts in the UMMA K-major layout, padded bias
    void* d_tc_cat   = nullptr;  // [K / KCH chunks][2 * NP rows][16 B]: hi rows then lo rows
    void* d_tc_win   = nullptr;  // conv_window.cuh: columns and channels permuted (32-channel inputs)
    float* d_tc_bias = nullptr;
    int tc_np        = 0;      // padded output width of the tensor-core tile, 0 = no tensor-core path for this shape
    bool tc_half     = false;  // fp16 hi/lo split (16- and 32-channel inputs) or TF32 split (8-channel inputs)
};

// What a launcher works out once per kernel instantiation and device: function attributes are per device, and engine
// instances of several host threads may reach a launcher at the same time.
struct LaunchPlan {
    int ctas_per_sm = 0;
    int n_sms       = 0;
};
constexpr int MAX_DEVICES = 64;
struct LaunchPlans {
    LaunchPlan plan[MAX_DEVICES];
    std::once_flag once[MAX_DEVICES];
    template <typename Init>
    const LaunchPlan& get(Init init) {
        int dev = 0;
        VM_CUDA(cudaGetDevice(&dev));
        dev = std::min(std::max(dev, 0), MAX_DEVICES - 1);
        std::call_once(once[dev], [&] { plan[dev] = init(dev); });
        return plan[dev];
    }
};

// Whether a layer's launch starts early: while its blocks (as many as there may be rows for) are few. The lines were found by trial on three
// networks; they do not follow from what a kernel's blocks take of an SM (a window layer's CTA takes all of it, and three or two of the
// staged ones: those of the next layer then start as the ones in front end). A pass with the layers started early, us, one frame of 2.7 | 11 | 25 |
// 57 | 121 | 242 k nodes: thirteen layers of 16 and 8 channels 86.9 | 90.3 | 92.8 | 101 | 128 | 154 -> 76.0 | 80.6 | 82.9 | 93.6 | 118 | 169; four layers
// 50.5 | 51.5 | 53.2 | 54.4 | 64.0 | 76.6 -> 45.7 | 48.5 | 48.4 | 53.2 | 63.6 | 85.9; ten of 32 channels 105 | 107 | 112 | 126 | 157 | 239 -> 84.7 | 85.9 | 104 |
// 134 | 193 | 255. So two blocks (of a window layer, two halves of a super-tile: 37.9 k rows) per SM, and four super-tiles of the staged layers
// (151.6 k rows): what measured slower lies beyond. Layers that few rows send to the kernel with part of the outputs per block lose (50
// -> 57 us at 11 k nodes, five times the blocks) and start the ordinary way, and so do the kernels of the projection (no gain),
// and a last layer that writes to the host (a call of two layers 36.9 -> 37.7 us).
inline bool starts_early(int64_t blocks, int blocks_per_sm, int n_sms) {
    return blocks <= static_cast<int64_t>(blocks_per_sm) * n_sms;
}
// A launch; early: it may start while the kernel in front of it in the stream finishes, and waits for that one's results itself
// (after_previous), with its own preparations - barriers, weights into shared memory - behind it.
template <typename... Params, typename... Args>
void launch_kernel(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t s, bool early, const Args&... args) {
    cudaLaunchAttribute attribute{};
    attribute.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim          = grid;
    config.blockDim         = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream           = s;
    config.attrs            = &attribute;
    config.numAttrs         = early ? 1 : 0;
    VM_CUDA(cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...));
}

// ---- conv_ffma.cu: layers on the CUDA cores ----------------------------------------------------------------------
// a specialised kernel exists for this shape (anything else runs the generic kernel, which ignores ConvArgs::out_split)
bool has_fast_ffma_kernel(int cin, int cout);
bool ffma_stores_to_host(const DenseLayer& L);  // the layer's kernel honours ConvArgs::out_host
void launch_conv_ffma(const DenseLayer& L, const ConvArgs& a, int n_frames, int max_rows, cudaStream_t s);

// ---- conv_tc.cu: layers on the tensor cores, gather by global loads ----------------------------------------------
constexpr int TC_MAX_FRAMES    = 256;  // frames per launch of a tensor-core layer (shared table of tile counts)
constexpr uint32_t TC_DEFAULT_WAIT_LIMIT = 4000000;
bool has_tc_gather_kernel(const DenseLayer& L);  // gathers fp32 rows and splits them itself
bool has_tc_split_kernel(const DenseLayer& L);   // fed from the split feature layout
bool launch_conv_tc_gather(const DenseLayer& L, const ConvArgs& a, int n_frames, int max_rows, int32_t* abort_flags, uint32_t wait_limit, cudaStream_t s);
bool launch_conv_tc_split(const DenseLayer& L, const ConvArgs& a, int n_frames, int max_rows, int32_t* abort_flags, uint32_t wait_limit, cudaStream_t s);

// ---- conv_staged.cu: layers on the tensor cores, gather from shared-memory windows --------------------------------
// What the tile plan of a chunk holds (device pointers), see conv_staged.cuh.
struct StagedPlan {
    const uint16_t* nbl;
    const int32_t* halo_rows;
    const int32_t* halo_count;
};
constexpr int STAGED_NBL_STRIDE = 8;    // 16-bit neighbour positions per row
constexpr int STAGED_ST         = 256;  // rows of a super-tile
constexpr int STAGED_HALO       = 384;  // halo slots of a super-tile
bool has_staged_kernel(const DenseLayer& L);
bool launch_conv_staged(const DenseLayer& L, const ConvArgs& a, const StagedPlan& plan, int n_frames, int max_rows, int32_t* abort_flags,
                        uint32_t wait_limit, cudaStream_t s);
// ---- conv_window.cu: 32-channel layers on the tensor cores (tcgen05), gather from shared-memory windows ------------
bool has_window_kernel(const DenseLayer& L);
// the layer's weights as the kernel wants them in shared memory; weights is [n_slots * 32][cout]
std::vector<unsigned char> pack_window_weights(const float* weights, int n_slots, int cout);
bool launch_conv_window(const DenseLayer& L, const ConvArgs& a, const StagedPlan& plan, int n_frames, int max_rows, int32_t* abort_flags,
                        uint32_t wait_limit, cudaStream_t s);
// the plan for a neighbourhood that is already in memory (the hot path makes it inside the neighbour-remap kernel)
void launch_tile_plan_kernel(int n_neighbours, const int32_t* offsets, const int32_t* nb, uint16_t* nbl, int32_t* halo_rows, int32_t* halo_count,
                             int f0, int n_frames, int max_rows, cudaStream_t s);

}  // namespace vm
