// CUDA-core graph-convolution layers with 32 channels in, and of widths without a kernel of their own (conv_ffma_launch.cuh).
#include "conv_ffma_launch.cuh"

namespace vm {

bool launch_conv_wide(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
#define VM_CONV(CI, CO, RR) if (launch_conv_shape<CI, CO, RR>(L, a, grid, max_rows, s)) return true;
    VM_CONV_SHAPES_WIDE(VM_CONV)
#undef VM_CONV
    return false;
}

// Shapes without a kernel of their own, in multiples of 4 up to 32. One row per thread and small blocks until two rows per thread
// still give every SM a block (few_rows).
template <int COUTP, int WMAX>
static void launch_conv_any_t(const DenseLayer& L, const ConvArgs& a, dim3 grid_rows, int max_rows, cudaStream_t s) {
    ConvWeights<WMAX> wp;
    std::memcpy(wp.w, L.host_packed.data(), L.host_packed.size() * sizeof(float));
    constexpr int threads = 128;
    if (few_rows(max_rows, grid_rows.y)) {
        dim3 grid((max_rows + threads - 1) / threads, grid_rows.y);
        const size_t smem = std::max(L.host_packed.size() * sizeof(float), stage_bytes(a, L.cout, threads, 1));
        k_graph_conv_any<COUTP, 1, threads, WMAX><<<grid, threads, smem, s>>>(a, L.cin / 4, L.cout, wp);
    }
    else {
        dim3 grid((max_rows + 2 * threads - 1) / (2 * threads), grid_rows.y);
        k_graph_conv_any<COUTP, 2, threads, WMAX><<<grid, threads, stage_bytes(a, L.cout, threads, 2), s>>>(a, L.cin / 4, L.cout, wp);
    }
}
bool launch_conv_any(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
    if (L.cin % 4 != 0 || L.host_packed.size() > static_cast<size_t>(CW_MOST) || a.out_split) return false;
    const bool small = L.host_packed.size() <= static_cast<size_t>(CW_MAX);
#define VM_ANY(CP)                                                             \
    if (L.coutp == CP) {                                                       \
        if (small) launch_conv_any_t<CP, CW_MAX>(L, a, grid, max_rows, s);     \
        else launch_conv_any_t<CP, CW_MOST>(L, a, grid, max_rows, s);          \
        return true;                                                           \
    }
    VM_ANY(4) VM_ANY(8) VM_ANY(12) VM_ANY(16) VM_ANY(20) VM_ANY(24) VM_ANY(28) VM_ANY(32)
#undef VM_ANY
    return false;
}

}  // namespace vm
