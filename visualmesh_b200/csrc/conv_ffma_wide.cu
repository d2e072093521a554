// CUDA-core graph-convolution layers with 32 channels in, and of widths without a kernel of their own (conv_ffma_launch.cuh).
#include "conv_ffma_launch.cuh"

namespace vm {

bool launch_conv_wide(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
#define VM_CONV(CI, CO, RR) if (launch_conv_shape<CI, CO, RR>(L, a, grid, max_rows, s)) return true;
    VM_CONV_SHAPES_WIDE(VM_CONV)
#undef VM_CONV
    return false;
}

// Few rows, any widths in multiples of 4 up to 32: OW outputs per thread and block.
template <int OW>
static bool launch_conv_few_t(const DenseLayer& L, const ConvArgs& a, dim3 grid_rows, int max_rows, cudaStream_t s) {
    constexpr int threads = 128;
    const size_t smem     = static_cast<size_t>(L.n_slots) * L.cin * OW * sizeof(float) + stage_bytes(a, L.cout, threads, 1);
    if (smem > 48 * 1024) return false;
    const dim3 grid((max_rows + threads - 1) / threads, grid_rows.y, (L.coutp + OW - 1) / OW);
    k_graph_conv_few<OW, threads><<<grid, threads, smem, s>>>(a, L.cin / 4, L.cout, L.coutp);
    return true;
}
bool launch_conv_few(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, int blocks_per_sm, cudaStream_t s) {
    if (L.cin % 4 != 0 || L.cin > 32 || L.coutp > 32 || a.out_split) return false;
    const int64_t blocks = static_cast<int64_t>((max_rows + 127) / 128) * grid.y * ((L.coutp + 7) / 8);
    if (blocks > static_cast<int64_t>(blocks_per_sm) * sm_count()) return false;
    // all outputs in a block where a row's outputs meet
    const int outputs = a.activation == VM_SOFTMAX || a.out_host != nullptr ? L.coutp : std::min(L.coutp, 8);
    if (outputs <= 4) return launch_conv_few_t<4>(L, a, grid, max_rows, s);
    if (outputs <= 8) return launch_conv_few_t<8>(L, a, grid, max_rows, s);
    if (outputs <= 16) return launch_conv_few_t<16>(L, a, grid, max_rows, s);
    return launch_conv_few_t<32>(L, a, grid, max_rows, s);
}

// Shapes without a kernel of their own, in multiples of 4 up to 32.
template <int COUTP, int WMAX>
static void launch_conv_any_t(const DenseLayer& L, const ConvArgs& a, dim3 grid_rows, int max_rows, cudaStream_t s) {
    ConvWeights<WMAX> wp;
    std::memcpy(wp.w, L.host_packed.data(), L.host_packed.size() * sizeof(float));
    constexpr int threads = 128;
    dim3 grid((max_rows + 2 * threads - 1) / (2 * threads), grid_rows.y);
    k_graph_conv_any<COUTP, 2, threads, WMAX><<<grid, threads, stage_bytes(a, L.cout, threads, 2), s>>>(a, L.cin / 4, L.cout, wp);
}
bool launch_conv_any(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
    if (few_rows(max_rows, grid.y) && launch_conv_few(L, a, grid, max_rows, FEW_BLOCKS, s)) return true;
    if (L.cin % 4 != 0 || L.coutp > 32 || L.host_packed.size() > static_cast<size_t>(CW_MOST) || a.out_split) return false;
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
