// CUDA-core graph-convolution layers: which kernel runs a layer, and those with 4 and 8 channels in (conv_ffma_launch.cuh).
#include "conv_ffma_launch.cuh"

namespace vm {

bool has_fast_ffma_kernel(int cin, int cout) {
#define VM_IS(CI, CO, RR) if (cin == CI && cout == CO) return true;
    VM_CONV_SHAPES_NARROW(VM_IS) VM_CONV_SHAPES_MID(VM_IS) VM_CONV_SHAPES_WIDE(VM_IS)
#undef VM_IS
    return false;
}

bool ffma_stores_to_host(const DenseLayer& L) {
    if (L.cout > 16 || L.cin % 4 != 0 || !const_weights()) return false;
    return L.host_packed.size() <= static_cast<size_t>(has_fast_ffma_kernel(L.cin, L.cout) ? CW_MAX : CW_MOST);
}

bool launch_conv_narrow(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
#define VM_CONV(CI, CO, RR) if (launch_conv_shape<CI, CO, RR>(L, a, grid, max_rows, s)) return true;
    VM_CONV_SHAPES_NARROW(VM_CONV)
#undef VM_CONV
    return false;
}

// Shapes with a specialised kernel; then the widths that are multiples of 4; anything else takes the generic kernel.
void launch_conv_ffma(const DenseLayer& L, const ConvArgs& a, int n_frames, int max_rows, cudaStream_t s) {
    const dim3 grid(1, n_frames);
    if ((static_cast<size_t>(L.n_slots) * L.cin * L.coutp + L.coutp) * sizeof(float) <= 96 * 1024) {
        if (launch_conv_narrow(L, a, grid, max_rows, s) || launch_conv_mid(L, a, grid, max_rows, s) || launch_conv_wide(L, a, grid, max_rows, s)) return;
    }
    if (launch_conv_any(L, a, grid, max_rows, s)) return;
    const dim3 g((max_rows + CONV_THREADS - 1) / CONV_THREADS, n_frames);
    k_graph_conv_generic<<<g, CONV_THREADS, 0, s>>>(a, L.cin, L.cout, L.coutp);
}

}  // namespace vm
