// CUDA-core graph-convolution layers with 12 and 16 channels in (conv_ffma_launch.cuh).
#include "conv_ffma_launch.cuh"

namespace vm {

bool launch_conv_mid(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
#define VM_CONV(CI, CO, RR) if (launch_conv_shape<CI, CO, RR>(L, a, grid, max_rows, s)) return true;
    VM_CONV_SHAPES_MID(VM_CONV)
#undef VM_CONV
    return false;
}

}  // namespace vm
