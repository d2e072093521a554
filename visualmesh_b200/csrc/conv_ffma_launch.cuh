// Launchers of the CUDA-core graph-convolution layer kernels (conv_ffma.cuh). The shapes are spread over three translation units,
// which compile side by side: conv_ffma.cu (4 and 8 channels in, and the choice between them), conv_ffma_mid.cu (12 and 16) and
// conv_ffma_wide.cu (32, and the widths without a kernel of their own).
#pragma once

#include <cstdlib>
#include <cstring>

#include "conv_dispatch.hpp"
#include "conv_ffma.cuh"

namespace vm {

// layer shapes (C_in, C_out, rows per thread) with a specialised FFMA kernel
#define VM_CONV_SHAPES_NARROW(X)                                                                            \
    X(4, 2, 4) X(4, 3, 4) X(4, 4, 4) X(4, 8, 4) X(4, 12, 4) X(4, 16, 4) X(4, 32, 2)                         \
    X(8, 2, 4) X(8, 3, 4) X(8, 4, 4) X(8, 5, 4) X(8, 8, 4) X(8, 12, 4) X(8, 16, 4)
#define VM_CONV_SHAPES_MID(X)                                                                               \
    X(12, 2, 4) X(12, 3, 4) X(12, 4, 4) X(12, 8, 4) X(12, 12, 4) X(12, 16, 4)                               \
    X(16, 2, 4) X(16, 3, 4) X(16, 4, 4) X(16, 5, 4) X(16, 8, 4) X(16, 12, 4) X(16, 16, 4) X(16, 32, 2)
#define VM_CONV_SHAPES_WIDE(X) X(32, 2, 4) X(32, 3, 4) X(32, 4, 4) X(32, 8, 4) X(32, 16, 4) X(32, 32, 2)

bool launch_conv_narrow(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s);
bool launch_conv_mid(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s);
bool launch_conv_wide(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s);
bool launch_conv_any(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s);
bool launch_conv_few(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, int blocks_per_sm, cudaStream_t s);

constexpr int CW_MAX  = 2320;  // floats: a 16 -> 16 layer with 8 neighbours and its biases
constexpr int CW_MOST = 8120;  // what the parameter space holds beside the other arguments: 28 -> 32 with 8 neighbours

inline int sm_count() {
    static LaunchPlans plans;
    return plans.get([](int device) {
        LaunchPlan p;
        VM_CUDA(cudaDeviceGetAttribute(&p.n_sms, cudaDevAttrMultiProcessorCount, device));
        return p;
    }).n_sms;
}
// Two rows per thread and 256 threads per block would leave SMs without a block: such launches run one row per thread in blocks of 128
// threads.
inline bool few_rows(int max_rows, int n_frames) {
    return static_cast<int64_t>((max_rows + 511) / 512) * n_frames < sm_count();
}
// The kernel with part of the outputs per block (launch_conv_few) pays while those blocks are few. A specialised layer with its weights
// in the parameter space, one frame, us of that layer less with it: 16 -> 16 with six neighbours 3.5 at 0.9 blocks per SM, 2.0 at 2.2,
// nothing from 2.8 on, 2.2 more at 7.2; 16 -> 8 1 to 2 up to 1.1, nothing at 2.5. Against the kernels of the other widths, and of the
// layers too large for the parameter space, it pays further (24,20,12,5, six neighbours, us a call: 4.0 blocks per SM 67.9 -> 64.3, 4.6
// 70.9 -> 65.8, 6.9 76.6 -> 76.2, 8.0 75.5 -> 79.3; 32 -> 16 13 at 0.5, 10 at 5.0, 5 at 7.2).
// Twelve outputs leave half of their second part empty: 16 -> 12 gains 0.5 to 2.7 us up to one block per SM, 12 -> 12 and 8 -> 12 nothing,
// and from there on all three lose, 2 to 3 us at 3.7.
constexpr int FEW_BLOCKS_SPECIALISED = 3;
constexpr int FEW_BLOCKS_TWELVE      = 1;
constexpr int FEW_BLOCKS             = 7;
// ... and while there are weights to share: below this many floats the parameter space is faster even for few blocks (8 -> 8, 328 to 584
// floats: 1.1 to 1.5 us a layer; from 648 on, 16 -> 8 and 8 -> 16 with four neighbours, it is 1 to 2 us slower).
constexpr size_t FEW_WEIGHTS = 640;
// weights small enough for the kernel parameter space are read through the constant cache (measured 15-40 %
// faster than the shared-memory copy: the weight reads leave the L1/shared data path to the gather)
inline bool const_weights() {
    static const bool on = [] {
        const char* v = std::getenv("VMCUDA_CONST_WEIGHTS");
        return v == nullptr || v[0] != '0';
    }();
    return on;
}

// shared memory in which the warps of a block arrange split rows, or the block its results for the host, before they store them
inline size_t stage_bytes(const ConvArgs& a, int cout, int threads, int rows_per_thread) {
    if (a.out_host != nullptr) return static_cast<size_t>(threads) * rows_per_thread * cout * sizeof(float);
    const int warp = a.out_split == SPLIT_ROWS ? SPLIT_ROW_STAGE : a.out_split == SPLIT_QUADS ? SPLIT_QUAD_STAGE : 0;
    return static_cast<size_t>(threads / 32) * warp;
}

template <int CIN, int COUT, int R, int T = CONV_THREADS, int MINB = 1>
static void launch_conv_t(const ConvArgs& a, dim3 grid_rows, int max_rows, cudaStream_t s) {
    constexpr int COUTP = (COUT + 3) & ~3;
    const size_t smem   = (static_cast<size_t>(a.n_slots) * CIN * COUTP + COUTP) * sizeof(float) + stage_bytes(a, COUT, T, R);
    static LaunchPlans plans;
    plans.get([](int) {
        VM_CUDA(cudaFuncSetAttribute(k_graph_conv<CIN, COUT, R, T, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024));
        return LaunchPlan{};
    });
    dim3 grid((max_rows + T * R - 1) / (T * R), grid_rows.y);
    k_graph_conv<CIN, COUT, R, T, MINB><<<grid, T, smem, s>>>(a);
}

template <int CIN, int COUT, int R, int WMAX, int T = CONV_THREADS>
static bool launch_conv_cw(const DenseLayer& L, const ConvArgs& a, dim3 grid_rows, int max_rows, cudaStream_t s) {
    if (L.host_packed.size() > static_cast<size_t>(WMAX)) return false;
    ConvWeights<WMAX> wp;
    std::memcpy(wp.w, L.host_packed.data(), L.host_packed.size() * sizeof(float));
    dim3 grid((max_rows + T * R - 1) / (T * R), grid_rows.y);
    // Layers bound by the latency of their gather rather than by the FP32 pipe - 4-channel first layers, 8 -> 8, and
    // the narrow last layers - run with the slot loop unrolled (slot count as a template parameter): the loads of the
    // next slots are then issued ahead of the current slot's arithmetic. Measured on 4.4 M rows: 4 -> 16 183 -> 114 us
    // (with the weights in the parameter space instead of shared memory), 8 -> 8 133 -> 112 us, 32 -> 4 448 -> 413 us;
    // the 16- and 32-channel layers in between, bound by the FP32 pipe, measured 3-6 % slower unrolled and stay rolled.
    const size_t smem            = stage_bytes(a, COUT, T, R);
    const bool early             = a.early && starts_early(static_cast<int64_t>(grid.x) * grid.y, 2, sm_count());
    // 12 -> 8 and 8 -> 12 go with the narrow ones.
    constexpr bool LATENCY_BOUND = CIN * COUT <= 96 || CIN == 4 || COUT <= 4;
    if (LATENCY_BOUND && a.n_slots == 5) { launch_kernel(k_graph_conv_cw<CIN, COUT, R, WMAX, T, LATENCY_BOUND ? 5 : 0>, grid, T, smem, s, early, a, wp); }
    else if (LATENCY_BOUND && a.n_slots == 7) {
        launch_kernel(k_graph_conv_cw<CIN, COUT, R, WMAX, T, LATENCY_BOUND ? 7 : 0>, grid, T, smem, s, early, a, wp);
    }
    else if (LATENCY_BOUND && a.n_slots == 9) {
        launch_kernel(k_graph_conv_cw<CIN, COUT, R, WMAX, T, LATENCY_BOUND ? 9 : 0>, grid, T, smem, s, early, a, wp);
    }
    else {
        launch_kernel(k_graph_conv_cw<CIN, COUT, R, WMAX, T>, grid, T, smem, s, early, a, wp);
    }
    return true;
}

// One shape: parameter-space weights where they fit (two rows per thread and 256 threads measured best for every shape tried). For few
// rows one row per thread, or the kernel that keeps part of the outputs' weights in shared memory.
template <int CIN, int COUT, int RR>
static bool launch_conv_shape(const DenseLayer& L, const ConvArgs& a, dim3 grid, int max_rows, cudaStream_t s) {
    if (L.cin != CIN || L.cout != COUT) return false;
    if (const_weights() && few_rows(max_rows, grid.y)) {
        const int blocks = L.host_packed.size() > static_cast<size_t>(CW_MAX) ? FEW_BLOCKS : COUT == 12 ? FEW_BLOCKS_TWELVE : FEW_BLOCKS_SPECIALISED;
        if (L.host_packed.size() > FEW_WEIGHTS && launch_conv_few(L, a, grid, max_rows, blocks, s)) return true;
        if (launch_conv_cw<CIN, COUT, 1, CW_MAX, 128>(L, a, grid, max_rows, s)) return true;
    }
    if (const_weights() && launch_conv_cw<CIN, COUT, 2, CW_MAX, 256>(L, a, grid, max_rows, s)) return true;
    launch_conv_t<CIN, COUT, RR>(a, grid, max_rows, s);
    return true;
}

}  // namespace vm
