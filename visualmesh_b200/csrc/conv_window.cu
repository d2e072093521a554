// Launchers of the window graph-convolution layers (conv_window.cuh).
#include <cstring>

#include "conv_dispatch.hpp"
#include "../../include/vmcuda.h"
#include "conv_window.cuh"

namespace vm {

template <int NP, int NSLOTS>
static void launch_conv_window_t(const DenseLayer& L, const ConvArgs& a, const st::Plan& plan, int n_frames, int max_rows, int32_t* abort_flags,
                                 uint32_t wait_limit, cudaStream_t s) {
    constexpr auto kernel = win::k_graph_conv_window<NP, NSLOTS>;
    constexpr size_t smem = win::smem_bytes<NP>(NSLOTS);
    static LaunchPlans plans;
    const LaunchPlan& lp = plans.get([](int dev) {
        LaunchPlan p;
        VM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        VM_CUDA(cudaDeviceGetAttribute(&p.n_sms, cudaDevAttrMultiProcessorCount, dev));
        p.ctas_per_sm = 1;  // a CTA takes all tensor memory of its SM
        return p;
    });
    win::Args t{};
    t.weights     = L.d_tc_win;
    t.bias        = L.d_tc_bias;
    t.n_frames    = n_frames;
    t.cout        = L.cout;
    t.abort_flags = abort_flags;
    t.wait_limit  = wait_limit;
    const int tiles_upper = n_frames * 2 * ((max_rows + st::ST - 1) / st::ST);  // few super-tiles: half a super-tile per CTA
    const int grid        = std::max(1, std::min(tiles_upper, lp.n_sms));
    launch_kernel(kernel, dim3(grid), win::THREADS, smem, s, a.early && starts_early(tiles_upper, 2, lp.n_sms), a, t, plan);
}

bool has_window_kernel(const DenseLayer& L) {
    return L.d_tc_win != nullptr && L.cin == win::CIN && (L.n_slots == 5 || L.n_slots == 7 || L.n_slots == 9);
}

std::vector<unsigned char> pack_window_weights(const float* weights, int n_slots, int cout) {
    const int np = cout <= 16 ? 16 : 32;
    std::vector<unsigned char> packed(static_cast<size_t>(n_slots) * 4 * 2 * np * 16, 0);
    for (int slot = 0; slot < n_slots; ++slot) {
        for (int k = 0; k < 32; ++k) {  // 16 columns of channel pairs; what follows them repeats
            const int channel = 2 * win::pair_of_column(k / 2) + k % 2;
            for (int n = 0; n < np; ++n) {
                const int out = win::channel_of_column(np, n);
                if (out >= cout) continue;
                const float w   = weights[(static_cast<size_t>(slot) * win::CIN + channel) * cout + out];
                const __half h  = __float2half_rn(w);
                const __half l  = __float2half_rn(w - __half2float(h));
                const size_t at = (static_cast<size_t>(slot) * 4 + k / 8) * 2 * np * 16 + (k % 8) * 2;
                std::memcpy(&packed[at + static_cast<size_t>(n) * 16], &h, 2);
                std::memcpy(&packed[at + static_cast<size_t>(np + n) * 16], &l, 2);
            }
        }
    }
    return packed;
}

bool launch_conv_window(const DenseLayer& L, const ConvArgs& a, const StagedPlan& plan, int n_frames, int max_rows, int32_t* abort_flags,
                        uint32_t wait_limit, cudaStream_t s) {
    const st::Plan p{plan.nbl, plan.halo_rows, plan.halo_count};
#define VM_WIN(NPAD, NS)                                                                           \
    if (L.tc_np == NPAD && L.n_slots == NS) {                                                      \
        launch_conv_window_t<NPAD, NS>(L, a, p, n_frames, max_rows, abort_flags, wait_limit, s);   \
        return true;                                                                               \
    }
    VM_WIN(16, 5) VM_WIN(16, 7) VM_WIN(16, 9) VM_WIN(32, 5) VM_WIN(32, 7) VM_WIN(32, 9)
#undef VM_WIN
    return false;
}

}  // namespace vm
