// Host side of the engine and its C ABI (include/vmcuda.h).
//
// One engine instance owns its streams, its grow-only device scratch and its pinned result buffers; like the
// reference engines it is not thread-safe - use one instance per host thread. A batch is cut into chunks of frames;
// chunks rotate over a few lanes (streams + scratch) so that the host-to-device copy of one chunk's images, the
// kernels of another and the device-to-host copy of a third overlap. Nothing waits for the device before the batch's end:
// offsets, results and abort flags are written into pinned host memory by the kernels themselves, and a chunk of a shape that
// returns is one launch of a recorded graph.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/vmcuda.h"
#include "host_math.hpp"
#include "kernels.cuh"
#include "conv_dispatch.hpp"
#include "upload.hpp"
#include "libm_tables.hpp"

namespace vm {

static thread_local std::string g_error;

static vm_status fail(vm_status s, const std::string& msg) {
    g_error = msg;
    return s;
}

// the per-frame constants could not be computed: a projection the lens math does not know (the reference throws from
// unproject, cpp/visualmesh/utility/projection.hpp:224)
struct UnsupportedLens {};

// The status of the exception in flight: nothing leaves a C entry point as an exception. Called inside a handler.
static vm_status status_of_exception() {
    cudaGetLastError();
    try {
        throw;
    }
    catch (const CudaFailure& f) {
        const vm_status s = f.code == cudaErrorMemoryAllocation ? VM_ERR_OUT_OF_MEMORY : VM_ERR_CUDA;
        return fail(s, std::string(cudaGetErrorName(f.code)) + ": " + cudaGetErrorString(f.code) + " in " + f.what);
    }
    catch (const UnsupportedLens&) {
        return fail(VM_ERR_UNSUPPORTED_LENS, "Cannot project: Unknown lens type");
    }
    catch (const std::bad_alloc&) {
        return fail(VM_ERR_OUT_OF_MEMORY, "out of host memory");
    }
    catch (const std::exception& x) {
        return fail(VM_ERR_CUDA, x.what());
    }
}

// Grow-only device and pinned-host arrays (the reference's OpenCL engine keeps the same kind of caches,
// cpp/visualmesh/engine/opencl/engine.hpp:740-835).
template <typename T>
struct DeviceArray {
    T* p       = nullptr;
    size_t cap = 0;
    bool ensure(size_t n) {  // true when the array was reallocated
        if (n <= cap) return false;
        if (p != nullptr) VM_CUDA(cudaFree(p));
        p   = nullptr;
        cap = 0;
        const size_t want = n + n / 8 + 64;
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&p), want * sizeof(T)));
        cap = want;
        return true;
    }
    void release() {
        if (p != nullptr) cudaFree(p);
        p   = nullptr;
        cap = 0;
    }
};

template <typename T>
struct PinnedArray {
    T* p       = nullptr;
    size_t cap = 0;
    bool ensure(size_t n) {  // true when the array was reallocated
        if (n <= cap) return false;
        if (p != nullptr) VM_CUDA(cudaFreeHost(p));
        p   = nullptr;
        cap = 0;
        const size_t want = n + n / 8 + 64;
        VM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&p), want * sizeof(T), cudaHostAllocDefault));
        cap = want;
        return true;
    }
    void release() {
        if (p != nullptr) cudaFreeHost(p);
        p   = nullptr;
        cap = 0;
    }
};

static_assert(libm::FIRST_BITS[libm::ACOS] == LIBM_FIRST_BITS && libm::END_BITS[libm::ACOS] == LIBM_ONE_BITS
                && libm::FIRST_BITS[libm::SIN] == LIBM_FIRST_BITS && libm::END_BITS[libm::SIN] == LIBM_TWO_BITS
                && libm::FIRST_BITS[libm::TAN] == LIBM_FIRST_BITS && libm::END_BITS[libm::TAN] == LIBM_TWO_BITS,
              "the device reads the last-bit tables over the ranges the host builds them for");

// Device copies of the libm last-bit tables, built on first use and shared by all engines of a process (per device).
constexpr int LIBM_MAX_DEVICES = 64;
static uint32_t* g_libm_device[LIBM_MAX_DEVICES][libm::N_FUNCTIONS] = {};
static std::mutex g_libm_mutex;

static const uint32_t* libm_table(int device, int fn, bool build_if_missing) {
    static const bool disabled = [] {
        const char* v = std::getenv("VMCUDA_LIBM_TABLES");
        return v != nullptr && v[0] == '0';
    }();
    if (disabled || device < 0 || device >= LIBM_MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> lock(g_libm_mutex);
    if (g_libm_device[device][fn] == nullptr && build_if_missing) {
        const std::vector<uint32_t> packed = libm::build(fn);
        uint32_t* d = nullptr;
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&d), packed.size() * sizeof(uint32_t)));
        VM_CUDA(cudaMemcpy(d, packed.data(), packed.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
        g_libm_device[device][fn] = d;
    }
    return g_libm_device[device][fn];
}

constexpr int MAX_LANES = 4;

struct Lane {
    cudaStream_t stream = nullptr;
    cudaStream_t side   = nullptr;     // runs beside `stream` within a chunk: sampling next to the neighbour remap, result copies
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    cudaEvent_t ev_offsets = nullptr;  // this chunk's offsets are on the device
    cudaEvent_t ev_projected = nullptr;  // everything of its projection is
    cudaEvent_t ev_images  = nullptr;  // its images are
    cudaEvent_t ev_done    = nullptr;  // everything of this chunk, result copies included, has finished
    bool busy = false;
    // staging block of a chunk, copied to the device in one piece: header, frame constants, range pairs and starts, group counts
    // (zeros), small images
    PinnedArray<uint8_t> h_staging;
    DeviceArray<uint8_t> d_staging;
    DeviceArray<uint8_t> d_state;
    DeviceArray<float2> d_cand_px;
    DeviceArray<int32_t> d_cand_node;
    DeviceArray<int32_t> d_block_counts;
    DeviceArray<int32_t> d_node_rank;
    DeviceArray<float> d_feat[2];
    DeviceArray<uint8_t> d_images;
    PinnedArray<uint8_t> h_images;  // staging of images that come from pageable memory
    // tile plan of the chunk for the staged tensor-core layers (conv_staged.cuh)
    DeviceArray<uint16_t> d_nbl;
    DeviceArray<int32_t> d_halo_rows;
    DeviceArray<int32_t> d_halo_count;

    // Makes the streams and events, when the lane is first used: a call of one chunk takes one lane of the four.
    void open(bool blocking_sync) {
        if (stream != nullptr) return;
        if (side == nullptr) VM_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        // ev_offsets and ev_done are the ones the host waits on: spinning (lowest latency) or, with VMCUDA_BLOCKING_SYNC=1, sleeping - for
        // boxes where several engines' host threads share few cores
        for (cudaEvent_t* ev : {&ev_fork, &ev_join, &ev_images, &ev_projected, &ev_offsets, &ev_done}) {
            const unsigned waits = (ev == &ev_offsets || ev == &ev_done) && blocking_sync ? cudaEventBlockingSync : 0;
            if (*ev == nullptr) VM_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming | waits));
        }
        VM_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    }
};

// One set of result arrays in pinned host memory. An engine writes its results into the set it holds; a caller may keep the set
// of the last call (vm_results_keep), and the engine takes another one for the next.
struct Results {
    PinnedArray<int32_t> offsets;
    PinnedArray<float2> px;
    PinnedArray<int32_t> gi;
    PinnedArray<int32_t> nb;
    PinnedArray<float> cls;
    ~Results() {
        offsets.release();
        px.release();
        gi.release();
        nb.release();
        cls.release();
    }
};
// The sets of an engine that are not in its hands: kept by callers, or given back and free. Outlives the engine while some are kept,
// and is given back to from any thread.
constexpr int MAX_KEPT_RESULTS = 4;
static_assert(MAX_KEPT_RESULTS == VM_MAX_KEPT_RESULTS, "as the header says");
struct ResultPool {
    ResultPool() {
        free.reserve(MAX_KEPT_RESULTS + 1);  // all sets there can be: giving one back allocates nothing
    }
    std::mutex mutex;
    std::vector<std::unique_ptr<Results>> free;
    int kept    = 0;
    bool closed = false;  // the engine is gone: sets that come back are freed
};
struct KeptResults {
    std::shared_ptr<ResultPool> pool;
    std::unique_ptr<Results> results;
};

struct StageTimer {
    const char* name;
    cudaEvent_t start, stop;
};

// What the recorded graph of a chunk's kernels depends on besides the contents of its buffers: everything that ends up in a launch's
// grid or arguments. Compared byte for byte. The staging block's layout is in it by every offset that a kernel gets (its size alone does
// not fix where the group counts lie: range slots before them and small images behind them may make up for each other).
struct GraphKey {
    int32_t part, lane, n_frames, f0, n_neighbours, blocks_per_frame, bsp_blocks, options;
    uint32_t wait_limit;
    int32_t feature_stride;
    uint64_t staging_bytes, counts_at;
};
struct GraphEntry {
    GraphKey key;
    cudaGraphExec_t exec = nullptr;
    int64_t kernels      = 0;
    uint64_t last_use    = 0;
    bool refused         = false;  // could not be recorded: its kernels are launched one by one
};
constexpr size_t MAX_GRAPHS = 48;  // per engine; the least recently used one goes first

}  // namespace vm

struct vm_mesh {
    const vm_engine* owner = nullptr;  // the engine it was uploaded through (and whose device holds it)
    int32_t n_nodes = 0, n_neighbours = 0, n_bsp = 0;
    float4* d_rays        = nullptr;
    int32_t* d_neighbours = nullptr;
    float4* d_cones_a     = nullptr;
    float* d_cones_s      = nullptr;
    int4* d_topology      = nullptr;
};

struct vm_engine {
    int device = 0;
    std::vector<vm::DenseLayer> layers;
    int max_width = 4;
    int n_classes = 0;
    vm::Lane lanes[vm::MAX_LANES];
    int n_lanes = vm::MAX_LANES;
    cudaStream_t copy_stream = nullptr;  // images on their way to the device, chunk after chunk
    int64_t chunk_candidates = 2 << 20;
    int chunk_frames         = 16;
    bool chunk_override      = false;  // set by the environment: use the limits above for every batch
    // batch-wide results
    vm::DeviceArray<int32_t> d_offsets;
    vm::DeviceArray<float2> d_px;
    vm::DeviceArray<int32_t> d_gi;
    vm::DeviceArray<int32_t> d_nb;
    vm::DeviceArray<float> d_cls;
    std::unique_ptr<vm::Results> host;  // ... and where they arrive on the host
    std::shared_ptr<vm::ResultPool> pool = std::make_shared<vm::ResultPool>();
    int32_t* flags = nullptr;  // abort flags, pinned host memory that the kernels raise them in
    std::vector<vm_mesh*> meshes;
    // recorded graphs
    bool use_graphs       = true;
    uint64_t graph_uses   = 0;
    bool buffers_moved    = false;  // a device buffer was reallocated: the recorded graphs name addresses that are gone
    std::vector<vm::GraphEntry> graphs;
    // constants of the last lens seen
    vm_lens lens{};
    bool lens_known = false;
    vm::host::EdgeRays lens_rays{};
    float lens_cos_fov = 0, lens_sin_fov = 0;
    // stage timing
    std::vector<vm::StageTimer> timers;
    std::vector<cudaEvent_t> event_pool;
    size_t events_used = 0;
    bool timing        = false;
    std::vector<std::pair<const char*, float>> stage_ms;
    int64_t launches = 0;
    bool use_tc      = true;
    int tc_mode      = 1;
    // mode 1: layers with C_in x C_out at least this run on the tensor cores. Narrower ones are slower there: 32 -> 4 over 7.4 M rows takes
    // 790 us on the CUDA cores and 2241 us on the window kernel.
    int tc_min_product = 512;
    bool tc_no_split = false;   // debugging: never use the split feature layout
    bool staged          = true;    // tensor-core layers read their gather from shared-memory windows (conv_staged.cuh)
    bool may_stage       = false;   // some layer could run as a staged tensor-core layer under the engine's policy
    uint32_t tc_wait_limit = vm::TC_DEFAULT_WAIT_LIMIT;  // polls of one mbarrier wait in the tensor-core kernels (vm_set_wait_limit)
    cudaEvent_t ev_timer_start = nullptr, ev_timer_stop = nullptr;
    bool blocking_sync         = false;    // host waits sleep instead of spinning
    bool nvtx                  = false;    // NVTX ranges around every kernel launch and batch (VMCUDA_NVTX=1)
    std::shared_ptr<vm::UploadHelpers> helpers;  // taken at the first upload from pageable memory
};

namespace vm {

// Device buffers and staging blocks of the batch path: a reallocation makes the recorded graphs stale.
template <typename Array>
static void need(vm_engine* e, Array& a, size_t n) {
    if (a.ensure(n)) e->buffers_moved = true;
}

// A stage is one kernel launch. With VMCUDA_NVTX=1 every launch sits in an NVTX range of the stage's name (the header-only
// NVTX does nothing unless a profiler is attached); with stage timing on, between two CUDA events.
static void begin_stage(vm_engine* e, cudaStream_t s, const char* name) {
    ++e->launches;
    if (e->nvtx) nvtxRangePushA(name);
    if (!e->timing) return;
    while (e->event_pool.size() < e->events_used + 2) {
        cudaEvent_t ev;
        VM_CUDA(cudaEventCreate(&ev));
        e->event_pool.push_back(ev);
    }
    StageTimer t{name, e->event_pool[e->events_used], e->event_pool[e->events_used + 1]};
    e->events_used += 2;
    VM_CUDA(cudaEventRecord(t.start, s));
    e->timers.push_back(t);
}
static void end_stage(vm_engine* e, cudaStream_t s) {
    VM_CUDA(cudaGetLastError());
    if (e->nvtx) nvtxRangePop();
    if (!e->timing) return;
    VM_CUDA(cudaEventRecord(e->timers.back().stop, s));
}

enum ConvKind { CONV_FFMA = 0, CONV_TC_GATHER = 1, CONV_TC_SPLIT = 2, CONV_TC_STAGED = 3, CONV_TC_WINDOW = 4 };

// Whether the kernel that runs layer L as `kind` honours ConvArgs::out_split. The tensor-core kernels write the split
// layout when their tile is exactly as wide as the layer; the specialised FFMA kernels when the width is a multiple
// of 8; the generic kernel never does.
static bool producer_writes_split(const DenseLayer& L, ConvKind kind) {
    if (kind == CONV_TC_STAGED || kind == CONV_TC_WINDOW) return L.cout % 8 == 0;
    if (kind != CONV_FFMA) return L.cout == L.tc_np;
    return has_fast_ffma_kernel(L.cin, L.cout) && L.cout % 8 == 0;
}
// the same for SPLIT_ROWS, the layout of the window kernel's 32 input channels
static bool producer_writes_rows(const DenseLayer& L, ConvKind kind) {
    return L.cout == 32 && kind != CONV_TC_GATHER && kind != CONV_TC_SPLIT && producer_writes_split(L, kind);
}

// Scratch of a chunk's tile plan (tile_plan.cuh): neighbour positions per row, halo lists per super-tile.
static void ensure_tile_plan(vm_engine* e, Lane& lane, size_t rows_cap, size_t supertiles_cap) {
    need(e, lane.d_nbl, rows_cap * STAGED_NBL_STRIDE + 64);
    need(e, lane.d_halo_rows, supertiles_cap * STAGED_HALO + 64);
    need(e, lane.d_halo_count, supertiles_cap + 64);
}
static st::PlanOut tile_plan(Lane& lane) {
    return st::PlanOut{lane.d_nbl.p, lane.d_halo_rows.p, lane.d_halo_count.p};
}

static void launch_conv(vm_engine* e, const DenseLayer& L, ConvArgs a, int n_frames, int max_rows, cudaStream_t s, ConvKind kind, const StagedPlan& plan) {
    a.weights     = L.d_weights;
    a.biases      = L.d_weights + static_cast<size_t>(L.n_slots) * L.cin * L.coutp;
    a.n_slots     = L.n_slots;
    a.activation  = L.activation;
    begin_stage(e, s, L.stage.c_str());
    // A layer's kind fixes the layout of its input: there is no other kernel to fall back to.
    bool launched = false;
    switch (kind) {
        case CONV_TC_WINDOW: launched = launch_conv_window(L, a, plan, n_frames, max_rows, e->flags, e->tc_wait_limit, s); break;
        case CONV_TC_STAGED: launched = launch_conv_staged(L, a, plan, n_frames, max_rows, e->flags, e->tc_wait_limit, s); break;
        case CONV_TC_SPLIT: launched = launch_conv_tc_split(L, a, n_frames, max_rows, e->flags, e->tc_wait_limit, s); break;
        case CONV_TC_GATHER: launched = launch_conv_tc_gather(L, a, n_frames, max_rows, e->flags, e->tc_wait_limit, s); break;
        case CONV_FFMA:
            launch_conv_ffma(L, a, n_frames, max_rows, s);
            launched = true;
            break;
    }
    if (!launched) throw std::logic_error("no kernel for layer " + L.stage + " in the layout of its input");
    end_stage(e, s);
}

// Runs all layers over a chunk whose input features are in feat[0]; the last layer writes out_final.
static void run_network(vm_engine* e,
                        Lane& lane,
                        bool plan_valid,
                        const int32_t* d_offsets,
                        const int32_t* d_nb,
                        int n_neighbours,
                        int f0,
                        int n_frames,
                        int max_rows,
                        float* out_final,
                        bool final_global,
                        int feature_stride,
                        float* const* out_host = nullptr) {
    // Which kernel runs each layer (VMCUDA_TC: 0 = CUDA cores only; 1, the default, and 2 = tensor cores too).
    // A 16-channel layer whose producer can write the split layout runs as a staged layer (conv_staged.cuh), a dense one with 32
    // channels in on the window kernel (conv_window.cuh; VMCUDA_STAGED=0 turns both off). Otherwise the tcgen05 kernels take a layer when its contraction is dense enough to
    // pay (mode 1: C_in x C_out >= 512) or whenever one exists (mode 2): fed by plain copies from the split layout
    // (CONV_TC_SPLIT) or gathering and splitting fp32 themselves (CONV_TC_GATHER).
    const size_t n_layers = e->layers.size();
    std::vector<ConvKind> kind(n_layers, CONV_FFMA);
    for (size_t l = 0; l < n_layers; ++l) {
        const DenseLayer& L = e->layers[l];
        if (!e->use_tc || L.tc_np == 0 || L.n_slots == 1 || n_frames > TC_MAX_FRAMES) continue;
        const bool producer_can_split = l > 0 && producer_writes_split(e->layers[l - 1], kind[l - 1]) && !e->tc_no_split;
        // the staged kernel wherever it exists (it writes features, not results: never the last layer)
        if (e->staged && plan_valid && producer_can_split && has_staged_kernel(L) && l + 1 < n_layers) {
            kind[l] = CONV_TC_STAGED;
            continue;
        }
        // the tcgen05 kernels where the contraction is dense enough for them to pay (mode 1) or wherever they exist (mode 2)
        const bool producer_can_rows = l > 0 && producer_writes_rows(e->layers[l - 1], kind[l - 1]) && !e->tc_no_split;
        if (e->tc_mode == 1 && L.cin * L.cout < e->tc_min_product) continue;
        if (e->staged && plan_valid && producer_can_rows && has_window_kernel(L) && (l + 1 == n_layers || L.cout % 4 == 0)) kind[l] = CONV_TC_WINDOW;
        else if (has_tc_split_kernel(L) && producer_can_split) kind[l] = CONV_TC_SPLIT;
        else if (has_tc_gather_kernel(L)) kind[l] = CONV_TC_GATHER;
        // anything else (dense-only layers, shapes without a tensor-core instantiation) stays on the FFMA kernels
    }
    const StagedPlan plan{lane.d_nbl.p, lane.d_halo_rows.p, lane.d_halo_count.p};
    int cur = 0;
    for (size_t l = 0; l < n_layers; ++l) {
        const bool last = l + 1 == n_layers;
        ConvArgs a{};
        a.in           = lane.d_feat[cur].p;
        a.out          = last ? out_final : lane.d_feat[cur ^ 1].p;
        a.nb           = d_nb;
        a.offsets      = d_offsets;
        a.n_neighbours = n_neighbours;
        a.f0           = f0;
        a.out_global   = (last && final_global) ? 1 : 0;
        a.in_stride    = feature_stride;
        a.out_stride   = feature_stride;
        a.out_planar   = (!last && e->layers[l].cout % 4 == 0) ? 1 : 0;
        a.out_split    = last ? SPLIT_NONE : kind[l + 1] == CONV_TC_WINDOW ? SPLIT_ROWS : kind[l + 1] == CONV_TC_STAGED ? SPLIT_QUADS : kind[l + 1] >= CONV_TC_SPLIT ? SPLIT_PLANES : SPLIT_NONE;
        a.out_host     = last ? out_host : nullptr;
        a.range_flag   = e->flags;
        // not the first layer, which follows two streams that have joined, and none behind a window kernel but another: a CTA of that one
        // fills its SM, and the 32 -> 4 layer started behind ten of them cost 45 us of 157 (121 k nodes)
        const bool behind_window = l > 0 && kind[l - 1] == CONV_TC_WINDOW && kind[l] != CONV_TC_WINDOW;
        a.early                  = l > 0 && !behind_window && a.out_host == nullptr && !e->timing ? 1 : 0;
        launch_conv(e, e->layers[l], a, n_frames, max_rows, lane.stream, kind[l], plan);
        cur ^= 1;
    }
}

// ---- per-frame constants -----------------------------------------------------------------------------------------

static bool fill_frame_params(vm_engine* e, const vm_frame& fr, FrameParams& p, bool may_allocate = true) {
    const float* H = fr.Hoc;
    // Rco = block<3,3>(transpose(Hoc)), cpp/visualmesh/engine/cpu/engine.hpp:95
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) p.Rco[i * 3 + j] = H[j * 4 + i];
    p.focal_length = fr.lens.focal_length;
    p.centre[0]    = fr.lens.centre[0];
    p.centre[1]    = fr.lens.centre[1];
    p.half_dims[0] = float(fr.lens.dimensions[0]) * 0.5f;
    p.half_dims[1] = float(fr.lens.dimensions[1]) * 0.5f;
    host::inverse_coefficients(fr.lens.k, p.ik);
    p.dims[0]    = fr.lens.dimensions[0];
    p.dims[1]    = fr.lens.dimensions[1];
    p.projection = fr.lens.projection;
    p.format     = fr.format;
    // what depends on the lens alone and takes a dozen libm calls is worked out when the lens changes
    if (!e->lens_known || std::memcmp(&e->lens, &fr.lens, sizeof(vm_lens)) != 0) {
        e->lens_known = false;
        if (!host::edge_rays(fr.lens, e->lens_rays)) return false;
        // cpp/visualmesh/mesh.hpp:503-504
        e->lens_cos_fov = std::cos(fr.lens.fov * 0.5f);
        e->lens_sin_fov = std::sin(fr.lens.fov * 0.5f);
        e->lens         = fr.lens;
        e->lens_known   = true;
    }
    p.cos_fov = e->lens_cos_fov;
    p.sin_fov = e->lens_sin_fov;
    if (fr.ranges == nullptr) {
        std::array<host::Cone, 4> edges;
        host::screen_edges(H, fr.lens, e->lens_rays, edges);
        for (int i = 0; i < 4; ++i) {
            p.edges[i][0] = edges[i].axis[0];
            p.edges[i][1] = edges[i].axis[1];
            p.edges[i][2] = edges[i].axis[2];
            p.edges[i][3] = edges[i].cos_t;
            p.edges[i][4] = edges[i].sin_t;
        }
    }
    p.libm_acos = libm_table(e->device, libm::ACOS, may_allocate);
    p.libm_sin  = fr.lens.projection == VM_EQUISOLID ? libm_table(e->device, libm::SIN, may_allocate) : nullptr;
    p.libm_tan  = fr.lens.projection == VM_RECTILINEAR ? libm_table(e->device, libm::TAN, may_allocate) : nullptr;
    const vm_mesh* m = fr.mesh;
    p.rays           = m->d_rays;
    p.neighbours     = m->d_neighbours;
    p.bsp_cones_a    = m->d_cones_a;
    p.bsp_cones_s    = m->d_cones_s;
    p.bsp_topology   = m->d_topology;
    p.n_nodes        = m->n_nodes;
    p.n_bsp          = m->n_bsp;
    return true;
}

static size_t image_bytes(const vm_frame& fr) {
    const int cls = format_class(fr.format);
    return static_cast<size_t>(fr.lens.dimensions[0]) * fr.lens.dimensions[1] * format_bytes_per_pixel(cls);
}

static int64_t frame_candidates(const vm_frame& fr) {
    if (fr.ranges == nullptr) return fr.mesh->n_nodes;
    int64_t n = 0;
    for (int r = 0; r < fr.n_ranges; ++r) n += std::max(0, fr.ranges[2 * r + 1] - fr.ranges[2 * r]);
    return n;
}

static size_t aligned(size_t n) {
    return (n + 255) & ~size_t(255);
}

// Sizes that shape the launches are rounded up (by an eighth at most), so that calls whose poses differ a little share a graph.
static int64_t rounded(int64_t n) {
    if (n >= int64_t(1) << 30) return n;  // the next step would pass what the 32-bit indices hold
    int64_t step = 1024;
    while (step * 16 <= n) step *= 2;
    return (n + step - 1) / step * step;
}

// ---- one chunk -----------------------------------------------------------------------------------------------------

// Images up to this size travel inside the chunk's staging block: for them a copy of their own costs more than the bytes.
constexpr size_t SMALL_IMAGES = 128 << 10;

// Results of a single chunk up to this size are written to the host by the device; more are copied by the copy engines, which leave
// the SMs alone (a persistent layer kernel that finds some of its SM occupied runs in two waves), at the price of a wait for the
// number of points in the middle of the call.
constexpr int64_t MAX_EXPORT = 16 << 20;

// Host images of one chunk of a batch.
constexpr size_t CHUNK_IMAGE_BYTES = 21 << 20;

// Nodes, and BSP elements, of the meshes of one chunk's frames. With host ranges the candidates say nothing about either, and the
// node tables of 256 frames on a mesh of 8.4 M nodes would pass the 32-bit offsets that find them. The limit lies lower: the node table
// takes 4 bytes a node in every lane (512 MB here; 64 frames on a mesh of 1.7 M nodes fit). One frame is always accepted.
constexpr int64_t MAX_CHUNK_NODES = int64_t(1) << 27;

struct Chunk {
    int f0 = 0, f1 = 0, n_neighbours = 0;
    bool classify = false, device_lookup = false, packed4 = false, with_plan = false;
    bool images_apart = false;  // host images that travel on the copy stream
    bool exported     = false;  // results are written to the host by k_export
    bool copied       = false;  // ... or copied there once the host knows how many there are
    int blocks_per_frame = 0, n_groups = 0, bsp_blocks = 0, max_rows = 0, stride = 0;
    size_t staging_bytes = 0, counts_at = 0;
};

// Where a chunk's host images go in the lane's buffers: pageable ones first (their slices are sent as runs of the staging
// buffer), then the pinned ones.
struct ImagePlan {
    std::vector<size_t> at;  // per frame of the chunk
    size_t total = 0, pageable = 0;
    bool small = false;
};

static bool is_pageable(const void* p) {
    cudaPointerAttributes attributes{};
    if (cudaPointerGetAttributes(&attributes, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return attributes.type == cudaMemoryTypeUnregistered;
}

static ImagePlan plan_images(const vm_frame* frames, int f0, int f1) {
    ImagePlan plan;
    plan.at.assign(f1 - f0, 0);
    for (int f = f0; f < f1; ++f)
        if (!frames[f].image_on_device) plan.total += aligned(image_bytes(frames[f]));
    plan.small = plan.total <= SMALL_IMAGES;
    std::vector<char> pageable(f1 - f0, 0);
    for (int f = f0; f < f1 && !plan.small; ++f) pageable[f - f0] = !frames[f].image_on_device && is_pageable(frames[f].image);
    size_t cursor = 0;
    for (const char wanted : {1, 0}) {
        for (int f = f0; f < f1; ++f) {
            if (frames[f].image_on_device || pageable[f - f0] != wanted) continue;
            plan.at[f - f0] = cursor;
            cursor += aligned(image_bytes(frames[f]));
        }
        if (wanted) plan.pageable = cursor;
    }
    return plan;
}

// Starts the images of a chunk on their way. Pinned frames that follow one another in host memory (a caller's ring of camera
// buffers, the rows of one big array) travel as ONE copy: sixteen 5 MB copies per chunk cost measurably more host time and bus
// turn-around than one 84 MB copy. Pageable frames go through the upload helpers.
static std::unique_ptr<Upload> start_images(vm_engine* e, Lane& lane, const vm_frame* frames, int f0, int f1, const ImagePlan& plan) {
    need(e, lane.d_images, plan.total + 256);
    if (e->copy_stream == nullptr) VM_CUDA(cudaStreamCreateWithFlags(&e->copy_stream, cudaStreamNonBlocking));
    std::unique_ptr<Upload> upload;
    if (plan.pageable > 0) {
        if (!e->helpers) e->helpers = UploadHelpers::get();
        lane.h_images.ensure(plan.pageable);
        upload.reset(new Upload(e->helpers.get(), lane.d_images.p, e->copy_stream));
        for (int f = f0; f < f1; ++f)
            if (!frames[f].image_on_device && plan.at[f - f0] < plan.pageable)
                upload->job.add(static_cast<const uint8_t*>(frames[f].image), plan.at[f - f0], image_bytes(frames[f]));
        upload->start(lane.h_images.p);
    }
    const uint8_t* run_src = nullptr;
    size_t run_dst = 0, run_bytes = 0;
    int run_first = f0;
    auto copy = [&](const uint8_t* src, size_t dst, size_t bytes) {
        return cudaMemcpyAsync(lane.d_images.p + dst, src, bytes, cudaMemcpyHostToDevice, e->copy_stream);
    };
    auto flush = [&](int end) {
        if (run_bytes == 0) return;
        cudaError_t err = copy(run_src, run_dst, run_bytes);
        if (err == cudaErrorInvalidValue && run_bytes > image_bytes(frames[run_first])) {
            // frames that follow one another but were pinned one by one: a copy may not reach from one allocation into the next
            cudaGetLastError();
            err = cudaSuccess;
            for (int f = run_first; f < end && err == cudaSuccess; ++f) {
                if (frames[f].image_on_device || plan.at[f - f0] < plan.pageable) continue;
                err = copy(static_cast<const uint8_t*>(frames[f].image), plan.at[f - f0], image_bytes(frames[f]));
            }
        }
        VM_CUDA(err);
        run_bytes = 0;
    };
    for (int f = f0; f < f1; ++f) {
        if (frames[f].image_on_device || plan.at[f - f0] < plan.pageable) continue;
        const size_t bytes = image_bytes(frames[f]);
        const uint8_t* src = static_cast<const uint8_t*>(frames[f].image);
        if (run_bytes > 0 && src == run_src + run_bytes && plan.at[f - f0] == run_dst + run_bytes) { run_bytes += bytes; }
        else {
            flush(f);
            run_first = f;
            run_src   = src;
            run_dst   = plan.at[f - f0];
            run_bytes = bytes;
        }
    }
    flush(f1);
    return upload;
}

// Fills the chunk's staging block and works out its launches.
static Chunk stage_chunk(vm_engine* e, Lane& lane, const vm_frame* frames, int f0, int f1, bool classify, bool to_host, bool only_chunk, const ImagePlan& images) {
    const int nf = f1 - f0;
    Chunk c;
    c.f0           = f0;
    c.f1           = f1;
    c.classify     = classify;
    c.n_neighbours = frames[f0].mesh->n_neighbours;
    size_t n_ranges = 0, supertiles_cap = 0;
    int64_t cand_total = 0, node_total = 0, bsp_total = 0, max_cand = 0, max_bsp = 0;
    bool on_device = true;
    c.packed4      = true;
    for (int f = f0; f < f1; ++f) {
        const vm_frame& fr = frames[f];
        const int64_t nc   = frame_candidates(fr);
        if (fr.ranges != nullptr) { n_ranges += fr.n_ranges; }
        else {
            c.device_lookup = true;
            bsp_total += fr.mesh->n_bsp;
            max_bsp = std::max<int64_t>(max_bsp, fr.mesh->n_bsp);
        }
        cand_total += nc;
        node_total += fr.mesh->n_nodes;
        max_cand = std::max(max_cand, nc);
        supertiles_cap += static_cast<size_t>((nc + 1 + STAGED_ST - 1) / STAGED_ST);
        const int cls = format_class(fr.format);
        c.packed4     = c.packed4 && (cls == FMT_RGBA || cls == FMT_BGRA);
        on_device     = on_device && fr.image_on_device;
    }
    c.images_apart     = classify && !on_device && !images.small;
    c.exported         = to_host && only_chunk && cand_total * (12 + 4 * c.n_neighbours + 4 * (classify ? e->n_classes : 0)) <= MAX_EXPORT;
    c.copied           = to_host && !c.exported;
    c.blocks_per_frame = static_cast<int>(std::max<int64_t>(1, (rounded(max_cand) + SELECT_THREADS - 1) / SELECT_THREADS));
    c.n_groups         = (c.blocks_per_frame + GROUP_BLOCKS - 1) / GROUP_BLOCKS;
    c.bsp_blocks       = static_cast<int>((max_bsp + SELECT_THREADS - 1) / SELECT_THREADS);
    c.max_rows         = c.blocks_per_frame * SELECT_THREADS + 1;
    c.stride           = static_cast<int>(rounded(cand_total + nf));
    // the staged layer kernels want a tile plan of the chunk: the remap makes it while it has the indices in hand
    c.with_plan = classify && e->staged && e->use_tc && e->may_stage && nf <= TC_MAX_FRAMES;

    // layout of the staging block
    const size_t frames_at = aligned(sizeof(ChunkHeader));
    const size_t ranges_at = aligned(frames_at + sizeof(FrameParams) * nf);
    const size_t n_slots   = n_ranges == 0 ? 0 : std::max<size_t>(64, rounded(n_ranges));  // rounded like every size a graph depends on
    c.counts_at            = aligned(ranges_at + 3 * sizeof(int32_t) * n_slots);
    const size_t images_at = aligned(c.counts_at + sizeof(int32_t) * nf * c.n_groups);
    c.staging_bytes        = images_at + (classify && images.small ? images.total : 0);
    need(e, lane.h_staging, c.staging_bytes);
    need(e, lane.d_staging, c.staging_bytes);
    need(e, lane.d_cand_px, cand_total + 1);
    need(e, lane.d_cand_node, cand_total + 1);
    need(e, lane.d_node_rank, node_total + 1);
    need(e, lane.d_block_counts, static_cast<size_t>(c.blocks_per_frame) * nf);
    if (c.device_lookup) need(e, lane.d_state, bsp_total + 1);
    if (classify) {
        need(e, lane.d_feat[0], static_cast<size_t>(c.stride) * e->max_width);
        need(e, lane.d_feat[1], static_cast<size_t>(c.stride) * e->max_width);
    }
    if (c.with_plan) ensure_tile_plan(e, lane, static_cast<size_t>(c.stride), supertiles_cap);

    uint8_t* h = lane.h_staging.p;
    uint8_t* d = lane.d_staging.p;
    *reinterpret_cast<ChunkHeader*>(h) = ChunkHeader{e->host->px.p, e->host->gi.p, e->host->nb.p, e->host->cls.p, e->host->offsets.p};
    int32_t* pairs  = reinterpret_cast<int32_t*>(h + ranges_at);
    int32_t* starts = pairs + 2 * n_slots;
    auto on_gpu     = [&](const void* p) { return d + (static_cast<const uint8_t*>(p) - h); };
    size_t cursor   = 0;
    int64_t cand_off = 0, node_off = 0, bsp_off = 0;
    for (int f = f0; f < f1; ++f) {
        const vm_frame& fr = frames[f];
        FrameParams& p     = reinterpret_cast<FrameParams*>(h + frames_at)[f - f0];
        std::memset(&p, 0, sizeof(p));
        if (!fill_frame_params(e, fr, p)) throw UnsupportedLens{};
        p.cand_off = static_cast<int32_t>(cand_off);
        p.node_off = static_cast<int32_t>(node_off);
        p.bsp_off  = static_cast<int32_t>(bsp_off);
        if (fr.ranges == nullptr) {
            p.n_candidates = fr.mesh->n_nodes;
            bsp_off += fr.mesh->n_bsp;
        }
        else {
            // ranges and their exclusive prefix sums; an empty frame keeps non-null pointers, which mark host ranges
            p.n_ranges     = fr.n_ranges;
            p.ranges       = reinterpret_cast<const int2*>(on_gpu(pairs + 2 * cursor));
            p.range_starts = reinterpret_cast<const int32_t*>(on_gpu(starts + cursor));
            int32_t run    = 0;
            for (int r = 0; r < fr.n_ranges; ++r, ++cursor) {
                pairs[2 * cursor + 0] = fr.ranges[2 * r];
                pairs[2 * cursor + 1] = fr.ranges[2 * r + 1];
                starts[cursor]        = run;
                run += std::max(0, fr.ranges[2 * r + 1] - fr.ranges[2 * r]);
            }
            p.n_candidates = run;
        }
        cand_off += p.n_candidates;
        node_off += fr.mesh->n_nodes;
        if (!classify) continue;
        if (fr.image_on_device) { p.image = static_cast<const uint8_t*>(fr.image); }
        else if (images.small) {
            p.image = d + images_at + images.at[f - f0];
            std::memcpy(h + images_at + images.at[f - f0], fr.image, image_bytes(fr));
        }
        else {
            p.image = lane.d_images.p + images.at[f - f0];
        }
    }
    std::memset(h + c.counts_at, 0, sizeof(int32_t) * nf * c.n_groups);
    return c;
}

static const FrameParams* device_frames(const Lane& lane) {
    return reinterpret_cast<const FrameParams*>(lane.d_staging.p + aligned(sizeof(ChunkHeader)));
}
static const ChunkHeader* device_header(const Lane& lane) {
    return reinterpret_cast<const ChunkHeader*>(lane.d_staging.p);
}

// Exported arrays are copied by a few blocks that leave the SMs to the layers: 32 blocks of 512 threads keep the bus busy.
constexpr int EXPORT_BLOCKS = 32;

static void issue_export_points(vm_engine* e, Lane& lane, const Chunk& c, cudaStream_t s, bool neighbours) {
    begin_stage(e, s, "export_points");
    k_export<0><<<EXPORT_BLOCKS, EXPORT_THREADS, 0, s>>>(device_header(lane), e->d_offsets.p, c.f0, c.f1, c.n_neighbours, e->d_px.p, e->d_gi.p,
                                                         neighbours ? e->d_nb.p : nullptr);
    end_stage(e, s);
}
static void issue_export_neighbours(vm_engine* e, Lane& lane, const Chunk& c, cudaStream_t s) {
    begin_stage(e, s, "export_neighbours");
    k_export<2><<<EXPORT_BLOCKS, EXPORT_THREADS, 0, s>>>(device_header(lane), e->d_offsets.p, c.f0, c.f1, c.n_neighbours, nullptr, nullptr, e->d_nb.p);
    end_stage(e, s);
}

static void issue_sample(vm_engine* e, Lane& lane, const Chunk& c, cudaStream_t s) {
    const dim3 g((c.max_rows + ROW_THREADS * SAMPLE_ROWS - 1) / (ROW_THREADS * SAMPLE_ROWS), c.f1 - c.f0);
    float4* features = reinterpret_cast<float4*>(lane.d_feat[0].p);
    begin_stage(e, s, "sample_image");
    if (c.packed4) { k_sample<true><<<g, ROW_THREADS, 0, s>>>(device_frames(lane), e->d_offsets.p, c.f0, e->d_px.p, features); }
    else {
        k_sample<false><<<g, ROW_THREADS, 0, s>>>(device_frames(lane), e->d_offsets.p, c.f0, e->d_px.p, features);
    }
    end_stage(e, s);
}

static void issue_remap(vm_engine* e, Lane& lane, const Chunk& c) {
    cudaStream_t s = lane.stream;
    const dim3 g((c.max_rows + ROW_THREADS - 1) / ROW_THREADS, c.f1 - c.f0);
    const st::PlanOut plan = c.with_plan ? tile_plan(lane) : st::PlanOut{nullptr, nullptr, nullptr};
    begin_stage(e, s, "remap_neighbours");
#define VM_REMAP(NN)                                                                                                                      \
    if (c.n_neighbours == NN) {                                                                                                           \
        if (c.with_plan) k_remap<NN, true><<<g, ROW_THREADS, 0, s>>>(device_frames(lane), e->d_offsets.p, c.f0, e->d_gi.p, lane.d_node_rank.p, e->d_nb.p, plan); \
        else k_remap<NN, false><<<g, ROW_THREADS, 0, s>>>(device_frames(lane), e->d_offsets.p, c.f0, e->d_gi.p, lane.d_node_rank.p, e->d_nb.p, plan);  \
    }
    VM_REMAP(4) VM_REMAP(6) VM_REMAP(8)
#undef VM_REMAP
    end_stage(e, s);
}

// The staging block's way to the device: by a kernel where images are on their way too (k_fetch), else by a copy. A block is a few
// kilobytes, with ranges at most a few hundred: 32 thread blocks keep enough reads in flight.
constexpr int FETCH_BLOCKS = 32;

static void issue_staging(vm_engine* e, Lane& lane, const Chunk& c) {
    cudaStream_t s = lane.stream;
    if (!c.images_apart) {
        VM_CUDA(cudaMemcpyAsync(lane.d_staging.p, lane.h_staging.p, c.staging_bytes, cudaMemcpyHostToDevice, s));
        return;
    }
    const int n = static_cast<int>(c.staging_bytes / sizeof(uint4));  // whole pieces: every part of the block is aligned to 256 bytes
    begin_stage(e, s, "fetch_staging");
    k_fetch<<<std::min(FETCH_BLOCKS, (n + FETCH_THREADS - 1) / FETCH_THREADS), FETCH_THREADS, 0, s>>>(reinterpret_cast<const uint4*>(lane.h_staging.p),
                                                                                                    reinterpret_cast<uint4*>(lane.d_staging.p), n);
    end_stage(e, s);
}

// Staging block, lookup, projection, compaction, neighbour remap; images that are on the device already are sampled beside the
// remap (neither needs the other: 178 -> 140 us on 4.4 M rows).
static void issue_projection(vm_engine* e, Lane& lane, const Chunk& c, bool sample, bool remap = true) {
    cudaStream_t s            = lane.stream;
    const int nf              = c.f1 - c.f0;
    const FrameParams* frames = device_frames(lane);
    int32_t* groups           = reinterpret_cast<int32_t*>(lane.d_staging.p + c.counts_at);
    issue_staging(e, lane, c);
    if (c.device_lookup) {
        begin_stage(e, s, "bsp_state");
        k_bsp_state<<<dim3(c.bsp_blocks, nf), SELECT_THREADS, 0, s>>>(frames, lane.d_state.p);
        end_stage(e, s);
    }
    begin_stage(e, s, "select_project");
    k_select<<<dim3(c.blocks_per_frame, nf), SELECT_THREADS, 0, s>>>(frames, lane.d_state.p, lane.d_cand_px.p, lane.d_cand_node.p, lane.d_block_counts.p,
                                                                     groups, c.n_groups, e->flags);
    end_stage(e, s);
    begin_stage(e, s, "scatter_compact");
    k_scatter<SCATTER_UNITS><<<dim3((c.blocks_per_frame + SCATTER_UNITS - 1) / SCATTER_UNITS, nf), SELECT_THREADS, 0, s>>>(
      frames, device_header(lane), lane.d_cand_px.p, lane.d_cand_node.p, lane.d_block_counts.p, groups, c.blocks_per_frame, c.n_groups, e->d_offsets.p,
      c.f0, e->d_px.p, e->d_gi.p, lane.d_node_rank.p);
    end_stage(e, s);
    if (!remap) return;
    // What the scatter leaves can go to the host while the remap runs: a chunk that only projects has nothing else to overlap the bus
    // with (RING8, 1193 pixels wide, six cameras: 443 -> 427 us; with layers to overlap, the second kernel costs what it saves).
    const bool early = !c.classify && c.exported && !e->timing;
    const bool fork  = (sample && !e->timing) || early;
    if (fork) {
        VM_CUDA(cudaEventRecord(lane.ev_fork, s));
        VM_CUDA(cudaStreamWaitEvent(lane.side, lane.ev_fork, 0));
    }
    if (sample) issue_sample(e, lane, c, fork ? lane.side : s);
    if (early) issue_export_points(e, lane, c, lane.side, false);
    if (fork) VM_CUDA(cudaEventRecord(lane.ev_join, lane.side));
    issue_remap(e, lane, c);
    if (early) issue_export_neighbours(e, lane, c, s);
    if (fork) VM_CUDA(cudaStreamWaitEvent(s, lane.ev_join, 0));
}

// All layers, and the classifications to the host when they are wanted there: by the last layer itself where its kernel can (one kernel
// and one trip through memory less: thumbnail call 49 -> 47 us, 1280 x 1024 frame 243 -> 239 us, others -1 to -4 %).
static void issue_layers(vm_engine* e, Lane& lane, const Chunk& c, bool sample) {
    if (sample) issue_sample(e, lane, c, lane.stream);
    const DenseLayer& last = e->layers.back();
    const bool direct      = c.exported && ffma_stores_to_host(last) && (last.tc_np == 0 || !e->use_tc || e->tc_mode == 1) && last.cin * last.cout < e->tc_min_product;
    float* const* to_host  = reinterpret_cast<float* const*>(lane.d_staging.p + offsetof(ChunkHeader, cls));
    run_network(e, lane, c.with_plan, e->d_offsets.p, e->d_nb.p, c.n_neighbours, c.f0, c.f1 - c.f0, c.max_rows, e->d_cls.p, true, c.stride, direct ? to_host : nullptr);
    if (!c.exported || direct) return;
    begin_stage(e, lane.stream, "export_classes");
    k_export<1><<<EXPORT_BLOCKS, EXPORT_THREADS, 0, lane.stream>>>(device_header(lane), e->d_offsets.p, c.f0, c.f1, e->n_classes, nullptr, nullptr, e->d_cls.p);
    end_stage(e, lane.stream);
}

// ---- recorded graphs -------------------------------------------------------------------------------------------------

enum GraphPart { PART_ALL = 0, PART_PROJECTION = 1, PART_LAYERS = 2 };

static void forget_graphs(vm_engine* e) {
    for (auto& g : e->graphs)
        if (g.exec != nullptr) cudaGraphExecDestroy(g.exec);
    e->graphs.clear();
}

static GraphKey graph_key(const vm_engine* e, const Lane& lane, const Chunk& c, int part) {
    GraphKey k;
    std::memset(&k, 0, sizeof(k));
    k.part             = part;
    k.lane             = static_cast<int32_t>(&lane - e->lanes);
    k.n_frames         = c.f1 - c.f0;
    k.f0               = c.f0;
    k.n_neighbours     = c.n_neighbours;
    k.blocks_per_frame = c.blocks_per_frame;
    k.bsp_blocks       = c.bsp_blocks;
    k.options          = c.classify | c.exported << 1 | c.device_lookup << 2 | c.packed4 << 3 | c.with_plan << 4 | c.images_apart << 5 | int(e->use_tc) << 6 | c.copied << 7;
    k.wait_limit       = e->tc_wait_limit;
    k.feature_stride   = c.stride;
    k.staging_bytes    = c.staging_bytes;
    k.counts_at        = c.counts_at;
    return k;
}

// Enqueues what `issue` enqueues on the lane's stream. A chunk of this shape that comes back is recorded as a CUDA graph and from
// then on costs one launch: on a B200's host of 16 cores a launch takes 2.7 to 3.8 us of host time, so that 8 small kernels and a wait take
// 32 us one by one and 11 us as a graph, 16 kernels 49 and 15 us. The first time nothing is recorded: recording and instantiating
// costs more than it saves on a shape that may never return.
template <typename Issue>
static void run_part(vm_engine* e, Lane& lane, const Chunk& c, int part, Issue issue) {
    if (!e->use_graphs || e->timing || e->nvtx) {
        issue();
        return;
    }
    const GraphKey key = graph_key(e, lane, c, part);
    GraphEntry* entry  = nullptr;
    for (auto& g : e->graphs)
        if (std::memcmp(&g.key, &key, sizeof(key)) == 0) entry = &g;
    if (entry == nullptr || entry->refused) {
        if (entry == nullptr) {
            if (e->graphs.size() >= MAX_GRAPHS) {
                auto oldest = std::min_element(e->graphs.begin(), e->graphs.end(), [](const GraphEntry& a, const GraphEntry& b) { return a.last_use < b.last_use; });
                if (oldest->exec != nullptr) {
                    // it may still be running on its lane
                    VM_CUDA(cudaStreamSynchronize(e->lanes[oldest->key.lane].stream));
                    cudaGraphExecDestroy(oldest->exec);
                }
                e->graphs.erase(oldest);
            }
            GraphEntry fresh;
            fresh.key      = key;
            fresh.last_use = ++e->graph_uses;
            e->graphs.push_back(fresh);
        }
        issue();
        return;
    }
    entry->last_use = ++e->graph_uses;
    if (entry->exec == nullptr) {
        const int64_t before = e->launches;
        cudaGraph_t graph    = nullptr;
        VM_CUDA(cudaStreamBeginCapture(lane.stream, cudaStreamCaptureModeThreadLocal));
        bool recorded = true;
        try {
            issue();
        }
        catch (...) {  // the recording must end whatever happened; launched one by one below, it happens again or does not
            recorded = false;
        }
        recorded         = cudaStreamEndCapture(lane.stream, &graph) == cudaSuccess && recorded;
        entry->kernels   = e->launches - before;
        e->launches      = before;
        recorded         = recorded && cudaGraphInstantiate(&entry->exec, graph, 0) == cudaSuccess;
        if (graph != nullptr) cudaGraphDestroy(graph);
        if (!recorded) {
            cudaGetLastError();
            entry->exec    = nullptr;
            entry->refused = true;
            issue();
            return;
        }
    }
    VM_CUDA(cudaGraphLaunch(entry->exec, lane.stream));
    e->launches += entry->kernels;
}

// ---- one batch -------------------------------------------------------------------------------------------------------

// Enqueues a whole chunk except for results that are copied once their number is known; nothing here waits for the device.
static Chunk enqueue_chunk(vm_engine* e, Lane& lane, Lane* prev, bool after_prev, const vm_frame* frames, int f0, int f1, bool classify, bool to_host,
                           bool only_chunk, const ImagePlan& images, Upload* upload) {
    const Chunk c = stage_chunk(e, lane, frames, f0, f1, classify, to_host, only_chunk, images);
    if (upload != nullptr) upload->pump();
    if (e->buffers_moved) {
        // graphs of other lanes may be running: they stay valid until they have finished
        for (auto& l : e->lanes)
            if (l.busy) VM_CUDA(cudaStreamSynchronize(l.stream));
        forget_graphs(e);
        e->buffers_moved = false;
    }
    // this chunk's offsets continue those of the one before
    if (prev != nullptr && prev != &lane) VM_CUDA(cudaStreamWaitEvent(lane.stream, after_prev ? prev->ev_done : prev->ev_offsets, 0));
    lane.busy = true;
    if (only_chunk && !c.images_apart && !c.copied) {
        // everything as one graph, the results of the projection on their way to the host beside the layers
        run_part(e, lane, c, PART_ALL, [&] {
            issue_projection(e, lane, c, classify);
            const bool fork = c.exported && classify && !e->timing;
            if (fork) {
                VM_CUDA(cudaEventRecord(lane.ev_fork, lane.stream));
                VM_CUDA(cudaStreamWaitEvent(lane.side, lane.ev_fork, 0));
            }
            if (c.exported && (classify || e->timing)) issue_export_points(e, lane, c, fork ? lane.side : lane.stream, true);
            if (fork) VM_CUDA(cudaEventRecord(lane.ev_join, lane.side));
            if (classify) issue_layers(e, lane, c, false);
            if (fork) VM_CUDA(cudaStreamWaitEvent(lane.stream, lane.ev_join, 0));
        });
    }
    else {
        // results that are copied once their number is known, and no layers beside which to copy them: the copies begin before the remap
        // (six cameras of 1280 x 1024, 14 MB: 338 -> 332 us)
        const bool split = !classify && c.copied;
        run_part(e, lane, c, PART_PROJECTION, [&] { issue_projection(e, lane, c, classify && !c.images_apart, !split); });
        VM_CUDA(cudaEventRecord(lane.ev_offsets, lane.stream));
        if (split) issue_remap(e, lane, c);
        VM_CUDA(cudaEventRecord(lane.ev_projected, lane.stream));
        if (c.exported) {
            cudaStream_t beside = e->timing ? lane.stream : lane.side;
            VM_CUDA(cudaStreamWaitEvent(beside, lane.ev_offsets, 0));
            issue_export_points(e, lane, c, beside, true);
            VM_CUDA(cudaEventRecord(lane.ev_join, beside));
        }
        if (upload != nullptr) upload->finish();
        if (c.images_apart) {
            VM_CUDA(cudaEventRecord(lane.ev_images, e->copy_stream));
            VM_CUDA(cudaStreamWaitEvent(lane.stream, lane.ev_images, 0));
        }
        if (classify) run_part(e, lane, c, PART_LAYERS, [&] { issue_layers(e, lane, c, c.images_apart); });
        if (c.exported) VM_CUDA(cudaStreamWaitEvent(lane.stream, lane.ev_join, 0));
    }
    VM_CUDA(cudaEventRecord(lane.ev_done, lane.stream));
    return c;
}

// Copies a chunk's results to the host; waits for its offsets first. The projection's results leave while its layers run.
static void copy_results(vm_engine* e, Lane& lane, const Chunk& c) {
    if (!c.copied) return;
    VM_CUDA(cudaEventSynchronize(lane.ev_offsets));
    Results& to = *e->host;
    const int32_t* off = to.offsets.p;
    const size_t p0 = off[c.f0], p1 = off[c.f1];
    const size_t r0 = p0 + c.f0, r1 = p1 + c.f1;
    const size_t N = c.n_neighbours, C = e->n_classes;
    cudaStream_t beside = e->timing ? lane.stream : lane.side;
    VM_CUDA(cudaStreamWaitEvent(beside, lane.ev_offsets, 0));
    if (p1 > p0) {
        VM_CUDA(cudaMemcpyAsync(to.px.p + p0, e->d_px.p + p0, sizeof(float2) * (p1 - p0), cudaMemcpyDeviceToHost, beside));
        VM_CUDA(cudaMemcpyAsync(to.gi.p + p0, e->d_gi.p + p0, sizeof(int32_t) * (p1 - p0), cudaMemcpyDeviceToHost, beside));
    }
    VM_CUDA(cudaStreamWaitEvent(beside, lane.ev_projected, 0));
    VM_CUDA(cudaMemcpyAsync(to.nb.p + r0 * N, e->d_nb.p + r0 * N, sizeof(int32_t) * (r1 - r0) * N, cudaMemcpyDeviceToHost, beside));
    if (c.classify) VM_CUDA(cudaMemcpyAsync(to.cls.p + r0 * C, e->d_cls.p + r0 * C, sizeof(float) * (r1 - r0) * C, cudaMemcpyDeviceToHost, lane.stream));
    if (beside != lane.stream) {
        VM_CUDA(cudaEventRecord(lane.ev_join, beside));
        VM_CUDA(cudaStreamWaitEvent(lane.stream, lane.ev_join, 0));
    }
    VM_CUDA(cudaEventRecord(lane.ev_done, lane.stream));
}

static vm_status run_batch(vm_engine* e, const vm_frame* frames, int32_t n_frames, uint32_t flags, vm_batch_result* out) {
    if (e == nullptr || out == nullptr || n_frames < 0 || (n_frames > 0 && frames == nullptr)) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null engine, frames or result");
    }
    std::memset(out, 0, sizeof(*out));
    if (n_frames == 0) return VM_OK;
    struct BatchRange {  // one NVTX range per batch, closed on every way out
        bool on;
        explicit BatchRange(bool enabled) : on(enabled) {
            if (on) nvtxRangePushA("vm_run_batch");
        }
        ~BatchRange() {
            if (on) nvtxRangePop();
        }
    } batch_range(e->nvtx);

    // validation, before any device work - the reference throws from inside the call for the same conditions
    bool classify = frames[0].image != nullptr && !e->layers.empty();
    const int N   = frames[0].mesh != nullptr ? frames[0].mesh->n_neighbours : 0;
    int64_t cand_all = 0;
    for (int f = 0; f < n_frames; ++f) {
        const vm_frame& fr = frames[f];
        if (fr.mesh == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "frame without a mesh");
        if (fr.mesh->owner != e) return fail(VM_ERR_INVALID_ARGUMENT, "mesh was uploaded through another engine");
        if (fr.mesh->n_neighbours != N) return fail(VM_ERR_INVALID_ARGUMENT, "frames of one batch must share n_neighbours");
        if (fr.lens.projection != VM_RECTILINEAR && fr.lens.projection != VM_EQUISOLID && fr.lens.projection != VM_EQUIDISTANT) {
            return fail(VM_ERR_UNSUPPORTED_LENS, "Cannot project: Unknown lens type");
        }
        if (fr.lens.dimensions[0] <= 0 || fr.lens.dimensions[1] <= 0) return fail(VM_ERR_INVALID_ARGUMENT, "lens dimensions must be positive");
        if (fr.ranges == nullptr && fr.n_ranges != 0) return fail(VM_ERR_INVALID_ARGUMENT, "n_ranges without ranges");
        if (fr.ranges == nullptr && fr.mesh->n_bsp == 0) return fail(VM_ERR_NO_BSP, "device lookup needs vm_mesh_set_bsp");
        if (fr.n_ranges < 0) return fail(VM_ERR_INVALID_ARGUMENT, "negative n_ranges");
        for (int r = 0; r < fr.n_ranges; ++r) {
            if (fr.ranges[2 * r] < 0 || fr.ranges[2 * r + 1] > fr.mesh->n_nodes || fr.ranges[2 * r] > fr.ranges[2 * r + 1]) {
                return fail(VM_ERR_INVALID_ARGUMENT, "range outside the mesh");
            }
        }
        if ((fr.image != nullptr) != (frames[0].image != nullptr)) return fail(VM_ERR_INVALID_ARGUMENT, "either all frames carry an image or none");
        if (classify && format_class(fr.format) == FMT_UNKNOWN) {
            char code[5] = {char(fr.format & 0xFF), char(fr.format >> 8 & 0xFF), char(fr.format >> 16 & 0xFF), char(fr.format >> 24 & 0xFF), 0};
            return fail(VM_ERR_UNSUPPORTED_FORMAT, std::string("Unsupported image format ") + code);
        }
        cand_all += frame_candidates(fr);
    }
    if (classify && e->layers.front().cin != 4) return fail(VM_ERR_NETWORK_SHAPE, "first layer must take 4 channels");
    if (classify && e->layers.front().n_slots != N + 1) return fail(VM_ERR_NETWORK_SHAPE, "network was built for a different n_neighbours");
    if (cand_all + n_frames > (int64_t(1) << 31) - 1024) return fail(VM_ERR_INVALID_ARGUMENT, "batch too large: split it");

    auto drain = [&] {
        for (auto& lane : e->lanes) {
            if (lane.stream != nullptr) cudaStreamSynchronize(lane.stream);
            if (lane.side != nullptr) cudaStreamSynchronize(lane.side);
            lane.busy = false;
        }
        if (e->copy_stream != nullptr) cudaStreamSynchronize(e->copy_stream);
    };
    try {
        VM_CUDA(cudaSetDevice(e->device));
        e->timing = (flags & VM_TIME_STAGES) != 0;
        e->timers.clear();
        e->events_used = 0;
        e->stage_ms.clear();
        const bool to_host = (flags & VM_RESULTS_ON_DEVICE) == 0;
        const int n_lanes  = e->timing ? 1 : e->n_lanes;  // with the stages timed, one chunk after another

        ImagePlan images;
        std::unique_ptr<Upload> upload;

        const size_t rows_all = static_cast<size_t>(cand_all) + n_frames;
        need(e, e->d_offsets, n_frames + 1);
        need(e, e->d_px, cand_all + 1);
        need(e, e->d_gi, cand_all + 1);
        need(e, e->d_nb, rows_all * N);
        if (classify) need(e, e->d_cls, rows_all * e->n_classes);
        if (!e->host) {
            std::lock_guard<std::mutex> lock(e->pool->mutex);
            if (!e->pool->free.empty()) {
                e->host = std::move(e->pool->free.back());
                e->pool->free.pop_back();
            }
        }
        if (!e->host) e->host.reset(new Results());
        e->host->offsets.ensure(n_frames + 1);
        if (to_host) {
            e->host->px.ensure(cand_all + 1);
            e->host->gi.ensure(cand_all + 1);
            e->host->nb.ensure(rows_all * N);
            if (classify) e->host->cls.ensure(rows_all * e->n_classes);
        }
        for (int i = 0; i < ABORT_FLAGS; ++i) e->flags[i] = 0;

        // Chunks: runs of frames bounded by a candidate budget, a frame count and the bytes of their host images. Small ones let the
        // copies of one chunk overlap the kernels of another: 20 MB are 0.4 ms of the bus (32 frames of 5 MB to results on the
        // host: 3.87 ms in chunks of 16 frames, 3.56 in chunks of 8, 3.50 in chunks of 4, 3.60 in chunks of 2; both directions' bytes
        // alone take 3.45. Two engines with 32 frames each: 6.60, 6.59, 6.78 ms in chunks of 16, 8 and 4; the bytes alone 6.67). When no
        // images are to be copied in, a batch is one chunk as far as the scratch allows, and
        // chunks follow one another: fewer and fuller launches (64 frames of 1280 x 1024 pixels in one chunk: 1.61 ms, in two that
        // overlap 1.99, in eight 2.06 - persistent layer kernels of two chunks get in one another's way).
        bool host_images = false;
        for (int f = 0; f < n_frames; ++f) host_images = host_images || (classify && !frames[f].image_on_device);
        const bool small_chunks = e->chunk_override || host_images;
        const int64_t max_chunk_candidates = small_chunks ? e->chunk_candidates : 8 * e->chunk_candidates;
        const int max_chunk_frames         = small_chunks ? e->chunk_frames : TC_MAX_FRAMES;
        int f0 = 0, chunk = 0;
        Lane* prev = nullptr;
        Chunk last;
        while (f0 < n_frames) {
            int f1 = f0;
            int64_t c = 0, nodes = 0, elements = 0;
            size_t bytes = 0;
            while (f1 < n_frames) {
                const int64_t more          = frame_candidates(frames[f1]);
                const int64_t more_nodes    = frames[f1].mesh->n_nodes;
                const int64_t more_elements = frames[f1].ranges == nullptr ? frames[f1].mesh->n_bsp : 0;
                const size_t more_bytes     = classify && !frames[f1].image_on_device ? image_bytes(frames[f1]) : 0;
                if (f1 > f0 && (nodes + more_nodes > MAX_CHUNK_NODES || elements + more_elements > MAX_CHUNK_NODES)) break;
                if (f1 > f0 && (c + more > max_chunk_candidates || f1 - f0 >= max_chunk_frames || (bytes + more_bytes > CHUNK_IMAGE_BYTES && !e->chunk_override))) break;
                c += more;
                nodes += more_nodes;
                elements += more_elements;
                bytes += more_bytes;
                ++f1;
            }
            Lane& lane = e->lanes[chunk % n_lanes];
            lane.open(e->blocking_sync);
            if (lane.busy) {
                // its previous chunk must have left the lane's staging and scratch
                VM_CUDA(cudaEventSynchronize(lane.ev_done));
                lane.busy = false;
            }
            if (classify) {
                images = plan_images(frames, f0, f1);
                upload.reset();
                if (images.total > 0 && !images.small) upload = start_images(e, lane, frames, f0, f1, images);
            }
            const Chunk current = enqueue_chunk(e, lane, prev, !host_images, frames, f0, f1, classify, to_host, f0 == 0 && f1 == n_frames, images, upload.get());
            // while this chunk runs, fetch the results of the one before it
            if (n_lanes == 1) { copy_results(e, lane, current); }
            else if (prev != nullptr) {
                copy_results(e, *prev, last);
            }
            prev = &lane;
            last = current;
            f0   = f1;
            ++chunk;
        }
        if (n_lanes > 1) copy_results(e, *prev, last);
        for (auto& lane : e->lanes) {
            if (lane.busy) VM_CUDA(cudaEventSynchronize(lane.ev_done));
            lane.busy = false;
        }
        // read once, after the last kernel of EVERY lane
        if (e->flags[ABORT_TC_TIMEOUT]) return fail(VM_ERR_DEVICE_ABORT, "a tensor-core kernel gave up waiting on an mbarrier");
        if (e->flags[ABORT_BSP_DEPTH]) return fail(VM_ERR_DEVICE_ABORT, "a kernel gave up on a bounded loop (BSP deeper than 128 levels)");
        if (e->flags[ABORT_TC_RANGE] && e->use_tc) {
            // a feature value beyond the range of the fp16 split: this engine goes back to the FFMA kernels for good and
            // the batch is computed again
            e->use_tc = false;
            return run_batch(e, frames, n_frames, flags, out);
        }

        if (e->timing) {
            for (const auto& t : e->timers) {
                float ms = 0.0f;
                VM_CUDA(cudaEventElapsedTime(&ms, t.start, t.stop));
                e->stage_ms.emplace_back(t.name, ms);
            }
        }

        out->n_frames     = n_frames;
        out->n_neighbours = N;
        out->n_classes    = classify ? e->n_classes : 0;
        out->on_device    = to_host ? 0 : 1;
        out->offsets      = e->host->offsets.p;
        if (to_host) {
            out->pixel_coordinates = reinterpret_cast<const float*>(e->host->px.p);
            out->global_indices    = e->host->gi.p;
            out->neighbourhood     = e->host->nb.p;
            out->classifications   = classify ? e->host->cls.p : nullptr;
        }
        else {
            out->pixel_coordinates = reinterpret_cast<const float*>(e->d_px.p);
            out->global_indices    = e->d_gi.p;
            out->neighbourhood     = e->d_nb.p;
            out->classifications   = classify ? e->d_cls.p : nullptr;
        }
        return VM_OK;
    }
    catch (...) {
        drain();
        return status_of_exception();
    }
}

}  // namespace vm

using namespace vm;

extern "C" {

const char* vm_last_error(void) {
    return g_error.c_str();
}

// lets the host mesh translation unit report through the same per-thread message
void vm_set_last_error_(const char* message) {
    g_error = message != nullptr ? message : "";
}

vm_status vm_engine_create(int device, const vm_layer* layers, const int32_t* layers_per_group, int32_t n_groups, vm_engine** out) {
    if (out == nullptr || n_groups < 0 || (n_groups > 0 && (layers == nullptr || layers_per_group == nullptr))) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    }
    *out = nullptr;
    // shape check: cpp/visualmesh/engine/cpu/engine.hpp:213-256 multiplies whatever it is given; a mismatch there is
    // undefined behaviour, here it is an error
    {
        int l = 0, width = 4, slots_first = 0;
        for (int g = 0; g < n_groups; ++g) {
            if (layers_per_group[g] <= 0) return fail(VM_ERR_NETWORK_SHAPE, "a group needs at least one layer");
            for (int i = 0; i < layers_per_group[g]; ++i, ++l) {
                const vm_layer& L = layers[l];
                if (L.weights == nullptr || L.biases == nullptr || L.n_in <= 0 || L.n_out <= 0) return fail(VM_ERR_NETWORK_SHAPE, "empty layer");
                if (L.activation < VM_SELU || L.activation > VM_TANH) return fail(VM_ERR_NETWORK_SHAPE, "unknown activation");
                if (i == 0) {
                    if (L.n_in % width != 0) return fail(VM_ERR_NETWORK_SHAPE, "gather layer rows must be (N+1) x previous width");
                    const int slots = L.n_in / width;
                    if (slots != 5 && slots != 7 && slots != 9) return fail(VM_ERR_NETWORK_SHAPE, "gather layer rows must be (N+1) x previous width, N in {4,6,8}");
                    if (slots_first == 0) slots_first = slots;
                    if (slots != slots_first) return fail(VM_ERR_NETWORK_SHAPE, "all groups must gather the same number of neighbours");
                }
                else if (L.n_in != width) {
                    return fail(VM_ERR_NETWORK_SHAPE, "dense layer rows must equal the previous width");
                }
                width = L.n_out;
            }
        }
    }
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return fail(VM_ERR_CUDA, "no CUDA device: this engine has no CPU fallback");
    }
    std::unique_ptr<vm_engine> e;
    try {
        e.reset(new vm_engine());
        if (device < 0) VM_CUDA(cudaGetDevice(&device));
        if (device >= count) return fail(VM_ERR_INVALID_ARGUMENT, "no such device");
        e->device = device;
        VM_CUDA(cudaSetDevice(device));
        if (const char* v = std::getenv("VMCUDA_CHUNK_FRAMES")) {
            e->chunk_frames   = std::max(1, std::atoi(v));
            e->chunk_override = true;
        }
        if (const char* v = std::getenv("VMCUDA_CHUNK_CANDIDATES")) {
            e->chunk_candidates = std::max<long long>(1, std::atoll(v));
            e->chunk_override   = true;
        }
        if (const char* v = std::getenv("VMCUDA_TC")) {
            e->tc_mode = std::atoi(v);
            e->use_tc  = e->tc_mode != 0;
        }
        if (const char* v = std::getenv("VMCUDA_TC_MIN_PRODUCT")) e->tc_min_product = std::atoi(v);
        if (const char* v = std::getenv("VMCUDA_TC_NO_SPLIT")) e->tc_no_split = std::atoi(v) != 0;
        if (const char* v = std::getenv("VMCUDA_STAGED")) e->staged = std::atoi(v) != 0;
        if (const char* v = std::getenv("VMCUDA_BLOCKING_SYNC")) e->blocking_sync = std::atoi(v) != 0;
        if (const char* v = std::getenv("VMCUDA_NVTX")) e->nvtx = std::atoi(v) != 0;
        if (const char* v = std::getenv("VMCUDA_GRAPHS")) e->use_graphs = std::atoi(v) != 0;
        if (const char* v = std::getenv("VMCUDA_LANES")) e->n_lanes = std::min(MAX_LANES, std::max(1, std::atoi(v)));
        e->lanes[0].open(e->blocking_sync);  // the others, and the stream of the images, when they are first used
        VM_CUDA(cudaEventCreate(&e->ev_timer_start));
        VM_CUDA(cudaEventCreate(&e->ev_timer_stop));
        VM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&e->flags), sizeof(int32_t) * ABORT_FLAGS, cudaHostAllocDefault));
        for (int i = 0; i < ABORT_FLAGS; ++i) e->flags[i] = 0;
        int l = 0;
        int logical = 4, width = 4;  // channels of the layer before, as the network has them and as they are stored
        for (int g = 0; g < n_groups; ++g) {
            for (int i = 0; i < layers_per_group[g]; ++i, ++l) {
                const vm_layer& given = layers[l];
                DenseLayer d;
                d.n_slots    = i == 0 ? given.n_in / logical : 1;
                d.cin        = width;
                d.activation = given.activation;
                d.stage      = std::string(i == 0 ? "graph_conv_" : "dense_") + std::to_string(logical) + "x" + std::to_string(given.n_out);
                // Features of a width that is no multiple of 4 are stored with channels of zeros up to the next one: the kernels with
                // 16-byte loads then serve every width. (Every activation but softmax maps 0 to 0; weights of the zeros are zeros.)
                const bool last = g + 1 == n_groups && i + 1 == layers_per_group[g];
                d.cout  = last || given.activation == VM_SOFTMAX ? given.n_out : (given.n_out + 3) & ~3;
                d.coutp = (d.cout + 3) & ~3;
                vm_layer L = given;
                std::vector<float> padded_weights, padded_biases;
                if (width != logical || d.cout != given.n_out) {
                    L.n_in  = d.n_slots * width;
                    L.n_out = d.cout;
                    padded_weights.assign(static_cast<size_t>(L.n_in) * L.n_out, 0.0f);
                    padded_biases.assign(L.n_out, 0.0f);
                    for (int r = 0; r < given.n_in; ++r) {
                        std::memcpy(&padded_weights[(static_cast<size_t>(r / logical) * width + r % logical) * L.n_out],
                                    given.weights + static_cast<size_t>(r) * given.n_out, sizeof(float) * given.n_out);
                    }
                    std::memcpy(padded_biases.data(), given.biases, sizeof(float) * given.n_out);
                    L.weights = padded_weights.data();
                    L.biases  = padded_biases.data();
                }
                // [n_in][n_out] as handed over (cpp/visualmesh/network_structure.hpp:25-27), padded to coutp columns
                std::vector<float> packed((static_cast<size_t>(L.n_in) + 1) * d.coutp, 0.0f);
                for (int r = 0; r < L.n_in; ++r)
                    for (int c = 0; c < L.n_out; ++c) packed[static_cast<size_t>(r) * d.coutp + c] = L.weights[static_cast<size_t>(r) * L.n_out + c];
                for (int c = 0; c < L.n_out; ++c) packed[static_cast<size_t>(L.n_in) * d.coutp + c] = L.biases[c];
                VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&d.d_weights), packed.size() * sizeof(float)));
                VM_CUDA(cudaMemcpy(d.d_weights, packed.data(), packed.size() * sizeof(float), cudaMemcpyHostToDevice));
                d.host_packed = packed;
                // tensor-core copy of the weights: per 16-byte K chunk, NP rows of hi parts then NP rows of lo parts
                if ((width == 8 || width == 16 || width == 32) && L.n_out <= 32 && i == 0) {
                    const int np    = L.n_out <= 16 ? 16 : 32;
                    const int K     = L.n_in;
                    const bool half = width != 8;
                    const int kch   = half ? 8 : 4;
                    float w_max     = 0.0f;
                    for (size_t q = 0; q < size_t(K) * L.n_out; ++q) w_max = std::max(w_max, std::fabs(L.weights[q]));
                    const size_t smem_need = 256 + size_t(9) * 2 * (width / kch) * 128 * 16 + size_t(K / kch) * 2 * np * 16;
                    if (smem_need <= 200 * 1024 && (!half || w_max < 60000.0f)) {
                        const size_t chunks = size_t(K / kch);
                        std::vector<unsigned char> cat(chunks * 2 * np * 16, 0);
                        std::vector<float> bias(np, 0.0f);
                        for (int k = 0; k < K; ++k) {
                            for (int n = 0; n < L.n_out; ++n) {
                                const float w     = L.weights[size_t(k) * L.n_out + n];
                                const size_t base = size_t(k / kch) * 2 * np * 16;
                                if (half) {
                                    const __half h = __float2half_rn(w);
                                    const __half l = __float2half_rn(w - __half2float(h));
                                    std::memcpy(&cat[base + size_t(n) * 16 + (k % kch) * 2], &h, 2);
                                    std::memcpy(&cat[base + size_t(np + n) * 16 + (k % kch) * 2], &l, 2);
                                }
                                else {
                                    uint32_t bits;
                                    std::memcpy(&bits, &w, sizeof(bits));
                                    bits &= 0xFFFFE000u;
                                    float h;
                                    std::memcpy(&h, &bits, sizeof(h));
                                    const float l = w - h;
                                    std::memcpy(&cat[base + size_t(n) * 16 + (k % kch) * 4], &h, 4);
                                    std::memcpy(&cat[base + size_t(np + n) * 16 + (k % kch) * 4], &l, 4);
                                }
                            }
                        }
                        for (int n = 0; n < L.n_out; ++n) bias[n] = L.biases[n];
                        VM_CUDA(cudaMalloc(&d.d_tc_cat, cat.size()));
                        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&d.d_tc_bias), bias.size() * sizeof(float)));
                        VM_CUDA(cudaMemcpy(d.d_tc_cat, cat.data(), cat.size(), cudaMemcpyHostToDevice));
                        VM_CUDA(cudaMemcpy(d.d_tc_bias, bias.data(), bias.size() * sizeof(float), cudaMemcpyHostToDevice));
                        if (half && width == 32) {
                            const std::vector<unsigned char> win = pack_window_weights(L.weights, d.n_slots, L.n_out);
                            VM_CUDA(cudaMalloc(&d.d_tc_win, win.size()));
                            VM_CUDA(cudaMemcpy(d.d_tc_win, win.data(), win.size(), cudaMemcpyHostToDevice));
                        }
                        d.tc_np   = np;
                        d.tc_half = half;
                    }
                }
                e->layers.push_back(d);
                width        = L.n_out;
                logical      = given.n_out;
                e->max_width = std::max(e->max_width, width);
            }
        }
        e->n_classes = e->layers.empty() ? 0 : e->layers.back().cout;
        for (size_t l = 1; l < e->layers.size(); ++l) {
            const DenseLayer& L = e->layers[l];
            e->may_stage        = e->may_stage || (l + 1 < e->layers.size() && has_staged_kernel(L));
            e->may_stage        = e->may_stage || (has_window_kernel(L) && (e->tc_mode != 1 || L.cin * L.cout >= e->tc_min_product));
        }
    }
    catch (...) {
        return status_of_exception();
    }
    *out = e.release();
    return VM_OK;
}

static void free_mesh(vm_mesh* m) {
    if (m == nullptr) return;
    cudaFree(m->d_rays);
    cudaFree(m->d_neighbours);
    cudaFree(m->d_cones_a);
    cudaFree(m->d_cones_s);
    cudaFree(m->d_topology);
    delete m;
}

void vm_engine_destroy(vm_engine* e) {
    if (e == nullptr) return;
    cudaSetDevice(e->device);
    cudaDeviceSynchronize();
    for (auto* m : e->meshes) free_mesh(m);
    for (auto& L : e->layers) {
        cudaFree(L.d_weights);
        cudaFree(L.d_tc_cat);
        cudaFree(L.d_tc_win);
        cudaFree(L.d_tc_bias);
    }
    forget_graphs(e);
    for (auto& lane : e->lanes) {
        lane.h_staging.release();
        lane.d_staging.release();
        lane.d_state.release();
        lane.d_cand_px.release();
        lane.d_cand_node.release();
        lane.d_block_counts.release();
        lane.d_node_rank.release();
        lane.d_feat[0].release();
        lane.d_feat[1].release();
        lane.d_images.release();
        lane.h_images.release();
        lane.d_nbl.release();
        lane.d_halo_rows.release();
        lane.d_halo_count.release();
        if (lane.stream) cudaStreamDestroy(lane.stream);
        if (lane.side) cudaStreamDestroy(lane.side);
        for (cudaEvent_t ev : {lane.ev_fork, lane.ev_join, lane.ev_offsets, lane.ev_projected, lane.ev_images, lane.ev_done})
            if (ev) cudaEventDestroy(ev);
    }
    if (e->copy_stream) cudaStreamDestroy(e->copy_stream);
    e->d_offsets.release();
    e->d_px.release();
    e->d_gi.release();
    e->d_nb.release();
    e->d_cls.release();
    {
        std::lock_guard<std::mutex> lock(e->pool->mutex);
        e->pool->closed = true;
        e->pool->free.clear();
    }
    for (auto ev : e->event_pool) cudaEventDestroy(ev);
    if (e->ev_timer_start) cudaEventDestroy(e->ev_timer_start);
    if (e->ev_timer_stop) cudaEventDestroy(e->ev_timer_stop);
    cudaFreeHost(e->flags);
    delete e;
}

vm_status vm_mesh_upload(vm_engine* e, const float* rays, const int32_t* neighbours, int32_t n_nodes, int32_t n_neighbours, vm_mesh** out) {
    if (e == nullptr || rays == nullptr || neighbours == nullptr || out == nullptr || n_nodes <= 0) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument or empty mesh");
    }
    if (n_neighbours != 4 && n_neighbours != 6 && n_neighbours != 8) return fail(VM_ERR_INVALID_ARGUMENT, "n_neighbours must be 4, 6 or 8");
    *out = nullptr;
    std::unique_ptr<vm_mesh> m;
    try {
        m.reset(new vm_mesh());
        VM_CUDA(cudaSetDevice(e->device));
        m->owner        = e;
        m->n_nodes      = n_nodes;
        m->n_neighbours = n_neighbours;
        // rays padded to float4 as the OpenCL engine does (cpp/visualmesh/engine/opencl/engine.hpp:611-615)
        std::vector<float4> padded(n_nodes);
        for (int i = 0; i < n_nodes; ++i) padded[i] = make_float4(rays[3 * i], rays[3 * i + 1], rays[3 * i + 2], 0.0f);
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_rays), sizeof(float4) * n_nodes));
        VM_CUDA(cudaMemcpy(m->d_rays, padded.data(), sizeof(float4) * n_nodes, cudaMemcpyHostToDevice));
        const size_t nb_bytes = sizeof(int32_t) * static_cast<size_t>(n_nodes) * n_neighbours;
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_neighbours), nb_bytes));
        VM_CUDA(cudaMemcpy(m->d_neighbours, neighbours, nb_bytes, cudaMemcpyHostToDevice));
        e->meshes.push_back(m.get());
    }
    catch (...) {
        free_mesh(m.release());
        return status_of_exception();
    }
    *out = m.release();
    return VM_OK;
}

vm_status vm_mesh_set_bsp(vm_engine* e, vm_mesh* m, int32_t n, const int32_t* ranges, const int32_t* children, const float* cones) {
    if (e == nullptr || m == nullptr || n <= 0 || ranges == nullptr || children == nullptr || cones == nullptr) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument or empty BSP");
    }
    try {
        std::vector<float4> a(n);
        std::vector<float> s(n);
        std::vector<int4> t(n);
        for (int i = 0; i < n; ++i) {
            a[i] = make_float4(cones[5 * i], cones[5 * i + 1], cones[5 * i + 2], cones[5 * i + 3]);
            s[i] = cones[5 * i + 4];
            const int c0 = children[2 * i], c1 = children[2 * i + 1];
            if (c0 >= n || c1 >= n || (c0 < 0) != (c1 < 0)) return fail(VM_ERR_INVALID_ARGUMENT, "BSP child out of range");
            if (ranges[2 * i] < 0 || ranges[2 * i + 1] > m->n_nodes) return fail(VM_ERR_INVALID_ARGUMENT, "BSP range outside the mesh");
            t[i] = make_int4(c0, c1, c1 >= 0 ? ranges[2 * c1] : 0, 0);
        }
        VM_CUDA(cudaSetDevice(e->device));
        cudaFree(m->d_cones_a);
        cudaFree(m->d_cones_s);
        cudaFree(m->d_topology);
        m->d_cones_a = nullptr;
        m->d_cones_s = nullptr;
        m->d_topology = nullptr;
        m->n_bsp = 0;
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_cones_a), sizeof(float4) * n));
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_cones_s), sizeof(float) * n));
        VM_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_topology), sizeof(int4) * n));
        VM_CUDA(cudaMemcpy(m->d_cones_a, a.data(), sizeof(float4) * n, cudaMemcpyHostToDevice));
        VM_CUDA(cudaMemcpy(m->d_cones_s, s.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
        VM_CUDA(cudaMemcpy(m->d_topology, t.data(), sizeof(int4) * n, cudaMemcpyHostToDevice));
        m->n_bsp = n;
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

void vm_mesh_release(vm_engine* e, vm_mesh* m) {
    if (e == nullptr || m == nullptr) return;
    cudaSetDevice(e->device);
    cudaDeviceSynchronize();
    e->meshes.erase(std::remove(e->meshes.begin(), e->meshes.end(), m), e->meshes.end());
    free_mesh(m);
}

vm_status vm_run_batch(vm_engine* e, const vm_frame* frames, int32_t n_frames, uint32_t flags, vm_batch_result* out) {
    return run_batch(e, frames, n_frames, flags, out);
}

vm_status vm_project(vm_engine* e, const vm_mesh* mesh, const int32_t* ranges, int32_t n_ranges, const float Hoc[16], const vm_lens* lens, vm_batch_result* out) {
    if (Hoc == nullptr || lens == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null Hoc or lens");
    vm_frame fr{};
    fr.mesh     = mesh;
    fr.ranges   = ranges;
    fr.n_ranges = n_ranges;
    std::memcpy(fr.Hoc, Hoc, sizeof(fr.Hoc));
    fr.lens = *lens;
    return run_batch(e, &fr, 1, 0, out);
}

vm_status vm_classify(vm_engine* e, const vm_mesh* mesh, const int32_t* ranges, int32_t n_ranges, const float Hoc[16], const vm_lens* lens, const void* image, uint32_t format, vm_batch_result* out) {
    if (Hoc == nullptr || lens == nullptr || image == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null Hoc, lens or image");
    if (e != nullptr && e->layers.empty()) return fail(VM_ERR_NETWORK_SHAPE, "this engine was created without a network");
    vm_frame fr{};
    fr.mesh     = mesh;
    fr.ranges   = ranges;
    fr.n_ranges = n_ranges;
    std::memcpy(fr.Hoc, Hoc, sizeof(fr.Hoc));
    fr.lens   = *lens;
    fr.image  = image;
    fr.format = format;
    return run_batch(e, &fr, 1, 0, out);
}

vm_status vm_call(vm_engine* e, const vm_mesh* mesh, const vm_hostmesh* lookup, const float Hoc[16], const vm_lens* lens, const void* image, uint32_t format, vm_batch_result* out) {
    if (lookup == nullptr || mesh == nullptr || Hoc == nullptr || lens == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null mesh, Hoc or lens");
    if (image != nullptr && e != nullptr && e->layers.empty()) return fail(VM_ERR_NETWORK_SHAPE, "this engine was created without a network");
    if (vm_hostmesh_n_nodes(lookup) != mesh->n_nodes) return fail(VM_ERR_INVALID_ARGUMENT, "the host mesh is not the one that was uploaded");
    vm_frame fr{};
    fr.mesh = mesh;
    std::memcpy(fr.Hoc, Hoc, sizeof(fr.Hoc));
    fr.lens   = *lens;
    fr.image  = image;
    fr.format = format;
    // With the mesh's BSP on the device the lookup runs there, with the host's arithmetic and the host's result: one more small kernel
    // against 10 to 140 us on the calling thread, which is then free to copy the image (thumbnail on a mesh of 7 k nodes: 62 -> 48 us a
    // call, 21 MB frame on one of 1.7 M: 2.49 -> 2.27 ms, ten calls of both grid models and all sizes: -3 % to +29 %).
    if (mesh->n_bsp > 0) return run_batch(e, &fr, 1, 0, out);
    std::vector<int32_t> ranges;
    try {
        int32_t held = 1024;
        do {
            ranges.resize(2 * static_cast<size_t>(held = std::max(held, fr.n_ranges)));
            const vm_status s = vm_hostmesh_lookup(lookup, Hoc, lens, ranges.data(), held, &fr.n_ranges);
            if (s != VM_OK) return s;
        } while (fr.n_ranges > held);
    }
    catch (...) {
        return status_of_exception();
    }
    fr.ranges = ranges.data();
    return run_batch(e, &fr, 1, 0, out);
}

vm_status vm_results_keep(vm_engine* e, vm_results** kept) {
    if (e == nullptr || kept == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    *kept = nullptr;
    if (!e->host) return fail(VM_ERR_INVALID_ARGUMENT, "the engine has no results");
    try {
        std::unique_ptr<KeptResults> k(new KeptResults{e->pool, nullptr});
        std::lock_guard<std::mutex> lock(e->pool->mutex);
        if (e->pool->kept >= MAX_KEPT_RESULTS) return fail(VM_ERR_OUT_OF_MEMORY, "VM_MAX_KEPT_RESULTS results of this engine are kept already");
        ++e->pool->kept;
        k->results = std::move(e->host);
        *kept      = reinterpret_cast<vm_results*>(k.release());
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

void vm_results_release(vm_results* kept) {
    std::unique_ptr<KeptResults> k(reinterpret_cast<KeptResults*>(kept));
    if (!k) return;
    std::lock_guard<std::mutex> lock(k->pool->mutex);
    --k->pool->kept;
    if (!k->pool->closed) k->pool->free.push_back(std::move(k->results));
}

vm_status vm_sample(vm_engine* e, const float* px, int32_t n, const void* image, int32_t width, int32_t height, uint32_t format, float* out) {
    if (e == nullptr || px == nullptr || image == nullptr || out == nullptr || n < 0 || width <= 0 || height <= 0) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    }
    const int cls = format_class(format);
    if (cls == FMT_UNKNOWN) return fail(VM_ERR_UNSUPPORTED_FORMAT, "Unsupported image format");
    if (n == 0) return VM_OK;
    // The reference reads whatever address a coordinate outside the image leads to (cpp/visualmesh/engine/cpu/
    // pixel.hpp:131-134 clamp only one side); the engine itself only samples points that passed the on-screen test.
    // Here the coordinates come from the caller, so they are checked: a read outside the image would be a GPU fault.
    for (int32_t i = 0; i < n; ++i) {
        const float x = px[2 * i], y = px[2 * i + 1];
        if (!(x >= 0.0f && x <= static_cast<float>(width - 1) && y >= 0.0f && y <= static_cast<float>(height - 1))) {
            return fail(VM_ERR_INVALID_ARGUMENT, "pixel coordinate " + std::to_string(i) + " is outside the image (or not finite)");
        }
    }
    try {
        VM_CUDA(cudaSetDevice(e->device));
        Lane& lane        = e->lanes[0];
        const size_t bytes = static_cast<size_t>(width) * height * format_bytes_per_pixel(cls);
        need(e, lane.d_images, bytes);
        need(e, lane.d_cand_px, n);
        need(e, lane.d_feat[0], static_cast<size_t>(n) * 4);
        VM_CUDA(cudaMemcpyAsync(lane.d_images.p, image, bytes, cudaMemcpyHostToDevice, lane.stream));
        VM_CUDA(cudaMemcpyAsync(lane.d_cand_px.p, px, sizeof(float2) * n, cudaMemcpyHostToDevice, lane.stream));
        ++e->launches;
        k_sample_flat<<<(n + ROW_THREADS - 1) / ROW_THREADS, ROW_THREADS, 0, lane.stream>>>(
          lane.d_cand_px.p, n, lane.d_images.p, width, height, cls, reinterpret_cast<float4*>(lane.d_feat[0].p));
        VM_CUDA(cudaGetLastError());
        VM_CUDA(cudaMemcpyAsync(out, lane.d_feat[0].p, sizeof(float) * 4 * n, cudaMemcpyDeviceToHost, lane.stream));
        VM_CUDA(cudaStreamSynchronize(lane.stream));
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

vm_status vm_network(vm_engine* e, const float* input, const int32_t* neighbourhood, int32_t n_rows, int32_t n_neighbours, float* out) {
    if (e == nullptr || input == nullptr || neighbourhood == nullptr || out == nullptr || n_rows <= 0) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    }
    if (e->layers.empty()) return fail(VM_ERR_NETWORK_SHAPE, "this engine was created without a network");
    if (e->layers.front().n_slots != n_neighbours + 1) return fail(VM_ERR_NETWORK_SHAPE, "network was built for a different n_neighbours");
    for (size_t i = 0; i < static_cast<size_t>(n_rows) * n_neighbours; ++i) {
        if (neighbourhood[i] < 0 || neighbourhood[i] >= n_rows) return fail(VM_ERR_INVALID_ARGUMENT, "neighbour index outside the rows");
    }
    try {
        VM_CUDA(cudaSetDevice(e->device));
        Lane& lane = e->lanes[0];
        const size_t rows = n_rows;
        need(e, e->d_offsets, 2);
        need(e, e->d_nb, rows * n_neighbours);
        need(e, e->d_cls, rows * e->n_classes);
        need(e, lane.d_feat[0], rows * e->max_width);
        need(e, lane.d_feat[1], rows * e->max_width);
        const int32_t offsets[2] = {0, n_rows - 1};
        VM_CUDA(cudaMemcpyAsync(e->d_offsets.p, offsets, sizeof(offsets), cudaMemcpyHostToDevice, lane.stream));
        VM_CUDA(cudaMemcpyAsync(e->d_nb.p, neighbourhood, sizeof(int32_t) * rows * n_neighbours, cudaMemcpyHostToDevice, lane.stream));
        e->timing = false;
        for (int attempt = 0; attempt < 2; ++attempt) {
            // the layers ping-pong over the feature buffers, so a second attempt needs the input again
            VM_CUDA(cudaMemcpyAsync(lane.d_feat[0].p, input, sizeof(float) * rows * 4, cudaMemcpyHostToDevice, lane.stream));
            for (int i = 0; i < ABORT_FLAGS; ++i) e->flags[i] = 0;
            const bool with_plan = e->staged && e->use_tc && e->may_stage;
            if (with_plan) {
                ensure_tile_plan(e, lane, rows, (rows + STAGED_ST - 1) / STAGED_ST + 1);
                const st::PlanOut plan = tile_plan(lane);
                ++e->launches;
                launch_tile_plan_kernel(n_neighbours, e->d_offsets.p, e->d_nb.p, plan.nbl, plan.halo_rows, plan.halo_count, 0, 1, n_rows, lane.stream);
                VM_CUDA(cudaGetLastError());
            }
            run_network(e, lane, with_plan, e->d_offsets.p, e->d_nb.p, n_neighbours, 0, 1, n_rows, e->d_cls.p, true, n_rows);
            VM_CUDA(cudaMemcpyAsync(out, e->d_cls.p, sizeof(float) * rows * e->n_classes, cudaMemcpyDeviceToHost, lane.stream));
            VM_CUDA(cudaStreamSynchronize(lane.stream));
            if (e->flags[ABORT_TC_TIMEOUT]) return fail(VM_ERR_DEVICE_ABORT, "a kernel gave up on a bounded wait");
            if (e->flags[ABORT_TC_RANGE] && e->use_tc) {
                e->use_tc = false;  // a value beyond the fp16 split's range: recompute with the FFMA kernels
                continue;
            }
            break;
        }
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

// ---- projection without any allocation ----------------------------------------------------------------------------
// All scratch of this entry point is one array inside the library image. In host code `g_static_scratch` is only a
// stand-in for the symbol; the address the kernels need comes from cudaGetSymbolAddress, looked up once per device.
namespace {
constexpr size_t align256(size_t v) {
    return (v + 255) & ~size_t(255);
}
constexpr size_t ST_FRAME   = 0;
constexpr size_t ST_CELLS   = ST_FRAME + align256(sizeof(vm::FrameParams));  // offsets[2], the offsets' second copy, abort flags, group counts
constexpr size_t ST_HEADER  = ST_CELLS + 256;
constexpr size_t ST_BLOCKS  = ST_HEADER + align256(sizeof(vm::ChunkHeader));
constexpr size_t ST_STATE   = ST_BLOCKS + align256(sizeof(int32_t) * (VM_STATIC_MAX_NODES / vm::SELECT_THREADS + 2));
constexpr int ST_GROUPS     = VM_STATIC_MAX_NODES / (vm::SELECT_THREADS * vm::GROUP_BLOCKS) + 1;
static_assert(8 + ST_GROUPS <= 64, "the cells hold offsets, flags and group counts");
constexpr size_t ST_CAND_PX = ST_STATE + align256(VM_STATIC_MAX_BSP);
constexpr size_t ST_CAND_ID = ST_CAND_PX + align256(sizeof(float2) * VM_STATIC_MAX_NODES);
constexpr size_t ST_RANK    = ST_CAND_ID + align256(sizeof(int32_t) * VM_STATIC_MAX_NODES);
constexpr size_t ST_BYTES   = ST_RANK + align256(sizeof(int32_t) * VM_STATIC_MAX_NODES);

static __device__ __align__(256) unsigned char g_static_scratch[ST_BYTES];

constexpr int ST_MAX_DEVICES = 64;
unsigned char* g_static_address[ST_MAX_DEVICES] = {};
std::once_flag g_static_once[ST_MAX_DEVICES];
}  // namespace

vm_status vm_project_static(vm_engine* e,
                            const vm_mesh* mesh,
                            const float Hoc[16],
                            const vm_lens* lens,
                            float* d_px,
                            int32_t* d_gi,
                            int32_t* d_nb,
                            int32_t* d_n_points,
                            int32_t* n_points) {
    if (e == nullptr || mesh == nullptr || Hoc == nullptr || lens == nullptr || d_px == nullptr || d_gi == nullptr || d_nb == nullptr) {
        return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    }
    if (lens->projection != VM_RECTILINEAR && lens->projection != VM_EQUISOLID && lens->projection != VM_EQUIDISTANT) {
        return fail(VM_ERR_UNSUPPORTED_LENS, "Cannot project: Unknown lens type");
    }
    if (lens->dimensions[0] <= 0 || lens->dimensions[1] <= 0) return fail(VM_ERR_INVALID_ARGUMENT, "lens dimensions must be positive");
    if (mesh->owner != e) return fail(VM_ERR_INVALID_ARGUMENT, "mesh was uploaded through another engine");
    if (mesh->n_bsp == 0) return fail(VM_ERR_NO_BSP, "vm_project_static looks up on the device: the mesh needs vm_mesh_set_bsp");
    if (mesh->n_nodes > VM_STATIC_MAX_NODES) {
        return fail(VM_ERR_INVALID_ARGUMENT, "mesh has " + std::to_string(mesh->n_nodes) + " nodes; vm_project_static holds at most VM_STATIC_MAX_NODES = "
                                               + std::to_string(VM_STATIC_MAX_NODES));
    }
    if (mesh->n_bsp > VM_STATIC_MAX_BSP) {
        return fail(VM_ERR_INVALID_ARGUMENT, "mesh BSP has " + std::to_string(mesh->n_bsp) + " elements; vm_project_static holds at most VM_STATIC_MAX_BSP = "
                                               + std::to_string(VM_STATIC_MAX_BSP));
    }
    if (e->device < 0 || e->device >= ST_MAX_DEVICES) return fail(VM_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    try {
        VM_CUDA(cudaSetDevice(e->device));
        // once per device, with that device current; engines of several host threads may get here together
        cudaError_t lookup = cudaSuccess;
        std::call_once(g_static_once[e->device], [&] {
            unsigned char* address = nullptr;
            lookup = cudaGetSymbolAddress(reinterpret_cast<void**>(&address), g_static_scratch);
            if (lookup == cudaSuccess) g_static_address[e->device] = address;
        });
        if (lookup != cudaSuccess) throw CudaFailure{lookup, "cudaGetSymbolAddress(g_static_scratch)"};
        unsigned char* base = g_static_address[e->device];
        if (base == nullptr) return fail(VM_ERR_CUDA, "the address of the static scratch array could not be looked up on this device");
        auto* d_frame         = reinterpret_cast<FrameParams*>(base + ST_FRAME);
        auto* d_cells         = reinterpret_cast<int32_t*>(base + ST_CELLS);  // [0..1] offsets, [2..3] copy, [4..7] abort flags, [8..] group counts
        auto* d_header        = reinterpret_cast<ChunkHeader*>(base + ST_HEADER);
        auto* d_blocks        = reinterpret_cast<int32_t*>(base + ST_BLOCKS);
        auto* d_state         = reinterpret_cast<uint8_t*>(base + ST_STATE);
        auto* d_cand_px       = reinterpret_cast<float2*>(base + ST_CAND_PX);
        auto* d_cand_node     = reinterpret_cast<int32_t*>(base + ST_CAND_ID);
        auto* d_rank          = reinterpret_cast<int32_t*>(base + ST_RANK);

        vm_frame fr{};
        fr.mesh = mesh;
        std::memcpy(fr.Hoc, Hoc, sizeof(fr.Hoc));
        fr.lens = *lens;
        FrameParams p;
        std::memset(&p, 0, sizeof(p));
        // never builds the libm last-bit tables here (that allocates): they are used only if an earlier call built them
        if (!fill_frame_params(e, fr, p, false)) return fail(VM_ERR_UNSUPPORTED_LENS, "Cannot project: Unknown lens type");
        p.n_candidates = mesh->n_nodes;

        cudaStream_t s = e->lanes[0].stream;
        VM_CUDA(cudaMemcpyAsync(d_frame, &p, sizeof(p), cudaMemcpyHostToDevice, s));
        // the array keeps the last call's contents: the running offset and the abort flag must start at zero
        VM_CUDA(cudaMemsetAsync(d_cells, 0, 64 * sizeof(int32_t), s));
        const ChunkHeader header{nullptr, nullptr, nullptr, nullptr, d_cells + 2};
        VM_CUDA(cudaMemcpyAsync(d_header, &header, sizeof(header), cudaMemcpyHostToDevice, s));
        const int blocks = (mesh->n_nodes + SELECT_THREADS - 1) / SELECT_THREADS;
        k_bsp_state<<<dim3((mesh->n_bsp + SELECT_THREADS - 1) / SELECT_THREADS, 1), SELECT_THREADS, 0, s>>>(d_frame, d_state);
        const int groups = (blocks + GROUP_BLOCKS - 1) / GROUP_BLOCKS;
        k_select<<<dim3(blocks, 1), SELECT_THREADS, 0, s>>>(d_frame, d_state, d_cand_px, d_cand_node, d_blocks, d_cells + 8, groups, d_cells + 4);
        k_scatter<1><<<dim3(blocks, 1), SELECT_THREADS, 0, s>>>(d_frame, d_header, d_cand_px, d_cand_node, d_blocks, d_cells + 8, blocks, groups, d_cells, 0,
                                                             reinterpret_cast<float2*>(d_px), d_gi, d_rank);
        dim3 g((mesh->n_nodes + 1 + ROW_THREADS - 1) / ROW_THREADS, 1);
        const st::PlanOut no_plan{nullptr, nullptr, nullptr};
        if (mesh->n_neighbours == 4) k_remap<4, false><<<g, ROW_THREADS, 0, s>>>(d_frame, d_cells, 0, d_gi, d_rank, d_nb, no_plan);
        else if (mesh->n_neighbours == 6) k_remap<6, false><<<g, ROW_THREADS, 0, s>>>(d_frame, d_cells, 0, d_gi, d_rank, d_nb, no_plan);
        else k_remap<8, false><<<g, ROW_THREADS, 0, s>>>(d_frame, d_cells, 0, d_gi, d_rank, d_nb, no_plan);
        VM_CUDA(cudaGetLastError());
        e->launches += 4;
        if (d_n_points != nullptr) VM_CUDA(cudaMemcpyAsync(d_n_points, d_cells + 1, sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
        int32_t cells[8] = {};
        VM_CUDA(cudaMemcpyAsync(cells, d_cells, sizeof(cells), cudaMemcpyDeviceToHost, s));
        VM_CUDA(cudaStreamSynchronize(s));
        if (cells[4 + ABORT_BSP_DEPTH] != 0) return fail(VM_ERR_DEVICE_ABORT, "a kernel gave up on a bounded loop (BSP deeper than 128 levels)");
        if (n_points != nullptr) *n_points = cells[1];
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

vm_status vm_stage_times(vm_engine* e, const char** names, float* ms, int32_t capacity, int32_t* n) {
    if (e == nullptr || n == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    *n = static_cast<int32_t>(e->stage_ms.size());
    for (int i = 0; i < *n && i < capacity; ++i) {
        if (names != nullptr) names[i] = e->stage_ms[i].first;
        if (ms != nullptr) ms[i] = e->stage_ms[i].second;
    }
    return VM_OK;
}

vm_status vm_timer_start(vm_engine* e) {
    if (e == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null engine");
    try {
        VM_CUDA(cudaSetDevice(e->device));
        for (auto& lane : e->lanes)
            if (lane.stream != nullptr) VM_CUDA(cudaStreamSynchronize(lane.stream));
        VM_CUDA(cudaEventRecord(e->ev_timer_start, e->lanes[0].stream));
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

vm_status vm_timer_stop(vm_engine* e, float* milliseconds) {
    if (e == nullptr || milliseconds == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    try {
        VM_CUDA(cudaSetDevice(e->device));
        // lane 0 waits for the other lanes, then stamps the end
        for (int l = 1; l < MAX_LANES; ++l) {
            if (e->lanes[l].stream == nullptr) continue;
            VM_CUDA(cudaEventRecord(e->lanes[l].ev_fork, e->lanes[l].stream));
            VM_CUDA(cudaStreamWaitEvent(e->lanes[0].stream, e->lanes[l].ev_fork, 0));
        }
        VM_CUDA(cudaEventRecord(e->ev_timer_stop, e->lanes[0].stream));
        VM_CUDA(cudaEventSynchronize(e->ev_timer_stop));
        VM_CUDA(cudaEventElapsedTime(milliseconds, e->ev_timer_start, e->ev_timer_stop));
    }
    catch (...) {
        return status_of_exception();
    }
    return VM_OK;
}

vm_status vm_set_wait_limit(vm_engine* e, uint32_t polls) {
    if (e == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null engine");
    e->tc_wait_limit = polls;
    return VM_OK;
}

int64_t vm_launch_count(const vm_engine* e) {
    return e == nullptr ? 0 : e->launches;
}

vm_status vm_host_alloc(void** ptr, size_t bytes) {
    if (ptr == nullptr) return fail(VM_ERR_INVALID_ARGUMENT, "null argument");
    const cudaError_t err = cudaHostAlloc(ptr, bytes, cudaHostAllocDefault);
    if (err != cudaSuccess) {
        cudaGetLastError();
        return fail(err == cudaErrorMemoryAllocation ? VM_ERR_OUT_OF_MEMORY : VM_ERR_CUDA, cudaGetErrorString(err));
    }
    return VM_OK;
}

void vm_host_free(void* ptr) {
    if (ptr != nullptr) cudaFreeHost(ptr);
}

}  // extern "C"
