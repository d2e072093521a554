// Graph-convolution layer on the tensor cores with the gather served from shared memory.
//
// The other layer kernels gather every neighbour row with per-thread global loads; a quarter of them miss the L1 cache
// (the first touch of every row), each miss stalls its warp for a full memory latency, and the layers end up bound by
// that latency (tensor-core kernels of conv_tc.cuh) or by the FP32 pipe (conv_ffma.cuh). Mesh nodes are stored in the
// order of the reference's BSP (cpp/visualmesh/mesh.hpp:450-466), which is spatially compact: of the neighbour
// references of 256 consecutive on-screen rows about 87 % point inside the same 256 rows, and the rest touch ~95
// distinct rows outside.
//
// So the rows of a frame are cut into super-tiles of consecutive rows and a tile plan (tile_plan.cuh) is made once per
// chunk of frames: the list of outside rows each super-tile needs (its halo) and every row's neighbours as 16-bit
// positions inside "super-tile + halo". A layer then runs as a persistent kernel whose loader warp brings a
// super-tile's own rows and their positions into shared memory with one bulk asynchronous copy each and its halo rows with
// 16-byte asynchronous copies - every byte of the feature buffer is requested once per super-tile that needs it, a
// super-tile ahead of its use - and whose compute warps read neighbour rows from shared memory only. The product runs on
// the warp-level tensor-core path (mma.sync m16n8k16, fp16 hi/lo parts of both operands, fp32 accumulators in registers)
// rather than tcgen05: a 16-channel slot is a 16x16x16 product per sixteen rows, far too little work per instruction to
// amortise moving a gathered tile into tensor memory and a single-thread issue pipeline, while here every warp is an
// independent worker with nothing to hand over (the 16 -> 16 layer over 4.4 M rows: tcgen05 with global-load gather
// 337 us, tcgen05 with this staging 740 us at one CTA per SM; the FFMA kernel 308 us).
//
// What bounds it is the shared-memory data path, then the rate of mma.sync (measured: one m16n8k16 per 8.5 cycles and SM
// sub-partition, 89 cycles for the 42 of sixteen rows of the 16 -> 16 layer with six neighbours). Three choices keep that path short:
//   - The weights are the operand with sixteen rows and the gathered rows the one with eight columns. A feature row is four
//     16-byte pieces, each the hi and the lo parts of four channels, and a thread's piece of a row IS its two registers
//     of that operand, hi and lo: one 16-byte load, no register is moved. (As the operand with sixteen rows its four
//     registers come from two loads: 170 moves more per sixteen rows.)
//   - A quarter-warp reads two whole rows of 64 bytes, so only two rows of the same parity meet in a bank (a third of the
//     pairs on the meshes here: consecutive rows have neighbours that follow one another). Rows in planes of 16-byte
//     pieces, eight of them per quarter-warp as ldmatrix takes them, took 2.25 passes where this takes 1.4.
//   - Twelve warps per SM with 106 to 128 registers instead of 24 with 72: loads of the next slot are in flight during the products of
//     one, and nothing spills but a register of 16 -> 8 with eight neighbours. The eight-channel layers also keep their weights in
//     registers (the sixteen-channel ones have twice as many, which spills).
// 16 -> 16 over 4.48 M rows with six neighbours 212 -> 169 us (the weights' fragments are 28 of its 115 wavefronts of shared-memory
// loads per sixteen rows, the rows 56 and 24 of conflicts), 16 -> 8 176 -> 123 us (138 with the weights read for each slot). On the way:
// planes and ldmatrix with fewer instructions 212; the layout alone 219 and 152; weights as the first operand with 24 warps 200 and 152;
// with twelve 182 and 138; split rows transposed before they are stored (stores of a quarter-warp in one 128-byte line, not
// four) 169. Sixteen compute warps in two CTAs 192; groups of 64 rows 177 (spills).
// A neighbour without a halo slot (more outside rows than the plan has slots) is marked and fetched from global memory
// by its warp, so any neighbourhood is computed correctly, only slower.
//
// The only waits are for a window's copies (compute warps) and for a window to be handed back (loader), and they are
// bounded. No multicast of any kind; all copies read this GPU's own memory.
#pragma once

#include "conv_tc.cuh"
#include "tile_plan.cuh"

namespace vm {
namespace st {

    struct PlanArgs {
        const int32_t* offsets;  // batch-wide point offsets
        const int32_t* nb;       // batch-wide neighbourhood rows (frame-local indices)
        PlanOut out;
        int32_t f0;
    };

    // The plan for a neighbourhood that is already in memory: one block per super-tile (blockIdx.x) and frame
    // (blockIdx.y), one thread per row. (On the hot path the neighbour-remap kernel makes the plan as it writes the
    // neighbourhood.)
    template <int N>
    __global__ void __launch_bounds__(ST) k_tile_plan(const PlanArgs a) {
        const int f     = blockIdx.y;
        const int frame = a.f0 + f;
        const int start = a.offsets[frame];
        const int rows  = a.offsets[frame + 1] - start + 1;
        const int t0    = blockIdx.x * ST;
        if (t0 >= rows) return;
        const int row    = t0 + static_cast<int>(threadIdx.x);
        const bool valid = row < rows;
        int idx[N];
#pragma unroll
        for (int j = 0; j < N; ++j) idx[j] = 0;
        if (valid) {
            const int32_t* src = a.nb + static_cast<size_t>(start + frame + row) * N;
#pragma unroll
            for (int j = 0; j < N; ++j) idx[j] = __ldg(src + j);
        }
        plan_super_tile<N>(idx, valid, t0, f, a.offsets, a.f0, a.out);
    }

    using tc::bulk_copy;
    using tc::copies_arrive;
    using tc::copy16;
    using tc::expect_bytes;
    using tc::load_shared;

    // ---- warp-level tensor-core pieces ----------------------------------------------------------------------------------
    // D += A . B, A 16x16 fp16 (row), B 16x8 fp16 (col), D 16x8 fp32
    __device__ __forceinline__ void mma_16816(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
    }
    // an 8x8 matrix of fp16 values, two neighbours of row g per thread
    __device__ __forceinline__ uint32_t transpose(uint32_t v) {
        uint32_t r;
        asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
        return r;
    }
    struct Args {
        int32_t n_frames;
        int32_t* abort_flags;
        uint32_t wait_limit;  // polls of one wait for a window before the kernel gives up (0: the first wait fails at once)
    };

    constexpr uint32_t WAIT_LIMIT  = tc::WAIT_LIMIT;
    constexpr int MAX_FRAMES       = tc::MAX_FRAMES;
    constexpr int TILE             = 8;   // rows of one warp-level MMA tile (its N)
    constexpr int CIN              = 16;  // input channels
    constexpr int ROW              = 4 * CIN;  // bytes of a feature row: four pieces of four channels, hi parts then lo parts each
    constexpr int NBL_BYTES        = ST * NBL_STRIDE * 2;

    // 16x16 fragments of a slot's weights: hi and lo parts of 16 output channels each, or of eight channels in one
    template <int COUT>
    __host__ __device__ constexpr int weight_fragments() {
        return COUT == 8 ? 1 : COUT / 8;
    }
    template <int COUT, int NSLOTS>
    __host__ __device__ constexpr int weight_bytes() {
        return NSLOTS * weight_fragments<COUT>() * 32 * 16;
    }
    // Rows of the two windows together: as many as let CTAS blocks share an SM, which has 228 KB and keeps 1 KB of them for every block. A
    // window takes as many as its super-tile and its halo have. Windows of 192 halo slots each made every super-tile with more outside rows a slow
    // one: none of the rings', three in four of an XYGRID8's (269 on average with 2.3 M rows, 16 % have more than the plan's 384 slots), half of an
    // XYGRID6's, 43 % of an XYGRID4's. And 896 rows with sixteen channels and eight neighbours left room for two blocks, not three: 16 -> 16
    // over 4.5 M rows of RING8 217 -> 203 us, over 2.3 M of XYGRID8 314 -> 236 (343 with windows of 192 slots).
    constexpr int SMEM_ALIGN  = 128;
    constexpr int SMEM_STATIC = (4 * 8 + 2 * 4 * (MAX_FRAMES + 1) + 5 * 4 + SMEM_ALIGN - 1) / SMEM_ALIGN * SMEM_ALIGN;  // the kernel's other variables
    template <int COUT, int NSLOTS, int CTAS>
    __host__ __device__ constexpr int pool_rows() {
        constexpr int room = 228 * 1024 / CTAS - 1024 - SMEM_STATIC - 2 * NBL_BYTES - weight_bytes<COUT, NSLOTS>();
        constexpr int rows = room / (2 * ROW) * 2;
        static_assert(rows >= ST + HALO, "a window fits");
        return rows < 2 * (ST + HALO) ? rows : 2 * (ST + HALO);
    }
    // windows, their neighbour positions, weights
    template <int COUT, int NSLOTS, int CTAS>
    __host__ __device__ constexpr size_t smem_bytes() {
        return static_cast<size_t>(pool_rows<COUT, NSLOTS, CTAS>()) * ROW + 2 * NBL_BYTES + weight_bytes<COUT, NSLOTS>();
    }

    // One CTA walks super-tiles; while it computes on one window the next is on its way. Every warp owns groups of TILES 8-row
    // tiles of the super-tile: for each slot four threads read a neighbour row, 16 bytes each, and hold with it their part of the
    // operand; three MMAs per 16 output channels add hi.hi, lo.hi and hi.lo into fp32 accumulators in registers (dropping only lo.lo
    // keeps ~2^-21 relative accuracy; with 8 output channels two MMAs do all four), and the epilogue (activation, store as fp32
    // chunks or split again for the next such layer) runs on the accumulator registers. The weights sit in shared memory as
    // ready-made fragments (16 bytes per lane, read once per slot for all tiles of the group), or in registers. The last warp
    // of the CTA is the loader; a compute warp waits only for a window to land and tells the loader when it is done with one,
    // so no compute warp ever waits for another.
    template <int COUT, int NSLOTS, int TILES, int THREADS, int CTAS>
    __global__ void __launch_bounds__(THREADS, CTAS) k_graph_conv_mma(const ConvArgs a, const Args t, const Plan plan) {
        static_assert((COUT == 8 || COUT == 16 || COUT == 32) && ST % (TILES * TILE) == 0, "whole fragments, whole groups of tiles");
        constexpr int MBLK  = COUT == 32 ? 2 : 1;  // blocks of 16 rows of the weights' operand
        constexpr int FRAGS = weight_fragments<COUT>();
        constexpr int WARPS = THREADS / 32 - 1;    // compute warps; the last warp of the CTA is the loader
        constexpr int POOL  = pool_rows<COUT, NSLOTS, CTAS>();

        extern __shared__ __align__(SMEM_ALIGN) unsigned char smem_raw[];
        __shared__ uint64_t bars[4];                      // full[2]: a window has landed; empty[2]: every compute warp is done with it
        __shared__ int32_t tile_prefix[MAX_FRAMES + 1];   // in super-tiles
        __shared__ int32_t frame_start[MAX_FRAMES + 1];   // offsets[f0 + f]
        __shared__ int32_t window_miss[2];                // some neighbour of the super-tile was left out of its window
        __shared__ int32_t window_start[2];               // its first row in the pool
        __shared__ int32_t failed_s;
        volatile int32_t* failed = &failed_s;

        const int tid  = threadIdx.x;
        const int warp = tid >> 5;
        const int lane = tid & 31;
        const int g    = lane >> 2;  // row of a tile that the thread reads; output channels of the accumulator fragment
        const int tq   = lane & 3;   // its piece of that row; rows 2 tq and 2 tq + 1 of the accumulator fragment
        const uint32_t win_addr = tc::smem_u32(smem_raw);
        const uint32_t nbl_addr  = win_addr + POOL * ROW;
        const uint32_t frag_addr = nbl_addr + 2 * NBL_BYTES + lane * 16;  // this lane's 16 bytes of fragment 0
        const uint32_t bar_full  = tc::smem_u32(&bars[0]);
        const uint32_t bar_empty = tc::smem_u32(&bars[2]);

        if (tid == 0) {
            failed_s = 0;
            for (int i = 0; i < 2; ++i) {
                tc::mbar_init(bar_full + 8 * i, 1 + 32);  // the bulk copies' byte count + one arrival per loader lane
                tc::mbar_init(bar_empty + 8 * i, WARPS);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int f = tid; f <= t.n_frames; f += THREADS) frame_start[f] = a.offsets[a.f0 + f];
        __syncthreads();
        tc::tiles_before<ST>(tile_prefix, frame_start, t.n_frames);

        // ---- the weights' fragments: split into fp16 hi and lo parts, in the register layout of mma.m16n8k16's A ----
        // The contraction's K axis may come in any order that both operands share: thread (g, tq) holds input channels 4 tq .. 4 tq + 3 of
        // a row (its 16-byte piece) as k = 2 tq, 2 tq + 1, 2 tq + 8, 2 tq + 9. Which output channel a row of the operand stands for is free
        // too; a thread gets rows g and g + 8 of each block, and those are neighbouring channels. Eight channels are one block: their
        // hi parts are its rows 0 to 7, their lo parts rows 8 to 15.
        auto channel = [&](int block, int half) { return COUT == 8 ? g : COUT == 16 ? 4 * (g >> 1) + 2 * half + (g & 1) : 4 * g + 2 * block + half; };
        {
            constexpr int COUTP = (COUT + 3) & ~3;
            uint4* w_frag       = reinterpret_cast<uint4*>(smem_raw + POOL * ROW + 2 * NBL_BYTES);  // [slot][block][part][lane]
            for (int i = warp; i < NSLOTS * MBLK; i += WARPS + 1) {
                const int block = i % MBLK, slot = i / MBLK;
                const float* w  = a.weights + static_cast<size_t>(slot * CIN + 4 * tq) * COUTP;
                uint32_t h[4], l[4];  // register 2 k + half: channels 4 tq + 2 k, + 1 of the block's row g + 8 half
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float* from = w + (r & 2) * COUTP + channel(block, r & 1);
                    split_pair(__ldg(from), __ldg(from + COUTP), h[r], l[r]);
                }
                if (COUT == 8) { w_frag[slot * 32 + lane] = make_uint4(h[0], l[0], h[2], l[2]); }
                else {
                    w_frag[(2 * i) * 32 + lane]     = make_uint4(h[0], h[1], h[2], h[3]);
                    w_frag[(2 * i + 1) * 32 + lane] = make_uint4(l[0], l[1], l[2], l[3]);
                }
            }
        }
        float bias[MBLK][2];
#pragma unroll
        for (int m = 0; m < MBLK; ++m) {
            bias[m][0] = __ldg(a.biases + channel(m, 0));
            bias[m][1] = COUT == 8 ? 0.0f : __ldg(a.biases + channel(m, 1));
        }
        __syncthreads();
        const int total_st = tile_prefix[t.n_frames];

        struct StRef {
            int rows;        // rows of the frame, off-screen row included
            int t0;          // first row of the super-tile within the frame
            int local_base;  // first feature row of the frame in this launch
            size_t nb_base;  // first neighbourhood row of the frame
        };
        int frame_hint = 0;
        auto locate = [&](int s) {
            int f = frame_hint;
            while (f + 1 < t.n_frames && tile_prefix[f + 1] <= s) ++f;
            frame_hint      = f;
            const int start = frame_start[f];
            StRef r;
            r.rows       = frame_start[f + 1] - start + 1;
            r.t0         = (s - tile_prefix[f]) * ST;
            r.local_base = start - frame_start[0] + f;
            r.nb_base    = static_cast<size_t>(start + a.f0 + f);
            return r;
        };
        // all that read the features: the loader, and the compute warps behind its first window
        const unsigned char* in_bytes = reinterpret_cast<const unsigned char*>(a.in);

        if (warp == WARPS) {
            // ================= loader warp: one window ahead of the compute warps per buffer =================
            // The halo list of a super-tile (its length, then this lane's entries) is read one super-tile ahead, while
            // the loader waits for a buffer anyway: the copies of a window then start the moment its buffer is free
            // instead of two dependent trips to global memory later. As much of it as most have: the rest is read when it is copied.
            constexpr int EARLY    = 192;
            constexpr int PER_LANE = EARLY / 32;
            int n_halo = 0, listed = 0;
            int32_t halo_row[PER_LANE];
            auto fetch_halo_list = [&](int st) {
                listed                = __ldg(plan.halo_count + st);
                n_halo                = min(listed, HALO);
                const int32_t* h_rows = plan.halo_rows + static_cast<size_t>(st) * HALO;
#pragma unroll
                for (int k = 0; k < PER_LANE; ++k) halo_row[k] = __ldg(h_rows + lane + 32 * k);  // entries past n_halo are never used
            };
            uint32_t n = 0;
            int before = 0;  // rows of the window before
            bool ok    = true;
            if (static_cast<int>(blockIdx.x) < total_st) fetch_halo_list(blockIdx.x);
            in_bytes = after_previous(in_bytes);
            for (int s = blockIdx.x; s < total_st; s += gridDim.x, ++n) {
                const uint32_t b = n & 1u;
                // every compute warp must be done with the super-tile that used this buffer before
                // the warp decides together: what follows needs all of its lanes, and a window that some had begun would never become full
                ok = __all_sync(0xffffffffu, n < 2 || tc::mbar_wait_or_fail(bar_empty + 8 * b, ((n >> 1) - 1) & 1u, failed, t.wait_limit));
                if (!ok) break;
                // windows lie at the pool's beginning and at its end in turn; two that do not fit beside each other follow one another
                const int size = ST + n_halo;
                if (size + before > POOL) {
                    ok = __all_sync(0xffffffffu, tc::mbar_wait_or_fail(bar_empty + 8 * (b ^ 1u), ((n - 1) >> 1) & 1u, failed, t.wait_limit));
                    if (!ok) break;
                }
                before             = size;
                const int at       = b == 0 ? 0 : POOL - size;
                const StRef r      = locate(s);
                const int own      = min(ST, r.rows - r.t0);
                const uint32_t dst = win_addr + at * ROW;
                const uint32_t bar = bar_full + 8 * b;
                if (lane == 0) {
                    window_miss[b]  = listed > HALO;
                    window_start[b] = at;
                    expect_bytes(bar, static_cast<uint32_t>(own * (ROW + 2 * NBL_STRIDE)));
                    bulk_copy(nbl_addr + b * NBL_BYTES, reinterpret_cast<const uint4*>(plan.nbl) + r.local_base + r.t0, static_cast<uint32_t>(own * 2 * NBL_STRIDE),
                              bar);
                    bulk_copy(dst, in_bytes + static_cast<size_t>(r.local_base + r.t0) * ROW, static_cast<uint32_t>(own * ROW), bar);
                }
                // four lanes to a halo row: whole rows per request
                const unsigned char* feat = in_bytes + (lane & 3) * 16;
                const uint32_t to         = dst + ST * ROW + lane * 16;
#pragma unroll
                for (int k = 0; k < EARLY / 8; ++k) {
                    if (8 * k >= n_halo) break;
                    const int32_t row = __shfl_sync(0xffffffffu, halo_row[k / 4], 8 * (k % 4) + (lane >> 2));
                    if (8 * k + (lane >> 2) < n_halo) copy16(to + k * 8 * ROW, feat + static_cast<size_t>(row) * ROW);
                }
                const int32_t* h_rows = plan.halo_rows + static_cast<size_t>(s) * HALO;
#pragma unroll 4
                for (int h = EARLY + (lane >> 2); h < n_halo; h += 8) {
                    copy16(dst + (ST + h) * ROW + (lane & 3) * 16, feat + static_cast<size_t>(__ldg(h_rows + h)) * ROW);
                }
                __syncwarp();
                if (s + static_cast<int>(gridDim.x) < total_st) fetch_halo_list(s + gridDim.x);
                copies_arrive(bar);
            }
            if (!ok) *failed = 1;
            // Nothing may still be writing this CTA's shared memory when it exits. On the normal path the compute warps have
            // waited for every window; after a wait ran out the last windows may still be on their way: this lane's own
            // 16-byte copies are waited for here, the bulk copies through the windows' barriers (a window is the last one
            // issued into its buffer, so its barrier phase can only be pending or complete), with the full default limit.
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (lane == 0) {
                for (uint32_t m = n > 2 ? n - 2 : 0; m < n; ++m) tc::mbar_wait(bar_full + 8 * (m & 1u), (m >> 1) & 1u, WAIT_LIMIT);
            }
        }
        else {
        // ================= compute warps =================
        constexpr bool HELD = COUT == 8;  // weights in registers
        uint4 held[HELD ? NSLOTS : 1];
        if (HELD) {
#pragma unroll
            for (int i = 0; i < NSLOTS; ++i) held[i] = load_shared(frag_addr + i * 512);
        }
        in_bytes = wait_previous(in_bytes);
        uint32_t n = 0;
        bool ok    = true;
        for (int s = blockIdx.x; s < total_st; s += gridDim.x, ++n) {
            const uint32_t b  = n & 1u;
            const StRef r     = locate(s);
            const int own     = min(ST, r.rows - r.t0);
            const int n_groups = (own + TILES * TILE - 1) / (TILES * TILE);
            ok = __all_sync(0xffffffffu, tc::mbar_wait_or_fail(bar_full + 8 * b, (n >> 1) & 1u, failed, t.wait_limit));
            if (!ok) {
                *failed = 1;
                break;
            }
            const uint32_t win = win_addr + *static_cast<volatile int32_t*>(&window_start[b]) * ROW + tq * 16;
            const uint32_t nbl = nbl_addr + b * NBL_BYTES;
            const bool miss    = *static_cast<volatile int32_t*>(&window_miss[b]) != 0;
            for (int group = warp; group < n_groups; group += WARPS) {
                float acc[TILES][MBLK][4];
#pragma unroll
                for (int i = 0; i < TILES; ++i) {
#pragma unroll
                    for (int m = 0; m < MBLK; ++m) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[i][m][k] = bias[m][k >> 1];
                    }
                }
                // the products of a slot for all tiles, x[i]: this thread's piece of tile i, {hi, hi, lo, lo} of four channels; no
                // accumulator twice in a row
                auto products = [&](const uint4 (&x)[TILES], int slot, auto rolled) {
                    constexpr bool ROLLED = decltype(rolled)::value;  // the slot is not known at compile time
#pragma unroll
                    for (int m = 0; m < MBLK; ++m) {
                        const uint4 wh = HELD && !ROLLED ? held[slot] : load_shared(frag_addr + (slot * FRAGS + (COUT == 8 ? 0 : 2 * m)) * 512);
#pragma unroll
                        for (int i = 0; i < TILES; ++i) mma_16816(acc[i][m], wh, x[i].x, x[i].y);
                        if constexpr (COUT != 8) {
                            const uint4 wl = load_shared(frag_addr + (slot * FRAGS + 2 * m + 1) * 512);
#pragma unroll
                            for (int i = 0; i < TILES; ++i) mma_16816(acc[i][m], wl, x[i].x, x[i].y);
                        }
#pragma unroll
                        for (int i = 0; i < TILES; ++i) mma_16816(acc[i][m], wh, x[i].z, x[i].w);
                    }
                };
                // rows past the super-tile's last are copies of it
                auto window_row = [&](int i) { return static_cast<uint32_t>(min((group * TILES + i) * TILE + g, own - 1)); };
                if (!miss) {
                    uint32_t row[TILES];
                    uint4 pos[TILES];
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
                        row[i] = window_row(i);
                        pos[i] = load_shared(nbl + row[i] * (2 * NBL_STRIDE));
                    }
#pragma unroll
                    for (int slot = 0; slot < NSLOTS; ++slot) {
                        uint4 x[TILES];
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
                            uint32_t p = row[i];
                            if (slot > 0) {
                                const int k         = slot - 1;
                                const uint32_t word = (k >> 1) == 0 ? pos[i].x : (k >> 1) == 1 ? pos[i].y : (k >> 1) == 2 ? pos[i].z : pos[i].w;
                                p                   = (k & 1) ? (word >> 16) : (word & 0xFFFFu);
                            }
                            x[i] = load_shared(win + p * ROW);
                        }
                        products(x, slot, std::false_type{});
                    }
                }
                else {
                    // some neighbour of the super-tile was not staged (more outside rows than halo slots): it comes from global memory
#pragma unroll 1
                    for (int slot = 0; slot < NSLOTS; ++slot) {
                        uint4 x[TILES];
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
                            const uint32_t row = window_row(i);
                            uint32_t p         = row;
                            if (slot > 0) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(p) : "r"(nbl + row * (2 * NBL_STRIDE) + 2 * (slot - 1)));
                            if (slot > 0 && p == NBL_GLOBAL) {
                                const int idx = __ldg(a.nb + (r.nb_base + r.t0 + row) * a.n_neighbours + (slot - 1));
                                x[i]          = *reinterpret_cast<const uint4*>(in_bytes + static_cast<size_t>(r.local_base + idx) * ROW + tq * 16);
                            }
                            else {
                                x[i] = load_shared(win + p * ROW);
                            }
                        }
                        __syncwarp();
                        products(x, slot, std::true_type{});
                    }
                }
                if constexpr (COUT == 8) {  // what the hi and the lo parts of the weights gave
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
                        acc[i][0][0] += acc[i][0][2];
                        acc[i][0][1] += acc[i][0][3];
                    }
                }
                // ---- epilogue on the accumulator fragments: rows 2 tq and 2 tq + 1 of each tile, COUT / 8 neighbouring channels ----
                auto apply = [&](auto f) {
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
#pragma unroll
                        for (int m = 0; m < MBLK; ++m) {
#pragma unroll
                            for (int k = 0; k < (COUT == 8 ? 2 : 4); ++k) acc[i][m][k] = f(acc[i][m][k]);
                        }
                    }
                };
                if (a.activation == VM_SELU) apply([](float x) { return selu(x); });
                else if (a.activation == VM_RELU) apply([](float x) { return x < 0.0f ? 0.0f : x; });
                else if (a.activation == VM_TANH) apply([](float x) { return tanhf(x); });
                // fp32 is stored by threads g and g ^ 1 together, which hold channels of the same four (8 channels: two) of the same two
                // rows: each takes one of the rows and the other's part of it. With 32 channels a thread's own part is wide enough. Split
                // rows of 16 channels are transposed, so that four threads write the 64 bytes of row g.
                const bool odd       = (g & 1) != 0;
                const bool quads     = COUT == 16 && a.out_split != SPLIT_NONE;
                const int row0       = r.t0 + group * TILES * TILE + (quads ? g : 2 * tq + (COUT != 32 && odd ? 1 : 0));  // within the frame
                const int left       = r.rows - row0;  // row row0 + k exists: k < left
                const size_t out_row = static_cast<size_t>(r.local_base) + row0;
                unsigned char* out_b = reinterpret_cast<unsigned char*>(a.out);
                auto swap            = [&](uint32_t first, uint32_t second) { return __shfl_xor_sync(0xffffffffu, odd ? first : second, 4); };
                auto swap_f          = [&](float first, float second) { return __uint_as_float(swap(__float_as_uint(first), __float_as_uint(second))); };
                if constexpr (COUT == 8) {
                    // chunk-planar fp32 (no consumer takes 8 channels split)
                    unsigned char* to = out_b + (static_cast<size_t>(g >> 2) * a.out_stride + out_row) * 16 + (g >> 1 & 1) * 8;
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
                        const float other = swap_f(acc[i][0][0], acc[i][0][1]);
                        if (TILE * i < left) *reinterpret_cast<float2*>(to + TILE * i * 16) = odd ? make_float2(other, acc[i][0][1]) : make_float2(acc[i][0][0], other);
                    }
                }
                else if (a.out_split) {
                    __half2 largest = __float2half2_rn(0.0f);
                    if constexpr (COUT == 16) {
                        unsigned char* to  = out_b + out_row * ROW + tq * 16;
                        const size_t plane = static_cast<size_t>(a.out_stride) * 16;
                        if (a.out_split == SPLIT_PLANES) to = out_b + (tq >> 1) * plane + out_row * 16 + (tq & 1) * 8;
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
                            uint32_t h[2], l[2];
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                split_pair(acc[i][0][2 * k], acc[i][0][2 * k + 1], h[k], l[k]);
                                largest = __hmax2(largest, __habs2(*reinterpret_cast<const __half2*>(&h[k])));
                            }
                            const uint4 piece = make_uint4(transpose(h[0]), transpose(h[1]), transpose(l[0]), transpose(l[1]));
                            if (TILE * i >= left) continue;
                            if (a.out_split == SPLIT_QUADS) { *reinterpret_cast<uint4*>(to + TILE * i * ROW) = piece; }
                            else {
                                *reinterpret_cast<uint2*>(to + TILE * i * 16)             = make_uint2(piece.x, piece.y);
                                *reinterpret_cast<uint2*>(to + 2 * plane + TILE * i * 16) = make_uint2(piece.z, piece.w);
                            }
                        }
                    }
                    else {
                        // 32 channels, the thread's 4 g .. 4 g + 3 of either row: a piece of it, or eight bytes of the hi and of the lo planes
                        const size_t plane = static_cast<size_t>(a.out_stride) * 16;
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                uint32_t h[2], l[2];
#pragma unroll
                                for (int m = 0; m < MBLK; ++m) {
                                    split_pair(acc[i][m][k], acc[i][m][2 + k], h[m], l[m]);
                                    largest = __hmax2(largest, __habs2(*reinterpret_cast<const __half2*>(&h[m])));
                                }
                                if (TILE * i + k >= left) continue;
                                const size_t row = out_row + TILE * i + k;
                                if (a.out_split == SPLIT_ROWS) {
                                    // the halves of odd rows lie the other way round
                                    reinterpret_cast<uint4*>(out_b)[row * 8 + (g ^ (static_cast<int>(row & 1) * 4))] = make_uint4(h[0], l[0], h[MBLK - 1], l[MBLK - 1]);
                                    continue;
                                }
                                unsigned char* dst                     = out_b + (g >> 1) * plane + row * 16 + (g & 1) * 8;
                                *reinterpret_cast<uint2*>(dst)             = make_uint2(h[0], h[MBLK - 1]);
                                *reinterpret_cast<uint2*>(dst + 4 * plane) = make_uint2(l[0], l[MBLK - 1]);
                            }
                        }
                    }
                    if (__hgt(__hmax(__low2half(largest), __high2half(largest)), __float2half_rn(60000.0f))) raise_flag(a.range_flag, ABORT_TC_RANGE);
                }
                else {
                    // chunk-planar fp32
                    unsigned char* to = out_b + (static_cast<size_t>(COUT == 16 ? g >> 1 : g) * a.out_stride + out_row) * 16;
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
                        if constexpr (COUT == 16) {
                            const float o0 = swap_f(acc[i][0][0], acc[i][0][1]), o1 = swap_f(acc[i][0][2], acc[i][0][3]);
                            const float4 v = odd ? make_float4(o0, acc[i][0][1], o1, acc[i][0][3]) : make_float4(acc[i][0][0], o0, acc[i][0][2], o1);
                            if (TILE * i < left) *reinterpret_cast<float4*>(to + TILE * i * 16) = v;
                        }
                        else {
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                if (TILE * i + k >= left) continue;
                                *reinterpret_cast<float4*>(to + (TILE * i + k) * 16) =
                                  make_float4(acc[i][0][k], acc[i][0][2 + k], acc[i][MBLK - 1][k], acc[i][MBLK - 1][2 + k]);
                            }
                        }
                    }
                }
            }
            // this warp is done with the window: the loader may refill it once every compute warp has said so
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar_empty + 8 * b);
        }
        }
        __syncthreads();
        if (tid == 0 && failed_s) raise_flag(t.abort_flags, ABORT_TC_TIMEOUT);
    }

}  // namespace st
}  // namespace vm
