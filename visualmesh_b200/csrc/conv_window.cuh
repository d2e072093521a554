// Graph-convolution layer with 32 input channels on the 5th-generation tensor cores, its gather served from shared-memory windows.
//
// out[row] = act(bias + sum_s X[nbr_s(row)] . W_s) reads every feature row once per row it is a neighbour of: 9 times for eight
// neighbours. The rows of a frame are cut into super-tiles of 256 rows with a halo list each (tile_plan.cuh); a loader warp brings
// super-tile and halo into shared memory, windows ahead of their use, and the gather reads shared memory only. The gathered rows
// become the A operand of tcgen05.mma in tensor memory.
//
// Features travel between such layers as two fp16 parts (x = hi + lo), row after row (SPLIT_ROWS): eight pieces of 16 bytes, each two
// hi, two lo, two hi and two lo parts. Weights are split the same way, and all four products are added up in fp32. A feature row is two
// rows of the MMA, its hi parts and its lo parts (64 rows a tile), and the K axis may come in any order that both operands share. So
//   - four threads read a row, 16 bytes each of either half, and what a load leaves in four registers is what the tcgen05.st shape
//     that spreads a row over four threads (16x128b) takes: no register is moved. (With hi and lo parts as columns of one row of
//     the MMA, the registers of two loads had to be interleaved: 13 of 47 M instructions of a launch.)
//   - odd rows lie with their second half first: two rows of different parity, which a quarter-warp reads together, never meet in a bank.
//   - the columns of D are permuted so that the epilogue's thread holds neighbouring output channels of a row, four threads a row:
//     features are written in whole 32-byte sectors without a detour through shared memory.
//
// Roles: two gather groups of four warps, each with one tile's A in tensor memory, one accumulator and a warp that issues its MMAs (the
// weights' hi and lo parts side by side as N, so half as many to issue); a group of four warps for the epilogue; two loader warps. They
// meet at mbarriers only. A is stored, multiplied and given back in two parts, so that one is multiplied while the other is stored.
// Windows take as many rows of a common pool as their super-tile and halo have (369 on average with eight neighbours, 587 at most).
//
// What bounds it: clocks read by each role (eight neighbours, 7.4 M rows) show the epilogue at work 83 % of the time, the gather 72 %,
// with the load/store path near its rate in between; under the power limit the SM clock falls to 1.55 GHz in this kernel. A tile takes
// 1290 cycles. Measured on the way, 32 -> 32, one frame of 0.92 M rows | eight frames: 110 | 762 us at first (units of three slots in a
// ring, A as two loads interleaved, one issuer); registers in order but more and smaller units 127 | 870 - the issuer and the chain of
// barriers were what took the time, with row loads, stores to tensor memory or the epilogue left out one by one it stayed the same;
// a tile's A as one unit 107 | 742; in two parts with an issuer per group 102 | 706; windows from a pool 85 | 631 (the
// mean of eight layers, as the others; the last, which writes fp32, 610): before, a
// super-tile with more than 192 halo rows (3 % of them) was gathered by a slow path, and the CTAs that had two or three of those
// finished 25 % later than the others; and one loader warp was busy all along. Four and six steps of loads in flight instead of two: 2 %.
// Sixteen gather or epilogue warps (96 registers): 5 to 17 % slower. Registers shared out with setmaxnreg: 9 % slower.
//
// Every wait is bounded: a wait that runs out raises the abort flag, the CTA stops issuing work, waits (bounded) for its own copies
// and MMAs, frees its tensor memory and returns. No multicast; all copies read this GPU's own memory.
#pragma once

#include <type_traits>

#include "conv_tc.cuh"
#include "tile_plan.cuh"

namespace vm {
namespace win {

    constexpr int ST            = st::ST;
    constexpr int HALO          = st::HALO;
    constexpr int CIN           = 32;
    constexpr int ROW           = 4 * CIN;  // bytes of a feature row: hi part, lo part
    constexpr int TILE          = 64;       // feature rows of one MMA tile: their hi and their lo parts are its 128 rows
    constexpr int GATHER_GROUPS = 2;        // groups of four warps: the rows of one MMA tile
    constexpr int GATHER_WARPS  = 4 * GATHER_GROUPS;
    constexpr int OUT_WARPS     = 4;
    constexpr int LOADER        = GATHER_WARPS + OUT_WARPS;
    constexpr int LOADERS       = 2;
    constexpr int ISSUER        = LOADER + LOADERS;
    constexpr int THREADS       = 32 * (ISSUER + GATHER_GROUPS);  // an issuer for each gather group
    constexpr int BUFFERS       = 3;     // windows that are being read or on their way
    constexpr int POOL          = 1344;  // rows of the windows together: a window takes as many as its super-tile and its halo have
    constexpr int NBL_BYTES     = ST * st::NBL_STRIDE * 2;
    static_assert(ST + HALO <= POOL / 2, "a window fits beside the one that is being read");

    struct Args {
        const void* weights;  // [slot][4 chunks of K][NP rows of hi parts, NP rows of lo parts][16 bytes], permuted
        const float* bias;    // [NP], in channel order
        int32_t n_frames;
        int32_t cout;
        int32_t* abort_flags;
        uint32_t wait_limit;  // polls of one wait before the kernel gives up (0: every wait fails at once)
    };

    // channel pair of a row that column c of a slot's A holds
    __host__ __device__ constexpr int pair_of_column(int c) {
        return 8 * (c / 8) + 2 * (c % 4) + c / 4 % 2;
    }
    // output channel of column n of D
    __host__ __device__ constexpr int channel_of_column(int np, int n) {
        return (np / 4) * ((n % 8) / 2) + 2 * (n / 8) + n % 2;
    }
    // A gather group has one tile's A in tensor memory, and an accumulator. The A is stored and multiplied in two parts: one is
    // multiplied while the other is stored.
    template <int NP, int NSLOTS>
    struct Parts {
        static constexpr int FIRST = (NSLOTS + 1) / 2;   // slots of the first part
        static constexpr int COLS  = NSLOTS * CIN / 2;   // tensor-memory columns of a tile: a column holds two fp16 values
        static_assert(GATHER_GROUPS * (COLS + 2 * NP) <= 512, "all tensor memory there is");
    };

    template <int NP>
    __host__ __device__ constexpr size_t smem_bytes(int n_slots) {
        return static_cast<size_t>(POOL) * ROW + static_cast<size_t>(BUFFERS) * NBL_BYTES + static_cast<size_t>(n_slots) * 4 * 2 * NP * 16;
    }

    using tc::bulk_copy;
    using tc::copies_arrive;
    using tc::copy16;
    using tc::expect_bytes;
    using tc::load_shared;
    __device__ __forceinline__ uint32_t load_position(uint32_t addr) {
        uint32_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr));
        return v;
    }
    // Whether both loader warps may go on. A window is filled by both or by neither: one that a single loader had begun would never become
    // full, and the other's wait for its copies at the end would last until the default limit runs out.
    __device__ __forceinline__ bool loaders_agree(bool ok) {
        uint32_t r;
        asm volatile(
          "{\n\t"
          ".reg .pred p, q;\n\t"
          "setp.ne.u32 p, %1, 0;\n\t"
          "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
          "selp.u32 %0, 1, 0, q;\n\t"
          "}\n"
          : "=r"(r)
          : "r"(static_cast<uint32_t>(ok)), "n"(32 * LOADERS)
          : "memory");
        return r != 0;
    }
    // one lane of a converged warp; what it alone does keeps its operands uniform
    __device__ __forceinline__ bool elect_one() {
        uint32_t r;
        asm volatile(
          "{\n\t"
          ".reg .pred p;\n\t"
          "elect.sync _|p, 0xffffffff;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t"
          "}\n"
          : "=r"(r));
        return r != 0;
    }
    // D = A . B (+ D), A in tensor memory
    template <bool ADD>
    __device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint32_t b_low, uint32_t b_high, uint32_t idesc) {
        asm volatile(
          "{\n\t"
          ".reg .pred p;\n\t"
          ".reg .b64 b;\n\t"
          "mov.b64 b, {%2, %3};\n\t"
          "setp.ne.b32 p, %5, 0;\n\t"
          "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t"
          "}\n" ::"r"(d),
          "r"(a), "r"(b_low), "r"(b_high), "r"(idesc), "n"(ADD ? 1 : 0)
          : "memory");
    }
    // Sixteen rows of tensor memory, a row over four threads: register 2 i + j of thread t is column (t % 4) + 4 i of row t / 4 + 8 j.
    __device__ __forceinline__ void store_a(uint32_t taddr, const uint4& a, const uint4& b) {
        asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                     "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                     : "memory");
    }
    // Sixteen rows of 16 columns: register 4 i + 2 j + e of thread t is column 8 i + 2 (t % 4) + e of row t / 4 + 8 j.
    __device__ __forceinline__ void load_d(uint32_t taddr, uint32_t* r) {
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    }

    // a thread's pieces of one row: four channels of the first and of the second half
    struct Gathered {
        uint4 v[2];
    };

    template <int NP, int NSLOTS>
    __global__ void __launch_bounds__(THREADS, 1) k_graph_conv_window(const ConvArgs a, const Args t, const st::Plan plan) {
        static_assert((NP == 16 || NP == 32) && HALO % 32 == 0, "shapes the layouts above are written for");
        using Part             = Parts<NP, NSLOTS>;
        constexpr int WCHUNK   = 2 * NP * 16;
        constexpr int OWN      = NP / 4;     // output channels of a thread
        constexpr int ACC_COLS = 2 * NP;     // products with the weights' hi parts, then with their lo parts
        constexpr int A_COLUMN = GATHER_GROUPS * ACC_COLS;  // first tensor-memory column of A, behind the accumulators

        extern __shared__ __align__(1024) unsigned char smem_raw[];
        // window: full, free; per group: the two parts of A stored, multiplied (it may be overwritten; after the second part the accumulator is
        // full), accumulator free, drain
        __shared__ uint64_t bars[2 * BUFFERS + 6 * GATHER_GROUPS];
        __shared__ uint32_t tmem_base_slot;
        __shared__ int32_t window_miss[BUFFERS];             // some neighbour of the super-tile was left out of its window
        __shared__ int32_t tile_prefix[tc::MAX_FRAMES + 1];  // in super-tiles
        __shared__ int32_t frame_start[tc::MAX_FRAMES + 1];  // offsets[f0 + f]
        __shared__ int32_t window_start[BUFFERS];            // its first row in the pool
        __shared__ int32_t halo_s[LOADERS][HALO];            // the halo list of the window that is being filled
        __shared__ int32_t failed_s;
        volatile int32_t* failed = &failed_s;

        const int tid  = threadIdx.x;
        const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
        const int lane = tid & 31;
        const uint32_t win_addr     = tc::smem_u32(smem_raw);
        const uint32_t nbl_addr     = win_addr + POOL * ROW;
        const uint32_t w_addr       = nbl_addr + BUFFERS * NBL_BYTES;
        const uint32_t bar_full     = tc::smem_u32(&bars[0]);
        const uint32_t bar_free     = bar_full + 8 * BUFFERS;
        const uint32_t bar_stored   = bar_free + 8 * BUFFERS;
        const uint32_t bar_done     = bar_stored + 16 * GATHER_GROUPS;
        const uint32_t bar_acc_free = bar_done + 16 * GATHER_GROUPS;
        const uint32_t bar_drain    = bar_acc_free + 8 * GATHER_GROUPS;

        if (tid == 0) {
            failed_s = 0;
            for (int i = 0; i < BUFFERS; ++i) {
                tc::mbar_init(bar_full + 8 * i, 1 + 32 * LOADERS);  // the bulk copies' byte count + one arrival per loader lane
                tc::mbar_init(bar_free + 8 * i, GATHER_WARPS);
            }
            for (int i = 0; i < 2 * GATHER_GROUPS; ++i) {
                tc::mbar_init(bar_stored + 8 * i, 4);  // the warps of a gather group
                tc::mbar_init(bar_done + 8 * i, 1);    // a commit
            }
            for (int i = 0; i < GATHER_GROUPS; ++i) {
                tc::mbar_init(bar_acc_free + 8 * i, OUT_WARPS);
                tc::mbar_init(bar_drain + 8 * i, 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int f = tid; f <= t.n_frames; f += THREADS) frame_start[f] = a.offsets[a.f0 + f];
        {
            const uint4* g = reinterpret_cast<const uint4*>(t.weights);
            uint4* sw      = reinterpret_cast<uint4*>(smem_raw + POOL * ROW + BUFFERS * NBL_BYTES);
            for (int i = tid; i < NSLOTS * 4 * 2 * NP; i += THREADS) sw[i] = __ldg(g + i);
        }
        __syncthreads();
        tc::tiles_before<ST>(tile_prefix, frame_start, t.n_frames);
        if (warp == ISSUER) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_base_slot)), "r"(512) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_base = tmem_base_slot;

        // An item is a super-tile, all of its MMA tiles, or half of them where that leaves no SM without work.
        const int total_st    = tile_prefix[t.n_frames];
        const int halves      = 2 * total_st <= static_cast<int>(gridDim.x) ? 1 : 0;
        const int total_items = total_st << halves;
        struct Item {
            int rows;        // rows of the frame, off-screen row included
            int t0;          // first row of the super-tile within the frame
            int local_base;  // first feature row of the frame in this launch
            int first, end;  // MMA tiles of the super-tile
        };
        // items only move forward: shared memory is read when a frame begins
        int frame = -1, st_begin = 0, st_end = 0, frame_rows = 0, frame_base = 0;
        auto locate = [&](int item) {
            const int s = item >> halves;
            while (s >= st_end) {
                ++frame;
                st_begin   = st_end;
                st_end     = tile_prefix[frame + 1];
                frame_rows = frame_start[frame + 1] - frame_start[frame] + 1;
                frame_base = frame_start[frame] - frame_start[0] + frame;
            }
            Item r;
            r.rows       = frame_rows;
            r.t0         = (s - st_begin) * ST;
            r.local_base = frame_base;
            r.first      = halves ? (item & 1) * (ST / TILE / 2) : 0;
            r.end        = min(halves ? r.first + ST / TILE / 2 : ST / TILE, (r.rows - r.t0 + TILE - 1) / TILE);
            return r;
        };
        // first neighbourhood row of the frame
        auto neighbourhood_base = [&] { return static_cast<size_t>(frame_start[frame] + a.f0 + frame); };
        const unsigned char* in_bytes = reinterpret_cast<const unsigned char*>(a.in);
        // the whole warp waits, and decides together whether to go on
        auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
            bool done = false;
            for (uint32_t i = 0; i < t.wait_limit && !done; ++i) {
                done = tc::mbar_try_wait(bar, parity);
                if (!done && (i & 1023u) == 1023u && *failed) break;
            }
            if (__all_sync(0xffffffffu, done)) return true;
            *failed = 1;
            return false;
        };

        if (warp >= LOADER && warp < LOADER + LOADERS) {
            // ================= loader: windows ahead of the gather =================
            // The halo list of a super-tile is read one super-tile ahead, as much of it as most have. Both warps walk all windows, each
            // copies every other four halo rows: one warp took 4500 cycles per window, its requests queueing with those of the gather.
            constexpr int EARLY    = 192;
            constexpr int PER_LANE = EARLY / 32;
            constexpr int LPR      = ROW / 16;        // lanes that copy one halo row
            constexpr int STEP     = LOADERS * (32 / LPR);
            constexpr int BATCH    = 8;
            const int loader       = warp - LOADER;
            struct HaloList {
                int count;
                int32_t row[PER_LANE];
            };
            auto fetch_halo_list = [&](HaloList& l, int item) {
                const int s           = item >> halves;
                l.count               = __ldg(plan.halo_count + s);
                const int32_t* h_rows = plan.halo_rows + static_cast<size_t>(s) * HALO;
#pragma unroll
                for (int k = 0; k < PER_LANE; ++k) l.row[k] = __ldg(h_rows + lane + 32 * k);  // entries past the count are never used
            };
            int32_t* halo = halo_s[loader];
            uint32_t n = 0, buf = 0, phase = 0;
            // the windows before: [0] the last, [1] the one before it
            int start[2] = {0, 0}, end[2] = {0, 0};
            HaloList next = {};
            if (static_cast<int>(blockIdx.x) < total_items) fetch_halo_list(next, blockIdx.x);
            in_bytes = after_previous(in_bytes);
            for (int item = blockIdx.x; item < total_items; item += gridDim.x, ++n) {
                const HaloList list = next;
                if (item + static_cast<int>(gridDim.x) < total_items) fetch_halo_list(next, item + gridDim.x);
                bool there = n < BUFFERS || wait(bar_free + 8 * buf, phase ^ 1u);
                const int n_halo = min(list.count, HALO);
                // behind the last window, or from the pool's beginning; whatever window lies there still must have been read
                const int size = ST + n_halo;
                const int at   = end[0] + size <= POOL ? end[0] : 0;
#pragma unroll
                for (int back = 2; back >= 1; --back) {
                    const bool meets = n >= static_cast<uint32_t>(back) && at < end[back - 1] && start[back - 1] < at + size;
                    const uint32_t m = n - back;
                    if (there && meets) there = wait(bar_free + 8 * (m % BUFFERS), (m / BUFFERS) & 1u);
                }
                if (!loaders_agree(there)) break;
                start[1] = start[0];
                end[1]   = end[0];
                start[0] = at;
                end[0]   = at + size;
                const Item r       = locate(item);
                const int own      = min(ST, r.rows - r.t0);
                const uint32_t dst = win_addr + at * ROW;
                const uint32_t bar = bar_full + 8 * buf;
                if (loader == 0 && lane == 0) {
                    window_miss[buf]  = list.count > HALO;
                    window_start[buf] = at;
                    expect_bytes(bar, static_cast<uint32_t>(own * (ROW + 2 * st::NBL_STRIDE)));
                    bulk_copy(nbl_addr + buf * NBL_BYTES, reinterpret_cast<const uint4*>(plan.nbl) + r.local_base + r.t0,
                              static_cast<uint32_t>(own * 2 * st::NBL_STRIDE), bar);
                    bulk_copy(dst, in_bytes + static_cast<size_t>(r.local_base + r.t0) * ROW, static_cast<uint32_t>(own * ROW), bar);
                }
#pragma unroll
                for (int k = 0; k < PER_LANE; ++k) halo[lane + 32 * k] = list.row[k];
                for (int k = EARLY + lane; k < n_halo; k += 32) halo[k] = __ldg(plan.halo_rows + static_cast<size_t>(item >> halves) * HALO + k);
                __syncwarp();
                // LPR lanes to a row: whole rows per request; pieces of a row that goes to a place of other parity trade halves
                const int first           = loader * (32 / LPR) + lane / LPR;
                const unsigned char* feat = in_bytes + (lane % LPR) * 16;
                const uint32_t to         = dst + ST * ROW + (lane % LPR) * 16;
                const uint32_t place      = static_cast<uint32_t>(first + r.local_base + r.t0);  // parity of this lane's places: they are an even number apart
                for (int h = first; h < n_halo; h += BATCH * STEP) {
                    int32_t row[BATCH];  // read before the first copy: their latencies overlap
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) row[k] = halo[min(h + k * STEP, HALO - 1)];
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) {
                        if (h + k * STEP < n_halo) copy16((to + (h + k * STEP) * ROW) ^ ((place ^ row[k]) & 1u) << 6, feat + static_cast<size_t>(row[k]) * ROW);
                    }
                }
                __syncwarp();
                copies_arrive(bar);
                if (++buf == BUFFERS) {
                    buf = 0;
                    phase ^= 1u;
                }
            }
            // Nothing may still be writing this CTA's shared memory when it exits. On the normal path the gather has waited for every
            // window; after a wait ran out the last windows may still be on their way: this lane's own 16-byte copies are waited for
            // here, the bulk copies through the windows' barriers (a window is the last one issued into its buffer, so its barrier's
            // phase can only be pending or complete), with the full default limit.
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (lane == 0) {
                for (uint32_t m = n > BUFFERS ? n - BUFFERS : 0; m < n; ++m) tc::mbar_wait(bar_full + 8 * (m % BUFFERS), (m / BUFFERS) & 1u, tc::WAIT_LIMIT);
            }
        }
        else if (warp >= ISSUER) {
            // ================= MMAs of a gather group's tiles, issued by one lane =================
            constexpr uint32_t IDESC = (1u << 4) | (static_cast<uint32_t>(tc::TILE_ROWS >> 4) << 24) | (static_cast<uint32_t>(ACC_COLS >> 3) << 17);
            const uint64_t b0        = tc::smem_desc(w_addr, WCHUNK, 128);
            const uint32_t b_high    = static_cast<uint32_t>(b0 >> 32);
            const int group          = warp - ISSUER;
            const uint32_t d         = tmem_base + group * ACC_COLS;
            const uint32_t a0        = tmem_base + A_COLUMN + group * Part::COLS;
            const uint32_t stored    = bar_stored + 16 * group, done = bar_done + 16 * group;
            uint32_t phase = 0;
            int turn = 0;
            bool ok  = true;
            in_bytes = wait_previous(in_bytes);
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                const Item r = locate(item);
                for (int tile = r.first; tile < r.end; ++tile) {
                    const bool mine = turn == group;
                    if (++turn == GATHER_GROUPS) turn = 0;
                    if (!mine) continue;
                    ok = wait(bar_acc_free + 8 * group, phase ^ 1u) && wait(stored, phase);  // the accumulator is free the first time
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t b_low = static_cast<uint32_t>(b0);
                    asm volatile("" : "+r"(b_low));  // keeps the descriptors of all slots from being held in registers all along
                    constexpr int FIRST = Part::FIRST * (CIN / 16);  // K steps of the first part
                    if (elect_one()) {
                        mma_ts<false>(d, a0, b_low, b_high, IDESC);
#pragma unroll
                        for (int k = 1; k < FIRST; ++k) {
                            // a K step of the weights: NP rows of hi parts, behind them NP rows of lo parts
                            mma_ts<true>(d, a0 + 8 * k, b_low + k * (2 * WCHUNK / 16), b_high, IDESC);
                        }
                        tc::commit(done);
                    }
                    __syncwarp();
                    ok = wait(stored + 8, phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
#pragma unroll
                        for (int k = FIRST; k < NSLOTS * (CIN / 16); ++k) mma_ts<true>(d, a0 + 8 * k, b_low + k * (2 * WCHUNK / 16), b_high, IDESC);
                        tc::commit(done + 8);
                    }
                    __syncwarp();
                    phase ^= 1u;
                }
            }
            // MMAs issued so far may still be running against this CTA's tensor memory and shared memory, and commits be on their way to
            // its barriers: one more commit comes after them all (bounded, with the full default limit)
            if (elect_one()) {
                tc::commit(bar_drain + 8 * group);
                tc::mbar_wait(bar_drain + 8 * group, 0u, tc::WAIT_LIMIT);
            }
            __syncwarp();
        }
        else if (warp < GATHER_WARPS) {
            // ================= gather: window -> A =================
            constexpr int DEPTH       = 4;             // steps of 8 rows of a slot whose loads are in flight
            const int group           = warp >> 2;
            const int quad            = lane >> 2;     // this thread's rows of the warp's 16: quad, quad + 8
            const int piece           = lane & 3;
            const uint32_t lanes      = static_cast<uint32_t>((warp & 3) * 32) << 16;
            const uint32_t at         = tmem_base + A_COLUMN + group * Part::COLS + lanes;
            const uint32_t stored     = bar_stored + 16 * group, done = bar_done + 16 * group;
            uint32_t buf = 0, phase = 0, done_phase = 1;  // the first waits for a part to be multiplied pass at once
            int turn = 0;  // the group whose tile is next
            bool ok  = true;
            in_bytes = wait_previous(in_bytes);
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                int last, first_tile, end_tile;
                uint32_t parity;  // 64 where even places of the window hold odd rows
                {
                    const Item r = locate(item);
                    last         = min(ST, r.rows - r.t0) - 1;
                    first_tile   = r.first;
                    end_tile     = r.end;
                    parity       = static_cast<uint32_t>(r.local_base + r.t0) << 6 & 64u;
                }
                ok = wait(bar_full + 8 * buf, phase);
                if (!ok) break;
                const uint32_t base = win_addr + *static_cast<volatile int32_t*>(&window_start[buf]) * ROW + piece * 16;
                const bool miss     = *static_cast<volatile int32_t*>(&window_miss[buf]) != 0;
                for (int tile = first_tile; ok && tile < end_tile; ++tile) {
                    const int first_row = tile * TILE + (warp & 3) * 16 + quad;  // within the super-tile
                    auto fill = [&]() -> bool {
                        constexpr int STEPS = 2 * NSLOTS;
                        uint32_t own[2];  // rows past the super-tile's last are stored as copies of it
                        uint4 pos[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) own[j] = static_cast<uint32_t>(min(first_row + 8 * j, last));
#pragma unroll
                        for (int j = 0; j < 2; ++j) pos[j] = load_shared(nbl_addr + buf * NBL_BYTES + own[j] * 16);
                        auto position = [&](int j, int slot) -> uint32_t {
                            if (slot == 0) return own[j];
                            const int k         = slot - 1;
                            const uint32_t word = (k >> 1) == 0 ? pos[j].x : (k >> 1) == 1 ? pos[j].y : (k >> 1) == 2 ? pos[j].z : pos[j].w;
                            return (k & 1) ? (word >> 16) : (word & 0xFFFFu);
                        };
                        auto load = [&](Gathered& to, uint32_t p) {
                            const uint32_t at = base + p * ROW + ((p << 6 ^ parity) & 64u);
                            to.v[0]           = load_shared(at);
                            to.v[1]           = load_shared(at ^ 64u);
                        };
                        auto gather       = [&](Gathered& to, int step) { load(to, position(step & 1, step / 2)); };
                        auto store        = [&](const Gathered& g, int step) {
                            store_a(at + (step / 2) * (CIN / 2) + (static_cast<uint32_t>(16 * (step & 1)) << 16), g.v[0], g.v[1]);
                        };
                        // a part of the tile: the MMAs that read its tensor memory last must be done, then it is handed over
                        auto begin_part = [&](int part) -> bool {
                            if (!wait(done + 8 * part, done_phase)) return false;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            return true;
                        };
                        auto end_part = [&](int part) {
                            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive(stored + 8 * part);
                        };
                        constexpr int SECOND = 2 * Part::FIRST;  // first step of the second part
                        Gathered x[DEPTH];
                        if (!miss) {
#pragma unroll
                            for (int step = 0; step < DEPTH; ++step) gather(x[step], step);
                            if (!begin_part(0)) return false;
#pragma unroll
                            for (int step = 0; step < STEPS; ++step) {
                                if (step == SECOND) {
                                    end_part(0);
                                    if (!begin_part(1)) return false;
                                }
                                store(x[step % DEPTH], step);
                                if (step + DEPTH < STEPS) gather(x[step % DEPTH], step + DEPTH);
                            }
                        }
                        else {
                            // some rows have to come from global memory
                            const Item f         = locate(item);
                            const size_t nb_base = neighbourhood_base() + f.t0;
#pragma unroll 1
                            for (int step = 0; step < STEPS; ++step) {
                                if (step == SECOND) end_part(0);
                                if ((step == 0 || step == SECOND) && !begin_part(step / SECOND)) return false;
                                const int slot   = step / 2;
                                const int row    = min(first_row + 8 * (step & 1), last);
                                const uint32_t p = slot == 0 ? static_cast<uint32_t>(row) : load_position(nbl_addr + buf * NBL_BYTES + row * 16 + 2 * (slot - 1));
                                if (slot > 0 && p == st::NBL_GLOBAL) {
                                    const int idx            = f.local_base + __ldg(a.nb + (nb_base + row) * a.n_neighbours + (slot - 1));
                                    const unsigned char* src = in_bytes + static_cast<size_t>(idx) * ROW + piece * 16;
#pragma unroll
                                    for (int h = 0; h < 2; ++h) x[0].v[h] = *reinterpret_cast<const uint4*>(src + 64 * ((h ^ idx) & 1));
                                }
                                else {
                                    load(x[0], p);
                                }
                                __syncwarp();
                                store(x[0], step);
                            }
                        }
                        end_part(1);
                        done_phase ^= 1u;
                        return true;
                    };
                    if (turn == group) ok = fill();
                    if (++turn == GATHER_GROUPS) turn = 0;
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(bar_free + 8 * buf);  // the warp has read all it needs of the window
                if (++buf == BUFFERS) {
                    buf = 0;
                    phase ^= 1u;
                }
            }
        }
        else {
            // ================= epilogue: accumulator -> registers -> bias, activation -> global =================
            const int quad       = lane >> 2;
            const int piece      = lane & 3;
            const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
            float bias[OWN];
#pragma unroll
            for (int j = 0; j < OWN; ++j) bias[j] = __ldg(t.bias + piece * OWN + j);
            uint32_t acc = 0, phase = 0;
            bool ok  = true;
            in_bytes = wait_previous(in_bytes);
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                const Item r = locate(item);
                for (int tile = r.first; ok && tile < r.end; ++tile) {
                    ok = wait(bar_done + 16 * acc + 8, phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    float v[2][OWN];  // rows first_row, + 8
                    uint32_t d[2][ACC_COLS / 2];  // all columns of the hi and lo parts of 8 rows over 32 threads
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
#pragma unroll
                        for (int c = 0; c < ACC_COLS; c += 16) load_d(tmem_base + acc * ACC_COLS + lanes + (static_cast<uint32_t>(16 * h) << 16) + c, d[h] + c / 2);
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
#pragma unroll
                        for (int i = 0; i < OWN; ++i) {
                            const int at   = 4 * (i / 2) + i % 2;
                            const float hi = __uint_as_float(d[h][at]) + __uint_as_float(d[h][NP / 2 + at]);
                            const float lo = __uint_as_float(d[h][at + 2]) + __uint_as_float(d[h][NP / 2 + at + 2]);
                            v[h][i]        = (hi + lo) + bias[i];
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(bar_acc_free + 8 * acc);
                    if (++acc == GATHER_GROUPS) {
                        acc = 0;
                        phase ^= 1u;
                    }
                    const int first_row = r.t0 + tile * TILE + (warp & 3) * 16 + quad;  // within the frame
                    if (a.activation == VM_SOFTMAX) {
                        // exp of each, summed in channel order from thread to thread of the row
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            float total = 0.0f;
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                if (piece == q) {
#pragma unroll
                                    for (int i = 0; i < OWN; ++i) {
                                        if (q * OWN + i < t.cout) {
                                            v[j][i] = expf(v[j][i]);
                                            total   = __fadd_rn(total, v[j][i]);
                                        }
                                    }
                                }
                                total = __shfl_sync(0xffffffffu, total, (lane & ~3) | q);
                            }
#pragma unroll
                            for (int i = 0; i < OWN; ++i) v[j][i] = __fdiv_rn(v[j][i], total);
                        }
                    }
                    else {
#pragma unroll
                        for (int j = 0; j < 2; ++j) activate<OWN>(v[j], a.activation);
                    }
                    const int rows = r.rows - first_row;  // row j exists: 8 * j < rows
                    if (a.out_split) {
                        uint32_t hi[2][OWN / 2], lo[2][OWN / 2];
                        __half2 largest = __float2half2_rn(0.0f);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
#pragma unroll
                            for (int i = 0; i < OWN / 2; ++i) {
                                split_pair(v[j][2 * i], v[j][2 * i + 1], hi[j][i], lo[j][i]);
                                largest = __hmax2(largest, __habs2(*reinterpret_cast<const __half2*>(&hi[j][i])));
                            }
                        }
                        if (a.out_split == SPLIT_ROWS) {
                            // 32 channels, two pieces of a row; the halves of odd rows lie the other way round
                            const size_t row = static_cast<size_t>(r.local_base) + first_row;
                            uint4* dst       = reinterpret_cast<uint4*>(a.out) + row * 8 + ((2 * piece) ^ (static_cast<int>(row & 1) * 4));
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (OWN == 8 && 8 * j < rows) {
                                    dst[64 * j]     = make_uint4(hi[j][0], lo[j][0], hi[j][1], lo[j][1]);
                                    dst[64 * j + 1] = make_uint4(hi[j][OWN / 2 - 2], lo[j][OWN / 2 - 2], hi[j][OWN / 2 - 1], lo[j][OWN / 2 - 1]);
                                }
                            }
                        }
                        else if (a.out_split == SPLIT_QUADS) {
                            // 16 channels; pieces of four hi and four lo parts
                            if (OWN == 4) {
                                uint4* dst = reinterpret_cast<uint4*>(a.out) + (static_cast<size_t>(r.local_base) + first_row) * 4 + piece;
#pragma unroll
                                for (int j = 0; j < 2; ++j) {
                                    if (8 * j < rows) dst[32 * j] = make_uint4(hi[j][0], hi[j][1], lo[j][0], lo[j][1]);
                                }
                            }
                        }
                        else {
                            // planes of 16-byte chunks of 8 channels, the hi planes first
                            const int n        = piece * OWN < t.cout ? rows : 0;
                            const size_t row   = static_cast<size_t>(r.local_base) + first_row;
                            unsigned char* out = reinterpret_cast<unsigned char*>(a.out) + (piece * OWN % 8) * 2;
                            const size_t plane = piece * OWN / 8, lo_planes = t.cout / 8;
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (8 * j >= n) continue;
                                unsigned char* dst_hi = out + (plane * a.out_stride + row + 8 * j) * 16;
                                unsigned char* dst_lo = out + ((plane + lo_planes) * a.out_stride + row + 8 * j) * 16;
#pragma unroll
                                for (int i = 0; i < OWN / 2; ++i) {
                                    reinterpret_cast<uint32_t*>(dst_hi)[i] = hi[j][i];
                                    reinterpret_cast<uint32_t*>(dst_lo)[i] = lo[j][i];
                                }
                            }
                        }
                        if (__hgt(__hmax(__low2half(largest), __high2half(largest)), __float2half_rn(60000.0f))) raise_flag(a.range_flag, ABORT_TC_RANGE);
                    }
                    else if (a.out_planar) {
#pragma unroll
                        for (int c = 0; c < OWN / 4; ++c) {
                            const int n = piece * OWN + 4 * c < t.cout ? rows : 0;
                            float4* dst = reinterpret_cast<float4*>(a.out) + static_cast<size_t>(piece * (OWN / 4) + c) * a.out_stride + r.local_base + first_row;
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (8 * j < n) dst[8 * j] = make_float4(v[j][4 * c], v[j][4 * c + 1], v[j][4 * c + 2], v[j][4 * c + 3]);
                            }
                        }
                    }
                    else {
                        const size_t out_base = a.out_global ? neighbourhood_base() : static_cast<size_t>(r.local_base);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            if (8 * j >= rows) continue;
                            float* dst = a.out + (out_base + first_row + 8 * j) * t.cout + piece * OWN;
#pragma unroll
                            for (int i = 0; i < OWN; ++i) {
                                if (piece * OWN + i < t.cout) dst[i] = v[j][i];
                            }
                        }
                    }
                }
            }
        }

        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0 && failed_s) raise_flag(t.abort_flags, ABORT_TC_TIMEOUT);
        if (warp == ISSUER) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
        }
    }

}  // namespace win
}  // namespace vm
