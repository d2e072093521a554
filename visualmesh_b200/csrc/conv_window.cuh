// Graph-convolution layer with 32 input channels on the 5th-generation tensor cores, its gather served from shared-memory windows.
//
// out[row] = act(bias + sum_s X[nbr_s(row)] . W_s) reads every feature row once per row it is a neighbour of: 9 times for eight
// neighbours. The rows of a frame are cut into super-tiles of 256 rows with a halo list each (tile_plan.cuh); a loader warp brings
// super-tile and halo into shared memory, windows ahead of their use, and the gather reads shared memory only. The gathered rows
// become the A operand of tcgen05.mma in tensor memory.
//
// Features travel between such layers as two fp16 parts (x = hi + lo), row after row: 32 hi values, then 32 lo values. Weights are split
// the same way, and all four products are added up in fp32. The contraction does not care in which order its K axis comes as long as
// both operands agree, nor which of the two parts of x is which, since either meets both parts of W. That freedom pays twice:
//   - four threads read one row, 16 bytes each, and store them with the tcgen05.st shape that spreads a row over four threads
//     (16x128b); the threads of every other row take the two halves of the row in opposite order, so that the two rows a quarter-warp
//     reads never meet in a bank, whatever rows they are.
//   - the columns of D are permuted so that the epilogue's thread holds neighbouring output channels of a row, four threads a row:
//     features are written in whole 32-byte sectors without a detour through shared memory.
//
// Roles: two gather groups of four warps (128 rows, one MMA tile) that store units of up to three slots of A into a ring in tensor
// memory, one warp that issues the MMAs (the weights' hi and lo parts side by side as N, so half as many to issue), a group of four
// warps for the epilogue, one loader warp. They meet at mbarriers only. 14 warps leave 128 registers a thread, and two steps of the
// gather in flight. Measured on the way here, 32 -> 32 over 7.4 M rows, against 820 us when this form was settled: three groups with 96
// registers and one step 883 us, with two steps (spills) 1064; a second group for the epilogue 970 and units of one slot 1075 (the
// barriers), either about a tenth more than the form it was tried on; hi and lo parts as two MMAs 978.
// What bounds a 128-row tile with eight neighbours (counters of one frame, 0.93 M rows): it takes 3420 cycles of its SM. The load/store
// path works 2120 of them - the gathered rows 1152 and 300 of conflicts, the stores to tensor memory, the window and the output - and
// the tensor pipe 1150; the rest is the chain load -> store -> settle -> MMA of a unit with only two groups to overlap it. The layer
// takes 761 us over 7.4 M rows, against 1394 us with the kernel that gathers with global loads (conv_tc.cuh).
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
    constexpr int GATHER_GROUPS = 2;        // groups of four warps: the 128 rows of one MMA tile
    constexpr int GATHER_WARPS  = 4 * GATHER_GROUPS;
    constexpr int OUT_WARPS     = 4;
    constexpr int LOADER        = GATHER_WARPS + OUT_WARPS;
    constexpr int ISSUER        = LOADER + 1;
    constexpr int THREADS       = 32 * (ISSUER + 1);
    constexpr int ACCS          = 2;  // accumulators: tiles between their first MMA and their epilogue's load
    constexpr int BUFFERS       = 3;  // windows that are being read or on their way
    constexpr int WINDOW        = (ST + HALO) * ROW;
    constexpr int NBL_BYTES     = ST * st::NBL_STRIDE * 2;

    struct Args {
        const void* weights;  // [slot][4 chunks of K][NP rows of hi parts, NP rows of lo parts][16 bytes], permuted
        const float* bias;    // [NP], in channel order
        int32_t n_frames;
        int32_t cout;
        int32_t* abort_flags;
        uint32_t wait_limit;  // polls of one wait before the kernel gives up (0: every wait fails at once)
    };

    // 32-bit word (channel pair) of a row's hi or lo part that column c of a slot's A holds; columns 16..31 repeat
    __host__ __device__ constexpr int pair_of_column(int c) {
        return 4 * (c % 4) + (c % 16) / 4;
    }
    // output channel of column n of D
    __host__ __device__ constexpr int channel_of_column(int np, int n) {
        return (np / 4) * ((n % 8) / 2) + 2 * (n / 8) + n % 2;
    }
    // A tile's slots are stored in units of at most three; the units in tensor memory are a ring.
    template <int NP, int NSLOTS>
    struct Units {
        static constexpr int COUNT  = (NSLOTS + 2) / 3;
        static constexpr int SLOTS  = (NSLOTS + COUNT - 1) / COUNT;
        static constexpr int COLS   = SLOTS * CIN;  // a column holds two fp16 values
        static constexpr int FIT    = (512 - ACCS * 2 * NP) / COLS;
        static constexpr int STAGES = FIT < 8 ? FIT : 8;
        static_assert(COUNT <= 3 && STAGES >= GATHER_GROUPS, "every gather group has a unit to store into");
    };

    template <int NP>
    __host__ __device__ constexpr size_t smem_bytes(int n_slots) {
        return static_cast<size_t>(BUFFERS) * (WINDOW + NBL_BYTES) + static_cast<size_t>(n_slots) * 4 * 2 * NP * 16;
    }

    __device__ __forceinline__ void expect_bytes(uint32_t bar, uint32_t bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    }
    // contiguous global -> shared, completion counted in bytes on the mbarrier; no multicast
    __device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                     : "memory");
    }
    __device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    // one arrival on the mbarrier once all earlier 16-byte copies of this thread have landed (counted at init)
    __device__ __forceinline__ void copies_arrive(uint32_t bar) {
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    }
    __device__ __forceinline__ uint4 load_shared(uint32_t addr) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
        return v;
    }
    __device__ __forceinline__ uint32_t load_position(uint32_t addr) {
        uint32_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr));
        return v;
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
    __device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool add) {
        asm volatile(
          "{\n\t"
          ".reg .pred p;\n\t"
          "setp.ne.b32 p, %4, 0;\n\t"
          "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
          "}\n" ::"r"(d),
          "r"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u)
          : "memory");
    }
    // Sixteen rows of tensor memory, a row over four threads: register 2 i + j of thread t is column (t % 4) + 4 i of row t / 4 + 8 j.
    __device__ __forceinline__ void store_a(uint32_t taddr, const uint4& a, const uint4& b) {
        asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(a.x), "r"(b.x), "r"(a.y), "r"(b.y),
                     "r"(a.z), "r"(b.z), "r"(a.w), "r"(b.w)
                     : "memory");
    }
    // Sixteen rows of 16 columns: register 4 i + 2 j + e of thread t is column 8 i + 2 (t % 4) + e of row t / 4 + 8 j.
    __device__ __forceinline__ void load_d(uint32_t taddr, uint32_t* r) {
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    }

    // a thread's pieces of one slot: two rows of the warp that are 8 apart, two halves each
    struct Gathered {
        uint4 v[2][2];
    };

    template <int NP, int NSLOTS>
    __global__ void __launch_bounds__(THREADS, 1) k_graph_conv_window(const ConvArgs a, const Args t, const st::Plan plan) {
        static_assert((NP == 16 || NP == 32) && HALO % 32 == 0, "shapes the layouts above are written for");
        using Unit             = Units<NP, NSLOTS>;
        constexpr int STAGES   = Unit::STAGES;
        constexpr int WCHUNK   = 2 * NP * 16;
        constexpr int OWN      = NP / 4;     // output channels of a thread
        constexpr int ACC_COLS = 2 * NP;     // products with the weights' hi parts, then with their lo parts
        constexpr int A_COLUMN = ACCS * ACC_COLS;  // first tensor-memory column of the units of A, behind the accumulators

        extern __shared__ __align__(1024) unsigned char smem_raw[];
        // window: full, free; unit of A: stored, read; accumulator: full, free; drain
        __shared__ uint64_t bars[2 * BUFFERS + 2 * STAGES + 2 * ACCS + 1];
        __shared__ uint32_t tmem_base_slot;
        __shared__ int32_t window_miss[BUFFERS];             // some neighbour of the super-tile was left out of its window
        __shared__ int32_t tile_prefix[tc::MAX_FRAMES + 1];  // in super-tiles
        __shared__ int32_t frame_start[tc::MAX_FRAMES + 1];  // offsets[f0 + f]
        __shared__ int32_t halo_s[HALO];                     // the halo list of the window that is being filled
        __shared__ int32_t failed_s;
        volatile int32_t* failed = &failed_s;

        const int tid  = threadIdx.x;
        const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
        const int lane = tid & 31;
        const uint32_t win_addr     = tc::smem_u32(smem_raw);
        const uint32_t nbl_addr     = win_addr + BUFFERS * WINDOW;
        const uint32_t w_addr       = nbl_addr + BUFFERS * NBL_BYTES;
        const uint32_t bar_full     = tc::smem_u32(&bars[0]);
        const uint32_t bar_free     = bar_full + 8 * BUFFERS;
        const uint32_t bar_stored   = bar_free + 8 * BUFFERS;
        const uint32_t bar_read     = bar_stored + 8 * STAGES;
        const uint32_t bar_acc_full = bar_read + 8 * STAGES;
        const uint32_t bar_acc_free = bar_acc_full + 8 * ACCS;
        const uint32_t bar_drain    = bar_acc_free + 8 * ACCS;

        if (tid == 0) {
            failed_s = 0;
            for (int i = 0; i < BUFFERS; ++i) {
                tc::mbar_init(bar_full + 8 * i, 1 + 32);  // the bulk copies' byte count + one arrival per loader lane
                tc::mbar_init(bar_free + 8 * i, GATHER_WARPS);
            }
            for (int i = 0; i < STAGES; ++i) {
                tc::mbar_init(bar_stored + 8 * i, 4);  // the warps of a gather group
                tc::mbar_init(bar_read + 8 * i, 1);    // a commit
            }
            for (int i = 0; i < ACCS; ++i) {
                tc::mbar_init(bar_acc_full + 8 * i, 1);  // a commit
                tc::mbar_init(bar_acc_free + 8 * i, OUT_WARPS);
            }
            tc::mbar_init(bar_drain, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int f = tid; f <= t.n_frames; f += THREADS) frame_start[f] = a.offsets[a.f0 + f];
        {
            const uint4* g = reinterpret_cast<const uint4*>(t.weights);
            uint4* sw      = reinterpret_cast<uint4*>(smem_raw + BUFFERS * (WINDOW + NBL_BYTES));
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

        // An item is a super-tile, both of its MMA tiles, or one of the two where that leaves no SM without work.
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
            r.first      = halves ? item & 1 : 0;
            r.end        = min(halves ? r.first + 1 : 2, (r.rows - r.t0 + tc::TILE_ROWS - 1) / tc::TILE_ROWS);
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

        if (warp == LOADER) {
            // ================= loader: windows ahead of the gather =================
            // The halo list of a super-tile is read one super-tile ahead.
            constexpr int PER_LANE = HALO / 32;
            constexpr int LPR      = ROW / 16;  // lanes that copy one halo row
            constexpr int BATCH    = 8;
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
            uint32_t n = 0, buf = 0, phase = 0;
            HaloList next = {};
            if (static_cast<int>(blockIdx.x) < total_items) fetch_halo_list(next, blockIdx.x);
            for (int item = blockIdx.x; item < total_items; item += gridDim.x, ++n) {
                const HaloList list = next;
                if (item + static_cast<int>(gridDim.x) < total_items) fetch_halo_list(next, item + gridDim.x);
                if (n >= BUFFERS && !wait(bar_free + 8 * buf, phase ^ 1u)) break;
                const Item r       = locate(item);
                const int own      = min(ST, r.rows - r.t0);
                const uint32_t dst = win_addr + buf * WINDOW;
                const uint32_t bar = bar_full + 8 * buf;
                if (lane == 0) {
                    window_miss[buf] = list.count > HALO;
                    expect_bytes(bar, static_cast<uint32_t>(own * (ROW + 2 * st::NBL_STRIDE)));
                    bulk_copy(nbl_addr + buf * NBL_BYTES, reinterpret_cast<const uint4*>(plan.nbl) + r.local_base + r.t0,
                              static_cast<uint32_t>(own * 2 * st::NBL_STRIDE), bar);
                    bulk_copy(dst, in_bytes + static_cast<size_t>(r.local_base + r.t0) * ROW, static_cast<uint32_t>(own * ROW), bar);
                }
#pragma unroll
                for (int k = 0; k < PER_LANE; ++k) halo_s[lane + 32 * k] = list.row[k];
                __syncwarp();
                // LPR lanes to a row: whole rows per request
                const int n_halo          = min(list.count, HALO);
                const unsigned char* from = in_bytes + (lane % LPR) * 16;
                const uint32_t to         = dst + ST * ROW + (lane % LPR) * 16;
                for (int h = lane / LPR; h < n_halo; h += BATCH * (32 / LPR)) {
                    int32_t row[BATCH];  // read before the first copy: their latencies overlap
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) row[k] = halo_s[min(h + k * (32 / LPR), HALO - 1)];
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) {
                        if (h + k * (32 / LPR) < n_halo) copy16(to + (h + k * (32 / LPR)) * ROW, from + static_cast<size_t>(row[k]) * ROW);
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
        else if (warp == ISSUER) {
            // ================= MMAs, issued by one lane =================
            constexpr uint32_t IDESC = (1u << 4) | (static_cast<uint32_t>(tc::TILE_ROWS >> 4) << 24) | (static_cast<uint32_t>(ACC_COLS >> 3) << 17);
            const uint64_t b0        = tc::smem_desc(w_addr, WCHUNK, 128);
            uint32_t stage = 0, stage_phase = 0, acc = 0, acc_phase = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                const Item r = locate(item);
                for (int tile = r.first; ok && tile < r.end; ++tile) {
                    ok = wait(bar_acc_free + 8 * acc, acc_phase ^ 1u);  // passes at once the first time round
                    const uint32_t d = tmem_base + acc * ACC_COLS;
#pragma unroll 1
                    for (int u = 0; ok && u < Unit::COUNT; ++u) {
                        ok = wait(bar_stored + 8 * stage, stage_phase);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (elect_one()) {
                            const uint32_t a0 = tmem_base + A_COLUMN + stage * Unit::COLS;
                            uint64_t bu       = b0 + u * (Unit::SLOTS * 4 * WCHUNK / 16);
                            asm volatile("" : "+l"(bu));  // keeps the descriptors of all slots from being held in registers all along
#pragma unroll
                            for (int i = 0; i < Unit::SLOTS; ++i) {
                                if (u * Unit::SLOTS + i < NSLOTS) {
#pragma unroll
                                    for (int ks = 0; ks < CIN / 8; ++ks) {
                                        // K step ks & 1 of the slot's weights: NP rows of hi parts, behind them NP rows of lo parts
                                        mma_ts(d, a0 + i * CIN + 8 * ks, bu + (i * 4 + (ks & 1) * 2) * (WCHUNK / 16), IDESC, u != 0 || i != 0 || ks != 0);
                                    }
                                }
                            }
                            tc::commit(bar_read + 8 * stage);
                            if (u + 1 == Unit::COUNT) tc::commit(bar_acc_full + 8 * acc);
                        }
                        __syncwarp();
                        if (++stage == STAGES) {
                            stage = 0;
                            stage_phase ^= 1u;
                        }
                    }
                    if (++acc == ACCS) {
                        acc = 0;
                        acc_phase ^= 1u;
                    }
                }
            }
            // MMAs issued so far may still be running against this CTA's tensor memory and shared memory, and commits be on their way to
            // its barriers: one more commit comes after them all (bounded, with the full default limit)
            if (elect_one()) {
                tc::commit(bar_drain);
                tc::mbar_wait(bar_drain, 0u, tc::WAIT_LIMIT);
            }
            __syncwarp();
        }
        else if (warp < GATHER_WARPS) {
            // ================= gather: window -> units of A =================
            constexpr int DEPTH       = 2;             // steps of 16 rows of a slot whose loads are in flight
            const int group           = warp >> 2;
            const int quad            = lane >> 2;     // this thread's rows of the warp's 32: quad, quad + 8, + 16, + 24
            const int piece           = lane & 3;
            const uint32_t first_half = (quad & 1) * 64;  // every other row starts with its second half
            const uint32_t lanes      = static_cast<uint32_t>((warp & 3) * 32) << 16;
            const uint32_t a_base     = tmem_base + A_COLUMN + lanes;
            uint32_t buf = 0, phase = 0, stage = 0, stage_phase = 1;  // the first waits for a unit pass at once
            int turn = 0;  // the group whose unit is next
            bool ok  = true;
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                int last, first_tile, end_tile;
                {
                    const Item r = locate(item);
                    last         = min(ST, r.rows - r.t0) - 1;
                    first_tile   = r.first;
                    end_tile     = r.end;
                }
                ok = wait(bar_full + 8 * buf, phase);
                if (!ok) break;
                const uint32_t base = win_addr + buf * WINDOW + piece * 16 + first_half;
                const bool miss     = *static_cast<volatile int32_t*>(&window_miss[buf]) != 0;
                for (int tile = first_tile; ok && tile < end_tile; ++tile) {
                    const int first_row = tile * tc::TILE_ROWS + (warp & 3) * 32 + quad;  // within the super-tile
                    auto unit = [&](auto which) {
                        constexpr int U     = decltype(which)::value;
                        constexpr int FIRST = U * Unit::SLOTS;
                        constexpr int SLOTS = NSLOTS - FIRST < Unit::SLOTS ? NSLOTS - FIRST : Unit::SLOTS;
                        constexpr int STEPS = 2 * SLOTS;
                        uint32_t own[4];  // rows past the super-tile's last are stored as copies of it
                        uint4 pos[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) own[j] = static_cast<uint32_t>(min(first_row + 8 * j, last));
#pragma unroll
                        for (int j = 0; j < 4; ++j) pos[j] = load_shared(nbl_addr + buf * NBL_BYTES + own[j] * 16);
                        auto position = [&](int j, int slot) -> uint32_t {
                            if (slot == 0) return own[j];
                            const int k         = slot - 1;
                            const uint32_t word = (k >> 1) == 0 ? pos[j].x : (k >> 1) == 1 ? pos[j].y : (k >> 1) == 2 ? pos[j].z : pos[j].w;
                            return (k & 1) ? (word >> 16) : (word & 0xFFFFu);
                        };
                        auto gather = [&](Gathered& to, int step) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const uint32_t at = base + position(2 * (step & 1) + i, FIRST + step / 2) * ROW;
                                to.v[i][0]        = load_shared(at);
                                to.v[i][1]        = load_shared(at ^ 64u);
                            }
                        };
                        const uint32_t at = a_base + stage * Unit::COLS;
                        auto store        = [&](const Gathered& g, int step) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                store_a(at + (step / 2) * CIN + 16 * h + (static_cast<uint32_t>(16 * (step & 1)) << 16), g.v[0][h], g.v[1][h]);
                            }
                        };
                        Gathered x[DEPTH];
                        if (!miss) {
#pragma unroll
                            for (int step = 0; step < DEPTH && step < STEPS; ++step) gather(x[step], step);
                        }
                        // the MMAs that read this part of the tensor memory last must be done
                        if (!wait(bar_read + 8 * stage, stage_phase)) return false;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (!miss) {
#pragma unroll
                            for (int step = 0; step < STEPS; ++step) {
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
                                const int slot = FIRST + step / 2;
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    const int row    = min(first_row + 16 * (step & 1) + 8 * i, last);
                                    const uint32_t p = slot == 0 ? static_cast<uint32_t>(row) : load_position(nbl_addr + buf * NBL_BYTES + row * 16 + 2 * (slot - 1));
                                    if (slot > 0 && p == st::NBL_GLOBAL) {
                                        const int idx            = __ldg(a.nb + (nb_base + row) * a.n_neighbours + (slot - 1));
                                        const unsigned char* src = in_bytes + static_cast<size_t>(f.local_base + idx) * ROW + piece * 16;
#pragma unroll
                                        for (int h = 0; h < 2; ++h) x[0].v[i][h] = __ldg(reinterpret_cast<const uint4*>(src + ((first_half + 64 * h) & 127)));
                                    }
                                    else {
                                        const uint32_t from = base + p * ROW;
                                        x[0].v[i][0]        = load_shared(from);
                                        x[0].v[i][1]        = load_shared(from ^ 64u);
                                    }
                                }
                                __syncwarp();
                                store(x[0], step);
                            }
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(bar_stored + 8 * stage);
                        return true;
                    };
#pragma unroll
                    for (int u = 0; u < Unit::COUNT; ++u) {
                        if (turn == group && ok) {
                            if (u == 0) ok = unit(std::integral_constant<int, 0>{});
                            if (u == 1) ok = unit(std::integral_constant<int, (Unit::COUNT > 1 ? 1 : 0)>{});
                            if (u == 2) ok = unit(std::integral_constant<int, (Unit::COUNT > 2 ? 2 : 0)>{});
                        }
                        if (++turn == GATHER_GROUPS) turn = 0;
                        if (++stage == STAGES) {
                            stage = 0;
                            stage_phase ^= 1u;
                        }
                    }
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
            uint32_t acc = 0, acc_phase = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                const Item r = locate(item);
                for (int tile = r.first; ok && tile < r.end; ++tile) {
                    ok = wait(bar_acc_full + 8 * acc, acc_phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    float v[4][OWN];  // rows first_row, + 8, + 16, + 24
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t d[ACC_COLS / 2];  // all columns of 16 rows over 32 threads
#pragma unroll
                        for (int c = 0; c < ACC_COLS; c += 16) load_d(tmem_base + acc * ACC_COLS + lanes + (static_cast<uint32_t>(16 * h) << 16) + c, d + c / 2);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
#pragma unroll
                            for (int i = 0; i < OWN; ++i) {
                                const int at    = 4 * (i / 2) + 2 * j + i % 2;
                                v[2 * h + j][i] = (__uint_as_float(d[at]) + __uint_as_float(d[NP / 2 + at])) + bias[i];
                            }
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(bar_acc_free + 8 * acc);
                    if (++acc == ACCS) {
                        acc = 0;
                        acc_phase ^= 1u;
                    }
                    const int first_row = r.t0 + tile * tc::TILE_ROWS + (warp & 3) * 32 + quad;  // within the frame
                    if (a.activation == VM_SOFTMAX) {
                        // exp of each, summed in channel order from thread to thread of the row
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
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
                        for (int j = 0; j < 4; ++j) activate<OWN>(v[j], a.activation);
                    }
                    const int rows = r.rows - first_row;  // row j exists: 8 * j < rows
                    if (a.out_split) {
                        uint32_t hi[4][OWN / 2], lo[4][OWN / 2];
                        __half2 largest = __float2half2_rn(0.0f);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
#pragma unroll
                            for (int i = 0; i < OWN / 2; ++i) {
                                split_pair(v[j][2 * i], v[j][2 * i + 1], hi[j][i], lo[j][i]);
                                largest = __hmax2(largest, __habs2(*reinterpret_cast<const __half2*>(&hi[j][i])));
                            }
                        }
                        if (a.out_split == SPLIT_ROWS) {
                            // the channels this thread holds may all be padding; a row's hi parts, then its lo parts
                            const int n        = piece * OWN < t.cout ? rows : 0;
                            unsigned char* dst = reinterpret_cast<unsigned char*>(a.out) + (static_cast<size_t>(r.local_base) + first_row) * (4 * t.cout) + piece * (2 * OWN);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                if (8 * j < n) {
                                    if (OWN == 8) {
                                        *reinterpret_cast<uint4*>(dst)              = make_uint4(hi[j][0], hi[j][1], hi[j][OWN / 2 - 2], hi[j][OWN / 2 - 1]);
                                        *reinterpret_cast<uint4*>(dst + 2 * t.cout) = make_uint4(lo[j][0], lo[j][1], lo[j][OWN / 2 - 2], lo[j][OWN / 2 - 1]);
                                    }
                                    else {
                                        *reinterpret_cast<uint2*>(dst)              = make_uint2(hi[j][0], hi[j][1]);
                                        *reinterpret_cast<uint2*>(dst + 2 * t.cout) = make_uint2(lo[j][0], lo[j][1]);
                                    }
                                }
                                dst += 32 * t.cout;
                            }
                        }
                        else if (a.out_split == SPLIT_QUADS) {
                            // 16 channels; pieces of four hi and four lo parts
                            if (OWN == 4) {
                                uint4* dst = reinterpret_cast<uint4*>(a.out) + (static_cast<size_t>(r.local_base) + first_row) * 4 + piece;
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
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
                            for (int j = 0; j < 4; ++j) {
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
                            for (int j = 0; j < 4; ++j) {
                                if (8 * j < n) dst[8 * j] = make_float4(v[j][4 * c], v[j][4 * c + 1], v[j][4 * c + 2], v[j][4 * c + 3]);
                            }
                        }
                    }
                    else {
                        const size_t out_base = a.out_global ? neighbourhood_base() : static_cast<size_t>(r.local_base);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
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
