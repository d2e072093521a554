// Graph-convolution layer kernels on the CUDA cores (fused gather + dense + activation).
#pragma once

#include "conv_common.cuh"

namespace vm {

// Each thread owns R rows strided by the block size, so a warp's loads and stores of one row index are contiguous.
// The layer's weights sit in shared memory; every weight read is a 128-bit broadcast shared by the R rows.
template <int CIN, int COUT, int R, int T = CONV_THREADS, int MINB = 1>
__global__ void __launch_bounds__(T, MINB) k_graph_conv(const ConvArgs a) {
    constexpr int COUTP = (COUT + 3) & ~3;
    extern __shared__ float4 smem4[];
    float* w_s = reinterpret_cast<float*>(smem4);

    const int frame_in_chunk = blockIdx.y;
    const int frame          = a.f0 + frame_in_chunk;
    const int start          = a.offsets[frame];
    const int rows           = a.offsets[frame + 1] - start + 1;
    const int first          = blockIdx.x * (T * R);
    if (first >= rows) return;

    const int K = a.n_slots * CIN;
    {
        const float4* src = reinterpret_cast<const float4*>(a.weights);
        const int total4  = (K * COUTP + COUTP) / 4;  // weights then biases, contiguous on the device
        for (int i = threadIdx.x; i < total4; i += T) smem4[i] = __ldg(src + i);
    }
    __syncthreads();
    const float* b_s = w_s + K * COUTP;

    const int local_base  = start - a.offsets[a.f0] + frame_in_chunk;  // chunk-local row of this frame's row 0
    const size_t nb_base  = static_cast<size_t>(start + frame);        // batch-wide row of this frame's row 0

    int row[R];
    float acc[R][COUTP];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        row[q] = min(first + q * T + static_cast<int>(threadIdx.x), rows - 1);
#pragma unroll
        for (int j = 0; j < COUTP; ++j) acc[q][j] = b_s[j];
    }

    const float4* in4 = reinterpret_cast<const float4*>(a.in);
    for (int s = 0; s < a.n_slots; ++s) {
        const float* src[R];
        int src_row[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int idx = (s == 0) ? row[q] : __ldg(a.nb + (nb_base + row[q]) * a.n_neighbours + (s - 1));
            src_row[q]    = local_base + idx;
            src[q]        = a.in + static_cast<size_t>(local_base + idx) * CIN;
        }
        const float* w_slot = w_s + s * CIN * COUTP;
        if (CIN % 4 == 0) {
#pragma unroll
            for (int c4 = 0; c4 < CIN / 4; ++c4) {
                float4 x[R];
#pragma unroll
                for (int q = 0; q < R; ++q) x[q] = in4[static_cast<size_t>(c4) * a.in_stride + src_row[q]];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const float* w_row = w_slot + (c4 * 4 + kk) * COUTP;
#pragma unroll
                    for (int j4 = 0; j4 < COUTP / 4; ++j4) {
                        const float4 w = *reinterpret_cast<const float4*>(w_row + j4 * 4);
#pragma unroll
                        for (int q = 0; q < R; ++q) {
                            const float xv = kk == 0 ? x[q].x : kk == 1 ? x[q].y : kk == 2 ? x[q].z : x[q].w;
                            acc[q][j4 * 4 + 0] = fmaf(xv, w.x, acc[q][j4 * 4 + 0]);
                            acc[q][j4 * 4 + 1] = fmaf(xv, w.y, acc[q][j4 * 4 + 1]);
                            acc[q][j4 * 4 + 2] = fmaf(xv, w.z, acc[q][j4 * 4 + 2]);
                            acc[q][j4 * 4 + 3] = fmaf(xv, w.w, acc[q][j4 * 4 + 3]);
                        }
                    }
                }
            }
        }
        else {
#pragma unroll
            for (int c = 0; c < CIN; ++c) {
                float x[R];
#pragma unroll
                for (int q = 0; q < R; ++q) x[q] = src[q][c];
                const float* w_row = w_slot + c * COUTP;
#pragma unroll
                for (int j4 = 0; j4 < COUTP / 4; ++j4) {
                    const float4 w = *reinterpret_cast<const float4*>(w_row + j4 * 4);
#pragma unroll
                    for (int q = 0; q < R; ++q) {
                        acc[q][j4 * 4 + 0] = fmaf(x[q], w.x, acc[q][j4 * 4 + 0]);
                        acc[q][j4 * 4 + 1] = fmaf(x[q], w.y, acc[q][j4 * 4 + 1]);
                        acc[q][j4 * 4 + 2] = fmaf(x[q], w.z, acc[q][j4 * 4 + 2]);
                        acc[q][j4 * 4 + 3] = fmaf(x[q], w.w, acc[q][j4 * 4 + 3]);
                    }
                }
            }
        }
    }

    const size_t out_base = a.out_global ? nb_base : static_cast<size_t>(local_base);
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int i = first + q * T + static_cast<int>(threadIdx.x);
        activate<COUT>(acc[q], a.activation);
        if constexpr (COUT == 32) {
            if (a.out_split == SPLIT_ROWS) {
                uint4* stage = reinterpret_cast<uint4*>(smem4 + (K * COUTP + COUTP) / 4) + (threadIdx.x >> 5) * (SPLIT_ROW_STAGE / 16);
                store_split_rows(a.out, out_base + i, i < rows, acc[q], stage, a.range_flag);
                continue;
            }
        }
        if constexpr (COUT == 16) {
            if (a.out_split == SPLIT_QUADS) {
                uint4* stage = reinterpret_cast<uint4*>(smem4 + (K * COUTP + COUTP) / 4) + (threadIdx.x >> 5) * (SPLIT_QUAD_STAGE / 16);
                store_split_quads(a.out, out_base + i, i < rows, acc[q], stage, a.range_flag);
                continue;
            }
        }
        if (i >= rows) continue;
        float* dst = a.out + (out_base + i) * COUT;
        if (COUT % 8 == 0 && a.out_split) { store_split<(COUT % 8 == 0 ? COUT : 8)>(a.out, a.out_stride, out_base + i, acc[q], a.range_flag); }
        else if (COUT % 4 == 0 && a.out_planar) {
            float4* out4 = reinterpret_cast<float4*>(a.out);
#pragma unroll
            for (int j4 = 0; j4 < COUT / 4; ++j4) {
                out4[static_cast<size_t>(j4) * a.out_stride + out_base + i] =
                  make_float4(acc[q][j4 * 4], acc[q][j4 * 4 + 1], acc[q][j4 * 4 + 2], acc[q][j4 * 4 + 3]);
            }
        }
        else if (COUT % 4 == 0) {
#pragma unroll
            for (int j4 = 0; j4 < COUT / 4; ++j4) {
                *reinterpret_cast<float4*>(dst + j4 * 4) =
                  make_float4(acc[q][j4 * 4], acc[q][j4 * 4 + 1], acc[q][j4 * 4 + 2], acc[q][j4 * 4 + 3]);
            }
        }
        else {
#pragma unroll
            for (int j = 0; j < COUT; ++j) dst[j] = acc[q][j];
        }
    }
}

// The last layer's results straight into pinned host memory. The rows of a block lie one after another there; threads that stored
// their own would send the bus pieces of a few bytes, so the block arranges them in shared memory first and writes whole lines.
// All threads call; stage holds T * R rows. rows_left: rows of the frame from the block's first on.
template <int R, int T, int COUTP>
__device__ __forceinline__ void store_rows_to_host(float* dst, int rows_left, int cout, const float (&v)[R][COUTP], float* stage) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
#pragma unroll
        for (int j = 0; j < COUTP; ++j) {
            if (j < cout) stage[(q * T + static_cast<int>(threadIdx.x)) * cout + j] = v[q][j];
        }
    }
    __syncthreads();
    const int words = min(rows_left, T * R) * cout;
    for (int k = threadIdx.x; k < words; k += T) dst[k] = stage[k];
}

// The same layer with the weights in the kernel's parameter space (constant bank) instead of shared memory: every
// weight read is a constant-cache load that all lanes share and does not touch the L1/shared data path that the
// gather loads. Layers whose weights fit the parameter space (WMAX floats).
template <int WMAX>
struct ConvWeights {
    float w[WMAX];
};

// Packed single-precision FMA of sm_100 (two independent IEEE fused multiply-adds per instruction): halves the
// number of FMA instructions of a kernel that is bound by instruction issue, not by the FMA pipe.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Accumulators live as pairs of adjacent output columns, each weight pair is one 64-bit constant load shared by the R
// rows, each input value is duplicated into a pair once per row and k.
// The narrow 8-channel layers wait on their gather: six blocks of 256 threads per SM (42 registers) instead of five
// measured 102 -> 98 us on the 8 -> 3 layer over 4.4 M rows, eight (32 registers) spill. 0 = no bound for the others.
template <int CIN, int COUT, int R, int WMAX, int T = CONV_THREADS, int NS = 0>
__global__ void __launch_bounds__(T, (CIN == 8 && COUT <= 8 && T == 256) ? 6 : 0) k_graph_conv_cw(const ConvArgs a, const __grid_constant__ ConvWeights<WMAX> wp) {
    static_assert(CIN % 4 == 0, "vector loads of the input rows");
    constexpr int COUTP = (COUT + 3) & ~3;
    extern __shared__ uint4 split_stage[];  // SPLIT_ROW_STAGE (SPLIT_QUAD_STAGE) bytes per warp when the output is split in rows; the results for the host
    const int frame_in_chunk = blockIdx.y;
    const int frame          = a.f0 + frame_in_chunk;
    const int start          = a.offsets[frame];
    const int rows           = a.offsets[frame + 1] - start + 1;
    const int first          = blockIdx.x * (T * R);
    if (first >= rows) return;
    const int n_slots     = NS ? NS : a.n_slots;  // NS != 0: the slot loop is unrolled and its loads scheduled across slots
    const int K           = n_slots * CIN;
    const int local_base  = start - a.offsets[a.f0] + frame_in_chunk;
    const size_t nb_base  = static_cast<size_t>(start + frame);

    int row[R];
    unsigned long long acc[R][COUTP / 2];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        row[q] = min(first + q * T + static_cast<int>(threadIdx.x), rows - 1);
#pragma unroll
        for (int j = 0; j < COUTP / 2; ++j) acc[q][j] = pack2(wp.w[K * COUTP + 2 * j], wp.w[K * COUTP + 2 * j + 1]);
    }
    const float4* in4 = after_previous(reinterpret_cast<const float4*>(a.in));
#pragma unroll(NS ? NS : 1)
    for (int s = 0; s < n_slots; ++s) {
        int src_row[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int idx = (s == 0) ? row[q] : __ldg(a.nb + (nb_base + row[q]) * a.n_neighbours + (s - 1));
            src_row[q]    = local_base + idx;
        }
        const int w_slot = s * CIN * COUTP;
#pragma unroll
        for (int c4 = 0; c4 < CIN / 4; ++c4) {
            float4 x[R];
#pragma unroll
            for (int q = 0; q < R; ++q) x[q] = in4[static_cast<size_t>(c4) * a.in_stride + src_row[q]];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                unsigned long long xx[R];
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const float xv = kk == 0 ? x[q].x : kk == 1 ? x[q].y : kk == 2 ? x[q].z : x[q].w;
                    xx[q]          = pack2(xv, xv);
                }
#pragma unroll
                for (int j = 0; j < COUTP / 2; ++j) {
                    const int at               = w_slot + (c4 * 4 + kk) * COUTP + 2 * j;
                    const unsigned long long w = pack2(wp.w[at], wp.w[at + 1]);
#pragma unroll
                    for (int q = 0; q < R; ++q) ffma2(acc[q][j], xx[q], w);
                }
            }
        }
    }
    const size_t out_base = a.out_global ? nb_base : static_cast<size_t>(local_base);
    if (COUT <= 16 && a.out_host != nullptr) {
        float v[R][COUTP];
#pragma unroll
        for (int q = 0; q < R; ++q) {
#pragma unroll
            for (int j = 0; j < COUTP / 2; ++j) unpack2(acc[q][j], v[q][2 * j], v[q][2 * j + 1]);
            activate<COUT>(v[q], a.activation);
        }
        store_rows_to_host<R, T>(*a.out_host + (out_base + first) * COUT, rows - first, COUT, v, reinterpret_cast<float*>(split_stage));
        return;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int i = first + q * T + static_cast<int>(threadIdx.x);
        float v[COUTP];
#pragma unroll
        for (int j = 0; j < COUTP / 2; ++j) unpack2(acc[q][j], v[2 * j], v[2 * j + 1]);
        activate<COUT>(v, a.activation);
        if constexpr (COUT == 32) {
            if (a.out_split == SPLIT_ROWS) {
                store_split_rows(a.out, out_base + i, i < rows, v, split_stage + (threadIdx.x >> 5) * (SPLIT_ROW_STAGE / 16), a.range_flag);
                continue;
            }
        }
        if constexpr (COUT == 16) {
            if (a.out_split == SPLIT_QUADS) {
                store_split_quads(a.out, out_base + i, i < rows, v, split_stage + (threadIdx.x >> 5) * (SPLIT_QUAD_STAGE / 16), a.range_flag);
                continue;
            }
        }
        if (i >= rows) continue;
        float* dst = a.out + (out_base + i) * COUT;
        if (COUT % 8 == 0 && a.out_split) { store_split<(COUT % 8 == 0 ? COUT : 8)>(a.out, a.out_stride, out_base + i, v, a.range_flag); }
        else if (COUT % 4 == 0 && a.out_planar) {
            float4* out4 = reinterpret_cast<float4*>(a.out);
#pragma unroll
            for (int j4 = 0; j4 < COUT / 4; ++j4) {
                out4[static_cast<size_t>(j4) * a.out_stride + out_base + i] = make_float4(v[j4 * 4], v[j4 * 4 + 1], v[j4 * 4 + 2], v[j4 * 4 + 3]);
            }
        }
        else if (COUT % 4 == 0) {
#pragma unroll
            for (int j4 = 0; j4 < COUT / 4; ++j4) {
                *reinterpret_cast<float4*>(dst + j4 * 4) = make_float4(v[j4 * 4], v[j4 * 4 + 1], v[j4 * 4 + 2], v[j4 * 4 + 3]);
            }
        }
        else {
#pragma unroll
            for (int j = 0; j < COUT; ++j) dst[j] = v[j];
        }
    }
}

// Layers whose widths are multiples of 4 up to 32 but have no kernel of their own: the padded output width is a template parameter,
// the input width is not. Input chunks come in batches of four, the next batch (and the next slot's neighbour index) on its way
// while one is multiplied. Weights in the parameter space as above. Measured on 29 k rows with four neighbours, against the kernel that
// reads its weights through the cache: 24 -> 20 85 -> 21 us, 20 -> 12 47 -> 15 us, 4 -> 24 30 -> 13 us.
template <int COUTP, int R, int T, int WMAX>
__global__ void __launch_bounds__(T) k_graph_conv_any(const ConvArgs a, int32_t cin4, int32_t cout, const __grid_constant__ ConvWeights<WMAX> wp) {
    constexpr int BATCH      = 4;  // chunks of 4 channels
    const int frame_in_chunk = blockIdx.y;
    const int frame          = a.f0 + frame_in_chunk;
    const int start          = a.offsets[frame];
    const int rows           = a.offsets[frame + 1] - start + 1;
    const int first          = blockIdx.x * (T * R);
    if (first >= rows) return;
    const int local_base = start - a.offsets[a.f0] + frame_in_chunk;
    const size_t nb_base = static_cast<size_t>(start + frame);
    const float4* in4    = reinterpret_cast<const float4*>(a.in);

    int row[R], src[R], next_src[R];
    unsigned long long acc[R][COUTP / 2];
    float4 x[R][BATCH], next[R][BATCH];
    auto fetch_index = [&](int s) {
#pragma unroll
        for (int q = 0; q < R; ++q) next_src[q] = local_base + __ldg(a.nb + (nb_base + row[q]) * a.n_neighbours + (s - 1));
    };
    auto fetch = [&](int c) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                if (c + k < cin4) next[q][k] = __ldg(in4 + static_cast<size_t>(c + k) * a.in_stride + src[q]);
            }
        }
    };
    const int biases = a.n_slots * cin4 * 4 * COUTP;
    extern __shared__ float4 smem4[];  // the results for the host
#pragma unroll
    for (int q = 0; q < R; ++q) {
        row[q] = min(first + q * T + static_cast<int>(threadIdx.x), rows - 1);
        src[q] = local_base + row[q];
#pragma unroll
        for (int j = 0; j < COUTP / 2; ++j) acc[q][j] = pack2(wp.w[biases + 2 * j], wp.w[biases + 2 * j + 1]);
    }
    if (a.n_slots > 1) fetch_index(1);
    fetch(0);
    int at = 0;  // weights of the channel
    for (int s = 0; s < a.n_slots; ++s) {
        for (int c = 0; c < cin4; c += BATCH) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
#pragma unroll
                for (int k = 0; k < BATCH; ++k) x[q][k] = next[q][k];
            }
            if (c + BATCH < cin4) { fetch(c + BATCH); }
            else if (s + 1 < a.n_slots) {
#pragma unroll
                for (int q = 0; q < R; ++q) src[q] = next_src[q];
                fetch(0);
                if (s + 2 < a.n_slots) fetch_index(s + 2);
            }
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                if (c + k >= cin4) break;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    unsigned long long xx[R];
#pragma unroll
                    for (int q = 0; q < R; ++q) {
                        const float xv = kk == 0 ? x[q][k].x : kk == 1 ? x[q][k].y : kk == 2 ? x[q][k].z : x[q][k].w;
                        xx[q]          = pack2(xv, xv);
                    }
#pragma unroll
                    for (int j = 0; j < COUTP / 2; ++j) {
                        const unsigned long long w = pack2(wp.w[at + 2 * j], wp.w[at + 2 * j + 1]);
#pragma unroll
                        for (int q = 0; q < R; ++q) ffma2(acc[q][j], xx[q], w);
                    }
                    at += COUTP;
                }
            }
        }
    }
    const size_t out_base = a.out_global ? nb_base : static_cast<size_t>(local_base);
    float v[R][COUTP];
#pragma unroll
    for (int q = 0; q < R; ++q) {
#pragma unroll
        for (int j = 0; j < COUTP / 2; ++j) unpack2(acc[q][j], v[q][2 * j], v[q][2 * j + 1]);
        if (a.activation == VM_SOFTMAX) {
            float total = 0.0f;
#pragma unroll
            for (int j = 0; j < COUTP; ++j) {
                if (j < cout) {
                    v[q][j] = expf(v[q][j]);
                    total   = __fadd_rn(total, v[q][j]);
                }
            }
#pragma unroll
            for (int j = 0; j < COUTP; ++j) v[q][j] = __fdiv_rn(v[q][j], total);
        }
        else {
            activate<COUTP>(v[q], a.activation);
        }
    }
    if (a.out_host != nullptr) {
        store_rows_to_host<R, T>(*a.out_host + (out_base + first) * cout, rows - first, cout, v, reinterpret_cast<float*>(smem4));
        return;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int i = first + q * T + static_cast<int>(threadIdx.x);
        if (i >= rows) continue;
        if (a.out_planar) {
            float4* out4 = reinterpret_cast<float4*>(a.out);
#pragma unroll
            for (int j4 = 0; j4 < COUTP / 4; ++j4) {
                out4[static_cast<size_t>(j4) * a.out_stride + out_base + i] = make_float4(v[q][j4 * 4], v[q][j4 * 4 + 1], v[q][j4 * 4 + 2], v[q][j4 * 4 + 3]);
            }
        }
        else {
            float* dst = a.out + (out_base + i) * cout;
#pragma unroll
            for (int j = 0; j < COUTP; ++j) {
                if (j < cout) dst[j] = v[q][j];
            }
        }
    }
}

// Few rows: a block owns 128 rows and OW of the outputs (blockIdx.z), a thread one row. With all outputs of a row to a thread an SM would
// hold a block or two, four to eight warps, too few to hide either the gather or the arithmetic's own latency; part of the outputs
// makes it three or four times as many, each with a chain as much shorter (the rows read again come from the L1 cache). The weights of
// those outputs sit in shared memory. Input chunks come in batches of four, the next batch (and the next slot's neighbour index) on its
// way while one is multiplied.
template <int OW, int T>
__global__ void __launch_bounds__(T) k_graph_conv_few(const ConvArgs a, int32_t cin4, int32_t cout, int32_t coutp) {
    constexpr int BATCH      = 4;  // chunks of 4 channels
    const int frame_in_chunk = blockIdx.y;
    const int frame          = a.f0 + frame_in_chunk;
    const int start          = a.offsets[frame];
    const int rows           = a.offsets[frame + 1] - start + 1;
    const int first          = blockIdx.x * T;
    if (first >= rows) return;
    const int local_base = start - a.offsets[a.f0] + frame_in_chunk;
    const size_t nb_base = static_cast<size_t>(start + frame);
    const float4* in4    = reinterpret_cast<const float4*>(a.in);
    const int o0         = blockIdx.z * OW;
    extern __shared__ float4 smem4[];  // weights [channel][OW], then the results for the host

    const int i   = first + static_cast<int>(threadIdx.x);
    const int row = min(i, rows - 1);
    int src = local_base + row, next_src = src;
    float4 next[BATCH];
    auto fetch_index = [&](int s) { next_src = local_base + __ldg(a.nb + (nb_base + row) * a.n_neighbours + (s - 1)); };
    auto fetch       = [&](int c) {
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
            if (c + k < cin4) next[k] = __ldg(in4 + static_cast<size_t>(c + k) * a.in_stride + src);
        }
    };
    if (a.n_slots > 1) fetch_index(1);
    fetch(0);
    const int channels = a.n_slots * cin4 * 4;
    for (int k = threadIdx.x; k < channels * (OW / 4); k += T) {
        const int o = o0 + (k % (OW / 4)) * 4;
        smem4[k]    = o < coutp ? __ldg(reinterpret_cast<const float4*>(a.weights + static_cast<size_t>(k / (OW / 4)) * coutp + o)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    unsigned long long acc[OW / 2];
#pragma unroll
    for (int j = 0; j < OW / 2; ++j) {
        const bool there = o0 + 2 * j < coutp;
        acc[j]           = there ? pack2(__ldg(a.biases + o0 + 2 * j), __ldg(a.biases + o0 + 2 * j + 1)) : 0ull;
    }
    __syncthreads();
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(smem4);  // of the channel
    auto multiply       = [&](const float4& x) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const float xv              = kk == 0 ? x.x : kk == 1 ? x.y : kk == 2 ? x.z : x.w;
            const unsigned long long xx = pack2(xv, xv);
#pragma unroll
            for (int j = 0; j < OW / 4; ++j) {
                const ulonglong2 w2 = w[kk * (OW / 4) + j];
                ffma2(acc[2 * j], xx, w2.x);
                ffma2(acc[2 * j + 1], xx, w2.y);
            }
        }
        w += OW;
    };
    for (int s = 0; s < a.n_slots; ++s) {
        for (int c = 0; c < cin4; c += BATCH) {
            float4 x[BATCH];
#pragma unroll
            for (int k = 0; k < BATCH; ++k) x[k] = next[k];
            if (c + BATCH < cin4) { fetch(c + BATCH); }
            else if (s + 1 < a.n_slots) {
                src = next_src;
                fetch(0);
                if (s + 2 < a.n_slots) fetch_index(s + 2);
            }
            if (c + BATCH <= cin4) {
#pragma unroll
                for (int k = 0; k < BATCH; ++k) multiply(x[k]);
            }
            else {
#pragma unroll
                for (int k = 0; k < BATCH - 1; ++k) {
                    if (c + k < cin4) multiply(x[k]);
                }
            }
        }
    }
    const size_t out_base = a.out_global ? nb_base : static_cast<size_t>(local_base);
    float v[1][OW];
#pragma unroll
    for (int j = 0; j < OW / 2; ++j) unpack2(acc[j], v[0][2 * j], v[0][2 * j + 1]);
    if (a.activation == VM_SOFTMAX) {  // all outputs are this block's
        float total = 0.0f;
#pragma unroll
        for (int j = 0; j < OW; ++j) {
            if (j < cout) {
                v[0][j] = expf(v[0][j]);
                total   = __fadd_rn(total, v[0][j]);
            }
        }
#pragma unroll
        for (int j = 0; j < OW; ++j) v[0][j] = __fdiv_rn(v[0][j], total);
    }
    else {
        activate<OW>(v[0], a.activation);
    }
    if (a.out_host != nullptr) {
        store_rows_to_host<1, T>(*a.out_host + (out_base + first) * cout, rows - first, cout, v, reinterpret_cast<float*>(smem4 + channels * (OW / 4)));
        return;
    }
    if (i >= rows) return;
    if (a.out_planar) {
        float4* out4 = reinterpret_cast<float4*>(a.out);
#pragma unroll
        for (int j4 = 0; j4 < OW / 4; ++j4) {
            if (o0 + j4 * 4 < coutp) {
                out4[static_cast<size_t>(o0 / 4 + j4) * a.out_stride + out_base + i] = make_float4(v[0][j4 * 4], v[0][j4 * 4 + 1], v[0][j4 * 4 + 2], v[0][j4 * 4 + 3]);
            }
        }
    }
    else {
        float* dst = a.out + (out_base + i) * cout;
#pragma unroll
        for (int j = 0; j < OW; ++j) {
            if (o0 + j < cout) dst[o0 + j] = v[0][j];
        }
    }
}

// Any layer shape: one row per thread, outputs in tiles of 8, weights read through the read-only cache.
static __global__ void __launch_bounds__(CONV_THREADS) k_graph_conv_generic(const ConvArgs a, int32_t cin, int32_t cout, int32_t coutp) {
    const int frame_in_chunk = blockIdx.y;
    const int frame          = a.f0 + frame_in_chunk;
    const int start          = a.offsets[frame];
    const int rows           = a.offsets[frame + 1] - start + 1;
    const int i              = blockIdx.x * CONV_THREADS + threadIdx.x;
    if (i >= rows) return;
    const int local_base  = start - a.offsets[a.f0] + frame_in_chunk;
    const size_t nb_base  = static_cast<size_t>(start + frame);
    const size_t out_base = a.out_global ? nb_base : static_cast<size_t>(local_base);
    const bool in_planar  = (cin % 4) == 0;
    const bool out_planar = a.out_planar != 0;
    // element c of a row in either layout
    auto in_at = [&](size_t r, int c) -> float {
        return in_planar ? a.in[((static_cast<size_t>(c >> 2) * a.in_stride + r) << 2) + (c & 3)] : a.in[r * cin + c];
    };
    auto out_ptr = [&](int c) -> float* {
        return out_planar ? a.out + ((static_cast<size_t>(c >> 2) * a.out_stride + out_base + i) << 2) + (c & 3)
                          : a.out + (out_base + i) * cout + c;
    };
    const float* biases   = a.weights + static_cast<size_t>(a.n_slots) * cin * coutp;
    for (int j0 = 0; j0 < cout; j0 += 8) {
        float acc[8];
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) acc[jj] = (j0 + jj < cout) ? __ldg(biases + j0 + jj) : 0.0f;
        for (int s = 0; s < a.n_slots; ++s) {
            const int idx    = (s == 0) ? i : __ldg(a.nb + (nb_base + i) * a.n_neighbours + (s - 1));
            const size_t src = static_cast<size_t>(local_base + idx);
            for (int c = 0; c < cin; ++c) {
                const float x      = in_at(src, c);
                const float* w_row = a.weights + static_cast<size_t>(s * cin + c) * coutp + j0;
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    if (j0 + jj < coutp) acc[jj] = fmaf(x, __ldg(w_row + jj), acc[jj]);
                }
            }
        }
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            if (j0 + jj < cout) *out_ptr(j0 + jj) = acc[jj];
        }
    }
    // activation over the row this thread has just written
    if (a.activation == VM_SELU) {
        for (int j = 0; j < cout; ++j) *out_ptr(j) = selu(*out_ptr(j));
    }
    else if (a.activation == VM_RELU) {
        for (int j = 0; j < cout; ++j) *out_ptr(j) = (*out_ptr(j) < 0.0f) ? 0.0f : *out_ptr(j);
    }
    else if (a.activation == VM_TANH) {
        for (int j = 0; j < cout; ++j) *out_ptr(j) = tanhf(*out_ptr(j));
    }
    else if (a.activation == VM_SOFTMAX) {
        float total = 0.0f;
        for (int j = 0; j < cout; ++j) {
            const float e = expf(*out_ptr(j));
            *out_ptr(j)   = e;
            total         = __fadd_rn(total, e);
        }
        for (int j = 0; j < cout; ++j) *out_ptr(j) = __fdiv_rn(*out_ptr(j), total);
    }
}

}  // namespace vm
