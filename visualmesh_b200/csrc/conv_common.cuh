// Device code shared by the graph-convolution layer kernels: activations and the split (fp16 hi/lo) feature layout.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/vmcuda.h"
#include "conv_args.hpp"

namespace vm {

// ---- activations -------------------------------------------------------------------------------------------------
// cpp/visualmesh/engine/cpu/apply_activation.hpp:35-64
__device__ __forceinline__ float selu(float s) {
    const float lambda       = 1.0507009873554804934193349852946f;
    const float lambda_alpha = 1.7580993408473768599402175208123f;
    // exp is evaluated for every value and the result selected: straight-line code, so the chains of a row's outputs overlap. Written
    // as one multiply-add of 2^(s log2 e); the product before it loses |s| 2^-24 of an exponential that has become small by then. Over
    // 3 M negative values from 2^-30 to 2^7 the largest error against double is 1.96e-7, that of lambda * (alpha * exp(s) - alpha), which
    // rounds three times behind the exponential, 2.21e-7. 16 -> 16 layers over 4.4 M rows 223 -> 211 us each with it, 4 -> 16 116 -> 102.
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(__fmul_rn(s, 1.4426950408889634f)));
    const float negative = fmaf(lambda_alpha, e, -lambda_alpha);
    return (s >= 0.0f) ? __fmul_rn(lambda, s) : negative;
}

template <int COUT>
__device__ __forceinline__ void activate(float* v, int act) {
    if (act == VM_SELU) {
#pragma unroll
        for (int j = 0; j < COUT; ++j) v[j] = selu(v[j]);
    }
    else if (act == VM_RELU) {
#pragma unroll
        for (int j = 0; j < COUT; ++j) v[j] = (v[j] < 0.0f) ? 0.0f : v[j];
    }
    else if (act == VM_TANH) {
#pragma unroll
        for (int j = 0; j < COUT; ++j) v[j] = tanhf(v[j]);
    }
    else if (act == VM_SOFTMAX) {
        // exp of each, summed in index order from 0, no max subtraction
        float total = 0.0f;
#pragma unroll
        for (int j = 0; j < COUT; ++j) {
            v[j]  = expf(v[j]);
            total = __fadd_rn(total, v[j]);
        }
#pragma unroll
        for (int j = 0; j < COUT; ++j) v[j] = __fdiv_rn(v[j], total);
    }
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// x = h + l with h = fp16(x), l = fp16(x - h), for two values at once
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& h, uint32_t& l) {
    h               = pack_half2(x0, x1);
    const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&h));
    l               = pack_half2(x0 - hf.x, x1 - hf.y);
}

// The "split" feature layout, produced for a layer that runs on the tensor cores. Every fp32 value x is stored as two
// fp16 values, hi = fp16(x) and lo = fp16(x - hi) (x = hi + lo to ~2^-22 relative, absolute error <= 3e-8 for small
// x), in the shape the tensor-core kernel copies straight into shared memory: 16-byte chunks of 8 channels, chunk
// plane p of row r at byte ((p * stride + r) * 16), the C/8 hi planes first, then the C/8 lo planes. Same footprint as
// fp32. Values beyond the fp16 range raise the range flag; the host then recomputes without the tensor-core path.
template <int COUT>
__device__ __forceinline__ void store_split(float* out, int stride, size_t row, const float* v, int32_t* range_flag) {
    static_assert(COUT % 8 == 0, "split layout needs whole 8-channel chunks");
    constexpr int P = COUT / 8;
    unsigned char* base = reinterpret_cast<unsigned char*>(out);
    bool bad            = false;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float x0 = v[8 * p + 2 * q], x1 = v[8 * p + 2 * q + 1];
            bad |= fabsf(x0) > 60000.0f || fabsf(x1) > 60000.0f;
            const __half h0 = __float2half_rn(x0);
            const __half h1 = __float2half_rn(x1);
            const __half l0 = __float2half_rn(x0 - __half2float(h0));
            const __half l1 = __float2half_rn(x1 - __half2float(h1));
            h[q] = static_cast<uint32_t>(__half_as_ushort(h0)) | (static_cast<uint32_t>(__half_as_ushort(h1)) << 16);
            l[q] = static_cast<uint32_t>(__half_as_ushort(l0)) | (static_cast<uint32_t>(__half_as_ushort(l1)) << 16);
        }
        *reinterpret_cast<uint4*>(base + (static_cast<size_t>(p) * stride + row) * 16)     = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(base + (static_cast<size_t>(P + p) * stride + row) * 16) = make_uint4(l[0], l[1], l[2], l[3]);
    }
    if (bad) raise_flag(range_flag, ABORT_TC_RANGE);
}

// The same values row after row for the window kernel (SPLIT_ROWS): eight 16-byte pieces a row, each the hi and lo parts of two channels,
// then of the next two; odd rows begin with their second half, so that two rows of different parity never meet in a bank of shared
// memory. Stores the rows of a warp, one per thread and one after another; all threads call (valid: the row exists; those that do come
// first). stage: shared memory of the warp, 4 KB. A thread that stored its own row would write 16-byte pieces 128 bytes apart, half a sector and one line per thread and store; from shared
// memory a store writes 512 consecutive bytes. Pieces are swizzled by their row, so that neither side meets bank conflicts.
constexpr int SPLIT_ROW_STAGE = 32 * 128;  // bytes of shared memory per warp
__device__ __forceinline__ void store_split_rows(float* out, size_t row, bool valid, const float* v, uint4* stage, int32_t* range_flag) {
    constexpr int Q = 8;  // 16-byte pieces of a row
    const int lane  = threadIdx.x & 31;
    const int odd   = static_cast<int>(row & 1) * 4;
    bool bad        = false;
    __syncwarp();
#pragma unroll
    for (int p = 0; p < Q; ++p) {
        uint32_t h[2], l[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float x0 = v[4 * p + 2 * q], x1 = v[4 * p + 2 * q + 1];
            bad |= fabsf(x0) > 60000.0f || fabsf(x1) > 60000.0f;
            split_pair(x0, x1, h[q], l[q]);
        }
        stage[lane * Q + ((p ^ odd) ^ (lane & (Q - 1)))] = make_uint4(h[0], l[0], h[1], l[1]);
    }
    if (bad && valid) raise_flag(range_flag, ABORT_TC_RANGE);
    __syncwarp();
    const int pieces = __popc(__ballot_sync(0xffffffffu, valid)) * Q;
    uint4* dst       = reinterpret_cast<uint4*>(out) + (row - lane) * Q;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const int i = k * 32 + lane, r = i / Q, p = i % Q;
        if (i < pieces) dst[i] = stage[r * Q + (p ^ (r & (Q - 1)))];
    }
}

// Rows of 16 channels for the staged kernel (SPLIT_QUADS): four 16-byte pieces a row, each four hi parts and their four lo parts.
__device__ __forceinline__ uint4 split_quad(const float* v, bool& bad) {
    uint4 q;
#pragma unroll
    for (int k = 0; k < 4; ++k) bad |= fabsf(v[k]) > 60000.0f;
    split_pair(v[0], v[1], q.x, q.z);
    split_pair(v[2], v[3], q.y, q.w);
    return q;
}
// the row of a thread
__device__ __forceinline__ void store_split_quads(float* out, size_t row, const float* v, int32_t* range_flag) {
    bool bad = false;
    uint4* dst = reinterpret_cast<uint4*>(out) + row * 4;
#pragma unroll
    for (int p = 0; p < 4; ++p) dst[p] = split_quad(v + 4 * p, bad);
    if (bad) raise_flag(range_flag, ABORT_TC_RANGE);
}
// the rows of a warp by way of shared memory (as in store_split_rows; stage: 2 KB of the warp)
constexpr int SPLIT_QUAD_STAGE = 32 * 64;
__device__ __forceinline__ void store_split_quads(float* out, size_t row, bool valid, const float* v, uint4* stage, int32_t* range_flag) {
    const int lane = threadIdx.x & 31;
    bool bad       = false;
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 4; ++p) stage[lane * 4 + (p ^ (lane >> 1 & 3))] = split_quad(v + 4 * p, bad);
    if (bad && valid) raise_flag(range_flag, ABORT_TC_RANGE);
    __syncwarp();
    const int pieces = __popc(__ballot_sync(0xffffffffu, valid)) * 4;
    uint4* dst       = reinterpret_cast<uint4*>(out) + (row - lane) * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = k * 32 + lane, r = i / 4, p = i % 4;
        if (i < pieces) dst[i] = stage[r * 4 + (p ^ (r >> 1 & 3))];
    }
}

}  // namespace vm
