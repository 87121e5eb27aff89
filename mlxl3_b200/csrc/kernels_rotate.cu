// Input and output rotations of the EXL3 linear layer as stand-alone kernels
// (reference: native/src/linear.rs:855-861 and 978-996; native/shaders/_lane_prologue.metal,
// _lane_epilogue.metal, exl3.metal:204-235).  One warp per 128-block of one row.
#include "hadamard.cuh"
#include "kernels.h"

namespace b200exl3 {

// WIDE: rows and scales lie so that four elements are one access (whatever this library allocated does; rows cut out of a
// larger buffer need not).  An instantiation of its own, because a test per access cost 0.1 to 0.3 us of a call.
template <bool WIDE>
__global__ void __launch_bounds__(256)
prepare_kernel(const void* __restrict__ x, int x_dtype, const __half* __restrict__ suh, int64_t scale_rows,
               int64_t rows, int in, __half* __restrict__ xhat, const __half* __restrict__ glu_up, int groups) {
    pdl_launch_dependents();                    // the kernel after this one may start; it waits for our memory itself
    pdl_wait();                                 // what the kernel before this one wrote is visible from here on
    const int lane = threadIdx.x & 31;
    const int blocks_per_row = in >> 7;
    const int64_t total = rows * blocks_per_row;
    for (int64_t unit = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); unit < total;
         unit += static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5)) {
        const int64_t row = unit / blocks_per_row;
        const int col = static_cast<int>(unit % blocks_per_row) * 128 + lane * 4;
        __half v[4];
        if (glu_up != nullptr) {
            // SwiGLU of two fp16 row sets as the input (x = gate rows): half(gate * sigmoid(gate)) * up, each product
            // rounded to half, the arithmetic of the stand-alone SwiGLU kernel and of the small-batch prologue
            const uint2 gv = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(x) + row * in + col);
            const uint2 uv = *reinterpret_cast<const uint2*>(glu_up + row * in + col);
            const __half2* gh = reinterpret_cast<const __half2*>(&gv);
            const __half2* uh = reinterpret_cast<const __half2*>(&uv);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 f = __half22float2(gh[j]);
                const __half2 sg = __floats2half2_rn(1.0f / (1.0f + expf(-f.x)), 1.0f / (1.0f + expf(-f.y)));
                const __half2 a = __hmul2_rn(__hmul2_rn(gh[j], sg), uh[j]);
                v[2 * j] = __low2half(a);
                v[2 * j + 1] = __high2half(a);
            }
        } else {
            load4_as_half<WIDE>(x, x_dtype, row * in + col, v);
        }
        // a group's members read the same row, each with its own input scales
        const __half* s = suh + (scale_rows == 1 ? 0 : row * in) + col;
        __half* dst = xhat + row * in + col;
        for (int g = 0; g < groups; ++g, s += in, dst += rows * in) {
            __half scale[4];
            load4_as_half<WIDE>(s, kF16, 0, scale);
            __align__(8) __half h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __hmul_rn(v[j], scale[j]);
            warp_hadamard128_f16(h, lane);
            *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(h);
        }
    }
}

// The same for many rows, where the instructions of the rotation bound it and not the chain of one block: four blocks by a warp (see
// quad_hadamard128_f16).  WIDE: rows and scales start at multiples of 16 bytes.  1999 rows of 4096 for three members, 65 MB, cold:
// 32.9 -> 21.3 us; 512 rows of 14336 with SwiGLU 20.6 -> 15.5; with few rows the longer chain shows (16 rows 5120->2x25600 72.0 us
// with one block a warp, 73.7 with four).
template <bool WIDE>
__global__ void __launch_bounds__(256)
prepare_quads_kernel(const void* __restrict__ x, int x_dtype, const __half* __restrict__ suh, int64_t scale_rows,
               int64_t rows, int in, __half* __restrict__ xhat, const __half* __restrict__ glu_up, int groups) {
    pdl_launch_dependents();                    // the kernel after this one may start; it waits for our memory itself
    pdl_wait();                                 // what the kernel before this one wrote is visible from here on
    const int lane = threadIdx.x & 31;
    const int blocks_per_row = in >> 7;
    const int64_t total = rows * blocks_per_row;
    for (int64_t first = (static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 4; first < total;
         first += static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5) * 4) {
        const bool live = first + (lane >> 3) < total;                          // the warp's last blocks need not exist
        const int64_t unit = live ? first + (lane >> 3) : total - 1;
        const int64_t row = unit / blocks_per_row;
        const int col = static_cast<int>(unit - row * blocks_per_row) * 128 + (lane & 7) * 16;
        __half2 v[8];
        load16_as_half<WIDE>(x, x_dtype, row * in + col, v);
        if (glu_up != nullptr) {
            // SwiGLU of two fp16 row sets as the input (x = gate rows): half(gate * sigmoid(gate)) * up, each product
            // rounded to half, the arithmetic of the stand-alone SwiGLU kernel and of the small-batch prologue
            __half2 u[8];
            load16_as_half<WIDE>(glu_up, kF16, row * in + col, u);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float2 f = __half22float2(v[j]);
                const __half2 sg = __floats2half2_rn(1.0f / (1.0f + expf(-f.x)), 1.0f / (1.0f + expf(-f.y)));
                v[j] = __hmul2_rn(__hmul2_rn(v[j], sg), u[j]);
            }
        }
        // a group's members read the same row, each with its own input scales
        const __half* s = suh + (scale_rows == 1 ? 0 : row * in) + col;
        __half* dst = xhat + row * in + col;
        for (int g = 0; g < groups; ++g, s += in, dst += rows * in) {
            __half2 h[8];
            load16_as_half<WIDE>(s, kF16, 0, h);
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = __hmul2_rn(v[j], h[j]);
            quad_hadamard128_f16(h, lane);
            if (live) store16_half(dst, h);
        }
    }
}

template <bool WIDE>
__global__ void __launch_bounds__(256)
finish_kernel(const float* __restrict__ partials, int splits, int64_t split_stride, const __half* __restrict__ svh,
              int64_t scale_rows, const __half* __restrict__ bias, int64_t rows, int out, int y_dtype,
              void* __restrict__ y) {
    pdl_launch_dependents();                    // the kernel after this one may start; it waits for our memory itself
    pdl_wait();                                 // what the kernel before this one wrote is visible from here on
    const int lane = threadIdx.x & 31;
    const int blocks_per_row = out >> 7;
    const int64_t total = rows * blocks_per_row;
    for (int64_t unit = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); unit < total;
         unit += static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5)) {
        const int64_t row = unit / blocks_per_row;
        const int col = static_cast<int>(unit % blocks_per_row) * 128 + lane * 4;
        const float* src = partials + row * out + col;
        float4 acc = *reinterpret_cast<const float4*>(src);
        for (int s0 = 1; s0 < splits; s0 += 8) {         // splits are added in order, in fp32; loads go out together
            float4 part[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (s0 + j < splits) part[j] = *reinterpret_cast<const float4*>(src + (s0 + j) * split_stride);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (s0 + j < splits) {
                    acc.x = __fadd_rn(acc.x, part[j].x); acc.y = __fadd_rn(acc.y, part[j].y);
                    acc.z = __fadd_rn(acc.z, part[j].z); acc.w = __fadd_rn(acc.w, part[j].w);
                }
        }
        __half h[4] = {__float2half_rn(acc.x), __float2half_rn(acc.y), __float2half_rn(acc.z), __float2half_rn(acc.w)};
        warp_hadamard128_f16(h, lane);
        __half scale[4];
        load4_as_half<WIDE>(svh, kF16, (scale_rows == 1 ? 0 : row * out) + col, scale);
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __hmul_rn(h[j], scale[j]);
        store4_from_half<WIDE>(y, y_dtype, row * out + col, h, bias ? bias + col : nullptr);
    }
}

static unsigned grid_for(int64_t units) {
    int64_t blocks = (units + 7) / 8;
    int64_t cap = static_cast<int64_t>(sm_count()) * 8;
    return static_cast<unsigned>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

int64_t prepare_ctas(int64_t rows, int in) {
    const int64_t units = rows * (in / 128);
    return grid_for(units > kQuadRotationUnits ? (units + 3) / 4 : units);
}

cudaError_t launch_prepare(const void* x, int x_dtype, const __half* suh, int64_t scale_rows, int64_t rows, int in,
                           __half* xhat, cudaStream_t stream, const __half* glu_up, int groups) {
    if (rows == 0) return cudaSuccess;
    if (groups > 1 && scale_rows != 1) return cudaErrorInvalidValue;
    if (glu_up != nullptr && x_dtype != kF16) return cudaErrorInvalidValue;
    const int64_t units = rows * (in / 128);
    if (units > kQuadRotationUnits) {
        const bool wide = sixteen_bytes_at_once(x) && sixteen_bytes_at_once(suh) && sixteen_bytes_at_once(glu_up);
        return launch_dependent(wide ? prepare_quads_kernel<true> : prepare_quads_kernel<false>, dim3(static_cast<unsigned>(prepare_ctas(rows, in))), dim3(256), 0, stream, x,
                                x_dtype, suh, scale_rows, rows, in, xhat, glu_up, groups);
    }
    const bool wide = four_at_once(x, x_dtype) && four_at_once(suh, kF16);
    return launch_dependent(wide ? prepare_kernel<true> : prepare_kernel<false>, dim3(static_cast<unsigned>(prepare_ctas(rows, in))), dim3(256), 0, stream, x, x_dtype, suh, scale_rows, rows, in, xhat,
                            glu_up, groups);
}

cudaError_t launch_finish(const float* partials, int splits, int64_t split_stride, const __half* svh,
                          int64_t scale_rows, const __half* bias, int64_t rows, int out, int y_dtype, void* y,
                          cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const bool wide = four_at_once(svh, kF16) && four_at_once(bias, kF16) && four_at_once(y, y_dtype);
    return launch_dependent(wide ? finish_kernel<true> : finish_kernel<false>, dim3(grid_for(rows * (out / 128))), dim3(256), 0, stream, partials, splits, split_stride, svh,
                            scale_rows, bias, rows, out, y_dtype, y);
}

}  // namespace b200exl3
