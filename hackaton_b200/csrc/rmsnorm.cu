// RMSNorm on the fp32 residual stream, one pass each way, with the residual add folded in: the
// arithmetic of the reference's rmsnorm_kernel (solution/rmsnorm.py:17-49) in its four modes
//   0  forward            y = w * (x * rstd),            rstd = 1 / sqrt(mean(x^2) + eps)
//   1  backward           dx = rstd * (g - xhat * mean(g * xhat)),  g = dy * w, xhat = x * rstd
//   2  add + forward      s = x + delta (delta fp16), s stored, then mode 0 on s
//   3  backward + the gradient that reaches the sum directly: dx += d_total
// x, w, s, dx, d_total fp32; y (and dy) fp32 or fp16 (the projections that follow read fp16). Modes
// 1 and 3 also write dx in fp16 where asked: the gradient of mode 2's delta, without a second pass
// over dx (16,384 x 1536: 57 + 22 us as a kernel and a cast, 66 as one kernel).
// HBM bound: 6 to 16 bytes per element. A row is read once into registers with 16-byte loads that
// are all in flight together, and every output is written once. Who owns a row depends on what has
// to be in flight (us measured, one CTA per row against one warp per row):
//   forward, many rows of the 1.5B / 7B widths (1536, 3584): one warp; 16,384 x 3584 with the add
//     105.6 against 113.7
//   backward: one CTA with one float4 of each array per thread (mode 3, 16,384 x 1536 with the fp16
//     copy: 65.8 against 68.8, where a warp's 12 to 28 float4 of two arrays spill) or two (mode 1: 43.7
//     against 49.8)
//   up to 512 rows, where latency counts: one CTA with one float4 per thread (64 x 3584 with the add
//     2.7 against 5.8, 1 x 1536 1.7 against 1.9)
//   other widths: one CTA. Before, these took the generic kernel (scalar accesses, the row walked
//     twice), which is left for rows that are not whole float4 or longer than 16,384.
// Inputs are read through the read-only path (ld.global.nc), which lets the compiler issue a row's
// loads ahead of its stores: outputs must not overlap inputs.
#include <cuda_fp16.h>

#include "kernels.h"
#include "ptx.cuh"

namespace nf4 {

constexpr int RN_WARPS = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float4 load4_any(const void* base, long long idx4, int half) {
    if (half) {
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(base) + idx4);
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    return __ldg(reinterpret_cast<const float4*>(base) + idx4);
}

__device__ __forceinline__ void store4_any(void* base, long long idx4, int half, float4 v) {
    if (half) {
        const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
        uint2 raw;
        raw.x = *reinterpret_cast<const uint32_t*>(&a);
        raw.y = *reinterpret_cast<const uint32_t*>(&b);
        reinterpret_cast<uint2*>(base)[idx4] = raw;
    } else {
        reinterpret_cast<float4*>(base)[idx4] = v;
    }
}

__device__ __forceinline__ void store_dx(const RmsNormArgs& a, long long idx4, float4 dx) {
    reinterpret_cast<float4*>(a.dx)[idx4] = dx;
    if (a.dx16 != nullptr) store4_any(a.dx16, idx4, 1, dx);
}

// Forward over many rows: one warp per row. (Instances for the add ask for the mode again, although nothing
// else comes to them: with the answer known at compile time the loads are ordered differently, and 16,384 x 3584
// takes 110.8 us instead of 106.7.)
template <int NV, bool ADD>
__global__ void __launch_bounds__(RN_WARPS * 32, NV <= 16 ? 2 : 1)
rmsnorm_rows_kernel(const RmsNormArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * RN_WARPS + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    const long long base4 = row * (long long)(NV * 32);  // in units of 4 elements
    float4 x[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) x[i] = __ldg(reinterpret_cast<const float4*>(a.x) + base4 + i * 32 + lane);
    if (ADD && a.mode == 2) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float4 d = load4_any(a.delta, base4 + i * 32 + lane, 1);
            x[i].x += d.x; x[i].y += d.y; x[i].z += d.z; x[i].w += d.w;
            reinterpret_cast<float4*>(a.total)[base4 + i * 32 + lane] = x[i];
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        ss += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
    const float rstd = 1.f / sqrtf(warp_sum(ss) * (1.f / (float)(NV * 128)) + a.eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const float4 w = __ldg(reinterpret_cast<const float4*>(a.w) + i * 32 + lane);
        store4_any(a.y, base4 + i * 32 + lane, a.y_half,
                   make_float4(w.x * (x[i].x * rstd), w.y * (x[i].y * rstd),
                               w.z * (x[i].z * rstd), w.w * (x[i].w * rstd)));
    }
    if (lane == 0) a.rstd[row] = rstd;
}

// Sum over the CTA, the same value in every thread.
__device__ __forceinline__ float block_sum(float v) {
    __shared__ float part[32];
    v = warp_sum(v);
    const int warps = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    const int l = threadIdx.x & 31;
    return warp_sum(l < warps ? part[l] : 0.f);
}

// One CTA per row of hidden = 4 * h4 floats, or one warp where a CTA holds RN_WARPS narrow rows; NV float4
// per thread; everything the row needs is requested before the first value is used.
template <int NV, int MODE, bool WARP>
__global__ void __launch_bounds__(WARP ? RN_WARPS * 32 : 1024)
rmsnorm_block_kernel(const RmsNormArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    const int h4 = a.hidden >> 2;
    const long long row = WARP ? (long long)blockIdx.x * RN_WARPS + threadIdx.y : (long long)blockIdx.x;
    const long long base4 = row * h4;
    if (WARP && row >= a.rows) return;
    auto row_sum = [&](float v) { return WARP ? warp_sum(v) : block_sum(v); };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 x[NV], w[NV], d[NV], t[NV];   // d: mode 2 the delta, modes 1 and 3 dy; t: d_total
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        x[i] = w[i] = d[i] = t[i] = zero;
        if (c < h4) {
            x[i] = __ldg(reinterpret_cast<const float4*>(a.x) + base4 + c);
            if (MODE == 1 || MODE == 3) d[i] = load4_any(a.dy, base4 + c, a.y_half);
            if (MODE == 2) d[i] = load4_any(a.delta, base4 + c, 1);
            if (MODE == 3) t[i] = __ldg(reinterpret_cast<const float4*>(a.d_total) + base4 + c);
            w[i] = __ldg(reinterpret_cast<const float4*>(a.w) + c);
        }
    }
    const float inv_h = 1.f / (float)a.hidden;
    float sum = 0.f;
    if (MODE == 0 || MODE == 2) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (MODE == 2) { x[i].x += d[i].x; x[i].y += d[i].y; x[i].z += d[i].z; x[i].w += d[i].w; }
            sum += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
        }
        const float rstd = 1.f / sqrtf(row_sum(sum) * inv_h + a.eps);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            if (c >= h4) continue;
            if (MODE == 2) reinterpret_cast<float4*>(a.total)[base4 + c] = x[i];
            store4_any(a.y, base4 + c, a.y_half,
                       make_float4(w[i].x * (x[i].x * rstd), w[i].y * (x[i].y * rstd),
                                   w[i].z * (x[i].z * rstd), w[i].w * (x[i].w * rstd)));
        }
        if (threadIdx.x == 0) a.rstd[row] = rstd;
        return;
    }
    const float rstd = a.rstd[row];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        x[i].x *= rstd; x[i].y *= rstd; x[i].z *= rstd; x[i].w *= rstd;              // xhat
        d[i].x *= w[i].x; d[i].y *= w[i].y; d[i].z *= w[i].z; d[i].w *= w[i].w;      // g
        sum += d[i].x * x[i].x + d[i].y * x[i].y + d[i].z * x[i].z + d[i].w * x[i].w;
    }
    const float mean_gx = row_sum(sum) * inv_h;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < h4)
            store_dx(a, base4 + c, make_float4(rstd * (d[i].x - x[i].x * mean_gx) + t[i].x,
                                               rstd * (d[i].y - x[i].y * mean_gx) + t[i].y,
                                               rstd * (d[i].z - x[i].z * mean_gx) + t[i].z,
                                               rstd * (d[i].w - x[i].w * mean_gx) + t[i].w));
    }
}

template <int NV, bool WARP = false>
static cudaError_t launch_block(const RmsNormArgs& a, cudaStream_t stream) {
    const dim3 grid((unsigned)(WARP ? (a.rows + RN_WARPS - 1) / RN_WARPS : a.rows));
    const dim3 block(WARP ? 32 : (unsigned)((a.hidden / 4 + 32 * NV - 1) / (32 * NV) * 32), WARP ? RN_WARPS : 1);
    switch (a.mode) {
        case 0: return launch_pdl(rmsnorm_block_kernel<NV, 0, WARP>, grid, block, 0, stream, a);
        case 1: return launch_pdl(rmsnorm_block_kernel<NV, 1, WARP>, grid, block, 0, stream, a);
        case 2: return launch_pdl(rmsnorm_block_kernel<NV, 2, WARP>, grid, block, 0, stream, a);
        default: return launch_pdl(rmsnorm_block_kernel<NV, 3, WARP>, grid, block, 0, stream, a);
    }
}

// Any width: scalar accesses, the row is walked twice.
__global__ void __launch_bounds__(RN_WARPS * 32)
rmsnorm_generic_kernel(const RmsNormArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * RN_WARPS + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    const long long base = row * a.hidden;
    const float* xs = a.x + base;
    if (a.mode == 2) {
        const __half* d = static_cast<const __half*>(a.delta) + base;
        for (int c = lane; c < a.hidden; c += 32) a.total[base + c] = xs[c] + __half2float(d[c]);
        __syncwarp();
        xs = a.total + base;
    }
    const float inv_h = 1.f / (float)a.hidden;
    if ((a.mode & 1) == 0) {
        float ss = 0.f;
        for (int c = lane; c < a.hidden; c += 32) ss += xs[c] * xs[c];
        const float rstd = 1.f / sqrtf(warp_sum(ss) * inv_h + a.eps);
        for (int c = lane; c < a.hidden; c += 32) {
            const float v = a.w[c] * (xs[c] * rstd);
            if (a.y_half) static_cast<__half*>(a.y)[base + c] = __float2half_rn(v);
            else          static_cast<float*>(a.y)[base + c] = v;
        }
        if (lane == 0) a.rstd[row] = rstd;
    } else {
        const float rstd = a.rstd[row];
        float dot = 0.f;
        for (int c = lane; c < a.hidden; c += 32) {
            const float dy = a.y_half ? __half2float(static_cast<const __half*>(a.dy)[base + c])
                                      : static_cast<const float*>(a.dy)[base + c];
            dot += dy * a.w[c] * (xs[c] * rstd);
        }
        const float mean_gx = warp_sum(dot) * inv_h;
        for (int c = lane; c < a.hidden; c += 32) {
            const float dy = a.y_half ? __half2float(static_cast<const __half*>(a.dy)[base + c])
                                      : static_cast<const float*>(a.dy)[base + c];
            float dx = rstd * (dy * a.w[c] - xs[c] * rstd * mean_gx);
            if (a.mode == 3) dx += a.d_total[base + c];
            a.dx[base + c] = dx;
            if (a.dx16 != nullptr) static_cast<__half*>(a.dx16)[base + c] = __float2half_rn(dx);
        }
    }
}

cudaError_t launch_rmsnorm(const RmsNormArgs& a, cudaStream_t stream) {
    if (a.rows <= 0 || a.hidden <= 0) return cudaSuccess;
    const dim3 grid((unsigned)((a.rows + RN_WARPS - 1) / RN_WARPS)), block(RN_WARPS * 32);
    const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) |
                           reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.dy) |
                           reinterpret_cast<uintptr_t>(a.dx) | reinterpret_cast<uintptr_t>(a.delta) |
                           reinterpret_cast<uintptr_t>(a.total) | reinterpret_cast<uintptr_t>(a.d_total) |
                           reinterpret_cast<uintptr_t>(a.dx16);
    const bool vec = (bits & 15) == 0;
    const int h4 = a.hidden / 4;
    if (!vec || a.hidden % 4 != 0 || a.rows > 0x7FFFFFFF || h4 > 4096)
        return launch_pdl(rmsnorm_generic_kernel, grid, block, 0, stream, a);
    const bool few = a.rows <= 512, backward = (a.mode & 1) != 0;
    if (!few && !backward && a.hidden == 12 * 128)
        return a.mode == 2 ? launch_pdl(rmsnorm_rows_kernel<12, true>, grid, block, 0, stream, a)
                           : launch_pdl(rmsnorm_rows_kernel<12, false>, grid, block, 0, stream, a);
    if (!few && !backward && a.hidden == 28 * 128)
        return a.mode == 2 ? launch_pdl(rmsnorm_rows_kernel<28, true>, grid, block, 0, stream, a)
                           : launch_pdl(rmsnorm_rows_kernel<28, false>, grid, block, 0, stream, a);
    // Narrow rows, a warp each. A CTA of its own costs a row more than its bytes: 16,384 rows of 64 / 256 / 512
    // take 17.7 / 18.6 / 19.1 us forward whatever the width (modes 1 to 3 the same), with a warp each 3.6 / 5.3 /
    // 9.3 (the generic kernel: 5.7 / 8.5 / 14.9). Up to 2048 rows a CTA's shorter chain is ahead from 192 on (2048 x
    // 256: 2.5 against 2.7 with the add); with four arrays in flight 384 needs more rows (4096: 5.1 against 6.0,
    // 16,384: 19.0 against 15.3) and 512 never pays (19.9 against 22.4); with one up to 1024 do (16,384 x 640 19.7
    // against 13.2, x 1024 21.4 against 18.2).
    if (h4 <= 32) return launch_block<1, true>(a, stream);
    if (a.rows > 2048) {
        if (h4 <= 64) return launch_block<2, true>(a, stream);
        if (h4 <= 128 && a.mode != 3) return launch_block<4, true>(a, stream);
        if (h4 <= 96 && a.rows > 8192) return launch_block<4, true>(a, stream);
        if (h4 <= 256 && a.mode == 0)
            return launch_pdl(rmsnorm_block_kernel<8, 0, true>, grid, dim3(32, RN_WARPS), 0, stream, a);
    }
    // float4 per thread: one where latency counts or four arrays are in flight, otherwise two
    if (h4 <= 1024 && (few || a.mode == 3 || h4 <= 128)) return launch_block<1>(a, stream);
    if (h4 <= 2048 && (few || backward || h4 <= 256)) return launch_block<2>(a, stream);
    return launch_block<4>(a, stream);
}

}  // namespace nf4
