// Device helpers shared by the sm_103a kernels: warp/block reductions and the
// deterministic grid reduction ("last CTA finishes": every CTA writes its
// partial, the last one to arrive sums all partials in a fixed order, so the
// result depends only on the grid size, never on scheduling).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "kernels.hpp"

namespace lss {

// Programmatic dependent launch: a kernel launched by launch_pdl may be
// dispatched once every CTA of its predecessor in the stream has ended, ahead
// of the flush and launch latency between two dependent grids (2 to 6% of a
// solve of up to 100k DOFs).  pdl_enter waits for the predecessor's completion
// and memory; before it a kernel may only read what no kernel of the running
// sequence writes.  No kernel lets its successor in earlier
// (griddepcontrol.launch_dependents): waiting CTAs then fill the SMs that
// drain first and pile up there, which took a 648k-DOF FP64 solve from 214 to
// 311 ms.
__device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
void launch_pdl(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                Args &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    LSS_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

constexpr int WARP = 32;
constexpr int BANK = 32;  // MAS bank width (MASPreconditioner.cu:33)

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the CTA; the result is valid in thread 0.  smem: >= 32 * NV doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *smem)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) smem[wid * NV + k] = v[k];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double t = lane < nw ? smem[lane * NV + k] : 0.0;
            v[k] = warp_sum(t);
        }
    }
}

// Grid-wide deterministic sum.  Every thread of every CTA must call it.
// Returns true in exactly one thread (thread 0 of the last CTA), where
// total[] holds the sums; the arrival counter is reset for the next use.
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], GridReduce gr, double (&total)[NV])
{
    __shared__ double smem[32 * RED_MAX_VALUES];
    __shared__ bool last;
    block_sum<NV>(v, smem);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) gr.partials[blockIdx.x * NV + k] = v[k];
        __threadfence();
        unsigned t = atomicAdd(gr.counter, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k] += __ldcg(gr.partials + b * NV + k);
    block_sum<NV>(acc, smem);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) total[k] = acc[k];
        *gr.counter = 0u;
        return true;
    }
    return false;
}

// Conversions between FP64 and FP32 on the integer pipe, to the same bits as the
// casts: a cast costs the FP64 pipe (two lanes per clock and SM) as much as a
// multiply-add.  Values outside the ranges below (zeros, denormals, infinities,
// NaN, extreme exponents) take the cast.
__device__ __forceinline__ double to_double(float f)
{
    const uint32_t u = __float_as_uint(f), e = (u >> 23) & 0xffu;
    if (e == 0u || e == 255u) return (double)f;
    return __hiloint2double((int)((u & 0x80000000u) | ((e + 896u) << 20) | ((u >> 3) & 0xfffffu)), (int)(u << 29));
}

// v rounded to FP32 (round to nearest even)
__device__ __forceinline__ float to_float(double v)
{
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v), e = (hi >> 20) & 0x7ffu;
    if (e - 897u > 252u) return (float)v;
    const uint32_t m = ((hi & 0xfffffu) << 3) | (lo >> 29), rem = lo & 0x1fffffffu;
    const uint32_t up = rem > 0x10000000u || (rem == 0x10000000u && (m & 1u)) ? 1u : 0u;
    return __uint_as_float((hi & 0x80000000u) | ((((e - 896u) << 23) | m) + up));
}

// (fl32(v), fl32(v - fl32(v)))
__device__ __forceinline__ float2 split_double(double v)
{
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v), e = (hi >> 20) & 0x7ffu;
    if (e - 949u > 200u) {
        const float h = (float)v;
        return make_float2(h, (float)(v - (double)h));
    }
    const uint32_t m = ((hi & 0xfffffu) << 3) | (lo >> 29), rem = lo & 0x1fffffffu;
    const uint32_t up = rem > 0x10000000u || (rem == 0x10000000u && (m & 1u)) ? 1u : 0u;
    // v - fl32(v) = +-(rem or rem - 2^29) * 2^(e - 1075), an integer of 29 bits scaled exactly
    const int d = (int)rem - (int)(up << 29);
    const float l = __fmul_rn((float)((hi & 0x80000000u) ? -d : d), __uint_as_float((e - 948u) << 23));
    return make_float2(__uint_as_float((hi & 0x80000000u) | ((((e - 896u) << 23) | m) + up)), l);
}

// The PCG's scalar sums.  The kernel that forms the addends leaves the sum's
// parts with put_sum; the next kernel that needs the scalar adds them in every
// CTA with from_sum.  PcgSum::direct: one part per CTA, nothing else -- the
// fence, counter and last-CTA tail of grid_sum cost 3 to 4 us at the end of a
// kernel, the consumer's sum 0.6 us at its start.  Otherwise grid_sum leaves
// one part: with many CTAs per SM summing, the parts' FP64 adds would cost the
// pipe more than the tail (PCG_DIRECT_ROWS has both measured).
__device__ __forceinline__ void put_sum(double v, GridReduce gr, PcgSum out)
{
    double a[1] = {v};
    if (out.direct) {
        __shared__ double smem[32];
        block_sum<1>(a, smem);
        if (threadIdx.x == 0) out.part[blockIdx.x] = a[0];
        return;
    }
    double tot[1];
    if (grid_sum<1>(a, gr, tot)) out.part[0] = tot[0];
}

// f(sum), formed by thread 0, in every thread of the CTA (all of them must call
// it).  What a scalar costs the FP64 pipe is warps: 16 clocks an instruction
// whatever the lanes.  A warp takes 128 parts, four a lane, since every warp that
// takes part adds five shuffled sums of its own (304 parts over 8 warps: 61
// warp-wide adds, over 3: 27), and the quotients and tests that follow run in one
// warp, not in all eight of every CTA (a division in each: 5 to 10 us of an
// SM's pipe under the 8 to 16 CTAs of a long vector update).  An iteration went
// from 107 to 103 us at 207k DOF, 805 to 798 at 3M (mixed), 147.1 to 145.2 on a
// 150k Laplacian, 82.5 to 81.3 at 24k (FP64).
template <typename F>
__device__ __forceinline__ auto from_sum(PcgSum in, F f)
{
    __shared__ double smem[32];
    __shared__ decltype(f(0.0)) res;
    const int t = threadIdx.x, w = t >> 5, warps = min((int)blockDim.x / 32, (in.count + 127) / 128);
    double a = 0.0;
    if (in.count == 1) {
        if (t == 0) a = __ldcg(in.part);
    } else {
        if (w < warps) {
            for (int i0 = t; i0 < in.count; i0 += 128 * warps) {
                double b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + j * 32 * warps;
                    b[j] = i < in.count ? __ldcg(in.part + i) : 0.0;
                }
                a += (b[0] + b[1]) + (b[2] + b[3]);
            }
            a = warp_sum(a);
            if ((t & 31) == 0) smem[w] = a;
        }
        if (warps > 1) {
            __syncthreads();
            if (t == 0)
                for (int k = 1; k < warps; ++k) a += smem[k];
        }
    }
    if (t == 0) res = f(a);
    __syncthreads();
    return res;
}

// Grid-wide min/max (deterministic, order independent).
__device__ __forceinline__ double warp_min(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}


}  // namespace lss
