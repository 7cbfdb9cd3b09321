// Block-row SpMV building blocks (sm_103a).
//
// Operator layout in HBM ("row-sliced BSR"): block rows in partition order,
// rows[nb+1], cols[nnzb]; the bd*bd values of the len blocks of block row i
// are stored as bd*bd contiguous arrays of length len:
//     vals[rows[i]*bd*bd + k*len + l] = entry k (row major in the block) of
// the l-th block of row i.  A group of LANES threads handles one block row;
// lane l reads block l, l+LANES, ...: every value load of the group is one
// contiguous, fully used segment, and the column index load is too.  For
// bd == 1 this is plain CSR.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace lss {

template <int LANES, typename T>
__device__ __forceinline__ T group_sum(T v)
{
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, LANES);
    return v;
}

// The blocks l = lane, lane + LANES, ... of a row, block(l, column) each.  Up to
// eight lanes the steps are paired by hand: unrolled by the compiler, the lanes
// with an odd count ran the loop's remainder apart, three rounds of products
// for a row of 15 blocks on eight lanes instead of two (648k DOFs in FP64: 93
// against 70 us, 3.0M in double-float 225 against 208).  From 16 lanes on a row
// is mostly one step, where the plain loop is shorter (207k: 23 against 26 us).
template <int LANES, typename Block>
__device__ __forceinline__ void row_steps(const int32_t *__restrict__ cols, int32_t len, int lane, Block block)
{
    if constexpr (LANES >= 16) {
#pragma unroll 2
        for (int32_t l = lane; l < len; l += LANES) block(l, __ldcs(cols + l));
    } else {
        for (int32_t l = lane; l < len; l += 2 * LANES) {
            const bool two = l + LANES < len;
            const int32_t c = __ldcs(cols + l), c2 = two ? __ldcs(cols + l + LANES) : c;
            block(l, c);
            if (two) block(l + LANES, c2);
        }
    }
}

// y[0..BD) = this lane's part of (A x)[block row i]: the blocks l = lane,
// lane + LANES, ...  VT: stored value type; XT: x type; ACC: accumulator.  A
// group without a row passes valid = false and gets zeros.
template <int BD, int LANES, typename VT, typename XT, typename ACC>
__device__ __forceinline__ void bsr_block_row_part(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                                              const VT *__restrict__ vals, int32_t i, bool valid,
                                              const XT *__restrict__ x, int lane, ACC (&y)[BD])
{
    const int32_t b = valid ? rows[i] : 0, e = valid ? rows[i + 1] : 0, len = e - b;
    const VT *__restrict__ v = vals + (int64_t)b * (BD * BD);
#pragma unroll
    for (int r = 0; r < BD; ++r) y[r] = ACC(0);
    row_steps<LANES>(cols + b, len, lane, [&](int32_t l, int32_t c) {
        ACC xv[BD];
#pragma unroll
        for (int k = 0; k < BD; ++k) xv[k] = (ACC)x[(int64_t)c * BD + k];
#pragma unroll
        for (int r = 0; r < BD; ++r)
#pragma unroll
            for (int k = 0; k < BD; ++k) y[r] += (ACC)__ldcs(v + (int64_t)(r * BD + k) * len + l) * xv[k];
    });
}

// y[0..BD) = (A x)[block row i], reduced over the LANES-wide group (valid in
// every lane of the group).  Every lane of the warp must call it (the group
// reduction is a full-warp shuffle).
template <int BD, int LANES, typename VT, typename XT, typename ACC>
__device__ __forceinline__ void bsr_block_row(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                                              const VT *__restrict__ vals, int32_t i, bool valid,
                                              const XT *__restrict__ x, int lane, ACC (&y)[BD])
{
    bsr_block_row_part<BD, LANES, VT, XT, ACC>(rows, cols, vals, i, valid, x, lane, y);
#pragma unroll
    for (int r = 0; r < BD; ++r) y[r] = group_sum<LANES>(y[r]);
}

// A x in FP64 over the block rows, 256 threads per CTA, out(i, k, value) once
// per scalar row.  The lanes' parts meet in shared memory, one thread adding
// the LANES parts of one scalar row: an FP64 add costs the pipe a whole warp
// however it is predicated, and the group's shuffle reduction ran log2(LANES)
// of them per component in every warp (a third of the instructions of a 3 x 3
// product at eight lanes; here a sixth) and left the epilogue to one lane in
// eight.  `buf`: rows_smem<BD, LANES> doubles.
template <int BD, int LANES>
constexpr int rows_smem = LANES == 1 ? 1 : 256 / LANES * BD * (LANES + 1);

template <int BD, int LANES, typename Out>
__device__ __forceinline__ void fp64_rows(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                                          const double *__restrict__ vals, int32_t nb, const double *__restrict__ x,
                                          double *__restrict__ buf, Out out)
{
    constexpr int RP = 256 / LANES;  // block rows per CTA and sweep
    const int lane = threadIdx.x % LANES, row = threadIdx.x / LANES;
    for (int64_t r0 = (int64_t)blockIdx.x * RP; r0 < nb; r0 += (int64_t)gridDim.x * RP) {
        const bool valid = r0 + row < nb;
        double acc[BD];
        bsr_block_row_part<BD, LANES, double, double, double>(rows, cols, vals, (int32_t)(r0 + row), valid, x, lane,
                                                              acc);
        if (LANES == 1) {
            if (valid)
#pragma unroll
                for (int k = 0; k < BD; ++k) out((int32_t)(r0 + row), k, acc[k]);
            continue;
        }
#pragma unroll
        for (int k = 0; k < BD; ++k) buf[(row * BD + k) * (LANES + 1) + lane] = acc[k];
        __syncthreads();
        for (int o = threadIdx.x; o < RP * BD; o += 256) {
            const int32_t i = (int32_t)(r0 + o / BD);
            if (i >= nb) break;
            double sum = buf[o * (LANES + 1)];
#pragma unroll
            for (int q = 1; q < LANES; ++q) sum += buf[o * (LANES + 1) + q];
            out(i, o % BD, sum);
        }
        __syncthreads();
    }
}

// ---- double-float (an FP32 pair hi + lo) arithmetic on the FP32 pipe.  The
// intrinsics keep the compiler from contracting the error-free transforms.

// (sh, sl) += (ah + al) * (xh + xl): TwoProd of the high words (exact product
// and its rounding error by FMA), TwoSum into sh, the error terms and the two
// cross products into sl; al * xl (2^-48 relative) is dropped.
__device__ __forceinline__ void df_fma(float &sh, float &sl, float ah, float al, float xh, float xl)
{
    const float p = __fmul_rn(ah, xh);
    const float e = __fmaf_rn(ah, xh, -p);
    const float t = __fadd_rn(sh, p);
    const float z = __fsub_rn(t, sh);
    const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, z)), __fsub_rn(p, z));
    sh = t;
    sl = __fadd_rn(sl, __fadd_rn(err, __fadd_rn(e, __fmaf_rn(ah, xl, __fmul_rn(al, xh)))));
}

// (ah, al) += (bh, bl)
__device__ __forceinline__ void df_add(float &ah, float &al, float bh, float bl)
{
    const float t = __fadd_rn(ah, bh);
    const float z = __fsub_rn(t, ah);
    const float err = __fadd_rn(__fsub_rn(ah, __fsub_rn(t, z)), __fsub_rn(bh, z));
    ah = t;
    al = __fadd_rn(__fadd_rn(al, bl), err);
}

// Block row i of A x in double-float: values and x as (hi, lo) pairs, one
// 8-byte load each.  The group reduction runs on the pairs with FP32
// shuffles; the sums are valid in every lane of the group.
template <int BD, int LANES>
__device__ __forceinline__ void bsr_block_row_df(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                                                 const float2 *__restrict__ vals, int32_t i, bool valid,
                                                 const float2 *__restrict__ x, int lane, float (&sh)[BD],
                                                 float (&sl)[BD])
{
    const int32_t b = valid ? rows[i] : 0, e = valid ? rows[i + 1] : 0, len = e - b;
    const float2 *__restrict__ v = vals + (int64_t)b * (BD * BD);
#pragma unroll
    for (int r = 0; r < BD; ++r) sh[r] = sl[r] = 0.f;
    row_steps<LANES>(cols + b, len, lane, [&](int32_t l, int32_t c) {
        float2 xv[BD];
#pragma unroll
        for (int k = 0; k < BD; ++k) xv[k] = x[(int64_t)c * BD + k];
#pragma unroll
        for (int r = 0; r < BD; ++r)
#pragma unroll
            for (int k = 0; k < BD; ++k) {
                const float2 a = __ldcs(v + (int64_t)(r * BD + k) * len + l);
                df_fma(sh[r], sl[r], a.x, a.y, xv[k].x, xv[k].y);
            }
    });
#pragma unroll
    for (int r = 0; r < BD; ++r)
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            const float bh = __shfl_xor_sync(0xffffffffu, sh[r], o, LANES);
            const float bl = __shfl_xor_sync(0xffffffffu, sl[r], o, LANES);
            df_add(sh[r], sl[r], bh, bl);
        }
}

// bsr_block_row_df with x given as separate high and low FP32 arrays
template <int BD, int LANES>
__device__ __forceinline__ void bsr_block_row_df_split(const int32_t *__restrict__ rows,
                                                       const int32_t *__restrict__ cols,
                                                       const float2 *__restrict__ vals, int32_t i, bool valid,
                                                       const float *__restrict__ xh, const float *__restrict__ xl,
                                                       int lane, float (&sh)[BD], float (&sl)[BD])
{
    const int32_t b = valid ? rows[i] : 0, e = valid ? rows[i + 1] : 0, len = e - b;
    const float2 *__restrict__ v = vals + (int64_t)b * (BD * BD);
#pragma unroll
    for (int r = 0; r < BD; ++r) sh[r] = sl[r] = 0.f;
    for (int32_t l = lane; l < len; l += LANES) {
        const int32_t c = __ldcs(cols + b + l);
        float x1[BD], x2[BD];
#pragma unroll
        for (int k = 0; k < BD; ++k) {
            x1[k] = xh[(int64_t)c * BD + k];
            x2[k] = xl[(int64_t)c * BD + k];
        }
#pragma unroll
        for (int r = 0; r < BD; ++r)
#pragma unroll
            for (int k = 0; k < BD; ++k) {
                const float2 a = __ldcs(v + (int64_t)(r * BD + k) * len + l);
                df_fma(sh[r], sl[r], a.x, a.y, x1[k], x2[k]);
            }
    }
#pragma unroll
    for (int r = 0; r < BD; ++r)
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            const float bh = __shfl_xor_sync(0xffffffffu, sh[r], o, LANES);
            const float bl = __shfl_xor_sync(0xffffffffu, sl[r], o, LANES);
            df_add(sh[r], sl[r], bh, bl);
        }
}

}  // namespace lss
