// Operator and PCG kernels (sm_103a): FP64 BSR/CSR SpMV with fused epilogues,
// PCG vector updates with deterministic fused reductions, permutation and
// the pattern-restricted gradient of the adjoint.
//
// PCG follows GPUHybrid::pcg_solve (GPUHybrid.cu:1413-1512): recurrence
// residual, relative test rr / bb < rel_tol^2 and absolute test rr < abs_tol^2
// every iteration, breakdown stops on p.Ap == 0, alpha <= 0 and subnormal
// alpha.  The scalars live on the device; every kernel of an iteration
// returns immediately once st->done is set, so the host only polls the flag
// every few iterations (the reference synchronises on every dot product).
#include <cfloat>

#include "device_common.cuh"
#include "kernels.hpp"
#include "mas.cuh"
#include "spmv.cuh"

namespace lss {
namespace {

__global__ void gather_values_kernel(int64_t count, const int64_t *__restrict__ src, const double *__restrict__ csc,
                                     double *__restrict__ vals, float *__restrict__ vals32,
                                     float2 *__restrict__ vals_df)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < count;
         j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = src[j];
        const double v = k >= 0 ? csc[k] : 0.0;
        vals[j] = v;
        if (vals32) vals32[j] = (float)v;
        if (vals_df) {
            const float h = (float)v;
            vals_df[j] = make_float2(h, (float)(v - (double)h));
        }
    }
}

// y = A x
template <int BD, int LANES>
__global__ void __launch_bounds__(256) spmv_kernel(BsrDev A, const double *__restrict__ x, double *__restrict__ y,
                                                   const int *done)
{
    __shared__ double buf[rows_smem<BD, LANES>];
    if (done && *done) return;
    fp64_rows<BD, LANES>(A.rows, A.cols, A.vals, A.nb, x, buf,
                         [&](int32_t i, int k, double v) { y[(int64_t)i * BD + k] = v; });
}

// y = r - A x
template <int BD, int LANES>
__global__ void __launch_bounds__(256) residual_kernel(BsrDev A, const double *__restrict__ r,
                                                       const double *__restrict__ x, double *__restrict__ y,
                                                       const int *done)
{
    __shared__ double buf[rows_smem<BD, LANES>];
    pdl_enter();
    if (done && *done) return;
    fp64_rows<BD, LANES>(A.rows, A.cols, A.vals, A.nb, x, buf, [&](int32_t i, int k, double v) {
        const int64_t e = (int64_t)i * BD + k;
        y[e] = r[e] - v;
    });
}

// y = r - A x with every product and sum carried in two doubles (TwoProd,
// TwoSum: Ogita, Rump and Oishi's Dot2) and rounded once; LANES threads per
// block row.  It starts the PCG's restarts (run_pcg), one launch each, and is bound
// by the FP64 pipe, eleven instructions a term: 42 us at 24k DOFs (the plain FP64
// residual 9), 61 us on a 150k Laplacian, half an iteration either way.
template <int BD, int LANES>
__global__ void __launch_bounds__(256) residual_twice_kernel(BsrDev A, const double *__restrict__ r,
                                                             const double *__restrict__ x, double *__restrict__ y)
{
    const int lane = threadIdx.x % LANES;
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) / LANES;
    const bool valid = i < A.nb;
    const int32_t b = valid ? A.rows[i] : 0, len = valid ? A.rows[i + 1] - b : 0;
    const double *__restrict__ v = A.vals + (int64_t)b * (BD * BD);
    auto add = [](double &h, double &l, double p, double e) {  // (h, l) += p + e
        const double t = __dadd_rn(h, p), z = __dsub_rn(t, h);
        l = __dadd_rn(l, __dadd_rn(e, __dadd_rn(__dsub_rn(h, __dsub_rn(t, z)), __dsub_rn(p, z))));
        h = t;
    };
    double sh[BD], sl[BD];
#pragma unroll
    for (int k = 0; k < BD; ++k) {  // the first lane starts from -r
        sh[k] = valid && lane == 0 ? -r[i * BD + k] : 0.0;
        sl[k] = 0.0;
    }
    for (int32_t q = lane; q < len; q += LANES) {
        const int64_t c = A.cols[b + q];
#pragma unroll
        for (int j = 0; j < BD; ++j) {
            const double xv = x[c * BD + j];
#pragma unroll
            for (int k = 0; k < BD; ++k) {
                const double a = v[(int64_t)(k * BD + j) * len + q], p = __dmul_rn(a, xv);
                add(sh[k], sl[k], p, __fma_rn(a, xv, -p));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < BD; ++k) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            const double h = __shfl_xor_sync(0xffffffffu, sh[k], o), l = __shfl_xor_sync(0xffffffffu, sl[k], o);
            add(sh[k], sl[k], h, l);
        }
        if (valid && lane == 0) y[i * BD + k] = -__dadd_rn(sh[k], sl[k]);
    }
}

// y32 = r - A x for the mixed preconditioner, rounded to FP32 (its result
// feeds the FP32 MAS).  Rows flagged in `precise` (the stiff rows: there r - A
// z cancels terms many orders larger than the result -- entries of 1e7 times a
// nearly rigid z -- which FP32 would turn into noise of the result's size) are
// evaluated in double-float (values as (hi, lo) pairs, x = x32 + x_lo, r in
// FP64); all other rows entirely in FP32.  A warp takes the double-float branch
// for all of its rows when any of them is flagged, so the group shuffles stay
// warp-uniform.
template <int BD, int LANES>
__global__ void __launch_bounds__(256) residual32_kernel(BsrDev A, const float *__restrict__ r32,
                                                         const float *__restrict__ x32, float *__restrict__ y32,
                                                         const uint8_t *__restrict__ precise,
                                                         const double *__restrict__ r64,
                                                         const float *__restrict__ x_lo, const int *done)
{
    pdl_enter();
    if (done && *done) return;
    const int lane = threadIdx.x % LANES;
    constexpr int RPW = 32 / LANES;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t wr = w0 * RPW; wr < A.nb; wr += nw * RPW) {
        const int64_t i = wr + (threadIdx.x & 31) / LANES;
        const bool valid = i < A.nb;
        const bool mine = precise && valid && precise[i];
        if (__any_sync(0xffffffffu, mine)) {
            float sh[BD], sl[BD];
            bsr_block_row_df_split<BD, LANES>(A.rows, A.cols, A.vals_df, (int32_t)i, valid, x32, x_lo, lane, sh, sl);
            if (valid) {
#pragma unroll
                for (int k = 0; k < BD; ++k)
                    if (k % LANES == lane)
                        y32[i * BD + k] = (float)(r64[i * BD + k] - ((double)sh[k] + (double)sl[k]));
            }
        } else {
            float acc[BD];
            bsr_block_row<BD, LANES, float, float, float>(A.rows, A.cols, A.vals32, (int32_t)i, valid, x32, lane,
                                                          acc);
            if (valid) {
#pragma unroll
                for (int k = 0; k < BD; ++k)
                    if (k % LANES == lane) y32[i * BD + k] = r32[i * BD + k] - acc[k];
            }
        }
    }
}

// Ap = A p and p.Ap (GPUHybrid.cu:1458-1462)
template <int BD, int LANES>
__global__ void __launch_bounds__(256) spmv_alpha_kernel(BsrDev A, const double *__restrict__ p,
                                                         double *__restrict__ Ap, const PcgState *st, GridReduce gr,
                                                         PcgSum pap)
{
    __shared__ double buf[rows_smem<BD, LANES>];
    pdl_enter();
    if (st->done) return;
    double dot = 0.0;
    fp64_rows<BD, LANES>(A.rows, A.cols, A.vals, A.nb, p, buf, [&](int32_t i, int k, double v) {
        const int64_t e = (int64_t)i * BD + k;
        Ap[e] = v;
        dot += p[e] * v;
    });
    put_sum(dot, gr, pap);
}

// update_p_kernel takes VEC rows per thread, all loaded before any is stored (its
// stores keep the compiler from hoisting the next row's loads).
constexpr int VEC = 4, VEC_ROWS = 256 * VEC;

__device__ __forceinline__ double as_double(double v) { return v; }
__device__ __forceinline__ double as_double(float2 v) { return to_double(v.x) + to_double(v.y); }

// partitions a warp takes at a time: one of block size 1 alone leaves too few
// loads in flight and too many CTAs that sum p.Ap
__host__ __device__ constexpr int XR_PARTS(int bd) { return bd == 1 ? 2 : 1; }

// alpha with the breakdown tests; x += alpha p; r -= alpha Ap; r.r
// (GPUHybrid.cu:1463-1487), and the restriction of the new r to the MAS's level-1
// items: a warp takes whole partitions, whose rows it holds anyway.  As a launch
// of its own behind this one the restriction read r again; an iteration took
// 54.9 us instead of 52.6 at 2k DOF (FP64), 67.4 / 65.2 at 24k, 114 / 108 at 207k,
// 831 / 804 at 3M (mixed), 145.8 / 142.7 on a 150k Laplacian (FP64).
// Every CTA forms alpha from the parts of p.Ap, the first one
// records the iteration's scalars.  AT: double, or float2 for the (hi, lo) product
// of the df32 SpMV; T: the MAS's type.  r32 (optional): r rounded to FP32, the
// input of the mixed preconditioner's FP32 residual.
template <int BD, typename AT, typename T>
__global__ void __launch_bounds__(256) update_xr_kernel(MasDev m, double *__restrict__ x, double *__restrict__ r,
                                                        const double *__restrict__ p, const AT *__restrict__ Ap,
                                                        PcgState *st, GridReduce gr, PcgSum pap, PcgSum rr,
                                                        T *__restrict__ v, float *__restrict__ r32)
{
    constexpr int W = 8, K = XR_PARTS(BD);
    __shared__ T xs_all[W][K][32 * BD];
    __shared__ unsigned mask_all[W][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    int64_t q = ((int64_t)blockIdx.x * W + wl) * K;
    const int64_t step = (int64_t)gridDim.x * W * K;
    MasPart t[K];  // constant: read ahead of the preceding kernel's end
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] = mas_part(m, q + k, lane);
    pdl_enter();
    // the first CTA may set done while another reads it: no thread leaves ahead of
    // the sum's barriers, and all that stay come to the same verdict
    const bool over = st->done != 0;
    struct Step {
        double alpha;
        int stop;
    };
    const Step ab = from_sum(pap, [&](double pAp) {
        const double gamma = st->rz, a = gamma / pAp;
        int c = STOP_RUNNING;
        if (pAp == 0.0) c = STOP_ZERO_PAP;
        else if (!(a == a) || isinf(a)) c = STOP_NONFINITE;
        else if (a <= 0.0) c = STOP_NEGATIVE_ALPHA;
        else if (a < DBL_MIN) c = STOP_SUBNORMAL_ALPHA;
        if (blockIdx.x == 0 && !over) {
            const int it = st->iter + 1;
            st->iter = it;
            st->pAp = pAp;
            st->gamma = gamma;
            if (c) st->done = c;
            else {
                st->alpha = a;
                if (it <= PCG_HIST) st->hist_alpha[it - 1] = a;
            }
        }
        return Step{a, c};
    });
    if (over || ab.stop) return;
    const double alpha = ab.alpha;
    double s = 0.0;
    for (; q < m.nparts; q += step) {
        double xv[K][BD], pv[K][BD], rv[K][BD];
        AT av[K][BD];
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int j = 0; j < BD; ++j) {
                const int e = j * 32 + lane;
                if (e >= t[k].cnt * BD) break;
                const int64_t i = (int64_t)t[k].lo * BD + e;
                xv[k][j] = x[i];
                pv[k][j] = p[i];
                rv[k][j] = r[i];
                av[k][j] = Ap[i];
            }
        }
        MasPart next[K];
#pragma unroll
        for (int k = 0; k < K; ++k) next[k] = mas_part(m, q + step + k, lane);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            T *xs = xs_all[wl][k];
#pragma unroll
            for (int j = 0; j < BD; ++j) {
                const int e = j * 32 + lane;
                if (e >= t[k].cnt * BD) break;
                const int64_t i = (int64_t)t[k].lo * BD + e;
                x[i] = xv[k][j] + alpha * pv[k][j];
                const double ri = rv[k][j] - alpha * as_double(av[k][j]);
                r[i] = ri;
                if (sizeof(T) == 4 || r32) {
                    const float f = to_float(ri);
                    if (r32) r32[i] = f;
                    if (sizeof(T) == 4) xs[e] = (T)f;
                }
                if (sizeof(T) == 8) xs[e] = (T)ri;
                s += ri * ri;
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < K; ++k) {
            bank_segment_sums<BD, T>(xs_all[wl][k], t[k].key, mask_all[wl], t[k].nc,
                                     v + m.voff[1] + (int64_t)t[k].i0 * BD, lane);
            __syncwarp();
            t[k] = next[k];
        }
    }
    put_sum(s, gr, rr);
}

// beta = r.z / gamma, p = z + beta p (GPUHybrid.cu:1501-1507), first: p = z;
// optionally also the df32 split of p
__global__ void __launch_bounds__(256) update_p_kernel(int64_t n, double *__restrict__ p, const double *__restrict__ z,
                                                       PcgState *st, PcgSum rz, bool first, float2 *__restrict__ p_df)
{
    pdl_enter();
    if (st->done) return;
    const double beta = from_sum(rz, [&](double g) {
        const double b = first ? 0.0 : g / st->gamma;
        if (blockIdx.x == 0) {
            st->rz = g;
            if (!first) {
                st->beta = b;
                if (st->iter >= 1 && st->iter <= PCG_HIST) st->hist_beta[st->iter - 1] = b;
            }
        }
        return b;
    });
    for (int64_t i0 = (int64_t)blockIdx.x * VEC_ROWS + threadIdx.x; i0 < n; i0 += (int64_t)gridDim.x * VEC_ROWS) {
        double zv[VEC], pv[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const int64_t i = i0 + j * 256;
            if (i >= n) break;
            zv[j] = z[i];
            pv[j] = first ? 0.0 : p[i];
        }
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const int64_t i = i0 + j * 256;
            if (i >= n) break;
            const double v = first ? zv[j] : zv[j] + beta * pv[j];
            p[i] = v;
            if (p_df) p_df[i] = split_double(v);
        }
    }
}

__global__ void split_kernel(int64_t n, const double *__restrict__ src, float2 *__restrict__ dst)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dst[i] = split_double(src[i]);
    }
}

// spmv_alpha_kernel with the SpMV in double-float on the FP32 pipe.  A p
// leaves as (hi, lo) pairs and p.Ap accumulates in double-float, so the loop
// issues no FP64 instruction: the storing lanes (k % LANES == lane) would
// run them as partly predicated warps, each costing the FP64 pipe a full warp.
template <int BD, int LANES>
__global__ void __launch_bounds__(256) spmv_alpha_df_kernel(BsrDev A, const float2 *__restrict__ p_df,
                                                            float2 *__restrict__ Ap, const PcgState *st, GridReduce gr,
                                                            PcgSum pap)
{
    pdl_enter();
    if (st->done) return;
    const int lane = threadIdx.x % LANES;
    constexpr int RPW = 32 / LANES;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    float dh = 0.f, dl = 0.f;
    for (int64_t wr = w0 * RPW; wr < A.nb; wr += nw * RPW) {
        const int64_t i = wr + (threadIdx.x & 31) / LANES;
        const bool valid = i < A.nb;
        float sh[BD], sl[BD];
        bsr_block_row_df<BD, LANES>(A.rows, A.cols, A.vals_df, (int32_t)i, valid, p_df, lane, sh, sl);
        if (valid) {
#pragma unroll
            for (int k = 0; k < BD; ++k)
                if (k % LANES == lane) {
                    Ap[i * BD + k] = make_float2(sh[k], sl[k]);
                    const float2 pk = p_df[i * BD + k];
                    df_fma(dh, dl, pk.x, pk.y, sh[k], sl[k]);
                }
        }
    }
    put_sum((double)dh + (double)dl, gr, pap);
}

__global__ void __launch_bounds__(256) dot_kernel(int64_t n, const double *__restrict__ a, const double *__restrict__ b,
                                                  double *out, GridReduce gr)
{
    double s[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s[0] += a[i] * b[i];
    double tot[1];
    if (grid_sum<1>(s, gr, tot)) *out = tot[0];
}

__global__ void permute_kernel(int64_t nb, int bd, const int32_t *__restrict__ perm, const double *__restrict__ src,
                               double *__restrict__ dst, bool to_new)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nb * bd;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t blk = i / bd, c = i % bd;
        const int64_t q = (int64_t)perm[blk] * bd + c;
        if (to_new) dst[q] = src[i];
        else dst[i] = src[q];
    }
}

// dA[k] = -lambda[row] * x[col] over the stored pattern (outer = row)
__global__ void grad_pattern_kernel(int32_t n, const int32_t *__restrict__ outer, const int32_t *__restrict__ inner,
                                    const double *__restrict__ lambda, const double *__restrict__ x,
                                    double *__restrict__ dA)
{
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = w0; i < n; i += nw) {
        const double li = lambda[i];
        for (int32_t k = outer[i] + lane; k < outer[i + 1]; k += 32) dA[k] = -li * x[inner[k]];
    }
}

__global__ void __launch_bounds__(256) rz_kernel(int64_t n, const double *__restrict__ r, const double *__restrict__ z,
                                                 const PcgState *st, GridReduce gr, PcgSum rz)
{
    pdl_enter();
    if (st->done) return;
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += r[i] * z[i];
    put_sum(s, gr, rz);
}

__global__ void check_finite_kernel(int64_t n, const double *__restrict__ v, int *flag)
{
    bool bad = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        bad |= !isfinite(v[i]);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// Fused adjoint scatter: the pattern gradient -lambda_i x_j is formed on the
// fly for the stored entries an element touches and reduced into its
// parameter (one warp per parameter row of the element -> entry map).
__global__ void __launch_bounds__(256) grad_params_kernel(int32_t nparams, const int64_t *__restrict__ rp,
                                                          const int32_t *__restrict__ cols,
                                                          const double *__restrict__ vals,
                                                          const int32_t *__restrict__ row_of,
                                                          const int32_t *__restrict__ inner,
                                                          const double *__restrict__ lambda,
                                                          const double *__restrict__ x, double *__restrict__ dtheta)
{
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t e = w0; e < nparams; e += nw) {
        double acc = 0.0;
        for (int64_t k = rp[e] + lane; k < rp[e + 1]; k += 32) {
            const int32_t v = cols[k];
            acc -= vals[k] * lambda[row_of[v]] * x[inner[v]];
        }
        acc = warp_sum(acc);
        if (lane == 0) dtheta[e] = acc;
    }
}

// values[v] = sum_k mvals[k] theta[mcols[k]] over the CSR row v of M, + c[v]:
// one thread per stored entry of A (rows of a few dozen parameters)
__global__ void __launch_bounds__(256) assemble_values_kernel(int64_t nvals, const int64_t *__restrict__ rowptr,
                                                              const int32_t *__restrict__ mcols,
                                                              const double *__restrict__ mvals,
                                                              const double *__restrict__ theta,
                                                              const double *__restrict__ c, double *__restrict__ out)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvals; v += (int64_t)gridDim.x * blockDim.x) {
        double acc = c ? c[v] : 0.0;
        for (int64_t k = rowptr[v]; k < rowptr[v + 1]; ++k) acc += mvals[k] * theta[mcols[k]];
        out[v] = acc;
    }
}

__global__ void row_of_kernel(int32_t n, const int32_t *__restrict__ outer, int32_t *__restrict__ row_of)
{
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = w0; i < n; i += nw)
        for (int32_t k = outer[i] + lane; k < outer[i + 1]; k += 32) row_of[k] = (int32_t)i;
}

template <int BD>
void spmv_dispatch(const BsrDev &A, const double *x, double *y, const int *done, cudaStream_t s)
{
    const int grid = grid_for((int64_t)A.nb * A.lanes, 256, sm_grid(16));
    switch (A.lanes) {
    case 1: spmv_kernel<BD, 1><<<grid, 256, 0, s>>>(A, x, y, done); break;
    case 2: spmv_kernel<BD, 2><<<grid, 256, 0, s>>>(A, x, y, done); break;
    case 4: spmv_kernel<BD, 4><<<grid, 256, 0, s>>>(A, x, y, done); break;
    case 8: spmv_kernel<BD, 8><<<grid, 256, 0, s>>>(A, x, y, done); break;
    case 16: spmv_kernel<BD, 16><<<grid, 256, 0, s>>>(A, x, y, done); break;
    default: spmv_kernel<BD, 32><<<grid, 256, 0, s>>>(A, x, y, done); break;
    }
}

template <int BD>
void residual_dispatch(const BsrDev &A, const double *r, const double *x, double *y, const int *done, cudaStream_t s)
{
    const int grid = grid_for((int64_t)A.nb * A.lanes, 256, sm_grid(16));
#define LSS_RES(L_) launch_pdl(residual_kernel<BD, L_>, grid, 256, 0, s, A, r, x, y, done)
    switch (A.lanes) {
    case 1: LSS_RES(1); break;
    case 2: LSS_RES(2); break;
    case 4: LSS_RES(4); break;
    case 8: LSS_RES(8); break;
    case 16: LSS_RES(16); break;
    default: LSS_RES(32); break;
    }
#undef LSS_RES
}

// marks `sum` as produced by a launch of `grid` CTAs over n rows
void produced(PcgSum &sum, int64_t n, int grid)
{
    sum.direct = n <= PCG_DIRECT_ROWS;
    sum.count = sum.direct ? grid : 1;
}

// CTAs of the outer product.  Eight per SM are resident at most; where its
// consumers add a part per CTA there are no more than those (207k DOF: 2432 parts
// cost the update 1 us more than 1216).
template <int BD>
int product_grid(const BsrDev &A)
{
    return grid_for((int64_t)A.nb * A.lanes, 256, sm_grid((int64_t)A.nb * BD <= PCG_DIRECT_ROWS ? 8 : 16));
}

template <int BD>
void spmv_alpha_dispatch(const BsrDev &A, const double *p, double *Ap, const PcgState *st, GridReduce gr, PcgSum &pap,
                         cudaStream_t s)
{
    const int grid = product_grid<BD>(A);
    produced(pap, (int64_t)A.nb * BD, grid);
#define LSS_SA(L_) launch_pdl(spmv_alpha_kernel<BD, L_>, grid, 256, 0, s, A, p, Ap, st, gr, pap)
    switch (A.lanes) {
    case 1: LSS_SA(1); break;
    case 2: LSS_SA(2); break;
    case 4: LSS_SA(4); break;
    case 8: LSS_SA(8); break;
    case 16: LSS_SA(16); break;
    default: LSS_SA(32); break;
    }
#undef LSS_SA
}

}  // namespace

void launch_gather_values(int64_t count, const int64_t *src, const double *csc, double *vals, float *vals32,
                          cudaStream_t s, float2 *vals_df)
{
    if (count == 0) return;
    gather_values_kernel<<<grid_for(count, 256, sm_grid(16)), 256, 0, s>>>(count, src, csc, vals, vals32, vals_df);
    LSS_LAUNCH_CHECK();
}

void launch_spmv(const BsrDev &A, const double *x, double *y, const int *done, cudaStream_t s)
{
    if (A.bd == 1) spmv_dispatch<1>(A, x, y, done, s);
    else if (A.bd == 2) spmv_dispatch<2>(A, x, y, done, s);
    else spmv_dispatch<3>(A, x, y, done, s);
    LSS_LAUNCH_CHECK();
}

void launch_residual_spmv(const BsrDev &A, const double *r, const double *x, double *y, const int *done,
                          cudaStream_t s)
{
    if (A.bd == 1) residual_dispatch<1>(A, r, x, y, done, s);
    else if (A.bd == 2) residual_dispatch<2>(A, r, x, y, done, s);
    else residual_dispatch<3>(A, r, x, y, done, s);
    LSS_LAUNCH_CHECK();
}

void launch_residual_twice(const BsrDev &A, const double *r, const double *x, double *y, cudaStream_t s)
{
    if (A.nb == 0) return;
    if (A.bd == 1) residual_twice_kernel<1, 4><<<(unsigned)(((int64_t)A.nb * 4 + 255) / 256), 256, 0, s>>>(A, r, x, y);
    else {
        const unsigned grid = (unsigned)(((int64_t)A.nb * 8 + 255) / 256);
        if (A.bd == 2) residual_twice_kernel<2, 8><<<grid, 256, 0, s>>>(A, r, x, y);
        else residual_twice_kernel<3, 8><<<grid, 256, 0, s>>>(A, r, x, y);
    }
    LSS_LAUNCH_CHECK();
}

template <int BD>
void residual32_dispatch(const BsrDev &A, const float *r32, const float *x32, float *y32, const uint8_t *precise,
                         const double *r64, const float *x_lo, const int *done, cudaStream_t s)
{
    const int grid = grid_for((int64_t)A.nb * A.lanes32, 256, sm_grid(16));
#define LSS_R32(L_) launch_pdl(residual32_kernel<BD, L_>, grid, 256, 0, s, A, r32, x32, y32, precise, r64, x_lo, done)
    switch (A.lanes32) {
    case 1: LSS_R32(1); break;
    case 2: LSS_R32(2); break;
    case 4: LSS_R32(4); break;
    case 8: LSS_R32(8); break;
    case 16: LSS_R32(16); break;
    default: LSS_R32(32); break;
    }
#undef LSS_R32
}

void launch_residual32(const BsrDev &A, const float *r32, const float *x32, float *y32, const int *done,
                       cudaStream_t s, const uint8_t *precise, const double *r64, const float *x_lo)
{
    if (A.nb > 0 && (!A.vals32 || !r32 || !x32 || !y32))
        fail(LSS_ERR_INTERNAL, "FP32 residual SpMV launched without its operand arrays");
    if (precise && (!A.vals_df || !r64 || !x_lo))
        fail(LSS_ERR_INTERNAL, "double-float rows of the FP32 residual need their operand arrays");
    if (A.bd == 1) residual32_dispatch<1>(A, r32, x32, y32, precise, r64, x_lo, done, s);
    else if (A.bd == 2) residual32_dispatch<2>(A, r32, x32, y32, precise, r64, x_lo, done, s);
    else residual32_dispatch<3>(A, r32, x32, y32, precise, r64, x_lo, done, s);
    LSS_LAUNCH_CHECK();
}

void launch_dot(int64_t n, const double *a, const double *b, double *out, GridReduce gr, cudaStream_t s)
{
    dot_kernel<<<grid_for(n, 1024, sm_grid(16)), 256, 0, s>>>(n, a, b, out, gr);
    LSS_LAUNCH_CHECK();
}

void launch_pcg_spmv_alpha(const BsrDev &A, const double *p, double *Ap, const PcgState *st, GridReduce gr,
                           PcgSum &pap, cudaStream_t s)
{
    if (A.bd == 1) spmv_alpha_dispatch<1>(A, p, Ap, st, gr, pap, s);
    else if (A.bd == 2) spmv_alpha_dispatch<2>(A, p, Ap, st, gr, pap, s);
    else spmv_alpha_dispatch<3>(A, p, Ap, st, gr, pap, s);
    LSS_LAUNCH_CHECK();
}

template <int BD>
void spmv_alpha_df_dispatch(const BsrDev &A, const float2 *pd, float2 *Ap, const PcgState *st, GridReduce gr,
                            PcgSum &pap, cudaStream_t s)
{
    const int grid = product_grid<BD>(A);
    produced(pap, (int64_t)A.nb * BD, grid);
#define LSS_SA(L_) launch_pdl(spmv_alpha_df_kernel<BD, L_>, grid, 256, 0, s, A, pd, Ap, st, gr, pap)
    switch (A.lanes) {
    case 1: LSS_SA(1); break;
    case 2: LSS_SA(2); break;
    case 4: LSS_SA(4); break;
    case 8: LSS_SA(8); break;
    case 16: LSS_SA(16); break;
    default: LSS_SA(32); break;
    }
#undef LSS_SA
}

void launch_pcg_spmv_alpha_df(const BsrDev &A, const float2 *p_df, float2 *Ap_df, const PcgState *st, GridReduce gr,
                              PcgSum &pap, cudaStream_t s)
{
    if (A.nb > 0 && (!A.vals_df || !p_df || !Ap_df))
        fail(LSS_ERR_INTERNAL, "df32 SpMV launched without its operand arrays");
    if (A.bd == 1) spmv_alpha_df_dispatch<1>(A, p_df, Ap_df, st, gr, pap, s);
    else if (A.bd == 2) spmv_alpha_df_dispatch<2>(A, p_df, Ap_df, st, gr, pap, s);
    else spmv_alpha_df_dispatch<3>(A, p_df, Ap_df, st, gr, pap, s);
    LSS_LAUNCH_CHECK();
}

// dst[perm-ordered] = v_i = ((i * 2654435761) mod 2^32) / 2^32 - 0.5 of the
// original index i (the damping estimate's probe vector)
__global__ void probe_kernel(int64_t nb, int bd, const int32_t *__restrict__ perm, double *__restrict__ dst)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nb * bd;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t h = (uint32_t)((uint64_t)(uint32_t)i * 2654435761u);
        dst[(int64_t)perm[i / bd] * bd + i % bd] = (double)h / 4294967296.0 - 0.5;
    }
}

void launch_probe(int64_t nb, int bd, const int32_t *perm, double *dst, cudaStream_t s)
{
    if (nb == 0) return;
    probe_kernel<<<grid_for(nb * bd, 1024, sm_grid(16)), 256, 0, s>>>(nb, bd, perm, dst);
    LSS_LAUNCH_CHECK();
}

__global__ void df_to_double_kernel(int64_t n, const float2 *__restrict__ src, double *__restrict__ dst)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = as_double(src[i]);
}

void launch_df_to_double(int64_t n, const float2 *src, double *dst, cudaStream_t s)
{
    if (n == 0) return;
    df_to_double_kernel<<<grid_for(n, 1024, sm_grid(16)), 256, 0, s>>>(n, src, dst);
    LSS_LAUNCH_CHECK();
}

void launch_split(int64_t n, const double *src, float2 *dst, cudaStream_t s)
{
    if (n == 0) return;
    if (!src || !dst) fail(LSS_ERR_INTERNAL, "split launched without its arrays");
    split_kernel<<<grid_for(n, 1024, sm_grid(16)), 256, 0, s>>>(n, src, dst);
    LSS_LAUNCH_CHECK();
}

void launch_pcg_update_xr(const MasDev &m, double *x, double *r, const double *p, const double *Ap,
                          const float2 *Ap_df, PcgState *st, GridReduce gr, PcgSum pap, PcgSum &rr, void *v, bool fp32,
                          cudaStream_t s, float *r32)
{
    const int grid = grid_for(m.nparts, 8 * XR_PARTS(m.bd), sm_grid(8));
    produced(rr, (int64_t)m.nb * m.bd, grid);
#define LSS_XR(BD_, AT_, T_, A_) \
    launch_pdl(update_xr_kernel<BD_, AT_, T_>, grid, 256, 0, s, m, x, r, p, A_, st, gr, pap, rr, (T_ *)v, r32)
#define LSS_XR_BD(BD_)                                 \
    do {                                               \
        if (Ap_df && fp32) LSS_XR(BD_, float2, float, Ap_df); \
        else if (Ap_df) LSS_XR(BD_, float2, double, Ap_df);   \
        else if (fp32) LSS_XR(BD_, double, float, Ap);        \
        else LSS_XR(BD_, double, double, Ap);                 \
    } while (0)
    if (m.bd == 1) LSS_XR_BD(1);
    else if (m.bd == 2) LSS_XR_BD(2);
    else LSS_XR_BD(3);
#undef LSS_XR_BD
#undef LSS_XR
    LSS_LAUNCH_CHECK();
}

void launch_pcg_update_p(int64_t n, double *p, const double *z, PcgState *st, PcgSum rz, bool first, cudaStream_t s,
                         float2 *p_df)
{
    launch_pdl(update_p_kernel, grid_for(n, 1024, sm_grid(16)), 256, 0, s, n, p, z, st, rz, first, p_df);
    LSS_LAUNCH_CHECK();
}

void launch_permute(int64_t nb, int bd, const int32_t *perm, const double *src, double *dst, bool to_new,
                    cudaStream_t s)
{
    permute_kernel<<<grid_for(nb * bd, 1024, sm_grid(16)), 256, 0, s>>>(nb, bd, perm, src, dst, to_new);
    LSS_LAUNCH_CHECK();
}

void launch_pcg_rz(int64_t n, const double *r, const double *z, const PcgState *st, GridReduce gr, PcgSum &rz,
                   cudaStream_t s)
{
    const int grid = grid_for(n, 1024, sm_grid(16));
    produced(rz, n, grid);
    launch_pdl(rz_kernel, grid, 256, 0, s, n, r, z, st, gr, rz);
    LSS_LAUNCH_CHECK();
}

void launch_check_finite(int64_t n, const double *v, int *flag, cudaStream_t s)
{
    if (n == 0) return;
    check_finite_kernel<<<grid_for(n, 1024, sm_grid(16)), 256, 0, s>>>(n, v, flag);
    LSS_LAUNCH_CHECK();
}

void launch_grad_params(int32_t nparams, const int64_t *mt_rowptr, const int32_t *mt_cols, const double *mt_vals,
                        const int32_t *row_of, const int32_t *inner, const double *lambda, const double *x,
                        double *dtheta, cudaStream_t s)
{
    if (nparams <= 0) return;
    grad_params_kernel<<<grid_for((int64_t)nparams * 32, 256, sm_grid(16)), 256, 0, s>>>(
        nparams, mt_rowptr, mt_cols, mt_vals, row_of, inner, lambda, x, dtheta);
    LSS_LAUNCH_CHECK();
}

void launch_assemble_values(int64_t nvals, const int64_t *rowptr, const int32_t *mcols, const double *mvals,
                            const double *theta, const double *c, double *out, cudaStream_t s)
{
    if (nvals <= 0) return;
    assemble_values_kernel<<<grid_for(nvals, 256, sm_grid(16)), 256, 0, s>>>(nvals, rowptr, mcols, mvals, theta, c,
                                                                            out);
    LSS_LAUNCH_CHECK();
}

void launch_row_of(int32_t n, const int32_t *outer, int32_t *row_of, cudaStream_t s)
{
    row_of_kernel<<<grid_for((int64_t)n * 32, 256, sm_grid(16)), 256, 0, s>>>(n, outer, row_of);
    LSS_LAUNCH_CHECK();
}

void launch_grad_pattern(int32_t n, const int32_t *outer, const int32_t *inner, const double *lambda,
                         const double *x, double *dA, cudaStream_t s)
{
    grad_pattern_kernel<<<grid_for((int64_t)n * 32, 256, sm_grid(16)), 256, 0, s>>>(n, outer, inner, lambda, x, dA);
    LSS_LAUNCH_CHECK();
}

}  // namespace lss
