// Stiff-block direct solve (sm_103a), dense part.
//
// The reference factors each stiff subdomain with cuDSS (batched sparse
// LDL^T) or, up to max_dense_size, with cuBLAS getrf/getri explicit inverses
// (GPUHybrid.cu:993-1411), and applies next_z = z + S^T A_SS^-1 S (r - A z)
// (dss_precond_iter, GPUHybrid.cu:544-675).  Here a subdomain of up to
// STIFF_DENSE_MAX DOFs is gathered into a dense FP64 block, inverted in FP64
// by the symmetric sweep (up to 64 DOFs one CTA in shared memory, beyond by the
// blocked sweep of multifrontal.cu) and applied as a GEMV fused with the scatter; larger subdomains get the FP64
// multifrontal factor (multifrontal.cu).  The residual rows r - A z are only
// computed on the stiff rows (the reference forms the full product and
// gathers it).
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"
#include "spmv.cuh"

namespace lss {
namespace {

template <int BD>
__global__ void __launch_bounds__(256) extract_kernel(BsrDev A, StiffDev S, double *__restrict__ stage)
{
    const int lane = threadIdx.x & 31;
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= S.ndof_dense) return;
    const int32_t d = S.dofs[j], I = d / BD, comp = d % BD;
    const int32_t s = S.sub_of[j], o = S.off[s], m = S.off[s + 1] - o;
    const int32_t *list = S.dofs + o;
    double *row = stage + S.inv_off[s] + (int64_t)(j - o) * m;
    const int32_t b = A.rows[I], len = A.rows[I + 1] - b;
    const double *v = A.vals + (int64_t)b * BD * BD;
    for (int32_t l = lane; l < len; l += 32) {
        const int32_t J = A.cols[b + l];
#pragma unroll
        for (int k = 0; k < BD; ++k) {
            const int32_t col = J * BD + k;
            int32_t lo = 0, hi = m;
            while (lo < hi) {
                const int32_t mid = (lo + hi) >> 1;
                if (list[mid] < col) lo = mid + 1;
                else hi = mid;
            }
            if (lo < m && list[lo] == col) row[lo] = v[(int64_t)(comp * BD + k) * len + l];
        }
    }
}

__device__ void sweep_invert_small(double *S, int ld, int N, double *col, double *scol, int *bad)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    for (int p = 0; p < N; ++p) {
        const double piv = S[p * ld + p];
        for (int t = tid; t < N; t += nt) {
            const double cv = (t == p) ? 0.0 : S[t * ld + p];
            col[t] = cv;
            scol[t] = cv / piv;
        }
        if (tid == 0 && (!isfinite(piv) || piv == 0.0)) atomicOr(bad, 4);
        __syncthreads();
        for (int t = wid; t < N; t += nw) {
            if (t == p) continue;
            const double st = scol[t];
            for (int c = lane; c < N; c += 32)
                if (c != p) S[t * ld + c] -= st * col[c];
        }
        __syncthreads();
        for (int t = tid; t < N; t += nt) {
            if (t == p) S[p * ld + p] = -1.0 / piv;
            else {
                S[t * ld + p] = scol[t];
                S[p * ld + t] = scol[t];
            }
        }
        __syncthreads();
    }
}

// one CTA per subdomain of at most max_m DOFs (the others are swept blocked),
// in place in global storage
__global__ void __launch_bounds__(256) invert_small_kernel(const int32_t *__restrict__ off,
                                                           const int64_t *__restrict__ inv_off,
                                                           double *__restrict__ inv, int max_m, int *bad)
{
    extern __shared__ double sm[];
    const int32_t s = blockIdx.x;  // the dense subdomains come first
    const int m = off[s + 1] - off[s], ld = m + 1;
    if (m > max_m) return;
    double *S = sm, *col = sm + m * ld, *scol = col + m;
    double *g = inv + inv_off[s];
    for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
        const int r = idx / m, c = idx % m;
        S[r * ld + c] = (r <= c) ? g[(int64_t)r * m + c] : g[(int64_t)c * m + r];
    }
    __syncthreads();
    sweep_invert_small(S, ld, m, col, scol, bad);
    // stored transposed (column-major): thread j of the apply reads row j as a column
    for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
        const int r = idx / m, c = idx % m;
        const double val = -S[r * ld + c];
        if (!isfinite(val)) atomicOr(bad, 8);
        g[(int64_t)c * m + r] = val;
    }
}

// t_j = r_d (- (A z)_d) for the stiff DOFs d = dofs[j], LANES threads per DOF
// (blocks l = lane, lane + LANES, ... of its row; the sums meet by shuffles).
// The stiff DOFs are few, so this is bound by the latency of the row's chain
// bounds -> columns -> z: one thread walking a row of 15 blocks took 14 us,
// eight of them 6; the two or three shuffled FP64 adds cost the pipe less than
// the row's products.
template <int BD, int LANES>
__global__ void __launch_bounds__(256) gather_kernel(BsrDev A, StiffDev S, const double *__restrict__ r,
                                                     const double *__restrict__ z, bool residual, const int *done)
{
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int lane = threadIdx.x % LANES;
    const bool valid = j < S.ndof;
    const int32_t d = valid ? S.dofs[j] : 0, i = d / BD, comp = d % BD;
    const int32_t b = valid ? A.rows[i] : 0, len = valid ? A.rows[i + 1] - b : 0;
    pdl_enter();
    if (done && *done) return;
    double acc = 0.0;
    if (residual) {
        const double *v = A.vals + (int64_t)b * BD * BD;
#pragma unroll 2
        for (int32_t l = lane; l < len; l += LANES) {
            const int32_t c = A.cols[b + l];
#pragma unroll
            for (int k = 0; k < BD; ++k) acc += v[(int64_t)(comp * BD + k) * len + l] * z[(int64_t)c * BD + k];
        }
        acc = group_sum<LANES>(acc);
    }
    if (valid && lane == 0) S.t[j] = r[d] - acc;
}

// z_S += Inv t over the dense subdomains, by the warps of StiffDev::warps: a
// warp takes 32 rows of one subdomain (lane = row, read as a column of the
// transposed storage, so a load is one line) and one of nsl slices of the
// columns; the slices' sums meet in shared memory in slice order.  Slices hold
// at most 24 columns: one thread summing a whole row of up to 160 took 30 to
// 45 us of dependent loads.
template <typename VT>
__global__ void __launch_bounds__(256) apply_kernel(StiffDev S, const VT *__restrict__ inv, double *__restrict__ z,
                                                    float *__restrict__ z32, float *__restrict__ z_lo, const int *done)
{
    __shared__ double red[8][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int32_t wi = blockIdx.x * 8 + wl;
    const StiffWarp w = wi < S.nwarps ? S.warps[wi] : StiffWarp{};
    const bool row = lane < w.m - w.row0;
    const int32_t d = row ? S.dofs[w.off + w.row0 + lane] : 0;
    pdl_enter();
    if (done && *done) return;
    double acc = 0.0;
    if (row) {
        const VT *__restrict__ col = inv + w.inv_off + w.row0 + lane;
        const double *__restrict__ t = S.t + w.off;
        const int32_t q1 = min(w.m, (w.slice + 1) * w.width);
#pragma unroll 8
        for (int32_t q = w.slice * w.width; q < q1; ++q) acc += (double)col[(int64_t)q * w.m] * t[q];
    }
    red[wl][lane] = acc;
    __syncthreads();
    if (!row || w.slice > 0) return;
    for (int k = 1; k < w.nsl; ++k) acc += red[wl + k][lane];
    const double nz = z[d] + acc;
    z[d] = nz;
    if (z32) {
        const float h = (float)nz;
        z32[d] = h;
        if (z_lo) z_lo[d] = (float)(nz - (double)h);
    }
}

__global__ void to_fp32_kernel(int64_t count, const double *__restrict__ src, float *__restrict__ dst)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}

}  // namespace

void launch_stiff_extract(const BsrDev &A, const StiffDev &S, double *stage, cudaStream_t s)
{
    if (S.ndof_dense == 0) return;
    const int grid = (int)(((int64_t)S.ndof_dense * 32 + 255) / 256);
    switch (A.bd) {
    case 1: extract_kernel<1><<<grid, 256, 0, s>>>(A, S, stage); break;
    case 2: extract_kernel<2><<<grid, 256, 0, s>>>(A, S, stage); break;
    default: extract_kernel<3><<<grid, 256, 0, s>>>(A, S, stage); break;
    }
    LSS_LAUNCH_CHECK();
}

void launch_stiff_invert(const StiffDev &S, const int32_t *h_off, int32_t nsub, int max_m, double *inv, int *bad,
                         cudaStream_t s)
{
    int m = 0;
    for (int32_t q = 0; q < nsub; ++q)
        if (h_off[q + 1] - h_off[q] <= max_m) m = std::max(m, h_off[q + 1] - h_off[q]);
    if (m == 0) return;
    const size_t smem = (size_t)(m * (m + 1) + 2 * m) * sizeof(double);
    raise_smem_limit((const void *)invert_small_kernel, smem);
    invert_small_kernel<<<(unsigned)nsub, 256, smem, s>>>(S.off, S.inv_off, inv, max_m, bad);
    LSS_LAUNCH_CHECK();
}

void launch_stiff_to_fp32(int64_t count, const double *src, float *dst, cudaStream_t s)
{
    if (count > 0 && (!src || !dst)) fail(LSS_ERR_INTERNAL, "FP32 conversion launched without its arrays");
    if (count == 0) return;
    to_fp32_kernel<<<grid_for(count, 256, sm_grid(8)), 256, 0, s>>>(count, src, dst);
    LSS_LAUNCH_CHECK();
}

void launch_stiff_gather(const BsrDev &A, const StiffDev &S, const double *r, const double *z, bool residual,
                         const int *done, cudaStream_t s)
{
    if (S.ndof == 0) return;
    auto go = [&](auto kernel, int lanes) {
        launch_pdl(kernel, (unsigned)(((int64_t)S.ndof * lanes + 255) / 256), 256, 0, s, A, S, r, z, residual, done);
    };
    switch (A.bd) {
    case 1: go(gather_kernel<1, 4>, 4); break;
    case 2: go(gather_kernel<2, 8>, 8); break;
    default: go(gather_kernel<3, 8>, 8); break;
    }
    LSS_LAUNCH_CHECK();
}

void launch_stiff_apply(const StiffDev &S, bool fp32, double *z, const int *done, cudaStream_t s, float *z32,
                        float *z_lo)
{
    if (S.nwarps == 0) return;
    const unsigned grid = (unsigned)((S.nwarps + 7) / 8);
    if (fp32) launch_pdl(apply_kernel<float>, grid, 256, 0, s, S, S.inv32, z, z32, z_lo, done);
    else launch_pdl(apply_kernel<double>, grid, 256, 0, s, S, S.inv, z, z32, z_lo, done);
    LSS_LAUNCH_CHECK();
}

std::vector<StiffWarp> stiff_warps(const std::vector<int32_t> &off, const std::vector<int64_t> &inv_off,
                                   int32_t ndense)
{
    std::vector<StiffWarp> out;
    // groups of 8, 4, 2, 1 warps in this order: no group straddles a CTA
    for (int nsl = 8; nsl >= 1; nsl /= 2)
        for (int32_t s = 0; s < ndense; ++s) {
            const int32_t m = off[s + 1] - off[s];
            const int need = m <= 24 ? 1 : (m <= 48 ? 2 : (m <= 96 ? 4 : 8));
            if (need != nsl) continue;
            for (int32_t r = 0; r < m; r += 32)
                for (int k = 0; k < nsl; ++k)
                    out.push_back({inv_off[s], off[s], m, r, k, nsl, (m + nsl - 1) / nsl});
        }
    return out;
}

}  // namespace lss
