// Multilevel additive Schwarz (MAS) preconditioner kernels (sm_103a).
//
// Semantics follow MASPreconditioner (MASPreconditioner.cu:376-1164 in the
// reference): level 0 = one 32*bd x 32*bd block per partition ("bank"), coarse
// level l = banks of 32 consecutive components of level l-1; each bank's
// Galerkin block is inverted exactly; apply = restrict (sum) -> per-bank
// symmetric matrix-vector product -> prolong (inject and add).
//
// GB300 layout of the inverses ("circulant tiles").  Inside a bank the scalar
// index is component-major (comp * 32 + lane).  The N x N inverse is cut into
// 32 x 32 tiles (c, c2), c <= c2; tile element [d][r] holds
// Inv[c*32 + r][c2*32 + (r+d) % 32], d = 0..16 for diagonal tiles (d = 16 kept
// twice, so 17*32 entries = the packed-triangle size plus 16) and d = 0..31 for
// off-diagonal tiles.  Row r of a tile is at lane r of every 32-entry line,
// so a warp's access to a tile, direct or transposed, is 32 consecutive or
// rotated words (128 bytes in FP32, 256 in FP64): one half of the symmetric
// matrix is stored and read from HBM, both halves of the product run from
// shared memory.  Residual and coarse vectors stay in L2.
#include <cuda_bf16.h>

#include <type_traits>

#include "device_common.cuh"
#include "kernels.hpp"
#include "mas.cuh"

namespace lss {

int64_t mas_tile_elems(int bd) { return (int64_t)bd * 17 * 32 + (int64_t)bd * (bd - 1) / 2 * 1024; }
int64_t mas_bank_bytes_bf16(int bd) { return (int64_t)bd * 17 * 32 * 4 + (int64_t)bd * (bd - 1) / 2 * 1024 * 2; }

namespace {

template <int BD>
__host__ __device__ constexpr int64_t tile_elems() { return (int64_t)BD * 17 * 32 + (int64_t)BD * (BD - 1) / 2 * 1024; }

// The bank product y = Inv x, split over warps.  With x in shared memory,
// output row r (= lane) of component c1 takes, for every component c and
// rotation e = 0..31, Inv[c1*32 + r][c*32 + (r+e) % 32] * x[c*32 + (r+e) % 32].
// That entry is tile (c1, c)[e][r] for c1 <= c (e <= 16 on the diagonal) and,
// by symmetry, tile (c, c1)[32 - e][(r+e) % 32] otherwise: both a conflict-free
// (coalesced) access of 32 consecutive or rotated words, so neither operand nor
// product moves by shuffle and every multiply-add is one FMA.  (The shuffled
// form, one warp per bank, spent 429 FP64 instructions and two shuffles per
// entry on a 96 x 96 bank against 288 FMAs here, in one dependent chain: 42 us
// for a handful of FP64 banks.)
//
// ROTS rotations starting at e0; BF: off-diagonal tiles in BF16 words.
template <int BD, int ROTS, bool BF, typename T, typename Ld>
__device__ __forceinline__ void bank_rows(const Ld &ld, const T *__restrict__ xs, int e0, int lane, T (&y)[BD])
{
#pragma unroll
    for (int c = 0; c < BD; ++c) y[c] = T(0);
#pragma unroll 4
    for (int q = 0; q < ROTS; ++q) {
        const int e = e0 + q, idx = (lane + e) & 31, t = (32 - e) & 31;
#pragma unroll
        for (int c = 0; c < BD; ++c) {
            const T x = xs[c * 32 + idx];
#pragma unroll
            for (int c1 = 0; c1 < BD; ++c1) {
                // element offset of tile (lo, hi), row-major over c <= c2
                const int lo = c1 < c ? c1 : c, hi = c1 < c ? c : c1;
                const int ndiag = hi == lo ? lo : lo + 1;  // diagonal tiles before this one
                const int noff = lo * (BD - 1) - lo * (lo - 1) / 2 + (hi > lo ? hi - lo - 1 : 0);
                const int off = hi == lo ? (e <= 16 ? e * 32 + lane : t * 32 + idx)
                                         : (c1 < c ? e * 32 + lane : t * 32 + idx);
                y[c1] += ld(ndiag, noff, hi == lo, off) * x;
            }
        }
    }
}

// entry loaders: tile (ndiag diagonal and noff off-diagonal tiles before it)
template <typename T, bool BF>
struct TileLd {
    const unsigned char *base;
    __device__ __forceinline__ T operator()(int ndiag, int noff, bool diag, int off) const
    {
        if (BF) {
            const unsigned char *t = base + ndiag * (17 * 32 * 4) + noff * 2048;
            if (diag) return (T) reinterpret_cast<const float *>(t)[off];
            // word (d / 2) * 32 + r holds entries d (low half) and d + 1 (high half)
            const int d = off >> 5, r = off & 31;
            const unsigned h = reinterpret_cast<const unsigned short *>(t)[(d >> 1) * 64 + 2 * r + (d & 1)];
            return (T)__uint_as_float(h << 16);
        }
        return (reinterpret_cast<const T *>(base) + ndiag * (17 * 32) + noff * 1024)[off];
    }
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------ setup

// Galerkin blocks of every coarse level, deterministically, in three passes.
// Pass 1: one warp per chunk of at most MEMB_CHUNK = 32 member rows of a coarse
// item ci (its row strip of the bank matrix).  The lanes first look up, for all
// rows of the chunk together, the bank slot of every block's column item; then
// 32 / BD^2 groups of BD^2 lanes (one per block entry) add the blocks of a row
// into the group's own strip in shared memory, and the strips are added in
// group order.  Pass 2 adds up to SEG_CHUNKS consecutive chunks of an item,
// pass 3 an item's segments and writes the upper triangle (each entry belongs
// to exactly one item, so the stores never collide).  Every sum runs in one
// fixed order (no atomics): two factorizations of the same matrix give
// bit-identical coarse inverses.
//
// An FP64 add costs the pipe a whole warp however few lanes need it: matching
// lanes by column item and adding them group by group ran 9 adds per block of
// a row (27 ms on four levels of 1M rows); entry-parallel groups run one per
// three blocks.
template <int BD>
__global__ void __launch_bounds__(128) assemble_coarse_chunk_kernel(BsrDev A, MasDev m, CoarseMembers mb,
                                                                    double *__restrict__ partial)
{
    constexpr int NE = BD * BD, G = 32 / NE, W = 4;
    __shared__ double acc_all[W][G * 32 * NE];
    __shared__ uint8_t slot_all[W][32][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int64_t c = (int64_t)blockIdx.x * W + wl;
    if (c >= mb.nchunk) return;
    double *acc = acc_all[wl];
    uint8_t(*slot)[32] = slot_all[wl];
    int64_t ci = mb.chunk_item[c];
    int l = 1;
    while (l < m.L && ci >= m.nitems[l]) ci -= m.nitems[l++];
    const int32_t *map = m.cmap + (int64_t)(l - 1) * A.nb;
    const int32_t bank = (int32_t)(ci >> 5), r0 = mb.chunk_r0[c], nr = mb.chunk_r0[c + 1] - r0;
    const int32_t row = lane < nr ? mb.rows[r0 + lane] : 0;
    const int32_t rb = lane < nr ? A.rows[row] : 0, rlen = lane < nr ? A.rows[row + 1] - rb : 0;
    for (int k = lane; k < G * 32 * NE; k += 32) acc[k] = 0.0;
    auto lookup = [&](int32_t at) -> uint8_t {  // bank slot of block `at`'s column item, 255 outside the bank
        const int32_t cj = map[A.cols[at]];
        return (cj >> 5) == bank ? (uint8_t)(cj & 31) : (uint8_t)255;
    };
#pragma unroll 8
    for (int j = 0; j < nr; ++j) {
        const int32_t b = __shfl_sync(0xffffffffu, rb, j), len = __shfl_sync(0xffffffffu, rlen, j);
        if (lane < len) slot[j][lane] = lookup(b + lane);
    }
    __syncwarp();
    const int grp = lane / NE, k = lane - grp * NE;
    double *mine = acc + (grp * 32) * NE + k;
    for (int j = 0; j < nr; ++j) {
        const int32_t b = __shfl_sync(0xffffffffu, rb, j), len = __shfl_sync(0xffffffffu, rlen, j);
        if (grp >= G) continue;
        const double *v = A.vals + (int64_t)b * NE + (int64_t)k * len;
        int q = grp;
        for (; q < len && q < 32; q += 4 * G) {  // four values in flight
            double x[4];
            uint8_t s[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int at = q + t * G;
                s[t] = at < len && at < 32 ? slot[j][at] : (uint8_t)255;
                x[t] = s[t] != 255 ? v[at] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (s[t] != 255) mine[s[t] * NE] += x[t];
        }
        for (q = grp + (32 - grp + G - 1) / G * G; q < len; q += G) {  // rows of more than 32 blocks
            const uint8_t s = lookup(b + q);
            if (s != 255) mine[s * NE] += v[q];
        }
    }
    __syncwarp();
    // strip entry (slot, k) at [k][slot]
    double *out = partial + c * (NE * 32);
    for (int e = lane; e < NE * 32; e += 32) {
        double sum = 0.0;
#pragma unroll
        for (int g = 0; g < G; ++g) sum += acc[g * 32 * NE + e];
        out[(e % NE) * 32 + e / NE] = sum;
    }
}

// Adds partial strips [ptr[w], ptr[w + 1]) in order; eight strips in flight.
template <int BD>
__device__ __forceinline__ void sum_strips(const double *__restrict__ partial, int32_t c0, int32_t c1, int lane,
                                           double (&acc)[BD * BD])
{
#pragma unroll
    for (int k = 0; k < BD * BD; ++k) acc[k] = 0.0;
#pragma unroll 4
    for (int32_t c = c0; c < c1; ++c) {
        const double *p = partial + (int64_t)c * (BD * BD * 32);
#pragma unroll
        for (int k = 0; k < BD * BD; ++k) acc[k] += p[k * 32 + lane];
    }
}

template <int BD>
__global__ void __launch_bounds__(256) assemble_coarse_seg_kernel(CoarseMembers mb, const double *__restrict__ partial,
                                                                  double *__restrict__ seg)
{
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= mb.nseg) return;
    double acc[BD * BD];
    sum_strips<BD>(partial, mb.seg_c0[w], mb.seg_c0[w + 1], lane, acc);
#pragma unroll
    for (int k = 0; k < BD * BD; ++k) seg[w * (BD * BD * 32) + k * 32 + lane] = acc[k];
}

template <int BD>
__global__ void __launch_bounds__(256) assemble_coarse_sum_kernel(MasDev m, CoarseMembers mb,
                                                                  const double *__restrict__ seg,
                                                                  double *__restrict__ stage)
{
    constexpr int N = 32 * BD;
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= mb.nitem) return;
    int64_t ci = w;
    int l = 1;
    while (l < m.L && ci >= m.nitems[l]) ci -= m.nitems[l++];
    const int64_t g = m.boff[l] + (ci >> 5);
    double acc[BD * BD];
    sum_strips<BD>(seg, mb.item_seg[w], mb.item_seg[w + 1], lane, acc);
    double *base = stage + g * N * N;
#pragma unroll
    for (int bi = 0; bi < BD; ++bi)
#pragma unroll
        for (int bj = 0; bj < BD; ++bj) {
            const int row = bi * 32 + (int)(ci & 31), col = bj * 32 + lane;
            if (row <= col) base[(int64_t)row * N + col] = acc[bi * BD + bj];
        }
}

// place of entry (t, c), t <= c, in the packed upper triangle
template <int N>
__device__ __forceinline__ int tri(int t, int c) { return t * N - t * (t - 1) / 2 + c - t; }

// Symmetric sweep inversion of S (the upper triangle of an N x N matrix, packed
// by rows, in shared memory): the Gauss-Jordan variant of
// MASPreconditioner.cu:799-900, which leaves -A^-1 in S.  The sweep preserves
// symmetry, so half the FP64 updates suffice.  The triangle's entries are dealt
// to the CTA's threads in packed order: every update instruction runs on full
// warps (a partly predicated FP64 instruction costs the pipe a whole warp) and
// every access to S is consecutive, and 37 KB for a 96 x 96 bank leave room for
// four CTAs per SM to cover each other's barriers (square storage: two).
// Flags zero / non-finite pivots.  Needs blockDim.x == 256.
template <int N>
__device__ void sweep_invert(double *S, double *col, double *scol, int *bad)
{
    constexpr int NE = N * (N + 1) / 2;
    constexpr int PER = (NE + 255) / 256;
    const int tid = threadIdx.x;
    uint32_t tc[PER];  // (t << 16) | c of this thread's entries; ~0u past the end
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int e = tid + k * 256;
        tc[k] = ~0u;
        if (e < NE) {
            int t = 0, off = 0;
            while (off + (N - t) <= e) {
                off += N - t;
                ++t;
            }
            tc[k] = ((uint32_t)t << 16) | (uint32_t)(t + (e - off));
        }
    }
    // the division of a pivot is left to one warp, while the others write the
    // previous pivot's column back: run by all eight it cost the pipe as much as
    // two thirds of the updates
    __shared__ double rp;
    auto reciprocal = [&](int p) {
        const double piv = S[tri<N>(p, p)];
        if (!isfinite(piv) || piv == 0.0) atomicOr(bad, 1);
        rp = 1.0 / piv;
    };
    if (tid == 255) reciprocal(0);
    __syncthreads();
    for (int p = 0; p < N; ++p) {
        const double rpiv = rp;  // the column is scaled by multiplication
        for (int t = tid; t < N; t += 256) {
            const double cv = (t == p) ? 0.0 : S[t < p ? tri<N>(t, p) : tri<N>(p, t)];
            col[t] = cv;
            scol[t] = cv * rpiv;
        }
        __syncthreads();
        // the pivot's own row and column (zeros in col and scol) keep their
        // values here and are replaced below
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (tc[k] == ~0u) continue;
            S[tid + k * 256] -= scol[tc[k] >> 16] * col[tc[k] & 0xffffu];
        }
        __syncthreads();
        for (int t = tid; t < N; t += 256) {
            if (t == p) S[tri<N>(p, p)] = -rpiv;
            else S[t < p ? tri<N>(t, p) : tri<N>(p, t)] = scol[t];
        }
        if (tid == 255 && p + 1 < N) reciprocal(p + 1);
        __syncthreads();
    }
}

// One CTA per bank, the level-0 banks (CTAs [0, nparts)) first and the coarse
// ones after them in the same launch: a few banks are one sweep's latency (215
// us of dependent pivots), which a launch per level paid twice.  A level-0 bank
// is gathered straight from the operator's rows; a coarse bank from its dense
// Galerkin staging (upper triangle).
template <int BD, typename T, bool BF0>
__global__ void __launch_bounds__(256, 4) mas_invert_kernel(BsrDev A, const int32_t *__restrict__ part_off,
                                                            int64_t nparts, void *__restrict__ out0,
                                                            const double *__restrict__ stagec, T *__restrict__ outc,
                                                            int *bad, uint8_t *__restrict__ uncoupled)
{
    constexpr int N = 32 * BD, NE = N * (N + 1) / 2;
    extern __shared__ double sm[];
    double *S = sm, *col = sm + NE, *scol = col + N;
    const bool fine = (int64_t)blockIdx.x < nparts;
    const int64_t bank = fine ? blockIdx.x : (int64_t)blockIdx.x - nparts;
    if (fine) {
        for (int idx = threadIdx.x; idx < NE; idx += blockDim.x) S[idx] = 0.0;
        __syncthreads();
        const int32_t lo = part_off[bank], hi = part_off[bank + 1];
        const int g = threadIdx.x & 7;  // eight threads per block row
        for (int32_t i = lo + (int32_t)(threadIdx.x >> 3); i < hi; i += (int32_t)(blockDim.x >> 3)) {
            const int32_t b = A.rows[i], len = A.rows[i + 1] - b;
            const double *v = A.vals + (int64_t)b * BD * BD;
            for (int32_t l = g; l < len; l += 8) {
                const int32_t j = A.cols[b + l];
                if (j < lo || j >= hi) continue;
#pragma unroll
                for (int bi = 0; bi < BD; ++bi)
#pragma unroll
                    for (int bj = 0; bj < BD; ++bj) {
                        const int r = bi * 32 + (i - lo), c = bj * 32 + (j - lo);
                        if (r <= c) S[tri<N>(r, c)] = v[(int64_t)(bi * BD + bj) * len + l];
                    }
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < N; t += blockDim.x)
            if (S[tri<N>(t, t)] == 0.0) S[tri<N>(t, t)] = 1.0;  // padding (MASPreconditioner.cu:779-796)
    } else {
        const double *src = stagec + bank * N * N;
        bool coupled = false;  // an entry between two different items of the bank
        for (int idx = threadIdx.x; idx < N * N; idx += blockDim.x) {
            const int r = idx / N, c = idx % N;
            if (r > c) continue;  // the upper triangle is all the sweep uses
            double v = src[(int64_t)r * N + c];
            coupled |= ((r ^ c) & 31) != 0 && v != 0.0;
            if (r == c && v == 0.0) v = 1.0;
            S[tri<N>(r, c)] = v;
        }
        coupled = __syncthreads_or(coupled);
        if (threadIdx.x == 0) uncoupled[bank] = coupled ? 0 : 1;
    }
    __syncthreads();
    sweep_invert<N>(S, col, scol, bad);
    // the swept entry (i, j), i <= j
    auto entry = [&](int i, int j) -> double { return S[tri<N>(i, j)]; };
    // tiles
    if (BF0 && fine) {  // FP32 diagonal tiles, BF16 off-diagonal tiles (round to nearest even)
        unsigned char *dst = reinterpret_cast<unsigned char *>(out0) + bank * (int64_t)(BD * 17 * 32 * 4 + BD * (BD - 1) / 2 * 2048);
        for (int c = 0; c < BD; ++c)
            for (int c2 = c; c2 < BD; ++c2) {
                const int nd = (c == c2) ? 17 : 32;
                for (int e = threadIdx.x; e < nd * 32; e += blockDim.x) {
                    const int d = e >> 5, r = e & 31;
                    const int gi = c * 32 + r, gj = c2 * 32 + ((r + d) & 31);
                    const double val = -entry(min(gi, gj), max(gi, gj));
                    if (!isfinite(val)) atomicOr(bad, 2);
                    if (c == c2) reinterpret_cast<float *>(dst)[e] = (float)val;
                    else reinterpret_cast<__nv_bfloat16 *>(dst)[(d >> 1) * 64 + 2 * r + (d & 1)] =
                        __float2bfloat16_rn((float)val);
                }
                dst += (c == c2) ? 17 * 32 * 4 : 32 * 32 * 2;
            }
        return;
    }
    T *dst = (fine ? reinterpret_cast<T *>(out0) : outc) + bank * tile_elems<BD>();
    int64_t off = 0;
    for (int c = 0; c < BD; ++c)
        for (int c2 = c; c2 < BD; ++c2) {
            const int nd = (c == c2) ? 17 : 32;
            for (int e = threadIdx.x; e < nd * 32; e += blockDim.x) {
                const int d = e >> 5, r = e & 31;
                const int gi = c * 32 + r, gj = c2 * 32 + ((r + d) & 31);
                const double val = -entry(min(gi, gj), max(gi, gj));
                if (!isfinite(val)) atomicOr(bad, 2);
                dst[off + e] = (T)val;
            }
            off += nd * 32;
        }
}

// ------------------------------------------------------------------ apply

// The restriction of r to level 1: a warp sums one partition's rows into its
// level-1 items (the PCG's update does the same for the residual it leaves,
// update_xr_kernel).  In a large hierarchy a second launch sums the level-1 banks
// into level 2 (MasDev::base); the levels above are summed from the base level
// by the products that need them (symv_coarse_kernel).  Restricting completed
// banks further inside this launch, found by arrival counters, saved launches
// but paid a fence and an atomic per bank: 14 to 22 us with all levels, 41 us
// with one on 33k partitions.
template <int BD, typename T, typename XT>
__global__ void __launch_bounds__(256) restrict_kernel(MasDev m, const XT *__restrict__ r, T *__restrict__ v,
                                                       const int *done)
{
    constexpr int N = 32 * BD, W = 8;
    __shared__ T xs_all[W][N];
    __shared__ unsigned mask_all[W][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    T *xs = xs_all[wl];
    // a partition's bounds and items do not depend on the preceding kernel
    int64_t p = (int64_t)blockIdx.x * W + wl;
    const int64_t step = (int64_t)gridDim.x * W;
    MasPart t = mas_part(m, p, lane);
    pdl_enter();
    if (done && *done) return;
    for (; p < m.nparts; p += step) {
        // the part's values are one contiguous run: coalesced loads
#pragma unroll
        for (int q = 0; q < BD; ++q) {
            const int e = q * 32 + lane;
            xs[e] = e < t.cnt * BD ? (T)r[(int64_t)t.lo * BD + e] : T(0);
        }
        const MasPart next = mas_part(m, p + step, lane);
        __syncwarp();
        bank_segment_sums<BD, T>(xs, t.key, mask_all[wl], t.nc, v + m.voff[1] + (int64_t)t.i0 * BD, lane);
        __syncwarp();
        t = next;
    }
}

// level 1 -> level 2, a warp per level-1 bank
template <int BD, typename T>
__global__ void __launch_bounds__(256) restrict1_kernel(MasDev m, T *__restrict__ v, PcgState *st, PcgSum rr)
{
    constexpr int N = 32 * BD, W = 8;
    __shared__ T xs_all[W][N];
    __shared__ unsigned mask_all[W][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int32_t b = blockIdx.x * W + wl;
    const bool valid = b < m.nbanks[1];
    const int32_t i0 = b * 32;
    const int cnt = valid ? min(32, m.nitems[1] - i0) : 0, nc = valid ? m.ccnt[1][b] : 0;
    const int32_t j0 = valid ? m.cbase[1][b] : 0;
    const uint8_t key = lane < cnt ? m.key[1][i0 + lane] : (uint8_t)0xff;
    pdl_enter();
    if (pcg_stops(st, rr) || !valid) return;
    const T *vl = v + m.voff[1] + (int64_t)i0 * BD;
    T *xs = xs_all[wl];
#pragma unroll
    for (int q = 0; q < BD; ++q) {
        const int e = q * 32 + lane;
        xs[e] = e < cnt * BD ? vl[e] : T(0);
    }
    __syncwarp();
    bank_segment_sums<BD, T>(xs, key, mask_all[wl], nc, v + m.voff[2] + (int64_t)j0 * BD, lane);
}

// x of a coarse bank above the base level: every item's sum over the base-level
// items below it (memb: base items grouped by their item at this level, in
// order).  Items of up to 128 members take a warp, larger ones the whole CTA.
template <int BD, typename T>
__device__ __forceinline__ void gather_bank(const MasDev &m, int l, int32_t b, const T *__restrict__ v,
                                            T *__restrict__ xs, T (*red)[32 * BD])
{
    constexpr int W = 8, BIG = 128;
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int32_t *__restrict__ ptr = m.memb_ptr[l] + (int64_t)b * 32;
    const int32_t *__restrict__ memb = m.memb[l];
    const T *__restrict__ vb = v + m.voff[m.base];
    const int cnt = min(32, m.nitems[l] - b * 32);
    const int32_t lo = lane < cnt ? ptr[lane] : 0, hi = lane < cnt ? ptr[lane + 1] : 0;
    const unsigned big = __ballot_sync(0xffffffffu, hi - lo > BIG);
    for (int it = wl; it < 32; it += W) {
        if (big >> it & 1u) continue;
        const int32_t p0 = __shfl_sync(0xffffffffu, lo, it), p1 = __shfl_sync(0xffffffffu, hi, it);
        T acc[BD];
#pragma unroll
        for (int c = 0; c < BD; ++c) acc[c] = T(0);
#pragma unroll 4
        for (int32_t j = p0 + lane; j < p1; j += 32) {
            const T *e = vb + (int64_t)memb[j] * BD;
#pragma unroll
            for (int c = 0; c < BD; ++c) acc[c] += e[c];
        }
        if (p1 - p0 > 1)
#pragma unroll
            for (int c = 0; c < BD; ++c) acc[c] = warp_sum(acc[c]);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < BD; ++c) xs[c * 32 + it] = acc[c];
    }
    for (unsigned left = big; left; left &= left - 1) {
        const int it = __ffs(left) - 1;
        const int32_t p0 = __shfl_sync(0xffffffffu, lo, it), p1 = __shfl_sync(0xffffffffu, hi, it);
        T acc[BD];
#pragma unroll
        for (int c = 0; c < BD; ++c) acc[c] = T(0);
#pragma unroll 4
        for (int32_t j = p0 + tid; j < p1; j += 32 * W) {
            const T *e = vb + (int64_t)memb[j] * BD;
#pragma unroll
            for (int c = 0; c < BD; ++c) acc[c] += e[c];
        }
#pragma unroll
        for (int c = 0; c < BD; ++c) acc[c] = warp_sum(acc[c]);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < BD; ++c) red[wl][c * 32] = acc[c];
        __syncthreads();
        if (tid < BD) {
            T sum = red[0][tid * 32];
#pragma unroll
            for (int w = 1; w < W; ++w) sum += red[w][tid * 32];
            xs[tid * 32 + it] = sum;
        }
        __syncthreads();
    }
}

// u_g = Inv_g v_g for every coarse bank, one CTA of eight warps per bank: each
// warp takes four rotations, whose loads are all in flight together (the
// banks are few and L2-resident, so this is one latency, not a stream).  In a
// bank without couplings between its items (uncoupled: Dirichlet rows, which
// never merge and fill a third of the coarse banks of a clamped cube) every
// entry off rotation 0 is an exact zero, and only that rotation is taken.  Banks
// above the base level first sum their items.  Level vectors are whole banks back to back: bank g starts at element g * N.
template <int BD, typename T>
__global__ void __launch_bounds__(256) symv_coarse_kernel(MasDev m, const T *__restrict__ invc,
                                                          const T *__restrict__ v, T *__restrict__ u,
                                                          PcgState *st, PcgSum rr)
{
    constexpr int N = 32 * BD, W = 8;
    __shared__ T xs[N];
    __shared__ T red[W][N];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int64_t g = blockIdx.x;
    const int o = (tid % BD) * 32 + tid / BD;  // component-major place of element tid
    const bool uncoupled = m.uncoupled[g];
    pdl_enter();
    if (pcg_stops(st, rr)) return;
    int l = 1;
    while (l + 1 < m.L && g >= m.boff[l + 1]) ++l;
    if (l <= m.base) {
        if (tid < N) xs[o] = v[g * N + tid];
    } else {
        gather_bank<BD, T>(m, l, (int32_t)(g - m.boff[l]), v, xs, red);
    }
    __syncthreads();
    T y[BD];
    const TileLd<T, false> ld{reinterpret_cast<const unsigned char *>(invc + g * m.tile_elems)};
    if (uncoupled) {
        if (wl > 0) return;
        bank_rows<BD, 1, false, T>(ld, xs, 0, lane, y);
#pragma unroll
        for (int c = 0; c < BD; ++c) u[g * N + lane * BD + c] = y[c];
        return;
    }
    bank_rows<BD, 32 / W, false, T>(ld, xs, wl * (32 / W), lane, y);
#pragma unroll
    for (int c = 0; c < BD; ++c) red[wl][c * 32 + lane] = y[c];
    __syncthreads();
    if (tid < N) {
        T sum = red[0][o];
#pragma unroll
        for (int w = 1; w < W; ++w) sum += red[w][o];
        u[g * N + tid] = sum;
    }
}

// level 0: z = Inv_0 x (+ the coarse corrections), optional accumulate and r.z;
// x in FP64, or in FP32 (XT = float) when it comes from the FP32 residual.
//
// A CTA of four warps works on GB consecutive banks at a time (one 96-row,
// two 64-row or four 32-row banks: the banks of one group are one contiguous
// run of HBM).  The next groups' inverses stream into shared-memory stages by
// 16-byte asynchronous copies while this group's product runs from its stage,
// and the vector operands are loaded a group ahead; WB warps share a bank, each taking 32 / WB rotations, and their
// partial sums meet in shared memory in warp order.  A node adds its
// ancestors' coarse corrections here (cmap: its item at every level), so no
// separate prolongation runs.
template <int BD, bool BF>
constexpr int bank_bytes(size_t elem)
{
    return BF ? BD * 17 * 32 * 4 + BD * (BD - 1) / 2 * 2048 : (int)(tile_elems<BD>() * elem);
}
template <int BD>
struct BankGroup {
    static constexpr int WB = BD == 3 ? 4 : BD, GB = 4 / WB;
};
// Stages of shared memory per CTA: two of up to 20 KB, a group's product beside
// the next one's copy, in five CTAs per SM.  More stages leave fewer CTAs (FP32
// level 0 of 3.0M / 648k DOFs with two, three, four stages: 100.5 / 24.7, 113 /
// 28.2, 143 / 34.6 us).  The larger FP64 stages are bound by the FP64 pipe, where
// five one-stage CTAs cover each other's loads.
template <int BD, typename T, bool BF>
constexpr int bank_stages()
{
    return (BF ? 4 : (int)sizeof(T)) * tile_elems<BD>() * BankGroup<BD>::GB <= 20480 ? 2 : 1;
}

template <int BD, typename T, bool ACC, bool DOT, typename XT, bool BF = false>
__global__ void __launch_bounds__(128) symv0_kernel(MasDev m, const T *__restrict__ inv0, const T *__restrict__ u,
                                                    const XT *__restrict__ xin, double *__restrict__ z,
                                                    double scale, const double *__restrict__ rdot, PcgSum rz,
                                                    GridReduce gr, const int *done, float *__restrict__ z32,
                                                    float *__restrict__ z_lo)
{
    constexpr int N = 32 * BD, WB = BankGroup<BD>::WB, GB = BankGroup<BD>::GB;
    constexpr int BANK_B = bank_bytes<BD, BF>(sizeof(T)), STAGE_B = BANK_B * GB, NST = bank_stages<BD, T, BF>();
    extern __shared__ __align__(16) unsigned char stage[];
    __shared__ T xs[GB][N];
    __shared__ T red[4][N];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int64_t ngroups = (m.nparts + GB - 1) / GB;
    const unsigned char *src = reinterpret_cast<const unsigned char *>(inv0);
    auto fill = [&](int st_, int64_t g) {
        const int64_t b0 = g * GB, left = m.nparts - b0;
        const int bytes = left < GB ? (int)left * BANK_B : STAGE_B;
        for (int k = tid * 16; k < bytes; k += 128 * 16) cp_async16(stage + st_ * STAGE_B + k, src + b0 * BANK_B + k);
    };
    // thread t owns vector element t % N of bank t / N of the group
    const int bk = tid / N, el = tid % N, node = el / BD, comp = el % BD;
    // The chain partition -> node -> items -> corrections is loaded over three
    // groups (partition bounds two groups ahead, a node's operands and items one
    // group ahead), so that no step waits for the one before it.
    struct Bounds {
        int32_t lo, hi;
    };
    auto bounds = [&](int64_t g) {
        Bounds b{0, 0};
        const int64_t p = g * GB + bk;
        if (bk < GB && g < ngroups && p < m.nparts) b = {m.part_off[p], m.part_off[p + 1]};
        return b;
    };
    struct Operand {
        XT x;
        double z, rd;
        int32_t item[MAS_MAXL - 1];
        int64_t e;  // -1: no element
    };
    auto operand = [&](Bounds b) {
        Operand o;
        const int32_t i = b.lo + node;
        const bool ok = i < b.hi;
        o.e = ok ? (int64_t)i * BD + comp : -1;
        o.x = ok ? xin[o.e] : XT(0);
        o.z = ACC && ok ? z[o.e] : 0.0;
        o.rd = DOT && ok ? rdot[o.e] : 0.0;
#pragma unroll
        for (int l = 1; l < MAS_MAXL; ++l) o.item[l - 1] = ok && l < m.L ? m.cmap[(int64_t)(l - 1) * m.nb + i] : 0;
        return o;
    };
    double dot = 0.0;
    int64_t g = blockIdx.x;
    const int64_t step = gridDim.x;
    int cur = 0;
    // the inverses and maps do not change within a solve: their first loads need
    // not wait for the preceding kernel
    constexpr int AHEAD = NST > 1 ? NST - 1 : 1;
#pragma unroll
    for (int q = 0; q < AHEAD; ++q) {
        if (g + q * step < ngroups) fill(q, g + q * step);
        cp_async_commit();
    }
    const Bounds b0 = bounds(g);
    Bounds nb = bounds(g + step);
    pdl_enter();
    if (done && *done) {
        cp_async_wait<0>();
        return;
    }
    Operand o = operand(b0);
    for (; g < ngroups; g += step) {
        const int64_t gf = g + (NST - 1) * step;
        if (gf < ngroups && (NST > 1 || g != (int64_t)blockIdx.x))
            fill(cur + NST - 1 < NST ? cur + NST - 1 : cur - 1, gf);
        cp_async_commit();
        if (bk < GB) xs[bk][comp * 32 + node] = (T)o.x;
        T cu[MAS_MAXL - 1];
#pragma unroll
        for (int l = 1; l < MAS_MAXL; ++l)
            cu[l - 1] = o.e >= 0 && l < m.L ? u[m.voff[l] + (int64_t)o.item[l - 1] * BD + comp] : T(0);
        const Operand nx = operand(nb);
        nb = bounds(g + 2 * step);
        cp_async_wait<NST - 1>();
        __syncthreads();
        T y[BD];
        const TileLd<T, BF> ld{stage + cur * STAGE_B + (wl / WB) * BANK_B};
        bank_rows<BD, 32 / WB, BF, T>(ld, xs[wl / WB], (wl % WB) * (32 / WB), lane, y);
#pragma unroll
        for (int c = 0; c < BD; ++c) red[wl][c * 32 + lane] = y[c];
        __syncthreads();
        if (o.e >= 0) {
            T sum = red[bk * WB][comp * 32 + node];
#pragma unroll
            for (int w = 1; w < WB; ++w) sum += red[bk * WB + w][comp * 32 + node];
            T corr = cu[MAS_MAXL - 2];  // top level down, as level-by-level prolongation adds them
#pragma unroll
            for (int l = MAS_MAXL - 2; l >= 1; --l) corr = cu[l - 1] + corr;
            double val = ((double)sum + (double)corr) * scale;
            if (ACC) val += o.z;
            z[o.e] = val;
            if (z32) {
                const float h = (float)val;
                z32[o.e] = h;
                if (z_lo) z_lo[o.e] = (float)(val - (double)h);
            }
            if (DOT) dot += o.rd * val;
        }
        o = nx;
        cur = cur + 1 < NST ? cur + 1 : 0;
    }
    if (DOT) put_sum(dot, gr, rz);
}

// Grid of a level-0 launch: every resident CTA, at most one per bank group.
template <int BD, typename T, bool BF>
int symv0_grid(int64_t nparts)
{
    constexpr int GB = BankGroup<BD>::GB;
    constexpr int cta = bank_stages<BD, T, BF>() * bank_bytes<BD, BF>(sizeof(T)) * GB + (BD == 3 ? 4096 : 2048) + 5 * 32 * BD * (int)sizeof(T);
    constexpr int per_sm = 227 * 1024 / cta < 12 ? 227 * 1024 / cta : 12;
    return grid_for(nparts, GB, sm_grid(per_sm));
}

template <int BD, typename T, bool ACC, bool DOT, typename XT, bool BF>
void symv0_launch(const MasDev &m, const T *inv0, const T *u, const XT *xin, double *z, double scale,
                  const double *rdot, PcgSum *rz, GridReduce gr, const int *done, cudaStream_t s, float *z32,
                  float *z_lo)
{
    const size_t smem = (size_t)bank_stages<BD, T, BF>() * bank_bytes<BD, BF>(sizeof(T)) * BankGroup<BD>::GB;
    const int grid = symv0_grid<BD, T, BF>(m.nparts);
    if (rz) {
        rz->direct = (int64_t)m.nb * BD <= PCG_DIRECT_ROWS;
        rz->count = rz->direct ? grid : 1;
    }
    raise_smem_limit((const void *)symv0_kernel<BD, T, ACC, DOT, XT, BF>, smem);
    launch_pdl(symv0_kernel<BD, T, ACC, DOT, XT, BF>, grid, 128, smem, s, m, inv0, u, xin, z, scale, rdot,
               rz ? *rz : PcgSum{}, gr, done, z32, z_lo);
}

template <int BD, typename T, typename XT>
void mas_apply_dot_t(const MasDev &m, const T *inv0, const T *invc, T *v, T *u, const XT *xin, double *z,
                     bool acc, double scale, const double *rdot, PcgState *st, const PcgSum *rr, PcgSum *rz,
                     GridReduce gr, cudaStream_t s, float *z32, float *z_lo, bool restricted)
{
    if (m.L < 2) fail(LSS_ERR_INTERNAL, "a MAS hierarchy has at least one coarse level");
    const int *done = &st->done;
    // the first launch after the residual's update tests it for convergence
    PcgSum test = rr ? *rr : PcgSum{};
    if (!restricted)
        launch_pdl(restrict_kernel<BD, T, XT>, grid_for(m.nparts, 8, sm_grid(8)), 256, 0, s, m, xin, v, done);
    if (m.base > 1) {
        launch_pdl(restrict1_kernel<BD, T>, (unsigned)((m.nbanks[1] + 7) / 8), 256, 0, s, m, v, st, test);
        test = PcgSum{};
    }
    launch_pdl(symv_coarse_kernel<BD, T>, (unsigned)m.ncoarse, 256, 0, s, m, invc, (const T *)v, u, st, test);
#define LSS_S0(A_, D_)                                                                                          \
    do {                                                                                                        \
        if (std::is_same<T, float>::value && m.bank_bytes0 > 0)                                                 \
            symv0_launch<BD, T, A_, D_, XT, std::is_same<T, float>::value>(m, inv0, u, xin, z, scale, rdot, rz, \
                                                                           gr, done, s, z32, z_lo);             \
        else                                                                                                    \
            symv0_launch<BD, T, A_, D_, XT, false>(m, inv0, u, xin, z, scale, rdot, rz, gr, done, s, z32, z_lo); \
    } while (0)
    if (rz) {
        if (acc) LSS_S0(true, true);
        else LSS_S0(false, true);
    } else {
        if (acc) LSS_S0(true, false);
        else LSS_S0(false, false);
    }
#undef LSS_S0
    LSS_LAUNCH_CHECK();
}

}  // namespace

template <int BD>
static void assemble_coarse_t(const BsrDev &A, const MasDev &m, const CoarseMembers &mb, double *partial, double *stage,
                              cudaStream_t s)
{
    double *seg = partial + mb.nchunk * (BD * BD * 32);
    assemble_coarse_chunk_kernel<BD><<<(unsigned)((mb.nchunk + 3) / 4), 128, 0, s>>>(A, m, mb, partial);
    assemble_coarse_seg_kernel<BD><<<(unsigned)((mb.nseg + 7) / 8), 256, 0, s>>>(mb, partial, seg);
    assemble_coarse_sum_kernel<BD><<<(unsigned)((mb.nitem + 7) / 8), 256, 0, s>>>(m, mb, seg, stage);
    LSS_LAUNCH_CHECK();
}

void launch_mas_assemble_coarse(const BsrDev &A, const MasDev &m, const CoarseMembers &mb, double *partial,
                                double *stage, cudaStream_t s)
{
    if (mb.nitem == 0 || m.L < 2) return;
    if (A.bd == 1) assemble_coarse_t<1>(A, m, mb, partial, stage, s);
    else if (A.bd == 2) assemble_coarse_t<2>(A, m, mb, partial, stage, s);
    else assemble_coarse_t<3>(A, m, mb, partial, stage, s);
}

template <int BD, typename T, bool BF0 = false>
static void invert_t(const BsrDev &A, const MasDev &m, const double *stagec, void *out0, void *outc, int *bad,
                     uint8_t *uncoupled, cudaStream_t s)
{
    constexpr int N = 32 * BD;
    const size_t smem = (size_t)(N * (N + 1) / 2 + 2 * N) * sizeof(double);
    raise_smem_limit((const void *)mas_invert_kernel<BD, T, BF0>, smem);
    mas_invert_kernel<BD, T, BF0><<<(unsigned)((int64_t)m.nparts + m.ncoarse), 256, smem, s>>>(
        A, m.part_off, m.nparts, out0, stagec, (T *)outc, bad, uncoupled);
    LSS_LAUNCH_CHECK();
}

void launch_mas_invert(const BsrDev &A, const MasDev &m, const double *stagec, void *out0, void *outc, bool fp32,
                       bool bf16_offdiag, int *bad, uint8_t *uncoupled, cudaStream_t s)
{
    if ((int64_t)m.nparts + m.ncoarse == 0) return;
    if (bf16_offdiag && !fp32) fail(LSS_ERR_INTERNAL, "BF16 off-diagonal tiles need the FP32 MAS");
#define LSS_INV(...) invert_t<__VA_ARGS__>(A, m, stagec, out0, outc, bad, uncoupled, s)
    switch (A.bd) {
    case 1:
        if (fp32) LSS_INV(1, float);  // one tile: no off-diagonal tiles to store in BF16
        else LSS_INV(1, double);
        break;
    case 2:
        if (bf16_offdiag) LSS_INV(2, float, true);
        else if (fp32) LSS_INV(2, float);
        else LSS_INV(2, double);
        break;
    default:
        if (bf16_offdiag) LSS_INV(3, float, true);
        else if (fp32) LSS_INV(3, float);
        else LSS_INV(3, double);
        break;
    }
#undef LSS_INV
}

void launch_mas_level0(const MasDev &m, const void *inv0, const void *u, bool fp32, const double *xin, double *z,
                       cudaStream_t s)
{
    GridReduce gr{};
#define LSS_L0(BD_, T_)                                                                                          \
    symv0_launch<BD_, T_, false, false, double, false>(m, (const T_ *)inv0, (const T_ *)u, xin, z, 1.0, nullptr, nullptr, \
                                                   gr, nullptr, s, nullptr, nullptr)
#define LSS_L0BF(BD_)                                                                                            \
    symv0_launch<BD_, float, false, false, double, true>(m, (const float *)inv0, (const float *)u, xin, z, 1.0, nullptr, \
                                                     nullptr, gr, nullptr, s, nullptr, nullptr)
    if (fp32 && m.bank_bytes0 > 0) {
        if (m.bd == 2) LSS_L0BF(2);
        else LSS_L0BF(3);
    } else if (fp32) {
        if (m.bd == 1) LSS_L0(1, float);
        else if (m.bd == 2) LSS_L0(2, float);
        else LSS_L0(3, float);
    } else {
        if (m.bd == 1) LSS_L0(1, double);
        else if (m.bd == 2) LSS_L0(2, double);
        else LSS_L0(3, double);
    }
#undef LSS_L0
#undef LSS_L0BF
    LSS_LAUNCH_CHECK();
}

void launch_mas_apply(const MasDev &m, const void *inv0, const void *invc, void *v, void *u, bool fp32,
                      const double *xin, double *z, bool acc, double scale, const double *rdot, PcgState *st,
                      const PcgSum *rr, PcgSum *rz, GridReduce gr, cudaStream_t s, float *z32, const float *xin32,
                      float *z_lo, bool restricted)
{
#define LSS_MAS(BD_, T_)                                                                                          \
    mas_apply_dot_t<BD_, T_, double>(m, (const T_ *)inv0, (const T_ *)invc, (T_ *)v, (T_ *)u, xin, z, acc, scale, \
                                     rdot, st, rr, rz, gr, s, z32, z_lo, restricted)
#define LSS_MAS32(BD_)                                                                                            \
    mas_apply_dot_t<BD_, float, float>(m, (const float *)inv0, (const float *)invc, (float *)v, (float *)u, xin32, \
                                       z, acc, scale, rdot, st, rr, rz, gr, s, z32, z_lo, restricted)
    if (xin32) {
        if (!fp32) fail(LSS_ERR_INTERNAL, "an FP32 input needs the FP32 MAS");
        if (m.bd == 1) LSS_MAS32(1);
        else if (m.bd == 2) LSS_MAS32(2);
        else LSS_MAS32(3);
        return;
    }
    if (fp32) {
        if (m.bd == 1) LSS_MAS(1, float);
        else if (m.bd == 2) LSS_MAS(2, float);
        else LSS_MAS(3, float);
    } else {
        if (m.bd == 1) LSS_MAS(1, double);
        else if (m.bd == 2) LSS_MAS(2, double);
        else LSS_MAS(3, double);
    }
#undef LSS_MAS
#undef LSS_MAS32
}

}  // namespace lss
