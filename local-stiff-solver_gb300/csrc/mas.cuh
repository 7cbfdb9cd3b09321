// Restriction of one partition to its level-1 items, shared by the MAS apply and
// the kernels that leave a residual already restricted (sm_103a).
#pragma once

#include "device_common.cuh"
#include "kernels.hpp"

namespace lss {

// Segmented sums of one bank: 32 items (values staged item-major in xs; lane j
// passes the target aggregate of item j, 0xff for none) into ncc aggregates.
// Output slot s = k * BD + c (aggregate k, component c) belongs to a group of P
// lanes, P the largest power of two with ncc * BD * P <= 32 (1 beyond): lane q
// of the group adds the items j = q, q + P, ... of aggregate k in order, found
// by its mask, and the group's sums meet by shuffles.  An FP64 add costs the
// pipe a whole warp however few lanes take part: one aggregate (a connected
// partition) takes 4 + 3 adds and 32 aggregates (uncoupled items) one add per
// pass, where testing every item against every slot took 32 per pass.
template <int BD, typename T>
__device__ __forceinline__ void bank_segment_sums(const T *xs, uint8_t key, unsigned *mask, int ncc,
                                                  T *__restrict__ out, int lane)
{
    const unsigned same = __match_any_sync(0xffffffffu, (unsigned)key);
    if (key < 32 && __ffs(same) - 1 == lane) mask[key] = same;
    __syncwarp();
    const int slots = ncc * BD;
    int lg = 0;
    while (lg < 5 && (slots << (lg + 1)) <= 32) ++lg;
    const int sub = lane & ((1 << lg) - 1);
    // every 2^lg-th item, starting at sub
    const unsigned every = (lg == 0 ? ~0u : lg == 1 ? 0x55555555u : lg == 2 ? 0x11111111u : lg == 3 ? 0x01010101u
                            : lg == 4 ? 0x00010001u : 1u) << sub;
    for (int s0 = 0; s0 < slots; s0 += 32 >> lg) {
        const int sl = s0 + (lane >> lg), k = sl / BD, c = sl - k * BD;
        T acc = T(0);
        for (unsigned m = sl < slots ? mask[k] & every : 0u; m; m &= m - 1) acc += xs[(__ffs(m) - 1) * BD + c];
        for (int o = (1 << lg) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (sl < slots && sub == 0) out[sl] = acc;
    }
}

// A partition as a warp sees it: its first row and rows, its first level-1 item
// and items, and the lane's row's item (0xff: no row).
struct MasPart {
    int32_t lo, cnt, i0;
    int nc;
    uint8_t key;
};
__device__ __forceinline__ MasPart mas_part(const MasDev &m, int64_t p, int lane)
{
    MasPart t{0, 0, 0, 0, 0xff};
    if (p < m.nparts) {
        t.lo = m.part_off[p];
        t.cnt = m.part_off[p + 1] - t.lo;
        t.i0 = m.cbase0[p];
        t.nc = m.ccnt0[p];
        if (lane < t.cnt) t.key = m.key0[t.lo + lane];
    }
    return t;
}

// Whether the iterations are over (threads that return true leave the kernel).
// With rr, also the updated residual's convergence tests (GPUHybrid.cu:1488-1496):
// every CTA of the first kernel after the update runs them -- every thread of it
// must call -- and the first CTA records them.  It may set done while another
// reads it: no thread leaves ahead of the sum's barriers, and all that stay come
// to the same verdict.
__device__ __forceinline__ bool pcg_stops(PcgState *st, PcgSum rr)
{
    const bool over = st->done != 0;
    if (!rr.part) return over;
    const int stop = from_sum(rr, [&](double s) {
        int c = STOP_RUNNING;
        if (!(s == s) || isinf(s)) c = STOP_NONFINITE;
        else if (st->rel_eps > 0 && s / st->bb < st->rel_eps) c = STOP_CONVERGED_REL;
        else if (st->abs_eps > 0 && s < st->abs_eps) c = STOP_CONVERGED_ABS;
        else if (st->iter >= st->max_iter) c = STOP_MAX_ITER;
        if (blockIdx.x == 0 && !over) {
            st->rr = s;
            if (c) st->done = c;
        }
        return c;
    });
    return over || stop != STOP_RUNNING;
}

}  // namespace lss
