// Launches of the resident time loops for one half order.
#pragma once

#include "resident.h"

namespace pyfwi {

constexpr size_t RES_MAX_FLOATS = (232448 - 1024) / sizeof(float);  // 227 KB per CTA less the static words

// The limit that is set is the same for every launch: it belongs to the kernel, and plans
// of other sizes may be launching the same one on other threads.
template <class Args>
static cudaError_t launch_resident(const void *kern, const Args &a, size_t floats, cudaStream_t s)
{
    const size_t smem = floats * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_MAX_FLOATS * sizeof(float));
    if (e != cudaSuccess) return e;
    void *args[] = {const_cast<Args *>(&a)};
    return cudaLaunchCooperativeKernel(kern, dim3(a.tl.gz * a.tl.gx * a.tl.nslots), dim3(RES_THREADS), args, smem, s);
}

// Groups of 4 cells with receivers in a tile and its ring, at most.
inline int res_slots(int R, const Lines &L, int th, int nq)
{
    int n = 0;
    for (int l = 0; l < L.n; ++l) n += L.drow[l] ? th + 2 * R : nq + 2;
    return n;
}

// Shared memory of the adjoint loop without its staged residuals, in floats.
template <int R>
constexpr size_t adj_res_floats(int rb)
{
    return rb == 1 ? ADJ_RES_FLOATS<R, 1> : rb == 2 ? ADJ_RES_FLOATS<R, 2> : ADJ_RES_FLOATS<R, 3>;
}

// And of the exact adjoint, whose blocks have one or two rows (three would
// spill: 32 floats a cell are live).
constexpr int RES_EXACT_ROWS = 2;
template <int R>
constexpr size_t exact_res_floats(int rb)
{
    return rb == 1 ? EXA_RES_FLOATS<R, 1> : EXA_RES_FLOATS<R, 2>;
}

template <int R>
cudaError_t launch_exact_resident_r(AdjResArgs &a, cudaStream_t s)
{
    a.slots = res_slots(R, a.a.lines, a.tl.rb * a.tl.bz, a.tl.nq);
    const size_t f = exact_res_floats<R>(a.tl.rb) + RES_SLOT_FLOATS * (size_t)a.slots;
    const void *kern = a.tl.rb == 1 ? reinterpret_cast<const void *>(exact_resident<R, 1>)
                                    : reinterpret_cast<const void *>(exact_resident<R, 2>);
    return launch_resident(kern, a, f, s);
}

template <int R>
cudaError_t launch_rev_resident_r(RevResArgs &a, cudaStream_t s)
{
#define CASE(RB_) \
    if (a.tl.rb == RB_) return launch_resident(reinterpret_cast<const void *>(rev_resident<R, RB_>), a, REV_RES_FLOATS<R, RB_>, s);
    CASE(1) CASE(2) CASE(3)
#undef CASE
    return cudaErrorInvalidValue;
}

template <int R>
cudaError_t launch_fwd_resident_r(FwdResArgs &a, cudaStream_t s)
{
#define CASE(RB_, Q_) \
    if (a.tl.rb == RB_ && a.store == Q_)                                                                                      \
        return launch_resident(reinterpret_cast<const void *>(fwd_resident<R, RB_, Q_>), a, FWD_RES_FLOATS<R, RB_>, s);
    CASE(1, 0) CASE(1, 1) CASE(1, 2) CASE(1, 3) CASE(2, 0) CASE(2, 1) CASE(2, 2) CASE(2, 3) CASE(3, 0) CASE(3, 1) CASE(3, 2)
    CASE(3, 3)
#undef CASE
    return cudaErrorInvalidValue;
}

template <int R>
cudaError_t launch_adj_resident_r(AdjResArgs &a, cudaStream_t s)
{
    const int th = a.tl.rb * a.tl.bz;
    a.slots = res_slots(R, a.a.lines, th, a.tl.nq);
    const size_t f = adj_res_floats<R>(a.tl.rb) + RES_SLOT_FLOATS * (size_t)a.slots;
#define CASE(RB_) \
    if (a.tl.rb == RB_) return launch_resident(reinterpret_cast<const void *>(adj_resident<R, RB_>), a, f, s);
    CASE(1) CASE(2) CASE(3)
#undef CASE
    return cudaErrorInvalidValue;
}

}  // namespace pyfwi
