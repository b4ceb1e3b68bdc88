// twopass_dev.cuh -- device helpers shared by the TWOPASS and TRIP kernels.
#pragma once

#include "ptx.cuh"
#include "twopass.cuh"

namespace fft3d {

// Every thread: drop from L2, without a write-back, the scratch lines whose
// rows row item j has read for the last time (twopass_row_line).  A barrier
// must follow before the slot is released to the next volume's plane items.
template <class TG>
__device__ __forceinline__ void twopass_discard_rows(const void *slot, int j, int tid, int nt)
{
    constexpr int NQ = TG::YG::N0 * twopass_row_lines_per_plane<TG>();
    for (int q = tid; q < NQ; q += nt) {
        uintptr_t line;
        if (twopass_row_line<TG>(slot, j, q, &line)) discard_l2_line(line);
    }
}

// Thread 0 of every CTA, as it leaves: the last one clears the control block for
// the next launch.
__device__ __forceinline__ void twopass_leave(TwoPassCtl *ctl, int tid)
{
    if (tid != 0) return;
    __threadfence();
    const unsigned prev = atomicAdd(&ctl->done, 1u);
    if (prev != gridDim.x - 1) return;
    __threadfence();  // every other CTA's updates of the block precede the reset
    ctl->ticket = 0ull;
    for (int i = 0; i < 2 * TWOPASS_RMAX; ++i) ctl->cnt[i] = 0u;
    ctl->abort = 0u;
    __threadfence();
    ctl->done = 0u;
}

// L2-policy loads and stores of one complex value.
template <typename T>
__device__ __forceinline__ cx<T> ld_hint(const cx<T> *p, uint64_t policy)
{
    if constexpr (sizeof(T) == 8) {
        const double2 v = ld_nc_hint(reinterpret_cast<const double2 *>(p), policy);
        return {v.x, v.y};
    } else {
        const float2 v = ld_nc_hint(reinterpret_cast<const float2 *>(p), policy);
        return {v.x, v.y};
    }
}

template <typename T>
__device__ __forceinline__ void st_hint(cx<T> *p, cx<T> v, uint64_t policy)
{
    if constexpr (sizeof(T) == 8) st_cg_hint(reinterpret_cast<double2 *>(p), make_double2(v.re, v.im), policy);
    else st_cg_hint(reinterpret_cast<float2 *>(p), make_float2(v.re, v.im), policy);
}

}  // namespace fft3d
