// Message areas in global memory: which CTA works on which.
//
// Decoders whose check messages do not go to shared memory keep them in a
// scratch of the context, one area per CTA that the device can hold at a time
// (CTAs per SM x SMs).  Launches of one context may overlap -- the host-buffer
// pipeline decodes alternate chunks on two streams, a program may use streams
// of its own or replay a captured launch -- so an area cannot belong to a block
// index: the first CTAs of one launch run beside the last ones of another.  A
// CTA takes a free area when it starts and gives it back when it is done.
//
// There are as many areas as CTAs that can be resident, and a CTA holds one only
// while it runs, so a free one always exists; CTA b tries area b first, which
// alone costs one atomic operation at its start (no case of 1 to 12 ms changed by
// more than 0.5 %).  The search is bounded all the same: a CTA that finds none
// sets the context's status word and decodes nothing.
//
// A thread reads only message words that it wrote itself since its CTA took the
// area, so the fences below order one holder's writes before the next one's and
// no more is needed.
#pragma once
#include "tables.h"

namespace ldpc {

constexpr int AREA_TRIES = 1 << 20;   // of 32 areas each, under a microsecond: a second or so

// Takes an area for the CTA (all threads call; s_area is shared): its index, or
// -1.  areas.taken null: the launch has areas of its own, one per block index.
__device__ __forceinline__ int take_area(const MsgAreas& areas, int& s_area) {
    if (!areas.taken) return (int)blockIdx.x;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int got = -1;
        if (lane == 0 && atomicCAS(areas.taken + blockIdx.x, 0u, 1u) == 0u) got = (int)blockIdx.x;
        got = __shfl_sync(0xffffffffu, got, 0);
        // 32 areas at a time from this CTA's own on
        for (int i = 0, base = (int)blockIdx.x; got < 0 && i < AREA_TRIES; ++i, base = (base + 32) % areas.n) {
            const int at = (base + lane) % areas.n;
            const bool open = *reinterpret_cast<volatile unsigned int*>(areas.taken + at) == 0u;
            const unsigned any = __ballot_sync(0xffffffffu, open);
            if (!any) continue;
            const int first = __ffs(any) - 1;
            if (lane == first && atomicCAS(areas.taken + at, 0u, 1u) == 0u) got = at;
            got = __shfl_sync(0xffffffffu, got, first);
        }
        if (lane == 0) {
            __threadfence();   // the former holder's writes come before this CTA's
            if (got < 0) {
                *reinterpret_cast<volatile unsigned int*>(areas.status) = 1u;
                __threadfence_system();
            }
            s_area = got;
        }
    }
    __syncthreads();
    return s_area;
}

// Gives the area back (all threads call, after their last message access).
__device__ __forceinline__ void give_area(const MsgAreas& areas, const int& s_area) {
    if (!areas.taken) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicExch(areas.taken + s_area, 0u);
    }
}

}  // namespace ldpc
