// Counting of a slot into its cell, for the counting sort (sf_sort.cu): by its
// own key kernel or by the integrator, whose positions the next sort takes.
#pragma once

#include "sf_device.cuh"
#include "sf_kernels.h"

namespace sfg {

// Set in the place of a slot that is parked (p.w is 0), which holds the slot that
// it goes to: its own, unless kRankParked says another. Blank slots never leave
// the end of their scene, and after a sort the particles whose mass was set to 0
// lie before them in slot order, so a slot that is parked goes to another place
// only after masses were set or particles added.
constexpr unsigned int kParkedBit = 0x80000000u;

// Counts slot (position p, parked when p.w is 0) into its cell and writes its
// key and its place among the slots counted there. Every thread of the block
// calls it; the block's slots are consecutive and of one scene. The particles
// are nearly in cell order, so a warp counts its runs of equal keys with one
// atomic each; the parking cell, which may hold most slots of a handle, takes
// one per block.
__device__ __forceinline__ void countSlot(const SceneDev& S, int slot, float4 p, const CountScratch& cc) {
    const bool live = p.w != 0.f;
    const unsigned int key = slotKey(S, p);
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned int heads = __ballot_sync(0xffffffffu, lane == 0u || prev != key);
    unsigned int at = 0u;
    if (live && ((heads >> lane) & 1u)) {
        const unsigned int behind = lane == 31u ? 0u : heads >> (lane + 1u);
        at = atomicAdd(&cc.count[key], behind ? unsigned(__ffs(behind)) : 32u - lane);
    }
    const int leader = 31 - __clz(heads & (0xffffffffu >> (31u - lane)));
    at = __shfl_sync(0xffffffffu, at, leader) + (lane - unsigned(leader));
    cc.keyRank[slot] = make_uint2(key, live ? at : kParkedBit | unsigned(slot));
    const int blockParked = __syncthreads_count(!live);
    if (threadIdx.x == 0 && blockParked) atomicAdd(&cc.count[S.cell_off + S.ncell], unsigned(blockParked));
}

}  // namespace sfg
