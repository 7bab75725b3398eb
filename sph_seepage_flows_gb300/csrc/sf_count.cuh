// Counting of a slot into its cell, for the counting sort (sf_sort.cu): by its
// own key kernel or by the integrator, whose positions the next sort takes.
#pragma once

#include "sf_device.cuh"
#include "sf_kernels.h"

namespace sfg {

// Set in the place of a slot that is parked (p.w is 0). The place then holds its
// number among the parked slots of its warp and, above those five bits, the
// first block of kSlotAlign slots of its scene (at most 2^22 of them): what the
// scatter needs for parkedPlace without another chain of loads.
constexpr unsigned int kParkedBit = 0x80000000u;

// Counts slot (position p, parked when p.w is 0) into its cell and writes its
// key and its place among the slots counted there. Every thread of the block
// calls it; the block's slots are consecutive and of one scene. The particles
// are nearly in cell order, so a warp counts its runs of equal keys with one
// atomic each; the parking cell, which may hold most slots of a handle, takes
// one per block. Its slots are not ordered by those atomics: a particle whose
// mass was set to 0 is parked too, keeps its id and has to stay in slot order
// before the blank slots, so each warp leaves the number of its parked slots.
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
    const unsigned int parked = __ballot_sync(0xffffffffu, !live);
    if (lane == 0u) cc.parkedInWarp[slot >> 5] = static_cast<unsigned char>(__popc(parked));
    const unsigned int park = kParkedBit | unsigned(S.slot_off / kSlotAlign) << 5 | unsigned(__popc(parked & ((1u << lane) - 1u)));
    cc.keyRank[slot] = make_uint2(key, live ? at : park);
    const int blockParked = __syncthreads_count(!live);
    if (threadIdx.x == 0 && blockParked) atomicAdd(&cc.count[S.cell_off + S.ncell], unsigned(blockParked));
}

// Parked slots in the first `warps` warps of a block of kSlotAlign slots.
__device__ __forceinline__ unsigned int parkedInWarps(const CountScratch& cc, int block, int warps) {
    static_assert(kSlotAlign == 256, "the counts of a block's warps are one 8-byte word");
    uint2 w = reinterpret_cast<const uint2*>(cc.parkedInWarp)[block];
    if (warps < 4) {
        w.x &= (1u << (8 * warps)) - 1u;
        w.y = 0u;
    } else if (warps < 8) {
        w.y &= (1u << (8 * (warps - 4))) - 1u;
    }
    return __dp4a(w.x, 0x01010101u, __dp4a(w.y, 0x01010101u, 0u));
}

// Place of a parked slot, whose place in keyRank is park, among its scene's parked slots.
__device__ __forceinline__ unsigned int parkedPlace(const CountScratch& cc, int slot, unsigned int park) {
    const int block = slot / kSlotAlign, first = int((park & ~kParkedBit) >> 5);
    unsigned int place = cc.parkedBefore[block] - cc.parkedBefore[first] + parkedInWarps(cc, block, (slot >> 5) & 7) + (park & 31u);
    for (int t = first >> cc.parkedShift; t < block >> cc.parkedShift; ++t) place += cc.parkedTile[t];
    return place;
}

}  // namespace sfg
