// Stable LSD radix sort of 32-bit cell keys, cell-start table and reorder.
//
// Replaces the reference's neighbor-grid build (cuda_neighbor_searcher.cu:
// 36-51, 64-116): thrust::sort_by_key on the cell keys with the particle
// arrays as values (a stable sort, so particles of one cell keep their
// previous relative order), then an atomic histogram + exclusive scan for
// cellStart. Here one stable sort of (key, slot) pairs yields the
// permutation, one gather applies it to every persistent array, and
// cellStart[c] is the lower bound of c in the sorted keys. The result is the
// same permutation and the same table as the reference's.
//
// Per digit pass (8-bit digits, or 9-11 bits when that saves a pass): kHist
// (per-tile digit counts), kScanTiles (per digit, exclusive scan over tiles)
// and kScatter (digit offsets, in-tile stable rank: rounds of 256 keys in
// index order, warp match for the rank inside a warp, shared per-warp digit
// counts for the rank across warps, moved into the running digit offsets by
// the warp leaders of each round). The first pass takes its tile histograms
// from the key kernel (kKeysHist), and the reorder writes the cell table
// (cellStart[c] = lower bound of c) as it gathers, so a sort stage of two
// digit passes is seven launches.
#include <algorithm>

#include "sf_count.cuh"
#include "sf_device.cuh"
#include "sf_kernels.h"

namespace sfg {

int sortTiles(int n, int items) { return (n + kSortThreads * items - 1) / (kSortThreads * items); }

int sortItemsFor(int n, int smCount) {
    for (int items = 8; items > 1; items >>= 1)
        if (sortTiles(n, items) >= 2 * smCount) return items;
    return 1;
}

template <int kSortItems, int kBits>
__global__ void __launch_bounds__(kSortThreads) kHist(const unsigned int* __restrict__ keys, int n, int shift,
                                                      unsigned int* __restrict__ hist, int tiles) {
    constexpr int kTile = kSortThreads * kSortItems;
    constexpr int R = 1 << kBits, kPer = R / kSortThreads;
    __shared__ unsigned int h[R];
#pragma unroll
    for (int q = 0; q < kPer; ++q) h[threadIdx.x * kPer + q] = 0;
    __syncthreads();
    const int base = blockIdx.x * kTile;
    // all of the thread's keys are loaded before the first shared-memory add
    unsigned int k[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = base + r * kSortThreads + threadIdx.x;
        k[r] = idx < n ? keys[idx] : 0u;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r)
        if (base + r * kSortThreads + int(threadIdx.x) < n) atomicAdd(&h[(k[r] >> shift) & unsigned(R - 1)], 1u);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int d = threadIdx.x * kPer + q;
        hist[size_t(d) * tiles + blockIdx.x] = h[d];
    }
}

// The cell keys (slotKey) of one tile of slots and the tile's histogram of
// their first digit: kHist of the first pass fused into the key computation.
// Rounds of 256 slots are 256-slot blocks of one scene each.
template <int kSortItems, int kBits>
__global__ void __launch_bounds__(kSortThreads) kKeysHist(const SceneDev* __restrict__ scenes,
                                                          const int* __restrict__ blockScene,
                                                          const float4* __restrict__ pos4,
                                                          unsigned int* __restrict__ keys, unsigned int* errWord,
                                                          int n, unsigned int* __restrict__ hist, int tiles) {
    constexpr int kTile = kSortThreads * kSortItems;
    constexpr int R = 1 << kBits, kPer = R / kSortThreads;
    __shared__ unsigned int h[R];
#pragma unroll
    for (int q = 0; q < kPer; ++q) h[threadIdx.x * kPer + q] = 0;
    __syncthreads();
    const int base = blockIdx.x * kTile;
    // positions are loaded in groups of (up to) four before their keys
    constexpr int kGroup = kSortItems < 4 ? kSortItems : 4;
#pragma unroll 1
    for (int r0 = 0; r0 < kSortItems; r0 += kGroup) {
        float4 p[kGroup];
        int sid[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            const int slot = base + (r0 + u) * kSortThreads + threadIdx.x;
            sid[u] = slot < n ? blockScene[slot / kSlotAlign] : 0;
            p[u] = slot < n ? pos4[slot] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            const int slot = base + (r0 + u) * kSortThreads + threadIdx.x;
            if (slot < n) {
                const unsigned int k = slotKey(scenes[sid[u]], p[u]);
                checkPosition(p[u], errWord);
                keys[slot] = k;
                atomicAdd(&h[k & unsigned(R - 1)], 1u);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int d = threadIdx.x * kPer + q;
        hist[size_t(d) * tiles + blockIdx.x] = h[d];
    }
}

template <int kSortItems>
static void launchKeysHistI(const LaunchCtx& c, int n, const float4* pos4, unsigned int* keys,
                            const SortScratch& sc) {
    switch (sc.digitBits) {
    case 9:
        kKeysHist<kSortItems, 9><<<sc.tiles, kSortThreads, 0, c.stream>>>(c.scenes, c.blockScene, pos4, keys,
                                                                          c.errWord, n, sc.hist, sc.tiles);
        break;
    case 10:
        kKeysHist<kSortItems, 10><<<sc.tiles, kSortThreads, 0, c.stream>>>(c.scenes, c.blockScene, pos4, keys,
                                                                           c.errWord, n, sc.hist, sc.tiles);
        break;
    case 11:
        kKeysHist<kSortItems, 11><<<sc.tiles, kSortThreads, 0, c.stream>>>(c.scenes, c.blockScene, pos4, keys,
                                                                           c.errWord, n, sc.hist, sc.tiles);
        break;
    default:
        kKeysHist<kSortItems, 8><<<sc.tiles, kSortThreads, 0, c.stream>>>(c.scenes, c.blockScene, pos4, keys,
                                                                          c.errWord, n, sc.hist, sc.tiles);
        break;
    }
}

void launchKeysHist(const LaunchCtx& c, int n, const float4* pos4, unsigned int* keys, const SortScratch& sc) {
    switch (sc.items) {
    case 1: launchKeysHistI<1>(c, n, pos4, keys, sc); break;
    case 2: launchKeysHistI<2>(c, n, pos4, keys, sc); break;
    case 4: launchKeysHistI<4>(c, n, pos4, keys, sc); break;
    default: launchKeysHistI<8>(c, n, pos4, keys, sc); break;
    }
}

// Per-digit exclusive scan over tiles: block d scans hist[d * tiles ..
// d * tiles + tiles) in place and writes the digit's total.
__global__ void __launch_bounds__(kSortThreads) kScanTiles(unsigned int* __restrict__ hist, int tiles,
                                                           unsigned int* __restrict__ digitTotal) {
    __shared__ unsigned int part[kSortThreads];
    unsigned int* h = hist + size_t(blockIdx.x) * tiles;
    unsigned int carry = 0;
    for (int base = 0; base < tiles; base += kSortThreads) {
        const int t = base + threadIdx.x;
        const unsigned int v = t < tiles ? h[t] : 0u;
        part[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < kSortThreads; o <<= 1) {
            const unsigned int u = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
            __syncthreads();
            part[threadIdx.x] += u;
            __syncthreads();
        }
        if (t < tiles) h[t] = carry + part[threadIdx.x] - v;
        carry += part[kSortThreads - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) digitTotal[blockIdx.x] = carry;
}

template <int kSortItems, int kBits>
__global__ void __launch_bounds__(kSortThreads) kScatter(const unsigned int* __restrict__ keysIn,
                                                         const unsigned int* __restrict__ valsIn,
                                                         unsigned int* __restrict__ keysOut,
                                                         unsigned int* __restrict__ valsOut, int n, int shift,
                                                         const unsigned int* __restrict__ hist, int tiles,
                                                         const unsigned int* __restrict__ digitTotal) {
    constexpr int kWarps = kSortThreads / 32;
    constexpr int kTile = kSortThreads * kSortItems;
    constexpr int R = 1 << kBits, kPer = R / kSortThreads;
    __shared__ unsigned int base[R];
    __shared__ unsigned int running[R];
    __shared__ unsigned char cnt[kWarps][R];  // keys of a digit per warp in one round (<= 32)
    __shared__ unsigned int warpSum[kWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // digit offsets: exclusive scan of the digit totals (kPer consecutive
    // digits per thread, then a block scan of the threads' sums)
    unsigned int tot[kPer], sum = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        tot[q] = digitTotal[tid * kPer + q];
        sum += tot[q];
    }
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warpSum[warp] = incl;
    __syncthreads();
    unsigned int acc = incl - sum;
    for (int w = 0; w < warp; ++w) acc += warpSum[w];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int d = tid * kPer + q;
        base[d] = acc + hist[size_t(d) * tiles + blockIdx.x];
        acc += tot[q];
        running[d] = 0;
    }
    unsigned int* cnt32 = reinterpret_cast<unsigned int*>(&cnt[0][0]);
    for (int q = tid; q < kWarps * R / 4; q += kSortThreads) cnt32[q] = 0u;
    __syncthreads();
    const unsigned int ltMask = (1u << lane) - 1u;
    const int tileBase = blockIdx.x * kTile;
    // the thread's keys and values of every round are loaded up front, so the
    // rounds (three barriers each) do not wait for global loads
    unsigned int kr[kSortItems], vr[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = tileBase + r * kSortThreads + tid;
        kr[r] = idx < n ? keysIn[idx] : 0u;
        vr[r] = idx < n ? (valsIn ? valsIn[idx] : unsigned(idx)) : 0u;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = tileBase + r * kSortThreads + tid;
        const bool valid = idx < n;
        const unsigned int k = kr[r], v = vr[r];
        const unsigned int d = valid ? (k >> shift) & unsigned(R - 1) : unsigned(R);
        const unsigned int peers = __match_any_sync(0xffffffffu, d);
        const unsigned int rank = __popc(peers & ltMask);
        const bool leader = valid && rank == 0;
        if (leader) cnt[warp][d] = (unsigned char)__popc(peers);
        __syncthreads();
        if (valid) {
            unsigned int pre = 0;
            for (int w = 0; w < warp; ++w) pre += cnt[w][d];
            const unsigned int pos = base[d] + running[d] + pre + rank;
            keysOut[pos] = k;
            valsOut[pos] = v;
        }
        __syncthreads();
        // only the digits of this round: the warp leaders move their counts
        if (leader) {
            atomicAdd(&running[d], unsigned(__popc(peers)));
            cnt[warp][d] = 0;
        }
        __syncthreads();
    }
}

template <int kSortItems, int kBits>
static void launchPassT(cudaStream_t s, int n, int shift, const unsigned int* kIn, const unsigned int* vIn,
                        unsigned int* kOut, unsigned int* vOut, const SortScratch& sc, bool histDone) {
    const int tiles = sc.tiles;
    if (!histDone) kHist<kSortItems, kBits><<<tiles, kSortThreads, 0, s>>>(kIn, n, shift, sc.hist, tiles);
    kScanTiles<<<1 << kBits, kSortThreads, 0, s>>>(sc.hist, tiles, sc.digitTotal);
    kScatter<kSortItems, kBits><<<tiles, kSortThreads, 0, s>>>(kIn, vIn, kOut, vOut, n, shift, sc.hist, tiles,
                                                               sc.digitTotal);
}

template <int kSortItems>
static void launchPass(cudaStream_t s, int n, int shift, int bits, const unsigned int* kIn,
                       const unsigned int* vIn, unsigned int* kOut, unsigned int* vOut, const SortScratch& sc,
                       bool histDone) {
    switch (bits) {
    case 9: launchPassT<kSortItems, 9>(s, n, shift, kIn, vIn, kOut, vOut, sc, histDone); break;
    case 10: launchPassT<kSortItems, 10>(s, n, shift, kIn, vIn, kOut, vOut, sc, histDone); break;
    case 11: launchPassT<kSortItems, 11>(s, n, shift, kIn, vIn, kOut, vOut, sc, histDone); break;
    default: launchPassT<kSortItems, 8>(s, n, shift, kIn, vIn, kOut, vOut, sc, histDone); break;
    }
}

int sortDigitBits(int keyBits) {
    const int passes8 = (keyBits + 7) / 8, passes11 = (keyBits + 10) / 11;
    if (passes11 >= passes8) return 8;
    return (keyBits + passes11 - 1) / passes11;  // the narrowest digits for that many passes
}

int radixSort(cudaStream_t s, int n, int bits, unsigned int* keys, SortScratch& sc, unsigned int** keysOut,
              unsigned int** permOut, bool firstHistDone) {
    const int digit = sc.digitBits ? sc.digitBits : 8;
    const int passes = (bits + digit - 1) / digit;
    unsigned int* kIn = keys;
    unsigned int* kOut = sc.keysAlt;
    unsigned int* vIn = nullptr;
    unsigned int* vOut = sc.vals;
    int launches = 0;
    for (int p = 0; p < passes; ++p) {
        const int shift = digit * p;
        const bool histDone = p == 0 && firstHistDone;
        switch (sc.items) {
        case 1: launchPass<1>(s, n, shift, digit, kIn, vIn, kOut, vOut, sc, histDone); break;
        case 2: launchPass<2>(s, n, shift, digit, kIn, vIn, kOut, vOut, sc, histDone); break;
        case 4: launchPass<4>(s, n, shift, digit, kIn, vIn, kOut, vOut, sc, histDone); break;
        default: launchPass<8>(s, n, shift, digit, kIn, vIn, kOut, vOut, sc, histDone); break;
        }
        launches += histDone ? 2 : 3;
        // next pass reads what this one wrote
        unsigned int* t = kIn;
        kIn = kOut;
        kOut = t;
        vIn = vOut;
        vOut = (vOut == sc.vals) ? sc.valsAlt : sc.vals;
    }
    *keysOut = kIn;
    *permOut = vIn;
    return launches;
}

__global__ void kCellStart(int n, int nCells, const unsigned int* __restrict__ sk, unsigned int* __restrict__ cs) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c > nCells) return;
    int lo = 0, hi = n;  // first index with sk[i] >= c
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sk[mid] < unsigned(c))
            lo = mid + 1;
        else
            hi = mid;
    }
    cs[c] = unsigned(lo);
}

void launchCellStart(cudaStream_t s, int n, int nCells, const unsigned int* sortedKeys, unsigned int* cellStart) {
    kCellStart<<<(nCells + 1 + 255) / 256, 256, 0, s>>>(n, nCells, sortedKeys, cellStart);
}

// cellStart[c] = v for c in [lo, hi), written by the lanes of one warp
// (all 32 call it): short runs by their own lane, long runs (the empty cells
// before a sparse region, up to whole empty slabs of the grid) by the whole
// warp, one run after the other, in 16-byte stores (the table is 16-byte
// aligned).
__device__ __forceinline__ void fillCellRuns(unsigned int* __restrict__ cs, unsigned int lo, unsigned int hi,
                                             unsigned int v) {
    constexpr unsigned int kShort = 8;
    if (hi - lo <= kShort)
        for (unsigned int c = lo; c < hi; ++c) cs[c] = v;
    const unsigned int lane = threadIdx.x & 31u;
    for (unsigned int longRuns = __ballot_sync(0xffffffffu, hi - lo > kShort); longRuns; longRuns &= longRuns - 1u) {
        const int src = __ffs(longRuns) - 1;
        const unsigned int l = __shfl_sync(0xffffffffu, lo, src), h = __shfl_sync(0xffffffffu, hi, src);
        const unsigned int w = __shfl_sync(0xffffffffu, v, src);
        const unsigned int a = min(h, (l + 3u) & ~3u), b = a + ((h - a) & ~3u);  // [a, b): whole 16-byte words
        if (lane < a - l) cs[l + lane] = w;
        if (lane < h - b) cs[b + lane] = w;
        const uint4 w4 = make_uint4(w, w, w, w);
        for (unsigned int q = a / 4u + lane; q < b / 4u; q += 32u) reinterpret_cast<uint4*>(cs)[q] = w4;
    }
}

// The positions of one slot pair in structure-of-arrays form, written by the
// pair's two lanes (the whole warp calls it; slots are warp-aligned).
__device__ __forceinline__ void writePair(int i, float4 p, float4* __restrict__ pairXY, float2* __restrict__ pairZ) {
    const float qx = __shfl_xor_sync(0xffffffffu, p.x, 1), qy = __shfl_xor_sync(0xffffffffu, p.y, 1),
                qz = __shfl_xor_sync(0xffffffffu, p.z, 1);
    if (i & 1)
        pairZ[i >> 1] = make_float2(qz, p.z);
    else
        pairXY[i >> 1] = make_float4(p.x, qx, p.y, qy);
}

__global__ void kPairs(int n, const float4* __restrict__ pos, float4* __restrict__ pairXY,
                       float2* __restrict__ pairZ) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) writePair(i, pos[i], pairXY, pairZ);  // n is a multiple of 32: whole warps
}

void launchPairs2(cudaStream_t s, int n, const float4* pos, float4* pairXY, float2* pairZ) {
    kPairs<<<(n + 255) / 256, 256, 0, s>>>(n, pos, pairXY, pairZ);
}

__global__ void kReorder(int n, const unsigned int* __restrict__ perm, const float4* __restrict__ pos,
                         const float4* __restrict__ vel, const float4* __restrict__ col,
                         const float4* __restrict__ mat, const float2* __restrict__ amc, const int* __restrict__ pid,
                         float4* __restrict__ posOut, float4* __restrict__ velOut, float4* __restrict__ colOut,
                         float4* __restrict__ matOut, float2* __restrict__ amcOut, int* __restrict__ pidOut,
                         const unsigned int* __restrict__ sk, int nCells, unsigned int* __restrict__ cs,
                         float4* __restrict__ pairXY, float2* __restrict__ pairZ) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;  // n is a multiple of 32: whole warps stay
    // cell table (the lower bound of every cell in the sorted keys): index i
    // starts the cells after its predecessor's key up to its own key; the
    // last index also ends the table
    // (keys above nCells, which only a corrupt position could give, are
    // clamped: that leaves every lower bound in [0, nCells] unchanged)
    const unsigned int top = unsigned(nCells);
    const unsigned int k = min(sk[i], top);
    fillCellRuns(cs, i == 0 ? 0u : min(sk[i - 1], top) + 1u, k + 1u, unsigned(i));
    fillCellRuns(cs, k + 1u, i == n - 1 ? unsigned(nCells) + 1u : k + 1u, unsigned(n));
    const unsigned int o = perm[i];
    const float4 p = pos[o];
    posOut[i] = p;
    writePair(i, p, pairXY, pairZ);
    velOut[i] = vel[o];
    colOut[i] = col[o];
    matOut[i] = mat[o];
    amcOut[i] = amc[o];
    pidOut[i] = pid[o];
}

void launchReorder(cudaStream_t s, int n, const unsigned int* perm, const float4* pos, const float4* vel,
                   const float4* col, const float4* mat, const float2* amc, const int* pid, float4* posOut,
                   float4* velOut, float4* colOut, float4* matOut, float2* amcOut, int* pidOut,
                   const unsigned int* sortedKeys, int nCells, unsigned int* cellStart, float4* pairXY,
                   float2* pairZ) {
    kReorder<<<(n + 255) / 256, 256, 0, s>>>(n, perm, pos, vel, col, mat, amc, pid, posOut, velOut, colOut, matOut,
                                            amcOut, pidOut, sortedKeys, nCells, cellStart, pairXY, pairZ);
}

// ------------------------------------------------- counting sort by cell
// The sort stage where the cell table is not much larger than the particle
// arrays (useCountingSort): three or four launches instead of seven (two digits) or ten.
//   kCountKeys     the key of every slot and its place among the slots counted
//                  into its cell (in arrival order); the integrator leaves the
//                  same for the positions it writes, so this runs only after
//                  positions came from elsewhere
//   kScanParked,   after masses were set and the slots counted anew: where the
//   kRankParked    parked slots go, in slot order, as the atomics that count
//                  them have none
//   kCellScan      exclusive scan of the counts within each table tile
//   kCountScatter  adds the slots of the tiles before (the cell table), and
//                  lists the slots of each cell in arrival order, the parked
//                  slots where they go
//   kCellReorder   the place of each slot within its cell by slot number (the
//                  stable order), the gather of the persistent arrays, and the
//                  counts cleared for the next sort; a non-finite position is
//                  reported here and not where it was counted, since a caller
//                  may still replace what the integrator wrote
// The particles are nearly in cell order from the substep before, so a warp
// counts its runs of equal keys with one atomic each, and a cell's slots are
// next to each other in memory. Atomics on few addresses are kept out: a count
// per table tile beside the cells' (a few hundred addresses) made the 1M sort
// 115 us with one per run, 66 with one per warp.
// Sort stage against the radix sort: 1M embankment 77.5 -> 51.6 us (keys 10,
// scan 3, scatter 8, reorder 27 of 190 MB through L2), and 42 behind an integrator
// that counted; 252k 40.9 -> 13.6, 64-scene ensemble 86 -> 49; on small scenes
// its launches count: 40k 28.8 -> 8.3.
constexpr int kScanItems = 4;
constexpr int kScanChunk = kSortThreads * kScanItems;
constexpr int kTableBlocksPerSM = 8;  // each block of the scatter scans the tile sums once

bool useCountingSort(int slots, int cells) { return cells <= max(8LL * slots, 1LL << 20); }

int countTileShift(int cells) {
    int shift = 10;
    while ((cells >> shift) >= kMaxCountTiles) ++shift;
    return shift;
}

int tableBlocks(int slotBlocks, int cells, int smCount) {
    return std::max(slotBlocks, std::min((cells - 1) / (4 * kSortThreads) + 1, kTableBlocksPerSM * smCount));
}

int parkedTileShift(int slots) {
    int shift = 10;
    while ((slots / kSlotAlign >> shift) >= kMaxParkedTiles) ++shift;
    return shift;
}

__global__ void __launch_bounds__(kSlotAlign) kCountKeys(const SceneDev* __restrict__ scenes,
                                                         const int* __restrict__ blockScene,
                                                         const float4* __restrict__ pos4, CountScratch cc, bool ranked) {
    const int slot = blockIdx.x * kSlotAlign + afterPrevious(threadIdx.x);
    const float4 p = pos4[slot];
    countSlot(scenes[blockScene[blockIdx.x]], slot, p, cc);
    if (ranked) {
        const unsigned int parked = __ballot_sync(0xffffffffu, p.w == 0.f);
        if ((threadIdx.x & 31u) == 0u) cc.parkedInWarp[slot >> 5] = static_cast<unsigned char>(__popc(parked));
    }
}

// Parked slots of the first `warps` warps of a block of kSlotAlign slots.
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

// Block t: tile t of the blocks of kSlotAlign slots, the exclusive prefix of
// their parked slots and its sum.
__global__ void __launch_bounds__(kSortThreads) kScanParked(CountScratch cc, int blocks) {
    unsigned int carry = 0u, total;
    const int t = afterPrevious(int(blockIdx.x)), end = min((t + 1) << cc.parkedShift, blocks);
    for (int base = t << cc.parkedShift; base < end; base += kScanChunk) {
        const int first = base + int(threadIdx.x) * kScanItems;
        unsigned int v[kScanItems], sum = 0u;
#pragma unroll
        for (int u = 0; u < kScanItems; ++u) sum += v[u] = first + u < end ? parkedInWarps(cc, first + u, 8) : 0u;
        unsigned int a = carry + blockScan(sum, total);
#pragma unroll
        for (int u = 0; u < kScanItems; ++u) {
            if (first + u < end) cc.parkedBefore[first + u] = a;
            a += v[u];
        }
        carry += total;
    }
    if (threadIdx.x == 0) cc.parkedTile[t] = carry;
}

// Where each parked slot goes: its scene's parked slots fill the end of the
// scene's slots in slot order.
__global__ void __launch_bounds__(kSlotAlign) kRankParked(const SceneDev* __restrict__ scenes,
                                                          const int* __restrict__ blockScene, CountScratch cc) {
    const int block = blockIdx.x, slot = block * kSlotAlign + afterPrevious(threadIdx.x);
    const bool parked = (cc.keyRank[slot].y & kParkedBit) != 0u;
    const unsigned int warp = __ballot_sync(0xffffffffu, parked);
    if (!parked) return;
    const SceneDev& S = scenes[blockScene[block]];
    const int first = S.slot_off / kSlotAlign;
    unsigned int place = cc.parkedBefore[block] - cc.parkedBefore[first] + parkedInWarps(cc, block, int(threadIdx.x >> 5)) +
                         unsigned(__popc(warp & ((1u << (threadIdx.x & 31u)) - 1u)));
    for (int t = first >> cc.parkedShift; t < block >> cc.parkedShift; ++t) place += cc.parkedTile[t];
    cc.keyRank[slot].y = kParkedBit | (unsigned(S.slot_off + S.slot_cap) - cc.count[S.cell_off + S.ncell] + place);
}

// Block b scans table tile b (2^tileShift cells, a multiple of kScanChunk) in
// place and writes its sum.
__global__ void __launch_bounds__(kSortThreads) kCellScan(CountScratch cc, int nCells) {
    unsigned int carry = 0u, total;
    const int tileBeg = afterPrevious(int(blockIdx.x)) << cc.tileShift, tileEnd = min(tileBeg + (1 << cc.tileShift), nCells);
    for (int base = tileBeg; base < tileEnd; base += kScanChunk) {
        const int c = base + int(threadIdx.x) * kScanItems;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (c < tileEnd) v = *reinterpret_cast<const uint4*>(cc.count + c);  // padded to whole 16-byte words
        const unsigned int a = carry + blockScan(v.x + v.y + v.z + v.w, total);
        if (c < tileEnd)
            *reinterpret_cast<uint4*>(cc.count + c) = make_uint4(a, a + v.x, a + v.x + v.y, a + v.x + v.y + v.z);
        carry += total;
    }
    if (threadIdx.x == 0) cc.tileCount[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(kSortThreads) kCountScatter(CountScratch cc, int n, int nCells, int tiles,
                                                              unsigned int* __restrict__ cs) {
    // every block scans the (at most kMaxCountTiles) tile sums
    __shared__ unsigned int before[kMaxCountTiles];
    unsigned int carry = 0u, total;
    const int tid = afterPrevious(threadIdx.x);
    for (int base = 0; base < tiles; base += kSortThreads) {
        const int t = base + tid;
        const unsigned int a = blockScan(t < tiles ? cc.tileCount[t] : 0u, total);
        if (t < tiles) before[t] = carry + a;
        carry += total;
    }
    __syncthreads();
    const int first = blockIdx.x * kSortThreads + tid, threads = gridDim.x * kSortThreads;
    for (int i = first; i < n; i += threads) {
        const uint2 kr = cc.keyRank[i];
        const unsigned int at = kr.y & kParkedBit ? kr.y & ~kParkedBit
                                                  : cc.count[kr.x] + before[kr.x >> cc.tileShift] + kr.y;
        cc.arrived[at] = unsigned(i);
    }
    for (int c = first; c < nCells; c += threads) cs[c] = cc.count[c] + before[c >> cc.tileShift];
    if (first == 0) cs[nCells] = unsigned(n);
}

__global__ void __launch_bounds__(kSortThreads)
    kCellReorder(CountScratch cc, int n, int nCells, const unsigned int* __restrict__ cs, const float4* __restrict__ pos,
                 const float4* __restrict__ vel, const float4* __restrict__ col, const float4* __restrict__ mat,
                 const float2* __restrict__ amc, const int* __restrict__ pid, float4* __restrict__ posOut,
                 float4* __restrict__ velOut, float4* __restrict__ colOut, float4* __restrict__ matOut,
                 float2* __restrict__ amcOut, int* __restrict__ pidOut, float* __restrict__ pairXY,
                 float* __restrict__ pairZ, unsigned int* errWord) {
    const int i = blockIdx.x * kSortThreads + afterPrevious(threadIdx.x);
    for (int c = i; c < ((nCells + 3) & ~3); c += gridDim.x * kSortThreads) cc.count[c] = 0u;
    if (i >= n) return;
    const unsigned int o = cc.arrived[i];
    const float4 p = pos[o], v = vel[o], cl = col[o], m = mat[o];
    const float2 am = amc[o];
    const int id = pid[o];
    const unsigned int key = cc.keyRank[o].x;
    unsigned int d = unsigned(i);
    checkPosition(p, errWord);
    if (p.w != 0.f) {  // the parked slots are listed where they go
        const unsigned int beg = cs[key], end = cs[key + 1];
        d = beg;
        for (unsigned int q = beg; q < end; ++q) d += cc.arrived[q] < o ? 1u : 0u;
    }
    posOut[d] = p;
    velOut[d] = v;
    colOut[d] = cl;
    matOut[d] = m;
    amcOut[d] = am;
    pidOut[d] = id;
    cc.sortedKeys[d] = key;
    const unsigned int q = (d >> 1) * 4u + (d & 1u);
    pairXY[q] = p.x;
    pairXY[q + 2u] = p.y;
    pairZ[d] = p.z;
}

int launchCountKeys(const LaunchCtx& c, int n, const float4* pos, const CountScratch& cc, bool ranked) {
    const int blocks = n / kSlotAlign;
    launchChained(c.stream, blocks, kSlotAlign, 0, kCountKeys, c.scenes, c.blockScene, pos, cc, ranked);
    if (!ranked) return 1;
    launchChained(c.stream, ((blocks - 1) >> cc.parkedShift) + 1, kSortThreads, 0, kScanParked, cc, blocks);
    launchChained(c.stream, blocks, kSlotAlign, 0, kRankParked, c.scenes, c.blockScene, cc);
    return 3;
}

int launchCountingSort(const LaunchCtx& c, int n, int nCells, const CountScratch& cc, const float4* pos,
                       const float4* vel, const float4* col, const float4* mat, const float2* amc, const int* pid,
                       float4* posOut, float4* velOut, float4* colOut, float4* matOut, float2* amcOut, int* pidOut,
                       unsigned int* cellStart, float4* pairXY, float2* pairZ) {
    const int blocks = n / kSlotAlign, tiles = ((nCells - 1) >> cc.tileShift) + 1;
    launchChained(c.stream, tiles, kSortThreads, 0, kCellScan, cc, nCells);
    const int all = tableBlocks(blocks, nCells, c.smCount);
    launchChained(c.stream, std::min(all, kTableBlocksPerSM * c.smCount), kSortThreads, 0, kCountScatter, cc, n, nCells, tiles,
                  cellStart);
    launchChained(c.stream, all, kSortThreads, 0, kCellReorder, cc, n, nCells, cellStart, pos, vel, col, mat, amc,
                  pid, posOut, velOut, colOut, matOut, amcOut, pidOut, reinterpret_cast<float*>(pairXY),
                  reinterpret_cast<float*>(pairZ), c.errWord);
    return 3;
}

}  // namespace sfg
