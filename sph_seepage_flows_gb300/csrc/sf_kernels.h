// Host-side launch interface of the substep kernels (sf_kernels.cu, sf_sort.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sfg {

// Launches a kernel that starts with afterPrevious (sf_device.cuh), which lets
// the GPU set it up while the kernel before it in the stream drains; captured
// graphs keep the edge as such. A substep of ten kernels: 1,770 particles 52 ->
// 50 us, 20k column 76 -> 74, 1M embankment 572 -> 565. The kernels do not
// release their successors early (griddepcontrol.launch_dependents): the next
// kernel's blocks then wait on the SMs for all of this one, and the substeps
// became 2-3 us longer.
template <typename... P, typename... A>
inline void launchChained(cudaStream_t s, int blocks, int threads, size_t shared, void (*kernel)(P...), A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(blocks));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = shared;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

struct SceneDev;
struct SceneState;

// Passes whose block size the tuner picks (threads per block, a divisor of
// kSlotAlign so that a block never spans two scenes).
enum TunedPass { kPassDensity = 0, kPassAvgFlow, kPassVoidage, kPassSand, kPassWater, kPassIntegrate, kTunedPasses };

// Launch context shared by all passes of one handle.
struct LaunchCtx {
    cudaStream_t stream;
    const SceneDev* scenes;   // device array [n_scenes]
    const int* blockScene;    // device array [slotBlocks]: scene of each kSlotAlign block
    SceneState* state;        // device array [n_scenes]
    unsigned int* errWord;    // device error word
    int slotBlocks;           // total slots / kSlotAlign
    int block[kTunedPasses];  // threads per block of each tuned pass
    int lanes[kTunedPasses];  // threads per slot of each neighbour pass (1, 2, 4 or 8)
    int densityStaged;        // 1: the one-lane density pass stages its candidates in shared memory
    int smCount;              // SMs of the device
};

// Largest shared staging of the density pass, in positions (16 B each): with
// the pass's own shared table it stays within the 48 KB a block gets without
// an opt-in.
constexpr int kDensityStageMax = 3008;

// Neighbour lists of the current substep (column-major: entry k of slot i at
// k * M + i). Particle lists hold sand neighbours from entry 0 upwards and
// water neighbours from entry cap - 1 downwards; cnt packs the two counts
// (sand in the low 16 bits, each saturating at 0xFFFF). Counts summing above
// cap mean the list overflowed: walk the stencil instead. A boundary count
// above kMaxBNbr means the same for the boundary list. The capacity cap is
// chosen per handle from the neighbour counts of its scenes (a multiple of
// 32 between kMinNbr and kMaxNbr).
constexpr int kMinNbr = 64;
constexpr int kMaxNbr = 256;
constexpr int kMaxBNbr = 48;
// Sand-sand pairs within DEM contact + liquid-bridge reach of a sand particle
// (the only pairs with DEM or capillary forces); more means "filter the sand list".
constexpr int kMaxContact = 16;
struct NbrLists {
    const unsigned int* cnt;
    const unsigned int* nbr;
    const int* bcnt;
    const unsigned int* bnbr;
    const int* ccnt;
    const unsigned int* cnbr;
    const unsigned int* cs;   // particle cell table (total_cells + 1)
    const unsigned int* bcs;  // boundary cell table (total_cells + 1)
    // per cell: 1 if a boundary particle lies in the cell or one of its 26
    // neighbours (the boundary is static, so this is set once at creation);
    // null means every cell walks its boundary ranges
    const unsigned char* bnear;
    long long M;              // total slots
    int cap;                  // particle list capacity
};
struct NbrListsW {
    unsigned int* cnt;
    unsigned int* nbr;
    int* bcnt;
    unsigned int* bnbr;
    int* ccnt;
    unsigned int* cnbr;
    const unsigned int* cs;
    const unsigned int* bcs;
    const unsigned char* bnear;
    const unsigned int* bcell;  // cell of each boundary particle
    long long M;
    int cap;
};

// Device buffers the neighbor passes read and write (current sort order).
struct PassBuffers {
    NbrLists lists;
    NbrListsW listsW;
    float4* pos4;
    // positions of slot pairs (2p, 2p + 1), written by the sort: (x0, x1, y0, y1)
    // and (z0, z1), the operands of the density pass's packed reach tests
    const float4* pairXY;
    const float2* pairZ;
    float4* vel4;
    float4* aux4;
    float4* flow4;
    float4* adh4;
    float4* avgadh4;
    float4* drag4;
    float4* acc4;
    float4* col4;
    float4* mat4;
    const float4* bpos4;
    // water: (D, P) = (rho / max(eps, voidage), p / max(eps, D^2)), the
    // effective density and pressure term every momentum pair term of the
    // particle uses (written by the voidage / adhesion pass); sand: the
    // denominators of its voidage quotient and of its average drag (written
    // by the voidage and sand momentum passes), which the adjoint reads
    // instead of summing them again. adh4.w of water holds the denominator
    // of its average adhesion for the same reason.
    float2* dp;
    // Gather records, rewritten every substep so that a neighbour term loads
    // one record besides the neighbour's position (values bit-identical to
    // the ones the terms used to gather from several arrays):
    //   vrec2, average-flow pass -> voidage / adhesion pass: water (fluid
    //     voidage x volume m / rho, volume), sand (adhesion Bezier factor of
    //     its saturation, volume);
    //   grec4: sand (velocity, saturation) from the average-flow pass, for the
    //     DEM contacts; water (velocity, pressure term P) from the voidage /
    //     adhesion pass, for the water momentum pairs.
    // avgadh4.w of water holds its effective density D for the sand momentum pass.
    float2* vrec2;
    float4* grec4;
};

// Threads per slot of the voidage / adhesion and momentum passes for
// totalSlots slots on a GPU with smCount SMs: doubled, up to 8, while fewer
// than 2048 threads per SM would run. The two momentum passes in us with 1, 2, 4
// and 8 lanes, columns / embankments: 20k 47 30 21 17 / 35 22 17 14, 50k 55 34
// 26 25 / 36 24 21 22, 75k 51 34 28 32 / 37 26 26 29, 100k 58 39 35 39 / 39 28 29
// 36, 150k 59 43 44 53 / 43 37 39 51, 200k 82 51 54 69 / 46 41 49 67, 300k 79 68
// 76 100 / 65 60 73 99, 340k 83 72 85 111 / 69 65 80 112, 420k 91 85 102 134 / 74
// 75 98 137. The line dates from 48 registers a thread (five blocks per SM);
// with the 64 of today 4 lanes are the better by a tenth from 55k to 78k slots, and 2
// to 400k. It stays, as other lanes group the momentum sums differently, so
// that results would differ from before in their rounding.
int lanesForSlots(long long totalSlots, int smCount);
// The same for the adjoint pair kernels, but 2 up to 4096 threads per SM: with
// 24 warps per SM at most, one lane per particle leaves their last wave short
// until there are more. A reverse substep in us with 1, 2, 4 and 8 lanes: 20k
// 136 89 65 55, 40k 158 101 76 75, 80k 182 125 109 116, 160k 193 158 158 200,
// 320k 285 255 286 394, 640k 439 446 575 856, 1M 633 689 936 1401.
int adjointLanesForSlots(long long totalSlots, int smCount);
// Threads per slot of the density pass, whose one-lane form does a third of the
// work in all but is one long chain per particle: 8 while no more than 1152
// threads per SM run, 4 while no more than 2304, else 1. Density in us with 1,
// 4 and 8 lanes at the start / after 1200 substeps, when lists are longer:
// columns of 30k 69 37 42 / 86 42 44, 60k 76 59 69 / 95 63 73, 80k 84 71 86 / 91
// 77 92; flat 40k scene 48 43 48 / 93 53 61; embankments of 80k 65 64 80 / 92 70
// 93, 120k 65 88 116 / 95 101 134.
int densityLanesForSlots(long long totalSlots, int smCount);
// Threads per slot of the average-flow pass: as the density pass, but 2 for 1 up
// to 4096 slots per SM. A substep in us with 1, 2, 4 and 8 lanes (/ after 1200
// substeps): flat 40k scene 80.9 81.0 79.8 79.8 / 127.8 118.9 110.6 108.7 (8
// adaptive substeps of another 40k state: 751 us with 2, 761 with 4, 794 with 8),
// columns of 30k 95.0 88.4 83.2 81.9 and 60k 130.6 123.7 119.4 118.9, embankments
// of 80k 124.7 121.7 121.5 122.3 / 159.4 151.3 150.2 150.7, 120k 134.6 131.5
// 131.1 134.3 / 195.3 186.7 186.7 188.6, 300k 223.3 220.3 223.6 235.3; 791k
// column 547 545 560 594.
int flowLanesForSlots(long long totalSlots, int smCount);

void launchBoundaryVolume(const LaunchCtx& c, int sid, int nb, float4* bpos4, const int* blabel,
                          const unsigned int* bcs);
// chained: the average flow follows at once, and takes the sand volume summed here
void launchDensity(const LaunchCtx& c, const PassBuffers& b, bool chained);
// chained: the density pass ran just before (chained), with nothing set in between
void launchAvgFlow(const LaunchCtx& c, const PassBuffers& b, bool chained);
void launchVoidageAdhesion(const LaunchCtx& c, const PassBuffers& b);
void launchSandMomentum(const LaunchCtx& c, const PassBuffers& b);
void launchWaterMomentum(const LaunchCtx& c, const PassBuffers& b);
// Scratch of the counting sort (sf_sort.cu); n: slots, a multiple of 256.
struct CountScratch {
    unsigned int* count;       // nCells rounded up to a multiple of 4
    unsigned int* tileCount;   // kMaxCountTiles: slots per table tile
    uint2* keyRank;            // n: key of each slot before the sort, place among the slots counted into its cell
                               // (of a parked slot: the slot it goes to)
    unsigned char* parkedInWarp;  // n / 32: parked slots of each 32
    unsigned int* parkedBefore;   // n / 256: parked slots before each block of 256, within its tile of blocks
    unsigned int* parkedTile;     // kMaxParkedTiles: parked slots of each tile of blocks
    unsigned int* arrived;     // n: slots of each cell, in arrival order
    unsigned int* sortedKeys;  // n: keys after the sort
    int tileShift;             // log2 of the cells per table tile (countTileShift)
    int parkedShift;           // log2 of the blocks of 256 slots per tile (parkedTileShift)
};
// timeArgDev: when not null, the kernel reads timeArg from this device scalar
// (graph-replayed steps whose render interval changes from call to call).
// cc: where the next sort's keys and counts go (keyRank null: nowhere).
void launchIntegrate(const LaunchCtx& c, const PassBuffers& b, float timeArg, int adaptive, const float* timeArgDev,
                     const CountScratch& cc);
// Largest number of particles within the interaction reach of any particle
// (itself included), atomically maxed into *maxCount; needs the cell table.
void launchNeighborCountMax(const LaunchCtx& c, const float4* pos4, const unsigned int* cs, unsigned int* maxCount);

// ---- stable LSD radix sort of 32-bit cell keys (sf_sort.cu) ----
// Scratch sizes for sorting n keys.
struct SortScratch {
    unsigned int* keysAlt;   // n
    unsigned int* vals;      // n
    unsigned int* valsAlt;   // n
    unsigned int* hist;      // 256 * tiles
    unsigned int* digitTotal;  // 256
    int tiles;               // sortTiles(n, items)
    int items;               // keys per thread of a tile: 1, 2, 4 or 8 (0 means 8)
    int digitBits;           // 8-11 (0 means 8); hist holds 2^digitBits * tiles, digitTotal 2^digitBits
};
// Digit width for keys of keyBits bits: 8, or the narrowest of 9-11 that
// needs fewer passes than 8-bit digits.
int sortDigitBits(int keyBits);
// Tiles of 256 threads x items keys over n keys.
int sortTiles(int n, int items = 8);
// Keys per thread for n keys: the largest of 8, 4, 2 that still gives every
// SM two tiles, else 1 (small sorts are a chain of short launches; smaller
// tiles spread them over more SMs).
int sortItemsFor(int n, int smCount);
// Sorts keys[0..n) (only the low `bits` bits are examined) and writes the
// stable permutation to *permOut (new index -> old index) and the sorted keys
// to *keysOut; both point into keys/scratch buffers. firstHistDone: sc.hist
// already holds the first digit's tile histograms (launchKeysHist). Returns
// kernels launched.
int radixSort(cudaStream_t s, int n, int bits, unsigned int* keys, SortScratch& sc, unsigned int** keysOut,
              unsigned int** permOut, bool firstHistDone = false);
// The cell key of every slot of the handle (n slots, a multiple of 256) and
// the first radix pass's tile histograms into sc.hist, in one launch.
void launchKeysHist(const LaunchCtx& c, int n, const float4* pos4, unsigned int* keys, const SortScratch& sc);
// cellStart[c] = first index i with sortedKeys[i] >= c, for c in [0, nCells]
void launchCellStart(cudaStream_t s, int n, int nCells, const unsigned int* sortedKeys, unsigned int* cellStart);
// Gather the persistent per-slot arrays into sorted order (n a multiple of
// 32) and write the cell table cellStart of the sorted keys (as
// launchCellStart) and the slot-pair positions in the same launch.
void launchReorder(cudaStream_t s, int n, const unsigned int* perm, const float4* pos, const float4* vel,
                   const float4* col, const float4* mat, const float2* amc, const int* pid, float4* posOut,
                   float4* velOut, float4* colOut, float4* matOut, float2* amcOut, int* pidOut,
                   const unsigned int* sortedKeys, int nCells, unsigned int* cellStart, float4* pairXY,
                   float2* pairZ);
// ---- counting sort by cell (sf_sort.cu) ----
constexpr int kMaxCountTiles = 1024;
// Whether the counting sort is used: its table passes cost 12 B per cell, which
// stays behind the radix sort's cost while there are at most 8 cells per slot
// (or a million cells, which the L2 holds).
bool useCountingSort(int slots, int cells);
// log2 of the cells per table tile: 1024 cells, doubled until at most
// kMaxCountTiles tiles are left (every block of the scatter scans the tile sums).
int countTileShift(int cells);
// log2 of the blocks of slots per tile of the scan of the parked slots: 1024,
// doubled until at most kMaxParkedTiles tiles are left (a parked slot adds the
// sums of those of its scene before it).
constexpr int kMaxParkedTiles = 64;
int parkedTileShift(int slots);
// Blocks of 256 threads for a kernel that passes over the slots (slotBlocks) and
// over the cell table: with the slots' blocks alone, a few slots in a large grid
// leave the table to a few threads. Four cells per thread, and up to 8 blocks per
// SM for the table. Sort stage with the blocks of the slots / with these:
// 250 slots in 97k cells 94 / 9 us, in 1M 895 / 12; 2000 in 97k 20 / 11, in 1M 121 /
// 14; 6750 in 1M 45 / 14; 100k in 1M 15.7 / 15.0 (the radix form: 35, 90, 33, 72, 71, 74).
int tableBlocks(int slotBlocks, int cells, int smCount);
// Keys and counts of n slots at pos, into zero counts. ranked: parked slots may
// have to go to another place (countSlot). Returns kernels launched.
int launchCountKeys(const LaunchCtx& c, int n, const float4* pos, const CountScratch& cc, bool ranked);
// The sort stage from the keys and counts: cell table, stable order and gather
// of the persistent arrays (with the slot-pair positions); the counts are zero
// afterwards. Returns kernels launched.
int launchCountingSort(const LaunchCtx& c, int n, int nCells, const CountScratch& cc, const float4* pos,
                       const float4* vel, const float4* col, const float4* mat, const float2* amc, const int* pid,
                       float4* posOut, float4* velOut, float4* colOut, float4* matOut, float2* amcOut, int* pidOut,
                       unsigned int* cellStart, float4* pairXY, float2* pairZ);
// The slot-pair positions of n slots (a multiple of 32), as launchReorder writes them.
void launchPairs2(cudaStream_t s, int n, const float4* pos, float4* pairXY, float2* pairZ);

}  // namespace sfg
