// Allocation-free cell sort (sf_cell_sort_noalloc): the sort stage of a
// single-scene handle on caller buffers, with every scratch word in one static
// device array instead of handle memory.
//
// Two forms, as in the handle's sort stage. The counting sort counts in the
// caller's cell table: clear, keys and counts, scan of each table tile, tiles
// added up (the table is then final), slots of each cell in arrival order,
// stable order. The radix sort (keys, digit passes, table by binary search)
// is for grids with many more cells than particles, and for input with a cell
// of more than kCrowded particles: finding their order slot by slot would cost
// the square of their number, so the last kernel reports such a cell instead.
// The call is a chain of short launches and a wait: 200k particles 84 -> 33 us.
//
// The scratch (g_noallocScratch) holds the keys and the arrays of either form.
// A call reports through one page of registered host memory, which its kernels
// write directly. Both are looked up once per device (scratchOf). Every scratch
// word is written before it is read.
// Calls that overlap on the GPU share the scratch and race.
#include "../../include/sf_capi.h"
#include "sf_device.cuh"
#include "sf_kernels.h"

#include <stdlib.h>
#include <unistd.h>

#include <mutex>
#include <string>

namespace sfg {
void setGlobalError(const std::string& msg);  // sf_capi.cu: text for sf_last_error_string(NULL)
}

namespace {

using namespace sfg;

constexpr int kMaxN = SF_NOALLOC_MAX_PARTICLES;
constexpr size_t kHistWords = 256 * size_t(kMaxN / 1024);  // >= 256 digit counts per sort tile
constexpr size_t kWords = 4 * size_t(kMaxN) + 256 + kHistWords;
constexpr unsigned int kCrowded = 256;          // most particles of a cell that the counting sort orders
constexpr int kMaxDevices = 64;

__device__ __align__(256) unsigned int g_noallocScratch[kWords];

// What a call's kernels report, in registered host memory: cleared by the host
// before the launches, set to 1 by any thread that finds the condition.
struct Report {
    unsigned int nonFinite, crowded;
};

// Pos2GridHash of a position (the key of the sort stage for a single-scene
// handle); a non-finite one is reported.
__device__ __forceinline__ unsigned int keyOf(const SceneDev& S, const float* __restrict__ pos, int i,
                                              Report* report) {
    const float3 q = mk3(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]);
    if (!(isfinite(q.x) && isfinite(q.y) && isfinite(q.z))) report->nonFinite = 1u;
    return unsigned(localHash(S, cellOf(S, q)));
}

__global__ void kNoAllocKeys(SceneDev S, const float* __restrict__ pos, int n, unsigned int* __restrict__ keys,
                             Report* report) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = keyOf(S, pos, i, report);
}

constexpr int kThreads = kSortThreads, kItems = 4;  // 1024 cells per turn of a scan block

// (key, place among the particles counted into its cell), counting in the
// table; runs of equal keys in a warp take one atomic.
__global__ void __launch_bounds__(kThreads) kNoAllocCount(SceneDev S, const float* __restrict__ pos, int n,
                                                          unsigned int* table, uint2* __restrict__ keyRank,
                                                          Report* report) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int key = i < n ? keyOf(S, pos, i, report) : 0xffffffffu;
    const unsigned int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned int heads = __ballot_sync(0xffffffffu, lane == 0u || prev != key);
    unsigned int at = 0u;
    if (i < n && ((heads >> lane) & 1u)) {
        const unsigned int behind = lane == 31u ? 0u : heads >> (lane + 1u);
        at = atomicAdd(&table[key], behind ? unsigned(__ffs(behind)) : 32u - lane);
    }
    const int leader = 31 - __clz(heads & (0xffffffffu >> (31u - lane)));
    at = __shfl_sync(0xffffffffu, at, leader) + (lane - unsigned(leader));
    if (i < n) keyRank[i] = make_uint2(key, at);
}

// Block b: exclusive scan of table tile b (2^shift cells) in place, and its sum.
__global__ void __launch_bounds__(kThreads) kNoAllocScan(unsigned int* table, int nCells, int shift,
                                                         unsigned int* __restrict__ tileSum) {
    const int beg = int(blockIdx.x) << shift, end = min(beg + (1 << shift), nCells);
    unsigned int carry = 0u, total;
    for (int base = beg; base < end; base += kThreads * kItems) {
        const int c = base + int(threadIdx.x) * kItems;
        unsigned int v[kItems], sum = 0u;
#pragma unroll
        for (int u = 0; u < kItems; ++u) sum += v[u] = c + u < end ? table[c + u] : 0u;
        unsigned int a = carry + blockScan(sum, total);
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            if (c + u < end) table[c + u] = a;
            a += v[u];
        }
        carry += total;
    }
    if (threadIdx.x == 0) tileSum[blockIdx.x] = carry;
}

// Adds the sums of the tiles before to every tile but the first (one block per
// tile); the table is then final.
__global__ void __launch_bounds__(kThreads) kNoAllocAddTiles(unsigned int* table, int nCells, int n, int shift,
                                                             const unsigned int* __restrict__ tileSum) {
    unsigned int before = 0u, total;
    for (int t = threadIdx.x; t < int(blockIdx.x); t += kThreads) before += tileSum[t];
    blockScan(before, total);
    const int beg = int(blockIdx.x) << shift, end = min(beg + (1 << shift), nCells);
    if (total)
        for (int c = beg + int(threadIdx.x); c < end; c += kThreads) table[c] += total;
    if (end == nCells && threadIdx.x == 0) table[nCells] = unsigned(n);
}

__global__ void __launch_bounds__(kThreads) kNoAllocScatter(int n, const unsigned int* __restrict__ table,
                                                            const uint2* __restrict__ keyRank,
                                                            unsigned int* __restrict__ arrived) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const uint2 kr = keyRank[i];
    arrived[table[kr.x] + kr.y] = unsigned(i);
}

// The stable order: a particle's place in its cell is the number of the cell's
// particles with a smaller index.
__global__ void __launch_bounds__(kThreads) kNoAllocOrder(int n, const unsigned int* __restrict__ table,
                                                          const uint2* __restrict__ keyRank,
                                                          const unsigned int* __restrict__ arrived,
                                                          int* __restrict__ perm, Report* report) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const unsigned int o = arrived[i], key = keyRank[o].x, beg = table[key], end = table[key + 1];
    if (end - beg > kCrowded) {
        report->crowded = 1u;
        return;
    }
    unsigned int d = beg;
    for (unsigned int q = beg; q < end; ++q) d += arrived[q] < o ? 1u : 0u;
    perm[d] = int(o);
}

sf_status failWith(sf_status st, const std::string& msg) {
    setGlobalError(msg);
    return st;
}

// Whether the runtime knows p as registered host memory.
bool isRegistered(const void* p) {
    cudaPointerAttributes a{};
    if (!p) return false;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();  // not sticky: clear it so later checks see only their own errors
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// What a call uses of a device.
struct Scratch {
    unsigned int* words = nullptr;    // g_noallocScratch
    Report* report = nullptr;         // host address of the report page
    Report* reportOnDevice = nullptr;
};

// The scratch of the current device: looked up on the first call on a device
// and again after its context was reset (cudaDeviceReset or any teardown of
// the primary context), when the module is loaded again and cached addresses
// may be stale. A reset frees pinned memory, so the report page is not the
// runtime's: it is a page of this library's own that stays allocated, and is
// registered with the context. The host may therefore always write it, no
// other allocation can be found at its address, and that the runtime no longer
// knows it as registered is what tells of a reset. (The device address alone
// does not: by the next call the module, or another allocation, may have taken
// the same place.)
bool scratchOf(int device, Scratch& out, std::string& why) {
    static std::mutex mu;
    static Scratch known[kMaxDevices];
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= kMaxDevices) return why = "device index out of range", false;
    Scratch& k = known[device];
    if (!k.words || !isRegistered(k.report)) {
        const size_t page = size_t(sysconf(_SC_PAGESIZE));
        void* p = k.report;
        if (!p && posix_memalign(&p, page, page) != 0) return why = "no host memory for the report page", false;
        k.report = static_cast<Report*>(p);
        k.words = nullptr;
        cudaError_t e = cudaSuccess;
        if (!isRegistered(p) &&
            (e = cudaHostRegister(p, page, cudaHostRegisterMapped)) != cudaSuccess)
            return why = std::string("cudaHostRegister: ") + cudaGetErrorString(e), false;
        void *d = nullptr, *s = nullptr;
        if ((e = cudaHostGetDevicePointer(&d, p, 0)) != cudaSuccess)
            return why = std::string("cudaHostGetDevicePointer: ") + cudaGetErrorString(e), false;
        if ((e = cudaGetSymbolAddress(&s, g_noallocScratch)) != cudaSuccess)
            return why = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e), false;
        k.reportOnDevice = static_cast<Report*>(d);
        k.words = static_cast<unsigned int*>(s);
    }
    out = k;
    return true;
}

}  // namespace

extern "C" sf_status sf_cell_sort_noalloc(const sf_boundary_params* grid, const float* pos_dev, int64_t n,
                                          int32_t* perm_out_dev, int32_t* cell_start_out_dev, void* stream) {
    if (!grid || !cell_start_out_dev || n < 0 || (n > 0 && (!pos_dev || !perm_out_dev)))
        return failWith(SF_ERR_INVALID, "sf_cell_sort_noalloc: null pointer or negative count");
    if (n > kMaxN)
        return failWith(SF_ERR_INVALID, "sf_cell_sort_noalloc: n = " + std::to_string(n) +
                                            " exceeds SF_NOALLOC_MAX_PARTICLES (" + std::to_string(kMaxN) + ")");
    if (!(grid->kernel_radius > 0.f)) return failWith(SF_ERR_INVALID, "sf_cell_sort_noalloc: kernel_radius must be > 0");
    for (int k = 0; k < 3; ++k)
        if (grid->grid_size[k] <= 0) return failWith(SF_ERR_INVALID, "sf_cell_sort_noalloc: grid_size must be positive");
    const int64_t cells = int64_t(grid->grid_size[0]) * grid->grid_size[1] * grid->grid_size[2];
    if (cells > (int64_t(1) << 30)) return failWith(SF_ERR_INVALID, "sf_cell_sort_noalloc: grid above 2^30 cells");
    if (size_t(sortTiles(kMaxN)) * 256 > kHistWords)
        return failWith(SF_ERR_UNSUPPORTED, "sf_cell_sort_noalloc: histogram scratch too small for the sort tiles");
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return failWith(SF_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    std::string why;
    Scratch scratch;
    if (!scratchOf(device, scratch, why)) return failWith(SF_ERR_CUDA, "sf_cell_sort_noalloc: " + why);
    unsigned int* base = scratch.words;
    volatile Report* report = scratch.report;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int ncell = int(cells);
    if (n == 0) {
        e = cudaMemsetAsync(cell_start_out_dev, 0, sizeof(int32_t) * (size_t(ncell) + 1), s);
        return e == cudaSuccess ? SF_OK : failWith(SF_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    }
    // grid of the sort stage (the cell fields of the scene description)
    SceneDev S{};
    S.lpx = grid->lowest_point[0];
    S.lpy = grid->lowest_point[1];
    S.lpz = grid->lowest_point[2];
    S.cell = grid->kernel_radius;
    S.gx = grid->grid_size[0];
    S.gy = grid->grid_size[1];
    S.gz = grid->grid_size[2];
    S.ncell = ncell;
    unsigned int* table = reinterpret_cast<unsigned int*>(cell_start_out_dev);
    const int blocks = int((n + kThreads - 1) / kThreads);
    report->nonFinite = report->crowded = 0u;
    bool done = false;
    if (useCountingSort(int(n), ncell)) {
        uint2* keyRank = reinterpret_cast<uint2*>(base);
        unsigned int *arrived = base + 2 * size_t(kMaxN), *tileSum = base + 3 * size_t(kMaxN);
        const int shift = countTileShift(ncell), tiles = ((ncell - 1) >> shift) + 1;
        if ((e = cudaMemsetAsync(table, 0, sizeof(int32_t) * size_t(ncell), s)) != cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
        kNoAllocCount<<<blocks, kThreads, 0, s>>>(S, pos_dev, int(n), table, keyRank, scratch.reportOnDevice);
        kNoAllocScan<<<tiles, kThreads, 0, s>>>(table, ncell, shift, tileSum);
        kNoAllocAddTiles<<<tiles, kThreads, 0, s>>>(table, ncell, int(n), shift, tileSum);
        kNoAllocScatter<<<blocks, kThreads, 0, s>>>(int(n), table, keyRank, arrived);
        kNoAllocOrder<<<blocks, kThreads, 0, s>>>(int(n), table, keyRank, arrived, perm_out_dev,
                                                  scratch.reportOnDevice);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("sf_cell_sort_noalloc launch: ") + cudaGetErrorString(e));
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("sf_cell_sort_noalloc sync: ") + cudaGetErrorString(e));
        done = report->crowded == 0u || report->nonFinite != 0u;
    }
    if (!done) {
        unsigned int* keys = base;
        SortScratch sc{};
        sc.keysAlt = keys + kMaxN;
        sc.vals = keys + 2 * size_t(kMaxN);
        sc.valsAlt = keys + 3 * size_t(kMaxN);
        sc.digitTotal = keys + 4 * size_t(kMaxN);
        sc.hist = sc.digitTotal + 256;
        sc.tiles = sortTiles(int(n));
        int bits = 1;
        while ((int64_t(1) << bits) <= int64_t(ncell)) ++bits;
        kNoAllocKeys<<<blocks, kThreads, 0, s>>>(S, pos_dev, int(n), keys, scratch.reportOnDevice);
        unsigned int *sortedKeys = nullptr, *perm = nullptr;
        radixSort(s, int(n), bits, keys, sc, &sortedKeys, &perm);
        launchCellStart(s, int(n), ncell, sortedKeys, table);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("sf_cell_sort_noalloc launch: ") + cudaGetErrorString(e));
        if ((e = cudaMemcpyAsync(perm_out_dev, perm, sizeof(int32_t) * size_t(n), cudaMemcpyDeviceToDevice, s)) !=
            cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("permutation copy: ") + cudaGetErrorString(e));
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess)
            return failWith(SF_ERR_CUDA, std::string("sf_cell_sort_noalloc sync: ") + cudaGetErrorString(e));
    }
    if (report->nonFinite) return failWith(SF_ERR_DEVICE, "sf_cell_sort_noalloc: non-finite particle position");
    return SF_OK;
}
