// noalloc_sort.cu — the spatial sort's stable counting sort by bin cell,
// for callers that cannot allocate device memory.
//
// Some hosts fix all device memory up front: a serving loop that admits
// systems against a planned HBM budget, or an embedding application whose
// allocator owns the whole device and forbids allocation once stepping has
// started (a cudaMalloc/cudaFree there would also synchronise the device and
// stall every other stream).  soil_bin_sort_noalloc gives them the same
// permutation as the spatial sort of soil_phase_sort without allocating:
// the caller passes positions, the per-atom cell output and the permutation
// output; the cell histogram, its scan and the scan's tile sums live in one
// file-scope device array of fixed size (kNoAllocScratchWords u32, 16 MiB),
// which every GPU that loads this library keeps until the process exits.
//
// The scratch is shared by every call on a device and keeps the previous
// call's contents; each call clears the histogram it uses before counting.
// Calls whose work overlaps on the GPU (two streams, or two host threads)
// race on that array and must be serialised by the caller.
#include <cstdio>
#include <cstring>

#include "device_ops.cuh"
#include "kernels.cuh"

struct soil_ctx;  // defined in soil_capi.cu

namespace soil {
int set_ctx_error(soil_ctx* ctx, int status, const char* msg);
}

namespace {

using namespace soil;

// Largest bin grid served: 2^21 = 2,097,152 cells.  The 32,768-atom box
// (41^3 cells), the 1,048,576-atom sheared box (~107^3) and every batched or
// served box fit; the 4,194,304-atom box at its default grid (133^3 cells)
// does not and gets SOIL_ERR_CAPACITY.
constexpr uint64_t kNoAllocMaxCells = 1ull << 21;
// histogram/cursor (cells+1) + scan output (cells+2) + scan tile sums
constexpr uint64_t kNoAllocScratchWords =
    (kNoAllocMaxCells + 1) + (kNoAllocMaxCells + 2) + (kNoAllocMaxCells / 2048 + 2);

static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocScratchWords];

// The positions come in the caller's order; unless that is nearly the sorted one,
// neighbouring threads rarely share a cell and an atomic per atom is the cost of a
// pass.  One such pass does: an atom's count on arrival is its place among its
// cell's atoms, kept in the bits of d_cell above the cell number until the scatter
// has used it (the few atoms that arrive in a cell after kLatePlace others take
// their places from the cell's final count instead).  On 2,000,003 atoms: 20 + 18
// us against 21 + 6 + 26 for counting, a copy of the starts and a scatter with
// atomics of its own; the rest is the rate of random accesses (four atoms in
// flight per thread are slower: 71 us a call against 68).
constexpr uint32_t kCellBits = 21;  // kNoAllocMaxCells cells
constexpr uint32_t kCellMask = (1u << kCellBits) - 1;
constexpr uint32_t kLatePlace = (1u << (32 - kCellBits)) - 1;
static_assert(kNoAllocMaxCells <= 1ull << kCellBits, "cells fit their bits");

// Lanes that share their cell with the next one from which a warp counts with one
// atomic per cell: in cells of a few atoms it makes little difference (45 against
// 43 us a call on 2,000,000 sorted atoms, 4 per cell), in crowded ones the lanes
// wait for one another's atomics (117 against 136 with 30 per cell).
constexpr int kAlikeLanes = 16;

__global__ void __launch_bounds__(kBlock) k_noalloc_cells(uint64_t n, const double* x,
                                                          const double* y, const double* z,
                                                          Grid gr, uint32_t* cell,
                                                          uint32_t* counts) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
        const uint64_t i = i0 + threadIdx.x;
        const bool valid = i < n;
        const uint32_t c = valid ? cell_of(gr, x[i], y[i], z[i]) : 0xffffffffu;
        const uint32_t next = __shfl_down_sync(kAll, c, 1);
        uint32_t place = 0;
        if (__popc(__ballot_sync(kAll, valid && lane < 31u && c == next)) >= kAlikeLanes) {
            const unsigned peers = __match_any_sync(kAll, c);
            const int leader = __ffs(peers) - 1;
            if (valid && (int)lane == leader) place = atomicAdd(&counts[c], (uint32_t)__popc(peers));
            place = __shfl_sync(kAll, place, leader) + __popc(peers & ((1u << lane) - 1u));
        } else if (valid) {
            place = atomicAdd(&counts[c], 1u);
        }
        if (valid) cell[i] = c | min(place, kLatePlace) << kCellBits;
    }
}

__global__ void __launch_bounds__(kBlock) k_noalloc_scatter(uint64_t n, const uint32_t* start,
                                                            uint32_t* cell, uint32_t* counts,
                                                            uint32_t* out) {
    // The wait alone: the segment sort starts when this kernel has completed.
    // Released earlier, its few CTAs pile up on the SMs that free up first, and
    // with many atoms per cell each is a long serial sort (131 against 89 us a call
    // on 2,000,000 atoms, 30 per cell).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = cell[i], c = v & kCellMask;
        uint32_t place = v >> kCellBits;
        if (place == kLatePlace) place = atomicSub(&counts[c], 1u) - 1u;
        out[start[c] + place] = (uint32_t)i;
        cell[i] = c;
    }
}

// Device address of g_noalloc_scratch on the current device.  The host-side
// name of the array is only a stand-in for the symbol, not a device address.
// The address is looked up on every call (the lookup is cheap), so a module
// reloaded after cudaDeviceReset is never reached through a stale pointer.
int scratch_for_current_device(soil_ctx* ctx, uint32_t** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0) {
        cudaGetLastError();
        return set_ctx_error(ctx, SOIL_ERR_NO_DEVICE, "soil_bin_sort_noalloc: no current CUDA device");
    }
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
        cudaGetLastError();
        char buf[160];
        snprintf(buf, sizeof buf, "soil_bin_sort_noalloc: cudaGetSymbolAddress failed: %s",
                 cudaGetErrorString(e));
        return set_ctx_error(ctx, SOIL_ERR_CUDA, buf);
    }
    *out = (uint32_t*)p;
    return SOIL_OK;
}

}  // namespace

extern "C" int soil_bin_sort_noalloc(soil_ctx* ctx, const double* d_x, const double* d_y,
                                     const double* d_z, uint64_t n, const double origin[3],
                                     const double bin_size[3], const int32_t bin_count[3],
                                     const double box_lo[3], const double box_size[3],
                                     const double tilt[3], int32_t triclinic, uint32_t* d_cell,
                                     uint32_t* d_perm, void* stream) {
    if (!origin || !bin_size || !bin_count || !box_lo || !box_size || !tilt)
        return set_ctx_error(ctx, SOIL_ERR_INVALID, "soil_bin_sort_noalloc: null grid argument");
    if (n && (!d_x || !d_y || !d_z || !d_cell || !d_perm))
        return set_ctx_error(ctx, SOIL_ERR_INVALID, "soil_bin_sort_noalloc: null device pointer");
    for (int d = 0; d < 3; ++d)
        if (bin_count[d] < 1 || !(bin_size[d] > 0.0) || !(box_size[d] > 0.0))
            return set_ctx_error(ctx, SOIL_ERR_INVALID, "soil_bin_sort_noalloc: invalid bin grid");
    // the product is built factor by factor and stops past the limit, so
    // counts whose 64-bit product would wrap are refused too
    uint64_t ncells = 1;
    for (int d = 0; d < 3 && ncells <= kNoAllocMaxCells; ++d) ncells *= (uint64_t)bin_count[d];
    if (ncells > kNoAllocMaxCells) {
        char buf[200];
        snprintf(buf, sizeof buf,
                 "soil_bin_sort_noalloc: %llu bin cells exceed the fixed scratch limit of %llu "
                 "cells; use soil_phase_sort (which allocates) for this grid",
                 (unsigned long long)ncells, (unsigned long long)kNoAllocMaxCells);
        return set_ctx_error(ctx, SOIL_ERR_CAPACITY, buf);
    }
    if (n >= 0x7fffffffull)
        return set_ctx_error(ctx, SOIL_ERR_CAPACITY, "soil_bin_sort_noalloc: n exceeds the u32 index range");
    uint32_t* scratch = nullptr;
    int r = scratch_for_current_device(ctx, &scratch);
    if (r != SOIL_OK) return r;
    if (n == 0) return SOIL_OK;

    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* counts = scratch;                      // histogram
    uint32_t* start = scratch + (kNoAllocMaxCells + 1);
    uint32_t* partials = start + (kNoAllocMaxCells + 2);

    Grid gr;
    for (int d = 0; d < 3; ++d) {
        gr.origin[d] = origin[d];
        gr.inv_bs[d] = 1.0 / bin_size[d];
        gr.n[d] = bin_count[d];
        gr.geom.lo[d] = box_lo[d];
        gr.geom.size[d] = box_size[d];
        gr.geom.tilt[d] = tilt[d];
    }
    gr.geom.triclinic = triclinic ? 1 : 0;
    cudaError_t e = cudaMemsetAsync(counts, 0, ncells * sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        note_launch();
        k_noalloc_cells<<<grid_wave<k_noalloc_cells>(n), kBlock, 0, st>>>(n, d_x, d_y, d_z, gr,
                                                                          d_cell, counts);
        exclusive_scan_u32(st, counts, start, ncells, partials);
        note_launch();
        pdl_launch(k_noalloc_scatter, grid_wave<k_noalloc_scatter>(n), kBlock, 0, st, n, start,
                   d_cell, counts, d_perm);
        launch_segsort(st, ncells, start, d_perm);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        char buf[200];
        snprintf(buf, sizeof buf, "soil_bin_sort_noalloc: %s", cudaGetErrorString(e));
        return set_ctx_error(ctx, SOIL_ERR_CUDA, buf);
    }
    return SOIL_OK;
}
