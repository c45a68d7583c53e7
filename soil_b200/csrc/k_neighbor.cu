// k_neighbor.cu — half-list CSR build of bin_neighbor_list
// (neighbor.rs:1127-1319) and the transposed ("incoming") lists the
// deterministic force gather reads.
//
// Row order is the reference's: the self-cell tail (sorted slots after the
// atom's own slot), then every forward-stencil cell in stencil order, each
// cell in sorted (ascending index) order.
//
// Pass 1 (k_pairs_rows): one thread per local row scans its candidates in
// that order, keeps the first K accepted indices in fixed per-row slots and
// records the row length.  An exclusive scan of the lengths gives
// neighbor_offsets; pass 2 (k_pairs_fill) copies every row into place and
// re-derives, sequentially and in the same order, the rare rows longer than
// K.  (A warp-per-cell variant with ballot compaction was measured slower:
// one dependent-load chain per warp, no overlap across rows.)
//
// Candidates are read as one 32-byte record {x, y, z, cutoff} per sorted slot
// (sorted_pos of the reference plus the cutoff radius of the polydisperse
// test).  Filter: FP64 `fma(dx,dx,fma(dy,dy,dz*dz)) < cut^2` exactly as the
// reference, or (FP32 mode) a float test on grid-relative coordinates that
// only REJECTS candidates provably outside the cutoff — the margin eps bounds
// the float rounding of coordinates, differences and squares — followed by
// the exact FP64 test on the rest, so the lists are identical in both modes.
#include "device_ops.cuh"
#include "kernels.cuh"

namespace soil {

// The block's filter statistics, then one atomic per counter and block (the
// FP64 filter rechecks nothing).
template <bool FP32>
__device__ __forceinline__ void add_block_stats(DevFlags* flags, uint64_t n_cand, uint64_t r) {
    __shared__ unsigned long long s_cand, s_rechk;
    if (threadIdx.x == 0) {
        s_cand = 0;
        s_rechk = 0;
    }
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) {
        n_cand += __shfl_down_sync(0xffffffffu, n_cand, o);
        r += __shfl_down_sync(0xffffffffu, r, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_cand, (unsigned long long)n_cand);
        if (FP32) atomicAdd(&s_rechk, (unsigned long long)r);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd((unsigned long long*)&flags->candidates, s_cand);
        if (FP32) atomicAdd((unsigned long long*)&flags->rechecked, s_rechk);
    }
}

// Pass 1: one thread per local row (rows of a warp are neighbours in space, so
// their candidate records are shared through L1); the first K entries go to
// the row's slots, the length to rowcount.
template <bool UNIFORM, bool FP32, int U, int NR>
__global__ void __launch_bounds__(kBlock) k_pairs_rows(PairParams p, uint32_t* rowcount,
                                                       uint32_t* slots, DevFlags* flags) {
    pdl_wait();  // launched with pdl_launch
    const Filter<UNIFORM, FP32> test(p);
    const uint32_t K = (uint32_t)p.row_slots;
    uint32_t n_rechk = 0, n_cand32 = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < p.nlocal;
         i += (uint64_t)gridDim.x * blockDim.x)
        rowcount[i] = row_scan<UNIFORM, FP32, true, U, NR>(p, test, i, slots + i * K, K, &n_rechk,
                                                           &n_cand32, flags, p.in_count);
    add_block_stats<FP32>(flags, n_cand32, n_rechk);
}

// Pass 1 of a system with too few rows to fill the chip with one thread each:
// G lanes per row.  What bounds it is the chain of a row's candidates through
// L2, G times shorter here.
template <int G, bool UNIFORM, bool FP32, int NR>
__global__ void __launch_bounds__(kBlock) k_pairs_group(PairParams p, uint32_t* rowcount,
                                                        uint32_t* slots, DevFlags* flags) {
    pdl_wait();  // launched with pdl_launch
    const Filter<UNIFORM, FP32> test(p);
    const uint32_t K = (uint32_t)p.row_slots;
    const uint32_t g = threadIdx.x & (G - 1);
    uint32_t n_rechk = 0, n_cand32 = 0;
    const uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / G;
    const bool valid = i < p.nlocal;
    const uint32_t cnt = row_scan_group<G, UNIFORM, FP32, NR>(p, test, i, valid, g, slots + i * K,
                                                              K, &n_rechk, &n_cand32, flags,
                                                              p.in_count);
    if (valid && g == 0) rowcount[i] = cnt;
    add_block_stats<FP32>(flags, n_cand32, n_rechk);
}

// Pass 2: rows into their CSR place; rows longer than K are re-derived.
template <bool UNIFORM, bool FP32>
__global__ void __launch_bounds__(kBlock) k_pairs_fill(PairParams p, const uint32_t* rowcount,
                                                       const uint32_t* slots,
                                                       const uint32_t* offsets, uint32_t* indices,
                                                       FillGuard g) {
    pdl_wait();  // launched with pdl_launch
    guard_publish(g);
    if (!guard_open(g)) return;
    const Filter<UNIFORM, FP32> test(p);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < p.nlocal;
         i += (uint64_t)gridDim.x * blockDim.x) {
        fill_row<UNIFORM, FP32>(p, test, i, rowcount, slots, offsets, indices);
    }
}

// Pass 2 by kFillLanes lanes per row, for systems whose rows do not fill the
// chip with one thread each: what bounds it is the chain of a row's entries
// through L2, four at a time with one thread.
constexpr int kFillLanes = 8;
template <bool UNIFORM, bool FP32>
__global__ void __launch_bounds__(kBlock) k_pairs_fill_group(PairParams p, const uint32_t* rowcount,
                                                             const uint32_t* slots,
                                                             const uint32_t* offsets,
                                                             uint32_t* indices, FillGuard g) {
    pdl_wait();  // launched with pdl_launch
    guard_publish(g);
    if (!guard_open(g)) return;
    const Filter<UNIFORM, FP32> test(p);
    const uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / kFillLanes;
    if (i < p.nlocal)
        fill_row_group<kFillLanes>(p, test, i, threadIdx.x % kFillLanes, rowcount, slots, offsets,
                                   indices);
}
// Up to 65,536 rows (with 1 / 8 lanes: 5.9 / 3.8 us on 1,000 rows, 6.9 / 3.8 on
// 8,009, 8.5 / 7.4 on 50,021, 13.9 / 19.8 on 200,003).
constexpr uint64_t kFillGroupRows = 65536;

// Pass 1's form.  8 lanes per row up to 12,288 rows, 4 up to 36,864 (measured
// with 1 / 4 / 8 lanes: 12.2 / 7.1 / 5.8 us on 8,009 rows, 13.4 / 8.3 / 11.5 on
// 24,001, 13.9 / 14.5 / 16.7 on 50,021).  Above, one thread per row: two
// candidates at a time where the cells hold enough atoms, else one.  With one /
// two at a time a whole sheared step of 1,048,576 equal spheres takes 324 / 330
// us at 0.23 atoms per cell, 381 / 385 at 0.89, 399 / 401 at 1.13, 440 / 438 at 1.32.
constexpr uint64_t kRows8Lanes = 12288, kRows4Lanes = 36864;
constexpr double kTwoAtATime = 1.25;  // mean atoms per cell

template <bool UNIFORM, bool FP32, int NR>
static void launch_rows_t(cudaStream_t st, const PairParams& p, uint32_t* rowcount,
                          uint32_t* slots, DevFlags* flags) {
    const bool pre = p.pre_ranges && p.nstencil < NR;  // never for NR = 0 (long stencils)
    const int g = !pre ? 1 : p.nlocal <= kRows8Lanes ? 8 : p.nlocal <= kRows4Lanes ? 4 : 1;
    const unsigned blocks = (unsigned)((p.nlocal * (uint64_t)g + kBlock - 1) / kBlock);
    auto launch = [&](auto k, unsigned grid) {
        pdl_launch(k, grid, kBlock, 0, st, p, rowcount, slots, flags);
    };
    if constexpr (NR > 0) {
        if (g == 8) return launch(k_pairs_group<8, UNIFORM, FP32, NR>, blocks);
        if (g == 4) return launch(k_pairs_group<4, UNIFORM, FP32, NR>, blocks);
    }
    if (p.cell_atoms >= kTwoAtATime)
        launch(k_pairs_rows<UNIFORM, FP32, 2, NR>, grid_wave<k_pairs_rows<UNIFORM, FP32, 2, NR>>(p.nlocal));
    else
        launch(k_pairs_rows<UNIFORM, FP32, 1, NR>, grid_wave<k_pairs_rows<UNIFORM, FP32, 1, NR>>(p.nlocal));
}

template <bool UNIFORM, bool FP32>
static void launch_pairs_t(cudaStream_t st, const PairParams& p, uint32_t* rowcount,
                           uint32_t* slots, const uint32_t* offsets, uint32_t* indices,
                           DevFlags* flags, const FillGuard* g) {
    note_launch();
    if (!g && p.nstencil < kPreRanges)
        launch_rows_t<UNIFORM, FP32, kPreRanges>(st, p, rowcount, slots, flags);
    else if (!g && p.nstencil < kPreRangesFull)
        launch_rows_t<UNIFORM, FP32, kPreRangesFull>(st, p, rowcount, slots, flags);
    else if (!g)
        launch_rows_t<UNIFORM, FP32, 0>(st, p, rowcount, slots, flags);
    else if (p.nlocal <= kFillGroupRows)
        pdl_launch(k_pairs_fill_group<UNIFORM, FP32>,
                   (unsigned)((p.nlocal * kFillLanes + kBlock - 1) / kBlock), kBlock, 0, st, p,
                   rowcount, slots, offsets, indices, *g);
    else
        pdl_launch(k_pairs_fill<UNIFORM, FP32>, grid_wave<k_pairs_fill<UNIFORM, FP32>>(p.nlocal), kBlock, 0, st, p, rowcount, slots,
                                                                            offsets, indices, *g);
}

// g == nullptr: pass 1; else pass 2 under guard *g
static void dispatch_pairs(cudaStream_t st, const PairParams& p, uint32_t* rowcount,
                           uint32_t* slots, const uint32_t* offsets, uint32_t* indices,
                           DevFlags* flags, const FillGuard* g) {
    const bool fp32 = p.filter == SOIL_FILTER_FP32_RECHECK;
    if (p.uniform) {
        if (fp32) launch_pairs_t<true, true>(st, p, rowcount, slots, offsets, indices, flags, g);
        else launch_pairs_t<true, false>(st, p, rowcount, slots, offsets, indices, flags, g);
    } else {
        if (fp32) launch_pairs_t<false, true>(st, p, rowcount, slots, offsets, indices, flags, g);
        else launch_pairs_t<false, false>(st, p, rowcount, slots, offsets, indices, flags, g);
    }
}

void launch_pair_count(cudaStream_t st, const PairParams& p, uint32_t* rowcount, uint32_t* slots,
                       DevFlags* flags) {
    if (p.nlocal == 0 || p.ncells == 0) return;
    dispatch_pairs(st, p, rowcount, slots, nullptr, nullptr, flags, nullptr);
}

void launch_pair_fill(cudaStream_t st, const PairParams& p, const uint32_t* rowcount,
                      const uint32_t* slots, const uint32_t* offsets, uint32_t* indices,
                      const FillGuard& g) {
    if (p.nlocal == 0) return;
    dispatch_pairs(st, p, const_cast<uint32_t*>(rowcount), const_cast<uint32_t*>(slots), offsets,
                   indices, nullptr, &g);
}

__global__ void __launch_bounds__(kBlock) k_in_count(uint64_t nlocal, const uint32_t* offsets,
                                                     const uint32_t* indices, uint32_t* incount) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlocal;
         i += (uint64_t)gridDim.x * blockDim.x)
        for (uint32_t q = offsets[i]; q < offsets[i + 1]; ++q) atomicAdd(&incount[indices[q]], 1u);
}

void launch_in_count(cudaStream_t st, uint64_t nlocal, const uint32_t* offsets,
                     const uint32_t* indices, uint32_t* incount) {
    if (nlocal == 0) return;
    note_launch();
    k_in_count<<<grid_wave<k_in_count>(nlocal), kBlock, 0, st>>>(nlocal, offsets, indices, incount);
}

__global__ void __launch_bounds__(kBlock) k_in_scatter(uint64_t nlocal, const uint32_t* offsets,
                                                       const uint32_t* indices, uint32_t* cursor,
                                                       uint32_t* in_list) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlocal;
         i += (uint64_t)gridDim.x * blockDim.x)
        for (uint32_t q = offsets[i]; q < offsets[i + 1]; ++q)
            in_list[atomicAdd(&cursor[indices[q]], 1u)] = (uint32_t)i;
}

void launch_in_scatter(cudaStream_t st, uint64_t nlocal, const uint32_t* offsets,
                       const uint32_t* indices, uint32_t* cursor, uint32_t* in_list) {
    if (nlocal == 0) return;
    note_launch();
    k_in_scatter<<<grid_wave<k_in_scatter>(nlocal), kBlock, 0, st>>>(nlocal, offsets, indices, cursor, in_list);
}

}  // namespace soil
