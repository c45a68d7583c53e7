// k_force.cu — the built-in pair consumer: linear repulsion
// f = k*overlap along the line of centres, the tutorial's
// soft_repulsion_force (docs/src/tutorial/write-your-own-physics.md:56-110).
//
// The reference accumulates pair forces in global pair order: for pair
// (i, j) it adds +f to i and -f to j, rows ascending, CSR order inside a row.
// So atom a receives, in order, -f(i,a) from every earlier row i that lists
// a (ascending i), then +f(a,j) for its own row, then (full lists only) -f
// from later rows.
//
// These kernels reproduce that sum bit for bit:
//
//  k_force_csr  the default: one thread per local root walks its and its
//               images' transposed lists and rows (8 lanes per root on small
//               systems, k_force_group, and for roots with several images),
//               then folds; k_force_step also ends the step and begins the
//               next one.
//
//  k_harmonic   one thread per atom walks the CSR and its transpose
//               (harmonic_atom), with a reverse pass of its own
//               (SOIL_FORCE=gather).
//
//  k_force_seq  (SOIL_FORCE=tiles2, tiles4) at every rebuild each atom's
//               contributions are merged into one partner sequence in the
//               reference's order (k_seq_fill).  IEEE negation is exact, so
//               f(i,j) = -f(j,i) bit for bit (d -> -d flips the sign of every
//               factor that carries it; every other factor is symmetric) and
//               F - f(i,a) is F + f(a,i): each entry is evaluated as
//               f(a, partner) and added.  The sequences are grouped by local
//               root: root t's sequence, then those of its ghost images in
//               reverse-comm fold order.  A warp takes 32 consecutive roots
//               and spreads the union of their groups over its lanes in
//               chunks (every lane busy, U independent gathers in flight per
//               lane); pair forces go to shared memory, and each lane then
//               adds its own group's entries in order, writes the forces of
//               its root and images and, with FOLD, folds the images into the
//               root exactly as reverse_send_force does (fold_root), so
//               reverse comm needs no pass of its own (force_ops.cuh).
#include <cstdlib>
#include <cstring>

#include "device_ops.cuh"
#include "force_ops.cuh"
#include "kernels.cuh"

namespace soil {

__global__ void __launch_bounds__(kBlock, 5) k_harmonic(uint64_t nlocal, uint64_t ntotal, AtomCols c,
                                                     const double* rad, double K, int newton,
                                                     const uint32_t* offsets,
                                                     const uint32_t* indices,
                                                     const uint32_t* in_start,
                                                     const uint32_t* in_list) {
    for (uint64_t a = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; a < ntotal;
         a += (uint64_t)gridDim.x * blockDim.x)
        harmonic_atom(c, a, nlocal, rad, K, newton, offsets, indices, in_start, in_list);
}

void launch_harmonic(cudaStream_t st, uint64_t nlocal, uint64_t ntotal, const AtomCols& c,
                     const double* radius, double k, int newton, const uint32_t* offsets,
                     const uint32_t* indices, const uint32_t* in_start, const uint32_t* in_list) {
    if (ntotal == 0) return;
    note_launch();
    // one resident wave (5 blocks of 256 per SM at <= 48 registers), grid-stride
    const unsigned full = 148u * 5u;
    const unsigned need = (unsigned)((ntotal + kBlock - 1) / kBlock);
    k_harmonic<<<need < full ? need : full, kBlock, 0, st>>>(nlocal, ntotal, c, radius, k, newton,
                                                              offsets, indices, in_start, in_list);
}

// ---- the grouped partner sequences (rebuilt with the lists) ----------------

__global__ void __launch_bounds__(kBlock) k_seq_count(SeqArgs q, uint32_t* cnt, uint32_t* grp) {
    for (uint64_t a = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; a < q.ntotal;
         a += (uint64_t)gridDim.x * blockDim.x)
        seq_count_atom(q, a, cnt, grp);
}

__global__ void __launch_bounds__(kBlock) k_seq_fill(SeqArgs q, const uint32_t* grp_start,
                                                     uint32_t* seq, uint8_t* owner) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < q.nlocal;
         t += (uint64_t)gridDim.x * blockDim.x)
        seq_fill_root(q, t, grp_start, seq, owner);
}

void launch_seq_count(cudaStream_t st, const SeqArgs& q, uint32_t* cnt, uint32_t* grp) {
    if (q.ntotal == 0) return;
    note_launch();
    k_seq_count<<<grid_wave<k_seq_count>(q.ntotal), kBlock, 0, st>>>(q, cnt, grp);
}

void launch_seq_fill(cudaStream_t st, const SeqArgs& q, const uint32_t* grp_start, uint32_t* seq,
                     uint8_t* owner) {
    if (q.nlocal == 0) return;
    note_launch();
    k_seq_fill<<<grid_wave<k_seq_fill>(q.nlocal), kBlock, 0, st>>>(q, grp_start, seq, owner);
}

// ---- the warp-cooperative consumer, one launch --------------------------------

template <int U, bool FOLD>
__global__ void __launch_bounds__(kBlock, 4) k_force_seq(ForceArgs p) {
    __shared__ ForceSmem<U> sm;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t ntiles = (p.q.nlocal + 31) / 32;
    for (uint64_t w = (uint64_t)blockIdx.x * kForceWarps + wib; w < ntiles;
         w += (uint64_t)gridDim.x * kForceWarps)
        force_tile<U, FOLD>(p.q, p.c, p.rev, w, sm, lane, wib);
}

// PK: partner records from the packed copy (p.q.pk / q.pk set).
template <bool FOLD, bool PK>
__global__ void __launch_bounds__(kBlock, 4) k_force_walk(ForceArgs p) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < p.q.nlocal;
         t += (uint64_t)gridDim.x * blockDim.x)
        force_walk_root<FOLD, PK>(p.q, p.c, p.rev, t);
}

// SORT: right after a neighbor build, whose transposed lists are unordered.  An
// atom's in-list is read by its root's walk alone, so the walk sorts it: one
// launch less, and the list is in the caches.  With k_segsort_split before it,
// 60 + 13 against 69 us on 1,048,576 sheared atoms, 18.4 + 6.1 against 22.1 on
// 200,003; k_force_group on 8,009 atoms 5.5 + 2.7 against 6.3.
template <bool FOLD, bool PK, bool SORT>
__global__ void __launch_bounds__(kBlock, 4) k_force_csr(ForceCsr q, AtomCols c, PlaneList rev,
                                                         const uint32_t* trip, FillGuard guard) {
    pdl_wait();  // launched with pdl_launch
    if (trip && *trip) return;  // the step rebuilds: its forces come later
    if (!guard_open(guard)) return;
    if (q.multi) {
        // The roots with two images or more (edges and corners of the box) by 8
        // lanes each, spread from the last block on (the first ones may have
        // one block of roots more); every other root and its image, if it has
        // one, by its thread below.  A corner root's eight items in series on
        // one thread set the kernel's time on systems of a few waves: 20.2
        // against 16.5 us on 200,003 atoms, 41.1 against 39.4 on 600,011.
        const uint64_t n = *q.nmulti;
        const uint64_t warp = (uint64_t)(gridDim.x - 1 - blockIdx.x) * (kBlock / 32) + threadIdx.x / 32;
        for (uint64_t k = warp * 4; k < n; k += (uint64_t)gridDim.x * (kBlock / 32) * 4) {
            const uint64_t at = k + (threadIdx.x & 31) / 8;
            force_group_root<FOLD, SORT>(q, c, rev, at < n ? q.multi[at] : 0, at < n);
        }
        for (uint64_t t = (uint64_t)blockIdx.x * kBlock + threadIdx.x; t < q.nlocal;
             t += (uint64_t)gridDim.x * kBlock)
            if (q.fold_start[t + 1] - q.fold_start[t] < 2)
                force_csr_root<FOLD, PK, SORT>(q, c, rev, t);
        return;
    }
    // grid-stride over whole blocks of kBlock roots, so a block's order
    // permutes its own roots
    for (uint64_t b = (uint64_t)blockIdx.x * kBlock; b < q.nlocal; b += (uint64_t)gridDim.x * kBlock) {
        const uint64_t k = b + threadIdx.x;
        if (k < q.nlocal) force_csr_root<FOLD, PK, SORT>(q, c, rev, q.order ? q.order[k] : k);
    }
}

// k_force_csr of a step inside a stretch, then each root's half-kicks, its next
// position and those of its images.  The walk is bound by its instructions and
// the latency of its gathers, the integration pass by memory bandwidth, so as
// one launch they overlap, and the forces just summed need no second read: a
// step on 4,194,304 atoms 234 us against 208 + 93 + 10 for the three launches,
// on 200,003 atoms 20.7 against 16.5 + 4.2 + 3.7.
__global__ void __launch_bounds__(kBlock, 4) k_force_step(ForceCsr q, AtomCols c, ForceStep p) {
    pdl_wait();  // launched with pdl_launch
    const unsigned long long w = *(volatile unsigned long long*)p.word;
    const bool head = p.head && *p.head;
    const bool skip = head || (w >= p.first && w <= p.number);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (head) *(volatile unsigned long long*)p.word = p.number;
        *(volatile uint32_t*)p.answer = (uint32_t)(2 * p.number) | (skip ? 1u : 0u);
    }
    if (skip) return;
    constexpr unsigned kAll = 0xffffffffu;
    const PlaneList none{};
    bool hit = false;
    {  // as in k_force_csr
        const uint64_t n = *q.nmulti;
        const uint64_t warp = (uint64_t)(gridDim.x - 1 - blockIdx.x) * (kBlock / 32) + threadIdx.x / 32;
        for (uint64_t k = warp * 4; k < n; k += (uint64_t)gridDim.x * (kBlock / 32) * 4) {
            const uint64_t at = k + (threadIdx.x & 31) / 8;
            const GroupItem it =
                force_group_root<true>(q, c, none, at < n ? q.multi[at] : 0, at < n);
            const bool root = it.mine && (threadIdx.x & 7) == 0;
            double x = it.x, y = it.y, z = it.z, vx = 0.0, vy = 0.0, vz = 0.0;
            if (root) hit |= step_local(p, c, it.a, it.Fx, it.Fy, it.Fz, x, y, z, vx, vy, vz);
            x = __shfl_sync(kAll, x, 0, 8);
            y = __shfl_sync(kAll, y, 0, 8);
            z = __shfl_sync(kAll, z, 0, 8);
            vx = __shfl_sync(kAll, vx, 0, 8);
            vy = __shfl_sync(kAll, vy, 0, 8);
            vz = __shfl_sync(kAll, vz, 0, 8);
            if (it.mine && !root) step_image(p, c, q.nlocal, it.gi, x, y, z, vx, vy, vz);
        }
    }
    const ColLd ld{c.x, c.y, c.z, q.rad};
    for (uint64_t t = (uint64_t)blockIdx.x * kBlock + threadIdx.x; t < q.nlocal;
         t += (uint64_t)gridDim.x * kBlock) {
        const uint32_t f0 = q.fold_start[t], nimg = q.fold_start[t + 1] - f0;
        if (nimg >= 2) continue;
        const uint32_t gi = nimg ? q.fold_list[f0] : 0u;
        double Fx = 0.0, Fy = 0.0, Fz = 0.0, x = 0.0, y = 0.0, z = 0.0;
        for (uint32_t j = 0; j <= nimg; ++j) {  // the root, then its image
            const uint64_t a = j ? q.nlocal + gi : t;
            const double4 pa = ld(a);
            double fx, fy, fz;
            csr_item_force(q, ld, a, pa, fx, fy, fz);
            if (j == 0) {
                Fx = fx;
                Fy = fy;
                Fz = fz;
                x = pa.x;
                y = pa.y;
                z = pa.z;
            } else {  // fold_root
                c.fx[a] = fx;
                c.fy[a] = fy;
                c.fz[a] = fz;
                Fx = Fx + fx;
                Fy = Fy + fy;
                Fz = Fz + fz;
            }
        }
        c.fx[t] = Fx;
        c.fy[t] = Fy;
        c.fz[t] = Fz;
        double vx, vy, vz;
        hit |= step_local(p, c, t, Fx, Fy, Fz, x, y, z, vx, vy, vz);
        if (nimg) step_image(p, c, q.nlocal, gi, x, y, z, vx, vy, vz);
    }
    const unsigned any = __ballot_sync(kAll, hit);
    if (any && (threadIdx.x & 31) == 0) *(volatile unsigned long long*)p.word = p.number + 1;
}

void launch_force_step(cudaStream_t st, const ForceCsr& q, const AtomCols& c, const ForceStep& p) {
    note_launch();
    const unsigned full = 148u * 4u;  // as k_force_csr
    const unsigned need = (unsigned)((q.nlocal + kBlock - 1) / kBlock);
    pdl_launch(k_force_step, need < full ? need : full, kBlock, 0, st, q, c, p);
}

// 8 lanes per root for a system whose roots do not fill the chip with one
// thread each.
template <bool FOLD, bool SORT>
__global__ void __launch_bounds__(kBlock, 4) k_force_group(ForceCsr q, AtomCols c, PlaneList rev,
                                                           const uint32_t* trip, FillGuard guard) {
    pdl_wait();  // launched with pdl_launch
    if (trip && *trip) return;  // the step rebuilds: its forces come later
    if (!guard_open(guard)) return;
    const uint64_t t = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) / 8;
    force_group_root<FOLD, SORT>(q, c, rev, t, t < q.nlocal);
}

// Entries of root t's walk: its and its images' in-lists and its row.
__device__ __forceinline__ uint32_t csr_work(const ForceCsr& q, uint64_t t) {
    uint32_t n = q.offsets[t + 1] - q.offsets[t] + q.in_start[t + 1] - q.in_start[t];
    if (q.newton)
        for (uint32_t f = q.fold_start[t]; f < q.fold_start[t + 1]; ++f) {
            const uint64_t g = q.nlocal + q.fold_list[f];
            n += q.in_start[g + 1] - q.in_start[g];
        }
    return n;
}

// One block per kBlock roots: a bitonic sort of (work, index) keys in
// shared memory.
__global__ void __launch_bounds__(kBlock) k_root_order(ForceCsr q, uint32_t* order) {
    __shared__ uint64_t key[kBlock];
    const uint64_t b = (uint64_t)blockIdx.x * kBlock;
    const uint32_t i = threadIdx.x;
    const uint64_t t = b + i;
    const uint32_t work = t < q.nlocal ? min(csr_work(q, t), 0xffffu) : 0xffffffffu;
    key[i] = ((uint64_t)work << 32) | (uint32_t)i;
    __syncthreads();
    for (uint32_t size = 2; size <= kBlock; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            const uint32_t j = i ^ stride;
            if (j > i) {
                const uint64_t a = key[i], c = key[j];
                const bool up = (i & size) == 0;
                if ((a > c) == up) {
                    key[i] = c;
                    key[j] = a;
                }
            }
            __syncthreads();
        }
    if (t < q.nlocal) order[t] = (uint32_t)(b + (uint32_t)key[i]);
}

void launch_root_order(cudaStream_t st, const ForceCsr& q, uint32_t* order) {
    if (q.nlocal == 0) return;
    note_launch();
    k_root_order<<<(unsigned)((q.nlocal + kBlock - 1) / kBlock), kBlock, 0, st>>>(q, order);
}

void launch_force_csr(cudaStream_t st, const ForceCsr& q0, const AtomCols& c, const PlaneList& rev,
                      bool fold, bool few_images, const uint32_t* trip, const FillGuard* guard) {
    if (q0.nlocal == 0) return;
    note_launch();
    const FillGuard gd = guard ? *guard : FillGuard{};
    ForceCsr q = q0;
    if (q.order) q.multi = nullptr;  // an order of whole blocks of roots
    if (q.nlocal <= kForceGroupRoots && few_images && !q.pk && !q.order) {
        const unsigned blocks = (unsigned)((q.nlocal * 8 + kBlock - 1) / kBlock);
        const auto k = q.unsorted ? (fold ? k_force_group<true, true> : k_force_group<false, true>)
                                  : (fold ? k_force_group<true, false> : k_force_group<false, false>);
        pdl_launch(k, blocks, kBlock, 0, st, q, c, rev, trip, gd);
        return;
    }
    // one resident wave at <= 64 registers, striding over blocks of roots
    // (measured faster than one block per kBlock roots, and than 5 blocks per
    // SM at 48 registers, which spills; and faster than spreading a block's
    // roots and their images over its threads as one item list with the fold
    // after a barrier: 0.287 against 0.251 ms at C2)
    const unsigned full = 148u * 4u;
    const unsigned need = (unsigned)((q.nlocal + kBlock - 1) / kBlock);
    const unsigned grid = need < full ? need : full;
    const auto k = q.pk         ? (fold ? k_force_csr<true, true, false> : k_force_csr<false, true, false>)
                   : q.unsorted ? (fold ? k_force_csr<true, false, true> : k_force_csr<false, false, true>)
                                : (fold ? k_force_csr<true, false, false> : k_force_csr<false, false, false>);
    pdl_launch(k, grid, kBlock, 0, st, q, c, rev, trip, gd);
}

template <int U>
static void launch_tiles(cudaStream_t st, const ForceArgs& p, bool fold) {
    const uint64_t ntiles = (p.q.nlocal + 31) / 32;
    const uint64_t need = (ntiles + kForceWarps - 1) / kForceWarps;
    const uint64_t full = 148ull * 4ull;  // one resident wave, grid-stride over the tiles
    const unsigned grid = (unsigned)(need < full ? need : full);
    if (fold) k_force_seq<U, true><<<grid, kBlock, 0, st>>>(p);
    else k_force_seq<U, false><<<grid, kBlock, 0, st>>>(p);
}

// The consumer kernel (SOIL_FORCE: gather, csr, tiles4, tiles2, walk); read at
// each call so a host can compare them on one system.
int force_variant() {
    const char* env = std::getenv("SOIL_FORCE");
    if (!env) return kDefaultForce;
    if (!std::strcmp(env, "gather")) return SOIL_FORCE_GATHER;
    if (!std::strcmp(env, "tiles4")) return SOIL_FORCE_TILES4;
    if (!std::strcmp(env, "tiles2")) return SOIL_FORCE_TILES2;
    if (!std::strcmp(env, "walk")) return SOIL_FORCE_WALK;
    if (!std::strcmp(env, "csr")) return SOIL_FORCE_CSR;
    return kDefaultForce;
}

void launch_force_seq(cudaStream_t st, const ForceArgs& p, bool fold, int variant) {
    if (p.q.nlocal == 0) return;
    note_launch();
    if (variant == SOIL_FORCE_WALK) {
        const unsigned full = 148u * 4u;  // one resident wave at <= 64 registers
        const unsigned need = (unsigned)((p.q.nlocal + kBlock - 1) / kBlock);
        const unsigned grid = need < full ? need : full;
        if (p.q.pk) {
            if (fold) k_force_walk<true, true><<<grid, kBlock, 0, st>>>(p);
            else k_force_walk<false, true><<<grid, kBlock, 0, st>>>(p);
        } else {
            if (fold) k_force_walk<true, false><<<grid, kBlock, 0, st>>>(p);
            else k_force_walk<false, false><<<grid, kBlock, 0, st>>>(p);
        }
    } else if (variant == SOIL_FORCE_TILES2) {
        launch_tiles<2>(st, p, fold);
    } else {
        launch_tiles<4>(st, p, fold);
    }
}

}  // namespace soil
