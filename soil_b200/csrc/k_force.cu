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
// Two kernels reproduce that sum bit for bit:
//
//  k_harmonic   one thread per atom walks the CSR and its transpose
//               (harmonic_atom); used by the batched engine and by systems
//               whose locals can have more than 7 ghost images.
//
//  k_force_seq  the single-system consumer.  At every rebuild each atom's
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

template <bool FOLD, bool PK>
__global__ void __launch_bounds__(kBlock, 4) k_force_csr(ForceCsr q, AtomCols c, PlaneList rev,
                                                         const uint32_t* trip, FillGuard guard) {
    pdl_wait();  // launched with pdl_launch
    if (trip && *trip) return;  // the step rebuilds: its forces come later
    if (!guard_open(guard)) return;
    // grid-stride over whole blocks of kBlock roots, so a block's order
    // permutes its own roots
    for (uint64_t b = (uint64_t)blockIdx.x * kBlock; b < q.nlocal; b += (uint64_t)gridDim.x * kBlock) {
        const uint64_t k = b + threadIdx.x;
        if (k < q.nlocal) force_csr_root<FOLD, PK>(q, c, rev, q.order ? q.order[k] : k);
    }
}

// The same forces by 8 lanes per root, for systems whose roots do not fill the
// chip with one thread each and whose roots have at most 7 images.  Lane j
// holds item j of the group (0: the root, j: its j-th image in fold order); the
// items' entries are numbered through, 8 evaluated at a time, and every lane
// adds the results in entry order, keeping its own item's sum; the fold moves
// the images' sums to their parents' lanes in fold order.  Same operations in
// the same order as force_csr_root.  What bounds it is one chain of dependent
// loads (fold list, list bounds, entry, partner) instead of one per image.
template <bool FOLD>
__global__ void __launch_bounds__(kBlock, 4) k_force_group(ForceCsr q, AtomCols c, PlaneList rev,
                                                           const uint32_t* trip, FillGuard guard) {
    pdl_wait();  // launched with pdl_launch
    if (trip && *trip) return;  // the step rebuilds: its forces come later
    if (!guard_open(guard)) return;
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t g = threadIdx.x & 7u;
    const uint64_t t = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) / 8;
    const bool valid = t < q.nlocal;
    const uint32_t f0 = valid ? q.fold_start[t] : 0u;
    const uint32_t nimg = valid ? q.fold_start[t + 1] - f0 : 0u;
    // this lane's item
    uint64_t a = t;
    uint32_t gi = 0, qs = 0, nin = 0, npre = 0, rs = 0, nrow = 0, org = 0;
    double4 pa = make_double4(0.0, 0.0, 0.0, 0.0);
    const bool mine = valid && g <= nimg;
    if (mine) {
        if (g) {
            gi = q.fold_list[f0 + g - 1];
            a = q.nlocal + gi;
            org = (uint32_t)c.origin[a];
        }
        if (g == 0 || q.newton) {
            qs = q.in_start[a];
            nin = q.in_start[a + 1] - qs;
        }
        if (g == 0) {
            npre = q.in_split[a];
            rs = q.offsets[t];
            nrow = q.offsets[t + 1] - rs;
        }
        pa = make_double4(c.x[a], c.y[a], c.z[a], q.rad[a]);
    }
    // items numbered through: this lane's are entries [from, to)
    const uint32_t n = nin + nrow;
    uint32_t to = n;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kAll, to, o, 8);
        if (g >= (uint32_t)o) to += v;
    }
    const uint32_t total = __shfl_sync(kAll, to, 7, 8);
    uint32_t ends[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) ends[j] = __shfl_sync(kAll, to, j, 8);
    const uint32_t rounds = __reduce_max_sync(kAll, (total + 7) / 8);
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;     // this lane's item
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t k = r * 8 + g;
        int item = 0;
#pragma unroll
        for (int j = 0; j < 7; ++j) item += k >= ends[j];
        // the item's lists and position from its lane
        const uint32_t iqs = __shfl_sync(kAll, qs, item, 8), inpre = __shfl_sync(kAll, npre, 0, 8);
        const uint32_t irs = __shfl_sync(kAll, rs, 0, 8), inrow = __shfl_sync(kAll, nrow, 0, 8);
        const uint32_t base = __shfl_sync(kAll, to - n, item, 8);
        const double px = __shfl_sync(kAll, pa.x, item, 8), py = __shfl_sync(kAll, pa.y, item, 8);
        const double pz = __shfl_sync(kAll, pa.z, item, 8), pr = __shfl_sync(kAll, pa.w, item, 8);
        double fx = 0.0, fy = 0.0, fz = 0.0;
        bool touch = false;
        if (k < total) {
            const uint32_t e = k - base;
            uint32_t o;
            if (item) o = q.in_list[iqs + e];
            else if (e < inpre) o = q.in_list[iqs + e];
            else if (e < inpre + inrow) o = q.indices[irs + (e - inpre)];
            else o = q.in_list[iqs + (e - inrow)];
            touch = pair_force(px, py, pz, pr, c.x[o], c.y[o], c.z[o], q.rad[o], q.K, fx, fy, fz);
        }
        const unsigned hits = __ballot_sync(kAll, touch) >> ((threadIdx.x & 31u) & ~7u);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double ex = __shfl_sync(kAll, fx, j, 8), ey = __shfl_sync(kAll, fy, j, 8);
            const double ez = __shfl_sync(kAll, fz, j, 8);
            const uint32_t kk = r * 8 + j;
            if (((hits >> j) & 1u) && kk >= to - n && kk < to) {
                Fx = Fx + ex;
                Fy = Fy + ey;
                Fz = Fz + ez;
            }
        }
    }
    if (FOLD) {  // fold_root's order
        uint32_t par = 0;  // this image's parent item
        if (mine && g && org >= q.nlocal) par = 0xffu;
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            const uint32_t gj = __shfl_sync(kAll, gi, j, 8);
            if (par && (uint32_t)j <= nimg && org == q.nlocal + gj) par = (uint32_t)j;
        }
        const uint32_t most = __reduce_max_sync(kAll, nimg);
        for (uint32_t j = 1; j <= most; ++j) {
            const double ex = __shfl_sync(kAll, Fx, j, 8), ey = __shfl_sync(kAll, Fy, j, 8);
            const double ez = __shfl_sync(kAll, Fz, j, 8);
            const uint32_t p = __shfl_sync(kAll, par, j, 8);
            if (j <= nimg && p == g) {
                Fx = Fx + ex;
                Fy = Fy + ey;
                Fz = Fz + ez;
            }
        }
        if (valid && g == 0)
            for (uint32_t f = f0; f < f0 + nimg && rev.n; ++f) {
                const uint64_t gh = q.nlocal + q.fold_list[f];
                const uint32_t o = (uint32_t)c.origin[gh];
                for (int k = 0; k < rev.n; ++k)
                    c.planes[rev.idx[k]][o] = c.planes[rev.idx[k]][o] + c.planes[rev.idx[k]][gh];
            }
    }
    if (mine) {
        c.fx[a] = Fx;
        c.fy[a] = Fy;
        c.fz[a] = Fz;
    }
}

// Largest system that takes 8 lanes per root: one resident wave of them
// (on 8,009 sheared atoms 5 against 12.5 us).
constexpr uint64_t kForceGroupRoots = 148ull * 4 * kBlock / 8;

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

void launch_force_csr(cudaStream_t st, const ForceCsr& q, const AtomCols& c, const PlaneList& rev,
                      bool fold, bool few_images, const uint32_t* trip, const FillGuard* guard) {
    if (q.nlocal == 0) return;
    note_launch();
    const FillGuard gd = guard ? *guard : FillGuard{};
    if (q.nlocal <= kForceGroupRoots && few_images && !q.pk && !q.order) {
        const unsigned blocks = (unsigned)((q.nlocal * 8 + kBlock - 1) / kBlock);
        if (fold) pdl_launch(k_force_group<true>, blocks, kBlock, 0, st, q, c, rev, trip, gd);
        else pdl_launch(k_force_group<false>, blocks, kBlock, 0, st, q, c, rev, trip, gd);
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
    if (q.pk) {
        if (fold) pdl_launch(k_force_csr<true, true>, grid, kBlock, 0, st, q, c, rev, trip, gd);
        else pdl_launch(k_force_csr<false, true>, grid, kBlock, 0, st, q, c, rev, trip, gd);
    } else {
        if (fold) pdl_launch(k_force_csr<true, false>, grid, kBlock, 0, st, q, c, rev, trip, gd);
        else pdl_launch(k_force_csr<false, false>, grid, kBlock, 0, st, q, c, rev, trip, gd);
    }
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
