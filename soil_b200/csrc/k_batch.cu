// k_batch.cu — segmented kernels of the batched engine (see batch.cuh).
//
// Three launch shapes:
//   element spans   blocks walk the flattened element range in chunks of
//                   Span::items rows of kBlock elements; a warp locates the
//                   chunk's segment once and its lanes advance per element
//                   (boxes hold hundreds of atoms or more);
//   scan tiles      one CTA per 8,192 counts of a box (scan_direct_tile);
//   tile spans      border and staged pair tiles, one warp per 32 locals.
// Every element calls the same device function as the single-system kernels.
#include "batch.cuh"
#include "block_scan.cuh"
#include "border_ops.cuh"
#include "force_ops.cuh"
#include "pairs_staged.cuh"
#include "sys_internal.cuh"

namespace soil {

// Segment holding flattened element g (the last segment whose start is <= g),
// found by the 32 lanes of one warp together: each level probes 32 evenly
// spaced starts, so 4,096 segments take three dependent loads.  Call with all
// 32 lanes of the warp; every lane returns the answer.
__device__ __forceinline__ uint32_t seg_of_warp(const Span& sp, uint64_t g) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = sp.nseg;  // start[lo] <= g < start[hi]
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        const bool ok = idx < hi && sp.start[idx] <= g;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const uint32_t last = 31u - (uint32_t)__clz(m);  // starts are sorted: ok is a prefix
        lo = lo + last * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// f(box, element index inside the box, segment) for every element of the
// span.  Chunks go to CTAs cyclically, so the CTAs running at any moment work
// on neighbouring chunks (the same few boxes, whose data then stays in L2).
// Each warp looks up the segment of its first element itself (no block
// barrier) and its lanes walk forward from there.
template <class F>
__device__ __forceinline__ void for_span(const Span& sp, F f) {
    pdl_wait();  // every span kernel is launched with pdl_launch
    const uint64_t chunk = (uint64_t)blockDim.x * sp.items;
    const uint64_t warp0 = threadIdx.x & ~31u;
    for (uint64_t g0 = (uint64_t)blockIdx.x * chunk; g0 < sp.total;
         g0 += (uint64_t)gridDim.x * chunk) {
        const uint64_t gw = g0 + warp0 < sp.total ? g0 + warp0 : g0;
        uint32_t k = seg_of_warp(sp, gw);
        for (uint32_t it = 0; it < sp.items; ++it) {
            const uint64_t g = g0 + (uint64_t)it * blockDim.x + threadIdx.x;
            if (g >= sp.total) break;
            while (g >= sp.start[k + 1]) ++k;
            f(sp.box[k], (uint64_t)sp.base[k] + (g - sp.start[k]), k);
        }
    }
}

static unsigned span_grid(const Span& sp) { return grid_for((sp.total + sp.items - 1) / sp.items); }

// One resident wave of span kernel K (grid_wave), never more than the span needs.
template <auto K>
static unsigned span_wave(const Span& sp) {
    return grid_wave<K>((sp.total + sp.items - 1) / sp.items);
}

#define SPAN_KERNEL(name, ...)                                                        \
    __global__ void __launch_bounds__(kBlock) name(Span sp, BatchArgs A) {            \
        for_span(sp, [&](uint32_t b, uint64_t i, uint32_t k) {                        \
            const BoxDev& D = A.dev[b];                                               \
            const BoxStep& S = A.step[b];                                             \
            (void)D;                                                                  \
            (void)S;                                                                  \
            (void)k;                                                                  \
            __VA_ARGS__                                                               \
        });                                                                           \
    }

#define SPAN_LAUNCH(fn, kern)                                        \
    void fn(cudaStream_t st, const Span& sp, const BatchArgs& a) {   \
        if (sp.total == 0) return;                                   \
        note_launch();                                               \
        pdl_launch(kern, span_wave<kern>(sp), kBlock, 0, st, sp, a); \
    }

// ---- integrate --------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) kb_initial(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t k) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const uint8_t f = sp.flag[k];
        const AtomCols& c = D.set[S.post];  // current at the start of a step
        double x, y, z;
        initial_atom(c, i, S.dt, (f & 2) != 0, (f & 4) != 0, x, y, z);
        if ((f & 1) && moved_too_far(x, y, z, D.lbx[i], D.lby[i], D.lbz[i], S.box, S.ibox, S.thr_sq))
            atomicOr(&A.flags[b].rebuild, 1u);
    });
}
SPAN_LAUNCH(b_initial, kb_initial)

SPAN_KERNEL(kb_final, { final_atom(D.set[S.post], i, S.dt); })
SPAN_LAUNCH(b_final, kb_final)

// soil_deform/src/lib.rs:568-574 (first shear step)
SPAN_KERNEL(kb_profile, {
    const AtomCols& c = D.set[S.post];
    c.vx[i] = c.vx[i] + D.shear_rate * (c.y[i] - D.yc);
})
SPAN_LAUNCH(b_profile, kb_profile)

SPAN_KERNEL(kb_zero_forces, {
    const AtomCols& c = D.set[S.cur];
    c.fx[i] = 0.0;
    c.fy[i] = 0.0;
    c.fz[i] = 0.0;
    for (int q = 0; q < D.zero.n; ++q) c.planes[D.zero.idx[q]][i] = 0.0;
})
SPAN_LAUNCH(b_zero_forces, kb_zero_forces)

// ---- bins -----------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) kb_pbc_cells(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t k) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const AtomCols& c = D.set[S.cur];
        const uint8_t f = sp.flag[k];
        double x, y, z;
        if (f & 1) {
            pbc_atom(c, i, S.geom, S.bvel[0], S.bvel[1], S.bvel[2], x, y, z);
        } else {
            x = c.x[i];
            y = c.y[i];
            z = c.z[i];
        }
        if (f & 2) {
            const uint32_t cell = cell_of(S.grid, x, y, z);
            D.sort_cell[i] = cell;
            atomicAdd(&D.cell_counts[cell], 1u);
        }
    });
}
SPAN_LAUNCH(b_pbc_cells, kb_pbc_cells)

SPAN_KERNEL(kb_ghost_cells, {
    // the border pass's ghosts get their columns here; the consumer overwrites
    // every force of the step
    const double3 q = make_ghost(D.set[S.post], S.nlocal, i - S.nlocal, D.ghost_root,
                                 D.ghost_chain, S.sc, false);
    const uint32_t cell = cell_of(S.grid, q.x, q.y, q.z);
    D.atom_cell[i] = cell;
    atomicAdd(&D.cell_counts[cell], 1u);
})
SPAN_LAUNCH(b_ghost_cells, kb_ghost_cells)

// One CTA per tile of a box's counts, no waits between them (scan_direct_tile).
// (One CTA per box walked the tiles of the largest box in series: 43 us a scan
// on 128 boxes of up to 65,536 atoms, 8.3 with a CTA per tile.)
__global__ void __launch_bounds__(kDirectThreads) kb_scan(Span sp, BatchArgs A) {
    pdl_wait();  // launched with pdl_launch
    const uint32_t k = seg_of_warp(sp, blockIdx.x);
    const uint32_t b = sp.box[k];
    const BoxDev& D = A.dev[b];
    const uint64_t tile = blockIdx.x - sp.start[k], ntiles = sp.start[k + 1] - sp.start[k];
    const uint64_t n = sp.base[k];
    const int which = sp.flag[k];
    const uint32_t* in = D.cell_counts;
    const uint32_t* add = nullptr;
    uint32_t* out = D.sort_start;
    if (which == BA_NEIGH_CELLS) {
        out = D.cell_start;
        add = D.sort_start;
    } else if (which == BA_ROWS) {
        in = D.rowcount;
        out = D.offsets;
    } else if (which == BA_IN) {
        in = D.in_count;
        out = D.in_start;
    } else if (which == BA_GRP) {
        in = D.grp_cnt;
        out = D.grp_start;
    }
    const uint32_t total = scan_direct_tile(in, out, n, tile, ntiles, add);
    if (which == BA_ROWS && tile + 1 == ntiles && threadIdx.x == 0) A.totals[b] = total;
}
void b_scan(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    pdl_launch(kb_scan, (unsigned)sp.total, kDirectThreads, 0, st, sp, a);
}

__global__ void __launch_bounds__(kBlock) kb_scatter(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t k) {
        const BoxDev& D = A.dev[b];
        const uint32_t cell = D.sort_cell[i];
        (sp.flag[k] ? D.sort_perm : D.bins)[D.sort_start[cell] + atomicSub(&D.cell_counts[cell], 1u) -
                                            1u] = (uint32_t)i;
    });
}
SPAN_LAUNCH(b_scatter, kb_scatter)

// as k_sort_gather
SPAN_KERNEL(kb_sort_gather, {
    const uint32_t p = D.bins[i];
    const uint32_t c = D.sort_cell[p];
    const uint32_t first = D.sort_start[c];
    const uint32_t end = D.sort_start[c + 1];
    uint32_t to = first;
    for (uint32_t j = first; j < end; ++j) to += D.bins[j] < p;
    perm_gather_atom(D.set[S.cur], D.set[S.post], to, p, false);
    D.sort_perm[to] = p;
    D.sorted_local_cell[to] = c;
})
SPAN_LAUNCH(b_sort_gather, kb_sort_gather)

SPAN_KERNEL(kb_segsort, { insertion_sort(D.sort_perm, D.sort_start[i], D.sort_start[i + 1]); })
SPAN_LAUNCH(b_segsort, kb_segsort)

SPAN_KERNEL(kb_permute_cells, { D.sorted_local_cell[i] = D.sort_cell[D.sort_perm[i]]; })
SPAN_LAUNCH(b_permute_cells, kb_permute_cells)

SPAN_KERNEL(kb_identity, {
    if (D.sort_perm[i] != (uint32_t)i) atomicOr(&A.flags[b].not_identity, 1u);
})
SPAN_LAUNCH(b_identity, kb_identity)

SPAN_KERNEL(kb_perm_gather, { perm_gather_atom(D.set[S.cur], D.set[S.post], i, D.sort_perm[i]); })
SPAN_LAUNCH(b_perm_gather, kb_perm_gather)

// ---- borders (chain categories; the single-system kernels are in k_ghost.cu) ---
// Warp-tile spans: every warp takes one tile of 32 locals of one box;
// f(box, warp tile index inside the box, segment).
template <class F>
__device__ __forceinline__ void for_warp_tiles(const Span& sp, F f) {
    pdl_wait();  // every tile kernel is launched with pdl_launch
    const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x / 32);
    for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; g < sp.total;
         g += nwarps) {
        const uint32_t k = seg_of_warp(sp, g);
        f(sp.box[k], (uint64_t)sp.base[k] + (g - sp.start[k]), k);
    }
}

__global__ void __launch_bounds__(kBlock) kb_border_faces(Span sp, BatchArgs A, BorderCats cats) {
    const uint32_t lane = threadIdx.x & 31u;
    for_warp_tiles(sp, [&](uint32_t b, uint64_t w, uint32_t k) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const uint64_t nw = sp.start[k + 1] - sp.start[k];
        border_warp_counts(D.set[S.post], S.nlocal, S.geom, S.geom.triclinic, S.thresh_lo,
                           S.thresh_hi, cats, D.face_flags, D.bcount, nw, w, lane);
    });
}
void b_border_faces(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    pdl_launch(kb_border_faces, grid_wave<kb_border_faces>(sp.total * 32), kBlock, 0, st, sp, a,
               border_cats());
}

// one CTA per (box, category): exclusive scan of the warp counts
__global__ void __launch_bounds__(kBlock) kb_border_cat_scan(Span sp, BatchArgs A) {
    pdl_wait();  // launched with pdl_launch
    const uint32_t seg = blockIdx.x / (kBorderCats + 1), k = blockIdx.x % (kBorderCats + 1);
    const uint32_t b = sp.box[seg];
    const BoxDev& D = A.dev[b];
    const uint64_t nw = sp.start[seg + 1] - sp.start[seg];
    const uint32_t total = cta_scan_array<8>(D.bcount + k * nw, D.boff + k * nw, nullptr, nw);
    if (threadIdx.x == 0) A.bstate[(uint64_t)b * kBorderStateWords + kBorderTotals + k] = total;
}
void b_border_cat_scan(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.nseg == 0) return;
    note_launch();
    pdl_launch(kb_border_cat_scan, sp.nseg * (kBorderCats + 1), kBlock, 0, st, sp, a);
}

__global__ void __launch_bounds__(kBlock) kb_border_images(Span sp, BatchArgs A, BorderCats cats) {
    __shared__ BorderWarpSmem sm[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31u;
    for_warp_tiles(sp, [&](uint32_t b, uint64_t w, uint32_t k) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        uint32_t* bs = A.bstate + (uint64_t)b * kBorderStateWords;
        const uint64_t nw = sp.start[k + 1] - sp.start[k];
        const uint32_t tot = lane < kBorderCats ? bs[kBorderTotals + lane] : 0u;
        const uint32_t base_lane = (uint32_t)S.nlocal + warp_exclusive_sum(tot, lane);
        if (w == 0) border_state_words(cats, base_lane, lane, bs, nullptr);
        border_warp_images(D.set[S.post], S.nlocal, D.cap, cats, D.face_flags,
                           ScannedOffs{D.boff, nullptr, 1, nw, w}, w, lane, base_lane, bs, D.ghost_root, D.ghost_chain, D.send,
                           D.fold_start, D.fold_list, sm[threadIdx.x / 32]);
    });
}
void b_border_images(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    pdl_launch(kb_border_images, grid_wave<kb_border_images>(sp.total * 32), kBlock, 0, st, sp, a,
               border_cats());
}

SPAN_KERNEL(kb_forward, {
    forward_ghost(D.set[S.post], S.nlocal, i, D.ghost_root, D.ghost_chain, S.sc, D.fwd, false);
})
SPAN_LAUNCH(b_forward, kb_forward)

// ---- neighbor build ---------------------------------------------------------
__device__ __forceinline__ SortedViews sorted_views(const BoxDev& D, const BoxStep& S) {
    SortedViews v;
    v.c = D.set[S.post];
    v.sorted = D.sorted_atoms;
    v.asi = D.asi;
    v.sp = D.sp;
    v.spf = S.filter ? D.spf : nullptr;
    for (int d = 0; d < 3; ++d) v.origin[d] = S.geom.lo[d];
    v.bp.x = D.lbx;
    v.bp.y = D.lby;
    v.bp.z = D.lbz;
    v.bp.nlocal = S.nlocal;
    v.atom_in_w = S.uniform;
    v.clear = nullptr;
    return v;
}

// as k_place_bins and k_ghost_rank
SPAN_KERNEL(kb_place_bins, {
    if (i < S.nlocal) {
        const uint32_t c = D.sorted_local_cell[i];
        put_sorted(sorted_views(D, S), D.cell_start[c] + ((uint32_t)i - D.sort_start[c]), (uint32_t)i);
    } else {
        const uint32_t c = D.atom_cell[i];
        D.bins[ghost_slots(D.cell_start, D.sort_start, c) + atomicSub(&D.cell_counts[c], 1u) - 1u] =
            (uint32_t)i;
    }
})
SPAN_LAUNCH(b_place_bins, kb_place_bins)

SPAN_KERNEL(kb_ghost_rank, {
    rank_ghost(sorted_views(D, S), (uint32_t)i, D.atom_cell[i], D.cell_start, D.sort_start, D.bins);
})
SPAN_LAUNCH(b_ghost_rank, kb_ghost_rank)

__device__ __forceinline__ PairParams pair_params(const BoxDev& D, const BoxStep& S) {
    PairParams p;
    p.atom_cell = D.sorted_local_cell;  // read for rows, which are locals
    p.atom_sorted_idx = D.asi;
    p.bin_start = D.cell_start;
    p.sorted_atoms = D.sorted_atoms;
    p.sp = D.sp;
    p.spf = D.spf;
    p.stencil = S.stencil;
    p.nstencil = S.nstencil;
    p.ncells = S.ncells;
    p.nlocal = S.nlocal;
    p.has_self = S.has_self;
    p.newton = S.newton;
    p.uniform = S.uniform;
    p.filter = S.filter;
    p.row_slots = soil_host::kRowSlotsPerAtom;
    p.cut_sq = S.cut_sq;
    p.sf_sq = S.sf_sq;
    p.sf = S.sf;
    p.eps32 = S.eps32;
    p.in_count = D.in_count;
    p.in_start = D.in_start;
    p.in_list = D.in_list;
    p.pre_ranges = S.pre_ranges;
    return p;
}

template <bool UNIFORM, bool FP32>
__device__ __forceinline__ void pairs_row(const PairParams& p, uint64_t i, uint32_t* rowcount,
                                          uint32_t* slots, DevFlags* flags, uint32_t& cd,
                                          uint32_t& rk) {
    const Filter<UNIFORM, FP32> test(p);
    const uint32_t K = (uint32_t)p.row_slots;
    rowcount[i] = row_scan<UNIFORM, FP32, true>(p, test, i, slots + i * K, K, &rk, &cd, flags,
                                                p.in_count);
}

__device__ __forceinline__ void add_filter_stats(DevFlags* f, uint32_t cd, uint32_t rk) {
    if (cd) atomicAdd((unsigned long long*)&f->candidates, (unsigned long long)cd);
    if (rk) atomicAdd((unsigned long long*)&f->rechecked, (unsigned long long)rk);
}

// Pair count pass over the rows of every box in the span.  The candidate and
// recheck statistics are summed per box inside each warp (lanes matched by
// box) before one atomic per box and warp.
// (One kernel for every cutoff kind and filter took 106 registers: 109 us on
// 128 boxes, 1.5 million atoms, against 108 with the transposed lists counted
// too.)
template <bool UNIFORM, bool FP32>
__global__ void __launch_bounds__(kBlock, FP32 ? 3 : 4) kb_pairs_rows(Span sp, BatchArgs A) {
    uint32_t cur = 0xffffffffu, cd = 0, rk = 0;
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t) {
        if (b != cur) {
            if (cur != 0xffffffffu) add_filter_stats(A.flags + cur, cd, rk);
            cur = b;
            cd = 0;
            rk = 0;
        }
        const BoxDev& D = A.dev[b];
        pairs_row<UNIFORM, FP32>(pair_params(D, A.step[b]), i, D.rowcount, D.row_slots, A.flags + b,
                                 cd, rk);
    });
    const unsigned peers = __match_any_sync(0xffffffffu, cur);
    const uint32_t scd = __reduce_add_sync(peers, cd);
    const uint32_t srk = __reduce_add_sync(peers, rk);
    if (cur != 0xffffffffu && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
        add_filter_stats(A.flags + cur, scd, srk);
}

// A span kernel's instance for the boxes of one cutoff kind and filter.
#define PAIR_LAUNCH(fn, kern)                                                                      \
    void fn(cudaStream_t st, const Span& sp, const BatchArgs& a, bool uniform, bool fp32) {        \
        if (sp.total == 0) return;                                                                 \
        note_launch();                                                                             \
        auto go = [&](auto k, unsigned grid) { pdl_launch(k, grid, kBlock, 0, st, sp, a); };       \
        if (uniform && fp32) go(kern<true, true>, span_wave<kern<true, true>>(sp));                \
        else if (uniform) go(kern<true, false>, span_wave<kern<true, false>>(sp));                 \
        else if (fp32) go(kern<false, true>, span_wave<kern<false, true>>(sp));                    \
        else go(kern<false, false>, span_wave<kern<false, false>>(sp));                            \
    }
PAIR_LAUNCH(b_pairs_rows, kb_pairs_rows)

// The staged pair count over warp tiles of every box (the single-system
// kernel is k_pairs_staged); boxes whose stencil does not fit PairSegs scan
// their rows from global memory.
template <bool UNIFORM, bool FP32>
__device__ __forceinline__ bool batch_tile(const PairParams& p, const BoxStep& S, const BoxDev& D,
                                           uint64_t w, unsigned char* recs, uint64_t* bar,
                                           uint32_t& phase, uint32_t* lo, uint32_t* base,
                                           DevFlags* fl, uint32_t& cd, uint32_t& rk) {
    if (S.segs_ok)
        return staged_tile<UNIFORM, FP32>(p, S.segs, w, recs, bar, phase, lo, base, D.rowcount,
                                          D.row_slots, fl, rk, cd);
    const uint64_t i = w * 32 + (threadIdx.x & 31);
    if (i < p.nlocal) pairs_row<UNIFORM, FP32>(p, i, D.rowcount, D.row_slots, fl, cd, rk);
    return true;
}

__global__ void __launch_bounds__(kStageWarps * 32) kb_pairs_staged(Span sp, BatchArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t s_lo[kStageWarps][kMaxPairSegs];
    __shared__ uint32_t s_base[kStageWarps][kMaxPairSegs];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char* recs = smem_raw + (size_t)wib * kStageRecs * 32;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + (size_t)kStageWarps * kStageRecs * 32) + wib;
    staged_init(bar);
    uint32_t phase = 0;
    bool ok = true;
    for_warp_tiles(sp, [&](uint32_t b, uint64_t w, uint32_t) {
        if (!ok) return;
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const PairParams p = pair_params(D, S);
        DevFlags* fl = A.flags + b;
        uint32_t cd = 0, rk = 0;
        if (S.uniform) {
            if (S.filter) ok = batch_tile<true, true>(p, S, D, w, recs, bar, phase, s_lo[wib], s_base[wib], fl, cd, rk);
            else ok = batch_tile<true, false>(p, S, D, w, recs, bar, phase, s_lo[wib], s_base[wib], fl, cd, rk);
        } else {
            if (S.filter) ok = batch_tile<false, true>(p, S, D, w, recs, bar, phase, s_lo[wib], s_base[wib], fl, cd, rk);
            else ok = batch_tile<false, false>(p, S, D, w, recs, bar, phase, s_lo[wib], s_base[wib], fl, cd, rk);
        }
        const uint32_t scd = __reduce_add_sync(0xffffffffu, cd);
        const uint32_t srk = __reduce_add_sync(0xffffffffu, rk);
        if (lane == 0) add_filter_stats(fl, scd, srk);
    });
}

void b_pairs_staged(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    const size_t smem = (size_t)kStageWarps * kStageRecs * 32 + kStageWarps * sizeof(uint64_t);
    const uint64_t per = kStageWarps;
    uint64_t blocks = (sp.total + per - 1) / per;
    if (blocks > 148ull * 8ull) blocks = 148ull * 8ull;
    pdl_launch(kb_pairs_staged, (unsigned)blocks, kStageWarps * 32, smem, st, sp, a);
}

// Row i into its CSR place (from its slots, or derived again when longer) and
// into every partner's transposed list, taking the counts back to zero.
template <bool UNIFORM, bool FP32>
__global__ void __launch_bounds__(kBlock) kb_pairs_fill(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t) {
        const BoxDev& D = A.dev[b];
        const PairParams p = pair_params(D, A.step[b]);
        const Filter<UNIFORM, FP32> test(p);
        fill_row<UNIFORM, FP32>(p, test, i, D.rowcount, D.row_slots, D.offsets, D.indices);
    });
}
PAIR_LAUNCH(b_pairs_fill, kb_pairs_fill)

SPAN_KERNEL(kb_in_sort, {
    D.in_split[i] = sort_segment(D.in_list, D.in_start[i], D.in_start[i + 1], (uint32_t)i);
})
SPAN_LAUNCH(b_in_sort, kb_in_sort)

// ---- force and reverse comm ---------------------------------------------------
// The single system's walk (k_force_csr): one thread per root, its images
// after it, then the fold.  (At 64 registers, four CTAs per SM, the boxes'
// pointers spill: 159 against 133 us on 1.5 million atoms in 128 boxes.)
__global__ void __launch_bounds__(kBlock, 3) kb_force_csr(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const AtomCols& c = D.set[S.post];
        ForceCsr q;
        q.rad = c.planes[D.radius_plane];
        q.K = S.K;
        q.nlocal = S.nlocal;
        q.newton = S.newton;
        q.offsets = D.offsets;
        q.indices = D.indices;
        q.in_start = D.in_start;
        q.in_list = D.in_list;
        q.in_split = D.in_split;
        q.fold_start = D.fold_start;
        q.fold_list = D.fold_list;
        force_csr_items(q, ColLd{c.x, c.y, c.z, q.rad}, c, i);
        if (S.newton) fold_root(c, S.nlocal, i, D.fold_start, D.fold_list, D.rev);
    });
}
SPAN_LAUNCH(b_force_csr, kb_force_csr)

// The per-atom gather (SOIL_FORCE=gather) with its reverse pass.
__global__ void __launch_bounds__(kBlock, 5) kb_harmonic(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const AtomCols& c = D.set[S.post];
        harmonic_atom(c, i, S.nlocal, c.planes[D.radius_plane], S.K, S.newton, D.offsets,
                      D.indices, D.in_start, D.in_list);
    });
}
SPAN_LAUNCH(b_harmonic, kb_harmonic)

SPAN_KERNEL(kb_reverse, { fold_root(D.set[S.post], S.nlocal, i, D.fold_start, D.fold_list, D.rev); })
SPAN_LAUNCH(b_reverse, kb_reverse)

// ---- the grouped consumer (the single-system kernels are in k_force.cu) -------
__device__ __forceinline__ SeqArgs seq_args(const BoxDev& D, const BoxStep& S) {
    SeqArgs q;
    q.nlocal = S.nlocal;
    q.ntotal = S.nlocal + S.nghost;
    q.newton = S.newton;
    q.offsets = D.offsets;
    q.indices = D.indices;
    q.in_start = D.in_start;
    q.in_list = D.in_list;
    q.fold_start = D.fold_start;
    q.fold_list = D.fold_list;
    return q;
}

SPAN_KERNEL(kb_seq_count, { seq_count_atom(seq_args(D, S), i, D.seq_cnt, D.grp_cnt); })
SPAN_LAUNCH(b_seq_count, kb_seq_count)

SPAN_KERNEL(kb_seq_fill, { seq_fill_root(seq_args(D, S), i, D.grp_start, D.seq, D.seq_owner); })
SPAN_LAUNCH(b_seq_fill, kb_seq_fill)

__device__ __forceinline__ ForceSeq force_seq_of(const BoxDev& D, const BoxStep& S,
                                                 const AtomCols& c) {
    ForceSeq q;
    q.rad = c.planes[D.radius_plane];
    q.K = S.K;
    q.nlocal = S.nlocal;
    q.grp_start = D.grp_start;
    q.cnt = D.seq_cnt;
    q.seq = D.seq;
    q.owner = D.seq_owner;
    q.fold_start = D.fold_start;
    q.fold_list = D.fold_list;
    q.pk = nullptr;
    return q;
}

__global__ void __launch_bounds__(kBlock, 3) kb_force_grouped(Span sp, BatchArgs A) {
    __shared__ ForceSmem<4> sm;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for_warp_tiles(sp, [&](uint32_t b, uint64_t w, uint32_t) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const AtomCols& c = D.set[S.post];
        const ForceSeq q = force_seq_of(D, S, c);
        if (S.newton) force_tile<4, true>(q, c, D.rev, w, sm, lane, wib);
        else force_tile<4, false>(q, c, D.rev, w, sm, lane, wib);
    });
}
__global__ void __launch_bounds__(kBlock, 4) kb_force_walk(Span sp, BatchArgs A) {
    for_span(sp, [&](uint32_t b, uint64_t i, uint32_t) {
        const BoxDev& D = A.dev[b];
        const BoxStep& S = A.step[b];
        const AtomCols& c = D.set[S.post];
        const ForceSeq q = force_seq_of(D, S, c);
        if (S.newton) force_walk_root<true, false>(q, c, D.rev, i);
        else force_walk_root<false, false>(q, c, D.rev, i);
    });
}
void b_force_walk(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    const unsigned g = span_grid(sp);
    pdl_launch(kb_force_walk, g < 148u * 4u ? g : 148u * 4u, kBlock, 0, st, sp, a);
}

void b_force_grouped(cudaStream_t st, const Span& sp, const BatchArgs& a) {
    if (sp.total == 0) return;
    note_launch();
    uint64_t blocks = (sp.total + kBlock / 32 - 1) / (kBlock / 32);
    if (blocks > 148ull * 3ull) blocks = 148ull * 3ull;  // one resident wave
    pdl_launch(kb_force_grouped, (unsigned)blocks, kBlock, 0, st, sp, a);
}

}  // namespace soil
