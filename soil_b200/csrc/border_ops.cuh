// border_ops.cuh — warp-tile routines of the borders pass (chain categories,
// see k_ghost.cu), shared by the single-system and the batched kernels.
//
// A warp tile is 32 consecutive locals, one per lane.  Pass 1 stores the face
// bits and, per category, the tile's member count (counts[k * nw + w]; row
// kBorderCats holds all images of the tile).  After a per-category scan
// (offs, same layout), pass 2 ranks each member inside its tile with a ballot
// and writes its image's root, chain and origin, its send entry and its root's
// fold program; the images' columns follow with one thread per ghost
// (make_ghost), whose writes are coalesced whatever the number of images per
// root.  Every routine is called by all 32 lanes of a warp.
#pragma once

#include "block_scan.cuh"
#include "device_ops.cuh"

namespace soil {

__device__ __forceinline__ bool cat_member(const BorderCats& cats, uint32_t bits, int k) {
    return (bits & cats.need[k]) == cats.need[k];
}

__device__ __forceinline__ uint32_t warp_exclusive_sum(uint32_t v, uint32_t lane) {
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    return incl - v;
}

// Pass 1 for warp tile w: local r = 32 w + lane.
__device__ __forceinline__ void border_warp_counts(const AtomCols& c, uint64_t nlocal,
                                                   const Geom& geom, int triclinic,
                                                   const double* lo, const double* hi,
                                                   const BorderCats& cats, uint8_t* face,
                                                   uint32_t* counts, uint64_t nw, uint64_t w,
                                                   uint32_t lane) {
    const uint64_t r = w * 32 + lane;
    uint32_t bits = 0;
    if (r < nlocal) {
        bits = face_bits(c, geom, triclinic, lo, hi, r);
        face[r] = (uint8_t)bits;
    }
    uint32_t mine = 0, images = 0;
    // a category can have members only if the tile's faces cover its need:
    // the categories of the OR of its bits (uniform over the warp)
    const uint32_t any = __reduce_or_sync(0xffffffffu, bits);
    const uint32_t mine_cats = cats.member[bits];
    for (uint32_t cand = cats.member[any]; cand; cand &= cand - 1) {
        const int k = __ffs(cand) - 1;
        const uint32_t n = __popc(__ballot_sync(0xffffffffu, (mine_cats >> k) & 1u));
        if (lane == (uint32_t)k) mine = n;
        images += n;
    }
    if (lane < kBorderCats) counts[lane * nw + w] = mine;
    if (lane == kBorderCats) counts[kBorderCats * nw + w] = images;
}

// Per-dim border state in the format the host reads (bs[0..9]; and its own
// copy, when given), by one warp: base_lane as for border_warp_images (on lane
// 26 the end of all ghosts).  A swap's categories follow one another, so its
// ghosts are those from its first category's base to the next swap's.  (One
// lane adding up the totals from memory was what a small system's border pass
// waited for: k_border_images 9.3 us on 8,009 atoms.)
__device__ __forceinline__ void border_state_words(const BorderCats& cats, uint32_t base_lane,
                                                   uint32_t lane, uint32_t* bs,
                                                   uint32_t* host_bs) {
    // word 0: nlocal; 1-3: the end of dim d; 4-6, 7-9: ghosts of its lo / hi swap
    const int d = lane == 0 ? 0 : (int)(lane - 1) % 3;
    const int from = lane < 7 ? 2 * d : 2 * d + 1;
    const int to = lane == 0 ? 0 : lane < 4 ? 2 * d + 2 : lane < 7 ? 2 * d + 1 : 2 * d + 2;
    const int first = cats.swap_first[from], last = to < kNumSwaps ? cats.swap_first[to] : kBorderCats;
    const uint32_t lo = __shfl_sync(0xffffffffu, base_lane, first);
    const uint32_t hi = __shfl_sync(0xffffffffu, base_lane, last);
    if (lane >= 10) return;
    const uint32_t v = lane < 4 ? hi : hi - lo;
    bs[lane] = v;
    if (host_bs) host_bs[lane] = v;
}

// Warp tiles per scan chunk: the category scans run one CTA per (category,
// chunk); chunk prefixes (cpre[k * nchunks + chunk]; NULL: a single chunk) are
// added back here.
constexpr uint64_t kScanChunk = 8192;
struct ScannedOffs {
    const uint32_t* offs;
    const uint32_t* cpre;
    uint64_t nchunks, nw, w;
    __device__ __forceinline__ uint32_t operator()(uint32_t k) const {
        return offs[k * nw + w] + (cpre ? cpre[k * nchunks + w / kScanChunk] : 0u);
    }
};

// A pass of few tiles needs no scan launch: each CTA of pass 2 sums the
// counts before its own tiles itself.
struct BorderCtaOffs {
    uint32_t before[kBorderCats + 1];               // in the tiles before this CTA's
    uint32_t total[kBorderCats + 1];                // in all tiles
    uint32_t tile[kBorderCats + 1][kBlock / 32];    // in each of its tiles
};
// (all threads; a barrier follows)
__device__ __forceinline__ void border_cta_offs(const uint32_t* counts, uint64_t nw, uint64_t first,
                                                BorderCtaOffs& sm) {
    constexpr uint32_t kWarps = kBlock / 32, kCats = (kBorderCats + kWarps) / kWarps;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x / 32;
    uint32_t before[kCats] = {}, total[kCats] = {};
    for (uint64_t t0 = 0; t0 < nw; t0 += 256) {  // every load of 256 tiles in flight
        uint32_t v[kCats][8];
#pragma unroll
        for (int q = 0; q < (int)kCats; ++q)
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint64_t t = t0 + u * 32 + lane;
                const uint32_t k = w + q * kWarps;
                v[q][u] = t < nw && k <= (uint32_t)kBorderCats ? counts[k * nw + t] : 0u;
            }
#pragma unroll
        for (int q = 0; q < (int)kCats; ++q)
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint64_t t = t0 + u * 32 + lane;
                total[q] += v[q][u];
                before[q] += t < first ? v[q][u] : 0u;
                if (t >= first && t < first + kWarps && w + q * kWarps <= (uint32_t)kBorderCats)
                    sm.tile[w + q * kWarps][t - first] = v[q][u];
            }
    }
#pragma unroll
    for (int q = 0; q < (int)kCats; ++q) {
        const uint32_t k = w + q * kWarps;
        const uint32_t b = __reduce_add_sync(0xffffffffu, before[q]);
        const uint32_t n = __reduce_add_sync(0xffffffffu, total[q]);
        if (lane == 0 && k <= (uint32_t)kBorderCats) {
            sm.before[k] = b;
            sm.total[k] = n;
        }
    }
}
struct CtaOffs {
    const BorderCtaOffs& sm;
    uint32_t wib;
    __device__ __forceinline__ uint32_t operator()(uint32_t k) const {
        uint32_t v = sm.before[k];
        for (uint32_t t = 0; t < wib; ++t) v += sm.tile[k][t];
        return v;
    }
};

// Shared-memory scratch of one warp in pass 2: per category its members among
// the tile's lanes and the ghost index of the first, and the first ghost index
// of each swap.  Kept this small on purpose: with dependent launches an SM is
// never idle between the kernels of a step, so it keeps the split of L1 and
// shared memory of the kernel that needed most.  With every lane's index per
// category here (27 KB a CTA, 6 CTAs) the pair count and the consumer that
// follow ran on a third of the L1: k_force_csr 339 against 208 us on 4,194,304
// atoms.
struct BorderWarpSmem {
    uint32_t members[kBorderCats];
    uint32_t first[kBorderCats];
    uint32_t recv[kNumSwaps];
};

// Ghost index of a member lane's image of category k (below: the lanes before it).
__device__ __forceinline__ uint32_t image_index(const BorderWarpSmem& sm, int k, unsigned below) {
    return sm.first[k] + __popc(sm.members[k] & below);
}

// Pass 2 for warp tile w.  base_lane: on lane k < 26 the first ghost index of
// category k (nlocal + the totals of the categories before it).  off(k): the
// members of category k (k = 26: images) in the tiles before.  sm: this warp's scratch.  host_bs (optional): the host's
// copy of bs, which gets the capacity word too.  multi (optional): the roots
// with two images or more, in no particular order, counted in
// bs[kBorderMulti].
template <class Off>
__device__ __forceinline__ void border_warp_images(
    const AtomCols& c, uint64_t nlocal, uint64_t cap, const BorderCats& cats, const uint8_t* face,
    const Off& off, uint64_t w, uint32_t lane, uint32_t base_lane, uint32_t* bs, uint32_t* root, uint32_t* chain, uint32_t* const* send,
    uint32_t* fold_start, uint32_t* fold_list, BorderWarpSmem& sm, uint32_t* host_bs = nullptr,
    uint32_t* multi = nullptr) {
    const unsigned below = (1u << lane) - 1u;
    const uint64_t r = w * 32 + lane;
    const uint32_t bits = r < nlocal ? face[r] : 0u;
    const uint32_t any = __reduce_or_sync(0xffffffffu, bits);
    if (!any) {  // no images: empty fold programs
        const uint32_t fold0 = off(kBorderCats);
        if (r < nlocal) fold_start[r] = fold0;
        if (r + 1 == nlocal) fold_start[nlocal] = fold0;
        return;
    }
    // lane k <= 26: offset of this tile's members of category k (k = 26: images)
    const uint32_t off_lane = lane <= (uint32_t)kBorderCats ? off(lane) : 0u;
    const uint32_t fold0 = __shfl_sync(0xffffffffu, off_lane, kBorderCats);
    const uint32_t rv =
        __shfl_sync(0xffffffffu, base_lane, lane < (uint32_t)kNumSwaps ? cats.swap_first[lane] : 0);
    if (lane < (uint32_t)kNumSwaps) sm.recv[lane] = rv;
    const uint32_t mine_cats = cats.member[bits];
    const uint32_t own = __popc(mine_cats);  // images of this lane's root
    // only categories the tile's faces cover can have members (uniform over
    // the warp); only members read their category, and a member's parent
    // category has it as a member too
    for (uint32_t cand = cats.member[any]; cand; cand &= cand - 1) {
        const int k = __ffs(cand) - 1;
        const unsigned bal = __ballot_sync(0xffffffffu, (mine_cats >> k) & 1u);
        const uint32_t base = __shfl_sync(0xffffffffu, base_lane + off_lane, k);
        if (lane == 0) {
            sm.members[k] = bal;
            sm.first[k] = base;
        }
    }
    __syncwarp();
    const uint32_t fs = fold0 + warp_exclusive_sum(own, lane);
    if (r < nlocal) fold_start[r] = fs;
    if (r + 1 == nlocal) fold_start[nlocal] = fs + own;
    if (multi) {
        const unsigned many = __ballot_sync(0xffffffffu, own >= 2);
        uint32_t at = 0;
        if (many && lane == 0) at = atomicAdd(&bs[kBorderMulti], (uint32_t)__popc(many));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (own >= 2) multi[at + __popc(many & below)] = (uint32_t)r;
    }
    if (bits) {
        for (uint32_t mk = mine_cats; mk; mk &= mk - 1) {
            const int k = __ffs(mk) - 1;
            const uint32_t g = image_index(sm, k, below);
            if (g >= cap) {
                bs[10] = 1u;  // out of capacity: the host grows the arrays and repeats
                if (host_bs) host_bs[10] = 1u;
                continue;
            }
            const uint32_t parent =
                cats.parent[k] < 0 ? (uint32_t)r : image_index(sm, cats.parent[k], below);
            root[g - nlocal] = (uint32_t)r;
            chain[g - nlocal] = cats.code[k];
            c.origin[g] = (int32_t)parent;
            const int s = cats.swap_of[k];
            send[s][g - sm.recv[s]] = parent;
        }
        uint32_t j = fs;
        for (uint32_t mf = cats.member_fold[bits]; mf; mf &= mf - 1) {
            const int k = cats.fold[__ffs(mf) - 1];
            const uint32_t g = image_index(sm, k, below);
            if (g < cap && j < cap) fold_list[j] = g - (uint32_t)nlocal;
            ++j;
        }
    }
    __syncwarp();  // every lane is done with the scratch before the warp's next tile
}

}  // namespace soil
