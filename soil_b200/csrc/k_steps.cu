// k_steps.cu — device-resident communicate-only steps.
//
// The reference decides every step whether the lists must be rebuilt
// (decide_rebuild, crates/soil_core/src/neighbor.rs:796-822); its GPU
// prototype runs K resident steps with no host read in between
// (crates/soil_gpu/src/gpu_state.rs:352-418).  k_steps runs consecutive steps
// that keep their lists in ONE cooperative launch.
//
// What bounds such a step on a system of up to ~150,000 atoms is latency:
// dependent loads through L2, the FP64 square root and divide of a pair, the
// grid barrier.  So:
//
//   - A group of G lanes (8, 4, 2 or 1: as many as keep the whole system in
//     one CTA per SM) owns one root for the whole launch.  Its position,
//     velocity, build position and mass stay in registers.
//   - The root's partner entries and those of its ghost images, in the
//     reference's summation order (CsrIdx order, the images in fold order),
//     are copied once per launch into shared memory.  Each step the lanes
//     evaluate G entries at a time and every lane adds the results in entry
//     order (shuffles), so the sums are those of the one-thread walk.  Image
//     forces go to shared memory and are folded by the group's first lane in
//     fold_root's order; with 8 lanes and at most 7 images per root, lane j
//     keeps its j-th image's position and force sum in registers instead and
//     the fold is a few shuffles (FEW: the roots at the box's corners, with
//     seven images, set the time of a step).
//   - Positions are exchanged as packed (x, y, z, r) records in two buffers
//     used in turn: a step reads one while the next step's integration, by
//     the same threads, writes the other.  One grid barrier per step, not
//     two.
//   - The barrier word carries the displacement check: an arrival adds 1, and
//     2^32 if an atom of the CTA moved too far; three words in rotation, the
//     one of the last step cleared by CTA 0 (its pollers have all arrived at
//     the next).
//
// The launch ends after max_steps or when a check trips; then (and only then)
// the columns of locals and ghosts are written.  Each step runs the same
// per-atom operations in the same order as the launch-per-phase path, so
// results are bit-identical.  A CTA whose entries or images do not fit its
// shared memory says so at the first barrier, and every CTA leaves with
// nothing written; the host learns what the CTA that has most needs, and
// launches again with room for that or not at all.  Barrier waits are bounded:
// a CTA whose wait runs out records SOIL_STEPS_ERR_BARRIER and returns; the
// cooperative launch guarantees co-residency, so the bound is a guard, never
// the expected exit.
//
// Measured per light step against one thread per root walking the CSR with
// its images in series, columns in global memory and two barriers a step:
// 3.2 against 22 us on 1,000 atoms, 11 against 32 us on 65,537.
#include <cuda/atomic>

#include "device_ops.cuh"
#include "force_ops.cuh"
#include "kernels.cuh"

namespace soil {

namespace {

// Spins of a barrier wait (each >= 100 ns of __nanosleep): about a second.
constexpr uint64_t kBarrierSpinLimit = 1ull << 23;

using Word = unsigned long long;
constexpr Word kTripUnit = 1ull << 32;  // added by a CTA whose check tripped
constexpr Word kOverUnit = 1ull << 48;  // added by a CTA whose lists do not fit
constexpr uint16_t kRootParent = 0xffffu;

// Arrive at `w` with `add` and wait for nb arrivals; *seen gets the word.
__device__ bool arrive_and_wait(Word* w, unsigned nb, Word add, Word* seen) {
    cuda::atomic_ref<Word, cuda::thread_scope_device> a(*w);
    Word v = a.fetch_add(add, cuda::memory_order_acq_rel) + add;
    for (uint64_t spins = 0; (uint32_t)v < nb; ++spins) {
        if (spins > kBarrierSpinLimit) return false;
        if (spins > 1024) __nanosleep(100);  // a short busy wait first
        v = a.load(cuda::memory_order_acquire);
    }
    *seen = v;
    return true;
}

// Exclusive scan over the CTA of two counts packed in one word (low and high
// 32 bits); *total gets the CTA's sums.
__device__ uint64_t cta_exclusive_pair(uint64_t v, uint64_t* total) {
    __shared__ uint64_t wsum[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint64_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint64_t w = lane < nw ? wsum[lane] : 0, wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        wsum[lane] = wi - w;
        if (lane == 31) wsum[32] = wi;
    }
    __syncthreads();
    *total = wsum[32];
    return wsum[warp] + inc - v;
}

// Shared memory of one CTA for e entries and m images.
struct StepsSmem {
    double* fimg;    // 3 per image: its force
    double* irad;    // its radius
    uint32_t* ent;   // partner of each entry
    uint32_t* ig;    // ghost index (minus nlocal) of each image
    uint32_t* iend;  // one past its last entry
    uint16_t* code;  // its swap chain
    uint16_t* par;   // image slot of its origin, or kRootParent
    uint8_t* eown;   // item of each entry: 0 the root, j its j-th image
};

// What only the integration needs of a thread's atom: in registers, or (PARK)
// in shared memory where 1,024 threads leave 64 registers each.
template <bool PARK>
struct Parked {
    double vx, vy, vz, h, lx, ly, lz;
    __device__ __forceinline__ void bind(double*) {}
    __device__ __forceinline__ Parked& get() { return *this; }
    __device__ __forceinline__ void put(const Parked&) {}
};
template <>
struct Parked<true> {
    double* p;  // this thread's, one per kind every blockDim.x
    __device__ __forceinline__ void bind(double* base) { p = base + threadIdx.x; }
    __device__ __forceinline__ Parked<false> get() const {
        const unsigned n = blockDim.x;
        return {p[0], p[n], p[2 * n], p[3 * n], p[4 * n], p[5 * n], p[6 * n]};
    }
    __device__ __forceinline__ void put(const Parked<false>& v) {
        const unsigned n = blockDim.x;
        p[0] = v.vx;
        p[n] = v.vy;
        p[2 * n] = v.vz;
    }
    __device__ __forceinline__ void set(const Parked<false>& v) {
        const unsigned n = blockDim.x;
        put(v);
        p[3 * n] = v.h;
        p[4 * n] = v.lx;
        p[5 * n] = v.ly;
        p[6 * n] = v.lz;
    }
};

__device__ StepsSmem carve(unsigned char* p, uint32_t e, uint32_t m) {
    StepsSmem s;
    s.fimg = reinterpret_cast<double*>(p);
    s.irad = s.fimg + 3 * m;
    s.ent = reinterpret_cast<uint32_t*>(s.irad + m);
    s.ig = s.ent + e;
    s.iend = s.ig + m;
    s.code = reinterpret_cast<uint16_t*>(s.iend + m);
    s.par = s.code + m;
    s.eown = reinterpret_cast<uint8_t*>(s.par + m);
    return s;
}

// Position (or velocity) of an image: its root's plus its chain's offsets, in
// chain order (forward_images).
__device__ __forceinline__ void shift_chain(uint32_t code, const double (*off)[3], double& x,
                                            double& y, double& z) {
    const uint32_t len = code >> 12;
    for (uint32_t k = 0; k < len; ++k) {
        const int s = (code >> (3 * k)) & 7;
        x = x + off[s][0];
        y = y + off[s][1];
        z = z + off[s][2];
    }
}

}  // namespace

// FOLD: newton, with the reverse fold; else only locals receive and the
// ghosts' forces are zero.
template <int G, bool FOLD, int TMAX, bool FEW>
__global__ void __launch_bounds__(TMAX, 1) k_steps(const __grid_constant__ StepsArgs a) {
    static_assert(!FEW || G == 8, "an item per lane");
    constexpr bool kPark = TMAX > (int)kStepsParkAbove;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Word s_seen;
    __shared__ int s_ok;
    const StepsSmem sm =
        carve(smem_raw + (kPark ? blockDim.x * kBytesParked : 0), a.ent_cap, a.img_cap);
    const AtomCols& c = a.c;
    const uint64_t nl = a.nlocal;
    const uint32_t g = threadIdx.x & (G - 1);
    const uint64_t t = (uint64_t)blockIdx.x * (blockDim.x / G) + threadIdx.x / G;
    const bool valid = t < nl;
    const bool lead = valid && g == 0;

    // ---- the group's lists -----------------------------------------------------
    uint32_t f0 = 0, nimg = 0, qs = 0, nin = 0, npre = 0, rs = 0, nrow = 0, cnt = 0;
    if (valid) {
        f0 = a.fc.fold_start[t];
        nimg = a.fc.fold_start[t + 1] - f0;
        qs = a.fc.in_start[t];
        nin = a.fc.in_start[t + 1] - qs;
        npre = a.fc.in_split[t];
        rs = a.fc.offsets[t];
        nrow = a.fc.offsets[t + 1] - rs;
        cnt = nin + nrow;
        if (FOLD)
            for (uint32_t q = 0; q < nimg; ++q) {
                const uint64_t gi = nl + a.fc.fold_list[f0 + q];
                cnt += a.fc.in_start[gi + 1] - a.fc.in_start[gi];
            }
    }
    uint64_t tot;
    const uint64_t at = cta_exclusive_pair(lead ? ((uint64_t)nimg << 32) | cnt : 0u, &tot);
    const bool over = (uint32_t)tot > a.ent_cap || (uint32_t)(tot >> 32) > a.img_cap;
    if (threadIdx.x == 0) {  // read by CTA 0 after the first barrier
        atomicMax(a.need, (uint32_t)tot);
        atomicMax(a.need + 1, (uint32_t)(tot >> 32));
    }
    // the first lane's prefix is its whole group's (the other lanes' counts are 0)
    const uint64_t at0 = __shfl_sync(0xffffffffu, at, 0, G);
    const uint32_t eb = (uint32_t)at0, ib = (uint32_t)(at0 >> 32);
    if (over) nimg = cnt = nin = nrow = npre = 0;
    // FEW: this lane's image (lane 0: the root itself)
    uint32_t my_gi = 0, my_code = 0, my_par = 0;
    double my_rad = 0.0;
    const bool has_item = valid && g <= nimg;
    const uint32_t ee = eb + cnt, e0 = eb + nin + nrow;
    for (uint32_t k = g; k < nin + nrow; k += G) {
        sm.ent[eb + k] = k < npre          ? a.fc.in_list[qs + k]
                         : k < npre + nrow ? a.fc.indices[rs + (k - npre)]
                                           : a.fc.in_list[qs + (k - nrow)];
        sm.eown[eb + k] = 0;
    }
    uint32_t k0 = e0;
    for (uint32_t q = 0; q < nimg; ++q) {
        const uint32_t gi = a.fc.fold_list[f0 + q];
        if (FOLD) {
            const uint32_t b = a.fc.in_start[nl + gi], n = a.fc.in_start[nl + gi + 1] - b;
            for (uint32_t k = g; k < n; k += G) {
                sm.ent[k0 + k] = a.fc.in_list[b + k];
                sm.eown[k0 + k] = (uint8_t)(q + 1);
            }
            k0 += n;
        }
        if (g == (FEW ? q + 1 : 0)) {
            for (int p = 0; p < a.fw.fwd.n; ++p)  // the first step's forward planes
                c.planes[a.fw.fwd.idx[p]][nl + gi] = c.planes[a.fw.fwd.idx[p]][t];
            const uint32_t code = a.fw.chain[gi];
            const double rad = a.fc.rad[nl + gi];
            const uint32_t o = (uint32_t)c.origin[nl + gi];
            uint32_t par = kRootParent;
            if (o >= nl)  // an image one chain shorter of the same root
                for (uint32_t r = 0; r < nimg; ++r)
                    if (a.fc.fold_list[f0 + r] == o - (uint32_t)nl) par = FEW ? r + 1 : ib + r;
            if (FEW) {
                my_gi = gi;
                my_code = code;
                my_rad = rad;
                my_par = par == kRootParent ? 0 : par;
            } else {
                sm.ig[ib + q] = gi;
                sm.iend[ib + q] = k0;
                sm.code[ib + q] = (uint16_t)code;
                sm.irad[ib + q] = rad;
                sm.par[ib + q] = (uint16_t)par;
            }
        }
    }
    const uint32_t rounds = __reduce_max_sync(0xffffffffu, (cnt + G - 1) / G);

    const uint32_t most_images = FEW ? __reduce_max_sync(0xffffffffu, nimg) : 0u;

    // ---- the group's atom ------------------------------------------------------
    double x = 0, y = 0, z = 0, Rx = 0, Ry = 0, Rz = 0, r = 0;
    Parked<kPark> parked;
    parked.bind(reinterpret_cast<double*>(smem_raw));
    {
        Parked<false> w{};
        if (valid) {
            w.h = 0.5 * a.dt * c.inv_mass[t];
            w.vx = c.vx[t];
            w.vy = c.vy[t];
            w.vz = c.vz[t];
            w.lx = a.ck.lbx[t];
            w.ly = a.ck.lby[t];
            w.lz = a.ck.lbz[t];
            x = c.x[t];
            y = c.y[t];
            z = c.z[t];
            Rx = c.fx[t];
            Ry = c.fy[t];
            Rz = c.fz[t];
            r = a.fc.rad[t];
        }
        if constexpr (kPark) parked.set(w);
        else parked = w;
    }
    if (g == 0) my_rad = r;
    double ix = 0, iy = 0, iz = 0;  // FEW: this lane's item
    double Ix = 0, Iy = 0, Iz = 0;  // FEW: its force
    __syncwarp();

    uint64_t done = 0;
    bool stop = false;
    for (uint64_t step = 0; step < a.max_steps; ++step) {
        // integrate (the previous step's final half-kick first), check, and
        // publish the new positions
        double* const rec = a.rec[step & 1];
        bool hit;
        {
            auto w = parked.get();
            initial_regs(w.h, a.dt, step > 0 || a.first_fused, Rx, Ry, Rz, w.vx, w.vy, w.vz, x, y, z);
            hit = valid && check_moved_at(a.ck, x, y, z, w.lx, w.ly, w.lz);
            if constexpr (kPark) parked.put(w);
            else parked = w;
        }
        if (FEW) {
            ix = x;
            iy = y;
            iz = z;
            shift_chain(my_code, a.fw.sc.off, ix, iy, iz);  // the root's chain is empty
            if (has_item) put_pk(rec, g ? nl + my_gi : t, ix, iy, iz, my_rad);
        } else {
            if (lead) put_pk(rec, t, x, y, z, r);
            for (uint32_t q = g; q < nimg; q += G) {
                double px = x, py = y, pz = z;
                shift_chain(sm.code[ib + q], a.fw.sc.off, px, py, pz);
                put_pk(rec, nl + sm.ig[ib + q], px, py, pz, sm.irad[ib + q]);
            }
        }
        if (a.rev.n && step > 0 && lead)  // forward planes a fold has changed
            for (uint32_t q = f0; q < f0 + nimg; ++q)
                for (int p = 0; p < a.fw.fwd.n; ++p)
                    c.planes[a.fw.fwd.idx[p]][nl + a.fc.fold_list[q]] = c.planes[a.fw.fwd.idx[p]][t];
        const int any = __syncthreads_or(hit);
        if (threadIdx.x == 0) {
            const Word add = 1u + (any ? kTripUnit : 0u) + (over ? kOverUnit : 0u);
            const uint64_t e = a.epoch + step;
            Word seen = 0;
            s_ok = arrive_and_wait(a.bar + e % 3, gridDim.x, add, &seen);
            s_seen = seen;
            if (!s_ok) *(volatile uint32_t*)(a.out + 3) = SOIL_STEPS_ERR_BARRIER;
            // every CTA has left the word of the step before
            if (blockIdx.x == 0)
                cuda::atomic_ref<Word, cuda::thread_scope_device>(a.bar[(e + 2) % 3])
                    .store(0u, cuda::memory_order_relaxed);
        }
        __syncthreads();
        const Word seen = s_seen;
        if (!s_ok || seen >= kOverUnit) {  // nothing is written
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                for (int k = 0; k < 2; ++k) a.out[4 + k] = atomicExch(a.need + k, 0u);
                a.out[2] = s_ok ? SOIL_STEPS_OVERFLOW : SOIL_STEPS_ERR_BARRIER;
            }
            return;
        }
        if (seen >= kTripUnit) {
            stop = true;
            break;
        }
        // the consumer: G entries at a time, added in entry order
        double Fx = 0.0, Fy = 0.0, Fz = 0.0;
        uint32_t item = 0, iend = e0;
        auto close = [&] {  // (not FEW) the item is complete
            if (item == 0) {
                Rx = Fx;
                Ry = Fy;
                Rz = Fz;
            } else if (g == 0) {
                double* f = sm.fimg + 3 * (ib + item - 1);
                f[0] = Fx;
                f[1] = Fy;
                f[2] = Fz;
            }
            Fx = Fy = Fz = 0.0;
            ++item;
            iend = item <= nimg ? sm.iend[ib + item - 1] : 0xffffffffu;
        };
        // (the next entry's record loaded one trip ahead measured slower: 17.2
        // against 15.4 us a step on 140,000 atoms)
        for (uint32_t rd = 0; rd < rounds; ++rd) {
            const uint32_t k = eb + rd * G + g;
            double fx = 0.0, fy = 0.0, fz = 0.0;
            bool touch = false;
            uint32_t own = 0;
            double4 q;
            if (k < ee) {
                own = FOLD ? sm.eown[k] : 0u;
                q = ld_pk(rec, sm.ent[k]);
            }
            double px = x, py = y, pz = z, pr = r;
            if (FEW && FOLD) {
                px = __shfl_sync(0xffffffffu, ix, own, 8);
                py = __shfl_sync(0xffffffffu, iy, own, 8);
                pz = __shfl_sync(0xffffffffu, iz, own, 8);
                pr = __shfl_sync(0xffffffffu, my_rad, own, 8);
            } else if (FOLD && own) {
                shift_chain(sm.code[ib + own - 1], a.fw.sc.off, px, py, pz);
                pr = sm.irad[ib + own - 1];
            }
            if (k < ee) touch = pair_force(px, py, pz, pr, q.x, q.y, q.z, q.w, a.fc.K, fx, fy, fz);
            const unsigned hits = __ballot_sync(0xffffffffu, touch) >> ((threadIdx.x & 31) & ~(G - 1));
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const double ex = G > 1 ? __shfl_sync(0xffffffffu, fx, j, G) : fx;
                const double ey = G > 1 ? __shfl_sync(0xffffffffu, fy, j, G) : fy;
                const double ez = G > 1 ? __shfl_sync(0xffffffffu, fz, j, G) : fz;
                // FEW: each lane sums its own item (the shuffle is every lane's)
                const uint32_t item_j = FEW && FOLD ? __shfl_sync(0xffffffffu, own, j, G) : g;
                const bool add = ((hits >> j) & 1u) && item_j == g;
                if (FOLD && !FEW) {
                    const uint32_t kk = eb + rd * G + j;
                    if (kk < ee)
                        while (kk >= iend) close();
                }
                if (add) {
                    Fx = Fx + ex;
                    Fy = Fy + ey;
                    Fz = Fz + ez;
                }
            }
        }
        if (FEW && FOLD) {  // fold_root's order: image by image onto its parent's lane
            for (uint32_t j = 1; j <= most_images; ++j) {
                const double ex = __shfl_sync(0xffffffffu, Fx, j, 8);
                const double ey = __shfl_sync(0xffffffffu, Fy, j, 8);
                const double ez = __shfl_sync(0xffffffffu, Fz, j, 8);
                const uint32_t p = __shfl_sync(0xffffffffu, my_par, j, 8);
                if (j <= nimg && p == g) {
                    Fx = Fx + ex;
                    Fy = Fy + ey;
                    Fz = Fz + ez;
                }
            }
            Ix = Fx;
            Iy = Fy;
            Iz = Fz;
        } else if (FOLD) {
            while (item <= nimg) close();
            if (nimg && g == 0)  // fold_root's order
                for (uint32_t q = ib; q < ib + nimg; ++q) {
                    const double* f = sm.fimg + 3 * q;
                    const uint32_t p = sm.par[q];
                    if (p == kRootParent) {
                        Rx = Rx + f[0];
                        Ry = Ry + f[1];
                        Rz = Rz + f[2];
                    } else {
                        double* o = sm.fimg + 3 * p;
                        o[0] = o[0] + f[0];
                        o[1] = o[1] + f[1];
                        o[2] = o[2] + f[2];
                    }
                }
        } else {
            Rx = Fx;
            Ry = Fy;
            Rz = Fz;
        }
        if (FOLD && G > 1) {  // the root's sum to the whole group
            __syncwarp();
            Rx = __shfl_sync(0xffffffffu, FEW ? Fx : Rx, 0, G);
            Ry = __shfl_sync(0xffffffffu, FEW ? Fy : Ry, 0, G);
            Rz = __shfl_sync(0xffffffffu, FEW ? Fz : Rz, 0, G);
        }
        if (FOLD && a.rev.n && lead)
            for (uint32_t q = f0; q < f0 + nimg; ++q) {
                const uint64_t gh = nl + a.fc.fold_list[q];
                const uint32_t o = (uint32_t)c.origin[gh];
                for (int w = 0; w < a.rev.n; ++w) {
                    double* pl = c.planes[a.rev.idx[w]];
                    pl[o] = pl[o] + pl[gh];
                }
            }
        ++done;
    }

    // ---- the columns -----------------------------------------------------------
    const auto w = parked.get();
    if (lead) {
        c.x[t] = x;
        c.y[t] = y;
        c.z[t] = z;
        c.vx[t] = w.vx;
        c.vy[t] = w.vy;
        c.vz[t] = w.vz;
        c.fx[t] = Rx;
        c.fy[t] = Ry;
        c.fz[t] = Rz;
    }
    __syncwarp();
    for (uint32_t q = FEW ? g - 1 : g; q < nimg; q += G) {  // (FEW, lane 0: no image)
        const uint64_t gi = nl + (FEW ? my_gi : sm.ig[ib + q]);
        const uint32_t code = FEW ? my_code : sm.code[ib + q];
        double px = x, py = y, pz = z, ux = w.vx, uy = w.vy, uz = w.vz;
        shift_chain(code, a.fw.sc.off, px, py, pz);
        shift_chain(code, a.fw.sc.voff, ux, uy, uz);
        c.x[gi] = px;
        c.y[gi] = py;
        c.z[gi] = pz;
        c.vx[gi] = ux;
        c.vy[gi] = uy;
        c.vz[gi] = uz;
        if (done) {
            const double* f = FEW ? nullptr : sm.fimg + 3 * (ib + q);
            c.fx[gi] = !FOLD ? 0.0 : FEW ? Ix : f[0];
            c.fy[gi] = !FOLD ? 0.0 : FEW ? Iy : f[1];
            c.fz[gi] = !FOLD ? 0.0 : FEW ? Iz : f[2];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = (uint32_t)done;
        a.out[1] = stop ? 1u : 0u;
        a.out[2] = 0u;
        for (int k = 0; k < 2; ++k) a.out[4 + k] = atomicExch(a.need + k, 0u);
    }
}

namespace {

template <int G, int TMAX, bool FEW = false>
const void* steps_kernel(bool fold) {
    return fold ? (const void*)k_steps<G, true, TMAX, FEW> : (const void*)k_steps<G, false, TMAX, FEW>;
}

}  // namespace

cudaError_t launch_steps(cudaStream_t st, const StepsArgs& a, const StepsShape& p, bool fold,
                         bool few_images) {
    const void* k;
    if (p.group == 8 && p.threads <= (int)kStepsParkAbove)
        k = few_images ? steps_kernel<8, 256, true>(fold) : steps_kernel<8, 256>(fold);
    else if (p.group == 8)
        k = few_images ? steps_kernel<8, 1024, true>(fold) : steps_kernel<8, 1024>(fold);
    else if (p.group == 4) k = steps_kernel<4, 1024>(fold);
    else if (p.group == 2) k = steps_kernel<2, 1024>(fold);
    else k = steps_kernel<1, 1024>(fold);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)p.smem);
    if (e != cudaSuccess) return e;
    StepsArgs arg = a;
    void* params[] = {&arg};
    e = cudaLaunchCooperativeKernel(k, dim3(p.grid), dim3(p.threads), params, p.smem, st);
    if (e == cudaSuccess) note_launch();
    return e;
}

}  // namespace soil
