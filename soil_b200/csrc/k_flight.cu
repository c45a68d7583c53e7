// k_flight.cu — communicate-only steps of a system without a consumer.
//
// With no force on any atom, nothing couples two atoms in a step that keeps
// its lists: each moves on by its own velocity, and the ghosts are their
// roots' images.  Only the step at which the first displacement check trips
// is shared.  So a stretch of steps takes two plain launches, whatever its
// length and the system's size:
//
//   k_flight_find   every atom is carried forward in registers, step by step
//                   with the operations of the integration pass and its
//                   check, until its check trips; the earliest such step of
//                   all atoms is the stretch's end (one word, atomicMax);
//   k_flight_apply  every atom is carried to that step again from memory and
//                   written back, with its images (forward comm) and zero
//                   forces.
//
// Bit-identical to one integration pass and forward comm per step.  A step
// costs its arithmetic instead of a pass over the columns and a grid barrier:
// on 32,768 atoms in free flight (some ten steps between rebuilds) a stretch
// takes 6.1 + 8.0 us (the second launch with its wait for the first), where a
// step took 8.1 us in a cooperative launch with one grid barrier per step, and
// 200 steps with their 20 rebuilds went from 3.78 to 2.16 ms.
#include "device_ops.cuh"
#include "kernels.cuh"

namespace soil {

namespace {

// Atom i of a flight: its state in registers, advanced one step at a time.
struct FlightAtom {
    double x, y, z, vx, vy, vz;
    double h, fx, fy, fz;

    __device__ __forceinline__ void load(const AtomCols& c, uint64_t i, double dt) {
        h = 0.5 * dt * c.inv_mass[i];
        fx = c.fx[i];
        fy = c.fy[i];
        fz = c.fz[i];
        vx = c.vx[i];
        vy = c.vy[i];
        vz = c.vz[i];
        x = c.x[i];
        y = c.y[i];
        z = c.z[i];
    }
    // one integration pass; the forces are zero from the second on
    __device__ __forceinline__ void step(double dt, bool fuse_final) {
        initial_regs(h, dt, fuse_final, fx, fy, fz, vx, vy, vz, x, y, z);
        fx = fy = fz = 0.0;
    }
};

// Polls of the shared end step: an atom that never trips stops within this
// many steps of the earliest trip.
constexpr uint32_t kFlightPoll = 4;

}  // namespace

// *late: max_steps minus the earliest tripping step (0: none), by atomicMax.
__global__ void __launch_bounds__(kBlock) k_flight_find(FlightArgs a) {
    const uint32_t max = a.max_steps;
    uint32_t mine = 0;  // of this thread's atoms
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < a.nlocal;
         i += (uint64_t)gridDim.x * blockDim.x) {
        FlightAtom p;
        p.load(a.c, i, a.dt);
        const double lx = a.ck.lbx[i], ly = a.ck.lby[i], lz = a.ck.lbz[i];
        uint32_t end = max - mine;  // steps worth looking at
        for (uint32_t s = 0; s < end; ++s) {
            if (s % kFlightPoll == 0) {
                const uint32_t late = *(volatile uint32_t*)a.late;
                if (max - late < end) end = max - late;
                if (s >= end) break;
            }
            p.step(a.dt, s > 0 || a.first_fused);
            if (check_moved_at(a.ck, p.x, p.y, p.z, lx, ly, lz)) {
                mine = max - s;
                atomicMax(a.late, mine);
                break;
            }
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_flight_apply(FlightArgs a) {
    pdl_wait();  // launched with pdl_launch
    const uint32_t late = *a.late;
    const uint32_t done = a.max_steps - late;      // completed steps
    const uint32_t passes = done + (late ? 1 : 0);  // the tripped step is integrated too
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.next_late = 0u;  // the next flight's word
        a.out[0] = done;
        a.out[1] = late ? 1u : 0u;
    }
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < a.nlocal;
         i += (uint64_t)gridDim.x * blockDim.x) {
        FlightAtom p;
        p.load(a.c, i, a.dt);
        for (uint32_t s = 0; s < passes; ++s) p.step(a.dt, s > 0 || a.first_fused);
        a.c.vx[i] = p.vx;
        a.c.vy[i] = p.vy;
        a.c.vz[i] = p.vz;
        a.c.x[i] = p.x;
        a.c.y[i] = p.y;
        a.c.z[i] = p.z;
        a.c.fx[i] = 0.0;
        a.c.fy[i] = 0.0;
        a.c.fz[i] = 0.0;
        forward_images(a.c, a.nlocal, i, p.x, p.y, p.z, p.vx, p.vy, p.vz, a.fw.fold_start,
                       a.fw.fold_list, a.fw.chain, a.fw.sc, a.fw.fwd, true);
    }
}

void launch_flight(cudaStream_t st, const FlightArgs& a) {
    note_launch();
    k_flight_find<<<grid_wave<k_flight_find>(a.nlocal), kBlock, 0, st>>>(a);
    note_launch();
    pdl_launch(k_flight_apply, grid_wave<k_flight_apply>(a.nlocal), kBlock, 0, st, a);
}

}  // namespace soil
