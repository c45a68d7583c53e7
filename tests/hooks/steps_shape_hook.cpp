// The launch shape of the resident steps (soil_b200/csrc/steps_shape.cuh) by a
// plain call.
#include "steps_shape.cuh"

extern "C" int shape_of(uint64_t nlocal, uint64_t npairs, uint64_t sms, uint32_t ent, uint32_t img,
                        uint64_t out[6]) {
    soil::StepsShape p{};
    soil::StepsNeed need;
    need.ent = ent;
    need.img = img;
    const bool ok = soil::steps_shape(nlocal, npairs, sms, need, &p);
    const uint64_t v[6] = {(uint64_t)p.group, (uint64_t)p.threads, (uint64_t)p.grid,
                           p.ent_cap, p.img_cap, p.smem};
    for (int k = 0; k < 6; ++k) out[k] = v[k];
    return ok;
}
