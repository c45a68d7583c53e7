// steps_shape.cuh — host only: the launch shape of the resident light steps
// (k_steps.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace soil {

// Launch shape of k_steps: lanes per root, threads per CTA, CTAs (one per SM),
// and the shared memory for ent_cap entries and img_cap images.
struct StepsShape {
    int group, threads, grid;
    uint32_t ent_cap, img_cap;
    size_t smem;
};

// Entries and images of the CTA that has most, as a launch reported them
// (0: not known).
struct StepsNeed {
    uint32_t ent = 0, img = 0;
};

// Shared memory of an entry, of an image, and of what a thread parks of its atom
// where its CTA has more than 256.
constexpr uint64_t kBytesPerImage = 3 * 8 + 8 + 4 + 4 + 2 + 2;
constexpr uint64_t kBytesPerEntry = 4 + 1;
constexpr uint64_t kBytesParked = 7 * 8;
constexpr uint64_t kStepsThreads = 1024, kStepsParkAbove = 256, kStepsSmem = 220 * 1024;

// Largest system of one resident launch on `sms` SMs.
constexpr uint64_t steps_max_roots(uint64_t sms) { return sms * kStepsThreads; }

// Lanes per root: the widest group with the whole system in one CTA per SM.
inline int steps_group(uint64_t nlocal, uint64_t sms) {
    for (int g = 8; g > 1; g /= 2)
        if (nlocal * (uint64_t)g <= steps_max_roots(sms)) return g;
    return 1;
}

// The shape for a system on `sms` SMs; false when it has too many atoms for one
// resident launch, or its lists need more shared memory than a CTA has.
// Without a need, a CTA has room for 1.3 times the mean entries per root and 1.5
// images per root (on a face of the box it has a little over one).  With one it
// has room for that and an eighth more (lists change from build to build), and
// where both do not fit, for what is needed of images and entries for the rest.
inline bool steps_shape(uint64_t nlocal, uint64_t npairs, uint64_t sms, const StepsNeed& need,
                        StepsShape* p) {
    if (nlocal == 0 || nlocal > steps_max_roots(sms)) return false;
    p->group = steps_group(nlocal, sms);
    const uint64_t lanes = nlocal * (uint64_t)p->group;
    const uint64_t threads = std::max<uint64_t>(64, ((lanes + sms - 1) / sms + 31) / 32 * 32);
    p->threads = (int)threads;
    const uint64_t roots = threads / (uint64_t)p->group;
    p->grid = (int)((nlocal + roots - 1) / roots);
    const uint64_t park = threads > kStepsParkAbove ? threads * kBytesParked : 0;
    const uint64_t room = kStepsSmem - park;
    const double mean = 2.0 * (double)npairs / (double)nlocal * (double)roots;
    const auto more = [](uint64_t v) { return v + v / 8; };
    uint64_t img = std::max(roots + roots / 2 + 64, more(need.img));
    uint64_t ent = std::max((uint64_t)(1.3 * mean) + 16 * roots / 8 + 256, more(need.ent));
    img = std::min(img, 26 * roots);
    if (img * kBytesPerImage + ent * kBytesPerEntry > room) {
        if (need.ent) img = need.img;
        if (img * kBytesPerImage > room) return false;
        ent = (room - img * kBytesPerImage) / kBytesPerEntry;
    }
    p->ent_cap = (uint32_t)((ent + 7) / 8 * 8);
    if (p->ent_cap * kBytesPerEntry + img * kBytesPerImage > room) p->ent_cap -= 8;
    p->img_cap = (uint32_t)img;
    p->smem = park + img * kBytesPerImage + p->ent_cap * kBytesPerEntry + 16;
    return p->ent_cap >= need.ent;
}

}  // namespace soil
