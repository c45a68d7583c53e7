// arena.cuh — host only: the places of a system's arrays in its slabs of device
// memory, and the slabs that closed systems leave to the next ones.
#pragma once

#include <algorithm>
#include <cstdint>
#include <map>
#include <vector>

namespace soil_host {

// Device memory of one system: its arrays are cut from a few slabs of the
// context's pool, each as large as all before it together, because a driver call
// per array costs microseconds (milliseconds once many streams share the
// pool: the first step of 128 boxes spent a second in 8,000 of them).  What
// an array gives back serves the system's next arrays, in the order of its one
// stream.  Arrays above kArenaMax, and every array of a context with a budget,
// come from the pool directly.  Sizes are multiples of 256.
constexpr uint64_t kArenaMax = 8ull << 20;
constexpr uint64_t kSlabMin = 1ull << 20, kSlabMax = 32ull << 20;

struct Arena {
    struct Slab {
        char* p;
        uint64_t size, used;
    };
    std::vector<Slab> slabs;
    std::multimap<uint64_t, char*> free;  // by size
    uint64_t total = 0;

    // A block that an array gave back (not much larger, so that the large ones
    // stay whole; the rest of it stays free), else the next bytes of a slab;
    // nullptr: no room.
    char* take(uint64_t bytes) {
        const auto it = free.lower_bound(bytes);
        if (it != free.end() && it->first <= bytes + bytes / 2 + 4096) {
            char* p = it->second;
            const uint64_t rest = it->first - bytes;
            free.erase(it);
            if (rest) free.emplace(rest, p + bytes);
            return p;
        }
        for (size_t k = slabs.size(); k-- > 0;) {
            Slab& b = slabs[k];
            if (b.size - b.used >= bytes) {
                char* p = b.p + b.used;
                b.used += bytes;
                return p;
            }
        }
        return nullptr;
    }
    void give(char* p, uint64_t bytes) { free.emplace(bytes, p); }
    uint64_t next_slab(uint64_t bytes) const {
        return std::max(bytes, std::min(std::max(total, kSlabMin), kSlabMax));
    }
    // A new slab, its first `bytes` taken.
    char* add(char* p, uint64_t size, uint64_t bytes) {
        slabs.push_back({p, size, bytes});
        total += size;
        return p;
    }
};

// Slabs of systems that are gone, at most kKeptSlabBytes of them.
constexpr uint64_t kKeptSlabBytes = 512ull << 20;

struct KeptSlabs {
    std::multimap<uint64_t, char*> slabs;  // by size
    uint64_t bytes = 0;

    bool give(char* p, uint64_t size) {
        if (bytes + size > kKeptSlabBytes) return false;
        slabs.emplace(size, p);
        bytes += size;
        return true;
    }
    // One of at least `size` bytes, or else of at least `least`, but of no more
    // than twice `size`: a system of 1 MB does not hold 32.  Its size goes to *got
    // (0: none).
    char* take(uint64_t size, uint64_t least, uint64_t* got) {
        auto it = slabs.lower_bound(size);
        if (it == slabs.end() || it->first > 2 * size) it = slabs.lower_bound(least);
        *got = 0;
        if (it == slabs.end() || it->first > 2 * size) return nullptr;
        char* p = it->second;
        *got = it->first;
        bytes -= it->first;
        slabs.erase(it);
        return p;
    }
};

}  // namespace soil_host
