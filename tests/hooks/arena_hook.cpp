// The slab allocator's host-only rules (soil_b200/csrc/arena.cuh) by plain calls.
#include "arena.cuh"

using namespace soil_host;

extern "C" {
Arena* arena_new() { return new Arena(); }
void arena_delete(Arena* a) { delete a; }
uint64_t arena_take(Arena* a, uint64_t bytes) { return (uint64_t)a->take(bytes); }
void arena_give(Arena* a, uint64_t p, uint64_t bytes) { a->give((char*)p, bytes); }
uint64_t arena_next_slab(Arena* a, uint64_t bytes) { return a->next_slab(bytes); }
uint64_t arena_add(Arena* a, uint64_t p, uint64_t size, uint64_t bytes) {
    return (uint64_t)a->add((char*)p, size, bytes);
}
// bytes that neither an array has nor a later one can get
uint64_t arena_lost(const Arena* a, uint64_t live) {
    uint64_t have = live;
    for (const auto& f : a->free) have += f.first;
    for (const auto& b : a->slabs) have += b.size - b.used;
    return a->total - have;
}

KeptSlabs* kept_new() { return new KeptSlabs(); }
void kept_delete(KeptSlabs* k) { delete k; }
int kept_give(KeptSlabs* k, uint64_t p, uint64_t size) { return k->give((char*)p, size); }
uint64_t kept_take(KeptSlabs* k, uint64_t size, uint64_t least) {
    uint64_t got;
    k->take(size, least, &got);
    return got;
}
uint64_t kept_bytes(const KeptSlabs* k) { return k->bytes; }
}
