// How an arena's device memory grows (engine.h, Arena), for host tests.
#ifndef NSP_ARENA_PLAN_H
#define NSP_ARENA_PLAN_H

#include <algorithm>
#include <cstddef>

namespace nsp {

// The size of the chunk after one of `last` bytes (0: the first): twice that,
// 64 MB to 1 GB, so a small build holds little and a large one needs few; at
// least the `n` bytes asked for.
inline size_t arena_chunk(size_t last, size_t n) {
    size_t cap = size_t{64} << 20;
    if (last > 0) cap = std::min(std::max(cap, 2 * last), size_t{1} << 30);
    return std::max(cap, n);
}

// A chunk of `cap` bytes by allocate(bytes) -> pointer, null when there is no
// room; then one of the `n` bytes asked for alone, so that the reserve does not
// refuse what the device holds. `cap` becomes the chunk's size.
template <class Allocate>
void* arena_allocate(size_t& cap, size_t n, Allocate allocate) {
    void* p = allocate(cap);
    if (p == nullptr && n < cap) {
        cap = n;
        p = allocate(cap);
    }
    return p;
}

}  // namespace nsp

#endif  // NSP_ARENA_PLAN_H
