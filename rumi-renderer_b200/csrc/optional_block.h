// A block of memory that a call can do without: grown when it is too small, and left as it is when
// the larger one cannot be had.
#pragma once
#include <cstddef>

namespace rumi {

// Grows (p, bytes) to `want` bytes: true when it holds them.  The old block is released only once the
// new one is there.  A size that was refused is not asked for again (a refusal may cost a trip through
// the driver on every call): `refused` remembers the smallest.  alloc(n): a block or nullptr.
template <typename Alloc, typename Release>
bool grow_optional(void *&p, size_t &bytes, size_t &refused, size_t want, Alloc alloc, Release release) {
    if (bytes >= want) return true;
    if (refused && want >= refused) return false;
    void *larger = alloc(want);
    if (!larger) {
        refused = want;
        return false;
    }
    if (p) release(p);
    p = larger;
    bytes = want;
    return true;
}

}  // namespace rumi
