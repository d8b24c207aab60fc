// Host build of grow_optional (optional_block.h) over a counting allocator with a limit.  Test
// infrastructure, not part of the library.
#include "../../rumi-renderer_b200/csrc/optional_block.h"
#include <cstdlib>

static size_t limit_bytes;
static int asked, released;
static void *held;
static size_t held_bytes, refused;

extern "C" {
void block_reset(size_t limit) {
    free(held);
    held = nullptr;
    held_bytes = refused = 0;
    asked = released = 0;
    limit_bytes = limit;
}
int block_grow(size_t want) {
    return rumi::grow_optional(
        held, held_bytes, refused, want,
        [](size_t n) -> void * {
            ++asked;
            return n <= limit_bytes ? malloc(n) : nullptr;
        },
        [](void *p) {
            ++released;
            free(p);
        });
}
size_t block_bytes() { return held_bytes; }
int block_asked() { return asked; }
int block_released() { return released; }
}
