// Every page that a byte range touches.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace fnn {

// True if `ok(address)` holds for an address of the range in each of its pages (`page`: a power of two).  Host memory is
// pinned page by page, so this decides whether all of a range is.
template <typename Pred>
inline bool every_page(uintptr_t first, size_t bytes, size_t page, Pred ok) {
    for (uintptr_t p = first; p < first + bytes; p = (p & ~(uintptr_t)(page - 1)) + page)
        if (!ok(p)) return false;
    return true;
}

}  // namespace fnn
