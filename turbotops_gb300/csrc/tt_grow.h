// tt_grow.h — a buffer that only grows. Where the allocation fails, nothing is
// left behind: no size without memory.
#pragma once
#include <cstddef>

namespace tt {

struct Grown {
    void* p = nullptr;
    size_t bytes = 0;
    // alloc(bytes): the memory, or throws; free(p)
    template <typename Alloc, typename Free>
    void* get(size_t want, Alloc&& alloc, Free&& free) {
        if (bytes < want) {
            if (p) free(p);
            p = nullptr;
            bytes = 0;
            p = alloc(want);
            bytes = want;
        }
        return p;
    }
};

}  // namespace tt
