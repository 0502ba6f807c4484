// grow_shim.cpp — test harness only: a growing buffer over a host allocator that
// can be told to fail, compiled with the host compiler.
#include <cstdint>
#include <cstdlib>
#include <new>

#include "../turbotops_gb300/csrc/tt_grow.h"

static tt::Grown g;
static int live = 0;

// 0: the buffer holds `want` bytes; 1: the allocation failed. *bytes: its size, *held: memory in use.
extern "C" int grow(uint64_t want, int fail, uint64_t* bytes, int* held) {
    int r = 0;
    try {
        void* p = g.get(want,
                        [&](size_t n) -> void* {
                            if (fail) throw std::bad_alloc();
                            ++live;
                            return std::malloc(n);
                        },
                        [&](void* q) {
                            --live;
                            std::free(q);
                        });
        r = p == nullptr && want > 0 ? 2 : 0;
    } catch (const std::bad_alloc&) {
        r = 1;
    }
    *bytes = g.bytes;
    *held = live;
    return r;
}
