// arena.h - arrays laid out in one block of device memory; plain C++ (tested without a device).
#pragma once
#include <algorithm>
#include <cstddef>
#include <functional>

namespace lam {

// Allocates `bytes`; 0 on success.
typedef std::function<int(void** p, size_t bytes)> ArenaAlloc;
constexpr size_t ARENA_SMALL = size_t(1) << 20, ARENA_ALIGN = 256;

// The arrays that a layout function takes, in three ways: measured, out of one block, or allocated one by one.
class Arena {
    char* base = nullptr;
    const ArenaAlloc* each = nullptr;

public:
    size_t used = 0, largest = 0;
    int rc = 0;
    Arena() {}
    explicit Arena(void* block) : base(static_cast<char*>(block)) {}
    explicit Arena(const ArenaAlloc& alloc) : each(&alloc) {}
    template <class T>
    void take(T** p, size_t count) {
        const size_t bytes = count * sizeof(T);
        void* at = base && count ? base + used : nullptr;
        if (each && count && !rc) rc = (*each)(&at, bytes);
        *p = static_cast<T*>(at);
        used += (bytes + ARENA_ALIGN - 1u) / ARENA_ALIGN * ARENA_ALIGN;
        largest = std::max(largest, bytes);
    }
};

// Bytes that place() asks for in one block.
template <class Layout>
size_t arena_bytes(Layout layout) {
    Arena a;
    layout(a);
    return a.used;
}

// Allocates what `layout` takes: one block, or an allocation per array where none is over ARENA_SMALL (the
// driver serves those from memory that it has mapped already) and where no block of that size is to be had.
template <class Layout>
int place(const ArenaAlloc& alloc, Layout layout) {
    Arena sizes;
    layout(sizes);
    void* block = nullptr;
    if (sizes.largest > ARENA_SMALL && alloc(&block, sizes.used) == 0) {
        Arena a(block);
        layout(a);
        return 0;
    }
    Arena a(alloc);
    layout(a);
    return a.rc;
}

}  // namespace lam
