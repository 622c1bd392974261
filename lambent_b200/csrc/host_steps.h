// host_steps.h - host-side sequences whose failure paths matter, in plain C++ (tested without a device).
#pragma once
#include <cstddef>

namespace lam {

// Steps of which each one needs those before it: after one that failed, none is taken.  A kernel whose
// producer was not launched would take whatever its input holds for indexes.
template <class Status>
struct Steps {
    Status status{};
    template <class F>
    void operator()(F step) {
        if (status == Status{}) status = step();
    }
};

// Two arrays of `count` that are only ever there together: one allocation, so that none is left without
// the other when memory runs out.  `alloc(T**, n)` returns 0 on success.
template <class T, class Alloc>
int alloc_pair(T** a, T** b, size_t count, Alloc alloc) {
    T* both = nullptr;
    if (const int rc = alloc(&both, 2 * count)) return rc;
    *a = both;
    *b = both + count;
    return 0;
}

// Launches a grid whose blocks wait for one another with at most `grid` blocks: halved while the launch says
// that so many are not resident together (a partition of the device holds fewer than the device).
template <class Status, class Launch>
Status launch_resident(unsigned grid, Status too_large, Launch launch) {
    Status s = launch(grid);
    while (s == too_large && grid > 1) s = launch(grid = (grid + 1) / 2);
    return s;
}

}  // namespace lam
