// host_steps.h - host-side sequences whose failure paths matter, in plain C++ (tested without a device).
#pragma once

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

}  // namespace lam
