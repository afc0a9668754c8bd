// graph_slot.h -- which captured graph may be launched (host code without CUDA
// types).
#pragma once

namespace amg {

// True when `exec` is a graph that may be launched.  A stale one (captured for
// another box, other flags, or arrays that have been reallocated since) is
// captured again by `capture`; if that fails, what is left of the old one is
// given up with `destroy`, and the caller enqueues the kernels themselves.
template <class Exec, class Capture, class Destroy>
bool launchable(Exec& exec, bool stale, Capture capture, Destroy destroy) {
    if (exec && !stale) return true;
    if (capture()) return exec != nullptr;
    if (exec) destroy(exec);
    exec = nullptr;
    return false;
}

}  // namespace amg
