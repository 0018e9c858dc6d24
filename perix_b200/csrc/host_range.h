// Which host buffers kernels may read and write themselves (the per-step rate call's ends).
#pragma once

#include <cstddef>
#include <cstdint>

namespace pxb {

// The driver's answer for an address: memory type (CUmemorytype, 1 = host), whether it is managed, and the page-locked
// range that holds it.
struct HostRange {
    unsigned int type = 0, managed = 0;
    unsigned long long start = 0;
    size_t size = 0;
};

// All of [p, p + bytes) lies in r.  The first byte alone does not say so: cudaHostRegister takes any part of a buffer,
// and two registered parts may leave a hole between them.
inline bool range_holds(const HostRange &r, const void *p, size_t bytes) {
    const unsigned long long at = (unsigned long long)reinterpret_cast<uintptr_t>(p);
    return r.type == 1 && !r.managed && at >= r.start && at - r.start <= r.size && bytes <= r.size - (at - r.start);
}

}  // namespace pxb
