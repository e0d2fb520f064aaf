// Which of the caller's host arrays a kernel may read or write in place of a copy.
#pragma once

#include <cstddef>
#include <cstdint>

namespace vfd {

// What the driver reports about an address: whether it is pinned host memory, the address kernels
// use for it, and the allocation (or registration) that holds it.
struct HostRange {
    bool pinned;
    const void* device;
    const void* start;
    size_t size;
};

// Whether kernels reach the floats [p, p + bytes) at their host address: all of them in one pinned
// range (the ends of an array may lie in two ranges with unmapped pages between) and aligned as
// floats (a copy moves bytes from any address).
inline bool kernel_reaches(const void* p, size_t bytes, const HostRange& r) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), s = reinterpret_cast<uintptr_t>(r.start);
    return r.pinned && r.device == p && a % alignof(float) == 0 && a >= s && a - s <= r.size && bytes <= r.size - (a - s);
}

}  // namespace vfd
