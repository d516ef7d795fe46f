// devrange.h — which allocations a range of device addresses lies in.
#pragma once
#include <cstddef>
#include <cstdint>

namespace suli {

enum RangeKind {
    kRangeUnmapped = -1,   // some address of it belongs to no allocation
    kRangeSeveral = 0,     // it crosses from one allocation into the next
    kRangeOne = 1,         // one allocation holds it
};

// Range of [p, p + bytes).  lookup(address, &base, &size) gives the allocation that holds an address,
// false if none does.
template <class Lookup>
RangeKind range_kind(std::uintptr_t p, std::size_t bytes, Lookup lookup) {
    const std::uintptr_t end = p + bytes;
    for (int n = 0; p < end; ++n) {
        std::uintptr_t base = 0;
        std::size_t size = 0;
        if (!lookup(p, &base, &size) || p < base || p - base >= size) return kRangeUnmapped;
        if (n == 0 && end - base <= size) return kRangeOne;
        p = base + size;
    }
    return kRangeSeveral;
}

}  // namespace suli
