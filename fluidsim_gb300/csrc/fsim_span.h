// fsim_span.h — when a kernel may read or write a caller's host buffer directly.
// Plain C++ (no CUDA headers), so that the rule is tested without a GPU.
#pragma once

#include <cstddef>
#include <cstdint>

namespace fsim_rt {

// What the driver says of a host pointer: whether it is page-locked host memory,
// the device's address of it, and the one allocation (or registration) around that
// address.  All zero for a pointer it does not know.
struct HostSpan {
    bool host;
    uintptr_t dev, start;
    size_t size;
};

// Whether the device can address all `bytes` from the pointer on: they must lie in
// ONE allocation.  That both ends are page-locked is not enough: between two
// allocations there may be pages that the device cannot reach.
inline bool span_addressable(const HostSpan &s, size_t bytes)
{
    return s.host && s.dev && s.start <= s.dev && s.size >= bytes && s.dev - s.start <= s.size - bytes;
}

// Whether the buffers [p, p + bytes) overlap: what a call leaves in buffers that
// share bytes is the last field's, which copies one after another give and copies
// side by side do not.
inline bool spans_overlap(uintptr_t p, size_t pbytes, uintptr_t q, size_t qbytes)
{
    return pbytes && qbytes && (p < q ? q - p < pbytes : p - q < qbytes);
}

} // namespace fsim_rt
