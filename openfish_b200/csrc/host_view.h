// host_view.h -- whether a kernel may write a caller's host buffer itself.  Plain C++, so that the rule can be
// tried without a GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>

// What the driver says about an address: page-locked or not, where the device sees it, and the whole
// registered range (in the device's addresses) that it lies in.
struct HostRange {
    bool page_locked;
    uintptr_t device, start;
    size_t size;
};

// Where the device can write the `bytes` bytes of a host buffer whose first byte `r` is about; null if it
// cannot write all of them.  Only the first byte's page being locked is not enough: a buffer may begin in one
// registration and end outside of it, and a store there is a fault that nothing checks.
inline unsigned char *writable_by_device(const HostRange &r, size_t bytes) {
    if (!r.page_locked || !r.device || r.device < r.start) return nullptr;
    const size_t before = r.device - r.start;
    if (before > r.size || bytes > r.size - before) return nullptr;
    return reinterpret_cast<unsigned char *>(r.device);
}
