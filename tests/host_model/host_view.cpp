// Host build of the rule by which a decode writes a caller's buffers directly (host_view.h).  Test code only.
#include "../../openfish_b200/csrc/host_view.h"

extern "C" uintptr_t host_writable(int page_locked, uintptr_t device, uintptr_t start, size_t size, size_t bytes) {
    const HostRange r = {page_locked != 0, device, start, size};
    return reinterpret_cast<uintptr_t>(writable_by_device(r, bytes));
}
