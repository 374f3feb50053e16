// Host-only.
#pragma once
#include <cstddef>

namespace rqc {

// Touches the pages of an output buffer that a copy from the device will fill. Called while
// the device works: a fresh 56 MB field buffer otherwise costs its page faults (about 7 ms)
// inside the copy, after the solve. Each touch is a write that leaves the byte as it is (an
// atomic or with zero), so that a call that fails leaves its caller's arrays alone.
inline void prefault(void *p, size_t bytes) {
    constexpr size_t page = 4096;
    char *c = static_cast<char *>(p);
    for (size_t i = 0; i < bytes; i += page)
        __atomic_fetch_or(c + i, 0, __ATOMIC_RELAXED);
    if (bytes)
        __atomic_fetch_or(c + bytes - 1, 0, __ATOMIC_RELAXED);
}

} // namespace rqc
