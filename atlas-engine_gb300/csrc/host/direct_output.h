// Which output buffers a kernel may write in place of the library's own.
#pragma once

#include <cstddef>
#include <cstdint>

#include <driver_types.h>

namespace atlas::rt::host {

// True when kernels on `device` may write `out`, 16 bytes and atomically too:
// 16-byte aligned memory of that very device (another GPU's may not be
// mapped, and managed pages may lie in host memory), apart from the input
// that is read meanwhile.  a: the attributes of `out`.
inline bool DirectOutput(const cudaPointerAttributes& a, int device, const void* out, size_t bytes, const void* in,
                         size_t in_bytes) {
    const uintptr_t o = reinterpret_cast<uintptr_t>(out), i = reinterpret_cast<uintptr_t>(in);
    if (!out || a.type != cudaMemoryTypeDevice || a.device != device || (o & 15u) != 0) return false;
    return o + bytes <= i || i + in_bytes <= o;
}

}  // namespace atlas::rt::host
