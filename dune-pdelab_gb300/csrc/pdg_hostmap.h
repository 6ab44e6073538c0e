// pdg_hostmap.h -- whether a kernel may store straight into a host vector
// (host code only: what CUDA says about the address comes in).
#pragma once

#include <cstddef>
#include <cstdint>

namespace pdg {

// what is known of a host address: pinned, the device's address of it, the range
// [start, start + size) of the one allocation or registration it lies in (as the
// device sees it), and whether the device may write there
struct HostMapping {
  bool pinned, writable;
  uintptr_t device, start;
  size_t size;
};

// The device's address of `bytes` bytes at the host address, or 0 unless all of them
// lie in that one range.  Two ends that are both pinned do not show that: pages
// between two registrations need not be mapped, and a store there is a memory fault,
// where a copy is refused or staged by the runtime.
inline uintptr_t mapped_range(const HostMapping &m, size_t bytes) {
  if (!m.pinned || !m.writable || !m.device || m.device < m.start) return 0;
  const uintptr_t off = m.device - m.start;
  return off <= m.size && bytes <= m.size - off ? m.device : 0;
}

}  // namespace pdg
