// gbr_host_range.h — whether a kernel may write a caller's host buffer through
// its device address, from what the driver says of its allocations (plain C++,
// shared with its host check).
#pragma once

#include <cstddef>
#include <cstdint>

namespace gbr {

// The page-locked, mapped allocation (or registration) that holds an address:
// the address as the device sees it, and the device range of the allocation.
struct HostSpan {
  uintptr_t device, start;
  size_t size;
};

// The device address of [p, p + bytes) when p is 4-byte aligned (kernels write
// 32-bit words) and every byte lies in mapped allocations that follow one
// another on the device, else nullptr.  The words at both ends say nothing of
// the pages between them: under unified addressing two registrations with
// pageable memory between them look like one.  query(q, &span) looks an
// address up and returns false where no mapped allocation holds it.
template <class Query>
uint8_t* mapped_range(void* p, size_t bytes, Query query) {
  if (!p || !bytes || (reinterpret_cast<uintptr_t>(p) & 3) != 0) return nullptr;
  uintptr_t first = 0;
  for (size_t done = 0; done < bytes;) {
    HostSpan s{};
    if (!query(static_cast<uint8_t*>(p) + done, &s) || !s.device) return nullptr;
    if (s.device < s.start || s.device - s.start >= s.size) return nullptr;
    if (done == 0)
      first = s.device;
    else if (s.device != first + done)
      return nullptr;
    done += s.size - (s.device - s.start);
  }
  return reinterpret_cast<uint8_t*>(first);
}

}  // namespace gbr
