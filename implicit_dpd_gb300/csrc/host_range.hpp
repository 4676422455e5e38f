// Which host arrays kernels may read or write over the host link: those that lie, whole, in
// one page-locked allocation or registration. Plain host code, compiled in the CPU tests.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace idpd {

// What the driver says of a pointer.
struct HostPointer {
  bool page_locked = false;   // host memory that it knows
  uintptr_t device = 0;       // the address that kernels use
  uintptr_t start = 0;        // the allocation or registration that holds it
  size_t size = 0;
  bool writable = false;      // by kernels
};

// The device address of the `bytes` bytes at p, or 0 where a part of them lies outside p's
// allocation, the address is not aligned to 8 bytes, or `write` is asked of memory that
// kernels only read.
inline uintptr_t link_address(const HostPointer& a, uintptr_t p, size_t bytes, bool write) {
  if (!a.page_locked || !a.device || a.device % 8 != 0 || (write && !a.writable)) return 0;
  if (p < a.start || a.size < bytes || p - a.start > a.size - bytes) return 0;
  return a.device;
}

}  // namespace idpd
