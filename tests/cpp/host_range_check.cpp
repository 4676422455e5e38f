// link_address (host_range.hpp) on made-up answers of the driver.
#include "host_range.hpp"

#include <cstdio>

using namespace idpd;

static int bad = 0;
static void want(bool ok, const char* what) {
  if (!ok) {
    bad++;
    std::printf("%s\n", what);
  }
}

int main() {
  const uintptr_t base = 0x70000000;
  HostPointer a;
  a.page_locked = a.writable = true;
  a.start = base;
  a.size = 4096;
  auto at = [&](uintptr_t off, size_t bytes, bool write = false) {
    a.device = base + off + 0x1000000000;  // an address of its own
    return link_address(a, base + off, bytes, write);
  };
  want(at(0, 4096) == base + 0x1000000000, "the whole allocation");
  want(at(0, 4096, true) == base + 0x1000000000, "the whole allocation, written");
  want(at(8, 4088) == base + 8 + 0x1000000000, "its tail");
  want(at(8, 4096) == 0, "past the end");
  want(at(0, 4104) == 0, "longer than the allocation");
  want(at(4088, 8) != 0, "its last number");
  want(at(4096, 8) == 0, "behind the end");
  want(at(0, (size_t)-8) == 0, "a size that wraps");
  want(at(4, 24) == 0, "an odd address");
  // two registrations of one array with a gap: the first holds p, not the array's end
  a.size = 1024;
  want(at(0, 3072) == 0, "an array that ends in another registration");
  a.size = 4096;
  a.writable = false;
  want(at(0, 64) != 0, "read from read-only memory");
  want(at(0, 64, true) == 0, "written to read-only memory");
  a.writable = true;
  a.page_locked = false;
  want(at(0, 64) == 0, "pageable memory");
  a.page_locked = true;
  a.device = 0;
  want(link_address(a, base, 64, false) == 0, "memory without a device address");
  return bad;
}
