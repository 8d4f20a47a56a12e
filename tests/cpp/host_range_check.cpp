// Checks mapped_range (gbr_host_range.h) on made-up allocations: a buffer is
// taken when mapped allocations cover every byte of it, one after another on
// the device, and no other buffer is.  Exit code 0 when all hold.
#include <cstdio>

#include "gbr_host_range.h"

using gbr::HostSpan;

struct Alloc {
  uintptr_t host, device;
  size_t size;
};

int main() {
  // two registrations with a gap, one that follows the second, one whose device address differs, one that follows it
  // on the host alone, and one at the end of the address range of the test
  const Alloc allocs[] = {{0x10000, 0x10000, 0x2000}, {0x14000, 0x14000, 0x2000}, {0x16000, 0x16000, 0x1000},
                          {0x20000, 0x90000, 0x1000}, {0x21000, 0xA0000, 0x1000}};
  auto query = [&](uint8_t* q, HostSpan* s) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(q);
    for (const Alloc& x : allocs)
      if (a >= x.host && a - x.host < x.size) {
        *s = HostSpan{x.device + (a - x.host), x.device, x.size};
        return true;
      }
    return false;
  };
  struct Case {
    uintptr_t p;
    size_t bytes;
    uintptr_t device;  // 0: refused
  };
  const Case cases[] = {
      {0x10000, 0x2000, 0x10000}, {0x10000, 4, 0x10000},      {0x11FFC, 4, 0x11FFC},   {0x10004, 0x1FFC, 0x10004},
      {0x10000, 0x2001, 0},       {0x11FFC, 8, 0},            {0x12000, 4, 0},         {0x0FFFC, 8, 0},
      {0x10000, 0x6000, 0},       {0x10000, 0x4004, 0},       {0x13FFC, 0x2000, 0},  // ends mapped, or only one of them
      {0x14000, 0x3000, 0x14000}, {0x15FFC, 8, 0x15FFC},      {0x14000, 0x3001, 0},    {0x14000, (size_t)-1, 0},
      {0x20000, 0x1000, 0x90000}, {0x20010, 0xFF0, 0x90010},  {0x20000, 0x1004, 0},    {0x21000, 0x1000, 0xA0000},
      {0x10001, 4, 0},            {0x10002, 4, 0},            {0, 4, 0},               {0x10000, 0, 0},
  };
  int bad = 0;
  for (const Case& c : cases) {
    const uintptr_t got = reinterpret_cast<uintptr_t>(gbr::mapped_range(reinterpret_cast<void*>(c.p), c.bytes, query));
    if (got != c.device) {
      std::printf("%#zx + %#zx: %#zx, not %#zx\n", (size_t)c.p, c.bytes, (size_t)got, (size_t)c.device);
      bad++;
    }
  }
  // an answer that does not hold the address is no answer
  auto wrong = [](uint8_t*, HostSpan* s) {
    *s = HostSpan{0x3000, 0x4000, 0x1000};
    return true;
  };
  if (gbr::mapped_range(reinterpret_cast<void*>(0x3000), 4, wrong)) bad++;
  return bad ? 1 : 0;
}
