// Pages of a host buffer that were never touched (csrc/host_pages.h): fresh,
// written and partly written mappings, buffers that start and end inside a page,
// more pages than are looked at in one call.
#include <cstdio>
#include <initializer_list>

#include "host_pages.h"

int main() {
  int bad = 0;
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  for (size_t pages : {(size_t)1, (size_t)3, (size_t)64, (size_t)16384, (size_t)16385, (size_t)40000})
    for (int part = 0; part <= 4; part++) {  // quarters written
      char* m = (char*)mmap(nullptr, pages * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
      if (m == MAP_FAILED) return 2;
      madvise(m, pages * page, MADV_NOHUGEPAGE);
      const size_t written = pages * part / 4;
      for (size_t i = 0; i < written; i++) m[i * page] = 1;
      const size_t a = knnsj::absent_bytes(m, pages * page);
      const size_t inner = knnsj::absent_bytes(m + 7, pages * page - 9);
      if (a != (pages - written) * page || inner != a) {
        std::printf("pages=%zu written=%zu absent=%zu %zu\n", pages, written, a / page, inner / page);
        bad++;
      }
      munmap(m, pages * page);
    }
  // not mapped: taken as present
  char* gone = (char*)mmap(nullptr, 4 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  munmap(gone, 4 * page);
  if (knnsj::absent_bytes(gone, 4 * page) != 0 || knnsj::absent_bytes(gone, 0) != 0) bad++;
  std::printf("bad=%d\n", bad);
  return bad != 0;
}
