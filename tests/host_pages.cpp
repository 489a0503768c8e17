// Test driver of populate_pages (tests/test_host_pages_cpu.py). Prints one
// line per check that fails and ends with the number of them.
#include "../hydra_lotus_b200/csrc/host_pages.h"

#include <cstdio>
#include <cstring>
#include <vector>

static int failures = 0;
static void check(bool ok, const char* what) {
  if (ok) return;
  std::printf("%s\n", what);
  ++failures;
}

static size_t page() { return (size_t)sysconf(_SC_PAGESIZE); }

static char* fresh(size_t pages, int protection = PROT_READ | PROT_WRITE) {
  void* p = mmap(nullptr, pages * page(), protection, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  return p == MAP_FAILED ? nullptr : (char*)p;
}

static std::vector<unsigned char> resident(char* p, size_t pages) {
  std::vector<unsigned char> v(pages, 0);
  check(mincore(p, pages * page(), v.data()) == 0, "mincore");
  for (auto& x : v) x &= 1;
  return v;
}

int main() {
  const size_t n = page();
  // Whole pages of a range that begins and ends within a page, none beyond it.
  {
    char* p = fresh(8);
    lotus::populate_pages(p + 16, 6 * n);
    const auto r = resident(p, 8);
    check(!r[0], "the page that the range begins within");
    for (int k = 1; k <= 5; ++k) check(r[k], "a whole page is not there");
    check(!r[6] && !r[7], "a page past the range's whole ones");
    bool zero = true;
    for (size_t i = 0; i < 8 * n; ++i) zero = zero && p[i] == 0;
    check(zero, "contents of fresh pages");
    munmap(p, 8 * n);
  }
  // What pages hold stays.
  {
    char* p = fresh(4);
    std::memset(p + n, 7, n);
    lotus::populate_pages(p, 4 * n);
    for (const auto x : resident(p, 4)) check(x, "a page of an aligned range");
    bool kept = true;
    for (size_t i = 0; i < 4 * n; ++i) kept = kept && p[i] == (i / n == 1 ? 7 : 0);
    check(kept, "contents");
    munmap(p, 4 * n);
  }
  // Ranges without a whole page, of no bytes and of no address.
  {
    char* p = fresh(2);
    lotus::populate_pages(p + 1, n);
    lotus::populate_pages(p, 0);
    lotus::populate_pages(p + 5, n - 5);
    lotus::populate_pages(nullptr, 16 * n);
    for (const auto x : resident(p, 2)) check(!x, "a page of no range");
    munmap(p, 2 * n);
  }
  // What cannot be populated is left as it is.
  {
    char* p = fresh(4, PROT_READ);
    lotus::populate_pages(p, 4 * n);
    mprotect(p, 4 * n, PROT_READ | PROT_WRITE);
    bool zero = true;
    for (size_t i = 0; i < 4 * n; ++i) zero = zero && p[i] == 0;
    check(zero, "contents of read-only pages");
    munmap(p, 4 * n);
    lotus::populate_pages(p, 4 * n);
  }
  std::printf("%d\n", failures);
  return failures;
}
