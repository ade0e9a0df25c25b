// Drives HostCopier over the stand-in runtime: one scenario per run, "ok" when
// it holds.
#include <atomic>
#include <cstdio>
#include <new>
#include <string>

#include "host_copy.hpp"

using nicp::HostCopier;
using Bytes = std::vector<char>;

static std::atomic<bool> no_new{false};
void *operator new(size_t n) {
  void *p = no_new ? nullptr : std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

static int failures = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); failures++; } } while (0)

static Bytes source(size_t n, unsigned seed) {
  Bytes b(n);
  for (size_t i = 0; i < n; i++) b[i] = (char)((i * 2654435761u + seed * 97u) >> 13);
  return b;
}

// Page-locked destinations are copied into directly, beside pageable ones.
static void locked() {
  const size_t big = ((size_t)3 << 20) + 17;
  const Bytes a = source(big, 1), b = source(big, 2);
  Bytes da(big), db(big);
  fake.locked[da.data()] = big;
  {
    HostCopier c;
    const HostCopier::Part one[] = {{da.data(), a.data(), big}};
    CHECK(c.down(one, 1, nullptr) == cudaSuccess);
    CHECK(da == a && fake.copies.size() == 1 && fake.copies[0].dst == da.data() && fake.allocated == 0);
    da.assign(big, 0);
    const HostCopier::Part two[] = {{db.data(), b.data(), big}, {nullptr, a.data(), 5}, {da.data(), a.data(), big}};
    CHECK(c.down(two, 3, nullptr) == cudaSuccess);
    CHECK(da == a && db == b);
    int direct = 0;
    for (const Fake::Copy &k : fake.copies) direct += k.dst == da.data();
    CHECK(direct == 2);
  }
  // only the front half page-locked: not taken for a page-locked buffer
  fake.locked[da.data()] = big / 2;
  fake.copies.clear();
  da.assign(big, 0);
  HostCopier c;
  const HostCopier::Part one[] = {{da.data(), a.data(), big}};
  CHECK(c.down(one, 1, nullptr) == cudaSuccess && da == a);
  for (const Fake::Copy &k : fake.copies) CHECK(k.dst != da.data());
  fake.locked.erase(da.data());
}

// A copy that has its slots and workers allocates nothing (an exception on the
// way would leave the workers writing into memory that the caller takes back);
// a failing transfer is reported, and the copier works on.
static void no_memory() {
  const size_t big = ((size_t)40 << 20) + 9;
  const Bytes a = source(big, 4);
  Bytes da(big);
  HostCopier c;
  const HostCopier::Part one[] = {{da.data(), a.data(), big}};
  CHECK(c.down(one, 1, nullptr) == cudaSuccess && da == a);
  fake.copies.clear();
  fake.copies.reserve(1000);
  da.assign(big, 0);
  no_new = true;
  bool thrown = false;
  cudaError_t e = cudaSuccess;
  try {
    e = c.down(one, 1, nullptr);
  } catch (const std::bad_alloc &) {
    thrown = true;
  }
  no_new = false;
  CHECK(!thrown && e == cudaSuccess && da == a);
  fake.copies.clear();
  fake.fail_copy = 20;
  CHECK(c.down(one, 1, nullptr) == cudaErrorInvalidValue);
  fake.fail_copy = -1;
  cudaGetLastError();
  da.assign(big, 0);
  CHECK(c.down(one, 1, nullptr) == cudaSuccess && da == a);
}

// Without page-locked memory for the slots (or their events) a copy still
// arrives, and the slots are used once they can be had.
static void no_slots() {
  const size_t big = ((size_t)9 << 20) + 5;
  const Bytes a = source(big, 3);
  Bytes da(big), db(100);
  HostCopier c;
  const HostCopier::Part parts[] = {{da.data(), a.data(), big}, {db.data(), a.data(), 100}};
  for (int k = 0; k < 4; k++) {
    fake.lock_fails = k == 0;
    fake.event_fails = k == 1;
    da.assign(big, 0);
    db.assign(100, 0);
    CHECK(c.down(parts, 2, nullptr) == cudaSuccess && cudaGetLastError() == cudaSuccess);
    CHECK(da == a && std::equal(db.begin(), db.end(), a.begin()));
  }
  CHECK(fake.allocated == 1);
}

int main(int, char **argv) {
  const std::string what = argv[1];
  if (what == "locked") locked();
  else if (what == "no_slots") no_slots();
  else if (what == "no_memory") no_memory();
  else CHECK(!"a scenario");
  CHECK(fake.allocated == fake.freed && fake.events == 0);
  std::puts(failures ? "failed" : "ok");
  return failures != 0;
}
