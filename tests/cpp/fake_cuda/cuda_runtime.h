// A host stand-in for the few runtime calls of host_copy.hpp: "device" memory
// is host memory, copies happen at once, page-locked ranges are a list, and
// allocations can be made to fail.
#pragma once
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes { cudaMemoryType type; };
typedef void *cudaStream_t;
typedef int *cudaEvent_t;
constexpr unsigned cudaEventDisableTiming = 2;

struct Fake {
  std::map<char *, size_t> locked;  // page-locked ranges
  struct Copy { char *dst; size_t bytes; };
  std::vector<Copy> copies;
  bool lock_fails = false, event_fails = false;
  int fail_copy = -1;  // this copy and all later ones fail
  int allocated = 0, freed = 0, events = 0;
  cudaError_t last = cudaSuccess;
  bool is_locked(const void *p) const {
    auto it = locked.upper_bound((char *)p);
    if (it == locked.begin()) return false;
    --it;
    return (char *)p < it->first + it->second;
  }
};
inline Fake fake;

inline cudaError_t raise_error(cudaError_t e) { return fake.last = e; }
inline cudaError_t cudaGetLastError() { const cudaError_t e = fake.last; fake.last = cudaSuccess; return e; }
inline cudaError_t cudaMallocHost(char **p, size_t n) {
  if (fake.lock_fails) return raise_error(cudaErrorMemoryAllocation);
  *p = (char *)std::malloc(n);
  fake.locked[*p] = n;
  fake.allocated++;
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void *p) { fake.locked.erase((char *)p); std::free(p); fake.freed++; return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  if (fake.event_fails) return raise_error(cudaErrorMemoryAllocation);
  *e = new int(0);
  fake.events++;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; fake.events--; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  a->type = fake.is_locked(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fake.fail_copy >= 0 && (int)fake.copies.size() >= fake.fail_copy) return raise_error(cudaErrorInvalidValue);
  std::memcpy(d, s, n);
  fake.copies.push_back({(char *)d, n});
  return cudaSuccess;
}
