// Runs kc_host_copy.cuh on the host against a stand-in for the runtime calls that
// it makes. The stand-in's copies are deferred as far as the real ones may be: to
// the event or stream synchronisation that waits for them, so a slot used again too
// early, or read too early, shows in the bytes.
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <thread>
#include <vector>

#include "../koral-zig_b200/csrc/kc_host_copy.cuh"

using namespace kc;

// ---- the stand-in ------------------------------------------------------------
namespace {
struct Op {
  void* dst;
  const void* src;
  size_t n;
};
std::mutex mu;
Op ops[1 << 12];  // one stream's copies, those from done_ on not run yet
size_t done_ = 0, issued_ = 0;
std::map<const char*, size_t> locked;      // page-locked ranges
size_t largest = 0;
int copies = 0, fail_copy_at = 0, fail_lock = 0;
std::atomic<int> news_left(-1);  // allocations until one fails; < 0: none does
void run_to(size_t k) {
  while (done_ < k) {
    const Op o = ops[done_++ % (1 << 12)];
    memcpy(o.dst, o.src, o.n);
  }
}
std::vector<void*> taken;  // memory of the runtime's own
void device_reset() {      // ends the locking and the runtime's memory
  std::lock_guard<std::mutex> l(mu);
  locked.clear();
  for (void* p : taken) munmap(p, 8 << 20);
  taken.clear();
}
bool is_locked(const void* p) {
  auto it = locked.upper_bound((const char*)p);
  return it != locked.begin() && (--it, (const char*)p < it->first + it->second);
}
}  // namespace
void* operator new(size_t n) {
  if (news_left.load() >= 0 && news_left.fetch_sub(1) == 0) throw std::bad_alloc();
  void* p = malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::lock_guard<std::mutex> l(mu);
  a->type = is_locked(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  std::lock_guard<std::mutex> l(mu);
  if (fail_lock) return cudaErrorMemoryAllocation;
  *p = mmap(nullptr, 8 << 20, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  taken.push_back(*p);
  locked[(const char*)*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> l(mu);
  for (size_t k = 0; k < taken.size(); ++k)
    if (taken[k] == p) {
      munmap(p, 8 << 20);
      taken.erase(taken.begin() + k);
      locked.erase((const char*)p);
      return cudaSuccess;
    }
  return cudaErrorInvalidValue;
}
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
  std::lock_guard<std::mutex> l(mu);
  if (fail_lock) return cudaErrorMemoryAllocation;
  locked[(const char*)p] = n;
  return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
  std::lock_guard<std::mutex> l(mu);
  return locked.erase((const char*)p) ? cudaSuccess : cudaErrorHostMemoryNotRegistered;
}
// an event is the count of copies before it
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)calloc(1, sizeof(size_t)), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free((void*)e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  std::lock_guard<std::mutex> l(mu);
  *(size_t*)e = issued_;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> l(mu);
  run_to(*(size_t*)e);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::lock_guard<std::mutex> l(mu);
  run_to(issued_);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::lock_guard<std::mutex> l(mu);
  if (fail_copy_at && ++copies >= fail_copy_at) return cudaErrorLaunchFailure;
  largest = n > largest ? n : largest;
  ops[issued_++ % (1 << 12)] = {d, s, n};
  return cudaSuccess;
}
}

// ---- the checks ----------------------------------------------------------------
namespace {
std::vector<unsigned char> pattern(size_t n, unsigned seed) {
  std::vector<unsigned char> v(n);
  for (size_t i = 0; i < n; ++i) v[i] = (unsigned char)((i * 2654435761u + seed * 97u) >> 13);
  return v;
}
// both directions, with the bytes around the destination
bool copies_right(size_t n, unsigned seed) {
  const size_t pad = 64;
  const std::vector<unsigned char> src = pattern(n, seed);
  std::vector<unsigned char> dst(n + 2 * pad, 0xA5);
  for (int up = 0; up < 2; ++up) {
    std::fill(dst.begin(), dst.end(), 0xA5);
    const cudaError_t e = up ? hostcopy::to_device(dst.data() + pad, src.data(), n, 0)
                             : hostcopy::to_host(dst.data() + pad, src.data(), n, 0);
    if (e != cudaSuccess || memcmp(dst.data() + pad, src.data(), n)) return false;
    for (size_t i = 0; i < pad; ++i)
      if (dst[i] != 0xA5 || dst[pad + n + i] != 0xA5) return false;
  }
  return true;
}
int fails = 0;
void check(bool ok, const char* what) {
  if (!ok) {
    ++fails;
    printf("wrong: %s\n", what);
  }
}
bool staged(size_t n) {  // by chunks, not in one piece
  largest = 0;
  const bool ok = copies_right(n, 1);
  return ok && largest <= hostcopy::kChunk;
}

void sizes() {
  const size_t c = hostcopy::kChunk, m = hostcopy::kMin;
  for (size_t n : {(size_t)1, c - 1, m - 1}) {
    largest = 0;
    check(copies_right(n, 2) && largest == n, "a small copy, by the driver");
  }
  for (size_t n : {m, m + 1, m + c - 1, m + c, m + c + 1, 20 * c + 7, 41 * c + c / 2}) check(staged(n), "a staged copy");
  std::vector<unsigned char> pinned(m + 5);
  const std::vector<unsigned char> src = pattern(m + 5, 3);
  cudaHostRegister(pinned.data(), pinned.size(), 0);
  largest = 0;
  check(hostcopy::to_host(pinned.data(), src.data(), src.size(), 0) == cudaSuccess && pinned == src && largest == m + 5,
        "a page-locked array, by the driver");
  cudaHostUnregister(pinned.data());
}
void threads() {
  bool ok[4] = {};
  std::thread th[4];
  for (int k = 0; k < 4; ++k)
    th[k] = std::thread([&ok, k] {
      ok[k] = true;
      for (int r = 0; r < 6; ++r) ok[k] = ok[k] && copies_right(hostcopy::kMin + 77777 * k + r, 10 * k + r);
    });
  for (auto& t : th) t.join();
  check(ok[0] && ok[1] && ok[2] && ok[3], "copies of four threads at once");
  bool busy = false;
  {
    std::lock_guard<std::mutex> held(hostcopy::area().busy);
    largest = 0;
    std::thread([&] { busy = copies_right(hostcopy::kMin + 9, 5); }).join();
  }
  check(busy && largest == hostcopy::kMin + 9, "a copy while the area is in use, by the driver");
}
void handles() {
  hostcopy::handle_made();
  hostcopy::handle_made();
  check(staged(hostcopy::kMin), "a copy with handles");
  hostcopy::handle_gone();
  check(hostcopy::area().mem != nullptr, "the area while a handle lives");
  hostcopy::handle_gone();
  check(hostcopy::area().mem == nullptr && locked.empty(), "the area given back with the last handle");
  check(staged(hostcopy::kMin + 3), "a copy after the last handle");
  hostcopy::handle_made();
  hostcopy::handle_gone();
  fail_lock = 1;
  largest = 0;
  check(copies_right(hostcopy::kMin + 1, 6) && largest == hostcopy::kMin + 1, "a copy without an area, by the driver");
  fail_lock = 0;
}
void resets() {
  check(staged(hostcopy::kMin), "a copy before a device reset");
  device_reset();
  check(staged(hostcopy::kMin + 1), "a copy after a device reset");
  hostcopy::handle_made();
  device_reset();
  hostcopy::handle_gone();
  check(hostcopy::area().mem == nullptr && staged(hostcopy::kMin + 2), "a copy after the area went with a reset");
}
void errors() {
  const std::vector<unsigned char> src = pattern(hostcopy::kMin * 2, 7);
  std::vector<unsigned char> dst(src.size());
  for (int at : {1, 2, 5, 8}) {
    copies = 0;
    fail_copy_at = at;
    check(hostcopy::to_device(dst.data(), src.data(), src.size(), 0) == cudaErrorLaunchFailure && done_ == issued_,
          "a failing copy reported, with nothing left in flight");
    fail_copy_at = 0;
  }
  check(staged(hostcopy::kMin), "a copy after a failed one");
}
// helper threads that cannot be made, for want of memory: the copy is complete all the same
void no_helpers() {
  const std::vector<unsigned char> src = pattern(hostcopy::kMin + 11, 8);
  std::vector<unsigned char> dst(src.size());
  for (int left = 0; left < 12; ++left) {
    std::fill(dst.begin(), dst.end(), 0);
    news_left = left;
    const cudaError_t e = hostcopy::to_device(dst.data(), src.data(), src.size(), 0);
    news_left = -1;
    check(e == cudaSuccess && dst == src, "a copy without memory for its helpers");
  }
}
}  // namespace

int main() {
  sizes();
  threads();
  handles();
  resets();
  errors();
  no_helpers();
  printf("%d\n", fails);
  return fails != 0;
}
