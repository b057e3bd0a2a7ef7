// kc_host_copy.cuh — copies between device memory and a caller's host array,
// complete on return.
//
// Host arrays of the C ABI are the caller's: pinned ones are copied directly, but
// a pageable one goes through the driver's own staging by one thread, at 10 GB/s
// up and, into pages not touched yet (a fresh result array), 2 GB/s down. Here
// large pageable arrays are staged by several threads through a small pinned
// area, so that page faults and host copies run in parallel with each other and
// with the bus. Measured for 40 MB on 16 host cores: up 4.1 to 1.5 ms, down into
// fresh pages 20.5 to 3.7 ms, into touched ones 2.6 to 1.6 ms.
//
// The area is one per process, 4 MiB, made at the first large copy and given back
// when the last engine handle is destroyed; a process that makes no handle, only
// batch calls, keeps it until it ends. Its memory is the process's own and only
// page-locked: a device reset undoes the locking, which the next copy makes good. A
// copy that finds the area in use by another thread, or cannot have it, takes the
// driver's way.
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <atomic>
#include <mutex>
#include <new>
#include <thread>

namespace kc {
namespace hostcopy {

constexpr size_t kChunk = 256 << 10, kMin = 2 << 20;
constexpr int kWorkers = 8, kSlots = 2;
constexpr size_t kArea = kWorkers * kSlots * kChunk;
static_assert(kArea == 4 << 20, "the area's size");

struct Area {
  std::mutex busy;           // held by the copy that uses the area
  unsigned char* mem = nullptr;
  int handles = 0;           // live engine handles (guarded by busy)
};
inline Area& area() {
  // never destroyed: calls may outlive static destruction
  alignas(Area) static unsigned char place[sizeof(Area)];
  static Area* a = new (place) Area;
  return *a;
}
inline void handle_made() {
  std::lock_guard<std::mutex> lock(area().busy);
  ++area().handles;
}
inline void handle_gone() {
  std::lock_guard<std::mutex> lock(area().busy);
  Area& a = area();
  if (--a.handles > 0 || !a.mem) return;
  if (cudaHostUnregister(a.mem) != cudaSuccess) cudaGetLastError();  // after a device reset
  free(a.mem);
  a.mem = nullptr;
}

inline bool pageable(const void* p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

// Makes the area, or locks its pages again; false: it cannot be had. With a.busy held.
// In huge pages where the system has them: made and locked in 0.7 ms, against 2.2 to
// 4.6 ms in small ones and 1.5 to 4 ms by cudaHostAlloc.
inline bool ready(Area& a) {
  if (!a.mem) {
    a.mem = (unsigned char*)aligned_alloc(kArea, kArea);
    if (!a.mem) return false;
    madvise(a.mem, kArea, MADV_HUGEPAGE);
    memset(a.mem, 0, kArea);
  }
  if (!pageable(a.mem) || cudaHostRegister(a.mem, kArea, cudaHostRegisterPortable) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

// One worker: takes chunks of [0, n) from *next until none is left. Two slots, so
// that a chunk's transfer runs beside the host copy of the one before.
inline void work(int device, unsigned char* slots, unsigned char* dev, unsigned char* host, size_t n, bool up,
                 cudaStream_t st, std::atomic<size_t>* next, std::atomic<int>* err) {
  cudaError_t e = cudaSetDevice(device);
  cudaEvent_t ev[kSlots] = {};
  for (int k = 0; k < kSlots && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
  size_t held[kSlots];  // the offset whose transfer is in flight in a slot
  bool flying[kSlots] = {};
  const auto settle = [&](int k) {
    if (!flying[k]) return;
    flying[k] = false;
    const cudaError_t w = cudaEventSynchronize(ev[k]);
    if (e == cudaSuccess) e = w;
    if (up || e != cudaSuccess) return;
    memcpy(host + held[k], slots + k * kChunk, n - held[k] < kChunk ? n - held[k] : kChunk);
  };
  for (int k = 0; e == cudaSuccess && err->load() == cudaSuccess; k ^= 1) {
    settle(k);
    if (e != cudaSuccess) break;
    const size_t off = next->fetch_add(kChunk);
    if (off >= n) break;
    const size_t len = n - off < kChunk ? n - off : kChunk;
    unsigned char* slot = slots + k * kChunk;
    if (up) {
      memcpy(slot, host + off, len);
      e = cudaMemcpyAsync(dev + off, slot, len, cudaMemcpyHostToDevice, st);
    } else {
      e = cudaMemcpyAsync(slot, dev + off, len, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaEventRecord(ev[k], st);
    held[k] = off;
    flying[k] = e == cudaSuccess;
  }
  for (int k = 0; k < kSlots; ++k) settle(k);
  for (int k = 0; k < kSlots; ++k)
    if (ev[k]) cudaEventDestroy(ev[k]);
  if (e != cudaSuccess) {
    cudaStreamSynchronize(st);  // nothing of the area is in flight after a failure either
    err->store(e);
  }
}

// Copies n bytes, ordered on st, and waits for it.
inline cudaError_t copy(void* dev, const void* host, size_t n, bool up, cudaStream_t st) {
  if (n >= kMin && pageable(host)) {
    Area& a = area();
    std::unique_lock<std::mutex> lock(a.busy, std::try_to_lock);
    int device = 0;
    if (lock.owns_lock() && ready(a) && cudaGetDevice(&device) == cudaSuccess) {
      std::atomic<size_t> next(0);
      std::atomic<int> err(cudaSuccess);
      std::thread th[kWorkers];
      int nt = 1;
      const int cores = (int)std::thread::hardware_concurrency();
      try {  // as many helpers as the system gives: the chunks are taken by whoever is there
        for (; nt < kWorkers && nt < cores; ++nt)
          th[nt] = std::thread(work, device, a.mem + nt * kSlots * kChunk, (unsigned char*)dev, (unsigned char*)host, n,
                               up, st, &next, &err);
      } catch (...) {  // no thread, or no memory for one
      }
      work(device, a.mem, (unsigned char*)dev, (unsigned char*)host, n, up, st, &next, &err);
      for (int k = 1; k < kWorkers; ++k)
        if (th[k].joinable()) th[k].join();
      return (cudaError_t)err.load();
    }
  }
  cudaError_t e = up ? cudaMemcpyAsync(dev, host, n, cudaMemcpyHostToDevice, st)
                     : cudaMemcpyAsync((void*)host, dev, n, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e;
}
inline cudaError_t to_device(void* dev, const void* host, size_t n, cudaStream_t st) { return copy(dev, host, n, true, st); }
inline cudaError_t to_host(void* host, const void* dev, size_t n, cudaStream_t st) {
  return copy((void*)dev, host, n, false, st);
}

}  // namespace hostcopy
}  // namespace kc
