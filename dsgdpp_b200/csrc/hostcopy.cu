// hostcopy.cu -- see hostcopy.h.
#include "hostcopy.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace dsgdpp {
namespace {

// Measured on a B200 host with 16 cores, 358 MB of factors to the device / back:
// 32 / 75 ms through the driver, 8.6 / 16 ms in pieces of 1 MB, 12.5 / 20 ms in
// pieces of 512 KB.
constexpr size_t kPiece = 1 << 20;
// Smaller arrays go the driver's way, where making the threads takes longer than
// they save.  us in / back, direct against pieces: 2.1 MB 152 / 182 against 240 /
// 479, 4 MB 270 / 320 against 265 / 590, 8 MB 475 / 590 against 473 / 600, 16 MB
// 910 / 1230 against 660 / 1000.  (Runs of the quick start, whose factors are
// two arrays of 8 MB, take 5.4 ms with pieces and 6.8 without.)
constexpr size_t kDirect = 6 << 20;
constexpr unsigned kThreads = 8;
// One slab serves one copy.  Page-locking it costs some 7 ms, what the pieces
// save on about 90 MB, so the first is made once some of that order has been
// copied: until then, and again after the last holder is gone, copies go the
// direct way (a program that loads little never pays for the slab).
constexpr size_t kSlabPieces = 2 * kThreads;
constexpr size_t kMaxSlabs = 2;  // 32 MB
constexpr size_t kSlabAfter = 64 << 20;

std::mutex g_mutex;
void* g_slabs[kMaxSlabs];
size_t g_nslabs = 0;
void* g_free[kMaxSlabs * kSlabPieces];  // pieces not in use
size_t g_nfree = 0;
size_t g_holders = 0;
size_t g_copied = 0;  // bytes copied directly since there was no slab
std::atomic<uint64_t> g_staged{0};  // bytes that went through pieces (dsgdpp_staged_bytes)

void free_slabs_if_unused() {  // under the mutex
  if (g_nslabs == 0 || g_holders > 0 || g_nfree != g_nslabs * kSlabPieces) return;
  for (size_t k = 0; k < g_nslabs; ++k) cudaFreeHost(g_slabs[k]);
  g_nslabs = g_nfree = 0;
  g_copied = 0;
}

bool worth_staging(size_t bytes) {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_nslabs > 0) return true;
  g_copied += bytes;
  return g_copied >= kSlabAfter;
}

void* take_piece() {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_nfree == 0) {
    if (g_nslabs >= kMaxSlabs) return nullptr;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kPiece * kSlabPieces, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();  // not an error of the copy: it goes the direct way
      return nullptr;
    }
    g_slabs[g_nslabs++] = p;
    for (size_t k = 0; k < kSlabPieces; ++k) g_free[g_nfree++] = static_cast<char*>(p) + k * kPiece;
  }
  return g_free[--g_nfree];
}

void give_piece(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lock(g_mutex);
  g_free[g_nfree++] = p;
  free_slabs_if_unused();
}

bool page_locked(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// One worker: pieces first, first + step, ... of the copy through two
// page-locked pieces of its own, one travelling while the other is filled or
// emptied.  Without pieces (none to be had) it copies directly.
cudaError_t work(char* dst, const char* src, size_t bytes, size_t first, size_t step, bool to_host,
                 int device, cudaStream_t st) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return e;
  struct Slot {
    void* p = nullptr;
    cudaEvent_t done = nullptr;
    size_t at = 0, len = 0;  // the piece of the copy it holds (to_host)
    bool busy = false;
  } slot[2];
  for (Slot& s : slot) {
    s.p = take_piece();
    if (cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming) != cudaSuccess) s.done = nullptr;
  }
  const bool staged = slot[0].p && slot[1].p && slot[0].done && slot[1].done;
  auto finish = [&](Slot& s) {  // the slot's transfer is over; hand out what it brought
    if (!s.busy) return cudaSuccess;
    s.busy = false;
    const cudaError_t r = cudaEventSynchronize(s.done);
    if (r == cudaSuccess && to_host) std::memcpy(dst + s.at, s.p, s.len);
    return r;
  };
  int k = 0;
  for (size_t at = first * kPiece; at < bytes && e == cudaSuccess; at += step * kPiece, k ^= 1) {
    const size_t len = std::min(kPiece, bytes - at);
    if (!staged) {
      e = cudaMemcpyAsync(dst + at, src + at, len,
                          to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st);
      continue;
    }
    Slot& s = slot[k];
    e = finish(s);
    if (e != cudaSuccess) break;
    if (to_host) {
      e = cudaMemcpyAsync(s.p, src + at, len, cudaMemcpyDeviceToHost, st);
    } else {
      std::memcpy(s.p, src + at, len);
      e = cudaMemcpyAsync(dst + at, s.p, len, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) e = cudaEventRecord(s.done, st);
    s.at = at;
    s.len = len;
    s.busy = e == cudaSuccess;
    if (s.busy) g_staged += len;
  }
  for (int j = 0; j < 2; ++j) {  // in the order they were started
    const cudaError_t r = finish(slot[k ^ j]);
    if (e == cudaSuccess) e = r;
  }
  if (!staged && to_host && e == cudaSuccess) e = cudaStreamSynchronize(st);
  // after a failure a transfer may still use the pieces
  if (e != cudaSuccess) cudaStreamSynchronize(st);
  for (Slot& s : slot) {
    give_piece(s.p);
    if (s.done) cudaEventDestroy(s.done);
  }
  return e;
}

cudaError_t copy(void* dst, const void* src, size_t bytes, bool to_host, int device,
                 cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  const void* host = to_host ? dst : src;
  if (bytes < kDirect || page_locked(host) || !worth_staging(bytes))
    return cudaMemcpyAsync(dst, src, bytes, kind, st);
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
  const unsigned n = (unsigned)std::min<size_t>({kThreads, cores, (pieces + 1) / 2});
  cudaError_t status[kThreads];
  std::thread pool[kThreads];
  auto one = [&](unsigned t) {
    status[t] = work(static_cast<char*>(dst), static_cast<const char*>(src), bytes, t, n, to_host,
                     device, st);
  };
  unsigned started = 1;
  for (; started < n; ++started) {
    try {
      pool[started] = std::thread(one, started);
    } catch (...) {  // std::system_error, std::bad_alloc
      break;  // no more threads: this one does the rest
    }
  }
  one(0);
  for (unsigned t = started; t < n; ++t) one(t);
  for (unsigned t = 1; t < started; ++t) pool[t].join();
  for (unsigned t = 0; t < n; ++t)
    if (status[t] != cudaSuccess) return status[t];
  return cudaSuccess;
}

}  // namespace

cudaError_t copy_to_device(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
  return copy(dst, src, bytes, false, device, st);
}

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
  return copy(dst, src, bytes, true, device, st);
}

void BackgroundCopy::start(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
  join();
  auto run = [this, dst, src, bytes, device, st]() {
    status_ = cudaSetDevice(device);
    if (status_ == cudaSuccess) status_ = copy_to_device(dst, src, bytes, device, st);
  };
  if (bytes < kDirect || page_locked(src)) {
    run();
    return;
  }
  try {
    thread_ = std::thread(run);
  } catch (...) {
    run();
  }
}

cudaError_t BackgroundCopy::join() {
  if (thread_.joinable()) thread_.join();
  return status_;
}

void hostcopy_hold() {
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_holders;
}

void hostcopy_drop() {
  std::lock_guard<std::mutex> lock(g_mutex);
  --g_holders;
  free_slabs_if_unused();
}

}  // namespace dsgdpp

extern "C" uint64_t dsgdpp_staged_bytes() { return dsgdpp::g_staged; }
