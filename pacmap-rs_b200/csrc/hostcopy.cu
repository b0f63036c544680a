// Copies between a caller's ordinary (pageable) host memory and the device.
//
// The driver moves pageable memory through its own staging buffers on the calling thread, and an output's pages are
// first touched there, one by one: 64 MB take it 4.7 ms up and 13.6 down, where the link needs 1.2. Larger copies are
// cut into one range per worker: each worker moves its range piece by piece through two page-locked slots of its own,
// copying one piece on a core while the other is on the link (64 MB: 3.0 and 3.1 ms). The threads live for one copy;
// the slots (32 MB) stay with the device until the library is unloaded. Calls on a device hold its lock, so one copy
// uses them at a time. Memory that the caller page-locked goes to the link directly, and everything goes the driver's way
// when the slots cannot be page-locked.
#include <algorithm>
#include <cstring>
#include <system_error>
#include <thread>

#include "engine.cuh"

namespace pacmap {
namespace {

constexpr int COPY_WORKERS = 8;
constexpr size_t COPY_SLOT = 2u << 20;
// Downloads are staged from 1 MB (0.11 against 0.23 ms; 4 MB 0.45 against 0.63), uploads from 32 MB (1.6 against 1.9;
// at 16 MB the two are equal). A worker is worth starting for 8 MB: smaller shares made 4 MB downloads 0.7 to 1.2 ms.
// 12 and 16 workers moved 256 MB up in 9.0 and 9.3 ms, 8 in 8.4.
constexpr size_t DOWN_MIN = 1u << 20, UP_MIN = 32u << 20, COPY_SHARE = 8u << 20;

}  // namespace

struct HostStaging {
  char* buf = nullptr;
  cudaEvent_t ev[COPY_WORKERS][2] = {};
  HostStaging() {
    if (cudaHostAlloc(reinterpret_cast<void**>(&buf), 2 * COPY_WORKERS * COPY_SLOT, cudaHostAllocDefault) != cudaSuccess)
      throw Fail{PACMAP_ERR_OOM, "cudaHostAlloc (staging)"};  // whatever the reason: the copy has another way
    for (auto& w : ev)
      for (auto& e : w)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
          release();
          throw Fail{PACMAP_ERR_OOM, "cudaEventCreateWithFlags (staging)"};
        }
  }
  void release() {
    for (auto& w : ev)
      for (auto& e : w)
        if (e) cudaEventDestroy(e);
    if (buf) cudaFreeHost(buf);
    buf = nullptr;
  }
  ~HostStaging() { release(); }
  HostStaging(const HostStaging&) = delete;
  HostStaging& operator=(const HostStaging&) = delete;
};

namespace {

std::unique_ptr<HostStaging> g_staging[64];  // by device, used under the device's lock

// Worker w's range [lo, hi): the first error, or success. Pieces alternate between the worker's two slots.
cudaError_t move_range(HostStaging& st, int w, int device, cudaStream_t stream, char* dst, const char* src, size_t lo,
                       size_t hi, bool to_device) {
  cudaError_t e = cudaSetDevice(device);
  char* slots[2] = {st.buf + (2 * w) * COPY_SLOT, st.buf + (2 * w + 1) * COPY_SLOT};
  const size_t piece = std::min(COPY_SLOT, std::max<size_t>((hi - lo) / 4, 128u << 10));
  const size_t pieces = (hi - lo + piece - 1) / piece;
  auto at = [&](size_t p) { return lo + p * piece; };
  auto len = [&](size_t p) { return std::min(piece, hi - at(p)); };
  for (size_t p = 0; p < pieces + (to_device ? 0 : 1) && e == cudaSuccess; ++p) {
    const int s = static_cast<int>(p & 1);
    if (to_device) {
      e = cudaEventSynchronize(st.ev[w][s]);  // the slot's last piece (or the last copy's) has left
      if (e != cudaSuccess) break;
      std::memcpy(slots[s], src + at(p), len(p));
      e = cudaMemcpyAsync(dst + at(p), slots[s], len(p), cudaMemcpyHostToDevice, stream);
      if (e == cudaSuccess) e = cudaEventRecord(st.ev[w][s], stream);
    } else {
      if (p < pieces) {
        if (p < 2) e = cudaEventSynchronize(st.ev[w][s]);  // an earlier upload from this slot
        if (e == cudaSuccess) e = cudaMemcpyAsync(slots[s], src + at(p), len(p), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(st.ev[w][s], stream);
      }
      if (p > 0 && e == cudaSuccess) {
        e = cudaEventSynchronize(st.ev[w][s ^ 1]);
        if (e == cudaSuccess) std::memcpy(dst + at(p - 1), slots[s ^ 1], len(p - 1));
      }
    }
  }
  return e;
}

void copy_host(Ctx& c, void* dst, const void* src, size_t bytes, bool to_device) {
  if (!bytes) return;
  const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  cudaPointerAttributes at{};
  const bool pageable = bytes >= (to_device ? UP_MIN : DOWN_MIN) &&
                        cudaPointerGetAttributes(&at, to_device ? src : dst) == cudaSuccess &&
                        at.type == cudaMemoryTypeUnregistered;
  if (!pageable || !try_scratch([&] {
        if (!g_staging[c.device]) g_staging[c.device] = std::make_unique<HostStaging>();
      })) {
    PM_CUDA(cudaMemcpyAsync(dst, src, bytes, kind, c.stream));
    return;
  }
  HostStaging& st = *g_staging[c.device];
  const int cores = static_cast<int>(std::max(1u, std::thread::hardware_concurrency()));
  const int workers = static_cast<int>(
      std::min<size_t>(std::min(COPY_WORKERS, std::max(1, cores / 2)), std::max<size_t>(1, bytes / COPY_SHARE)));
  const size_t share = (bytes / workers + 4095) & ~static_cast<size_t>(4095);
  cudaError_t err[COPY_WORKERS] = {};
  std::thread th[COPY_WORKERS];
  auto work = [&](int w) {
    const size_t lo = std::min(bytes, w * share), hi = w + 1 == workers ? bytes : std::min(bytes, lo + share);
    err[w] = move_range(st, w, c.device, c.stream, static_cast<char*>(dst), static_cast<const char*>(src), lo, hi,
                        to_device);
  };
  int started = 1;
  try {
    for (; started < workers; ++started) th[started] = std::thread(work, started);
  } catch (const std::system_error&) {  // no more threads: this one takes the remaining ranges
  }
  work(0);
  for (int w = started; w < workers; ++w) work(w);
  for (int w = 1; w < started; ++w) th[w].join();
  for (int w = 0; w < workers; ++w)
    if (err[w] != cudaSuccess) {
      cudaStreamSynchronize(c.stream);
      PM_CUDA(err[w]);
    }
}

}  // namespace

void copy_to_device(Ctx& c, void* d_dst, const void* src, size_t bytes) { copy_host(c, d_dst, src, bytes, true); }
void copy_to_host(Ctx& c, void* dst, const void* d_src, size_t bytes) { copy_host(c, dst, d_src, bytes, false); }

}  // namespace pacmap
