// Large copies between pageable host memory and the device. A plain cudaMemcpyAsync from pageable memory moves a few
// GB/s: one thread of the driver copies everything through a buffer of its own before the bus sees it. Here several
// threads copy, each through two page-locked buffers of its own: while the bus moves one, the thread fills (or empties)
// the other. How many threads, and how much at a time, is measured (us, 16 cores):
//   to the device   five threads keep the bus busy and more only contend for it; 2 MB at a time, or 512 KB where that would leave
//                   threads with less than four chunks (6 MB 970 -> 590, 24 MB 2000 -> 1030, 112 MB 4740 -> 3890,
//                   against eight threads and 1 MB)
//   to the host     the pages written to are often fresh, and faulting them in is what takes the time: eight threads, 1 MB at a
//                   time (112 MB 6800; five threads 9700)
// A staging object belongs to its creator (a Runtime): 32 MB of page-locked memory and 7 sleeping threads, made at the
// first large copy and given back by bt_stage_destroy. Calls on one object take turns.
#include "common.cuh"
#include <condition_variable>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

using namespace bt;

namespace {

constexpr size_t kBuffer = 2 << 20;
constexpr size_t kMostThreads = 8, kUpThreads = 5;

struct Stage {
  struct Lane {                       // one thread's buffers and the events that say when each is free
    char *buf[2] = {};
    cudaEvent_t free[2] = {};
  };
  int device;
  std::vector<Lane> lanes;
  std::vector<std::thread> threads;   // lane 0 is the calling thread's
  std::mutex call, lock;
  std::condition_variable wake, idle;
  uint64_t round = 0;                 // copies so far: a thread works once per round
  int working = 0;
  bool stop = false;
  // the copy at hand
  bool up = false;
  char *host = nullptr, *dev = nullptr;
  size_t bytes = 0, chunk = 0, active = 0;   // the lanes from `active` on sit this one out
  cudaStream_t stream = nullptr;
  std::atomic<size_t> next{0};
  std::atomic<int> failed{0};

  cudaError_t chunks(Lane &l) {
    size_t at[2], n[2] = {0, 0};      // of a chunk on its way to the host: where it goes from this buffer
    for (int b = 0;; b ^= 1) {
      if (cudaError_t e = cudaEventSynchronize(l.free[b])) return e;
      if (n[b]) memcpy(host + at[b], l.buf[b], n[b]), n[b] = 0;
      const size_t i = failed ? SIZE_MAX / kBuffer : next++;
      const size_t from = i * chunk;
      if (from >= bytes) {
        if (n[b ^ 1]) continue;       // the other buffer still has one
        return cudaSuccess;
      }
      const size_t size = bytes - from < chunk ? bytes - from : chunk;
      if (up) memcpy(l.buf[b], host + from, size);
      else at[b] = from, n[b] = size;
      if (cudaError_t e = up ? cudaMemcpyAsync(dev + from, l.buf[b], size, cudaMemcpyHostToDevice, stream) : cudaMemcpyAsync(l.buf[b], dev + from, size, cudaMemcpyDeviceToHost, stream)) return e;
      if (cudaError_t e = cudaEventRecord(l.free[b], stream)) return e;
    }
  }
  void work(Lane &l) {
    if (cudaError_t e = chunks(l)) failed = (int)e;
  }
  void run(size_t lane) {
    cudaSetDevice(device);
    for (uint64_t seen = 0;;) {
      {
        std::unique_lock<std::mutex> hold(lock);
        wake.wait(hold, [&] { return stop || round != seen; });
        if (stop) return;
        seen = round;
        if (lane >= active) continue;
      }
      work(lanes[lane]);
      std::lock_guard<std::mutex> hold(lock);
      if (--working == 0) idle.notify_one();
    }
  }
  cudaError_t copy(bool up_, void *host_, uint64_t dev_, size_t bytes_, cudaStream_t stream_) {
    std::lock_guard<std::mutex> one(call);
    up = up_, host = static_cast<char *>(host_), dev = as_ptr<char>(dev_), bytes = bytes_, stream = stream_, next = 0, failed = 0;
    const size_t most = up && lanes.size() > kUpThreads ? kUpThreads : lanes.size();
    chunk = !up ? kBuffer / 2 : bytes < 4 * kBuffer * most ? kBuffer / 4 : kBuffer;
    const bool several = bytes > 2 * chunk && most > 1;
    if (several) {
      std::lock_guard<std::mutex> hold(lock);
      round++, active = most, working = (int)most - 1;
      wake.notify_all();
    }
    work(lanes[0]);
    if (several) {
      std::unique_lock<std::mutex> hold(lock);
      idle.wait(hold, [&] { return working == 0; });
    }
    return (cudaError_t)(int)failed;
  }
  ~Stage() {
    {
      std::lock_guard<std::mutex> hold(lock);
      stop = true;
      wake.notify_all();
    }
    for (auto &t : threads) t.join();
    for (auto &l : lanes)
      for (int b = 0; b < 2; b++) {
        if (l.free[b]) cudaEventSynchronize(l.free[b]), cudaEventDestroy(l.free[b]);
        if (l.buf[b]) cudaFreeHost(l.buf[b]);
      }
  }
};

}  // namespace

extern "C" {

int bt_stage_create(int device, uint64_t *stage) {
  BT_REQUIRE(stage, "bt_stage_create: null result");
  if (int s = use_device(device)) return s;
  const unsigned cores = std::thread::hardware_concurrency();
  try {                                // memory, and threads where a process may have only so many
    auto st = std::make_unique<Stage>();
    st->device = device;
    st->lanes.resize(cores < 2 ? 1 : cores < kMostThreads ? cores : kMostThreads);
    for (auto &l : st->lanes)
      for (int b = 0; b < 2; b++) {
        cudaError_t e = cudaMallocHost(&l.buf[b], kBuffer);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&l.free[b], cudaEventDisableTiming);
        if (e != cudaSuccess) {
          cudaGetLastError();
          return fail(BT_NO_MEMORY, "no page-locked memory for a staging object: %s", cudaGetErrorString(e));
        }
      }
    st->threads.reserve(st->lanes.size());
    for (size_t i = 1; i < st->lanes.size(); i++) st->threads.emplace_back(&Stage::run, st.get(), i);
    *stage = reinterpret_cast<uint64_t>(st.release());
    return BT_OK;
  } catch (const std::exception &e) {
    return fail(BT_NO_MEMORY, "no memory or threads for a staging object: %s", e.what());
  }
}

int bt_stage_destroy(uint64_t stage) {
  delete as_ptr<Stage>(stage);
  return BT_OK;
}

int bt_stage_upload(uint64_t stage, uint64_t dst, const void *src, size_t bytes, uint64_t stream) {
  BT_REQUIRE(stage && dst && src && bytes, "bt_stage_upload: null staging object or address, or no bytes");
  Stage *st = as_ptr<Stage>(stage);
  if (int s = use_device(st->device)) return s;
  return cuda_status(st->copy(true, const_cast<void *>(src), dst, bytes, as_stream(stream)), "bt_stage_upload");
}

int bt_stage_download(uint64_t stage, void *dst, uint64_t src, size_t bytes, uint64_t stream) {
  BT_REQUIRE(stage && dst && src && bytes, "bt_stage_download: null staging object or address, or no bytes");
  Stage *st = as_ptr<Stage>(stage);
  if (int s = use_device(st->device)) return s;
  return cuda_status(st->copy(false, dst, src, bytes, as_stream(stream)), "bt_stage_download");
}

}  // extern "C"
