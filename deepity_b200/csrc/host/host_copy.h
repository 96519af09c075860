// Copies from ordinary host memory to the device, for the networks' inputs.
//
// A train step from host batches starts with a copy into pinned memory and one to the device: one core
// moves about 10 GB/s, a fifth of what the link takes, so 12 MB of inputs cost 1.2 ms of a 2.4 ms
// prediction.  Large inputs go in chunks instead: the caller and up to three helper threads each copy a
// chunk into the pinned buffer and send it on its way at once.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "deepity_b200.h"

namespace Deep
{
// The helper threads: one set per process, started by the first large copy, shared by all networks
// and joined when the last network that used them is gone.  Calls from several threads are safe: one
// of them gets the helpers, the others copy by themselves meanwhile.
class HostCopier
{
public:
  static std::shared_ptr<HostCopier> Shared();
  ~HostCopier();
  // data -> stage (pinned) -> dst (device), stream-ordered on the context; stage must not be in use.
  // Returns when data has been read and every chunk is enqueued.  Returns a dpc_status.
  int Upload(dpc_ctx* ctx, int device, float* dst, float* stage, const float* data, size_t count);

  // Below this the wake-up of the helpers costs what they save.
  static constexpr size_t kMinFloats = 96 * 1024;

private:
  HostCopier();
  struct Job
  {
    dpc_ctx* ctx;
    int device;
    char *dst, *stage;
    const char* data;
    size_t bytes, chunk;
    std::atomic<size_t> next{0};
    std::atomic<int> status{0};
  };
  static void Work(Job& job);
  void Loop();

  std::vector<std::thread> helpers;
  std::mutex callers; // held by the call that has the helpers
  std::mutex lock;
  std::condition_variable wake, done;
  Job* job = nullptr;
  unsigned generation = 0;
  int busy = 0;
  bool stop = false;
};
} // namespace Deep
