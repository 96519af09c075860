#include "host_copy.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

namespace Deep
{
std::shared_ptr<HostCopier> HostCopier::Shared()
{
  static std::mutex m;
  static std::weak_ptr<HostCopier> current;
  std::lock_guard<std::mutex> g(m);
  std::shared_ptr<HostCopier> p = current.lock();
  if (!p)
    current = p = std::shared_ptr<HostCopier>(new HostCopier());
  return p;
}

HostCopier::HostCopier()
{
  const unsigned cores = std::thread::hardware_concurrency();
  const int n = cores >= 8 ? 3 : cores >= 4 ? 1 : 0;
  for (int i = 0; i < n; ++i)
    helpers.emplace_back([this] { Loop(); });
}

HostCopier::~HostCopier()
{
  {
    std::lock_guard<std::mutex> g(lock);
    stop = true;
  }
  wake.notify_all();
  for (auto& t : helpers)
    t.join();
}

void HostCopier::Work(Job& j)
{
  for (;;)
  {
    const size_t at = j.next.fetch_add(j.chunk);
    if (at >= j.bytes)
      return;
    const size_t n = std::min(j.chunk, j.bytes - at);
    std::memcpy(j.stage + at, j.data + at, n);
    const int rc = dpc_copy_h2d(j.ctx, j.dst + at, j.stage + at, n);
    if (rc != DPC_OK)
      j.status.store(rc);
  }
}

void HostCopier::Loop()
{
  unsigned seen = 0;
  std::unique_lock<std::mutex> g(lock);
  for (;;)
  {
    wake.wait(g, [&] { return stop || (job && generation != seen); });
    if (stop)
      return;
    seen = generation;
    Job* j = job;
    ++busy;
    g.unlock();
    if (cudaSetDevice(j->device) == cudaSuccess)
      Work(*j);
    g.lock();
    if (--busy == 0)
      done.notify_all();
  }
}

int HostCopier::Upload(dpc_ctx* ctx, int device, float* dst, float* stage, const float* data, size_t count)
{
  Job j;
  j.ctx = ctx, j.device = device;
  j.dst = reinterpret_cast<char*>(dst), j.stage = reinterpret_cast<char*>(stage);
  j.data = reinterpret_cast<const char*>(data);
  j.bytes = count * sizeof(float);
  // about four chunks per thread, 128 KB to 1 MB
  j.chunk = std::min<size_t>(std::max<size_t>(j.bytes / 16, 128 << 10), 1 << 20) & ~(size_t)4095;
  const bool mine = !helpers.empty() && callers.try_lock();
  if (mine)
  {
    {
      std::lock_guard<std::mutex> g(lock);
      job = &j;
      ++generation;
    }
    wake.notify_all();
  }
  Work(j);
  if (mine)
  {
    // no helper may still be in a chunk, or pick the job up later
    std::unique_lock<std::mutex> g(lock);
    job = nullptr;
    done.wait(g, [&] { return busy == 0; });
    g.unlock();
    callers.unlock();
  }
  return j.status.load();
}
} // namespace Deep
