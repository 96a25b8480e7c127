#include "device.h"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

namespace gb {

namespace {
DeviceState g_dev;
std::map<void *, size_t> g_live;
size_t g_live_bytes = 0;
// allocations made since track_alloc(true), by label, with their high-water mark: the reference's
// _debug_track_alloc / _debug_live_alloc / _debug_peak_alloc (python/kk/kk_core.cpp:143-184)
bool g_track = false;
std::map<void *, std::pair<std::string, size_t>> g_tracked;
size_t g_tracked_bytes = 0, g_tracked_peak = 0;
}    // namespace

void track_alloc(bool on)
{
  g_tracked.clear();
  g_tracked_bytes = g_tracked_peak = 0;
  g_track = on;
}

size_t tracked_peak_bytes() { return g_tracked_peak; }

std::vector<std::pair<std::string, size_t>> tracked_live()
{
  std::map<std::string, size_t> by;
  for (const auto &kv : g_tracked) by[kv.second.first] += kv.second.second;
  std::vector<std::pair<std::string, size_t>> v(by.begin(), by.end());
  std::sort(v.begin(), v.end(), [](const auto &a, const auto &b) { return a.second > b.second; });
  return v;
}

DeviceState &dev() { return g_dev; }

void require_initialized()
{
  if (!g_dev.initialized) throw DeviceError("the GPU backend is not initialised (call grace_initialize first) or was finalised");
}

void cuda_check(cudaError_t e, const char *what)
{
  if (e == cudaSuccess) return;
  const std::string msg = std::string("CUDA error: ") + cudaGetErrorString(e) + " in " + what;
  if (e == cudaErrorMemoryAllocation) {
    (void) cudaGetLastError();    // the allocation error is not sticky: clear it so the context stays usable
    throw OutOfMemory(msg);
  }
  throw DeviceError(msg);
}

namespace {
struct ProfSpan { std::string name; cudaEvent_t a, b; };
const char *g_tag = nullptr;
bool g_prof_on = false;
std::vector<ProfSpan> g_prof;
std::vector<cudaEvent_t> g_prof_pool;
size_t g_prof_used = 0;
cudaEvent_t prof_event()
{
  if (g_prof_used == g_prof_pool.size()) {
    cudaEvent_t e;
    GB_CUDA(cudaEventCreate(&e));
    g_prof_pool.push_back(e);
  }
  return g_prof_pool[g_prof_used++];
}
}    // namespace

void launch_tag(const char *tag) { g_tag = tag; }

void profile_enable(bool on)
{
  g_prof_on = on;
  g_prof.clear();
  g_prof_used = 0;
}

std::string profile_report()
{
  if (g_dev.initialized) cudaStreamSynchronize(g_dev.stream);
  std::map<std::string, std::pair<long long, double>> acc;
  for (const auto &s : g_prof) {
    float ms = 0.0f;
    if (cudaEventElapsedTime(&ms, s.a, s.b) != cudaSuccess) continue;
    auto &e = acc[s.name];
    e.first++;
    e.second += ms;
  }
  std::string out;
  for (const auto &kv : acc) out += kv.first + " " + std::to_string(kv.second.first) + " " + std::to_string(kv.second.second) + "\n";
  return out;
}

void before_launch(const char *name)
{
  if (!g_prof_on) return;
  ProfSpan s{g_tag ? std::string(name) + ":" + g_tag : std::string(name), prof_event(), prof_event()};
  cudaEventRecord(s.a, g_dev.stream);
  g_prof.push_back(s);
}

void after_launch(const char *name)
{
  if (g_prof_on && !g_prof.empty()) cudaEventRecord(g_prof.back().b, g_dev.stream);
  g_dev.launches++;
  if (g_dev.fail_launch_nth > 0 && --g_dev.fail_launch_nth == 0)
    throw OutOfMemory(std::string("kernel launch ran out of device memory (injected) in ") + name);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) cuda_check(e, name);
}

namespace {
constexpr size_t POOL_BLOCK = (size_t) 1 << 30, POOL_TOTAL = (size_t) 4 << 30;
std::mutex g_pool_mu;
std::multimap<size_t, void *> g_pool;    // free blocks by size
std::map<void *, size_t> g_block;        // size of every block that came from the driver
size_t g_pool_bytes = 0;

// a pooled block of at least `bytes` that wastes at most as much again (small ones: 64 KB), or null
void *pool_take(size_t bytes)
{
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pool.lower_bound(bytes);
  if (it == g_pool.end() || it->first > 2 * bytes + ((size_t) 64 << 10)) return nullptr;
  void *p = it->second;
  g_pool_bytes -= it->first;
  g_pool.erase(it);
  return p;
}

void driver_free(void *p)
{
  if (g_dev.initialized) cudaFree(p);
}

void pool_give(void *p)
{
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_block.find(p);
    if (it != g_block.end() && it->second <= POOL_BLOCK && g_pool_bytes + it->second <= POOL_TOTAL && g_dev.initialized) {
      g_pool.emplace(it->second, p);
      g_pool_bytes += it->second;
      return;
    }
    if (it != g_block.end()) g_block.erase(it);
  }
  driver_free(p);
}
}    // namespace

void device_pool_trim()
{
  std::lock_guard<std::mutex> lk(g_pool_mu);
  for (auto &kv : g_pool) {
    g_block.erase(kv.second);
    driver_free(kv.second);
  }
  g_pool.clear();
  g_pool_bytes = 0;
}

size_t device_free_bytes()
{
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = (size_t) 8 << 30;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  return free_b + g_pool_bytes;
}

void *device_alloc(size_t bytes, const char *label)
{
  require_initialized();
  if (bytes == 0) bytes = 16;
  void *p = pool_take(bytes);
  if (!p) {
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
      (void) cudaGetLastError();
      device_pool_trim();
      GB_CUDA(cudaMalloc(&p, bytes));
    }
    std::lock_guard<std::mutex> lk(g_pool_mu);
    g_block[p] = bytes;
  }
  // the injected failure comes after the allocation, as the reference's hook does (kk_core.cpp:128-141): the buffer is
  // returned before the error is raised
  if (g_dev.fail_alloc_nth > 0 && label && std::strstr(label, g_dev.fail_label.c_str()) != nullptr &&
      --g_dev.fail_alloc_nth == 0) {
    pool_give(p);
    throw OutOfMemory(std::string("out of device memory (injected) allocating '") + label + "'");
  }
  g_live[p] = bytes;
  g_live_bytes += bytes;
  if (g_track) {
    g_tracked[p] = {label ? label : "buffer", bytes};
    g_tracked_bytes += bytes;
    g_tracked_peak = std::max(g_tracked_peak, g_tracked_bytes);
  }
  return p;
}

void device_free(void *p)
{
  if (!p) return;
  auto it = g_live.find(p);
  if (it != g_live.end()) {
    g_live_bytes -= it->second;
    g_live.erase(it);
  }
  auto tr = g_tracked.find(p);
  if (tr != g_tracked.end()) {    // allocated before tracking started: not counted
    g_tracked_bytes -= tr->second.second;
    g_tracked.erase(tr);
  }
  pool_give(p);
}

char *PinnedBuf::ensure(size_t bytes)
{
  if (bytes <= cap_) return p_;
  release();
  const size_t want = bytes + bytes / 2 + 4096;
  void *p = nullptr;
  if (cudaMallocHost(&p, want) != cudaSuccess) {
    (void) cudaGetLastError();
    return nullptr;
  }
  p_ = static_cast<char *>(p);
  cap_ = want;
  return p_;
}

void PinnedBuf::release()
{
  if (p_ && g_dev.initialized) cudaFreeHost(p_);
  p_ = nullptr;
  cap_ = 0;
}

size_t device_bytes_live() { return g_live_bytes; }

StageTimer::~StageTimer()
{
  if (!g_dev.initialized) return;
  for (auto e : pool_) cudaEventDestroy(e);
}

int StageTimer::mark()
{
  if (used_ > 0 && at_launch_ == g_dev.launches) return (int) used_ - 1;    // nothing launched since the last event
  if (used_ == pool_.size()) {
    cudaEvent_t e;
    GB_CUDA(cudaEventCreate(&e));
    pool_.push_back(e);
  }
  GB_CUDA(cudaEventRecord(pool_[used_], g_dev.stream));
  at_launch_ = g_dev.launches;
  return (int) used_++;
}

void StageTimer::reset()
{
  spans_.clear();
  used_ = 0;
  at_launch_ = ~0ull;
  for (int s = 0; s < NSTAGE; s++) open_[s] = -1;
}

void StageTimer::begin(int stage)
{
  open_[stage] = (int) spans_.size();
  spans_.push_back(Span{stage, mark(), -1});
}

void StageTimer::end(int stage)
{
  if (open_[stage] < 0) return;
  spans_[open_[stage]].b = mark();
  open_[stage] = -1;
}

void StageTimer::collect(double *ms)
{
  for (int s = 0; s < NSTAGE; s++) ms[s] = 0.0;
  for (const Span &sp : spans_) {
    if (sp.b <= sp.a) continue;    // not closed, or nothing was launched inside
    float t = 0.0f;
    if (cudaEventElapsedTime(&t, pool_[sp.a], pool_[sp.b]) == cudaSuccess) ms[sp.stage] += t;
  }
}

}    // namespace gb
