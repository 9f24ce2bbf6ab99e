// The pool of device blocks behind tl_alloc / tl_free (host code only).
#include "tl_pool.cuh"

#include <algorithm>
#include <cstdint>
#include <iterator>

namespace {
std::mutex pools_lock;  // taken before a pool's own
std::vector<TlBlockPool*>& pools() {
  static auto* all = new std::vector<TlBlockPool*>;  // never destroyed: a context may go after the library's statics
  return *all;
}
}  // namespace

TlBlockPool::TlBlockPool() {
  std::lock_guard<std::mutex> hold(pools_lock);
  pools().push_back(this);
}

TlBlockPool::~TlBlockPool() {
  std::lock_guard<std::mutex> hold(pools_lock);
  pools().erase(std::find(pools().begin(), pools().end(), this));
}

void TlBlockPool::release_device() {
  std::lock_guard<std::mutex> hold(pools_lock);
  for (TlBlockPool* p : pools())
    if (p->device == device) p->release();
}

cudaError_t TlBlockPool::device_malloc(void** out, size_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  release_device();
  return cudaMalloc(out, bytes);
}

void TlBlockPool::fenced() {
  while (!waiting.empty()) {
    const auto w = waiting.back();
    ready.emplace(w.second, w.first);
    waiting.pop_back();
    ready_bytes += w.second;
    waiting_bytes -= w.second;
  }
}

void TlBlockPool::trim(size_t keep) {
  while (!ready.empty() && ready_bytes > keep) {
    auto last = std::prev(ready.end());
    if (cudaFree(last->second) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    ready_bytes -= last->first;
    ready.erase(last);
  }
}

void TlBlockPool::release() {
  std::lock_guard<std::mutex> hold(lock);
  while (!waiting.empty()) {
    if (cudaFree(waiting.back().first) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    waiting_bytes -= waiting.back().second;
    waiting.pop_back();
  }
  trim(0);
  if (mark && cudaFree(mark) == cudaSuccess) mark = nullptr;
}

void TlBlockPool::keep_at_most(size_t bytes) {
  release();
  std::lock_guard<std::mutex> hold(lock);
  keep = bytes;
}

cudaError_t TlBlockPool::alloc(size_t bytes, void** out) {
  // capacities in steps of 512 bytes, or of 1/64 to 1/32 of the size where that is more: sizes that differ a little
  // from call to call share blocks, and little is lost in weights that stay
  size_t step = 512;
  while (bytes <= kLargestBytes && step < bytes / 64) step *= 2;
  const size_t cap = bytes > SIZE_MAX / 2 ? bytes : std::max<size_t>(1, (bytes + step - 1) / step) * step;
  std::unique_lock<std::mutex> hold(lock);
  auto it = ready.lower_bound(cap);
  if (it != ready.end() && it->first <= cap + cap / 4) {
    live[it->second] = it->first;
    *out = it->second;
    ready_bytes -= it->first;
    ready.erase(it);
    return cudaSuccess;
  }
  size_t got = cap;
  cudaError_t e = cudaMalloc(out, cap);
  if (e == cudaErrorMemoryAllocation) {  // give back what is kept, then ask for no more than was asked for
    cudaGetLastError();
    hold.unlock();
    release_device();
    hold.lock();
    got = bytes ? bytes : 1;
    e = cudaMalloc(out, got);
  }
  if (e != cudaSuccess) return e;
  try {
    live[*out] = got;
  } catch (...) {
    cudaFree(*out);
    *out = nullptr;
    throw;
  }
  return cudaSuccess;
}

cudaError_t TlBlockPool::free(void* p, bool* known) {
  std::lock_guard<std::mutex> hold(lock);
  auto it = live.find(p);
  *known = it != live.end();
  if (!*known) {
    for (auto& w : waiting) *known = *known || w.first == p;
    for (auto& r : ready) *known = *known || r.second == p;
    return *known ? cudaErrorInvalidValue : cudaSuccess;  // given back twice, or not from here
  }
  const size_t cap = it->second;
  const size_t part = keep / 4;  // kLargestBytes and kWaitingBytes
  const bool full = waiting.size() + 1 >= kWaitingBlocks || waiting_bytes + cap >= part;
  bool kept = cap <= part;
  if (kept && full) {
    cudaError_t e = mark ? cudaSuccess : cudaMalloc(&mark, 256);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      mark = nullptr;
      kept = false;  // short of memory: this block goes back, and is the fence
    } else {
      if (e == cudaSuccess) e = cudaFree(mark);
      if (e != cudaSuccess) return e;
      mark = nullptr;
    }
  }
  if (!kept) {
    cudaError_t e = cudaFree(p);
    if (e != cudaSuccess) return e;
    live.erase(it);
    fenced();
  } else if (full) {
    ready.emplace(cap, p);
    ready_bytes += cap;
    live.erase(it);
    fenced();
  } else {
    waiting.emplace_back(p, cap);
    waiting_bytes += cap;
    live.erase(it);
    return cudaSuccess;
  }
  trim(keep - part);
  return cudaSuccess;
}
