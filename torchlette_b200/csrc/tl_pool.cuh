// Device blocks behind tl_alloc / tl_free.  cudaMalloc and cudaFree map and unmap memory and stop the device: 1.5 ms
// a call that returns 50 MB, 0.5 ms a decoder layer with its fourteen results.  A block that was given back is kept
// and handed out again, but only after a fence that came after it was given back, the promise that cudaFree makes:
// whatever any stream still does with the old contents is over by then.  One fence serves many blocks (kWaitingBlocks,
// kWaitingBytes).
// The fence is a cudaFree, of a 256-byte block made for it: it returns when everything that the device was given before
// is over, on any stream (beside 343 ms of work on a non-blocking stream it took 343 ms, on an idle device 4 us with
// the cudaMalloc).  cudaDeviceSynchronize does the same, but not while any stream of the device is being captured, by
// whatever thread: it is refused then and the capture is lost.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

struct TlBlockPool {
  TlBlockPool();
  ~TlBlockPool();
  TlBlockPool(const TlBlockPool&) = delete;
  TlBlockPool& operator=(const TlBlockPool&) = delete;
  static constexpr size_t kKeptBytes = size_t(1) << 30;     // blocks kept in all, waiting ones included
  static constexpr size_t kLargestBytes = kKeptBytes / 4;   // larger blocks go straight back
  static constexpr size_t kWaitingBytes = kKeptBytes / 4;
  static constexpr size_t kWaitingBlocks = 64;
  std::mutex lock;                            // tl_alloc and tl_free may come from several threads
  std::map<void*, size_t> live;               // handed out: capacity
  std::multimap<size_t, void*> ready;         // free and behind a fence, by capacity
  std::vector<std::pair<void*, size_t>> waiting;  // given back since the last fence
  size_t ready_bytes = 0, waiting_bytes = 0;
  void* mark = nullptr;                       // the fence's block, where its cudaFree failed
  cudaError_t alloc(size_t bytes, void** out);
  // *known: the block is one of the pool's (a pointer from elsewhere is left to the caller).  After an error the block is
  // still the caller's.
  cudaError_t free(void* p, bool* known);
  // cudaMalloc for the library itself (scratch, schedules): where memory is short, what the device's pools keep goes
  // back first
  cudaError_t device_malloc(void** out, size_t bytes);
  void release();  // gives back all that is kept
  void keep_at_most(size_t bytes);  // in place of kKeptBytes; 0: tl_free gives every block straight back
  int device = -1;
  size_t keep = kKeptBytes;

 private:
  void release_device();   // of every context of the device (not with `lock` held)
  void fenced();           // a fence has just passed: waiting blocks become ready
  void trim(size_t keep);  // gives ready blocks back until at most `keep` bytes of them are left, the largest first
};
