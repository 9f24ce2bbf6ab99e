// The block pool of tl_alloc / tl_free on a fake device: addresses are made up, every call is counted, and the next
// cudaMalloc or cudaFree can be made to fail.  Built with tl_pool.cu by tests/test_pool_cpu.py; argv[1] names the test.
#include "tl_pool.cuh"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>

static std::map<uintptr_t, size_t> device;  // what is allocated
static uintptr_t next_address = 1 << 20;
static int mallocs = 0, frees = 0;
static cudaError_t fail_malloc = cudaSuccess, fail_free = cudaSuccess;  // every call fails with this
static size_t memory = SIZE_MAX;  // cudaMalloc fails beyond this

extern "C" {
cudaError_t cudaMalloc(void** out, size_t bytes) {
  ++mallocs;
  if (fail_malloc != cudaSuccess) return fail_malloc;
  size_t used = 0;
  for (const auto& d : device) used += d.second;
  if (bytes > memory || used > memory - bytes) return cudaErrorMemoryAllocation;
  *out = reinterpret_cast<void*>(next_address);
  device[next_address] = bytes;
  next_address += (bytes + 511) / 512 * 512 + 512;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  ++frees;
  if (fail_free != cudaSuccess) return fail_free;
  return device.erase(reinterpret_cast<uintptr_t>(p)) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {  // spoils the captures of others
  fprintf(stderr, "cudaDeviceSynchronize called\n");
  exit(1);
}
}

#define CHECK(x) \
  do { if (!(x)) { fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #x); exit(1); } } while (0)

static void* take(TlBlockPool& pool, size_t bytes) {
  void* p = nullptr;
  CHECK(pool.alloc(bytes, &p) == cudaSuccess && p && device.count(reinterpret_cast<uintptr_t>(p)));
  CHECK(device[reinterpret_cast<uintptr_t>(p)] >= bytes);
  return p;
}
static void give(TlBlockPool& pool, void* p) {
  bool known = false;
  CHECK(pool.free(p, &known) == cudaSuccess && known);
}

// a block comes out again only after a cudaFree that came after it was given back
static void reuse() {
  TlBlockPool pool;
  std::map<void*, int> given;  // block: frees so far when it was given back
  std::set<void*> held;
  int again = 0;
  for (int i = 0; i < 4000; ++i) {
    void* p = take(pool, size_t(1) << (i % 11 + 3));
    CHECK(held.insert(p).second);
    if (given.count(p)) { CHECK(frees > given[p]); ++again; }
    if (i % 3) { given[p] = frees; held.erase(p); give(pool, p); }
  }
  CHECK(again > 1000);
  for (void* p : held) give(pool, p);
  pool.release();
  CHECK(device.empty() && pool.live.empty() && pool.ready_bytes == 0 && pool.waiting_bytes == 0);
}

// a fence that fails leaves the block with the caller, and everything else as it was
static void failing_fence() {
  for (size_t bytes : {size_t(100), size_t(30) << 20}) {
    TlBlockPool pool;
    std::set<void*> held;
    for (int i = 0; i < 80; ++i) held.insert(take(pool, bytes));
    CHECK(held.size() == 80);
    fail_free = cudaErrorStreamCaptureUnsupported;
    int refused = 0;
    for (auto it = held.begin(); it != held.end();) {
      bool known = false;
      const cudaError_t e = pool.free(*it, &known);
      CHECK(known);
      refused += e != cudaSuccess;
      it = e == cudaSuccess ? held.erase(it) : std::next(it);
    }
    CHECK(refused > 0 && refused == int(held.size()) && pool.live.size() == held.size());
    for (int i = 0; i < 80; ++i) {
      void* p = take(pool, bytes);
      CHECK(held.insert(p).second);  // none of the caller's, none of those that wait
    }
    fail_free = cudaSuccess;
    for (void* p : held) give(pool, p);
    pool.release();
    CHECK(device.empty() && pool.live.empty());
  }
}

// without memory for the fence's own block the given block goes back and is the fence
static void no_memory_for_the_fence() {
  TlBlockPool pool;
  std::vector<void*> held;
  for (int i = 0; i < 64; ++i) held.push_back(take(pool, 100));
  fail_malloc = cudaErrorMemoryAllocation;
  for (void* p : held) give(pool, p);
  CHECK(pool.waiting.empty() && pool.ready.size() == 63 && device.size() == 63);
  fail_malloc = cudaSuccess;
  pool.release();
  CHECK(device.empty());
}

static void bounds() {
  TlBlockPool pool;
  void* p = take(pool, TlBlockPool::kLargestBytes + 1);
  give(pool, p);  // straight back
  CHECK(device.empty());
  std::vector<void*> held;
  for (int i = 0; i < 40; ++i) held.push_back(take(pool, size_t(60) << 20));
  for (void* q : held) {
    give(pool, q);
    CHECK(pool.ready_bytes + pool.waiting_bytes <= TlBlockPool::kKeptBytes);
  }
  pool.keep_at_most(size_t(100) << 20);
  CHECK(device.size() == pool.live.size() && pool.ready_bytes + pool.waiting_bytes == 0);  // all that was kept went back
  held.clear();
  for (int i = 0; i < 20; ++i) held.push_back(take(pool, size_t(20) << 20));
  for (void* q : held) {
    give(pool, q);
    CHECK(pool.ready_bytes + pool.waiting_bytes <= size_t(100) << 20);
  }
  CHECK(pool.ready_bytes + pool.waiting_bytes > 0);
  pool.keep_at_most(0);
  give(pool, take(pool, 1));
  CHECK(device.empty());
  pool.keep_at_most(TlBlockPool::kKeptBytes);
  bool known = false;
  p = take(pool, 100);
  give(pool, p);
  CHECK(pool.free(p, &known) == cudaErrorInvalidValue && known);  // given back twice
  CHECK(pool.free(&known, &known) == cudaSuccess && !known);                 // not from here
  pool.release();
  CHECK(device.empty());
}

// memory is short: what every pool of the device keeps goes back, for the library's own buffers as for blocks
static void short_of_memory() {
  for (int own = 0; own < 2; ++own) {
    TlBlockPool a, b, other;
    a.device = b.device = 0;
    other.device = 1;
    void* still = take(a, 10 << 20);
    for (TlBlockPool* p : {&a, &b, &other}) give(*p, take(*p, 100 << 20));
    memory = size_t(320) << 20;
    void* p = nullptr;
    const cudaError_t e = own ? b.device_malloc(&p, 200 << 20) : b.alloc(200 << 20, &p);
    CHECK(e == cudaSuccess && p && device.count(reinterpret_cast<uintptr_t>(still)));
    CHECK(a.waiting_bytes + a.ready_bytes == 0 && b.waiting_bytes + b.ready_bytes == 0 && other.waiting_bytes + other.ready_bytes > 0);
    CHECK((own ? a.device_malloc(&p, 200 << 20) : a.alloc(200 << 20, &p)) == cudaErrorMemoryAllocation);
    memory = SIZE_MAX;
    device.clear();
    a.live.clear(); b.live.clear(); other.waiting.clear();
  }
}

int main(int, char** argv) {
  const struct { const char* name; void (*run)(); } tests[] = {
      {"reuse", reuse}, {"failing_fence", failing_fence}, {"no_memory_for_the_fence", no_memory_for_the_fence}, {"bounds", bounds},
      {"short_of_memory", short_of_memory}};
  for (const auto& t : tests)
    if (!strcmp(t.name, argv[1])) { t.run(); return 0; }
  return 2;
}
