// Runs copy_fields (csrc/dropin_copy.cu, compiled as host C++) over a stand-in
// for the CUDA runtime whose "device" is host memory and whose streams hold
// their copies until something waits for them, so that what a call leaves in
// flight can be counted and any runtime call can be made to fail.
// usage: dropin_copy_check <scenario>; exit status 0: as it should be.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "dropin_ctx.cuh"

namespace {

struct Copy {
  void* dst;
  const void* src;
  size_t n;
};
struct Stream {
  std::vector<Copy> queued;
};
std::mutex mu;
std::set<Stream*> streams;
std::map<void*, Stream*> events;           // event -> stream it was recorded on
std::vector<char*> pinned;                 // live pinned buffers
int allocations = 0;                       // pinned buffers made so far
int copies = 0, waits = 0;                 // calls so far
int fail_copy = -1, fail_wait = -1;        // the call that fails, counted from 0
int plain = 0, pieces = 0;                 // copies on the caller's stream, and on others
Stream* caller = nullptr;
thread_local int device = 0;               // each thread's current device
std::map<const void*, cudaMemoryType> kinds;   // arrays that are not ordinary host memory

void finish(Stream* s) {
  for (const Copy& c : s->queued) std::memcpy(c.dst, c.src, c.n);
  s->queued.clear();
}
bool wrong_device = false;                 // a worker's copy issued on another device than the pool's (1)
size_t in_flight() {
  size_t n = 0;
  for (Stream* s : streams) n += s->queued.size();
  return n;
}
Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  std::lock_guard<std::mutex> g(mu);
  pinned.push_back((char*)(*p = std::malloc(n)));
  ++allocations;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> g(mu);
  pinned.erase(std::find(pinned.begin(), pinned.end(), (char*)p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::mutex> g(mu);
  Stream* n = new Stream;
  streams.insert(n);
  *s = reinterpret_cast<cudaStream_t>(n);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  finish(of(s));
  streams.erase(of(s));
  delete of(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  finish(of(s));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new char);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<char*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  events[e] = of(s);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> g(mu);
  if (waits++ == fail_wait) return cudaErrorUnknown;
  finish(events[e]);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = kinds.count(p) ? kinds[p] : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  if (of(s) != caller && device != 1) wrong_device = true;
  if (!dst || !src) return cudaErrorInvalidValue;
  if (copies++ == fail_copy) return cudaErrorUnknown;
  of(s)->queued.push_back(Copy{dst, src, n});
  ++(of(s) == caller ? plain : pieces);
  return cudaSuccess;
}
}

using namespace amss;

namespace {

#define EXPECT(c)                                              \
  do {                                                         \
    if (!(c)) {                                                \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #c);     \
      std::exit(1);                                            \
    }                                                          \
  } while (0)

constexpr int kFields = 12;
constexpr size_t kBytes = (size_t)1300 * 1000;   // a piece and a remainder; 15.6 MB in all
std::vector<std::vector<char>> host(kFields), dev(kFields);
cudaStream_t stream;

// Pools of which the next large call makes one.
struct Ready : CopyPools {
  Ready() { plain = kPoolEarned; }
};

std::vector<CopyField> fields() {
  std::vector<CopyField> f;
  for (int m = 0; m < kFields; ++m) f.push_back(CopyField{dev[m].data(), host[m].data()});
  return f;
}
void fill() {
  for (int m = 0; m < kFields; ++m) {
    host[m].assign(kBytes, 0);
    dev[m].assign(kBytes, 0);
    for (size_t i = 0; i < kBytes; ++i) {
      host[m][i] = (char)(7 * m + i % 251);
      dev[m][i] = (char)(5 * m + i % 241 + 1);
    }
  }
}

// A failed call leaves nothing in flight: its pinned pieces and the device
// arrays may be reused at once.  The calls after it take the plain copies.
void failed(int at_copy, int at_wait) {
  for (const bool to_device : {true, false}) {
    Ready pool;
    fill();
    copies = waits = 0;
    fail_copy = at_copy;
    fail_wait = at_wait;
    EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, to_device, stream) == cudaErrorUnknown);
    EXPECT(in_flight() == 0);
    fail_copy = fail_wait = -1;
    fill();
    plain = pieces = 0;
    EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, to_device, stream) == cudaSuccess);
    cudaStreamSynchronize(stream);
    EXPECT(plain == kFields && pieces == 0);
    EXPECT(host == dev);
  }
}

void works() {
  for (const bool to_device : {true, false}) {
    Ready pool;
    fill();
    plain = pieces = 0;
    EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, to_device, stream) == cudaSuccess);
    EXPECT(in_flight() == 0 && plain == 0 && pieces == 2 * kFields);
    EXPECT(host == dev);
  }
}

// Arrays that are pinned or managed already go by plain copies, the others of
// the same call by threads.
void not_pageable(cudaMemoryType t, int n, bool rest_threaded) {
  for (const bool to_device : {true, false}) {
    Ready pool;
    fill();
    kinds.clear();
    for (int m = 0; m < n; ++m) kinds[host[m].data()] = t;
    plain = pieces = 0;
    EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, to_device, stream) == cudaSuccess);
    cudaStreamSynchronize(stream);
    EXPECT(plain == (rest_threaded ? n : kFields) && pieces == (rest_threaded ? 2 * (kFields - n) : 0));
    EXPECT(host == dev);
  }
}

// A null pointer is refused with the runtime's error, as by the plain copies.
void null_pointer() {
  for (const bool to_device : {true, false}) {
    Ready pool;
    fill();
    std::vector<CopyField> f = fields();
    f[3].host = nullptr;
    EXPECT(copy_fields(pool, f.data(), kFields, kBytes, to_device, stream) == cudaErrorInvalidValue);
    cudaStreamSynchronize(stream);
  }
}

// Output arrays that share memory hold the later field's values, as after
// copies one after another; inputs that do are only read.
void shared(size_t offset) {
  Ready pool;
  fill();
  std::vector<CopyField> f = fields();
  host[2].resize(kBytes + offset);
  f[7].host = host[2].data() + offset;
  f[2].host = host[2].data();
  plain = pieces = 0;
  EXPECT(copy_fields(pool, f.data(), kFields, kBytes, false, stream) == cudaSuccess);
  cudaStreamSynchronize(stream);
  EXPECT(plain == kFields && pieces == 0);
  EXPECT(std::memcmp(f[7].host, dev[7].data(), kBytes) == 0);
  plain = pieces = 0;
  EXPECT(copy_fields(pool, f.data(), kFields, kBytes, true, stream) == cudaSuccess);
  EXPECT(plain == 0 && pieces == 2 * kFields);
  EXPECT(std::memcmp(f[7].host, dev[7].data(), kBytes) == 0 && std::memcmp(f[2].host, dev[2].data(), kBytes) == 0);
}

// Outputs that lie one behind the other share nothing.
void adjacent() {
  Ready pool;
  fill();
  std::vector<char> all(kFields * kBytes);
  std::vector<CopyField> f = fields();
  for (int m = 0; m < kFields; ++m) f[m].host = all.data() + m * kBytes;
  plain = pieces = 0;
  EXPECT(copy_fields(pool, f.data(), kFields, kBytes, false, stream) == cudaSuccess);
  EXPECT(plain == 0 && pieces == 2 * kFields);
  for (int m = 0; m < kFields; ++m) EXPECT(std::memcmp(f[m].host, dev[m].data(), kBytes) == 0);
}

// The copies leave the calling thread's current device as it is, and a call
// made on another device than the pool's takes the plain copies.
void devices() {
  Ready pool;
  cudaSetDevice(1);
  fill();
  wrong_device = false;
  EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, true, stream) == cudaSuccess);
  EXPECT(device == 1 && !wrong_device && host == dev);
  cudaSetDevice(2);
  for (const bool to_device : {true, false}) {
    fill();
    plain = pieces = 0;
    EXPECT(copy_fields(pool, fields().data(), kFields, kBytes, to_device, stream) == cudaSuccess);
    cudaStreamSynchronize(stream);
    EXPECT(device == 2 && plain == kFields && pieces == 0 && host == dev);
  }
}

// Calls that each come from a thread of their own share a pool, and none is
// made before its cost is earned.
void thread_a_call() {
  CopyPools pools;
  const size_t all = kFields * kBytes;
  size_t done = 0;
  for (int call = 0; call < 60; ++call, done += all) {
    fill();
    plain = pieces = 0;
    cudaError_t e = cudaErrorUnknown;
    std::thread([&] { e = copy_fields(pools, fields().data(), kFields, kBytes, call & 1, stream); }).join();
    EXPECT(e == cudaSuccess);
    cudaStreamSynchronize(stream);
    EXPECT(host == dev);
    EXPECT(done < kPoolEarned ? plain == kFields && allocations == 0 : pieces == 2 * kFields && allocations == 1);
  }
}

// Six threads at once: at most kMaxPools pools, and each thread's own data.
void threads_at_once() {
  CopyPools pools;
  std::vector<std::thread> t;
  std::vector<int> good(6, 0);
  for (int k = 0; k < 6; ++k)
    t.emplace_back([&, k] {
      const size_t bytes = 3 << 20;
      std::vector<std::vector<char>> h(4, std::vector<char>(bytes)), d(4, std::vector<char>(bytes));
      std::vector<CopyField> f;
      for (int m = 0; m < 4; ++m) f.push_back(CopyField{d[m].data(), h[m].data()});
      for (int call = 0; call < 40; ++call) {
        for (int m = 0; m < 4; ++m) std::memset((call & 1 ? h : d)[m].data(), 31 * k + 7 * m + call, bytes);
        if (copy_fields(pools, f.data(), 4, bytes, call & 1, stream) != cudaSuccess) return;
        cudaStreamSynchronize(stream);
        if (h != d) return;
      }
      good[k] = 1;
    });
  for (auto& x : t) x.join();
  EXPECT(std::count(good.begin(), good.end(), 1) == 6);
  EXPECT(allocations >= 1 && allocations <= kMaxPools);
}

}  // namespace

int main(int, char** argv) {
  cudaStreamCreateWithFlags(&stream, 0);
  caller = of(stream);
  const std::string s = argv[1];
  if (s == "works") works();
  else if (s == "copy_fails") failed(20, -1);
  else if (s == "wait_fails") failed(-1, 5);
  else if (s == "pinned") not_pageable(cudaMemoryTypeHost, kFields, false);
  else if (s == "managed") not_pageable(cudaMemoryTypeManaged, kFields, false);
  else if (s == "some_pinned") not_pageable(cudaMemoryTypeHost, 4, true);
  else if (s == "few_pageable") not_pageable(cudaMemoryTypeHost, 8, false);   // 5.2 MB of pageable arrays
  else if (s == "device") not_pageable(cudaMemoryTypeDevice, kFields, false);
  else if (s == "null") null_pointer();
  else if (s == "same_array") shared(0);
  else if (s == "overlap") shared(sizeof(double));
  else if (s == "adjacent") adjacent();
  else if (s == "devices") devices();
  else if (s == "thread_a_call") thread_a_call();
  else if (s == "threads_at_once") threads_at_once();
  else return 2;
  EXPECT(pinned.empty());   // given back with the pool
  return 0;
}
