// dropin_copy.cu -- the drop-in entries' copies between the caller's arrays
// and the device.
//
// The entries take pageable arrays.  cudaMemcpyAsync moves such an array
// through the driver's staging buffer on the calling thread alone, and the
// first write to a fresh output array faults its pages in on that thread too:
// 20 of the 22 ms of a 54^3 right-hand side (43 MB in, 69 MB out).  Several
// worker threads therefore copy pieces through pinned buffers of their own,
// each with two pieces in flight, so that host copies, page faults and DMA
// overlap: 21.4 -> 9.4 ms a call with 16 cores.  Pieces of 1 MB: 54^3 points take
// 1.4 ms in and 2.5 ms out, with 512 KB 1.8 and 3.2, with 256 KB 2.2 and 3.9, by
// plain copies 2.6 and 5.2.  Small calls, calls that get no pool, arrays that are
// not ordinary host memory and outputs that share memory take the plain copies.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <utility>
#include <vector>

#include "dropin_ctx.cuh"

namespace amss {

CopyPool::~CopyPool() {
  for (int w = 0; w < kCopyWorkers; ++w) {
    for (int s = 0; s < 2; ++s)
      if (done[w][s]) cudaEventDestroy(done[w][s]);
    if (stream[w]) cudaStreamDestroy(stream[w]);
  }
  if (pinned) cudaFreeHost(pinned);
}

bool CopyPool::init(int dev) {
  device = dev;
  bool ok = cudaHostAlloc((void**)&pinned, 2 * kCopyWorkers * kCopyPiece, cudaHostAllocDefault) == cudaSuccess;
  for (int w = 0; ok && w < kCopyWorkers; ++w) {
    ok = cudaStreamCreateWithFlags(&stream[w], cudaStreamNonBlocking) == cudaSuccess;
    for (int s = 0; ok && s < 2; ++s) ok = cudaEventCreateWithFlags(&done[w][s], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) (void)cudaGetLastError();
  return ok;
}

CopyPools& copy_pools() {
  static CopyPools p;   // made after the runtime's own state, so given back before that goes
  return p;
}

std::unique_ptr<CopyPool> CopyPools::take(size_t bytes) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  {
    std::lock_guard<std::mutex> g(lock);
    for (auto& p : idle)
      if (p->device == dev) {
        std::unique_ptr<CopyPool> got = std::move(p);
        p = std::move(idle.back());
        idle.pop_back();
        return got;
      }
    if (failed || made == kMaxPools) return nullptr;
    if (plain < kPoolEarned) {
      plain += bytes;
      return nullptr;
    }
    plain = 0;
    idle.reserve(kMaxPools);   // give() allocates nothing
    ++made;
  }
  std::unique_ptr<CopyPool> pool(new (std::nothrow) CopyPool);
  if (pool && pool->init(dev)) return pool;
  std::lock_guard<std::mutex> g(lock);
  failed = true;
  return nullptr;
}

void CopyPools::give(std::unique_ptr<CopyPool> pool) {
  std::lock_guard<std::mutex> g(lock);
  idle.push_back(std::move(pool));
}

namespace {

struct Piece {
  char* dev;
  char* host;
  size_t n;
};

// One worker: takes pieces until none is left, two in flight.
void work(CopyPool& P, int w, const std::vector<Piece>& v, std::atomic<size_t>& next, bool to_device,
          std::atomic<int>& err) {
  auto ck = [&](cudaError_t e) {
    if (e != cudaSuccess) err.store((int)e);
    return e == cudaSuccess;
  };
  const Piece* held[2] = {nullptr, nullptr};   // the piece in flight in each slot
  auto settle = [&](int s) {
    if (!held[s]) return true;
    if (!ck(cudaEventSynchronize(P.done[w][s]))) return false;
    if (!to_device) std::memcpy(held[s]->host, P.slot(w, s), held[s]->n);
    held[s] = nullptr;
    return true;
  };
  for (int s = 0; err.load() == 0; s ^= 1) {
    if (!settle(s)) return;
    const size_t i = next.fetch_add(1);
    if (i >= v.size()) break;
    const Piece& p = v[i];
    if (to_device) {
      std::memcpy(P.slot(w, s), p.host, p.n);
      if (!ck(cudaMemcpyAsync(p.dev, P.slot(w, s), p.n, cudaMemcpyHostToDevice, P.stream[w]))) return;
    } else {
      if (!ck(cudaMemcpyAsync(P.slot(w, s), p.dev, p.n, cudaMemcpyDeviceToHost, P.stream[w]))) return;
    }
    if (!ck(cudaEventRecord(P.done[w][s], P.stream[w]))) return;
    held[s] = &p;
  }
  for (int s = 0; s < 2; ++s)
    if (!settle(s)) return;
}

// Ordinary host memory.  Pinned and managed arrays move at full rate without
// the threads (55 outputs of 54^3 points: 3.0 ms a call, 4.5 ms through the
// pieces), and a null or a device pointer is the runtime's to refuse.
bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (!p) return false;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// Whether two fields share host memory: of outputs that do, the later field's
// values stay, which only copies one after another keep.
bool share_memory(const CopyField* fields, int nfields, size_t bytes) {
  std::vector<const char*> at;
  for (int m = 0; m < nfields; ++m) at.push_back((const char*)fields[m].host);
  std::sort(at.begin(), at.end());
  for (int m = 1; m < nfields; ++m)
    if ((size_t)(at[m] - at[m - 1]) < bytes) return true;
  return false;
}

}  // namespace

cudaError_t copy_fields(CopyPools& pools, const CopyField* fields, int nfields, size_t bytes, bool to_device,
                        cudaStream_t s) try {
  // Starting the threads costs more than they save on less: at 26^3 points
  // (4.8 MB in, 7.7 MB out) 2.4 ms a call by plain copies, 2.7 to 3.1 ms by
  // threads.  From the line on, where the arrays' pages are there already: at
  // 27^3 (8.7 MB out) 1.67 ms by plain copies and 1.24 with threads, at 30^3 2.07
  // and 1.51, at 34^3 2.67 and 1.70, at 54^3 8.2 and 4.5.
  constexpr size_t kLeast = (size_t)8 << 20;
  // the fields that the threads take
  std::vector<bool> threaded(nfields, false);
  size_t total = 0;
  if (bytes * nfields >= kLeast && (to_device || !share_memory(fields, nfields, bytes)))
    for (int m = 0; m < nfields; ++m)
      if (pageable(fields[m].host)) {
        threaded[m] = true;
        total += bytes;
      }
  std::vector<Piece> v;
  std::unique_ptr<CopyPool> pool;
  if (total >= kLeast) {
    v.reserve(nfields * ((bytes + kCopyPiece - 1) / kCopyPiece));
    pool = pools.take(total);
  }
  if (!pool) {
    threaded.assign(nfields, false);
  } else {
    CopyPool& P = *pool;
    for (int m = 0; m < nfields; ++m)
      for (size_t o = 0; threaded[m] && o < bytes; o += kCopyPiece)
        v.push_back(Piece{(char*)fields[m].dev + o, (char*)fields[m].host + o, std::min(kCopyPiece, bytes - o)});
    std::atomic<size_t> next{0};
    // work of this context's stream that the copies must follow (outputs), or
    // that still reads the arrays they fill (inputs)
    std::atomic<int> err{(int)cudaStreamSynchronize(s)};
    if (err.load() == 0) {
      const unsigned cores = std::thread::hardware_concurrency();
      const int nw = std::max(1, std::min((int)std::min<size_t>(kCopyWorkers, v.size()), cores ? (int)cores : 1));
      std::vector<std::thread> t;
      try {
        t.reserve(nw);
        for (int w = 1; w < nw; ++w)
          t.emplace_back([&, w] {
            const cudaError_t d = cudaSetDevice(P.device);   // a thread starts on device 0
            if (d != cudaSuccess) err.store((int)d);
            else work(P, w, v, next, to_device, err);
          });
      } catch (const std::exception&) {   // no more threads, or no memory for one: those there are, and this one, do it
      }
      work(P, 0, v, next, to_device, err);
      for (std::thread& x : t) x.join();
    }
    if (err.load() != 0) {
      // a worker stopped with copies in flight: they end before the caller's
      // arrays, the device's and the pieces are used again, and the pool goes.
      // Later calls take the plain copies.
      for (int w = 0; w < kCopyWorkers; ++w) (void)cudaStreamSynchronize(P.stream[w]);
      std::lock_guard<std::mutex> g(pools.lock);
      pools.failed = true;
      return (cudaError_t)err.load();
    }
    pools.give(std::move(pool));
  }
  for (int m = 0; m < nfields; ++m) {
    if (threaded[m]) continue;
    const CopyField& f = fields[m];
    const cudaError_t e = to_device ? cudaMemcpyAsync(f.dev, f.host, bytes, cudaMemcpyHostToDevice, s)
                                    : cudaMemcpyAsync(f.host, f.dev, bytes, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
} catch (const std::exception&) {   // no memory for the piece list, before any copy: nothing passes the C entries
  return cudaErrorMemoryAllocation;
}

}  // namespace amss
