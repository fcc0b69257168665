// dropin_copy.cu -- the drop-in entries' copies between the caller's arrays
// and the device.
//
// The entries take pageable arrays.  cudaMemcpyAsync moves such an array
// through the driver's staging buffer on the calling thread alone, and the
// first write to a fresh output array faults its pages in on that thread too:
// 20 of the 22 ms of a 54^3 right-hand side (43 MB in, 69 MB out).  Several
// worker threads therefore copy pieces through pinned buffers of their own,
// each with two pieces in flight, so that host copies, page faults and DMA
// overlap: 21.4 -> 9.4 ms a call with 16 cores.  The pool belongs to the calling thread's context:
// kCopyWorkers streams and 2 kCopyWorkers pieces of kCopyPiece bytes, freed
// with it.  Small calls, calls that get no pool, and arrays that are not ordinary
// host memory and outputs that share memory take the plain copies.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#include <vector>

#include "dropin_ctx.cuh"

namespace amss {

CopyPool::~CopyPool() { release(); }

void CopyPool::release() {
  for (int w = 0; w < kCopyWorkers; ++w) {
    for (int s = 0; s < 2; ++s)
      if (done[w][s]) cudaEventDestroy(done[w][s]);
    if (stream[w]) cudaStreamDestroy(stream[w]);
    done[w][0] = done[w][1] = nullptr;
    stream[w] = nullptr;
  }
  if (pinned) cudaFreeHost(pinned);
  pinned = nullptr;
  ready = false;
}

bool CopyPool::init() {
  if (failed) return false;
  int now = 0;
  if (cudaGetDevice(&now) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  // the caller has since chosen another device: the runtime's copies serve it
  if (ready) return now == device;
  device = now;
  bool ok = cudaHostAlloc((void**)&pinned, 2 * kCopyWorkers * kCopyPiece, cudaHostAllocDefault) == cudaSuccess;
  for (int w = 0; ok && w < kCopyWorkers; ++w) {
    ok = cudaStreamCreateWithFlags(&stream[w], cudaStreamNonBlocking) == cudaSuccess;
    for (int s = 0; ok && s < 2; ++s) ok = cudaEventCreateWithFlags(&done[w][s], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    (void)cudaGetLastError();
    release();
    failed = true;
    return false;
  }
  ready = true;
  return true;
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

cudaError_t copy_fields(CopyPool& P, const CopyField* fields, int nfields, size_t bytes, bool to_device,
                        cudaStream_t s) try {
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
  // Starting the threads costs more than they save where the arrays' pages are
  // there already: at 26^3 points (4.8 MB in, 7.7 MB out) 2.4 ms a call by
  // plain copies, 2.7 to 3.1 ms by threads; at 28^3 (6.0 and 9.7 MB) 5.0 and 2.3.
  if (total < kLeast || !P.init()) {
    threaded.assign(nfields, false);
  } else {
    // work of this context's stream that the copies must follow (outputs), or
    // that still reads the arrays they fill (inputs)
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    std::vector<Piece> v;
    for (int m = 0; m < nfields; ++m)
      for (size_t o = 0; threaded[m] && o < bytes; o += kCopyPiece)
        v.push_back(Piece{(char*)fields[m].dev + o, (char*)fields[m].host + o, std::min(kCopyPiece, bytes - o)});
    std::atomic<size_t> next{0};
    std::atomic<int> err{0};
    const unsigned cores = std::thread::hardware_concurrency();
    const int nw = std::max(1, std::min((int)std::min<size_t>(kCopyWorkers, v.size()), cores ? (int)cores : 1));
    std::vector<std::thread> t;
    t.reserve(nw);
    try {
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
    if (err.load() != 0) {
      // a worker stopped with copies in flight: they end before the caller's
      // arrays, the device's and the pieces are used again.  Later calls take
      // the plain copies.
      for (int w = 0; w < kCopyWorkers; ++w) (void)cudaStreamSynchronize(P.stream[w]);
      P.release();
      P.failed = true;
      return (cudaError_t)err.load();
    }
  }
  for (int m = 0; m < nfields; ++m) {
    if (threaded[m]) continue;
    const CopyField& f = fields[m];
    const cudaError_t e = to_device ? cudaMemcpyAsync(f.dev, f.host, bytes, cudaMemcpyHostToDevice, s)
                                    : cudaMemcpyAsync(f.host, f.dev, bytes, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
} catch (const std::bad_alloc&) {   // of the piece list, before any copy: nothing passes the C entries
  return cudaErrorMemoryAllocation;
}

}  // namespace amss
