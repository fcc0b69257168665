// dropin_ctx.cuh -- per-thread device scratch of the drop-in entry points.
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <mutex>
#include <vector>

#include "dev_util.cuh"

namespace amss {

// Pinned pieces and streams of the threaded copies (dropin_copy.cu).
constexpr int kCopyWorkers = 8;
constexpr size_t kCopyPiece = (size_t)1 << 20;
struct CopyPool {
  char* pinned = nullptr;
  cudaStream_t stream[kCopyWorkers] = {};
  cudaEvent_t done[kCopyWorkers][2] = {};
  int device = 0;
  ~CopyPool();
  bool init(int dev);
  char* slot(int w, int s) { return pinned + (size_t)(2 * w + s) * kCopyPiece; }
};
// The process's pools: a call takes one and gives it back, so that threads that
// call one after another share it.  A pool costs 9 to 20 ms to make (16 MB of
// pinned memory) and saves about 40 us a MB, so it is made once kPoolEarned
// bytes have been copied without it; at most kMaxPools, kept to the end of the
// process.
constexpr int kMaxPools = 4;
constexpr size_t kPoolEarned = (size_t)256 << 20;
struct CopyPools {
  std::mutex lock;
  std::vector<std::unique_ptr<CopyPool>> idle;
  int made = 0;
  size_t plain = 0;      // bytes copied for want of a pool since the last was made
  bool failed = false;   // a pool could not be made, or a copy through one failed: no more of them
  std::unique_ptr<CopyPool> take(size_t bytes);   // on the calling thread's device; null: plain copies
  void give(std::unique_ptr<CopyPool> pool);
};
CopyPools& copy_pools();
struct CopyField {
  void* dev;
  void* host;
};
// Copies `bytes` of every field host -> device or back.  In stream order with
// s; the copies that threads made have also completed on return.
cudaError_t copy_fields(CopyPools& pools, const CopyField* fields, int nfields, size_t bytes, bool to_device,
                        cudaStream_t s);

// Per-thread device scratch of the drop-in entries (grow-only, reused).
struct DropinCtx {
  cudaStream_t stream = nullptr;
  double* dbuf = nullptr;
  size_t cap = 0;      // doubles
  unsigned* dstatus = nullptr;
  bool ok = false;
  ~DropinCtx() {
    if (dbuf) cudaFree(dbuf);
    if (dstatus) cudaFree(dstatus);
    if (stream) cudaStreamDestroy(stream);
  }
  int init() {
    if (ok) return 0;
    if (check_device("drop-in") != 0) return -1;
    if (cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) return -1;
    if (cudaMalloc(&dstatus, sizeof(unsigned)) != cudaSuccess) return -1;
    ok = true;
    return 0;
  }
  double* reserve(size_t n) {
    if (n > cap) {
      if (dbuf) cudaFree(dbuf);
      dbuf = nullptr;
      cap = 0;
      if (cudaMalloc(&dbuf, n * sizeof(double)) != cudaSuccess) return nullptr;
      cap = n;
    }
    return dbuf;
  }
};

// The calling thread's context (one stream and one grow-only buffer per thread).
DropinCtx& dropin_ctx();

}  // namespace amss
