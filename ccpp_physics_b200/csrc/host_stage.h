// host_stage.h -- pinned staging of small host-memory calls (lw_api.cu,
// sw_api.cu).
//
// A call on host arrays has some thirty fields.  Copied one by one from the
// caller's pageable memory, each is a driver call that stages and waits; here
// they are gathered into one pinned buffer, which travels in pieces while the
// gathering goes on, and the outputs come back in one copy.  32 columns x 64
// layers of rrtmg_lw_run: 361 -> 309 us; 57 x 127 of rrtmg_sw_run: 1,000 -> 933 us.
// The buffer belongs to a calling thread's workspace, is freed with it and never
// exceeds kHostStageMax; larger calls keep the copies per field, whose cost
// their own size hides, while the gathering grows with it.  Staged / per field,
// us: longwave, 64 layers, 300 columns (9.7 MiB) 978 / 1,008, 400 (12.9) 1,204 /
// 1,199, 540 (17) 1,628 / 1,535; 127 layers, 200 (12.8) 1,248 / 1,252, 270 (17)
// 1,644 / 1,517, 400 (26) 2,290 / 2,019; shortwave, 127 layers, 100 (7.2) 1,099 /
// 1,155, 200 (14) 1,574 / 1,524, 480 (34) 3,108 / 2,644: the line lies at 12 MiB.
#pragma once
#include <algorithm>
#include <cstring>
#include <cuda_runtime.h>

constexpr size_t kHostStageMax = (size_t)12 << 20;

struct HostStage {
  char* p = nullptr;
  size_t bytes = 0;

  // room for n bytes; false (nothing pinned) beyond the limit or if the host refuses
  bool ensure(size_t n) {
    if (n > kHostStageMax) return false;
    if (n <= bytes) return true;
    release();
    const size_t want = std::min(kHostStageMax, n + n / 4);
    if (cudaMallocHost((void**)&p, want) != cudaSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
      return false;
    }
    bytes = want;
    return true;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
  }
};

// Gathers fields into a stage laid out like the device buffer dev.  A call that
// ends early waits for the copies it has sent, so that the next one, on whatever
// stream, finds the stage at rest.
struct HostGather {
  static constexpr size_t kPiece = (size_t)256 << 10;
  char *host, *dev;
  cudaStream_t st;
  size_t sent = 0;
  bool waited = false;   // the call has synchronised st

  HostGather(char* h, char* d, cudaStream_t s) : host(h), dev(d), st(s) {}
  HostGather(const HostGather&) = delete;
  HostGather& operator=(const HostGather&) = delete;
  ~HostGather() {
    if (sent && !waited) (void)cudaStreamSynchronize(st);
  }
  cudaError_t put(size_t off, const void* src, size_t n, size_t next) {   // next: where the following field starts
    std::memcpy(host + off, src, n);
    return next - sent >= kPiece ? send(next) : cudaSuccess;
  }
  cudaError_t send(size_t upto) {
    if (upto <= sent) return cudaSuccess;
    const cudaError_t e = cudaMemcpyAsync(dev + sent, host + sent, upto - sent, cudaMemcpyHostToDevice, st);
    sent = upto;
    return e;
  }
};

// the npts-wide part of each of `rows` rows of `pitch` elements of `elem` bytes
inline void copy_rows(void* dst, const void* src, size_t rows, size_t pitch, size_t npts, size_t elem) {
  if (pitch == npts) {
    std::memcpy(dst, src, rows * pitch * elem);
    return;
  }
  for (size_t r = 0; r < rows; ++r)
    std::memcpy(static_cast<char*>(dst) + r * pitch * elem, static_cast<const char*>(src) + r * pitch * elem, npts * elem);
}
