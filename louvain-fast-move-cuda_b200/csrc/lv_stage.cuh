// lv_stage.cuh -- copies between pageable host memory and the device through pinned buffers.
//
// A cudaMemcpyAsync from pageable memory is staged by the driver on the calling thread (about
// 4-6 GB/s measured here, and calls of several threads queue up): it was most of an ingest (64 MB
// of text). A Stager copies in pieces of kPiece bytes, each thread through its own two pinned
// buffers, so that the host copy of one piece overlaps the transfer of the one before. Ingest of
// 64 MB: 16.3 -> 3.9 ms together with its buffers taken from the pool; a served burst (350 MB of
// CSR arrays), where the slots' copies overlap GPU work anyway: 62.7 -> 61.9 ms.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <thread>
#include <vector>

namespace lv {

class Stager {
 public:
  explicit Stager(int threads) : lanes_((size_t)std::max(1, std::min(threads, (int)std::thread::hardware_concurrency()))) {}
  Stager(const Stager&) = delete;
  Stager& operator=(const Stager&) = delete;
  ~Stager() { release(); }

  // Gives the buffers back; the copies issued from them must have finished.
  void release() {
    for (Lane& l : lanes_) {
      for (int i = 0; i < 2; ++i) {
        if (l.ev[i]) cudaEventDestroy(l.ev[i]);
        if (l.buf[i]) cudaFreeHost(l.buf[i]);
      }
      l = Lane{};
    }
  }

  // As cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st): on return `src` is free again.
  cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (!staged(src, bytes)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    return spread(bytes, [=](Lane& l, size_t first, size_t step) {
      int k = 0;
      for (size_t at = first; at < bytes; at += step, k ^= 1) {
        const size_t len = std::min(kPiece, bytes - at);
        cudaError_t e = l.wait(k);
        if (e != cudaSuccess) return e;
        std::memcpy(l.buf[k], static_cast<const char*>(src) + at, len);
        e = cudaMemcpyAsync(static_cast<char*>(dst) + at, l.buf[k], len, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = l.mark(k, st);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    });
  }

  // As cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st): `dst` holds the data once `st` is
  // synchronised (staged copies: on return).
  cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (!staged(dst, bytes)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    return spread(bytes, [=](Lane& l, size_t first, size_t step) {
      int k = 0;
      size_t held[2] = {bytes, bytes};  // where the piece in each buffer belongs
      auto drain = [&](int i) {
        if (held[i] >= bytes) return cudaSuccess;
        const cudaError_t e = l.wait(i);
        if (e == cudaSuccess)
          std::memcpy(static_cast<char*>(dst) + held[i], l.buf[i], std::min(kPiece, bytes - held[i]));
        held[i] = bytes;
        return e;
      };
      for (size_t at = first; at < bytes; at += step, k ^= 1) {
        cudaError_t e = drain(k);
        if (e == cudaSuccess) e = l.wait(k);  // (an earlier call's copy from this buffer)
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(l.buf[k], static_cast<const char*>(src) + at, std::min(kPiece, bytes - at),
                              cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = l.mark(k, st);
        if (e != cudaSuccess) return e;
        held[k] = at;
      }
      const cudaError_t e = drain(k);
      return e == cudaSuccess ? drain(k ^ 1) : e;
    });
  }

 private:
  static constexpr size_t kPiece = 1 << 20;
  static constexpr size_t kMin = 256 << 10;  // smaller copies are the driver's

  struct Lane {
    char* buf[2] = {nullptr, nullptr};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    bool busy[2] = {false, false};
    cudaError_t open() {
      for (int i = 0; i < 2; ++i) {
        cudaError_t e = cudaSuccess;
        if (!buf[i]) e = cudaMallocHost(reinterpret_cast<void**>(&buf[i]), kPiece);
        if (e == cudaSuccess && !ev[i]) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
    cudaError_t wait(int i) {
      if (!busy[i]) return cudaSuccess;
      busy[i] = false;
      return cudaEventSynchronize(ev[i]);
    }
    cudaError_t mark(int i, cudaStream_t st) {
      busy[i] = true;
      return cudaEventRecord(ev[i], st);
    }
  };

  // Whether a copy is worth staging: large, and the host side not pinned.
  static bool staged(const void* host, size_t bytes) {
    if (bytes < kMin) return false;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
  }

  // Runs body(lane, first byte, step) on as many lanes as there are pieces for.
  template <class F>
  cudaError_t spread(size_t bytes, F body) {
    const size_t n = std::max<size_t>(1, std::min(lanes_.size(), bytes / (2 * kPiece)));
    for (size_t i = 0; i < n; ++i) {
      const cudaError_t e = lanes_[i].open();
      if (e != cudaSuccess) return e;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    std::vector<cudaError_t> res(n, cudaSuccess);
    std::vector<std::thread> more;
    size_t started = 1;
    try {
      for (; started < n; ++started)
        more.emplace_back([&, i = started] {
          cudaSetDevice(device);
          res[i] = body(lanes_[i], i * kPiece, n * kPiece);
        });
    } catch (...) {  // no thread to be had: this one takes the remaining lanes' pieces
    }
    res[0] = body(lanes_[0], 0, n * kPiece);
    for (size_t i = started; i < n; ++i) res[i] = body(lanes_[i], i * kPiece, n * kPiece);
    for (std::thread& t : more) t.join();
    for (cudaError_t r : res)
      if (r != cudaSuccess) return r;
    return cudaSuccess;
  }

  std::vector<Lane> lanes_;
};

}  // namespace lv
