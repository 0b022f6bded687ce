// Device memory of one call: an arena over the memory cache, with staged uploads and grouped zeroing.
#pragma once

#include <algorithm>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "device_cache.cuh"
#include "pdhg_host.cuh"

namespace sih26 {

#define SIH26_CUDA(expr, code)                                                           \
  do {                                                                                   \
    const cudaError_t e_ = (expr);                                                       \
    if (e_ != cudaSuccess)                                                               \
      throw Failure{code, std::string(#expr) + ": " + cudaGetErrorString(e_)};           \
  } while (0)

// Owns every device allocation of one solve and counts the bytes it copies. Buffers are
// carved, 256-byte aligned, out of a few large chunks (one per 64 MiB or per larger buffer) of
// the memory cache, so a solve's ~60 buffers cost no allocation once a call has been made.
//
// Small uploads are staged: between begin_staging and end_staging the arrays of upload_same go
// side by side into one pinned buffer and one device range, sent with one copy (30 separate
// copies of a few KB took longer than a small LP's whole solve). zeros between begin_zeros and
// end_zeros likewise clears with one memset per chunk.
class Arena {
 public:
  long long h2d_bytes = 0;
  long long d2h_bytes = 0;
  ~Arena() {
    // whatever ended the call, nothing may still be using the chunks when they are kept
    const bool idle = cudaStreamSynchronize(stream_) == cudaSuccess;
    for (const auto& c : chunks_) {
      if (idle) MemoryCache::get().give_device(c);
      else cudaFree(c.p);
    }
  }
  template <class T>
  T* alloc(size_t count) {
    if (count == 0) count = 1;
    const size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
    if (bytes > left_) {
      end_range();
      constexpr size_t kChunk = size_t(64) << 20;
      const Chunk c = MemoryCache::get().take_device(device_, std::max(bytes, kChunk));
      if (!c) throw Failure{SANKHYA_GPU_OUT_OF_MEMORY, "cudaMalloc: out of memory"};
      chunks_.push_back(c);
      next_ = static_cast<unsigned char*>(c.p);
      left_ = c.bytes;
      range_ = next_;
    }
    void* p = next_;
    next_ += bytes;
    left_ -= bytes;
    return static_cast<T*>(p);
  }
  void set_device(int device) { device_ = device; }
  // The stream every later use of the arena's buffers is ordered on: zeroing goes there too,
  // so a kernel on that stream never overtakes the memset of a buffer it reads (a
  // non-blocking stream does not wait for the legacy default stream).
  void set_stream(cudaStream_t s) { stream_ = s; }
  cudaStream_t stream() const { return stream_; }
  void begin_zeros() {
    zeroing_ = true;
    range_ = next_;
  }
  void end_zeros() {
    end_range();
    zeroing_ = false;
  }
  template <class T>
  T* zeros(size_t count) {
    T* p = alloc<T>(count);
    if (!zeroing_)
      SIH26_CUDA(cudaMemsetAsync(p, 0, std::max<size_t>(count, 1) * sizeof(T), stream_),
                 SANKHYA_GPU_COPY_FAILED);
    return p;
  }
  void begin_staging(size_t bytes) {
    stage_ = std::make_unique<PinnedBuffer>(bytes);
    stage_size_ = std::min(stage_->size(), bytes);
    stage_at_ = 0;
    stage_base_ = stage_size_ ? alloc<unsigned char>(stage_size_) : nullptr;
  }
  void end_staging() {
    const size_t bytes = stage_at_;
    stage_size_ = 0;  // the buffer itself is in flight: kept until the arena goes
    if (bytes)
      SIH26_CUDA(cudaMemcpyAsync(stage_base_, stage_->data(), bytes, cudaMemcpyHostToDevice, stream_),
                 SANKHYA_GPU_COPY_FAILED);
  }
  template <class T>
  T* upload_raw(const T* host, size_t count) {
    const size_t bytes = count * sizeof(T), padded = (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    if (stage_size_ && stage_at_ + padded <= stage_size_) {
      T* p = reinterpret_cast<T*>(stage_base_ + stage_at_);
      if (bytes) std::memcpy(stage_->data() + stage_at_, host, bytes);
      stage_at_ += padded;
      h2d_bytes += bytes;
      return p;
    }
    T* p = alloc<T>(count);
    if (bytes) {
      SIH26_CUDA(cudaMemcpyAsync(p, host, bytes, cudaMemcpyHostToDevice, stream_), SANKHYA_GPU_COPY_FAILED);
      h2d_bytes += bytes;
    }
    return p;
  }
  template <class T>
  T* upload_same(const std::vector<T>& host) {
    return upload_raw(host.data(), host.size());
  }
  // host -> device copy of a plain buffer, counted
  void put(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    if (bytes == 0) return;
    SIH26_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream), SANKHYA_GPU_COPY_FAILED);
    h2d_bytes += bytes;
  }
  void get(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    if (bytes == 0) return;
    SIH26_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream), SANKHYA_GPU_COPY_FAILED);
    d2h_bytes += bytes;
  }

 private:
  void end_range() {
    if (zeroing_ && next_ != range_)
      SIH26_CUDA(cudaMemsetAsync(range_, 0, next_ - range_, stream_), SANKHYA_GPU_COPY_FAILED);
    range_ = next_;
  }
  std::vector<Chunk> chunks_;
  unsigned char* next_ = nullptr;
  size_t left_ = 0;
  int device_ = 0;
  cudaStream_t stream_ = nullptr;
  bool zeroing_ = false;
  unsigned char* range_ = nullptr;  // start of what begin_zeros still has to clear
  std::unique_ptr<PinnedBuffer> stage_;
  unsigned char* stage_base_ = nullptr;
  size_t stage_size_ = 0, stage_at_ = 0;
};

}  // namespace sih26
