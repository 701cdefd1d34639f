// sink.cpp -- the depth sink: finished batches' depth rows stream from HBM
// to the caller's host buffer while later batches are still traversing.
//
// Replaces the reference's result writer (write_result.cuh:5-36, commented
// out at its call site bfs_gpu_opt.cuh:89), which would have copied every
// depth array to the host after the whole run.  Here a batch's rows are
// handed to the sink as soon as its output pass has finished (a device flag
// in the device-loop schedule, an event in the plain one) and go down on a
// copy stream of their own, so the PCIe transfer of early batches overlaps
// the traversal of later ones:
//   * pinned destination (cudaMallocHost / cudaHostRegister memory): one
//     cudaMemcpyAsync per row straight into the caller's buffer;
//   * pageable destination: a ring of eight 4 MiB pinned staging slots that
//     rows are packed into -- later slots copy in while the host spreads the
//     oldest into the caller's buffer with all cores, which also take the page
//     faults of a fresh buffer in parallel.  512 rows of 4,194,304 depths
//     (2.1 GB) from R-MAT scale 22 to a fresh / a reused pageable array: 429 /
//     253 ms with four 32 MiB slots spread row by row once all were full, 158
//     to 184 / 58 ms now.
#include <algorithm>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "internal.h"

namespace ibfs {

static bool is_pinned(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

DepthSink::~DepthSink() { release(); }

void DepthSink::release() {
  for (auto& s : slots_) {
    if (s.buf) cudaFreeHost(s.buf);
    if (s.ev) cudaEventDestroy(s.ev);
  }
  slots_.clear();
  if (stream_) cudaStreamDestroy(stream_);
  stream_ = nullptr;
  device_ = -1;
}

cudaError_t DepthSink::begin(int device, void* dst_host, const uint8_t* src_dev) {
  dst_ = static_cast<uint8_t*>(dst_host);
  src_ = src_dev;
  next_ = 0;
  open_ = -1;
  fill_ = 0;
  pending_.clear();
  for (auto& sl : slots_) sl.pieces.clear();
  copied_ = 0;
  if (stream_ && device_ != device) release();
  device_ = device;
  if (!stream_) {
    const cudaError_t e = cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
  }
  pinned_ = is_pinned(dst_host);
  if (!pinned_ && slots_.empty()) {
    slots_.resize(kSlots);
    for (auto& sl : slots_) {
      cudaError_t e = cudaMallocHost(&sl.buf, kSlotBytes);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.ev, cudaEventDisableTiming);
      if (e != cudaSuccess) {
        release();
        return e;
      }
    }
  }
  return cudaSuccess;
}

cudaError_t DepthSink::wait_for(cudaEvent_t ev) {
  if (!ev) return cudaSuccess;
  return cudaStreamWaitEvent(stream_, ev, 0);
}

// Spread the oldest closed staging slot into the caller's buffer once its
// copies have landed.
cudaError_t DepthSink::drain_one() {
  Slot& sl = slots_[pending_.front()];
  const cudaError_t e = cudaEventSynchronize(sl.ev);
  if (e != cudaSuccess) return e;
  // the slot is cut into equal pieces whatever the rows' size: few long rows
  // and many short ones both keep every core busy
  constexpr size_t kPiece = 128u << 10;
  const size_t total = sl.pieces.empty() ? 0 : sl.pieces.back().at + sl.pieces.back().bytes;
  const long long cuts = (long long)((total + kPiece - 1) / kPiece);
#pragma omp parallel for schedule(static) if (cuts > 2)
  for (long long i = 0; i < cuts; i++) {
    const size_t lo = (size_t)i * kPiece, hi = std::min(total, lo + kPiece);
    // the first row that reaches past lo (rows are packed in order)
    auto it = std::upper_bound(sl.pieces.begin(), sl.pieces.end(), lo,
                               [](size_t x, const Piece& pc) { return x < pc.at + pc.bytes; });
    for (; it != sl.pieces.end() && it->at < hi; ++it) {
      const size_t a = std::max(lo, it->at), b = std::min(hi, it->at + it->bytes);
      std::memcpy(dst_ + it->off + (a - it->at), static_cast<const uint8_t*>(sl.buf) + a, b - a);
    }
  }
  sl.pieces.clear();
  pending_.erase(pending_.begin());
  return cudaSuccess;
}

// Close the open slot: its copies are queued, an event marks their end.
cudaError_t DepthSink::close_open() {
  if (open_ < 0) return cudaSuccess;
  const cudaError_t e = cudaEventRecord(slots_[open_].ev, stream_);
  if (e != cudaSuccess) return e;
  pending_.push_back(open_);
  open_ = -1;
  return cudaSuccess;
}

cudaError_t DepthSink::push(size_t off, size_t bytes) {
  copied_ += bytes;
  if (pinned_)
    return cudaMemcpyAsync(dst_ + off, src_ + off, bytes, cudaMemcpyDeviceToHost, stream_);
  // pack pieces into staging slots; a full slot is closed and the next one
  // opened (after spreading the oldest when all are in flight)
  while (bytes > 0) {
    if (open_ >= 0 && fill_ == kSlotBytes) {
      const cudaError_t e = close_open();
      if (e != cudaSuccess) return e;
      // spread what has landed while the next copies run
      while (!pending_.empty()) {
        const cudaError_t q = cudaEventQuery(slots_[pending_.front()].ev);
        if (q == cudaErrorNotReady) break;
        const cudaError_t d = q == cudaSuccess ? drain_one() : q;
        if (d != cudaSuccess) return d;
      }
    }
    if (open_ < 0) {
      if ((int)pending_.size() == kSlots) {
        const cudaError_t e = drain_one();
        if (e != cudaSuccess) return e;
      }
      open_ = next_;
      next_ = (next_ + 1) % kSlots;
      fill_ = 0;
    }
    const size_t n = std::min(bytes, kSlotBytes - fill_);
    Slot& sl = slots_[open_];
    const cudaError_t e = cudaMemcpyAsync(static_cast<uint8_t*>(sl.buf) + fill_, src_ + off, n,
                                          cudaMemcpyDeviceToHost, stream_);
    if (e != cudaSuccess) return e;
    sl.pieces.push_back({off, fill_, n});
    fill_ += n;
    off += n;
    bytes -= n;
  }
  return cudaSuccess;
}

cudaError_t DepthSink::finish() {
  cudaError_t e = pinned_ ? cudaSuccess : close_open();
  while (e == cudaSuccess && !pending_.empty()) e = drain_one();
  const cudaError_t e2 = stream_ ? cudaStreamSynchronize(stream_) : cudaSuccess;
  return e != cudaSuccess ? e : e2;
}

}  // namespace ibfs
