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
//     to 184 / 58 ms now.  The slots are one huge-page block, touched by all
//     cores and registered once: 1.7 to 2.5 ms to make and 1 to 1.5 to free, where
//     eight pinned allocations took 15 to 24 and 5.
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "internal.h"

namespace ibfs {

bool DepthSink::is_pinned(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

DepthSink::~DepthSink() { release(); }

void DepthSink::release() {
  for (auto& s : slots_)
    if (s.ev) cudaEventDestroy(s.ev);
  slots_.clear();
  if (registered_) cudaHostUnregister(ring_);
  registered_ = false;
  if (map_) munmap(map_, kMapBytes);
  map_ = ring_ = nullptr;
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
    const cudaError_t e = make_ring();
    if (e != cudaSuccess) {
      release();
      return e;
    }
  }
  return cudaSuccess;
}

// The block is a mapping of its own that a forked child does not inherit: a
// page shared with a child would be copied on the next write and leave the
// registration on the old one.
cudaError_t DepthSink::make_ring() {
  constexpr size_t kBytes = kSlots * kSlotBytes;
  void* m = mmap(nullptr, kMapBytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
  map_ = static_cast<uint8_t*>(m);
  ring_ = map_ + (kHuge - reinterpret_cast<uintptr_t>(map_) % kHuge) % kHuge;
  (void)madvise(ring_, kBytes, MADV_HUGEPAGE);
  (void)madvise(ring_, kBytes, MADV_DONTFORK);
#pragma omp parallel for schedule(static)
  for (long long i = 0; i < (long long)(kBytes / kHuge); i++)
    std::memset(ring_ + (size_t)i * kHuge, 0, kHuge);
  cudaError_t e = cudaHostRegister(ring_, kBytes, cudaHostRegisterDefault);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return e;
  }
  registered_ = true;
  slots_.resize(kSlots);
  for (int i = 0; i < kSlots; i++) {
    slots_[i].buf = ring_ + i * kSlotBytes;
    e = cudaEventCreateWithFlags(&slots_[i].ev, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// A run whose depths could as well go by one driver copy takes the ring once
// there is one, and makes one when it sends kRingPays bytes or when the runs
// before it have sent as many without: making and freeing the ring costs
// about 3 ms, what it saves is 0.03 to 0.04 ms per MB to a reused array and 0.15
// per MB to one whose pages are fresh (those of 32 MB and more, which malloc
// maps anew), so a program that opens a graph, takes a few small results and
// leaves does not pay for it.
bool DepthSink::ring_pays(size_t bytes) {
  if (slots_.empty() && unpaid_ < kRingPays) unpaid_ += bytes;
  return !slots_.empty() || unpaid_ >= kRingPays;
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
      std::memcpy(dst_ + it->off + (a - it->at), sl.buf + a, b - a);
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
    const cudaError_t e = cudaMemcpyAsync(sl.buf + fill_, src_ + off, n,
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
