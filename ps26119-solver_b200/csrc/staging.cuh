// staging.cuh — copies between pageable host arrays and the device.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

#include "common.cuh"
#include "parallel.hpp"

namespace b200 {

// Host <-> device copies of pageable host arrays through two page-locked staging blocks: the host
// threads fill (or empty) one block while the copy engine moves the other, so a copy runs at
// the host threads' memcpy rate instead of the single-threaded staging of a pageable
// cudaMemcpyAsync. `jobs` hold device and host addresses and sizes; blocks come from (and go back
// to) the process's pinned-block cache.
struct StagedCopy {
  void* dev;
  void* host;
  std::size_t bytes;
};
constexpr std::size_t kStageBytes = std::size_t{16} << 20;

// The pieces of the concatenated jobs, at most kStageBytes per block: block b takes bytes
// [b·kStageBytes, (b+1)·kStageBytes) of the concatenation.
template <class F>
inline void for_each_piece(const std::vector<StagedCopy>& jobs, std::size_t block, F&& f) {
  const std::size_t lo = block * kStageBytes, hi = lo + kStageBytes;
  std::size_t off = 0;
  for (const StagedCopy& j : jobs) {
    const std::size_t a = std::max(lo, off), e = std::min(hi, off + j.bytes);
    if (a < e) f(j, a - off, a - lo, e - a);  // job, offset in the job, offset in the block, bytes
    off += j.bytes;
  }
}

class StagingBlocks {
 public:
  explicit StagingBlocks(cudaStream_t st) : st_(st) {
    for (int b = 0; b < 2; ++b) {
      buf_[b] = static_cast<char*>(PinnedBlockCache::instance().acquire(kStageBytes));
      B200_CHECK(cudaEventCreateWithFlags(&ev_[b], cudaEventDisableTiming));
    }
  }
  ~StagingBlocks() {
    for (int b = 0; b < 2; ++b) {  // the copies of both blocks have completed before they go back
      cudaEventSynchronize(ev_[b]);
      cudaEventDestroy(ev_[b]);
      PinnedBlockCache::instance().release(buf_[b], kStageBytes);
    }
  }
  void upload(const std::vector<StagedCopy>& jobs) {
    const std::size_t nb = blocks(jobs);
    for (std::size_t k = 0; k < nb; ++k) {
      const int b = static_cast<int>(k & 1);
      B200_CHECK(cudaEventSynchronize(ev_[b]));  // this block's previous copy has left it
      std::vector<CopyJob> fill;
      for_each_piece(jobs, k, [&](const StagedCopy& j, std::size_t jo, std::size_t bo, std::size_t n) {
        fill.push_back({buf_[b] + bo, static_cast<const char*>(j.host) + jo, n});
      });
      parallel_copy(fill.data(), fill.size());
      for_each_piece(jobs, k, [&](const StagedCopy& j, std::size_t jo, std::size_t bo, std::size_t n) {
        B200_CHECK(cudaMemcpyAsync(static_cast<char*>(j.dev) + jo, buf_[b] + bo, n, cudaMemcpyHostToDevice, st_));
      });
      B200_CHECK(cudaEventRecord(ev_[b], st_));
    }
  }
  void download(const std::vector<StagedCopy>& jobs) {
    const std::size_t nb = blocks(jobs);
    auto issue = [&](std::size_t k) {
      const int b = static_cast<int>(k & 1);
      for_each_piece(jobs, k, [&](const StagedCopy& j, std::size_t jo, std::size_t bo, std::size_t n) {
        B200_CHECK(cudaMemcpyAsync(buf_[b] + bo, static_cast<const char*>(j.dev) + jo, n, cudaMemcpyDeviceToHost, st_));
      });
      B200_CHECK(cudaEventRecord(ev_[b], st_));
    };
    if (nb > 0) issue(0);
    for (std::size_t k = 0; k < nb; ++k) {
      const int b = static_cast<int>(k & 1);
      if (k + 1 < nb) issue(k + 1);  // the other block: its previous contents were copied out below
      B200_CHECK(cudaEventSynchronize(ev_[b]));
      std::vector<CopyJob> drain;
      for_each_piece(jobs, k, [&](const StagedCopy& j, std::size_t jo, std::size_t bo, std::size_t n) {
        drain.push_back({static_cast<char*>(j.host) + jo, buf_[b] + bo, n});
      });
      parallel_copy(drain.data(), drain.size());
    }
  }

 private:
  static std::size_t blocks(const std::vector<StagedCopy>& jobs) {
    std::size_t total = 0;
    for (const StagedCopy& j : jobs) total += j.bytes;
    return (total + kStageBytes - 1) / kStageBytes;
  }
  cudaStream_t st_;
  char* buf_[2] = {nullptr, nullptr};
  cudaEvent_t ev_[2] = {nullptr, nullptr};
};

}  // namespace b200
