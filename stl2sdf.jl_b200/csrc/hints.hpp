// hints.hpp -- sizes for the scratch buffers of a batch's workers (host only, see scratch() in capi.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <mutex>
#include <string>
#include <unordered_map>

namespace sdfgpu {

// Batch workers take whatever items come up, so each would grow its buffers for as long as new sizes reach it,
// and every cudaFree waits for all of them.  A worker's buffer that has to grow therefore grows to the largest
// size that any worker has asked for, up to kHintMax and while all workers' buffers together are at most
// kSlackMax, a hundredth of the device's memory, beyond their own needs.  32 meshes, 8 workers, six medians of
// 20 calls in turn (B200): 16.3 to 16.7 ms, against 16.8 to 17.6 without; a first call 0.28 to 0.51 s, against
// 0.39 s and more; 0.5 GB more.
struct ScratchHints {
  static constexpr std::size_t kHintMax = (std::size_t)128 << 20, kSlackMax = (std::size_t)2 << 30;
  std::mutex mu;
  std::unordered_map<std::string, std::size_t> bytes;  // the largest request per buffer
  std::size_t slack = 0;                               // granted beyond the requests and not given back

  // The size for a request of `need` bytes that would otherwise be given `want`; what it is above `want` counts
  // as slack until it is given back.
  std::size_t grant(const std::string& name, std::size_t need, std::size_t want) {
    std::lock_guard<std::mutex> lk(mu);
    std::size_t& most = bytes[name];
    most = std::max(most, need);
    const std::size_t hint = std::min(most, kHintMax), size = hint + hint / 8;
    if (size <= want || slack + (size - want) > kSlackMax) return want;
    slack += size - want;
    return size;
  }
  void give_back(std::size_t s) {
    std::lock_guard<std::mutex> lk(mu);
    slack -= s;
  }
};

}  // namespace sdfgpu
