// Device-to-host copies into pageable memory (host_copy.cpp).
#pragma once

#include "errors.h"

namespace hw {

constexpr int kCopyWorkers = 8;
constexpr size_t kCopyChunk = 1 << 20;
constexpr size_t kCopyMin = 2 << 20;  // smaller copies go the plain way

// Page-locked chunks and streams for up to kCopyWorkers threads, kept by the context (8 MiB); the
// threads themselves are made and joined by each copy.
class HostCopier {
  public:
    HostCopier() = default;
    HostCopier(const HostCopier &) = delete;
    HostCopier &operator=(const HostCopier &) = delete;
    ~HostCopier();
    // Device -> host after the work on the stream; returns when dst is complete.  Without chunks or
    // streams to be had the copy goes the plain way.
    int copy(int device, cudaStream_t s, void *dst, const void *src, size_t bytes);

  private:
    int ready(int want);  // how many threads can be served, at most `want`
    void *buf_[kCopyWorkers] = {};
    cudaStream_t stream_[kCopyWorkers] = {};
};

}  // namespace hw
