// copystage.h -- copies from the device into pageable host memory, staged
// through pinned pieces.  Host code only.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace moldy {

// One pinned allocation per engine, made on first use: a head for small
// results and two pieces for copies into pageable memory.
constexpr size_t kStageBytes = 256 << 10;
struct CopyStage {
    unsigned char *head = nullptr, *piece = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    // leaves no error pending when it fails: the caller may do without the pieces
    cudaError_t open(size_t head_bytes);
    // first hands on an error that an earlier launch of this thread left pending
    cudaError_t out(void *dst, const void *src, size_t bytes, cudaStream_t s);
    ~CopyStage();
};

}  // namespace moldy
