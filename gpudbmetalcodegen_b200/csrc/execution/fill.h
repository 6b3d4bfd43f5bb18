#pragma once
// One launch for all of a run's buffer fills, one for what it reads back
// (kernels/fill.cu).
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace gpudb {

struct BufferFill {
    void* ptr;
    size_t bytes;
    int value;  // of every byte
};

// Enqueue the fills on `stream`: kernel launches of up to kFillSegments
// buffers each, instead of a memset per buffer.
constexpr int kFillSegments = 32;
cudaError_t fillBuffers(const std::vector<BufferFill>& fills, cudaStream_t stream);

struct BufferRead {
    const void* src;  // device memory
    void* dst;        // pinned host memory
    size_t bytes;
};

// Enqueue small reads: the kernel writes the host memory itself, up to
// kReadSegments buffers a launch, instead of a copy per buffer.
constexpr int kReadSegments = 32;
cudaError_t readBuffers(const std::vector<BufferRead>& reads, cudaStream_t stream);

}  // namespace gpudb
