#pragma once
// One launch for all of a run's buffer fills (kernels/fill.cu).
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

}  // namespace gpudb
