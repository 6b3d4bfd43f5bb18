// A run's buffer fills in one launch, its small reads in another
// (execution/fill.h). A plan fills up to
// a dozen small buffers (counters, ticket words, bitmaps, output lists), and
// a memset costs about 2 us of stream time each, whatever its size: the
// join's nine took 17 us of a 600K-row query whose kernels take 50 (B200);
// this launch takes 3. Large buffers are written 16 bytes per thread and
// store, at memory rate.
#include <algorithm>

#include "../execution/fill.h"

namespace gpudb {

namespace {

constexpr int kThreads = 256;
constexpr unsigned long long kChunk = 32768;  // bytes per block step

struct Segments {
    unsigned char* p[kFillSegments];
    unsigned long long bytes[kFillSegments];
    unsigned long long chunk0[kFillSegments + 1];  // first chunk of each segment
    unsigned value[kFillSegments];                 // the byte, four times
    int n;
};

__global__ void __launch_bounds__(kThreads) kFill(const __grid_constant__ Segments s) {
    int g = 0;
    for (unsigned long long c = blockIdx.x; c < s.chunk0[s.n]; c += gridDim.x) {
        while (c >= s.chunk0[g + 1]) ++g;
        const unsigned long long a = (c - s.chunk0[g]) * kChunk, end = s.bytes[g];
        const unsigned long long b = a + kChunk < end ? a + kChunk : end;
        const unsigned v = s.value[g];
        const unsigned long long body = a + (b - a) / 16 * 16;
        for (unsigned long long i = a + 16ull * threadIdx.x; i < body; i += 16ull * kThreads)
            *reinterpret_cast<uint4*>(s.p[g] + i) = make_uint4(v, v, v, v);
        for (unsigned long long i = body + threadIdx.x; i < b; i += kThreads) s.p[g][i] = (unsigned char)v;
    }
}

struct Reads {
    const unsigned char* src[kReadSegments];
    unsigned char* dst[kReadSegments];
    unsigned long long bytes[kReadSegments];
};

// One block per buffer. A copy of a few bytes is about 3 us of stream time
// and 2 us of the host's; a run reads back its error word, its phases' start
// times and one to five result buffers.
__global__ void __launch_bounds__(kThreads) kRead(const __grid_constant__ Reads r) {
    const unsigned char* src = r.src[blockIdx.x];
    unsigned char* dst = r.dst[blockIdx.x];
    const unsigned long long n = r.bytes[blockIdx.x];
    const unsigned long long body =
        (reinterpret_cast<size_t>(src) | reinterpret_cast<size_t>(dst)) % 8 ? 0ull : n / 8 * 8;
    for (unsigned long long i = 8ull * threadIdx.x; i < body; i += 8ull * kThreads)
        *reinterpret_cast<unsigned long long*>(dst + i) = *reinterpret_cast<const unsigned long long*>(src + i);
    for (unsigned long long i = body + threadIdx.x; i < n; i += kThreads) dst[i] = src[i];
}

}  // namespace

cudaError_t readBuffers(const std::vector<BufferRead>& reads, cudaStream_t stream) {
    for (size_t at = 0; at < reads.size(); at += kReadSegments) {
        Reads r{};
        const unsigned n = (unsigned)std::min<size_t>(kReadSegments, reads.size() - at);
        for (unsigned i = 0; i < n; ++i) {
            r.src[i] = static_cast<const unsigned char*>(reads[at + i].src);
            r.dst[i] = static_cast<unsigned char*>(reads[at + i].dst);
            r.bytes[i] = reads[at + i].bytes;
        }
        kRead<<<n, kThreads, 0, stream>>>(r);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t fillBuffers(const std::vector<BufferFill>& fills, cudaStream_t stream) {
    Segments s{};
    auto flush = [&]() {
        if (s.n == 0) return cudaSuccess;
        const unsigned blocks = (unsigned)std::min<unsigned long long>(s.chunk0[s.n], 148 * 8);
        kFill<<<blocks, kThreads, 0, stream>>>(s);
        s.n = 0;
        return cudaGetLastError();
    };
    for (const auto& f : fills) {
        if (f.bytes == 0) continue;
        if (reinterpret_cast<size_t>(f.ptr) % 16) {  // a caller's own buffer
            const cudaError_t e = cudaMemsetAsync(f.ptr, f.value, f.bytes, stream);
            if (e != cudaSuccess) return e;
            continue;
        }
        s.p[s.n] = static_cast<unsigned char*>(f.ptr);
        s.bytes[s.n] = f.bytes;
        s.value[s.n] = 0x01010101u * (unsigned)(f.value & 0xFF);
        s.chunk0[s.n + 1] = s.chunk0[s.n] + (f.bytes + kChunk - 1) / kChunk;
        if (++s.n == kFillSegments) {
            const cudaError_t e = flush();
            if (e != cudaSuccess) return e;
        }
    }
    return flush();
}

}  // namespace gpudb
