#pragma once
// ===================================================================
// Collecting a hash aggregate's groups on the device.
//
// The reference walks its aggregate arrays on the host after the run
// (metal_result_collector.cpp:231-235). Here the table stays in HBM: its
// live slots are compacted and put in key order by kernels
// (kernels/group_collect.cu), and only the dense, sorted columns cross the
// host link, into a pinned block.
// ===================================================================
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

namespace gpudb {

// Host memory a result's columns live in. Blocks are page-locked and
// recycled through a process-wide pool while the bytes handed out stay
// under kPinnedHandedOut (the pool keeps at most kPinnedKept idle); beyond
// that, or when page-locking fails, a block is plain memory. Thread-safe.
struct HostBlock {
    void* ptr = nullptr;
    size_t bytes = 0;
    bool pinned = false;
    ~HostBlock();
};
constexpr size_t kPinnedHandedOut = size_t(1) << 30;
constexpr size_t kPinnedKept = size_t(256) << 20;
std::shared_ptr<HostBlock> hostBlock(size_t bytes);

// A hash table as its aggregation kernel left it.
struct GroupTable {
    static constexpr int kMaxAggs = 16;
    const void* keys = nullptr;   // u64, u32, or (packedStride) slots of u64 words
    int keyBytes = 8;
    int packedStride = 0;         // words per slot; word 0 holds ~key, aggregate a is word 1 + a
    uint64_t cap = 0;             // slots
    std::vector<const void*> aggs;  // u64 each (unused when packed)
    int nAggs = 0;
};

// Scratch of the collection, kept by its owner and grown on demand.
struct GroupWorkspace {
    void* dev = nullptr;
    size_t bytes = 0;
    uint64_t* head = nullptr;  // pinned: count, OR and AND of the keys
    ~GroupWorkspace();
};

// Live groups (a key, and any aggregate other than zero) as int64 columns
// {key, aggregates...}, column c at data[c * rows] inside `host`, in
// ascending key order when `sorted`. Runs on `stream` and waits for it. Returns false with
// `error` empty when device scratch could not be had (the caller collects
// on the host), and with `error` set when the device failed.
bool collectGroups(const GroupTable& t, bool sorted, GroupWorkspace& ws, cudaStream_t stream, uint64_t& rows,
                   const int64_t*& data, std::shared_ptr<HostBlock>& host, std::string& error);

// The same for a table of few slots, enqueued on `stream` without a wait:
// smallGroups() reads the columns once the stream has been waited for. False
// (with `error` empty) when the table is too large or there is no scratch or
// no pinned memory for it.
bool enqueueSmallGroups(const GroupTable& t, bool sorted, GroupWorkspace& ws, cudaStream_t stream,
                        std::shared_ptr<HostBlock>& host, std::string& error);
void smallGroups(const HostBlock& host, uint64_t& rows, const int64_t*& data);

}  // namespace gpudb
