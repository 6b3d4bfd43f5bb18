// Collecting a hash aggregate's groups on the device: compaction of the
// live slots, key order, dense columns (execution/group_collect.h).
//
// What it replaces: copying the whole table to pageable host memory, one
// host pass over its slots, a host sort and a row object per group. Measured
// on B200, whole calls: a hash join with 2^20 keys 350 ms before, 1.17 ms
// now (0.34 ms of it the join's kernels, 0.46 ms the 25 MB over the link); a
// group-by with 4,099 groups 788 us before, 80 us now.
//
// Tables of at most kSmallCap slots follow the query's own kernels without a
// wait between: compaction, key order (group keys are distinct, so a key's
// position is the number of smaller keys: few keys are compared with all
// others, more are sorted by chunks and then searched for in the other
// chunks) and a pass that writes the columns straight into the mapped host
// block. With a wait between, and one CTA for all comparisons of a key, the
// call with 4,099 groups took 119 us.
// Larger ones count first (the scratch is sized by the groups, not by the
// slots), then compact, sort the key with its slot number by a
// least-significant-digit radix sort and gather the aggregates in order.
// Digits in which no two keys differ are skipped (a 4-million-value key
// domain takes 3 passes, mixed 62-bit keys 8).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "../execution/group_collect.h"

namespace gpudb {

namespace {

// Slots of a small table (at most 2^18 groups at the planned load of 1/2).
// Whole calls on B200, as a small table / as a large one: 112 / 300 us with
// 16,385 groups, 237 / 396 with 131,072, 440 / 458 with 262,144: the searches
// grow with groups x chunks, and the columns cross the link at half the
// speed of a copy.
constexpr uint64_t kSmallCap = 1 << 19;
constexpr int kThreads = 256;
// Slots up to which every key is compared with every other (8192 groups at
// load 1/2); more are sorted by chunks. Whole group-by calls on B200,
// comparing / by chunks of 2048: 72 / 85 us with 100 groups, 81 / 96 with
// 4,099, 97 / 104 with 8,000, 117 / 107 with 12,000, 132 / 111 with 16,384.
// (Chunks of 512: 91 with 4,099, but 370 where 2048 take 233, at 131,072.)
constexpr uint64_t kFewCap = 1 << 14;
constexpr unsigned kRankSplit = 16;  // CTAs that share the ranking of a tile of few keys
constexpr unsigned kChunk = 2048;    // keys per CTA of a sorted chunk
constexpr unsigned kChunkThreads = kChunk / 2;
// Keys per thread of a radix tile: a pass waits for memory and ranks, so more
// and smaller CTAs win. Whole calls on B200 with 16 / 8 / 4: 474 / 429 / 405
// us at 300,000 groups, 886 / 876 / 853 at 1M, 3,078 / 2,968 / 2,967 at 4M.
constexpr int kItems = 4;
constexpr int kTile = kThreads * kItems;  // keys per CTA of a radix pass
constexpr int kWarps = kThreads / 32;

struct TableArgs {
    const void* keys;
    const unsigned long long* aggs[GroupTable::kMaxAggs];
    unsigned long long cap;
    int nAggs, keyBytes, packedStride;
};

// Key of slot s as an order-preserving u64 (signed order, sign bit
// flipped), and whether the slot holds a group.
__device__ __forceinline__ bool slotKey(const TableArgs& t, unsigned long long s, unsigned long long& key) {
    if (t.packedStride) {
        const unsigned long long* w = static_cast<const unsigned long long*>(t.keys) + s * t.packedStride;
        if (*w == 0ull) return false;
        bool any = false;
        for (int a = 0; a < t.nAggs; ++a) any |= w[1 + a] != 0ull;
        key = ~*w ^ 0x8000000000000000ull;
        return any;
    }
    if (t.keyBytes == 4) {
        const unsigned k = static_cast<const unsigned*>(t.keys)[s];
        if (k == 0xFFFFFFFFu) return false;
        key = (unsigned long long)(long long)(int)k ^ 0x8000000000000000ull;
    } else {
        const unsigned long long k = static_cast<const unsigned long long*>(t.keys)[s];
        if (k == ~0ull) return false;
        key = k ^ 0x8000000000000000ull;
    }
    for (int a = 0; a < t.nAggs; ++a)
        if (t.aggs[a][s] != 0ull) return true;  // else inserted but never aggregated (an unmatched build key)
    return false;
}

__device__ __forceinline__ unsigned long long slotAgg(const TableArgs& t, unsigned long long s, int a) {
    return t.packedStride ? static_cast<const unsigned long long*>(t.keys)[s * t.packedStride + 1 + a] : t.aggs[a][s];
}

// head: [0] live groups, [1] OR and [2] AND of their keys.
__global__ void __launch_bounds__(kThreads) kCount(TableArgs t, unsigned long long* head) {
    unsigned n = 0;
    unsigned long long o = 0ull, a = ~0ull;
    for (unsigned long long s = blockIdx.x * (unsigned long long)kThreads + threadIdx.x; s < t.cap;
         s += (unsigned long long)gridDim.x * kThreads) {
        unsigned long long k;
        if (!slotKey(t, s, k)) continue;
        ++n;
        o |= k;
        a &= k;
    }
    for (int d = 16; d > 0; d >>= 1) {
        n += __shfl_xor_sync(0xffffffffu, n, d);
        o |= __shfl_xor_sync(0xffffffffu, o, d);
        a &= __shfl_xor_sync(0xffffffffu, a, d);
    }
    if ((threadIdx.x & 31u) == 0u && n) {
        atomicAdd(head, (unsigned long long)n);
        atomicOr(head + 1, o);
        atomicAnd(head + 2, a);
    }
}

// Live slots to dense (key, slot) pairs, one position atomic per CTA round.
__global__ void __launch_bounds__(kThreads) kCompact(TableArgs t, unsigned long long* n, unsigned long long cap,
                                                     unsigned long long* __restrict__ keys, unsigned* __restrict__ slots) {
    __shared__ unsigned wsum[kWarps];
    __shared__ unsigned long long base;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned long long stride = (unsigned long long)gridDim.x * kThreads;
    for (unsigned long long b = blockIdx.x * (unsigned long long)kThreads; b < t.cap; b += stride) {
        const unsigned long long s = b + threadIdx.x;
        unsigned long long k = 0ull;
        const bool live = s < t.cap && slotKey(t, s, k);
        const unsigned m = __ballot_sync(0xffffffffu, live);
        if (lane == 0u) wsum[warp] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned tot = 0;
            for (int w = 0; w < kWarps; ++w) {
                const unsigned c = wsum[w];
                wsum[w] = tot;
                tot += c;
            }
            base = tot ? atomicAdd(n, (unsigned long long)tot) : 0ull;
        }
        __syncthreads();
        const unsigned long long p = base + wsum[warp] + __popc(m & ((1u << lane) - 1u));
        if (live && p < cap) {
            keys[p] = k;
            slots[p] = (unsigned)s;
        }
        __syncthreads();
    }
}

// Few keys: position = number of smaller keys. The kThreads keys of
// blockIdx.x are compared with every kRankSplit-th tile of kThreads keys,
// read through shared memory; the last of their CTAs to add its part places
// them.
__global__ void __launch_bounds__(kThreads) kRankAll(const unsigned long long* n,
                                                     const unsigned long long* __restrict__ keys,
                                                     const unsigned* __restrict__ slots, unsigned* ranks,
                                                     unsigned* tickets, unsigned long long* __restrict__ keysOut,
                                                     unsigned* __restrict__ slotsOut) {
    __shared__ unsigned long long tile[kThreads];
    __shared__ bool last;
    const unsigned cnt = (unsigned)*n;
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (blockIdx.x * kThreads >= cnt) return;
    const unsigned long long mine = i < cnt ? keys[i] : 0ull;
    unsigned rank = 0;
    for (unsigned b = blockIdx.y * kThreads; b < cnt; b += kRankSplit * kThreads) {
        // past the end the tile holds the largest word, smaller than no key
        tile[threadIdx.x] = b + threadIdx.x < cnt ? keys[b + threadIdx.x] : ~0ull;
        __syncthreads();
#pragma unroll 8
        for (int j = 0; j < kThreads; ++j) rank += tile[j] < mine;
        __syncthreads();
    }
    if (i < cnt && rank) atomicAdd(ranks + i, rank);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(tickets + blockIdx.x, 1u) == kRankSplit - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (i < cnt) {
        const unsigned r = __ldcg(ranks + i);
        keysOut[r] = mine;
        slotsOut[r] = slots[i];
    }
}

// More keys, first of two launches: each CTA sorts kChunk keys with their
// slots (bitonic, in shared memory; the keys are distinct). Past the end
// chunks hold the largest word, after a key equal to it.
__global__ void __launch_bounds__(kChunkThreads) kChunkSort(const unsigned long long* n,
                                                       const unsigned long long* __restrict__ keys,
                                                       const unsigned* __restrict__ slots,
                                                       unsigned long long* __restrict__ chunkKeys,
                                                       unsigned* __restrict__ chunkSlots) {
    __shared__ unsigned long long k[kChunk];
    __shared__ unsigned short x[kChunk];
    const unsigned cnt = (unsigned)*n, b = blockIdx.x * kChunk;
    if (b >= cnt) return;
#pragma unroll
    for (unsigned u = threadIdx.x; u < kChunk; u += kChunkThreads) {
        k[u] = b + u < cnt ? keys[b + u] : ~0ull;
        x[u] = (unsigned short)u;
    }
    for (unsigned size = 2; size <= kChunk; size *= 2)
        for (unsigned d = size / 2; d > 0; d /= 2) {
            __syncthreads();
            const unsigned l = 2 * threadIdx.x - (threadIdx.x & (d - 1)), r = l + d;
            const unsigned long long kl = k[l], kr = k[r];
            const unsigned short xl = x[l], xr = x[r];
            const bool swapped = kl > kr || (kl == kr && xl > xr);
            if (swapped == ((l & size) == 0u)) {
                k[l] = kr;
                k[r] = kl;
                x[l] = xr;
                x[r] = xl;
            }
        }
    __syncthreads();
#pragma unroll
    for (unsigned u = threadIdx.x; u < kChunk; u += kChunkThreads) {
        chunkKeys[b + u] = k[u];
        if (b + u < cnt) chunkSlots[b + u] = slots[b + x[u]];
    }
}

// Second: a key's position is its place in its own chunk plus, for every
// other chunk, the number of smaller keys there (binary searches, four
// chunks' at a time so that their loads overlap).
__global__ void __launch_bounds__(kThreads) kRank(const unsigned long long* n,
                                                  const unsigned long long* __restrict__ chunkKeys,
                                                  const unsigned* __restrict__ chunkSlots,
                                                  unsigned long long* __restrict__ keys, unsigned* __restrict__ slots) {
    const unsigned cnt = (unsigned)*n, i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= cnt) return;
    const unsigned long long mine = chunkKeys[i];
    const unsigned chunks = (cnt + kChunk - 1) / kChunk, own = i / kChunk;
    unsigned rank = i % kChunk;
    for (unsigned c = 0; c < chunks; c += 4) {
        unsigned p[4] = {0u, 0u, 0u, 0u};
        const unsigned long long* a[4];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) a[u] = chunkKeys + (c + u < chunks ? c + u : own) * kChunk;
#pragma unroll
        for (unsigned d = kChunk / 2; d > 0; d /= 2)
#pragma unroll
            for (unsigned u = 0; u < 4; ++u) p[u] += a[u][p[u] + d - 1] < mine ? d : 0u;
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) {
            p[u] += a[u][p[u]] < mine;
            if (c + u < chunks && c + u != own) rank += p[u];
        }
    }
    keys[rank] = mine;
    slots[rank] = chunkSlots[i];
}

// Small tables: the columns in order, written straight into the mapped host
// block: out[0] holds the group count, column c starts at out[1 + c * n].
__global__ void __launch_bounds__(kThreads) kSmallOut(TableArgs t, const unsigned long long* n,
                                                      const unsigned long long* __restrict__ keys,
                                                      const unsigned* __restrict__ slots, long long* out) {
    const unsigned cnt = (unsigned)*n;
    const unsigned r = blockIdx.x * kThreads + threadIdx.x;
    if (r == 0) out[0] = cnt;
    if (r >= cnt) return;
    const unsigned s = slots[r];
    out[1 + r] = (long long)(keys[r] ^ 0x8000000000000000ull);
    for (int a = 0; a < t.nAggs; ++a) out[1 + (unsigned long long)(1 + a) * cnt + r] = (long long)slotAgg(t, s, a);
}

// ---- least-significant-digit radix sort of (key, slot), 8-bit digits -------
// counts[digit * blocks + block]
__global__ void __launch_bounds__(kThreads) kDigitCount(const unsigned long long* __restrict__ keys, unsigned n, int shift,
                                                        unsigned* __restrict__ counts) {
    __shared__ unsigned h[256];
    h[threadIdx.x] = 0u;
    __syncthreads();
    const unsigned b = blockIdx.x * kTile;
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const unsigned i = b + u * kThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(unsigned)(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// One CTA per digit: its blocks' counts become exclusive prefixes, and its
// total goes to totals[digit].
__global__ void __launch_bounds__(kThreads) kDigitScan(unsigned* __restrict__ counts, int blocks,
                                                       unsigned* __restrict__ totals) {
    __shared__ unsigned wsum[kWarps];
    unsigned* c = counts + (unsigned long long)blockIdx.x * blocks;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned carry = 0u;
    for (int b = 0; b < blocks; b += kThreads) {
        const int i = b + (int)threadIdx.x;
        const unsigned v = i < blocks ? c[i] : 0u;
        unsigned x = v;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, d);
            if ((int)lane >= d) x += y;
        }
        if (lane == 31u) wsum[warp] = x;
        __syncthreads();
        unsigned before = carry, all = 0u;
        for (unsigned w = 0; w < kWarps; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (i < blocks) c[i] = before + x - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// The lanes with the same 8-bit digit (of those that are `in`, or of the
// others): nine ballots. A match-any per item instead: 1,185 us for a hash
// join with 2^20 groups that takes 1,157, 857 / 831 for a group-by with 1M.
__device__ __forceinline__ unsigned digitPeers(unsigned d, bool in) {
    const unsigned m = __ballot_sync(0xffffffffu, in);
    unsigned peers = in ? m : ~m;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = d >> b & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, one);
        peers &= one ? v : ~v;
    }
    return peers;
}

// Stable scatter of a tile: each warp owns kItems * 32 consecutive pairs and
// ranks equal digits by match-any, 32 at a time; the warps' counts then
// become offsets from the digit's base.
__global__ void __launch_bounds__(kThreads) kDigitScatter(const unsigned long long* __restrict__ keys,
                                                          const unsigned* __restrict__ slots, unsigned n, int shift,
                                                          const unsigned* __restrict__ counts,
                                                          const unsigned* __restrict__ totals,
                                                          unsigned long long* __restrict__ keysOut,
                                                          unsigned* __restrict__ slotsOut) {
    __shared__ unsigned cnt[kWarps][256];
    __shared__ unsigned wsum[kWarps];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, d0 = threadIdx.x;
    for (int w = 0; w < kWarps; ++w) cnt[w][d0] = 0u;
    // exclusive prefix of the digit totals, digit d0 in thread d0
    const unsigned tot = totals[d0];
    unsigned x = tot;
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, d);
        if ((int)lane >= d) x += y;
    }
    if (lane == 31u) wsum[warp] = x;
    __syncthreads();
    unsigned digitBase = x - tot;
    for (unsigned w = 0; w < warp; ++w) digitBase += wsum[w];
    const unsigned b = blockIdx.x * kTile + warp * (kItems * 32u) + lane;
    unsigned long long k[kItems];
    unsigned pos[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const unsigned i = b + u * 32u;
        k[u] = i < n ? keys[i] : ~0ull;
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const bool in = b + u * 32u < n;
        const unsigned dg = (unsigned)(k[u] >> shift) & 255u;
        const unsigned peers = digitPeers(dg, in);
        const unsigned before = in ? cnt[warp][dg] : 0u;
        __syncwarp();
        if (in && (int)lane == __ffs(peers) - 1) cnt[warp][dg] = before + __popc(peers);
        __syncwarp();
        pos[u] = before + __popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    unsigned at = digitBase + counts[d0 * gridDim.x + blockIdx.x];
    for (int w = 0; w < kWarps; ++w) {
        const unsigned c = cnt[w][d0];
        cnt[w][d0] = at;
        at += c;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const unsigned i = b + u * 32u;
        if (i >= n) continue;
        const unsigned p = cnt[warp][(unsigned)(k[u] >> shift) & 255u] + pos[u];
        keysOut[p] = k[u];
        slotsOut[p] = slots[i];
    }
}

// The dense columns in order: keys back to int64, aggregates gathered.
__global__ void __launch_bounds__(kThreads) kGather(TableArgs t, const unsigned long long* __restrict__ keys,
                                                    const unsigned* __restrict__ slots, unsigned n,
                                                    long long* __restrict__ out) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    out[i] = (long long)(keys[i] ^ 0x8000000000000000ull);
    const unsigned s = slots[i];
    for (int a = 0; a < t.nAggs; ++a) out[(unsigned long long)(1 + a) * n + i] = (long long)slotAgg(t, s, a);
}

std::string cudaWhy(const char* what, cudaError_t e) { return std::string(what) + ": " + cudaGetErrorString(e); }

bool reserve(GroupWorkspace& ws, size_t want) {
    if (want <= ws.bytes) return true;
    if (ws.dev) cudaFree(ws.dev);
    ws.dev = nullptr;
    ws.bytes = 0;
    if (cudaMalloc(&ws.dev, want) != cudaSuccess) {
        cudaGetLastError();
        ws.dev = nullptr;
        return false;
    }
    ws.bytes = want;
    return true;
}

// ---- pinned host blocks -----------------------------------------------------
struct Pool {
    std::mutex mu;
    struct Idle {
        void* ptr;
        size_t bytes;
    };
    std::vector<Idle> idle;
    size_t out = 0, kept = 0;
};
Pool& pool() {
    static Pool* p = new Pool;  // outlives every result, whatever the exit order
    return *p;
}

}  // namespace

std::shared_ptr<HostBlock> hostBlock(size_t bytes) {
    auto b = std::make_shared<HostBlock>();
    bytes = std::max<size_t>(bytes, 4096);
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> g(p.mu);
        if (p.out + bytes <= kPinnedHandedOut) {
            size_t best = p.idle.size();
            for (size_t i = 0; i < p.idle.size(); i++)
                if (p.idle[i].bytes >= bytes && p.idle[i].bytes <= 4 * bytes + (1 << 20) &&
                    (best == p.idle.size() || p.idle[i].bytes < p.idle[best].bytes))
                    best = i;
            if (best < p.idle.size()) {
                b->ptr = p.idle[best].ptr;
                b->bytes = p.idle[best].bytes;
                b->pinned = true;
                p.idle.erase(p.idle.begin() + (long)best);
                p.kept -= b->bytes;
                p.out += b->bytes;
                return b;
            }
            p.out += bytes;  // taken before the allocation, so racing callers see it
            b->pinned = true;
        }
    }
    if (b->pinned) {
        if (cudaHostAlloc(&b->ptr, bytes, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            b->bytes = bytes;
            return b;
        }
        cudaGetLastError();
        b->ptr = nullptr;
        b->pinned = false;
        std::lock_guard<std::mutex> g(p.mu);
        p.out -= bytes;
    }
    b->ptr = ::operator new(bytes);
    b->bytes = bytes;
    return b;
}

HostBlock::~HostBlock() {
    if (!ptr) return;
    if (!pinned) {
        ::operator delete(ptr);
        return;
    }
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> g(p.mu);
        p.out -= bytes;
        if (p.kept + bytes <= kPinnedKept) {
            p.idle.push_back({ptr, bytes});
            p.kept += bytes;
            return;
        }
    }
    cudaFreeHost(ptr);
}

GroupWorkspace::~GroupWorkspace() {
    if (dev) cudaFree(dev);
    if (head) cudaFreeHost(head);
}

namespace {

TableArgs tableArgs(const GroupTable& gt) {
    TableArgs t{};
    t.keys = gt.keys;
    t.cap = gt.cap;
    t.nAggs = gt.nAggs;
    t.keyBytes = gt.keyBytes;
    t.packedStride = gt.packedStride;
    for (int a = 0; a < gt.nAggs && !gt.packedStride; a++) t.aggs[a] = static_cast<const unsigned long long*>(gt.aggs[a]);
    return t;
}

unsigned scanGrid(uint64_t cap) { return (unsigned)std::min<uint64_t>((cap + kThreads - 1) / kThreads, 148 * 8); }

size_t at256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace

bool enqueueSmallGroups(const GroupTable& gt, bool sorted, GroupWorkspace& ws, cudaStream_t stream,
                        std::shared_ptr<HostBlock>& host, std::string& error) {
    error.clear();
    if (gt.nAggs < 1 || gt.nAggs > GroupTable::kMaxAggs || gt.cap == 0 || gt.cap > kSmallCap) return false;
    auto blk = hostBlock((1 + (1 + gt.nAggs) * (size_t)gt.cap) * 8);
    void* mapped = nullptr;
    if (!blk->pinned || cudaHostGetDevicePointer(&mapped, blk->ptr, 0) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const unsigned blocks = (unsigned)((gt.cap + kThreads - 1) / kThreads);
    // few keys: counters and ranks that start at 0, beside the group count;
    // more: whole chunks of keys and slots
    const bool few = gt.cap <= kFewCap;
    const unsigned chunks = (unsigned)((gt.cap + kChunk - 1) / kChunk);
    const size_t oTickets = 256, oRanks = oTickets + at256(4 * blocks), oKeys = few ? oRanks + at256(4 * gt.cap) : 256,
                 oSlots = oKeys + at256(8 * gt.cap), oKeys2 = oSlots + at256(4 * gt.cap),
                 n2 = few ? (size_t)gt.cap : (size_t)kChunk * chunks, oSlots2 = oKeys2 + at256(8 * n2);
    if (!reserve(ws, oSlots2 + at256(4 * n2))) return false;
    char* d = static_cast<char*>(ws.dev);
    auto* n = reinterpret_cast<unsigned long long*>(d);
    auto* keys = reinterpret_cast<unsigned long long*>(d + oKeys);
    auto* slots = reinterpret_cast<unsigned*>(d + oSlots);
    auto* keys2 = reinterpret_cast<unsigned long long*>(d + oKeys2);
    auto* slots2 = reinterpret_cast<unsigned*>(d + oSlots2);
    const TableArgs t = tableArgs(gt);
    cudaError_t e = cudaMemsetAsync(d, 0, few ? oKeys : 256, stream);
    if (e == cudaSuccess) {
        kCompact<<<scanGrid(gt.cap), kThreads, 0, stream>>>(t, n, gt.cap, keys, slots);
        if (sorted && few) {
            kRankAll<<<dim3(blocks, kRankSplit), kThreads, 0, stream>>>(
                n, keys, slots, reinterpret_cast<unsigned*>(d + oRanks), reinterpret_cast<unsigned*>(d + oTickets), keys2, slots2);
            std::swap(keys, keys2);
            std::swap(slots, slots2);
        } else if (sorted) {
            kChunkSort<<<chunks, kChunkThreads, 0, stream>>>(n, keys, slots, keys2, slots2);
            kRank<<<blocks, kThreads, 0, stream>>>(n, keys2, slots2, keys, slots);
        }
        kSmallOut<<<blocks, kThreads, 0, stream>>>(t, n, keys, slots, static_cast<long long*>(mapped));
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        cudaStreamSynchronize(stream);  // nothing may still write the block
        error = cudaWhy("group collection", e);
        return false;
    }
    host = blk;
    return true;
}

void smallGroups(const HostBlock& host, uint64_t& rows, const int64_t*& data) {
    rows = *static_cast<const uint64_t*>(host.ptr);
    data = static_cast<const int64_t*>(host.ptr) + 1;
}

bool collectGroups(const GroupTable& gt, bool sorted, GroupWorkspace& ws, cudaStream_t stream, uint64_t& rows,
                   const int64_t*& data, std::shared_ptr<HostBlock>& host, std::string& error) {
    error.clear();
    rows = 0;
    data = nullptr;
    if (gt.nAggs < 1 || gt.nAggs > GroupTable::kMaxAggs || gt.cap == 0 || gt.cap > (1ull << 31)) return false;
    if (!ws.head && cudaHostAlloc((void**)&ws.head, 4 * sizeof(uint64_t), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        ws.head = nullptr;
        return false;
    }
    const TableArgs t = tableArgs(gt);
    const unsigned scanBlocks = scanGrid(gt.cap);
    const int ncols = 1 + gt.nAggs;
    auto fail = [&](const char* what, cudaError_t e) {
        error = cudaWhy(what, e);
        return false;
    };
    cudaError_t e;
    if (enqueueSmallGroups(gt, sorted, ws, stream, host, error)) {
        if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return fail("group collection", e);
        smallGroups(*host, rows, data);
        return true;
    }
    if (!error.empty()) return false;
    if (!reserve(ws, 256)) return false;
    auto* head = static_cast<unsigned long long*>(ws.dev);
    ws.head[0] = 0;
    ws.head[1] = 0;
    ws.head[2] = ~0ull;
    if ((e = cudaMemcpyAsync(head, ws.head, 24, cudaMemcpyHostToDevice, stream)) != cudaSuccess)
        return fail("group collection", e);
    kCount<<<scanBlocks, kThreads, 0, stream>>>(t, head);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(ws.head, head, 24, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess)
        return fail("group collection", e);
    const uint64_t n = ws.head[0], diff = ws.head[1] & ~ws.head[2];  // bits in which keys differ
    rows = n;
    if (n == 0) {
        host = hostBlock(8);
        data = static_cast<int64_t*>(host->ptr);
        return true;
    }
    const unsigned blocks = (unsigned)((n + kTile - 1) / kTile);
    const size_t oTot = 256, oCnt = oTot + 1024, oK0 = oCnt + at256(4ull * 256 * blocks), oK1 = oK0 + at256(8 * n),
                 oS0 = oK1 + at256(8 * n), oS1 = oS0 + at256(4 * n), oOut = oS1 + at256(4 * n);
    if (!reserve(ws, oOut + 8 * ncols * n)) return false;
    auto blk = hostBlock(8 * ncols * n);
    char* d = static_cast<char*>(ws.dev);
    head = reinterpret_cast<unsigned long long*>(d);  // the scratch may have moved
    auto* totals = reinterpret_cast<unsigned*>(d + oTot);
    auto* counts = reinterpret_cast<unsigned*>(d + oCnt);
    unsigned long long* k[2] = {reinterpret_cast<unsigned long long*>(d + oK0), reinterpret_cast<unsigned long long*>(d + oK1)};
    unsigned* s[2] = {reinterpret_cast<unsigned*>(d + oS0), reinterpret_cast<unsigned*>(d + oS1)};
    auto* out = reinterpret_cast<long long*>(d + oOut);
    if ((e = cudaMemsetAsync(head, 0, 8, stream)) != cudaSuccess) return fail("group collection", e);
    kCompact<<<scanBlocks, kThreads, 0, stream>>>(t, head, n, k[0], s[0]);
    int cur = 0;
    for (int shift = 0; sorted && shift < 64; shift += 8) {
        if (((diff >> shift) & 255u) == 0u) continue;
        kDigitCount<<<blocks, kThreads, 0, stream>>>(k[cur], (unsigned)n, shift, counts);
        kDigitScan<<<256, kThreads, 0, stream>>>(counts, (int)blocks, totals);
        kDigitScatter<<<blocks, kThreads, 0, stream>>>(k[cur], s[cur], (unsigned)n, shift, counts, totals, k[cur ^ 1],
                                                       s[cur ^ 1]);
        cur ^= 1;
    }
    kGather<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, stream>>>(t, k[cur], s[cur], (unsigned)n, out);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(blk->ptr, out, 8 * ncols * n, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess)
        return fail("group collection", e);
    host = blk;
    data = static_cast<int64_t*>(blk->ptr);
    return true;
}

}  // namespace gpudb
