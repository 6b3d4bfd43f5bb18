// Batched mixed-query execution (include/gpudb_batch.h).
//
// Every query of a batch owns a slice of one zero-initialised device arena
// (outputs, hash table, bitmap, error word). Each pipeline shape runs as ONE
// persistent kernel: CTAs take work items — (query, tile of rows) — from a
// global counter, in the order of a per-shape prefix sum of tiles, so uneven
// table sizes balance across the GPU and a whole batch costs one memset and
// a handful of launches (build, agg, group, top-k, top-k merge), replayable
// as a CUDA graph.
//
// Group tables are arrays of 16-byte slots {key + card (u32), count (u32),
// sum (u64)}: two slots per L2 sector, and the all-zero pattern is the empty
// slot, so a single memset initialises the whole arena. A table with at
// least 2 card - 1 slots is DENSE: slot i belongs to key i + 1 - card, a row
// costs two reductions and no probe, and the table cannot overflow; a
// smaller one is an open-addressing hash table (`int32 % card` lies in
// (-card, card), so key + card is never 0). Each CTA may first aggregate
// into a shared-memory table (kTableWords; bounded probing; a row
// whose key finds no room goes to the global table directly), which it
// flushes when it moves to another query: few-group queries then cost a
// handful of global atomics per CTA, and hot keys of skewed ones stay on
// chip. Nothing lists the created groups: the passes after the group-by walk
// the slots, since a list costs one atomic on one address per group.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../../include/gpudb_batch.h"
#include "gpudb_device.cuh"

namespace gpudb {
void setThreadError(const std::string& message);
}

namespace {

constexpr int kTopK = 16;             // largest k a top-k query may ask for
// Table slots per work item of the passes after the group-by: 32 items of a
// table, as far as an item keeps 1024 to 16384 slots.
constexpr long long kScanMin = 1024, kScanMax = 16384;
constexpr int kUnroll = 4;            // independent rows in flight per thread
constexpr int kSmemProbe = 4;         // probes into the shared table before spilling to global

struct __align__(16) Slot {
    unsigned key;    // key + card, 0 = empty
    unsigned count;  // rows of the group (slices are < 2^32 rows)
    unsigned long long sum;
};

__host__ __device__ __forceinline__ unsigned encKey(long long key, long long card) {
    return (unsigned)(key + card);
}
__host__ __device__ __forceinline__ long long decKey(unsigned enc, long long card) { return (long long)enc - card; }

struct QDesc {
    int tmpl, thr, k, attr_lt;
    long long card, rows;
    unsigned cardMagic;  // key % card by multiply-high for keys >= 0
    int cardSh1, cardSh2;
    const int* key;
    const int* filter;
    const long long* value;
    const int* fk;
    const int* dim_key;
    const int* dim_attr;
    long long dim_rows, bitmap_words;
    unsigned long long* agg;  // [count, sum word 0, sum word 1]
    unsigned long long* topk_n;
    unsigned long long* nslots;
    unsigned* err;
    unsigned* bitmap;
    Slot* ht;
    int log2cap, maxProbe;
    long long scanChunk;
    int aggMode;  // GPUDB_AGG_SHARED / _GLOBAL_WARP / _GLOBAL / _SHARED_DIRECT
    int dense;    // slot i belongs to encoded key i + 1
    unsigned directBase;  // SHARED_DIRECT: the encoded key of shared slot 0
    long long* tk_part;  // [tk_chunks][kTopK] of (value, key)
    long long tk_chunks;
    long long* topk_out;  // [kTopK] of (key, value)
    // exact statistics
    unsigned long long* st_pass;
    unsigned long long* st_distinct;
    unsigned* st_bitmap;
    long long st_words;
};

// Group key = key % card. Non-negative keys use division by the invariant
// card via a multiply-high (Granlund & Montgomery, "Division by invariant
// integers using multiplication", PLDI 1994, Fig. 4.1): with
// l = ceil(log2 d) and m = floor(2^32 (2^l - d) / d) + 1,
// n / d = (t + ((n - t) >> min(l, 1))) >> max(l - 1, 0), t = mulhi(m, n).
void cardDivisor(long long card, unsigned* magic, int* sh1, int* sh2) {
    const unsigned long long d = (unsigned long long)card;
    int l = 0;
    while ((1ull << l) < d) l++;
    *magic = (unsigned)(((1ull << 32) * ((1ull << l) - d)) / d + 1ull);
    *sh1 = l < 1 ? l : 1;
    *sh2 = l - 1 > 0 ? l - 1 : 0;
}

__device__ __forceinline__ long long keyMod(int k, const QDesc& q) {
    if (k >= 0) {
        const unsigned n = (unsigned)k;
        const unsigned t = __umulhi(n, q.cardMagic);
        const unsigned quo = (t + ((n - t) >> q.cardSh1)) >> q.cardSh2;
        return (long long)(n - quo * (unsigned)q.card);
    }
    return (long long)k % q.card;
}

// A work list: queries (indices into the descriptor array) and the prefix
// sum of their work items.
struct WorkList {
    const int* q;
    const long long* prefix;  // nq + 1 entries
    int nq;
};

__device__ __forceinline__ int findQuery(const WorkList& wl, long long w) {
    int lo = 0, hi = wl.nq - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(wl.prefix + mid) <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Filter words of rows b, b + step, ... (kUnroll of them); rows at or past
// r1 read as `thr`, which no row passes.
template <int N>
__device__ __forceinline__ void loadFilters(const int* __restrict__ filter, long long b, long long step, long long r1,
                                            int thr, int (&f)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u) f[u] = b + u * step < r1 ? __ldcs(filter + b + u * step) : thr;
}

// Words of rows b, b + step, ... (kUnroll of them) whatever the filter
// says; rows at or past r1 read as 0.
template <typename T, int N>
__device__ __forceinline__ void loadAhead(const T* __restrict__ col, long long b, long long step, long long r1,
                                          T (&x)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u) x[u] = b + u * step < r1 ? __ldcs(col + b + u * step) : (T)0;
}

// A warp whose first kUnroll x 32 rows of a work item pass the filter at
// least one time in four reads its dependent columns unconditionally, one
// iteration ahead with the filter words: at that selectivity nearly every
// 32-byte sector of those columns is needed anyway (each holds 4-8 rows),
// and the loads no longer wait for the filter. Sparser warps keep
// filter-guarded loads. Called by whole warps.
template <int N>
__device__ __forceinline__ bool denseWarp(const int (&f)[N], int thr) {
    int pass = 0;
#pragma unroll
    for (int u = 0; u < N; ++u) pass += __popc(__ballot_sync(0xffffffffu, f[u] < thr));
    return 4 * pass >= 32 * N;
}

// CTA-wide work pull; returns -1 when the list is exhausted.
__device__ __forceinline__ long long pullWork(unsigned long long* counter, long long total, long long* s_item) {
    __syncthreads();
    if (threadIdx.x == 0) *s_item = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    const long long w = *s_item;
    return w < total ? w : -1;
}

__device__ __forceinline__ void blockAdd2(long long c, long long s, unsigned long long* out, long long* red) {
    c = gpudb_warp_sum_i64(c);
    s = gpudb_warp_sum_i64(s);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) {
        red[2 * warp] = c;
        red[2 * warp + 1] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long tc = 0, ts = 0;
        for (int w = 0; w < nw; ++w) {
            tc += red[2 * w];
            ts += red[2 * w + 1];
        }
        if (tc) atomicAdd(out, (unsigned long long)tc);
        if (ts) gpudb_acc128_add(out + 1, ts);
    }
}

// Linear probing from slot `s`, whose key word `cur` is already loaded.
__device__ __forceinline__ long long slotFrom(Slot* ht, int log2cap, unsigned enc, unsigned long long s, unsigned cur,
                                              unsigned maxProbe, unsigned* err) {
    const unsigned long long mask = (1ull << log2cap) - 1ull;
    for (unsigned p = 0; p < maxProbe; ++p) {
        if (p) cur = *((volatile unsigned*)&ht[s].key);
        if (cur == enc) return (long long)s;
        if (cur == 0u) {
            const unsigned prev = atomicCAS(&ht[s].key, 0u, enc);
            if (prev == 0u || prev == enc) return (long long)s;
        }
        s = (s + 1ull) & mask;
    }
    gpudb_set_error(err, GPUDB_ERR_HASH_OVERFLOW);
    return -1;
}

__device__ __forceinline__ void slotAdd(Slot* s, unsigned c, unsigned long long v) {
    gpudb_red_add_u32(&s->count, c);
    gpudb_red_add_u64(&s->sum, v);
}

// Add (count, sum) to a group of the query's table.
template <bool DENSE>
__device__ __forceinline__ void globalAdd(const QDesc& q, Slot* ht, int log2cap, unsigned enc, unsigned c,
                                          unsigned long long v) {
    if (DENSE) {
        slotAdd(ht + (enc - 1u), c, v);
        return;
    }
    const unsigned long long s0 = gpudb_hash_slot((unsigned long long)enc, log2cap);
    const long long s = slotFrom(ht, log2cap, enc, s0, *((volatile unsigned*)&ht[s0].key), (unsigned)q.maxProbe, q.err);
    if (s >= 0) slotAdd(ht + s, c, v);
}

// A table slot's group, if it holds one.
__device__ __forceinline__ bool slotLive(const QDesc& q, const Slot& s) { return q.dense ? s.count != 0u : s.key != 0u; }
__device__ __forceinline__ long long slotKey(const QDesc& q, const Slot& s, long long i) {
    return decKey(q.dense ? (unsigned)i + 1u : s.key, q.card);
}

// ---- JOIN build: bitmap of dim keys with attr < attr_lt -------------------
__global__ void __launch_bounds__(1024) kJoinBuild(const QDesc* __restrict__ qs, WorkList wl, long long tile, unsigned long long* counter) {
    __shared__ long long s_item;
    const long long total = __ldg(wl.prefix + wl.nq);
    for (long long w; (w = pullWork(counter, total, &s_item)) >= 0;) {
        const int qi = findQuery(wl, w);
        const QDesc& q = qs[__ldg(wl.q + qi)];
        const int* __restrict__ dk = q.dim_key;
        const int* __restrict__ da = q.dim_attr;
        unsigned* bm = q.bitmap;
        const long long words = q.bitmap_words;
        const int attrLt = q.attr_lt;
        const long long r0 = (w - __ldg(wl.prefix + qi)) * tile, r1 = min(q.dim_rows, r0 + tile);
        for (long long i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            if (__ldcs(da + i) >= attrLt) continue;
            const long long k = __ldcs(dk + i);
            if (k < 0 || (k >> 5) >= words) {
                gpudb_set_error(q.err, GPUDB_ERR_BOUNDS);
                continue;
            }
            // lanes that set bits of one word (dimension keys tend to be
            // dense and in order) set them with one atomic
            const unsigned am = __activemask();
            const unsigned w = (unsigned)(k >> 5);
            const unsigned peers = __match_any_sync(am, w);
            const unsigned bits = __reduce_or_sync(peers, 1u << (unsigned)(k & 31));
            if ((int)(threadIdx.x & 31u) == __ffs(peers) - 1) atomicOr(bm + w, bits);
        }
    }
}

// ---- AGG / JOIN probe: filter [-> semi-join] -> count + sum ---------------
template <int U>
__global__ void __launch_bounds__(U == 4 ? 1024 : 512, U == 4 ? 1 : 4) kAgg(const QDesc* __restrict__ qs, WorkList wl, long long tile, unsigned long long* counter) {
    __shared__ long long s_item;
    __shared__ long long red[64];
    const long long total = __ldg(wl.prefix + wl.nq);
    for (long long w; (w = pullWork(counter, total, &s_item)) >= 0;) {
        const int qi = findQuery(wl, w);
        const QDesc& q = qs[__ldg(wl.q + qi)];
        const int* __restrict__ filter = q.filter;
        const long long* __restrict__ value = q.value;
        const int thr = q.thr;
        const long long r0 = (w - __ldg(wl.prefix + qi)) * tile, r1 = min(q.rows, r0 + tile);
        const long long step = (long long)blockDim.x;
        long long c = 0, s = 0;
        // the filter words of a thread's next U rows are loaded while
        // the current rows' dependent loads are in flight
        int fn[U];
        loadFilters(filter, r0 + threadIdx.x, step, r1, thr, fn);
        const bool dense = denseWarp(fn, thr);
        if (q.tmpl == GPUDB_TPL_JOIN && dense) {
            // most rows pass: fk and value ride along with the filter words
            const int* __restrict__ fk = q.fk;
            const unsigned* __restrict__ bm = q.bitmap;
            const long long words = q.bitmap_words;
            int kn[U];
            long long vn[U];
            loadAhead(fk, r0 + threadIdx.x, step, r1, kn);
            loadAhead(value, r0 + threadIdx.x, step, r1, vn);
            for (long long b = r0 + threadIdx.x; b < r1; b += U * step) {
                int f[U], key[U];
                long long v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    f[u] = fn[u];
                    key[u] = kn[u];
                    v[u] = vn[u];
                }
                loadFilters(filter, b + U * step, step, r1, thr, fn);
                loadAhead(fk, b + U * step, step, r1, kn);
                loadAhead(value, b + U * step, step, r1, vn);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const long long k = key[u];
                    if (f[u] < thr && k >= 0 && (k >> 5) < words && gpudb_bitmap_test(bm, k)) {
                        ++c;
                        s += v[u];
                    }
                }
            }
        } else if (q.tmpl == GPUDB_TPL_JOIN) {
            const int* __restrict__ fk = q.fk;
            const unsigned* __restrict__ bm = q.bitmap;
            const long long words = q.bitmap_words;
            for (long long b = r0 + threadIdx.x; b < r1; b += U * step) {
                int f[U];
#pragma unroll
                for (int u = 0; u < U; ++u) f[u] = fn[u];
                loadFilters(filter, b + U * step, step, r1, thr, fn);
                int key[U];
#pragma unroll
                for (int u = 0; u < U; ++u) key[u] = f[u] < thr ? __ldcs(fk + b + u * step) : -1;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const long long k = key[u];
                    if (k >= 0 && (k >> 5) < words && gpudb_bitmap_test(bm, k)) {
                        ++c;
                        s += __ldcs(value + b + u * step);
                    }
                }
            }
        } else if (dense) {
            long long vn[U];
            loadAhead(value, r0 + threadIdx.x, step, r1, vn);
            for (long long b = r0 + threadIdx.x; b < r1; b += U * step) {
                int f[U];
                long long v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    f[u] = fn[u];
                    v[u] = vn[u];
                }
                loadFilters(filter, b + U * step, step, r1, thr, fn);
                loadAhead(value, b + U * step, step, r1, vn);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (f[u] < thr) {
                        ++c;
                        s += v[u];
                    }
            }
        } else {
            for (long long b = r0 + threadIdx.x; b < r1; b += U * step) {
                int f[U];
#pragma unroll
                for (int u = 0; u < U; ++u) f[u] = fn[u];
                loadFilters(filter, b + U * step, step, r1, thr, fn);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (f[u] < thr) {
                        ++c;
                        s += __ldcs(value + b + u * step);
                    }
            }
        }
        blockAdd2(c, s, q.agg, red);
    }
}

// ---- GROUPBY / TOPK: filter -> key % card -> table (count, sum) -------------
// Per query, the strategy the host picked from the expected group count and
// the sample's key repetition:
//   SHARED_DIRECT the CTA's shared table indexed by the key itself;
//   SHARED      the CTA's hashed shared table;
//   GLOBAL_WARP warp aggregation, then the global table;
//   GLOBAL      the global table directly.
// A CTA keeps its shared table across a query's work items and flushes it
// into the query's global table when it moves to another query or runs out
// of work. Its sums are (low, high) words, added natively (a 64-bit
// shared-memory add is a compare-and-swap loop; gpudb_shared_add64): equal
// keys of a warp meet there more cheaply than in a warp aggregation.
//
// A row for the global hash table costs L2 round trips (find the slot, then
// the reductions). Lanes that need one wait in a queue of their warp until
// kColdBatch rows have gathered, so the round trips are paid once per 64
// rows instead of by every warp iteration with a single such lane in it
// (before: 9 of 32 lanes active per instruction, long-scoreboard stalls first).
//
// Shared memory per CTA follows its threads (kTableWords each): one CTA of
// 1,024 threads per SM or two of 512 then hold tables of 10 hashed or 13
// direct slots per thread.
//
// Measured (B200, group stage alone, before -> now; floor: 16 B per row at
// 6.65 TB/s): 27.1M rows, 71 % pass, 2,838 uniform keys 650 -> 116 us (65);
// 58.9M rows, 8,763 uniform keys 724 -> 221 (142); 47.9M rows, 57 % pass,
// Zipf(1.3) keys into 0.6M groups 992 -> 348 (115); 22.8M rows, Zipf over
// 10,908 keys 302 -> 109 (55); the mixed batch's 34 grouped queries 5.79 ->
// 2.80 ms. Queries of few keys run at 1.6 x their floor (their loads in
// flight), uniform ones of many keys at the L2's rate of reductions (two per
// row, 75 G rows/s).
constexpr int kTableWords = 40;  // of the shared table, per thread
constexpr int kColdBatch = 64;   // rows of the global hash path a warp takes at a time
constexpr int kColdCap = kColdBatch + 32;

__host__ __device__ constexpr int directSlots(int block) { return kTableWords * block / 3; }
__host__ __device__ constexpr int hashedSlots(int block) { return kTableWords * block / 4; }
constexpr size_t groupSmem(int block) { return (size_t)block * 4 * kTableWords + (size_t)(block / 32) * kColdCap * 12; }

// The CTA's shared table: count and sum words of each slot, then (hashed)
// its key word.
struct SharedTable {
    unsigned* w;
    int slots;
    __device__ __forceinline__ unsigned* cnt(int i) const { return w + i; }
    __device__ __forceinline__ unsigned* lo(int i) const { return w + slots + i; }
    __device__ __forceinline__ unsigned* hi(int i) const { return w + 2 * slots + i; }
    __device__ __forceinline__ unsigned* key(int i) const { return w + 3 * slots + i; }
    __device__ __forceinline__ void add(int i, unsigned long long v) const {
        gpudb_red_add_shared_u32(cnt(i), 1u);
        gpudb_shared_add64(lo(i), hi(i), v);
    }
};

// Encoded group key (key % card) + card of a 32-bit key, from the query's
// divisor held in registers.
struct KeyCode {
    unsigned card, magic;
    int sh1, sh2;
    __device__ __forceinline__ unsigned operator()(int k) const {
        if (k >= 0) {
            const unsigned n = (unsigned)k;
            const unsigned t = __umulhi(n, magic);
            return n - ((t + ((n - t) >> sh1)) >> sh2) * card + card;
        }
        return (unsigned)(k % (int)card) + card;
    }
};

// A warp's rows on their way to the global hash table.
struct ColdQueue {
    unsigned long long* v;
    unsigned* k;
    int n;  // the same in every lane
    // whole warps: the lanes with `cold` append their row
    template <typename Take>
    __device__ __forceinline__ void push(bool cold, unsigned enc, unsigned long long val, Take take) {
        const unsigned m = __ballot_sync(0xffffffffu, cold);
        if (!m) return;
        const unsigned lane = threadIdx.x & 31u;
        if (cold) {
            const int p = n + __popc(m & ((1u << lane) - 1u));
            k[p] = enc;
            v[p] = val;
        }
        n += __popc(m);
        __syncwarp();
        if (n >= kColdBatch) {
            n -= kColdBatch;
            take(n, kColdBatch);
            __syncwarp();
        }
    }
};

enum class GroupPath { Direct, Shared, Global };

template <int U, GroupPath PATH, bool DENSE>
__device__ __forceinline__ void groupTile(const QDesc& q, const SharedTable& st, unsigned directBase, ColdQueue& cq,
                                          long long r0, long long r1) {
    const int* __restrict__ filter = q.filter + r0;
    const int* __restrict__ keyc = q.key + r0;
    const long long* __restrict__ value = q.value + r0;
    const int thr = q.thr;
    const KeyCode code{(unsigned)q.card, q.cardMagic, q.cardSh1, q.cardSh2};
    Slot* ht = q.ht;
    const int log2cap = q.log2cap;
    const unsigned maxProbe = (unsigned)q.maxProbe;
    unsigned* err = q.err;
    const bool warp = PATH == GroupPath::Global && q.aggMode == GPUDB_AGG_GLOBAL_WARP;
    const int step = (int)blockDim.x, n = (int)(r1 - r0), lane = (int)(threadIdx.x & 31u);
    // rows queued for the global table (two per lane in flight)
    auto take = [&](int at, int count) {
        unsigned enc[2], cur[2];
        unsigned long long v[2], s0[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const bool in = lane + 32 * j < count;
            enc[j] = in ? cq.k[at + lane + 32 * j] : 0u;
            v[j] = in ? cq.v[at + lane + 32 * j] : 0ull;
            s0[j] = gpudb_hash_slot((unsigned long long)enc[j], log2cap);
            cur[j] = in ? *((volatile unsigned*)&ht[s0[j]].key) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (lane + 32 * j >= count) continue;
            long long s = (long long)s0[j];
            if (cur[j] != enc[j]) s = slotFrom(ht, log2cap, enc[j], s0[j], cur[j], maxProbe, err);
            if (s >= 0) slotAdd(ht + s, 1u, v[j]);
        }
    };
    const int first = (int)threadIdx.x - lane;  // the warp's first row of each round
    // Software pipeline: while a round's rows are processed, the next round's
    // keys and values (of its rows that pass: its filter words are here) and
    // the filter words of the round after it are on their way.
    auto loadFilter = [&](int b, int (&f)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = b + u * step;
            f[u] = i < n ? __ldcs(filter + i) : thr;  // no row passes at thr
        }
    };
    auto loadRows = [&](int b, const int (&f)[U], int (&k)[U], long long (&v)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool p = f[u] < thr;
            k[u] = p ? __ldcs(keyc + b + u * step) : 0;
            v[u] = p ? __ldcs(value + b + u * step) : 0;
        }
    };
    int f[U], f1[U], kr[U];
    long long v[U];
    loadFilter(first + lane, f);
    loadFilter(first + lane + U * step, f1);
    loadRows(first + lane, f, kr, v);
    for (int b = first + lane; b - lane < n; b += U * step) {
        int f2[U], k1[U];
        long long v1[U];
        loadFilter(b + 2 * U * step, f2);
        loadRows(b + U * step, f1, k1, v1);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool live = f[u] < thr;
            const unsigned enc = live ? code(kr[u]) : 0u;
            const unsigned long long val = (unsigned long long)v[u];
            bool cold = live;
            if (PATH == GroupPath::Direct) {
                const unsigned i = enc - directBase;
                if (live && i < (unsigned)st.slots) {
                    st.add((int)i, val);
                    cold = false;
                }
            } else if (PATH == GroupPath::Shared) {
                // the search ends before the adds: lanes that find their
                // slot at different probes then add together
                const unsigned lm = __ballot_sync(0xffffffffu, live);
                if (live) {
                    int at = -1;
                    int h = (int)__umulhi(enc * 0x9E3779B1u, (unsigned)st.slots);
#pragma unroll 1
                    for (int p = 0; p < kSmemProbe; ++p) {
                        unsigned cur = *(volatile unsigned*)st.key(h);
                        if (cur == 0u) {
                            const unsigned prev = atomicCAS(st.key(h), 0u, enc);
                            cur = prev == 0u ? enc : prev;
                        }
                        if (cur == enc) {
                            at = h;
                            break;
                        }
                        h = h + 1 < st.slots ? h + 1 : 0;
                    }
                    __syncwarp(lm);
                    if (at >= 0) st.add(at, val);
                    cold = at < 0;
                }
            } else if (warp) {
                if (live) {
                    const unsigned am = __activemask();
                    const unsigned peers = __match_any_sync(am, enc);
                    const unsigned long long sum = gpudb_peer_sum(am, peers, val);
                    if (lane == __ffs(peers) - 1) globalAdd<DENSE>(q, ht, log2cap, enc, (unsigned)__popc(peers), sum);
                }
                cold = false;
            }
            if (DENSE) {
                if (cold) slotAdd(ht + (enc - 1u), 1u, val);
            } else {
                cq.push(cold, enc, val, take);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f[u] = f1[u];
            f1[u] = f2[u];
            kr[u] = k1[u];
            v[u] = v1[u];
        }
    }
    if (!DENSE && cq.n) {  // the rest of this item's queued rows
        take(0, cq.n);
        cq.n = 0;
        __syncwarp();
    }
}

template <int U>
__global__ void __launch_bounds__(1024, 1) kGroup(const QDesc* __restrict__ qs, WorkList wl, long long tile,
                                                  unsigned long long* counter) {
    extern __shared__ unsigned long long groupShared[];
    __shared__ long long s_item[2];
    const int words = kTableWords * (int)blockDim.x;
    SharedTable st{reinterpret_cast<unsigned*>(groupShared), 0};
    unsigned long long* coldV = groupShared + words / 2;
    unsigned* coldK = reinterpret_cast<unsigned*>(coldV + (blockDim.x >> 5) * kColdCap);
    ColdQueue cq{coldV + (threadIdx.x >> 5) * kColdCap, coldK + (threadIdx.x >> 5) * kColdCap, 0};
    for (int i = threadIdx.x; i < words; i += blockDim.x) st.w[i] = 0u;
    const long long total = __ldg(wl.prefix + wl.nq);
    // the query whose groups the shared table holds, -1 when empty: the table
    // is flushed into that query's global table only when the CTA moves to
    // another query's rows or runs out of work, so a query's work items on
    // one CTA share one table and one flush
    int heldQ = -1;
    auto shape = [&](const QDesc& q) {
        st.slots = q.aggMode == GPUDB_AGG_SHARED_DIRECT ? directSlots((int)blockDim.x) : hashedSlots((int)blockDim.x);
    };
    auto flushShared = [&](const QDesc& q) {
        shape(q);
        const bool direct = q.aggMode == GPUDB_AGG_SHARED_DIRECT;
        for (int i = threadIdx.x; i < st.slots; i += blockDim.x) {
            const unsigned c = *st.cnt(i);
            if (c) {
                const unsigned k = direct ? (unsigned)i + q.directBase : *st.key(i);
                const unsigned long long v = ((unsigned long long)*st.hi(i) << 32) | *st.lo(i);
                if (q.dense) globalAdd<true>(q, q.ht, q.log2cap, k, c, v);
                else globalAdd<false>(q, q.ht, q.log2cap, k, c, v);
                *st.cnt(i) = 0u;
                *st.lo(i) = 0u;
                *st.hi(i) = 0u;
            }
            if (!direct) *st.key(i) = 0u;
        }
    };
    // Work items are pulled one ahead: the counter's answer arrives while the
    // current item is processed, and an item costs one barrier.
    if (threadIdx.x == 0) s_item[0] = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    for (int it = 0;; it ^= 1) {
        const long long w = s_item[it];
        if (w >= total) break;
        long long ahead = 0;
        if (threadIdx.x == 0) ahead = (long long)atomicAdd(counter, 1ull);
        const int qi = findQuery(wl, w);
        const int qd = __ldg(wl.q + qi);
        if (heldQ >= 0 && heldQ != qd) {
            // the item's closing barrier ordered every add of the held query
            // before this flush; the barrier after it orders the reset before
            // the next rows' adds
            flushShared(qs[heldQ]);
            heldQ = -1;
            __syncthreads();
        }
        const QDesc& q = qs[qd];
        const long long r0 = (w - __ldg(wl.prefix + qi)) * tile, r1 = min(q.rows, r0 + tile);
        shape(q);
        if (q.aggMode == GPUDB_AGG_SHARED_DIRECT) {
            if (q.dense) groupTile<U, GroupPath::Direct, true>(q, st, q.directBase, cq, r0, r1);
            else groupTile<U, GroupPath::Direct, false>(q, st, q.directBase, cq, r0, r1);
            heldQ = qd;
        } else if (q.aggMode == GPUDB_AGG_SHARED) {
            if (q.dense) groupTile<U, GroupPath::Shared, true>(q, st, 0u, cq, r0, r1);
            else groupTile<U, GroupPath::Shared, false>(q, st, 0u, cq, r0, r1);
            heldQ = qd;
        } else if (q.dense) {
            groupTile<U, GroupPath::Global, true>(q, st, 0u, cq, r0, r1);
        } else {
            groupTile<U, GroupPath::Global, false>(q, st, 0u, cq, r0, r1);
        }
        if (threadIdx.x == 0) s_item[it ^ 1] = ahead;
        __syncthreads();
    }
    // the closing barriers ordered the last adds before this flush
    if (heldQ >= 0) flushShared(qs[heldQ]);
}

// The warps' sorted lists (lane j of each holds its j-th best) -> warp 0
// holds the block's best kTopK: pairwise list merges through shared memory.
__device__ __forceinline__ void blockTopK(long long& rv, long long& rk, long long* sv, long long* sk) {
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5);
    __syncthreads();  // an earlier merge may still read sv / sk
    sv[threadIdx.x] = rv;
    sk[threadIdx.x] = rk;
    for (int s = 1; s < nw; s <<= 1) {
        __syncthreads();
        if ((warp & (2 * s - 1)) == 0 && warp + s < nw) {
            gpudb_topk_warp_merge_list<kTopK>(rv, rk, sv[(warp + s) * 32 + lane], sk[(warp + s) * 32 + lane]);
            sv[threadIdx.x] = rv;
            sk[threadIdx.x] = rk;
        }
    }
}

// ---- after the group-by: count every grouped query's groups and, for TOPK,
// keep the best kTopK of each chunk of its table. Each warp walks the slots
// 32 at a time and keeps its best kTopK one per lane (a ballot drops slots
// that cannot enter).
__global__ void __launch_bounds__(256) kScanGroups(const QDesc* __restrict__ qs, WorkList wl, unsigned long long* counter) {
    __shared__ long long s_item;
    __shared__ long long sv[256], sk[256];
    __shared__ unsigned s_n;
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const long long total = __ldg(wl.prefix + wl.nq);
    for (long long w; (w = pullWork(counter, total, &s_item)) >= 0;) {
        const int qi = findQuery(wl, w);
        const QDesc& q = qs[__ldg(wl.q + qi)];
        const long long c = w - __ldg(wl.prefix + qi);
        const long long i0 = c * q.scanChunk, i1 = min(1ll << q.log2cap, i0 + q.scanChunk);
        const bool top = q.tmpl == GPUDB_TPL_TOPK;
        const Slot* __restrict__ ht = q.ht;
        if (threadIdx.x == 0) s_n = 0u;
        __syncthreads();
        unsigned n = 0;
        long long rv = GPUDB_TOPK_NONE_VAL, rk = GPUDB_TOPK_NONE_KEY;
        for (long long b = i0 + warp * 32; b < i1; b += blockDim.x) {
            const long long i = b + lane;
            Slot s{0u, 0u, 0ull};
            if (i < i1) s = ht[i];
            const bool live = slotLive(q, s);
            n += (unsigned)__popc(__ballot_sync(0xffffffffu, live));
            if (top)
                gpudb_topk_warp_offer<kTopK>(rv, rk, live ? (long long)s.sum : GPUDB_TOPK_NONE_VAL,
                                             live ? slotKey(q, s, i) : GPUDB_TOPK_NONE_KEY);
        }
        if (lane == 0 && n) atomicAdd(&s_n, n);
        if (top) {
            blockTopK(rv, rk, sv, sk);
            if (threadIdx.x < (unsigned)kTopK) {
                long long* dst = q.tk_part + 2 * (kTopK * c + lane);
                dst[0] = rv;
                dst[1] = rk;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_n) atomicAdd(q.nslots, (unsigned long long)s_n);
    }
}

// ---- TOPK, pass 2: one CTA per query merges its chunks' lists --------------
__global__ void __launch_bounds__(256) kTopKMerge(const QDesc* __restrict__ qs, const int* __restrict__ qlist) {
    __shared__ long long sv[256], sk[256];
    const QDesc& q = qs[qlist[blockIdx.x]];
    const int lane = (int)(threadIdx.x & 31u);
    long long rv = GPUDB_TOPK_NONE_VAL, rk = GPUDB_TOPK_NONE_KEY;
    for (long long c = threadIdx.x >> 5; c < q.tk_chunks; c += blockDim.x >> 5) {
        const bool in = lane < kTopK;
        const long long v = in ? q.tk_part[2 * (kTopK * c + lane)] : GPUDB_TOPK_NONE_VAL;
        const long long k = in ? q.tk_part[2 * (kTopK * c + lane) + 1] : GPUDB_TOPK_NONE_KEY;
        gpudb_topk_warp_merge_list<kTopK>(rv, rk, v, k);
    }
    blockTopK(rv, rk, sv, sk);
    if (threadIdx.x < 32u) {
        const long long m = min((long long)q.k, (long long)*q.nslots);
        if (lane < m) {
            q.topk_out[2 * lane] = rk;
            q.topk_out[2 * lane + 1] = rv;
        }
        if (lane == 0) *q.topk_n = (unsigned long long)m;
    }
}

// ---- exact statistics: passing rows and distinct keys ----------------------
__global__ void __launch_bounds__(1024) kStats(const QDesc* __restrict__ qs, WorkList wl, long long tile, unsigned long long* counter) {
    __shared__ long long s_item;
    const long long total = __ldg(wl.prefix + wl.nq);
    for (long long w; (w = pullWork(counter, total, &s_item)) >= 0;) {
        const int qi = findQuery(wl, w);
        const QDesc& q = qs[__ldg(wl.q + qi)];
        const int* __restrict__ filter = q.filter;
        const int* __restrict__ keyc = q.key;
        const int thr = q.thr;
                unsigned* bm = q.st_bitmap;
        const long long words = q.st_words;
        const long long r0 = (w - __ldg(wl.prefix + qi)) * tile, r1 = min(q.rows, r0 + tile);
        const bool grouped = q.tmpl == GPUDB_TPL_GROUPBY || q.tmpl == GPUDB_TPL_TOPK;
        const long long step = (long long)blockDim.x;
        long long pass = 0, fresh = 0;
        for (long long b = r0 + threadIdx.x; b < r1; b += kUnroll * step) {
            int f[kUnroll], kr[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) f[u] = b + u * step < r1 ? __ldcs(filter + b + u * step) : thr;
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) kr[u] = (grouped && f[u] < thr) ? __ldcs(keyc + b + u * step) : 0;
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                if (f[u] >= thr) continue;
                ++pass;
                if (!grouped) continue;
                const long long k = keyMod(kr[u], q);
                const long long wd = k >> 5;
                const unsigned bit = 1u << (unsigned)(k & 31);
                if (k < 0 || wd >= words) {
                    gpudb_set_error(q.err, GPUDB_ERR_BOUNDS);
                    continue;
                }
                if ((bm[wd] & bit) == 0u && (atomicOr(bm + wd, bit) & bit) == 0u) ++fresh;
            }
        }
        pass = gpudb_warp_sum_i64(pass);
        fresh = gpudb_warp_sum_i64(fresh);
        if ((threadIdx.x & 31) == 0) {
            if (pass) atomicAdd(q.st_pass, (unsigned long long)pass);
            if (fresh) atomicAdd(q.st_distinct, (unsigned long long)fresh);
        }
    }
}

// ---- 4096-row feature sample: one CTA per query ----------------------------
// Evenly spaced rows of the slice: rows sampled, rows passing the filter,
// distinct group keys among them and the multiplicity of the most frequent
// key (the skew signal that picks the aggregation strategy).
// Latency: a thread's four sample rows load together (filter words, then the
// keys of those that pass), and the counts are 32-bit (a 64-bit shared add
// is a compare-and-swap loop, 4,096 of them on one word). B200, four queries
// of 1M-5M rows: 30 us with 256 threads and 64-bit counts -> 18 us.
constexpr int kSample = 4096, kSampleSlots = 8192;
constexpr int kSampleSmem = kSampleSlots * (8 + 4);
constexpr int kSampleThreads = 1024, kSampleRows = kSample / kSampleThreads;
__global__ void __launch_bounds__(kSampleThreads) kSampleStats(const QDesc* qs, unsigned long long* out /* [n][4] */) {
    extern __shared__ unsigned long long setKeys[];
    unsigned* setCnt = reinterpret_cast<unsigned*>(setKeys + kSampleSlots);
    __shared__ unsigned s_pass, s_distinct, s_top;
    const QDesc& q = qs[blockIdx.x];
    const long long m = q.rows < kSample ? q.rows : kSample;
    const bool grouped = q.tmpl == GPUDB_TPL_GROUPBY || q.tmpl == GPUDB_TPL_TOPK;
    long long r[kSampleRows];
    bool pass[kSampleRows];
    int key[kSampleRows];
#pragma unroll
    for (int u = 0; u < kSampleRows; ++u) {
        const long long j = threadIdx.x + u * kSampleThreads;
        r[u] = j < m ? (j * q.rows) / m : -1;  // evenly spaced rows of the slice
    }
#pragma unroll
    for (int u = 0; u < kSampleRows; ++u) pass[u] = r[u] >= 0 && q.filter[r[u]] < q.thr;
#pragma unroll
    for (int u = 0; u < kSampleRows; ++u) key[u] = grouped && pass[u] ? q.key[r[u]] : 0;
    for (int i = threadIdx.x; i < kSampleSlots; i += kSampleThreads) {
        setKeys[i] = GPUDB_EMPTY64;
        setCnt[i] = 0u;
    }
    if (threadIdx.x == 0) {
        s_pass = 0;
        s_distinct = 0;
        s_top = 0;
    }
    __syncthreads();
    unsigned n = 0, fresh = 0;
#pragma unroll
    for (int u = 0; u < kSampleRows; ++u) {
        if (!pass[u]) continue;
        ++n;
        if (!grouped) continue;
        const unsigned long long k = (unsigned long long)keyMod(key[u], q);
        unsigned h = (unsigned)gpudb_hash_slot(k, 13);
        for (int p = 0; p < kSampleSlots; ++p) {
            const unsigned long long cur = setKeys[h];
            bool mine = cur == k;
            if (cur == GPUDB_EMPTY64) {
                const unsigned long long prev = atomicCAS(setKeys + h, GPUDB_EMPTY64, k);
                if (prev == GPUDB_EMPTY64) ++fresh;
                mine = prev == GPUDB_EMPTY64 || prev == k;
            }
            if (mine) {
                atomicAdd(setCnt + h, 1u);
                break;
            }
            h = (h + 1) & (kSampleSlots - 1);
        }
    }
    n = __reduce_add_sync(0xffffffffu, n);
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0) {
        if (n) atomicAdd(&s_pass, n);
        if (fresh) atomicAdd(&s_distinct, fresh);
    }
    __syncthreads();
    unsigned top = 0;
    for (int i = threadIdx.x; i < kSampleSlots; i += kSampleThreads) top = max(top, setCnt[i]);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_top, top);
    __syncthreads();
    if (threadIdx.x == 0) {
        out[4 * blockIdx.x] = (unsigned long long)m;
        out[4 * blockIdx.x + 1] = s_pass;
        out[4 * blockIdx.x + 2] = s_distinct;
        out[4 * blockIdx.x + 3] = s_top;
    }
}

// ---- a batch's last launch: what the host needs to know of it (one CTA) ----
// Per-query result rows and their exclusive prefix, for kCollect and in the
// pinned `host` (rows[n], offs[n + 1]), the error words, and zeroed cursors.
// The host waits for the batch alone: asked for afterwards (a launch, two
// copies and a wait more), they were 40 us of a 300 us batch of four queries.
__global__ void kResultRows(const QDesc* __restrict__ qs, int n, unsigned long long* offs, unsigned long long* cursors,
                            const unsigned* __restrict__ errs, unsigned long long* host, unsigned* errHost) {
    unsigned long long* rowsHost = host;
    unsigned long long* offsHost = host + n;
    for (int i = threadIdx.x; i <= n; i += blockDim.x) cursors[i] = 0ull;
    for (int i = threadIdx.x; i < n; i += blockDim.x) errHost[i] = errs[i];
    __shared__ unsigned long long carry;
    __shared__ unsigned long long wsum[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n; base += blockDim.x) {
        const int i = base + threadIdx.x;
        unsigned long long r = 0;
        if (i < n) {
            const QDesc& q = qs[i];
            r = q.tmpl == GPUDB_TPL_GROUPBY ? *q.nslots : q.tmpl == GPUDB_TPL_TOPK ? *q.topk_n : 1ull;
            rowsHost[i] = r;
        }
        unsigned long long x = r;  // inclusive warp scan
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)(threadIdx.x & 31) >= o) x += y;
        }
        if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = x;
        __syncthreads();
        unsigned long long before = carry;
        for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) before += wsum[w];
        if (i < n) offsHost[i] = offs[i] = before + x - r;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) offsHost[n] = offs[n] = carry;
}

// ---- collect: compaction of every query's rows into one packed buffer ------
// `counter`, `cursor`: zero; one position counter per query (group rows come in no order).
__global__ void __launch_bounds__(256) kCollect(const QDesc* __restrict__ qs, WorkList wl, unsigned long long* counter,
                                                unsigned long long* cursor, const unsigned long long* __restrict__ offs,
                                                long long* __restrict__ out) {
    __shared__ long long s_item;
    const unsigned lane = threadIdx.x & 31u;
    const long long total = __ldg(wl.prefix + wl.nq);
    for (long long w; (w = pullWork(counter, total, &s_item)) >= 0;) {
        const int qi = findQuery(wl, w);
        const int id = __ldg(wl.q + qi);
        const QDesc& q = qs[id];
        long long* dst = out + 3 * (long long)offs[id];
        const long long c = w - __ldg(wl.prefix + qi);
        if (q.tmpl == GPUDB_TPL_AGG || q.tmpl == GPUDB_TPL_JOIN) {
            if (threadIdx.x == 0) {
                dst[0] = (long long)q.agg[0];
                // exact 128-bit sum = (int64)w1 * 2^32 + w0, split into (lo, hi)
                const __int128 s = (__int128)(long long)q.agg[2] * ((__int128)1 << 32) + (__int128)q.agg[1];
                dst[1] = (long long)(unsigned long long)s;
                dst[2] = (long long)(s >> 64);
            }
        } else if (q.tmpl == GPUDB_TPL_TOPK) {
            const long long m = (long long)*q.topk_n;
            for (long long i = threadIdx.x; i < m; i += blockDim.x) {
                dst[3 * i] = q.topk_out[2 * i];
                dst[3 * i + 1] = q.topk_out[2 * i + 1];
                dst[3 * i + 2] = 0;
            }
        } else {
            // a warp takes 128 slots at a time and reserves its rows with one atomic
            const long long i1 = min(1ll << q.log2cap, (c + 1) * q.scanChunk);
            for (long long b = c * q.scanChunk + (threadIdx.x >> 5) * 128; b < i1; b += 4 * blockDim.x) {
                Slot s[4];
                unsigned m[4], n = 0u;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const long long i = b + u * 32 + lane;
                    s[u] = i < i1 ? q.ht[i] : Slot{0u, 0u, 0ull};
                    m[u] = __ballot_sync(0xffffffffu, slotLive(q, s[u]));
                    n += __popc(m[u]);
                }
                unsigned long long p = 0ull;
                if (lane == 0u && n) p = atomicAdd(cursor + id, (unsigned long long)n);
                p = __shfl_sync(0xffffffffu, p, 0);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (m[u] >> lane & 1u) {
                        long long* row = dst + 3 * (p + __popc(m[u] & ((1u << lane) - 1u)));
                        row[0] = slotKey(q, s[u], b + u * 32 + lane);
                        row[1] = (long long)s[u].count;
                        row[2] = (long long)s[u].sum;
                    }
                    p += __popc(m[u]);
                }
            }
        }
    }
}

unsigned long long pow2ceil(unsigned long long v) {
    unsigned long long p = 16;
    while (p < v) p <<= 1;
    return p;
}
int log2u(unsigned long long v) {
    int l = 0;
    while ((1ull << l) < v) l++;
    return l;
}
bool grouped(int tmpl) { return tmpl == GPUDB_TPL_GROUPBY || tmpl == GPUDB_TPL_TOPK; }

#define B_CHECK(call, code)                                                                        \
    do {                                                                                           \
        const cudaError_t _e = (call);                                                             \
        if (_e != cudaSuccess) {                                                                   \
            gpudb::setThreadError(std::string("batch: ") + #call + ": " + cudaGetErrorString(_e)); \
            return code;                                                                           \
        }                                                                                          \
    } while (0)

// Grow-only device buffer from the stream-ordered pool allocator: growing
// it never synchronises the device (cudaFree would), so batches of other
// streams keep running while this one resizes; 25 % headroom on growth.
struct DeviceBuf {
    void* p = nullptr;
    size_t bytes = 0;
    int reserve(size_t want, cudaStream_t st) {
        if (want <= bytes) return GPUDB_OK;
        release(st);
        const size_t cap = want + want / 4 + 256;
        B_CHECK(cudaMallocAsync(&p, cap, st), GPUDB_E_ALLOC);
        bytes = cap;
        return GPUDB_OK;
    }
    void release(cudaStream_t st) {
        if (p) cudaFreeAsync(p, st);
        p = nullptr;
        bytes = 0;
    }
};

size_t al256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace

struct gpudb_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    int numSMs = 148;
    int block = 512, maxProbe = 128, warpAgg = 1;
    // threads per CTA and rows in flight per thread of the group-by kernel.
    // Measured on the 64-query mixed batch (group stage, ms): 512 threads
    // with 1 / 2 / 4 rows 3.92 / 3.62 / 5.08, 1,024 threads 3.39 / 3.06 /
    // 4.25 (2.80 for 2 rows since the shared search ends before its adds):
    // the larger CTA holds the larger shared table, four rows spill.
    int groupBlock = 1024, groupRows = 2;
    // rows in flight per thread of the agg / join kernel: 2 (32 registers,
    // every thread slot resident; measured 9.9 ms against 10.6 ms per
    // mixed batch) or 4 (64 registers)
    int aggRows = 2;
    long long tile = 32768;  // rows per work item (measured: 16K 5.31k, 32K 5.45k mixed queries/s)
    std::vector<gpudb_batch_query> queries;
    std::vector<QDesc> desc;
    DeviceBuf arena;  // zero-initialised per execution
    size_t zeroBytes = 0;
    DeviceBuf scratch;  // never initialised: result offsets and cursors, top-k partials
    DeviceBuf meta;     // descriptors + work lists
    DeviceBuf stats, collect;
    QDesc* dDesc = nullptr;
    WorkList wlBuild{}, wlAgg{}, wlGroup{}, wlScan{}, wlStats{}, wlCollect{};
    // rows per work item of each list: the tuning's, or fewer when the batch
    // would leave CTAs without work
    long long tileBuild = 0, tileAgg = 0, tileGroup = 0, tileStats = 0;
    int* dTopk = nullptr;
    int nTopk = 0;
    unsigned long long* counters = nullptr;  // work counters (first words of the arena)
    unsigned* errs = nullptr;                // one error word per query (behind the counters)
    unsigned long long* resOffs = nullptr;   // result offsets [n + 1]
    unsigned long long* cursors = nullptr;   // kCollect's work counter and the queries' positions
    bool cursorsZero = false;
    // pinned, written by the kernels: rows[n] and offsets[n + 1] of the last
    // execution, its error words, and the sample statistics
    unsigned long long* resHost = nullptr;
    unsigned* errHost = nullptr;
    unsigned long long* sampleHost = nullptr;
    size_t hostCap = 0;  // queries
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t graphExec = nullptr;
    bool dirty = true;
    bool executed = false;  // resHost holds the last execution's rows
    long long lastLaunches = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t evStage[GPUDB_BATCH_STAGES + 1] = {};
    double stageMs[GPUDB_BATCH_STAGES] = {};
    bool stagesValid = false;
};

namespace {

void dropGraph(gpudb_batch* b) {
    if (b->graphExec) cudaGraphExecDestroy(b->graphExec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->graphExec = nullptr;
    b->graph = nullptr;
}

long long scanChunk(unsigned long long cap) {
    return std::min(kScanMax, std::max<long long>(kScanMin, (long long)cap / 32));
}

// Lay out the arena and the work lists for the current queries.
int plan(gpudb_batch* b) {
    const int n = (int)b->queries.size();
    size_t z = al256(8 * 8);  // work counters
    const size_t zErr = z;
    z += al256(4 * (size_t)n);
    size_t sc = al256(8 * (2 * (size_t)n + 2));  // offsets, cursors
    std::vector<size_t> zOff(n), sOff(n);
    std::vector<unsigned long long> caps(n, 0);
    std::vector<long long> tkChunks(n, 0);
    for (int i = 0; i < n; i++) {
        const auto& q = b->queries[i];
        zOff[i] = z;
        z += 64;  // agg[3], topk_n, nslots
        if (q.tmpl == GPUDB_TPL_JOIN) z += 4 * ((size_t)q.dim_max_key / 32 + 1);
        if (grouped(q.tmpl)) {
            caps[i] = pow2ceil(2 * std::max<uint64_t>(q.groups, 1));
            z = al256(z);
            z += sizeof(Slot) * caps[i];
            if (q.tmpl == GPUDB_TPL_TOPK) {
                sOff[i] = sc;
                tkChunks[i] = (long long)((caps[i] + scanChunk(caps[i]) - 1) / scanChunk(caps[i]));
                sc += al256(16 * kTopK * (size_t)tkChunks[i] + 16 * kTopK);
            }
        }
        z = al256(z);
    }
    if (int st = b->arena.reserve(z, b->stream)) return st;
    if (int st = b->scratch.reserve(sc, b->stream)) return st;
    b->zeroBytes = z;
    char* zb = static_cast<char*>(b->arena.p);
    char* sb = static_cast<char*>(b->scratch.p);
    b->counters = reinterpret_cast<unsigned long long*>(zb);
    b->errs = reinterpret_cast<unsigned*>(zb + zErr);
    b->resOffs = reinterpret_cast<unsigned long long*>(sb);
    b->cursors = b->resOffs + n + 1;
    b->desc.assign(n, QDesc{});
    std::vector<int> lBuild, lAgg, lGroup, lTopk, lAll(n), lCollect;
    std::vector<long long> pBuild{0}, pAgg{0}, pGroup{0}, pScan{0}, pAll{0}, pCollect{0};
    // Two work items for each resident CTA (three of the group-by's larger
    // ones) before an item gets the tuning's rows: 8M rows in 32K-row items
    // are work for 233 of 592 CTAs (B200, four queries of 1M-5M rows, group
    // stage: 192 us in such items by the kernel of that time, 43 us now).
    long long rBuild = 0, rAgg = 0, rGroup = 0;
    for (const auto& q : b->queries) {
        if (q.tmpl == GPUDB_TPL_JOIN) rBuild += (long long)q.dim_rows;
        (grouped(q.tmpl) ? rGroup : rAgg) += (long long)q.rows;
    }
    auto tileFor = [&](long long rows, long long items) {
        const long long t = (rows / items + 1023) / 1024 * 1024;
        return std::min(b->tile, std::max<long long>(4096, t));
    };
    b->tileBuild = tileFor(rBuild, 8ll * b->numSMs);
    b->tileAgg = tileFor(rAgg, 8ll * b->numSMs);
    b->tileGroup = tileFor(rGroup, 3ll * b->numSMs * std::max(1, 1024 / b->groupBlock));
    b->tileStats = tileFor(rAgg + rGroup, 8ll * b->numSMs);
    for (int i = 0; i < n; i++) {
        const auto& q = b->queries[i];
        QDesc& d = b->desc[i];
        d.tmpl = q.tmpl;
        d.thr = q.thr;
        d.k = q.k;
        d.attr_lt = q.attr_lt;
        d.card = q.card > 0 ? q.card : 1;
        cardDivisor(d.card, &d.cardMagic, &d.cardSh1, &d.cardSh2);
        d.rows = (long long)q.rows;
        d.key = q.key;
        d.filter = q.filter;
        d.value = reinterpret_cast<const long long*>(q.value);
        d.fk = q.fk;
        d.dim_key = q.dim_key;
        d.dim_attr = q.dim_attr;
        d.dim_rows = (long long)q.dim_rows;
        d.maxProbe = b->maxProbe;
        // aggregation strategy: the caller's choice, else the shared-memory
        // table (with spill to the global one), which is never far off
        d.aggMode = q.agg_mode != GPUDB_AGG_AUTO ? q.agg_mode : GPUDB_AGG_SHARED;
        if (!b->warpAgg && d.aggMode == GPUDB_AGG_GLOBAL_WARP) d.aggMode = GPUDB_AGG_GLOBAL;
        // The direct table takes every key of (-card, card), or, of a larger
        // domain, the keys >= 0 (the column's statistics say that there are
        // no others; any that occur go to the global table). It never loses
        // to the hashed one while a CTA's flush stays small beside its rows:
        // below that, a large domain keeps the other strategies.
        const int slots = directSlots(b->groupBlock);
        const bool both = 2 * d.card - 1 <= slots, upper = d.card <= slots && q.key_min >= 0;
        const bool enough = both && d.card <= 1024 ? true : d.rows >= 4ll * b->numSMs * (1024 / b->groupBlock) * d.card;
        if (d.aggMode == GPUDB_AGG_SHARED && (both || upper) && enough) d.aggMode = GPUDB_AGG_SHARED_DIRECT;
        else if (d.aggMode == GPUDB_AGG_SHARED_DIRECT && !((both || upper) && enough))
            d.aggMode = both || upper ? GPUDB_AGG_GLOBAL : GPUDB_AGG_SHARED;
        d.directBase = both ? 1u : (unsigned)d.card;
        char* p = zb + zOff[i];
        d.agg = reinterpret_cast<unsigned long long*>(p);
        d.topk_n = d.agg + 3;
        d.nslots = d.agg + 4;
        d.err = b->errs + i;
        p += 64;
        if (q.tmpl == GPUDB_TPL_JOIN) {
            d.bitmap = reinterpret_cast<unsigned*>(p);
            d.bitmap_words = q.dim_max_key / 32 + 1;
            p += 4 * (size_t)d.bitmap_words;
        }
        if (grouped(q.tmpl)) {
            p = zb + al256((size_t)(p - zb));
            d.ht = reinterpret_cast<Slot*>(p);
            d.log2cap = log2u(caps[i]);
            d.scanChunk = scanChunk(caps[i]);
            // no probe and no overflow where the table can hold every key anyway
            d.dense = 2 * (unsigned long long)d.card - 1 <= caps[i];
            if (q.tmpl == GPUDB_TPL_TOPK) {
                d.tk_part = reinterpret_cast<long long*>(sb + sOff[i]);
                d.tk_chunks = tkChunks[i];
                d.topk_out = d.tk_part + 2 * kTopK * tkChunks[i];
            }
        }
        auto items = [](long long rows, long long tile) { return (rows + tile - 1) / tile; };
        lAll[i] = i;
        pAll.push_back(pAll.back() + items(d.rows, b->tileStats));
        if (q.tmpl == GPUDB_TPL_JOIN) {
            lBuild.push_back(i);
            pBuild.push_back(pBuild.back() + items(d.dim_rows, b->tileBuild));
        }
        if (q.tmpl == GPUDB_TPL_AGG || q.tmpl == GPUDB_TPL_JOIN) {
            lAgg.push_back(i);
            pAgg.push_back(pAgg.back() + items(d.rows, b->tileAgg));
        }
        const long long chunks = caps[i] ? items((long long)caps[i], d.scanChunk) : 0;
        if (grouped(q.tmpl)) {
            lGroup.push_back(i);
            pGroup.push_back(pGroup.back() + items(d.rows, b->tileGroup));
            pScan.push_back(pScan.back() + chunks);
        }
        if (q.tmpl == GPUDB_TPL_TOPK) lTopk.push_back(i);
        lCollect.push_back(i);
        pCollect.push_back(pCollect.back() + (q.tmpl == GPUDB_TPL_GROUPBY ? chunks : 1));
    }
    std::vector<char> host;
    auto put = [&](const void* src, size_t bytes) {
        const size_t off = al256(host.size());
        host.resize(off + std::max<size_t>(bytes, 8));
        if (bytes) std::memcpy(host.data() + off, src, bytes);
        return off;
    };
    const size_t oDesc = put(b->desc.data(), sizeof(QDesc) * n);
    auto putList = [&](const std::vector<int>& l, const std::vector<long long>& pf) {
        const size_t a = put(l.data(), 4 * l.size());
        const size_t c = put(pf.data(), 8 * pf.size());
        return std::make_pair(a, c);
    };
    const auto oB = putList(lBuild, pBuild), oA = putList(lAgg, pAgg), oG = putList(lGroup, pGroup),
               oT = putList(lGroup, pScan), oS = putList(lAll, pAll), oC = putList(lCollect, pCollect);
    const size_t oTop = put(lTopk.data(), 4 * lTopk.size());
    if (int st = b->meta.reserve(host.size(), b->stream)) return st;
    B_CHECK(cudaMemcpyAsync(b->meta.p, host.data(), host.size(), cudaMemcpyHostToDevice, b->stream), GPUDB_E_CUDA);
    char* m = static_cast<char*>(b->meta.p);
    auto wl = [&](std::pair<size_t, size_t> o, size_t nq) {
        return WorkList{reinterpret_cast<int*>(m + o.first), reinterpret_cast<long long*>(m + o.second), (int)nq};
    };
    b->dDesc = reinterpret_cast<QDesc*>(m + oDesc);
    b->wlBuild = wl(oB, lBuild.size());
    b->wlAgg = wl(oA, lAgg.size());
    b->wlGroup = wl(oG, lGroup.size());
    b->wlScan = wl(oT, lGroup.size());
    b->wlStats = wl(oS, n);
    b->wlCollect = wl(oC, lCollect.size());
    b->dTopk = reinterpret_cast<int*>(m + oTop);
    b->nTopk = (int)lTopk.size();
    if ((size_t)n > b->hostCap) {
        if (b->resHost) cudaFreeHost(b->resHost);
        b->resHost = nullptr;
        b->hostCap = 0;
        const size_t cap = std::max<size_t>(4096, 2 * (size_t)n);
        B_CHECK(cudaHostAlloc((void**)&b->resHost, 8 * (2 * cap + 1) + 32 * cap + 4 * cap, cudaHostAllocDefault),
                GPUDB_E_ALLOC);
        b->sampleHost = b->resHost + 2 * cap + 1;
        b->errHost = reinterpret_cast<unsigned*>(b->sampleHost + 4 * cap);
        b->hostCap = cap;
    }
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    dropGraph(b);
    b->executed = false;
    b->dirty = false;
    return GPUDB_OK;
}

int gridFor(gpudb_batch* b, const void* fn, int block, size_t smem = 0) {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, block, smem);
    return std::max(1, occ) * b->numSMs;
}

// Enqueue the memset + kernels of one execution on b->stream; with `stages`
// an event follows every step (not inside a graph capture).
int enqueue(gpudb_batch* b, bool stages) {
    const int n = (int)b->queries.size();
    long long launches = 0;
    auto mark = [&](int i) { if (stages) cudaEventRecord(b->evStage[i], b->stream); };
    mark(0);
    B_CHECK(cudaMemsetAsync(b->arena.p, 0, b->zeroBytes, b->stream), GPUDB_E_CUDA);
    mark(1);
    if (b->wlBuild.nq) {
        kJoinBuild<<<gridFor(b, (const void*)kJoinBuild, b->block), b->block, 0, b->stream>>>(b->dDesc, b->wlBuild,
                                                                                              b->tileBuild, b->counters + 0);
        launches++;
    }
    mark(2);
    if (b->wlAgg.nq) {
        if (b->aggRows == 2 && b->block <= 512)  // the 2-row form is built for blocks of <= 512
            kAgg<2><<<gridFor(b, (const void*)kAgg<2>, b->block), b->block, 0, b->stream>>>(
                b->dDesc, b->wlAgg, b->tileAgg, b->counters + 1);
        else
            kAgg<4><<<gridFor(b, (const void*)kAgg<4>, b->block), b->block, 0, b->stream>>>(
                b->dDesc, b->wlAgg, b->tileAgg, b->counters + 1);
        launches++;
    }
    mark(3);
    if (b->wlGroup.nq) {
        const int block = b->groupBlock;
        const size_t smem = groupSmem(block);
        auto launch = [&](void (*k)(const QDesc*, WorkList, long long, unsigned long long*)) {
            k<<<gridFor(b, (const void*)k, block, smem), block, smem, b->stream>>>(b->dDesc, b->wlGroup, b->tileGroup,
                                                                                  b->counters + 2);
        };
        if (b->groupRows == 1) launch(kGroup<1>);
        else if (b->groupRows == 2) launch(kGroup<2>);
        else launch(kGroup<4>);
        launches++;
    }
    mark(4);
    if (b->wlScan.nq) {
        kScanGroups<<<gridFor(b, (const void*)kScanGroups, 256), 256, 0, b->stream>>>(b->dDesc, b->wlScan, b->counters + 3);
        launches++;
    }
    mark(5);
    if (b->nTopk) {
        kTopKMerge<<<b->nTopk, 256, 0, b->stream>>>(b->dDesc, b->dTopk);
        launches++;
    }
    mark(6);
    B_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    if (n) {
        kResultRows<<<1, 1024, 0, b->stream>>>(b->dDesc, n, b->resOffs, b->cursors, b->errs, b->resHost, b->errHost);
        B_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
        launches++;
    }
    b->lastLaunches = launches;
    return GPUDB_OK;
}

float elapsed(gpudb_batch* b) {
    float t = 0;
    cudaEventElapsedTime(&t, b->ev0, b->ev1);
    return t;
}

// Zone-map statistics of a resident column: min and max of n int32 or
// int64 values (the sizer's column features). One grid-stride pass, warp
// shuffle reduction, one signed 64-bit atomicMin / atomicMax per warp.
template <typename T>
__global__ void __launch_bounds__(256) kColumnMinMax(const T* __restrict__ v, unsigned long long n,
                                                     long long* __restrict__ out) {
    long long lo = LLONG_MAX, hi = LLONG_MIN;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const long long x = (long long)__ldcs(v + i);
        lo = x < lo ? x : lo;
        hi = x > hi ? x : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    if ((threadIdx.x & 31u) == 0u) {
        atomicMin(out, lo);
        atomicMax(out + 1, hi);
    }
}

}  // namespace

extern "C" {

int gpudb_batch_create(gpudb_ctx* ctx, gpudb_batch** out) {
    if (!out) return GPUDB_E_INVALID;
    *out = nullptr;
    (void)ctx;  // the batch runs on the calling thread's current device
    auto b = std::make_unique<gpudb_batch>();
    int dev = 0;
    B_CHECK(cudaGetDevice(&dev), GPUDB_E_NOGPU);
    b->device = dev;
    B_CHECK(cudaDeviceGetAttribute(&b->numSMs, cudaDevAttrMultiProcessorCount, dev), GPUDB_E_CUDA);
    B_CHECK(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking), GPUDB_E_CUDA);
    B_CHECK(cudaEventCreate(&b->ev0), GPUDB_E_CUDA);
    B_CHECK(cudaEventCreate(&b->ev1), GPUDB_E_CUDA);
    for (auto& e : b->evStage) B_CHECK(cudaEventCreate(&e), GPUDB_E_CUDA);
    B_CHECK(cudaFuncSetAttribute(kSampleStats, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmem),
            GPUDB_E_LAUNCH);
    for (const void* k : {(const void*)kGroup<1>, (const void*)kGroup<2>, (const void*)kGroup<4>})
        B_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)groupSmem(1024)),
                GPUDB_E_LAUNCH);
    *out = b.release();
    return GPUDB_OK;
}

void gpudb_batch_free(gpudb_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    dropGraph(b);
    for (DeviceBuf* d : {&b->arena, &b->scratch, &b->meta, &b->stats, &b->collect}) d->release(b->stream);
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->resHost) cudaFreeHost(b->resHost);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    for (auto& e : b->evStage)
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

int gpudb_batch_set_queries(gpudb_batch* b, const gpudb_batch_query* q, int n) {
    if (!b || (n > 0 && !q) || n < 0) return GPUDB_E_INVALID;
    for (int i = 0; i < n; i++) {
        const auto& x = q[i];
        const std::string who = "batch: query " + std::to_string(i);
        if (x.tmpl < 0 || x.tmpl > GPUDB_TPL_TOPK || (x.rows && (!x.filter || !x.value))) {
            gpudb::setThreadError(who + " is malformed");
            return GPUDB_E_INVALID;
        }
        if (grouped(x.tmpl) && ((x.rows && !x.key) || x.card < 1 || x.card >= (1ll << 31) || x.rows >= (1ull << 32))) {
            gpudb::setThreadError(who + " needs a key column, 1 <= card < 2^31 and fewer than 2^32 rows");
            return GPUDB_E_INVALID;
        }
        if (grouped(x.tmpl) && x.groups > (1ull << 30)) {
            gpudb::setThreadError(who + " asks for more than 2^30 groups");
            return GPUDB_E_INVALID;
        }
        if (x.agg_mode < GPUDB_AGG_AUTO || x.agg_mode > GPUDB_AGG_SHARED_DIRECT) {
            gpudb::setThreadError(who + " has an unknown agg_mode");
            return GPUDB_E_INVALID;
        }
        if (x.tmpl == GPUDB_TPL_TOPK && (x.k < 1 || x.k > kTopK)) {
            gpudb::setThreadError(who + " needs 1 <= k <= 16");
            return GPUDB_E_INVALID;
        }
        if (x.tmpl == GPUDB_TPL_JOIN &&
            ((x.rows && !x.fk) || (x.dim_rows && (!x.dim_key || !x.dim_attr)) || x.dim_max_key < 0)) {
            gpudb::setThreadError(who + " needs fk, the dim columns and dim_max_key >= 0");
            return GPUDB_E_INVALID;
        }
    }
    cudaSetDevice(b->device);
    b->queries.assign(q, q + n);
    b->dirty = true;
    return plan(b);
}

int gpudb_batch_set_groups(gpudb_batch* b, int qi, uint64_t groups) {
    if (!b || qi < 0 || qi >= (int)b->queries.size() || groups > (1ull << 30)) return GPUDB_E_INVALID;
    if (b->queries[qi].groups != groups) {
        b->queries[qi].groups = groups;
        b->dirty = true;
    }
    return GPUDB_OK;
}

int gpudb_batch_set_agg_mode(gpudb_batch* b, int qi, int mode) {
    if (!b || qi < 0 || qi >= (int)b->queries.size() || mode < GPUDB_AGG_AUTO || mode > GPUDB_AGG_SHARED_DIRECT)
        return GPUDB_E_INVALID;
    if (b->queries[qi].agg_mode != mode) {
        b->queries[qi].agg_mode = mode;
        b->dirty = true;
    }
    return GPUDB_OK;
}

int gpudb_batch_set_option(gpudb_batch* b, const char* name, long long value) {
    if (!b || !name) return GPUDB_E_INVALID;
    const std::string n(name);
    if (n == "group_rows") {
        if (value != 1 && value != 2 && value != 4) {
            gpudb::setThreadError("group_rows must be 1, 2 or 4");
            return GPUDB_E_INVALID;
        }
        b->groupRows = (int)value;
        b->dirty = true;
        return GPUDB_OK;
    }
    if (n == "shared_warp") {
        if (value != 0 && value != 1) {
            gpudb::setThreadError("shared_warp must be 0 or 1");
            return GPUDB_E_INVALID;
        }
        return GPUDB_OK;  // rows go to the shared table directly in either case
    }
    if (n == "agg_rows") {
        if (value != 2 && value != 4) {
            gpudb::setThreadError("agg_rows must be 2 or 4");
            return GPUDB_E_INVALID;
        }
        b->aggRows = (int)value;
        b->dirty = true;
        return GPUDB_OK;
    }
    gpudb::setThreadError("unknown batch option '" + n + "'");
    return GPUDB_E_INVALID;
}

int gpudb_batch_set_tuning(gpudb_batch* b, int block, int tile_rows, int warp_aggregate, int max_probe) {
    if (!b || block < 64 || block > 1024 || block % 32 || tile_rows < 256 || max_probe < 1) return GPUDB_E_INVALID;
    b->block = b->groupBlock = block;
    b->tile = tile_rows;
    b->warpAgg = warp_aggregate ? 1 : 0;
    b->maxProbe = max_probe;
    b->dirty = true;
    return GPUDB_OK;
}

int gpudb_batch_execute(gpudb_batch* b, int use_graph, double* ms, uint32_t* errors) {
    if (!b) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    if (b->dirty)
        if (int st = plan(b)) return st;
    const int n = (int)b->queries.size();
    b->executed = false;
    B_CHECK(cudaEventRecord(b->ev0, b->stream), GPUDB_E_CUDA);
    if (use_graph) {
        if (!b->graphExec) {
            B_CHECK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), GPUDB_E_CUDA);
            const int st = enqueue(b, false);
            cudaGraph_t g = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
            if (st != GPUDB_OK) {
                if (g) cudaGraphDestroy(g);
                return st;
            }
            B_CHECK(ce, GPUDB_E_CUDA);
            b->graph = g;
            B_CHECK(cudaGraphInstantiate(&b->graphExec, g, 0), GPUDB_E_CUDA);
        }
        B_CHECK(cudaGraphLaunch(b->graphExec, b->stream), GPUDB_E_CUDA);
        b->stagesValid = false;
    } else {
        if (int st = enqueue(b, true)) return st;
    }
    B_CHECK(cudaEventRecord(b->ev1, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaEventSynchronize(b->ev1), GPUDB_E_CUDA);
    if (ms) *ms = elapsed(b);
    if (!use_graph) {
        for (int i = 0; i < GPUDB_BATCH_STAGES; i++) {
            float t = 0;
            cudaEventElapsedTime(&t, b->evStage[i], b->evStage[i + 1]);
            b->stageMs[i] = t;
        }
        b->stagesValid = true;
    }
    b->executed = true;
    b->cursorsZero = true;
    if (errors && n) std::memcpy(errors, b->errHost, sizeof(unsigned) * n);
    return GPUDB_OK;
}

int gpudb_batch_exact_stats(gpudb_batch* b, uint64_t* passing, uint64_t* distinct, double* ms) {
    if (!b) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    if (b->dirty)
        if (int st = plan(b)) return st;
    const int n = (int)b->queries.size();
    if (n == 0) return GPUDB_OK;
    // counter, pass[n], distinct[n], one distinct bitmap per grouped query
    size_t words = 0;
    for (const auto& q : b->queries)
        if (grouped(q.tmpl)) words += (size_t)q.card / 32 + 1;
    const size_t bytes = 8 + 16 * (size_t)n + 4 * words;
    if (int st = b->stats.reserve(bytes, b->stream)) return st;
    unsigned long long* counter = static_cast<unsigned long long*>(b->stats.p);
    unsigned long long* pass = counter + 1;
    unsigned long long* dist = pass + n;
    unsigned* bm = reinterpret_cast<unsigned*>(dist + n);
    std::vector<QDesc> d = b->desc;
    size_t w = 0;
    for (int i = 0; i < n; i++) {
        d[i].st_pass = pass + i;
        d[i].st_distinct = dist + i;
        if (grouped(b->queries[i].tmpl)) {
            d[i].st_bitmap = bm + w;
            d[i].st_words = d[i].card / 32 + 1;
            w += (size_t)d[i].st_words;
        }
    }
    // the pass runs on descriptors that carry the statistics buffers; the
    // execution's descriptors are put back behind it
    B_CHECK(cudaMemcpyAsync(b->dDesc, d.data(), sizeof(QDesc) * n, cudaMemcpyHostToDevice, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaEventRecord(b->ev0, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaMemsetAsync(b->stats.p, 0, bytes, b->stream), GPUDB_E_CUDA);
    kStats<<<gridFor(b, (const void*)kStats, b->block), b->block, 0, b->stream>>>(b->dDesc, b->wlStats, b->tileStats,
                                                                                  counter);
    B_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    B_CHECK(cudaEventRecord(b->ev1, b->stream), GPUDB_E_CUDA);
    std::vector<unsigned long long> h(2 * (size_t)n);
    B_CHECK(cudaMemcpyAsync(h.data(), pass, 16 * (size_t)n, cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaMemcpyAsync(b->dDesc, b->desc.data(), sizeof(QDesc) * n, cudaMemcpyHostToDevice, b->stream),
            GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    if (ms) *ms = elapsed(b);
    for (int i = 0; i < n; i++) {
        if (passing) passing[i] = h[i];
        if (distinct) distinct[i] = h[n + i];
    }
    return GPUDB_OK;
}

int gpudb_batch_features(gpudb_batch* b, float* f, double* ms) {
    if (!b || !f) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    if (b->dirty)
        if (int st = plan(b)) return st;
    const int n = (int)b->queries.size();
    if (n == 0) return GPUDB_OK;
    const unsigned long long* h = b->sampleHost;
    B_CHECK(cudaEventRecord(b->ev0, b->stream), GPUDB_E_CUDA);
    kSampleStats<<<n, kSampleThreads, kSampleSmem, b->stream>>>(b->dDesc, b->sampleHost);
    B_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    B_CHECK(cudaEventRecord(b->ev1, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    if (ms) *ms = elapsed(b);
    for (int i = 0; i < n; i++) {
        const auto& q = b->queries[i];
        const double m = (double)h[4 * i], pass = (double)h[4 * i + 1], dist = (double)h[4 * i + 2],
                     top = (double)h[4 * i + 3];
        const double rows = (double)q.rows;
        // key domain under the modulus, from the key column's min / max
        const double span = (double)q.key_max - (double)q.key_min + 1.0;
        const double card = std::max(1.0, std::min((double)std::max<int64_t>(q.card, 1), span > 0 ? span : 1.0));
        // predicate position inside the filter column's [min, max]
        const double frange = (double)q.filter_max - (double)q.filter_min + 1.0;
        const double predPos =
            frange > 0 ? std::min(1.0, std::max(0.0, ((double)q.thr - (double)q.filter_min) / frange)) : 0.0;
        const double sel = m > 0 ? pass / m : 0.0;
        const double expPass = rows * sel;
        const double uniformDistinct = card * (1.0 - std::exp(-expPass / card));
        float* x = f + (size_t)i * GPUDB_SIZER_FEATURES;
        for (int j = 0; j < GPUDB_SIZER_FEATURES; j++) x[j] = 0.0f;
        x[q.tmpl & 3] = 1.0f;                                      // template id, one-hot
        x[4] = (float)(std::log2(rows + 1.0) / 27.0);              // slice rows
        x[5] = (float)predPos;                                     // predicate constant vs column min / max
        x[6] = (float)(std::log2(card) / 24.0);                    // group-key domain
        x[7] = (float)sel;                                         // sample selectivity
        x[8] = (float)(pass > 0 ? dist / pass : 0.0);              // sample distinct / sample passing
        x[9] = (float)(std::log2(dist + 1.0) / 12.0);              // sample distinct count
        x[10] = (float)(std::log2(expPass + 1.0) / 27.0);          // estimated passing rows
        x[11] = (float)(std::log2((expPass + 1.0) / card) / 30.0);
        x[12] = (float)(pass > 0 ? top / pass : 0.0);              // share of the most frequent sample key
        x[13] = (float)(std::log2(pass + 1.0) / 12.0);             // sample passing count
        x[14] = (float)(std::log2(uniformDistinct + 1.0) / 24.0);  // uniform-key estimate of the groups
        x[15] = 1.0f;
    }
    return GPUDB_OK;
}

int gpudb_batch_collect(gpudb_batch* b, uint64_t* rows, void* host, uint64_t host_bytes, uint64_t* bytes_needed,
                        double* ms) {
    if (!b) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    if (b->dirty) {
        gpudb::setThreadError("batch: collect before execute");
        return GPUDB_E_INVALID;
    }
    const int n = (int)b->queries.size();
    if (n == 0) {
        if (bytes_needed) *bytes_needed = 0;
        return GPUDB_OK;
    }
    if (!b->executed) {
        gpudb::setThreadError("batch: collect before execute");
        return GPUDB_E_INVALID;
    }
    const unsigned long long total = b->resHost[2 * (size_t)n];
    if (rows)
        for (int i = 0; i < n; i++) rows[i] = b->resHost[i];
    if (bytes_needed) *bytes_needed = 24 * total;
    if (ms) *ms = 0.0;
    if (!host) return GPUDB_OK;
    if (host_bytes < 24 * total) {
        gpudb::setThreadError("batch: collect buffer too small");
        return GPUDB_E_INVALID;
    }
    if (total == 0) return GPUDB_OK;
    if (int st = b->collect.reserve(24 * total, b->stream)) return st;
    long long* out = static_cast<long long*>(b->collect.p);
    B_CHECK(cudaEventRecord(b->ev0, b->stream), GPUDB_E_CUDA);
    if (!b->cursorsZero)
        B_CHECK(cudaMemsetAsync(b->cursors, 0, 8 * ((size_t)n + 1), b->stream), GPUDB_E_CUDA);
    b->cursorsZero = false;
    kCollect<<<gridFor(b, (const void*)kCollect, 256), 256, 0, b->stream>>>(b->dDesc, b->wlCollect, b->cursors,
                                                                           b->cursors + 1, b->resOffs, out);
    B_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    B_CHECK(cudaMemcpyAsync(host, out, 24 * total, cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaEventRecord(b->ev1, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaEventSynchronize(b->ev1), GPUDB_E_CUDA);
    if (ms) *ms = elapsed(b);
    return GPUDB_OK;
}

int gpudb_batch_result_scalar(gpudb_batch* b, int qi, int64_t* count, uint64_t* sum_lo, int64_t* sum_hi) {
    if (!b || qi < 0 || qi >= (int)b->queries.size() || b->dirty) return GPUDB_E_INVALID;
    const QDesc& d = b->desc[qi];
    if (d.tmpl != GPUDB_TPL_AGG && d.tmpl != GPUDB_TPL_JOIN) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    unsigned long long w[3];
    B_CHECK(cudaMemcpyAsync(w, d.agg, 24, cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    const __int128 s = (__int128)(int64_t)w[2] * ((__int128)1 << 32) + (__int128)w[1];
    if (count) *count = (int64_t)w[0];
    if (sum_lo) *sum_lo = (uint64_t)s;
    if (sum_hi) *sum_hi = (int64_t)(s >> 64);
    return GPUDB_OK;
}

int gpudb_batch_result_groups(gpudb_batch* b, int qi, uint64_t cap, uint64_t* ngroups, int64_t* keys, int64_t* counts,
                              int64_t* sums) {
    if (!b || qi < 0 || qi >= (int)b->queries.size() || !ngroups || b->dirty) return GPUDB_E_INVALID;
    const QDesc& d = b->desc[qi];
    if (!grouped(d.tmpl)) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    unsigned long long n = 0;
    B_CHECK(cudaMemcpyAsync(&n, d.nslots, 8, cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    *ngroups = n;
    if (!keys || !counts || !sums || n == 0 || cap < n) return GPUDB_OK;
    std::vector<Slot> table((size_t)1 << d.log2cap);
    B_CHECK(cudaMemcpyAsync(table.data(), d.ht, sizeof(Slot) * table.size(), cudaMemcpyDeviceToHost, b->stream),
            GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    unsigned long long j = 0;
    for (size_t i = 0; i < table.size() && j < n; i++) {
        const Slot& s = table[i];
        if (!(d.dense ? s.count : s.key)) continue;
        keys[j] = (int64_t)decKey(d.dense ? (unsigned)i + 1u : s.key, d.card);
        counts[j] = (int64_t)s.count;
        sums[j] = (int64_t)s.sum;
        j++;
    }
    return GPUDB_OK;
}

int gpudb_batch_result_topk(gpudb_batch* b, int qi, int64_t* keys, int64_t* vals, int* n) {
    if (!b || qi < 0 || qi >= (int)b->queries.size() || !n || b->dirty) return GPUDB_E_INVALID;
    const QDesc& d = b->desc[qi];
    if (d.tmpl != GPUDB_TPL_TOPK) return GPUDB_E_INVALID;
    cudaSetDevice(b->device);
    unsigned long long cnt = 0;
    long long kv[2 * kTopK];
    B_CHECK(cudaMemcpyAsync(&cnt, d.topk_n, 8, cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaMemcpyAsync(kv, d.topk_out, sizeof(kv), cudaMemcpyDeviceToHost, b->stream), GPUDB_E_CUDA);
    B_CHECK(cudaStreamSynchronize(b->stream), GPUDB_E_CUDA);
    *n = (int)cnt;
    for (unsigned long long i = 0; i < cnt; i++) {
        if (keys) keys[i] = kv[2 * i];
        if (vals) vals[i] = kv[2 * i + 1];
    }
    return GPUDB_OK;
}

long long gpudb_batch_last_launches(gpudb_batch* b) { return b ? b->lastLaunches : 0; }

int gpudb_batch_stage_ms(gpudb_batch* b, double* ms) {
    if (!b || !ms) return GPUDB_E_INVALID;
    if (!b->stagesValid) {
        gpudb::setThreadError("batch: stage times need an execute without a graph");
        return GPUDB_E_INVALID;
    }
    for (int i = 0; i < GPUDB_BATCH_STAGES; i++) ms[i] = b->stageMs[i];
    return GPUDB_OK;
}

int gpudb_column_minmax(const void* column, uint64_t n, int elem_bytes, int64_t* min_out, int64_t* max_out,
                        void* stream) {
    if (!min_out || !max_out || (n && !column) || (elem_bytes != 4 && elem_bytes != 8)) {
        gpudb::setThreadError("column_minmax: needs int32 / int64 elements and output pointers");
        return GPUDB_E_INVALID;
    }
    if (n == 0) {
        *min_out = 0;
        *max_out = 0;
        return GPUDB_OK;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int dev = 0, sms = 0;
    B_CHECK(cudaGetDevice(&dev), GPUDB_E_NOGPU);
    B_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), GPUDB_E_CUDA);
    long long* d = nullptr;
    B_CHECK(cudaMallocAsync((void**)&d, 2 * sizeof(long long), st), GPUDB_E_ALLOC);
    const long long init[2] = {LLONG_MAX, LLONG_MIN};
    long long host[2] = {0, 0};
    cudaError_t e = cudaMemcpyAsync(d, init, sizeof init, cudaMemcpyHostToDevice, st);
    const unsigned long long want = (n + 255) / 256;
    const int blocks = (int)std::min<unsigned long long>(want, (unsigned long long)sms * 8);
    if (e == cudaSuccess) {
        if (elem_bytes == 4) kColumnMinMax<int><<<blocks, 256, 0, st>>>(static_cast<const int*>(column), n, d);
        else kColumnMinMax<long long><<<blocks, 256, 0, st>>>(static_cast<const long long*>(column), n, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, d, sizeof host, cudaMemcpyDeviceToHost, st);
    const cudaError_t f = cudaFreeAsync(d, st);
    if (e == cudaSuccess) e = f;
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        gpudb::setThreadError(std::string("column_minmax: ") + cudaGetErrorString(e));
        return GPUDB_E_CUDA;
    }
    *min_out = host[0];
    *max_out = host[1];
    return GPUDB_OK;
}

}  // extern "C"
