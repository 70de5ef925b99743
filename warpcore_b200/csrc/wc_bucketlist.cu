/*
 * wc_bucketlist.cu -- BucketListHashTable (the reference's
 * bucket_list_hash_table.cuh over BucketListStore, storage.cuh:651-1454):
 * kernels and the wc_blht_* C ABI.
 *
 * Layout: keys, handles (one 64-bit list handle per key slot) and the
 * value pool are three arrays; the reference keeps {key, handle} pairs and
 * a pool of value/header unions.  Every kernel runs one key per lane
 * (detail/bl_ops.cuh): the key's window, then its handle, then its list.
 */
#include <warpcore_b200.h>

#include "wc_internal.h"
#include "wc_compact.cuh"
#include <warpcore/detail/bl_ops.cuh>

#include <cstring>

using namespace warpcore::b200;

struct wc_blht {
    wc_table_config cfg{};
    uint64_t capacity = 0, num_buckets = 0, seed = 0;
    uint64_t value_capacity = 0, min_bucket = 1, max_bucket = 1, max_values = 1;
    float grow = 1.1f;
    uint32_t ib = 32, cb = 20, sb = 10;
    void *keys = nullptr;
    unsigned long long *handles = nullptr;
    unsigned long long *pool = nullptr;
    uint32_t *status = nullptr;             /* device Status word */
    unsigned long long *counters = nullptr; /* device: next free pool element, scratch */
    void *scan = nullptr;
    uint64_t scan_bytes = 0;
    bool initialized = false;
};

namespace {

#define BL_CUDA(call)                                                          \
    do {                                                                       \
        cudaError_t e_ = (call);                                               \
        if (e_ != cudaSuccess) return host_cuda_fail(e_, #call);               \
    } while (0)

constexpr int kBlock = 256;
constexpr unsigned kBlAuxBytes = 256; /* Status word at 0, counters from 64 on */

int bl_fail(int code, const char *msg) { return host_fail(code, msg); }

uint64_t kmask(uint32_t bytes) { return bytes == 4 ? 0xffffffffull : ~0ull; }

struct BlArgs : MultiArgs {
    BlView v;
};

/* bulk insert (:235-326).  Unlike the reference kernel, which leaves the
 * status of a key without a slot (invalid key, probing length exceeded)
 * unwritten, every key gets its status. */
template <class K, class V, int kW>
__global__ void __launch_bounds__(256, WC_MULTI_INSERT_BLOCKS) bl_insert_kernel(const BlArgs a)
{
    uint32_t join = 0;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < a.n; i += stride) {
        uint32_t j = 0;
        const uint32_t st = bl_insert_one<K, V, kW>(a.v, reinterpret_cast<const K *>(a.keys)[i],
                                                    reinterpret_cast<const V *>(a.values)[i],
                                                    a.max_windows, j);
        join |= j;
        multi_write_status(a, i, st);
    }
    const uint32_t wj = __reduce_or_sync(0xffffffffu, join); /* every lane arrives */
    if ((threadIdx.x & 31) == 0) join_status(a.v.t.status, wj);
}

/* Bulk insert (:235-326), as bl_insert_one, in two steps per block tile.  In
 * the first the lanes draw keys and find or claim their slots, one window
 * read or compare-and-swap per lane and step; a lane whose key is done takes
 * the next one, so no lane waits for the longest walk of its warp.  In the
 * second each thread appends to four lists at once: the handles, the newest
 * buckets' headers and the swaps of all four are in flight together, and
 * the lanes of a warp that grow their lists share one pool reservation
 * (which a loop of single steps per lane breaks up: 3330 us).  An append
 * that loses its swap goes on in bl_append.  24 M values, 8 per key, in
 * eight rounds: 1993 us with bl_insert_kernel, 1763 now; 16 M u64 values in
 * one batch, 8 per key: 1506 and 1010.  What is left is random reads and
 * compare-and-swaps outside L2. */
template <class K, class V, int kW>
__global__ void __launch_bounds__(kMultiThreads, WC_MULTI_INSERT_BLOCKS)
    bl_insert_tiles_kernel(const BlArgs a)
{
    constexpr int kPer = kMultiTile / kMultiThreads;
    constexpr uint64_t kDone = ~0ull;      /* no slot: the status is written */
    constexpr uint64_t kFound = 1ull << 63; /* the key was there */
    __shared__ K s_key[kMultiTile];
    __shared__ uint64_t s_slot[kMultiTile];
    __shared__ int s_drawn;
    const BlView &v = a.v;
    const TableView &t = v.t;
    const uint32_t W = kW ? uint32_t(kW) : t.cg_size;
    const K empty = K(t.empty_key), tomb = K(t.tombstone_key);
    K *const slots = reinterpret_cast<K *>(t.slots);
    const K *const keys_in = reinterpret_cast<const K *>(a.keys);
    const V *const vals_in = reinterpret_cast<const V *>(a.values);
    const uint64_t head = bl_head(v.ib);
    uint32_t join = 0;

    for (uint64_t base = uint64_t(blockIdx.x) * a.tile; base < a.n;
         base += uint64_t(gridDim.x) * a.tile) {
        const int m = int(a.n - base < a.tile ? a.n - base : a.tile);
        if (threadIdx.x == 0) s_drawn = 0;
        for (int i = threadIdx.x; i < m; i += kMultiThreads)
            s_key[i] = ld_stream(keys_in + base + uint64_t(i));
        __syncthreads();

        /* ---- the keys' slots ---- */
        {
            bool has = false, left = true;
            int at = 0;
            K key = K(0);
            uint64_t bucket = 0, step = 0, wins = 0;
            uint32_t free = 0; /* free slots still to be tried; 0: the window is due */
            for (;;) {
                if (draw_key(has, m, &s_drawn, left, at)) {
                    key = s_key[at];
                    if (key == empty || key == tomb) {
                        s_slot[at] = kDone;
                        join |= kStInvalidKey;
                        multi_write_status(a, base + uint64_t(at), kStInvalidKey);
                    } else {
                        has = true;
                        bucket = probe_begin<K>(t, key);
                        step = 0;
                        wins = 0;
                        free = 0;
                    }
                }
                if (!left && !__any_sync(0xffffffffu, has)) break;
                KeyWindow<K, kW> win;
                K old = empty;
                const int i = __ffs(free) - 1;
                if (has) {
                    if (free) old = mb_cas<K>(slots + bucket * W + uint64_t(i), empty, key);
                    else win.load(slots + bucket * W, W, key, empty);
                }
                if (!has) continue;
                uint64_t slot = kDone;
                if (free) {
                    if (old == empty) slot = bucket * W + uint64_t(i);
                    else if (old == key) slot = (bucket * W + uint64_t(i)) | kFound;
                    free &= free - 1u;
                } else {
                    const uint32_t hits = win.key_slots(key);
                    if (hits) slot = (bucket * W + uint64_t(__ffs(hits) - 1)) | kFound;
                    else free = win.free_slots(empty);
                }
                if (slot == kDone) {
                    if (free) continue;
                    if (++wins < a.max_windows) {
                        if (wins == 1) step = probe_step<K>(t, key);
                        bucket = probe_next(t, bucket, step);
                        continue;
                    }
                    join |= kStProbingLengthExceeded;
                    multi_write_status(a, base + uint64_t(at), kStProbingLengthExceeded);
                }
                s_slot[at] = slot;
                has = false;
            }
        }
        __syncthreads();

        /* ---- append, four lists per thread ---- */
        uint64_t slot[kPer];
        unsigned long long cur[kPer], want[kPer], old[kPer];
        uint64_t size[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int i = int(threadIdx.x) + j * kMultiThreads;
            slot[j] = i < m ? s_slot[i] : kDone;
            /* a new key's list is as init left it, unless an equal key's
             * append was faster (the swap finds out) */
            cur[j] = bl_pack(v, kBlUninit, head, 0, 0);
            if (slot[j] != kDone && (slot[j] & kFound))
                cur[j] = bl_load(v.handles + (slot[j] & ~kFound));
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const BlHandle c = bl_unpack(v, cur[j]);
            size[j] = v.min_bucket;
            if (slot[j] != kDone && c.state == kBlInit && c.count > v.min_bucket &&
                c.count < v.max_values)
                size[j] = bl_header_size(v, bl_load(v.pool + c.index));
        }
        /* the swap that takes a place or blocks the handle, where the list may
         * grow */
        bool tried[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const BlHandle c = bl_unpack(v, cur[j]);
            tried[j] = slot[j] != kDone && c.count < v.max_values &&
                       (c.state == kBlInit || c.state == kBlUninit);
            want[j] = c.state == kBlUninit ? bl_pack(v, kBlBlocking, head, 0, 0)
                      : c.tail == size[j]
                          ? bl_pack(v, kBlBlocking, c.index, c.count, c.tail)
                          : bl_pack(v, kBlInit, c.index, c.count + 1, c.tail + 1);
            old[j] = ~cur[j];
            if (tried[j]) old[j] = atomicCAS(v.handles + (slot[j] & ~kFound), cur[j], want[j]);
        }
        uint32_t ast[kPer];
        /* what the swaps won is finished for all four before any append that
         * lost one waits for another's list */
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            ast[j] = kStNone;
            if (!tried[j] || old[j] != cur[j]) continue;
            const int i = int(threadIdx.x) + j * kMultiThreads;
            const unsigned long long value = (unsigned long long)vals_in[base + uint64_t(i)];
            const BlHandle c = bl_unpack(v, cur[j]);
            if ((want[j] & 3u) == kBlInit) {
                v.pool[c.index + (c.count + 1 <= v.min_bucket ? c.tail : c.tail + 1)] = value;
                continue;
            }
            unsigned long long *const h = v.handles + (slot[j] & ~kFound);
            const bool first = c.state == kBlUninit; /* the first bucket has no header */
            uint64_t grow = v.min_bucket;
            if (!first) {
                const float grown = ceilf(float(size[j]) * v.grow);
                const float cap = float(v.max_bucket);
                grow = uint64_t(cap < grown ? cap : grown);
            }
            const uint64_t need = grow + (first ? 0 : 1);
            const unsigned long long alloc = bl_alloc(v, need);
            if (alloc + need <= v.capacity) {
                if (!first) v.pool[alloc] = bl_header(v, c.index, grow);
                v.pool[alloc + (first ? 0 : 1)] = value;
                __threadfence();
                atomicExch(h, bl_pack(v, kBlInit, alloc, c.count + 1, 1));
            } else {
                atomicExch(h, bl_pack(v, kBlFull, first ? head : c.index, c.count, c.tail));
                ast[j] = kStOutOfMemory;
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (slot[j] == kDone) continue;
            const int i = int(threadIdx.x) + j * kMultiThreads;
            if (!tried[j] || old[j] != cur[j]) {
                if (bl_unpack(v, cur[j]).count >= v.max_values) ast[j] = kStMaxValuesReached;
                else ast[j] = bl_append<V>(v, v.handles + (slot[j] & ~kFound),
                                           vals_in[base + uint64_t(i)],
                                           tried[j] ? old[j] : cur[j]);
            }
            const uint32_t st = ((slot[j] & kFound) ? kStDuplicateKey : kStNone) | ast[j];
            join |= st;
            multi_write_status(a, base + uint64_t(i), st);
        }
        __syncthreads(); /* the shared rows are rewritten by the next tile */
    }
    const uint32_t wj = __reduce_or_sync(0xffffffffu, join); /* every lane arrives */
    if ((threadIdx.x & 31) == 0) join_status(a.v.t.status, wj);
}

/* the key's slot (as bl_find looks for it), then its handle, which holds the
 * list's count, then for the values the list's buckets, newest first (as
 * bl_walk reads them): a bucket's header and its first four values are read
 * together, so a list costs one memory latency per bucket */
template <class K, class V, int kW>
struct BlWalk {
    using key_t = K;
    using val_t = V;
    using Args = BlArgs;
    static constexpr int kFindTile = multi_find_tile(sizeof(K), kW * int(sizeof(K)));
    struct State {
        uint64_t bucket, step, wins, num;
        uint64_t at;    /* the key's slot, then the list bucket's pool index */
        uint64_t count; /* list: values in all; num: values read */
        uint64_t size, read; /* list: values in the bucket (phase 3: at most), read of it */
        int phase;      /* 0 windows, 1 handle, 2 list, 3 list, size still in the header */
    };

    static __device__ __forceinline__ const TableView &view(const Args &a) { return a.v.t; }

    static __device__ __forceinline__ void start(const Args &a, K key, State &s)
    {
        s.bucket = probe_begin<K>(a.v.t, key);
        s.step = 0;
        s.wins = 0;
        s.num = 0;
        s.phase = 0;
    }

    static __device__ __forceinline__ bool count_step(const Args &a, K key, State &s, uint32_t &st)
    {
        if (s.phase == 0) return window(a, key, s, st);
        s.num = bl_unpack(a.v, a.v.handles[s.at]).count;
        st = kStNone;
        return true;
    }

    static __device__ __forceinline__ bool value_step(const Args &a, K key, State &s, V *out,
                                                      uint64_t room)
    {
        const BlView &v = a.v;
        if (s.phase == 0) {
            uint32_t st;
            return window(a, key, s, st);
        }
        if (s.phase == 1) {
            const BlHandle c = bl_unpack(v, v.handles[s.at]);
            if (c.state != kBlInit || c.index == bl_head(v.ib)) return true;
            s.at = c.index;
            s.count = c.count;
            s.size = c.tail;
            s.read = 0;
            s.phase = 2;
            return s.at >= v.capacity ||
                   s.at + (c.count <= v.min_bucket ? 0 : 1) + c.tail > v.capacity;
        }
        /* the list's first bucket (the last one read) has no header; an
         * older bucket is no larger than a newer one, so no value is read
         * that lies beyond what the bucket may hold */
        const bool last = s.count - s.num + s.read <= v.min_bucket;
        const uint64_t first = s.at + (last ? 0 : 1);
        if (last && s.phase == 3) s.size = v.min_bucket;
        unsigned long long x[4];
        const unsigned long long header = v.pool[s.at];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t p = first + s.read + uint64_t(u);
            x[u] = s.read + uint64_t(u) < s.size && p < v.capacity ? v.pool[p] : 0ull;
        }
        if (s.phase == 3) {
            if (!last) s.size = bl_header_size(v, header);
            s.phase = 2;
            if (first + s.size > v.capacity) return true;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (s.read < s.size && s.num < s.count) {
                if (s.num < room) out[s.num] = V(x[u]);
                ++s.num;
                ++s.read;
            }
        }
        if (s.num >= s.count) return true;
        if (s.read >= s.size) {
            s.size = bl_header_size(v, header);
            s.at = bl_header_prev(v, header);
            s.read = 0;
            s.phase = 3;
            return s.at >= v.capacity;
        }
        return false;
    }

    static __device__ __forceinline__ bool window(const Args &a, K key, State &s, uint32_t &st)
    {
        const TableView &t = a.v.t;
        const uint32_t W = kW ? uint32_t(kW) : t.cg_size;
        KeyWindow<K, kW> win;
        win.load(reinterpret_cast<const K *>(t.slots) + s.bucket * W, W, key, K(t.empty_key));
        const uint32_t hits = win.key_slots(key);
        const bool free = win.any_free(K(t.empty_key));
        if (hits) {
            s.at = s.bucket * W + uint64_t(__ffs(hits) - 1);
            s.phase = 1;
            return false;
        }
        if (free) {
            st = kStKeyNotFound;
            return true;
        }
        if (++s.wins >= a.max_windows) {
            st = kStProbingLengthExceeded;
            return true;
        }
        if (s.wins == 1) s.step = probe_step<K>(t, key);
        s.bucket = probe_next(t, s.bucket, s.step);
        return false;
    }
};

/* init: keys empty, handles uninitialized, pool headers {head, min}, Status and
 * counters 0 */
template <class K>
__global__ void __launch_bounds__(256) bl_init_kernel(const BlView v, uint64_t capacity)
{
    const unsigned long long u = bl_pack(v, kBlUninit, bl_head(v.ib), 0, 0);
    const unsigned long long hdr = bl_header(v, bl_head(v.ib), v.min_bucket);
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t tid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    for (uint64_t i = tid; i < capacity; i += stride) {
        reinterpret_cast<K *>(v.t.slots)[i] = K(v.t.empty_key);
        v.handles[i] = u;
    }
    for (uint64_t i = tid; i < v.capacity; i += stride) v.pool[i] = hdr;
    /* the table's small device block: the Status word and the counters */
    if (blockIdx.x == 0 && threadIdx.x < kBlAuxBytes / 4) v.t.status[threadIdx.x] = 0;
}

/* num_keys (valid keys), num_values (sum of list counts) and the keys,
 * compacted by block tiles (wc_compact.cuh) */
template <class K>
__global__ void __launch_bounds__(256) bl_scan_keys_kernel(const BlView v, uint64_t capacity,
                                                           void *keys_out,
                                                           unsigned long long *num_keys,
                                                           unsigned long long *num_values)
{
    const K empty = K(v.t.empty_key), tomb = K(v.t.tombstone_key);
    const K *const keys = reinterpret_cast<const K *>(v.t.slots);
    unsigned long long vals = 0;
    compact_tiles<K, K>(capacity, reinterpret_cast<K *>(keys_out), nullptr, num_keys,
                        [&](uint64_t i, K &k, K &) {
                            k = keys[i];
                            if (k == empty || k == tomb) return false;
                            vals += bl_unpack(v, v.handles[i]).count;
                            return true;
                        });
    vals = warp_sum_u64(vals);
    if ((threadIdx.x & 31) == 0 && vals) atomicAdd(num_values, vals);
}

struct BlKernels {
    uint32_t find_tile;
    const void *insert, *insert_tiles, *count, *offsets, *values, *init, *scan;
};

template <class K, class V, int kW>
BlKernels bl_kernels_of()
{
    return {BlWalk<K, V, kW>::kFindTile,
            reinterpret_cast<const void *>(bl_insert_kernel<K, V, kW>),
            reinterpret_cast<const void *>(bl_insert_tiles_kernel<K, V, kW>),
            reinterpret_cast<const void *>(multi_find_kernel<BlWalk<K, V, kW>, false>),
            reinterpret_cast<const void *>(multi_find_kernel<BlWalk<K, V, kW>, true>),
            reinterpret_cast<const void *>(multi_values_kernel<BlWalk<K, V, kW>>),
            reinterpret_cast<const void *>(bl_init_kernel<K>),
            reinterpret_cast<const void *>(bl_scan_keys_kernel<K>)};
}

template <class K, class V>
BlKernels bl_kernels_kv(uint32_t cg)
{
    return cg == 8 ? bl_kernels_of<K, V, 8>() : bl_kernels_of<K, V, 0>();
}

BlKernels bl_kernels(const wc_blht *t)
{
    using U32 = unsigned int;
    using U64 = unsigned long long;
    const uint32_t cg = t->cfg.cg_size;
    if (t->cfg.key_bytes == 4)
        return t->cfg.value_bytes == 4 ? bl_kernels_kv<U32, U32>(cg) : bl_kernels_kv<U32, U64>(cg);
    return t->cfg.value_bytes == 4 ? bl_kernels_kv<U64, U32>(cg) : bl_kernels_kv<U64, U64>(cg);
}

BlView view_of(const wc_blht *t)
{
    BlView v{};
    TableView &tv = v.t;
    tv.slots = t->keys;
    tv.status = t->status;
    tv.fps = nullptr;
    tv.num_buckets = t->num_buckets;
    tv.seed = t->seed;
    tv.empty_key = t->cfg.empty_key;
    tv.tombstone_key = t->cfg.tombstone_key;
    tv.max_count = ~0ull;
    tv.magic_nb = barrett_magic(t->num_buckets);
    tv.magic_nb1 = barrett_magic(t->num_buckets > 1 ? t->num_buckets - 1 : 1);
    tv.probing = t->cfg.probing;
    tv.hasher1 = t->cfg.hasher1;
    tv.hasher2 = t->cfg.hasher2;
    tv.cg_size = t->cfg.cg_size;
    v.handles = t->handles;
    v.pool = t->pool;
    v.next_free = t->counters;
    v.capacity = t->value_capacity;
    v.min_bucket = t->min_bucket;
    v.max_bucket = t->max_bucket;
    v.max_values = t->max_values;
    v.grow = t->grow;
    v.ib = t->ib;
    v.cb = t->cb;
    v.sb = t->sb;
    return v;
}

int check(const wc_blht *t)
{
    if (!t) return bl_fail(WC_ERR_INVALID_ARGUMENT, "table is NULL");
    if (!t->initialized) return bl_fail(WC_ERR_NOT_INITIALIZED, "table is not initialized");
    return WC_OK;
}

BlArgs args_of(const wc_blht *t, const void *keys, uint64_t n, uint64_t probing_length,
               void *status_out, int handler, uint32_t ignore)
{
    BlArgs a{};
    a.v = view_of(t);
    a.keys = keys;
    a.n = n;
    a.max_windows = max_windows(probing_length, t->cfg.cg_size, t->num_buckets);
    a.status_out = handler == WC_HANDLER_NOTHING ? nullptr : status_out;
    a.handler = handler;
    a.bool_mask = (~ignore) ^ 0xFFFu;
    return a;
}

int launch(const void *k, uint64_t items, BlArgs &a, cudaStream_t s)
{
    void *args[] = {&a};
    BL_CUDA(cudaLaunchKernel(k, dim3(host_grid(k, kBlock, items, kBlock)), dim3(kBlock), args, 0, s));
    note_launches(1);
    return WC_OK;
}

int read_counter(const unsigned long long *d, cudaStream_t s, uint64_t *out)
{
    return host_read_counter(d, s, out);
}

int count(wc_blht *t, const void *keys, uint64_t n, uint64_t *counts_dev, uint64_t *total,
          cudaStream_t s, uint64_t probing_length, void *status_out, int handler, uint32_t ignore)
{
    BlArgs a = args_of(t, keys, n, probing_length, status_out, handler, ignore);
    const BlKernels k = bl_kernels(t);
    return host_multi_count(k.count, k.find_tile, &a, &a, t->counters + 8, counts_dev, total, s);
}

int join_host(wc_blht *t, uint32_t bits, cudaStream_t s)
{
    return host_join_status(t->status, bits, s);
}

/* valid keys (into keys_out if not NULL) and the sum of their list counts */
int scan_keys(wc_blht *t, void *keys_out, uint64_t *num_keys, uint64_t *num_values,
              cudaStream_t s)
{
    unsigned long long *nk = t->counters + 2, *nv = t->counters + 3;
    BL_CUDA(cudaMemsetAsync(nk, 0, 2 * sizeof(unsigned long long), s));
    BlView v = view_of(t);
    uint64_t cap = t->capacity;
    const void *k = bl_kernels(t).scan;
    void *args[] = {&v, &cap, &keys_out, &nk, &nv};
    BL_CUDA(cudaLaunchKernel(k, dim3(host_grid(k, kBlock, cap, kBlock)), dim3(kBlock), args, 0, s));
    note_launches(1);
    unsigned long long h[2] = {0, 0};
    BL_CUDA(cudaMemcpyAsync(h, nk, sizeof(h), cudaMemcpyDeviceToHost, s));
    BL_CUDA(cudaStreamSynchronize(s));
    if (num_keys) *num_keys = h[0];
    if (num_values) *num_values = h[1];
    return WC_OK;
}

} // namespace

extern "C" {

int wc_blht_create(const wc_table_config *cfg, uint64_t key_capacity, uint64_t value_capacity,
                   uint64_t seed, float grow_factor, uint64_t min_bucket_size,
                   uint64_t max_bucket_size, uint64_t max_values_per_key, uint32_t index_bits,
                   uint32_t counter_bits, uint32_t size_bits, int no_init, wc_blht **out)
{
    if (!out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (!cfg) return bl_fail(WC_ERR_INVALID_ARGUMENT, "config is NULL");
    if (cfg->key_bytes != 4 && cfg->key_bytes != 8)
        return bl_fail(WC_ERR_UNSUPPORTED, "key_bytes must be 4 or 8");
    if (cfg->value_bytes != 4 && cfg->value_bytes != 8)
        return bl_fail(WC_ERR_UNSUPPORTED, "value_bytes must be 4 or 8");
    const uint32_t cg = cfg->cg_size;
    if (!(cg == 1 || cg == 2 || cg == 4 || cg == 8 || cg == 16 || cg == 32))
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "cg_size must be 1, 2, 4, 8, 16 or 32");
    if (cfg->probing > WC_PROBING_QUADRATIC || cfg->hasher1 > WC_HASH_IDENTITY64 ||
        cfg->hasher2 > WC_HASH_IDENTITY64)
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "unknown probing scheme or hasher");
    const uint64_t km = kmask(cfg->key_bytes);
    if ((cfg->empty_key & km) == (cfg->tombstone_key & km))
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "empty key and tombstone key must differ");
    if (index_bits == 0 || counter_bits == 0 || size_bits == 0 ||
        uint64_t(index_bits) + counter_bits + size_bits + 2 > 64 || index_bits + size_bits > 64)
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "bit widths must be positive and fit in 62 bits");
    /* the store's configuration check (storage.cuh:990-1014) */
    const uint64_t head = (1ull << index_bits) - 1, max_size = (1ull << size_bits) - 1;
    if (!(value_capacity < head && grow_factor >= 1.0f && min_bucket_size >= 1 &&
          max_bucket_size >= min_bucket_size && max_bucket_size <= max_size))
        return bl_fail(WC_ERR_INVALID_ARGUMENT,
                       "invalid bucket list configuration (value capacity, grow factor, bucket sizes)");
    const uint64_t cap = host_valid_capacity(key_capacity, cg);
    if (cap == 0) return bl_fail(WC_ERR_INVALID_ARGUMENT, "key_capacity exceeds the largest capacity");
    auto *t = new wc_blht();
    t->cfg = *cfg;
    t->cfg.empty_key &= km;
    t->cfg.tombstone_key &= km;
    t->capacity = cap;
    t->num_buckets = cap / cg;
    t->seed = seed & km;
    t->value_capacity = value_capacity;
    t->grow = grow_factor;
    t->min_bucket = min_bucket_size;
    t->max_bucket = max_bucket_size;
    const uint64_t max_count = (1ull << counter_bits) - 1;
    t->max_values = max_values_per_key < max_count ? max_values_per_key : max_count;
    t->ib = index_bits;
    t->cb = counter_bits;
    t->sb = size_bits;
    const uint64_t kbytes = (cap * cfg->key_bytes + 255) & ~uint64_t(255);
    const uint64_t hbytes = cap * 8;
    const uint64_t pbytes = (value_capacity ? value_capacity : 1) * 8;
    void *mem = nullptr;
    cudaError_t e = cudaMalloc(&mem, kbytes + hbytes + pbytes);
    if (e == cudaSuccess) e = cudaMalloc(&t->status, kBlAuxBytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (mem) cudaFree(mem);
        delete t;
        return host_cuda_fail(e, "cudaMalloc (bucket list table)");
    }
    t->keys = mem;
    t->handles = reinterpret_cast<unsigned long long *>(static_cast<char *>(mem) + kbytes);
    t->pool = reinterpret_cast<unsigned long long *>(static_cast<char *>(mem) + kbytes + hbytes);
    t->counters = reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(t->status) + 64);
    *out = t;
    if (!no_init) {
        const int rc = wc_blht_init(t, t->seed, nullptr);
        if (rc) {
            wc_blht_destroy(t);
            *out = nullptr;
            return rc;
        }
    }
    return WC_OK;
}

int wc_blht_destroy(wc_blht *t)
{
    if (!t) return WC_OK;
    if (t->keys) cudaFree(t->keys);
    if (t->status) cudaFree(t->status);
    if (t->scan) cudaFree(t->scan);
    delete t;
    return WC_OK;
}

int wc_blht_init(wc_blht *t, uint64_t seed, wc_stream_t stream)
{
    if (!t) return bl_fail(WC_ERR_INVALID_ARGUMENT, "table is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    t->seed = seed & kmask(t->cfg.key_bytes);
    BlView v = view_of(t);
    uint64_t cap = t->capacity;
    const void *k = bl_kernels(t).init;
    const uint64_t items = cap > t->value_capacity ? cap : t->value_capacity;
    void *args[] = {&v, &cap};
    BL_CUDA(cudaLaunchKernel(k, dim3(host_grid(k, kBlock, items, kBlock)), dim3(kBlock), args, 0, s));
    note_launches(1);
    BL_CUDA(cudaStreamSynchronize(s));
    t->initialized = true;
    return WC_OK;
}

int wc_blht_insert(wc_blht *t, const void *keys_in, const void *values_in, uint64_t num_in,
                   wc_stream_t stream, uint64_t probing_length, void *status_out,
                   int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (status_handler < WC_HANDLER_NOTHING || status_handler > WC_HANDLER_BOOLEAN)
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "unknown status handler");
    if (num_in == 0) return WC_OK;
    if (!keys_in || !values_in) return bl_fail(WC_ERR_INVALID_ARGUMENT, "keys_in / values_in is NULL");
    BlArgs a = args_of(t, keys_in, num_in, probing_length, status_out, status_handler, ignore);
    a.values = values_in;
    const BlKernels k = bl_kernels(t);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    /* Where every resident lane gets at most one key, no lane has a second
     * one to draw, and the kernel without tiles is the faster one; else the
     * tiles (u32 pairs, per round of 50 000 / 100 000 / 200 000 / 1 M new
     * values: 11.7 / 12.5 / 21.9 / 80.2 us without, 12.1 / 12.4 / 19.1 /
     * 63.8 with them). */
    if (num_in <= uint64_t(host_grid(k.insert, kBlock, num_in, kBlock)) * kBlock)
        return launch(k.insert, num_in, a, s);
    return host_multi_launch(k.insert_tiles, &a, &a, s);
}

int wc_blht_num_values(wc_blht *t, const void *keys_in, uint64_t num_in, uint64_t *num_out,
                       uint64_t *num_per_key_out, wc_stream_t stream, uint64_t probing_length,
                       void *status_out, int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    *num_out = 0;
    if (num_in == 0) return WC_OK;
    if (!keys_in) return bl_fail(WC_ERR_INVALID_ARGUMENT, "keys_in is NULL");
    return count(t, keys_in, num_in, num_per_key_out, num_out,
                 reinterpret_cast<cudaStream_t>(stream), probing_length, status_out,
                 status_handler, ignore);
}

int wc_blht_retrieve(wc_blht *t, const void *keys_in, uint64_t num_in,
                     uint64_t *begin_offsets_out, uint64_t *end_offsets_out, void *values_out,
                     uint64_t *num_out, wc_stream_t stream, uint64_t probing_length,
                     void *status_out, int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    *num_out = 0;
    if (num_in == 0) return WC_OK;
    if (!keys_in || !end_offsets_out || (values_out && !begin_offsets_out))
        return bl_fail(WC_ERR_INVALID_ARGUMENT, "NULL buffer");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!values_out) {
        rc = count(t, keys_in, num_in, end_offsets_out, num_out, s, probing_length, nullptr,
                   WC_HANDLER_NOTHING, ignore);
        if (rc) return rc;
        rc = host_dry_run_status(status_out, num_in, status_handler, ignore, s);
        if (rc) return rc;
        return join_host(t, kStDryRun, s);
    }
    BlArgs a = args_of(t, keys_in, num_in, probing_length, status_out, status_handler, ignore);
    const BlKernels k = bl_kernels(t);
    return host_multi_retrieve(k.offsets, k.find_tile, k.values, &a, &a, &t->scan, &t->scan_bytes,
                               begin_offsets_out, end_offsets_out, values_out, num_out, s);
}

int wc_blht_retrieve_all_keys(wc_blht *t, void *keys_out, uint64_t *num_out, wc_stream_t stream)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    return scan_keys(t, keys_out, num_out, nullptr, reinterpret_cast<cudaStream_t>(stream));
}

int wc_blht_num_keys(wc_blht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    return scan_keys(t, nullptr, out, nullptr, reinterpret_cast<cudaStream_t>(stream));
}

int wc_blht_total_values(wc_blht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    return scan_keys(t, nullptr, nullptr, out, reinterpret_cast<cudaStream_t>(stream));
}

int wc_blht_pool_used(wc_blht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    return read_counter(t->counters, reinterpret_cast<cudaStream_t>(stream), out);
}

int wc_blht_peek_status(wc_blht *t, wc_stream_t stream, uint32_t *out)
{
    if (!t || !out) return bl_fail(WC_ERR_INVALID_ARGUMENT, "NULL argument");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    BL_CUDA(cudaMemcpyAsync(out, t->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    BL_CUDA(cudaStreamSynchronize(s));
    return WC_OK;
}

int wc_blht_pop_status(wc_blht *t, wc_stream_t stream, uint32_t *out)
{
    int rc = wc_blht_peek_status(t, stream, out);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    BL_CUDA(cudaMemsetAsync(t->status, 0, sizeof(uint32_t), s));
    BL_CUDA(cudaStreamSynchronize(s));
    return WC_OK;
}

int wc_blht_get_info(const wc_blht *t, wc_blht_info *info)
{
    if (!t || !info) return bl_fail(WC_ERR_INVALID_ARGUMENT, "NULL argument");
    std::memset(info, 0, sizeof(*info));
    info->key_bytes = t->cfg.key_bytes;
    info->value_bytes = t->cfg.value_bytes;
    info->cg_size = t->cfg.cg_size;
    info->probing = t->cfg.probing;
    info->hasher1 = t->cfg.hasher1;
    info->hasher2 = t->cfg.hasher2;
    info->index_bits = t->ib;
    info->counter_bits = t->cb;
    info->size_bits = t->sb;
    info->grow_factor = t->grow;
    info->key_capacity = t->capacity;
    info->value_capacity = t->value_capacity;
    info->num_buckets = t->num_buckets;
    info->seed = t->seed;
    info->empty_key = t->cfg.empty_key;
    info->tombstone_key = t->cfg.tombstone_key;
    info->min_bucket_size = t->min_bucket;
    info->max_bucket_size = t->max_bucket;
    info->max_values_per_key = t->max_values;
    info->bytes_total = t->capacity * (t->cfg.key_bytes + 8) + t->value_capacity * 8 + 8;
    info->keys = t->keys;
    info->handles = t->handles;
    info->pool = t->pool;
    info->next_free = t->counters;
    info->status = t->status;
    info->is_initialized = t->initialized ? 1 : 0;
    return WC_OK;
}

} // extern "C"
