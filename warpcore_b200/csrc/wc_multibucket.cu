/*
 * wc_multibucket.cu -- MultiBucketHashTable (the reference's
 * multi_bucket_hash_table.cuh): kernels and the wc_mbht_* C ABI.
 *
 * Layout: the key array (capacity keys, bucket-aligned probe windows of
 * cg_size keys) and the bucket array (capacity x bucket values) are
 * separate; the reference keeps {key, value[bucket]} structures (AoSStore).
 * A probe window then costs cg_size keys (32 bytes for u32 at CG 8) whatever
 * the bucket size, and a key's values are read only where the key is.
 * Every kernel runs one key per lane (detail/mb_ops.cuh).
 */
#include <warpcore_b200.h>

#include "wc_internal.h"
#include "wc_compact.cuh"
#include <warpcore/detail/mb_ops.cuh>

#include <cstdio>
#include <cstring>

using namespace warpcore::b200;

struct wc_mbht {
    wc_table_config cfg{};
    uint32_t bucket = 1;
    uint64_t empty_value = 0;
    uint64_t capacity = 0, num_buckets = 0, seed = 0, max_values = ~0ull;
    void *keys = nullptr;
    void *vals = nullptr;
    uint32_t *status = nullptr;           /* device Status word */
    unsigned long long *counters = nullptr; /* device: num_keys, num_occupied, scratch */
    void *scan = nullptr;                 /* tiles of a retrieve, grown on demand */
    uint64_t scan_bytes = 0;
    bool initialized = false;
};

namespace {

#define MB_CUDA(call)                                                          \
    do {                                                                       \
        cudaError_t e_ = (call);                                               \
        if (e_ != cudaSuccess) return host_cuda_fail(e_, #call);               \
    } while (0)

constexpr int kBlock = 256;

int mb_fail(int code, const char *msg) { return host_fail(code, msg); }

uint64_t kmask(uint32_t bytes) { return bytes == 4 ? 0xffffffffull : ~0ull; }

struct MbArgs : MultiArgs {
    MbView m;
};

/* warp sums of two counters and the joined status, one atomic each per warp */
__device__ __forceinline__ void mb_flush(const MbView &m, uint32_t join, unsigned claimed,
                                         unsigned fresh)
{
    const uint32_t wj = __reduce_or_sync(0xffffffffu, join);
    const unsigned c = __reduce_add_sync(0xffffffffu, claimed);
    const unsigned f = __reduce_add_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0) {
        if (c) atomicAdd(m.num_occupied, (unsigned long long)c);
        if (f) atomicAdd(m.num_keys, (unsigned long long)f);
        join_status(m.t.status, wj);
    }
}

template <class K, class V, int kW, int kB>
__global__ void __launch_bounds__(256, WC_MULTI_INSERT_BLOCKS) mb_insert_kernel(const MbArgs a)
{
    uint32_t join = 0;
    unsigned claimed = 0, fresh = 0;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < a.n; i += stride) {
        bool c = false, f = false;
        const uint32_t st = mb_insert_one<K, V, kW, kB>(a.m, reinterpret_cast<const K *>(a.keys)[i],
                                                reinterpret_cast<const V *>(a.values)[i],
                                                a.max_windows, c, f);
        /* every status but a stored value's none / duplicate_key is joined */
        if (st != kStNone && st != kStDuplicateKey) join |= st;
        claimed += c;
        fresh += f;
        multi_write_status(a, i, st);
    }
    mb_flush(a.m, join, claimed, fresh); /* every lane arrives (no early exit) */
}

/* Bulk insert, as mb_insert_one, with buckets of two values or more.  A
 * warp's lanes walk the windows of its range of keys, one window per lane
 * and step, up to the first with a free slot, and put what they found into
 * a queue of the warp; a lane whose key is walked takes the next one, so no
 * lane waits for the longest walk.  Whenever 32 keys are queued, the warp
 * does for all of them what is left: read the key's last bucket, then swap
 * the value into a free place of it or claim the free slot.  A key that
 * loses its swap is inserted from the start by mb_insert_one.
 *
 * With one key per lane for the whole insert (mb_insert_kernel), the warp
 * waited for the longest of 32 walks and then for every other step.  2^25 u32
 * values, 8 per key in buckets of 4, in eight rounds 2036 -> 1836 us; 16 M u32
 * values of u64 keys in buckets of 8 865 -> 719; 10 M u64 in buckets of 2 758
 * -> 730, in one batch 886 -> 733.  Buckets of one value have no last bucket to
 * read and keep mb_insert_kernel (6 M u64 values of u32 keys 272 us, 313 here).
 * Tried as well: the two steps per block tile, four keys per thread in the
 * second (1991 us, in one batch slower), and every step of an insert in one
 * loop (2230). */
constexpr int kMbQueue = 64; /* keys a warp's queue holds */

template <class K, class V, int kW, int kB>
__global__ void __launch_bounds__(256, WC_MULTI_INSERT_BLOCKS)
    mb_insert_queue_kernel(const MbArgs a)
{
    /* slots that stand for: values up to max_values_per_key already (by
     * slots); windows used up; and for no last slot */
    constexpr uint64_t kCapped = ~0ull, kLength = ~1ull, kNone = ~0ull;
    __shared__ uint64_t s_last[8][kMbQueue], s_slot[8][kMbQueue];
    __shared__ uint32_t s_num[8][kMbQueue], s_at[8][kMbQueue];
    const MbView &mv = a.m;
    const TableView &t = mv.t;
    const uint32_t W = mb_w<kW>(mv), B = mb_b<kB>(mv);
    const K empty = K(t.empty_key), tomb = K(t.tombstone_key);
    const V ev = V(mv.empty_value);
    K *const slots = reinterpret_cast<K *>(t.slots);
    V *const places = reinterpret_cast<V *>(mv.vals);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    const uint32_t m = uint32_t(wb + per < a.n ? per : a.n - wb);
    const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;
    const V *const vals = reinterpret_cast<const V *>(a.values) + wb;

    uint32_t join = 0;
    unsigned claimed = 0, fresh = 0;
    int queued = 0;

    /* every status but a stored value's none / duplicate_key is joined */
    auto finish = [&](uint32_t i, uint32_t st) {
        if (st != kStNone && st != kStDuplicateKey) join |= st;
        multi_write_status(a, wb + i, st);
    };

    /* the last `take` queued keys, one per lane */
    auto place = [&](int take) {
        queued -= take;
        const bool in = lane < take;
        const int q = queued + lane;
        enum : int { kOver, kPlace, kClaim, kAgain };
        int todo = kOver;
        uint64_t slot = 0, last = kNone;
        uint32_t num = 0, at = 0, e = 0, st = kStNone;
        K key = K(0), old_key = K(0);
        V value = V(0), old_value = V(0);
        if (in) {
            slot = s_slot[wib][q];
            last = s_last[wib][q];
            num = s_num[wib][q];
            at = s_at[wib][q];
            key = keys[at];
            value = vals[at];
            if (B > 1 && last != kNone)
                e = mb_bucket_empties<V, kB>(places + last * B, B, ev, nullptr) & ~1u;
        }
        __syncwarp();
        if (in) {
            todo = kClaim;
            if (num == 0xffffffffu) {
                todo = kAgain; /* not counted exactly */
            } else if (B > 1 && last != kNone) {
                /* insert_into_bucket (:262-330): place 0 counts as full */
                const uint64_t before = uint64_t(num) - uint64_t(__popc(e));
                if (before >= mv.max_values) {
                    st = kStDuplicateKey | kStMaxValuesReached;
                    todo = kOver;
                } else if (e) {
                    st = before > 0 ? kStDuplicateKey : kStNone;
                    todo = kPlace;
                } else if (slot == kCapped) {
                    st = kStUnknownError;
                    todo = kOver;
                } else if (slot == kLength) {
                    st = kStProbingLengthExceeded | (num > 0 ? kStDuplicateKey : kStNone);
                    todo = kOver;
                }
            }
            if (todo == kPlace)
                old_value = mb_cas<V>(places + last * B + (__ffs(e) - 1), ev, value);
            else if (todo == kClaim)
                old_key = mb_cas<K>(slots + slot, empty, key);
        }
        if (todo == kPlace && old_value != ev) todo = kAgain;
        if (todo == kClaim) {
            if (old_key == empty) {
                /* the bucket's first place, after the key (:446-449) */
                places[slot * B] = value;
                ++claimed;
                fresh += num == 0;
                st = num == 0 ? kStNone : kStDuplicateKey;
            } else {
                todo = kAgain;
            }
        }
        if (todo == kAgain) {
            bool c = false, f = false;
            st = mb_insert_one<K, V, kW, kB>(mv, key, value, a.max_windows, c, f);
            claimed += c;
            fresh += f;
        }
        if (in) finish(at, st);
        __syncwarp();
    };

    uint32_t pf_base = 0, cursor = 0;
    K pfA = uint32_t(lane) < m ? ld_stream(keys + lane) : empty;
    K pfB = 32 + uint32_t(lane) < m ? ld_stream(keys + 32 + lane) : empty;
    bool has = false;
    uint32_t at = 0;
    K key = K(0);
    uint64_t bucket = 0, step = 0, wins = 0, num = 0, last = kNone;
    for (;;) {
        /* ---- lanes without a key take the next ones, in input order ---- */
        const unsigned need = __ballot_sync(0xffffffffu, !has);
        const uint32_t idle = uint32_t(__popc(need)), avail = m - cursor;
        const uint32_t take = idle < avail ? idle : avail;
        if (take == 0 && need == 0xffffffffu) break;
        if (take) {
            const uint32_t r = uint32_t(__popc(need & lanemask_lt));
            const uint32_t off = cursor - pf_base + r;
            const K ka = shfl_any(pfA, int(off & 31u)), kb = shfl_any(pfB, int(off & 31u));
            if (!has && r < take) {
                key = off < 32 ? ka : kb;
                at = cursor + r;
                const uint32_t st = key == empty || key == tomb ? kStInvalidKey
                                    : ld_stream(vals + at) == ev ? kStInvalidValue : kStNone;
                if (st != kStNone) {
                    finish(at, st);
                } else {
                    has = true;
                    bucket = probe_begin<K>(t, key);
                    step = 0;
                    wins = 0;
                    num = 0;
                    last = kNone;
                }
            }
            cursor += take;
            if (cursor - pf_base >= 32) {
                pf_base += 32;
                pfA = pfB;
                const uint32_t nx = pf_base + 32 + uint32_t(lane);
                if (nx < m) pfB = ld_stream(keys + nx);
            }
        }

        /* ---- one window per lane ---- */
        uint64_t slot = 0;
        bool walked = false;
        if (has) {
            KeyWindow<K, kW> win;
            win.load(slots + bucket * W, W, key, empty);
            const uint32_t hits = win.key_slots(key), free = win.free_slots(empty);
            if (hits) {
                last = bucket * W + uint64_t(31 - __clz(hits));
                num += uint64_t(B) * uint64_t(__popc(hits));
            }
            if (num >= mv.max_values) {
                has = false;
                walked = B > 1 && last != kNone;
                slot = kCapped;
                if (!walked) finish(at, kStDuplicateKey | kStMaxValuesReached);
            } else if (free) {
                has = false;
                walked = true;
                slot = bucket * W + uint64_t(__ffs(free) - 1);
            } else if (++wins >= a.max_windows) {
                has = false;
                walked = B > 1 && last != kNone;
                slot = kLength;
                if (!walked)
                    finish(at, kStProbingLengthExceeded | (num > 0 ? kStDuplicateKey : kStNone));
            } else {
                if (wins == 1) step = probe_step<K>(t, key);
                bucket = probe_next(t, bucket, step);
            }
        }
        const unsigned done = __ballot_sync(0xffffffffu, walked);
        if (walked) {
            const int q = queued + __popc(done & lanemask_lt);
            s_slot[wib][q] = slot;
            s_last[wib][q] = last;
            s_num[wib][q] = num < 0xffffffffull ? uint32_t(num) : 0xffffffffu;
            s_at[wib][q] = at;
        }
        queued += __popc(done);
        __syncwarp();
        if (queued >= 32) place(32);
    }
    if (queued) place(queued);
    mb_flush(a.m, join, claimed, fresh);
}

/* the key's slots window by window, as mb_for_each_one walks them: a window
 * is one memory operation; then one bucket each: the last one of the window
 * for the count (its free places are what the count needs), every one for
 * the values */
template <class K, class V, int kW, int kB>
struct MbWalk {
    using key_t = K;
    using val_t = V;
    using Args = MbArgs;
    static constexpr int kFindTile = multi_find_tile(sizeof(K), kW * int(sizeof(K)));
    struct State {
        uint64_t bucket, step, wins, num;
        uint32_t hits; /* slots of the window whose buckets are still to be read */
        bool free;     /* the window has a free slot */
    };

    static __device__ __forceinline__ const TableView &view(const Args &a) { return a.m.t; }

    static __device__ __forceinline__ void start(const Args &a, K key, State &s)
    {
        s.bucket = probe_begin<K>(a.m.t, key);
        s.step = 0;
        s.wins = 0;
        s.num = 0;
        s.hits = 0;
        s.free = false;
    }

    /* the lanes' windows and buckets are loaded before any is looked at */
    static __device__ __forceinline__ bool count_step(const Args &a, K key, State &s, uint32_t &st)
    {
        const uint32_t B = mb_b<kB>(a.m);
        KeyWindow<K, kW> win;
        uint32_t e = 0;
        const bool at_window = s.hits == 0;
        if (at_window) load(a, key, s, win);
        else e = places(a, s, 31 - __clz(s.hits), nullptr);
        if (at_window) {
            s.free = win.any_free(K(a.m.t.empty_key));
            s.hits = win.key_slots(key);
            if (s.hits) return false;
        } else {
            s.num += uint64_t(B) * uint64_t(__popc(s.hits)) - uint64_t(__popc(e));
            s.hits = 0;
        }
        return next(a, key, s, st, a.m.max_values);
    }

    static __device__ __forceinline__ bool value_step(const Args &a, K key, State &s, V *out,
                                                      uint64_t room)
    {
        const uint32_t B = mb_b<kB>(a.m);
        KeyWindow<K, kW> win;
        V v[kB ? kB : 32];
        uint32_t e = 0;
        const bool at_window = s.hits == 0;
        if (at_window) load(a, key, s, win);
        else e = places(a, s, __ffs(s.hits) - 1, v);
        if (at_window) {
            s.free = win.any_free(K(a.m.t.empty_key));
            s.hits = win.key_slots(key);
            if (s.hits) return false;
        } else {
            for (uint32_t r = 0; r < (kB ? uint32_t(kB) : B); ++r)
                if (!((e >> r) & 1u) && s.num + r < room) out[s.num + r] = v[r];
            s.num += B;
            s.hits &= s.hits - 1u;
            if (s.hits) return false;
            s.num -= uint64_t(__popc(e)); /* of the window's last bucket */
        }
        uint32_t st;
        return next(a, key, s, st, room < a.m.max_values ? room : a.m.max_values);
    }

    static __device__ __forceinline__ void load(const Args &a, K key, const State &s,
                                                KeyWindow<K, kW> &win)
    {
        const uint32_t W = mb_w<kW>(a.m);
        win.load(reinterpret_cast<const K *>(a.m.t.slots) + s.bucket * W, W, key,
                 K(a.m.t.empty_key));
    }
    /* the places of the bucket of window slot i: free ones, and all values */
    static __device__ __forceinline__ uint32_t places(const Args &a, const State &s, int i, V *v)
    {
        const uint32_t W = mb_w<kW>(a.m), B = mb_b<kB>(a.m);
        return mb_bucket_empties<V, kB>(
            reinterpret_cast<const V *>(a.m.vals) + (s.bucket * W + uint64_t(i)) * B, B,
            V(a.m.empty_value), v);
    }

    static __device__ __forceinline__ bool next(const Args &a, K key, State &s, uint32_t &st,
                                                uint64_t stop_at)
    {
        if (s.free || s.num >= stop_at) {
            st = s.num ? kStNone : kStKeyNotFound;
            return true;
        }
        if (++s.wins >= a.max_windows) {
            st = kStProbingLengthExceeded;
            return true;
        }
        if (s.wins == 1) s.step = probe_step<K>(a.m.t, key);
        s.bucket = probe_next(a.m.t, s.bucket, s.step);
        return false;
    }
};

/* retrieve_all_keys (gpu_engine.cuh:51-93): slot `gid` emits its key when
 * it is the lowest slot of the first window holding the key; compacted by
 * block tiles (wc_compact.cuh) */
template <class K>
__global__ void __launch_bounds__(256) mb_unique_keys_kernel(const MbView m, uint64_t capacity,
                                                             void *keys_out,
                                                             unsigned long long *count)
{
    const TableView &t = m.t;
    const K empty = K(t.empty_key), tomb = K(t.tombstone_key);
    const K *const keys = reinterpret_cast<const K *>(t.slots);
    compact_tiles<K, K>(capacity, reinterpret_cast<K *>(keys_out), nullptr, count,
                        [&](uint64_t gid, K &key, K &) {
                            key = keys[gid];
                            if (key == empty || key == tomb) return false;
                            uint64_t b = probe_begin<K>(t, key), step = 0;
                            for (uint64_t w = 0; w < t.num_buckets; ++w) {
                                uint32_t hits, emp;
                                mb_window<K, 0>(keys + b * t.cg_size, t.cg_size, key, empty,
                                                hits, emp);
                                if (hits) return b * t.cg_size + uint64_t(__ffs(hits) - 1) == gid;
                                if (w == 0) step = probe_step<K>(t, key);
                                b = probe_next(t, b, step);
                            }
                            return false;
                        });
}

/* size (gpu_engine.cuh:419-464): non-empty values of slots with a valid key */
template <class K, class V>
__global__ void __launch_bounds__(256) mb_size_kernel(const MbView m, uint64_t capacity,
                                                      unsigned long long *count)
{
    const K empty = K(m.t.empty_key), tomb = K(m.t.tombstone_key);
    const V ev = V(m.empty_value);
    const K *const keys = reinterpret_cast<const K *>(m.t.slots);
    const V *const vals = reinterpret_cast<const V *>(m.vals);
    unsigned long long c = 0;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < capacity; i += stride) {
        const K k = keys[i];
        if (k == empty || k == tomb) continue;
        for (uint32_t r = 0; r < m.bucket; ++r) c += vals[i * m.bucket + r] != ev;
    }
    const unsigned s = __reduce_add_sync(0xffffffffu, unsigned(c));
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(count, (unsigned long long)s);
}

struct MbKernels {
    uint32_t find_tile;
    const void *insert_one, *insert_more, *count, *offsets, *values, *unique, *size;
};

template <class K, class V, int kW, int kB>
MbKernels mb_kernels_of()
{
    /* buckets of one value, and of more */
    const void *one = nullptr, *more = nullptr;
    if constexpr (kB <= 1) one = reinterpret_cast<const void *>(mb_insert_kernel<K, V, kW, kB>);
    if constexpr (kB != 1)
        more = reinterpret_cast<const void *>(mb_insert_queue_kernel<K, V, kW, kB>);
    return {MbWalk<K, V, kW, kB>::kFindTile, one, more,
            reinterpret_cast<const void *>(multi_find_kernel<MbWalk<K, V, kW, kB>, false>),
            reinterpret_cast<const void *>(multi_find_kernel<MbWalk<K, V, kW, kB>, true>),
            reinterpret_cast<const void *>(multi_values_kernel<MbWalk<K, V, kW, kB>>),
            reinterpret_cast<const void *>(mb_unique_keys_kernel<K>),
            reinterpret_cast<const void *>(mb_size_kernel<K, V>)};
}

/* CG 8 (the reference's default) with buckets of 1, 2, 4 or 8 runs kernels
 * built for that shape; every other shape runs the run-time ones */
template <class K, class V>
MbKernels mb_kernels_kv(uint32_t cg, uint32_t bucket)
{
    if (cg == 8) {
        switch (bucket) {
        case 1: return mb_kernels_of<K, V, 8, 1>();
        case 2: return mb_kernels_of<K, V, 8, 2>();
        case 4: return mb_kernels_of<K, V, 8, 4>();
        case 8: return mb_kernels_of<K, V, 8, 8>();
        default: break;
        }
    }
    return mb_kernels_of<K, V, 0, 0>();
}

MbKernels mb_kernels(const wc_mbht *t)
{
    using U32 = unsigned int;
    using U64 = unsigned long long;
    const uint32_t cg = t->cfg.cg_size, b = t->bucket;
    if (t->cfg.key_bytes == 4)
        return t->cfg.value_bytes == 4 ? mb_kernels_kv<U32, U32>(cg, b) : mb_kernels_kv<U32, U64>(cg, b);
    return t->cfg.value_bytes == 4 ? mb_kernels_kv<U64, U32>(cg, b) : mb_kernels_kv<U64, U64>(cg, b);
}

MbView view_of(const wc_mbht *t)
{
    MbView m{};
    TableView &v = m.t;
    v.slots = t->keys;
    v.status = t->status;
    v.fps = nullptr;
    v.num_buckets = t->num_buckets;
    v.seed = t->seed;
    v.empty_key = t->cfg.empty_key;
    v.tombstone_key = t->cfg.tombstone_key;
    v.max_count = ~0ull;
    v.magic_nb = barrett_magic(t->num_buckets);
    v.magic_nb1 = barrett_magic(t->num_buckets > 1 ? t->num_buckets - 1 : 1);
    v.probing = t->cfg.probing;
    v.hasher1 = t->cfg.hasher1;
    v.hasher2 = t->cfg.hasher2;
    v.cg_size = t->cfg.cg_size;
    m.vals = t->vals;
    m.empty_value = t->empty_value;
    m.max_values = t->max_values;
    m.bucket = t->bucket;
    m.num_keys = t->counters;
    m.num_occupied = t->counters + 1;
    return m;
}

int check(const wc_mbht *t)
{
    if (!t) return mb_fail(WC_ERR_INVALID_ARGUMENT, "table is NULL");
    if (!t->initialized) return mb_fail(WC_ERR_NOT_INITIALIZED, "table is not initialized");
    return WC_OK;
}

MbArgs args_of(const wc_mbht *t, const void *keys, uint64_t n, uint64_t probing_length, bool find,
               void *status_out, int handler, uint32_t ignore)
{
    MbArgs a{};
    a.m = view_of(t);
    a.keys = keys;
    a.n = n;
    /* for_each caps the probing length at the capacity (:802) */
    const uint64_t pl = find && probing_length > t->capacity ? t->capacity : probing_length;
    a.max_windows = max_windows(pl, t->cfg.cg_size, t->num_buckets);
    a.status_out = handler == WC_HANDLER_NOTHING ? nullptr : status_out;
    a.handler = handler;
    a.bool_mask = (~ignore) ^ 0xFFFu; /* ~Status(Ignore), status.cuh:142-146 */
    return a;
}

int launch(const void *k, uint64_t items, MbArgs &a, cudaStream_t s)
{
    void *args[] = {&a};
    MB_CUDA(cudaLaunchKernel(k, dim3(host_grid(k, kBlock, items, kBlock)), dim3(kBlock), args, 0, s));
    note_launches(1);
    return WC_OK;
}

int read_counter(const unsigned long long *d, cudaStream_t s, uint64_t *out)
{
    return host_read_counter(d, s, out);
}

/* per-key counts (and their sum, read back) */
int count(wc_mbht *t, const void *keys, uint64_t n, uint64_t *counts_dev, uint64_t *total,
          cudaStream_t s, uint64_t probing_length, void *status_out, int handler, uint32_t ignore)
{
    MbArgs a = args_of(t, keys, n, probing_length, true, status_out, handler, ignore);
    const MbKernels k = mb_kernels(t);
    return host_multi_count(k.count, k.find_tile, &a, &a, t->counters + 8, counts_dev, total, s);
}

/* host join of status bits into the table's Status word */
int join_host(wc_mbht *t, uint32_t bits, cudaStream_t s)
{
    return host_join_status(t->status, bits, s);
}

/* fill `bytes` (a multiple of 4) with a repeated 4- or 8-byte word, and
 * n_zero words at `zero` with zeros */
int fill(void *p, uint64_t bytes, uint64_t word, uint32_t word_bytes, cudaStream_t s,
         uint32_t *zero = nullptr, uint32_t n_zero = 0)
{
    uint32_t w[4];
    if (word_bytes == 4) {
        w[0] = w[1] = w[2] = w[3] = uint32_t(word);
    } else {
        w[0] = w[2] = uint32_t(word);
        w[1] = w[3] = uint32_t(word >> 32);
    }
    uint4 pat = make_uint4(w[0], w[1], w[2], w[3]);
    uint32_t *dst = reinterpret_cast<uint32_t *>(p);
    uint64_t n = bytes / 4;
    const void *kfn = reinterpret_cast<const void *>(fill_kernel<0>);
    void *args[] = {&dst, &n, &pat, &zero, &n_zero};
    MB_CUDA(cudaLaunchKernel(kfn, dim3(host_grid(kfn, kBlock, n / 4, kBlock)), dim3(kBlock), args, 0,
                             s));
    note_launches(1);
    return WC_OK;
}

} // namespace

extern "C" {

int wc_mbht_create(const wc_table_config *cfg, uint32_t bucket_size, uint64_t empty_value,
                   uint64_t min_capacity, uint64_t seed, uint64_t max_values_per_key, int no_init,
                   wc_mbht **out)
{
    if (!out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (!cfg) return mb_fail(WC_ERR_INVALID_ARGUMENT, "config is NULL");
    if (cfg->key_bytes != 4 && cfg->key_bytes != 8)
        return mb_fail(WC_ERR_UNSUPPORTED, "key_bytes must be 4 or 8");
    if (cfg->value_bytes != 4 && cfg->value_bytes != 8)
        return mb_fail(WC_ERR_UNSUPPORTED, "value_bytes must be 4 or 8");
    const uint32_t cg = cfg->cg_size;
    if (!(cg == 1 || cg == 2 || cg == 4 || cg == 8 || cg == 16 || cg == 32))
        return mb_fail(WC_ERR_INVALID_ARGUMENT, "cg_size must be 1, 2, 4, 8, 16 or 32");
    if (bucket_size == 0 || bucket_size > cg)
        return mb_fail(WC_ERR_UNSUPPORTED, "bucket_size must be 1 .. cg_size");
    if (cfg->probing > WC_PROBING_QUADRATIC || cfg->hasher1 > WC_HASH_IDENTITY64 ||
        cfg->hasher2 > WC_HASH_IDENTITY64)
        return mb_fail(WC_ERR_INVALID_ARGUMENT, "unknown probing scheme or hasher");
    const uint64_t km = kmask(cfg->key_bytes);
    if ((cfg->empty_key & km) == (cfg->tombstone_key & km))
        return mb_fail(WC_ERR_INVALID_ARGUMENT, "empty key and tombstone key must differ");
    const uint64_t cap = host_valid_capacity(min_capacity, cg);
    if (cap == 0) return mb_fail(WC_ERR_INVALID_ARGUMENT, "min_capacity exceeds the largest capacity");
    auto *t = new wc_mbht();
    t->cfg = *cfg;
    t->cfg.empty_key &= km;
    t->cfg.tombstone_key &= km;
    t->bucket = bucket_size;
    t->empty_value = empty_value & kmask(cfg->value_bytes);
    t->capacity = cap;
    t->num_buckets = cap / cg;
    t->seed = seed & km;
    t->max_values = max_values_per_key;
    const uint64_t kbytes = (cap * cfg->key_bytes + 255) & ~uint64_t(255);
    const uint64_t vbytes = cap * bucket_size * cfg->value_bytes;
    cudaError_t e = cudaMalloc(&t->keys, kbytes + vbytes);
    if (e == cudaSuccess) e = cudaMalloc(&t->status, 256);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (t->keys) cudaFree(t->keys);
        delete t;
        return host_cuda_fail(e, "cudaMalloc (multi-bucket table)");
    }
    t->vals = static_cast<char *>(t->keys) + kbytes;
    t->counters = reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(t->status) + 64);
    *out = t;
    if (!no_init) {
        const int rc = wc_mbht_init(t, nullptr);
        if (rc) {
            wc_mbht_destroy(t);
            *out = nullptr;
            return rc;
        }
    }
    return WC_OK;
}

int wc_mbht_destroy(wc_mbht *t)
{
    if (!t) return WC_OK;
    if (t->keys) cudaFree(t->keys);
    if (t->status) cudaFree(t->status);
    if (t->scan) cudaFree(t->scan);
    delete t;
    return WC_OK;
}

int wc_mbht_init(wc_mbht *t, wc_stream_t stream)
{
    if (!t) return mb_fail(WC_ERR_INVALID_ARGUMENT, "table is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int rc = fill(t->keys, t->capacity * t->cfg.key_bytes, t->cfg.empty_key, t->cfg.key_bytes, s);
    if (rc) return rc;
    rc = fill(t->vals, t->capacity * t->bucket * t->cfg.value_bytes, t->empty_value,
              t->cfg.value_bytes, s, t->status, 256 / 4);
    if (rc) return rc;
    MB_CUDA(cudaStreamSynchronize(s));
    t->initialized = true;
    return WC_OK;
}

int wc_mbht_insert(wc_mbht *t, const void *keys_in, const void *values_in, uint64_t num_in,
                   wc_stream_t stream, uint64_t probing_length, void *status_out,
                   int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (status_handler < WC_HANDLER_NOTHING || status_handler > WC_HANDLER_BOOLEAN)
        return mb_fail(WC_ERR_INVALID_ARGUMENT, "unknown status handler");
    if (num_in == 0) return WC_OK;
    if (!keys_in || !values_in) return mb_fail(WC_ERR_INVALID_ARGUMENT, "keys_in / values_in is NULL");
    MbArgs a = args_of(t, keys_in, num_in, probing_length, false, status_out, status_handler, ignore);
    a.values = values_in;
    const MbKernels k = mb_kernels(t);
    return launch(t->bucket == 1 ? k.insert_one : k.insert_more, num_in, a,
                  reinterpret_cast<cudaStream_t>(stream));
}

int wc_mbht_num_values(wc_mbht *t, const void *keys_in, uint64_t num_in, uint64_t *num_out,
                       uint64_t *num_per_key_out, wc_stream_t stream, uint64_t probing_length,
                       void *status_out, int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    *num_out = 0;
    if (num_in == 0) return WC_OK;
    if (!keys_in) return mb_fail(WC_ERR_INVALID_ARGUMENT, "keys_in is NULL");
    return count(t, keys_in, num_in, num_per_key_out, num_out,
                 reinterpret_cast<cudaStream_t>(stream), probing_length, status_out,
                 status_handler, ignore);
}

int wc_mbht_retrieve(wc_mbht *t, const void *keys_in, uint64_t num_in,
                     uint64_t *begin_offsets_out, uint64_t *end_offsets_out, void *values_out,
                     uint64_t *num_out, wc_stream_t stream, uint64_t probing_length,
                     void *status_out, int status_handler, uint32_t ignore)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    *num_out = 0;
    if (num_in == 0) return WC_OK;
    if (!keys_in || !end_offsets_out || (values_out && !begin_offsets_out))
        return mb_fail(WC_ERR_INVALID_ARGUMENT, "NULL buffer");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!values_out) {
        /* dry run: per-key counts, status dry_run for every key */
        rc = count(t, keys_in, num_in, end_offsets_out, num_out, s, probing_length, nullptr,
                   WC_HANDLER_NOTHING, ignore);
        if (rc) return rc;
        rc = host_dry_run_status(status_out, num_in, status_handler, ignore, s);
        if (rc) return rc;
        return join_host(t, kStDryRun, s);
    }
    MbArgs a = args_of(t, keys_in, num_in, probing_length, true, status_out, status_handler, ignore);
    const MbKernels k = mb_kernels(t);
    return host_multi_retrieve(k.offsets, k.find_tile, k.values, &a, &a, &t->scan, &t->scan_bytes,
                               begin_offsets_out, end_offsets_out, values_out, num_out, s);
}

int wc_mbht_retrieve_all_keys(wc_mbht *t, void *keys_out, uint64_t *num_out, wc_stream_t stream)
{
    int rc = check(t);
    if (rc) return rc;
    if (!num_out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "num_out is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!keys_out) {
        rc = read_counter(t->counters, s, num_out);
        if (rc) return rc;
        return join_host(t, kStDryRun, s);
    }
    unsigned long long *tmp = t->counters + 2;
    MB_CUDA(cudaMemsetAsync(tmp, 0, sizeof(unsigned long long), s));
    MbView v = view_of(t);
    uint64_t cap = t->capacity;
    const MbKernels k = mb_kernels(t);
    void *args[] = {&v, &cap, &keys_out, &tmp};
    MB_CUDA(cudaLaunchKernel(k.unique, dim3(host_grid(k.unique, kBlock, cap, kBlock)), dim3(kBlock),
                             args, 0, s));
    note_launches(1);
    return read_counter(tmp, s, num_out);
}

int wc_mbht_num_keys(wc_mbht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    return read_counter(t->counters, reinterpret_cast<cudaStream_t>(stream), out);
}

int wc_mbht_num_occupied(wc_mbht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    return read_counter(t->counters + 1, reinterpret_cast<cudaStream_t>(stream), out);
}

int wc_mbht_size(wc_mbht *t, wc_stream_t stream, uint64_t *out)
{
    int rc = check(t);
    if (rc) return rc;
    if (!out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "out is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    unsigned long long *tmp = t->counters + 2;
    MB_CUDA(cudaMemsetAsync(tmp, 0, sizeof(unsigned long long), s));
    MbView v = view_of(t);
    uint64_t cap = t->capacity;
    const MbKernels k = mb_kernels(t);
    void *args[] = {&v, &cap, &tmp};
    MB_CUDA(cudaLaunchKernel(k.size, dim3(host_grid(k.size, kBlock, cap, kBlock)), dim3(kBlock), args,
                             0, s));
    note_launches(1);
    return read_counter(tmp, s, out);
}

int wc_mbht_peek_status(wc_mbht *t, wc_stream_t stream, uint32_t *out)
{
    if (!t || !out) return mb_fail(WC_ERR_INVALID_ARGUMENT, "NULL argument");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    MB_CUDA(cudaMemcpyAsync(out, t->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    MB_CUDA(cudaStreamSynchronize(s));
    return WC_OK;
}

int wc_mbht_pop_status(wc_mbht *t, wc_stream_t stream, uint32_t *out)
{
    int rc = wc_mbht_peek_status(t, stream, out);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    MB_CUDA(cudaMemsetAsync(t->status, 0, sizeof(uint32_t), s));
    MB_CUDA(cudaStreamSynchronize(s));
    return WC_OK;
}

int wc_mbht_get_info(const wc_mbht *t, wc_mbht_info *info)
{
    if (!t || !info) return mb_fail(WC_ERR_INVALID_ARGUMENT, "NULL argument");
    std::memset(info, 0, sizeof(*info));
    info->key_bytes = t->cfg.key_bytes;
    info->value_bytes = t->cfg.value_bytes;
    info->bucket_size = t->bucket;
    info->cg_size = t->cfg.cg_size;
    info->probing = t->cfg.probing;
    info->hasher1 = t->cfg.hasher1;
    info->hasher2 = t->cfg.hasher2;
    info->capacity = t->capacity;
    info->value_capacity = t->capacity * t->bucket;
    info->num_buckets = t->num_buckets;
    info->seed = t->seed;
    info->empty_key = t->cfg.empty_key;
    info->tombstone_key = t->cfg.tombstone_key;
    info->empty_value = t->empty_value;
    info->max_values_per_key = t->max_values;
    info->bytes_total = t->capacity * (t->cfg.key_bytes + uint64_t(t->bucket) * t->cfg.value_bytes) +
                        sizeof(uint64_t);
    info->keys = t->keys;
    info->values = t->vals;
    info->status = t->status;
    info->num_keys = t->counters;
    info->num_occupied = t->counters + 1;
    info->is_initialized = t->initialized ? 1 : 0;
    return WC_OK;
}

} // extern "C"
