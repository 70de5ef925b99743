/*
 * wc_mv.cuh -- MultiValueHashTable kernels (the reference's
 * multi_value_hash_table.cuh: insert :200-289, for_each / num_values
 * :607-663, bulk retrieve :371-520, unique keys gpu_engine.cuh:51-93).
 *
 * Every (key, value) pair takes a slot of its own.  A key's values live
 * along its bucket sequence, up to the first bucket that has a free slot:
 * insert counts them bucket by bucket (stopping at max_values_per_key) and
 * claims the first free slot of that bucket; num_values and retrieve walk
 * the same buckets and take the key's slots in slot order.  Buckets are the
 * table kernels' bucket-aligned windows, so a key's values come out in the
 * order they were inserted, as in the reference.
 *
 * Lookups go through multi_find_kernel (wc_multi.cuh).
 */
#ifndef WC_MV_CUH
#define WC_MV_CUH

#include "wc_lane_kernels.cuh"
#include "wc_multi.cuh"
#include <warpcore/detail/mv_ops.cuh>

namespace warpcore {
namespace b200 {

struct MvArgs : MultiArgs {
    TableView t;
    unsigned long long *num_keys;     /* insert: keys that got their first value */
    uint64_t max_values;
};

/* the key's slots window by window, as mv_for_each_one walks them */
template <class L, int W>
struct MvWalk {
    using key_t = typename L::key_t;
    using val_t = typename L::val_t;
    using Args = MvArgs;
    static constexpr int kFindTile = multi_find_tile(sizeof(key_t), W * L::kSlotBytes);
    struct State {
        uint64_t bucket, step, wins, num;
    };

    static __device__ __forceinline__ const TableView &view(const Args &a) { return a.t; }

    static __device__ __forceinline__ void start(const Args &a, key_t key, State &s)
    {
        s.bucket = probe_begin<key_t>(a.t, key);
        s.step = 0;
        s.wins = 0;
        s.num = 0;
    }

    /* one window; true where the walk ends */
    static __device__ __forceinline__ bool count_step(const Args &a, key_t key, State &s,
                                                      uint32_t &st)
    {
        return walk<false>(a, key, s, st, nullptr, 0, a.max_values);
    }
    static __device__ __forceinline__ bool value_step(const Args &a, key_t key, State &s,
                                                      val_t *out, uint64_t room)
    {
        uint32_t st;
        return walk<true>(a, key, s, st, out, room, room < a.max_values ? room : a.max_values);
    }

    /* ---- insert, as mv_insert_one: the key's values counted window by
     * window, then a claim of the lowest free slot of the first window that
     * has one; a claim that loses tries the next free slot it saw ---- */
    static constexpr int WB = W * L::kSlotBytes;
    static constexpr int kInsertBlocks = WB <= 64 ? WC_MULTI_INSERT_BLOCKS : 3;
    /* Many values of one key in one batch queue at the end of its walk, where
     * each step's compare-and-swaps of all its lanes but one are lost.  Past
     * kCrowd windows a lane that lost to its own key sits out up to kCrowdSkip
     * steps: 2^20 Zipf(0.8) keys over 2^20 (the most frequent 14 000 times) 13.6
     * -> 11.1 ms in u32 pairs, 13.4 -> 12.0 in u64; 2^17 Zipf(1.01) 9.2 -> 7.5,
     * 10.1 -> 8.4.  Shorter lists are left alone: from 32 windows on, 2^20
     * Zipf(0.5) keys took 397 us, 307 without any and 315 so. */
    static constexpr uint32_t kCrowd = 128, kCrowdSkip = 31;
    struct InsertState {
        uint64_t bucket, step, wins, num;
        uint32_t free; /* free slots still to be tried; 0: the window is due */
        val_t expect;  /* payload the slot is expected to hold */
        uint32_t skip; /* steps to sit out (kCrowd) */
    };
    struct InsertIo {
        uint32_t w[WB <= 128 ? WB / 4 : 1];
        uint32_t hits, free;
        key_t old;
        val_t old_payload;
    };
    struct Counts {
        unsigned fresh; /* keys that got their first value */
    };

    static __device__ __forceinline__ uint32_t insert_start(const Args &a, key_t key, val_t,
                                                            InsertState &s)
    {
        if (key == key_t(a.t.empty_key) || key == key_t(a.t.tombstone_key)) return kStInvalidKey;
        s.bucket = probe_begin<key_t>(a.t, key);
        s.step = 0;
        s.wins = 0;
        s.num = 0;
        s.free = 0;
        s.expect = 0;
        s.skip = 0;
        return kStNone;
    }

    static __device__ __forceinline__ unsigned char *slot_of(const Args &a, const InsertState &s)
    {
        return reinterpret_cast<unsigned char *>(a.t.slots) + s.bucket * uint64_t(WB) +
               (__ffs(s.free) - 1) * L::kSlotBytes;
    }

    static __device__ __forceinline__ void issue(const Args &a, key_t key, val_t val,
                                                 const InsertState &s, InsertIo &io)
    {
        if (s.skip) return;
        if (s.free) {
            io.old = cas_slot<L>(slot_of(a, s), key_t(a.t.empty_key), s.expect, key, val,
                                 &io.old_payload);
        } else if constexpr (WB <= 128) {
            load_window<WB>(reinterpret_cast<const unsigned char *>(a.t.slots) +
                                s.bucket * uint64_t(WB), io.w);
        } else {
            mv_bucket<L, W>(a.t, s.bucket, key, io.hits, io.free,
                            [](int, const LaneWords &, int) {});
        }
    }

    static __device__ __forceinline__ bool look(const Args &a, key_t key, val_t val,
                                                InsertState &s, const InsertIo &io, uint32_t &st,
                                                uint32_t &join, Counts &counts)
    {
        const key_t empty = key_t(a.t.empty_key);
        bool advance = false;
        if (s.skip) {
            --s.skip;
            return false;
        }
        if (s.free) {
            if (io.old == empty && io.old_payload == s.expect) {
                counts.fresh += s.num == 0;
                st = s.num ? kStDuplicateKey : kStNone;
                return true;
            }
            if (io.old == empty) {
                s.expect = io.old_payload; /* free slot, stale payload: again */
                return false;
            }
            if (io.old == key && ++s.num >= a.max_values) {
                st = kStDuplicateKey | kStMaxValuesReached;
                join |= st;
                return true;
            }
            if (io.old == key && s.wins >= kCrowd)
                s.skip = (threadIdx.x * 7u + blockIdx.x * 5u + uint32_t(s.num) * 3u) &
                         kCrowdSkip;
            s.free &= s.free - 1u;
            s.expect = 0;
            advance = s.free == 0;
        } else {
            uint32_t hits = io.hits, free = io.free;
            if constexpr (WB <= 128) {
                bool any_hit = false, any_free = false;
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    any_hit |= window_key<L>(io.w, i) == key;
                    any_free |= window_key<L>(io.w, i) == empty;
                }
                hits = free = 0;
                if (any_hit) {
#pragma unroll
                    for (int i = 0; i < W; ++i) hits += window_key<L>(io.w, i) == key;
                    s.num += hits;
                }
                if (any_free) {
#pragma unroll
                    for (int i = 0; i < W; ++i)
                        free |= uint32_t(window_key<L>(io.w, i) == empty) << i;
                }
            } else {
                s.num += uint64_t(__popc(hits));
            }
            if (s.num >= a.max_values) {
                st = kStDuplicateKey | kStMaxValuesReached;
                join |= st;
                return true;
            }
            s.free = free;
            advance = free == 0;
        }
        if (!advance) return false;
        if (++s.wins >= a.max_windows) {
            st = kStProbingLengthExceeded | (s.num ? kStDuplicateKey : kStNone);
            join |= st;
            return true;
        }
        if (s.wins == 1) s.step = probe_step<key_t>(a.t, key);
        s.bucket = probe_next(a.t, s.bucket, s.step);
        return false;
    }

    static __device__ __forceinline__ void add_counts(const Args &a, const Counts &c)
    {
        const unsigned f = __reduce_add_sync(kFull, c.fresh);
        if ((threadIdx.x & 31) == 0 && f) atomicAdd(a.num_keys, (unsigned long long)f);
    }

    template <bool kValues>
    static __device__ __forceinline__ bool walk(const Args &a, key_t key, State &s, uint32_t &st,
                                                val_t *out, uint64_t room, uint64_t stop_at)
    {
        const key_t empty = key_t(a.t.empty_key);
        bool free = false;
        if constexpr (WB <= 128) {
            uint32_t w[WB / 4];
            load_window<WB>(reinterpret_cast<const unsigned char *>(a.t.slots) +
                                s.bucket * uint64_t(WB), w);
            bool any = false; /* one compare per slot; more only where the key is */
#pragma unroll
            for (int i = 0; i < W; ++i) {
                any |= window_key<L>(w, i) == key;
                free |= window_key<L>(w, i) == empty;
            }
            if (any) {
#pragma unroll
                for (int i = 0; i < W; ++i)
                    if (window_key<L>(w, i) == key) {
                        if constexpr (kValues) {
                            if (s.num < room) out[s.num] = window_val<L>(w, i);
                        }
                        ++s.num;
                    }
            }
        } else {
            uint32_t hits, emp;
            mv_bucket<L, W>(a.t, s.bucket, key, hits, emp, [&](int, const LaneWords &lw, int i) {
                if constexpr (kValues) {
                    if (s.num < room) out[s.num] = slot_val<L>(lw, i);
                }
                ++s.num;
            });
            free = emp != 0;
        }
        if (free || s.num >= stop_at) {
            st = s.num ? kStNone : kStKeyNotFound;
            return true;
        }
        if (++s.wins >= a.max_windows) {
            st = kStProbingLengthExceeded;
            return true;
        }
        if (s.wins == 1) s.step = probe_step<key_t>(a.t, key);
        s.bucket = probe_next(a.t, s.bucket, s.step);
        return false;
    }
};

/* retrieve_all_keys: slot `gid` emits its key when it is the key's first
 * entry along its bucket sequence (lowest slot of the first bucket holding
 * the key), compacted by block tiles (wc_compact.cuh) */
template <class L, int W>
__global__ void __launch_bounds__(256) mv_unique_keys_kernel(TableView t, uint64_t capacity,
                                                             void *keys_out,
                                                             unsigned long long *count)
{
    using K = typename L::key_t;
    constexpr int SB = L::kSlotBytes;
    const K empty = K(t.empty_key), tomb = K(t.tombstone_key);
    const unsigned char *const slots = reinterpret_cast<const unsigned char *>(t.slots);
    compact_tiles<K, K>(capacity, reinterpret_cast<K *>(keys_out), nullptr, count,
                        [&](uint64_t gid, K &key, K &) {
                            key = *reinterpret_cast<const K *>(slots + gid * SB);
                            if (key == empty || key == tomb) return false;
                            uint64_t b = probe_begin<K>(t, key), step = 0;
                            for (uint64_t w = 0; w < t.num_buckets; ++w) {
                                uint32_t hits, emp;
                                mv_bucket<L, W>(t, b, key, hits, emp,
                                                [](int, const LaneWords &, int) {});
                                if (hits) return b * W + uint64_t(__ffs(hits) - 1) == gid;
                                if (w == 0) step = probe_step<K>(t, key);
                                b = probe_next(t, b, step);
                            }
                            return false;
                        });
}

} // namespace b200
} // namespace warpcore

#endif /* WC_MV_CUH */
