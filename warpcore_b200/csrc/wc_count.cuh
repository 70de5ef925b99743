/*
 * wc_count.cuh -- counting insert without per-key statuses
 * (counting_hash_table.cuh:75-249).
 *
 * What bounds a counting insert is the table's atomics, one per key, on few
 * addresses where the stream is skewed, and the instructions around them.
 * One block per SM keeps a count cache in shared memory: equal keys add up
 * there and each cached key reaches the table once, when the block ends.
 *   - Keys pass the cache 32 at a time per warp: a four-entry set is one
 *     vector read of shared memory, a hit one shared-memory add.  Keys that
 *     find their set full of others go to a queue of the warp.
 *   - Lanes take keys from the queue and probe the table, one memory
 *     operation per lane and step (the key's window, or a claim's
 *     compare-and-swap), as the one-key-per-lane kernel does; a lane whose
 *     key is done takes the next one.  The result of a count's atomicAdd,
 *     needed for the wrap check only, is looked at one step later.
 *   - The cached keys take the same way when the input is used up.
 * A warp whose first kCountSample keys hit the cache in less than one of
 * kCountMinHits leaves it out for a while: in a stream of nearly distinct
 * keys the cache only delays them.  Keys left for the queue are merged with
 * equal ones of the same 32, so that a stream in runs, or one whose frequent
 * keys found the cache full, sends one add for each.  (A warp that found no
 * equal keys four times looks at one 32 of eight.)  2^26 u32 keys in runs of
 * four 2 030 -> 955 us, 2^26 sorted Zipf(1.1) u64 keys 1 670 -> 987.
 *
 * Measured against table_op_kernel and its caches of 32 KiB per block, which
 * merged all equal keys with __match_any_sync, probed the table in the same
 * loop and counted the cached keys slot by slot at the end: u32 pairs, 2^27
 * Zipf(1.1) keys over 2^23 (84 MB) 2496 -> 1252 us (107 G keys/s); 2^25
 * Zipf(1.1) over 2^20 679 -> 330; u64 keys, 3 M Zipf(0.5) over 1 M 199 ->
 * 109; 300 000 u32 keys over 20 000 40 -> 22.
 *
 * Statuses of the table (duplicate_key, probing_length_exceeded,
 * index_overflow, invalid_key), the bucket sequence and the claim order
 * (lowest free slot of a window) are those of table_op_kernel.
 */
#ifndef WC_COUNT_CUH
#define WC_COUNT_CUH

#include "wc_lane_kernels.cuh"

namespace warpcore {
namespace b200 {

constexpr int kCountThreads = 1024; /* one block per SM, at most 64 registers */
constexpr int kCountWarps = kCountThreads / 32;
constexpr int kCountQueue = 64;     /* keys a warp's queue holds */
/* When a warp leaves the cache out: fewer than one of kCountMinHits of the
 * first kCountSample keys hit it.  Even few early hits pay later, when the
 * cache holds the frequent keys: Zipf(0.8), 2^25 u32 keys over 2^22, ran
 * 1757 / 792 / 703 / 692 us with one hit of 6 / 16 / 32 / 64 of the first 128
 * keys.  A stream may begin with rare keys, so the warp tries the cache again
 * for kCountResample keys after every kCountAgain: where each warp's first 300
 * keys were distinct and the others 16 hot ones, 2^24 u32 keys took 2 440 us
 * without that and 357 with it, u64 keys 3 430 and 590. */
constexpr uint32_t kCountSample = 128;
constexpr uint32_t kCountMinHits = 64;
constexpr uint32_t kCountAgain = 512, kCountResample = 64;

/* What a warp remembers from one 32 keys to the next: keys of the present
 * sample and its hits, for how many times 32 keys the cache is still left out,
 * and times since equal keys were found.  In one register where keys take 8
 * bytes, whose kernels have none left (2^24 Zipf(0.5) keys over 2^20: 455 us
 * with each in its own, 438 so); for 4-byte keys that costs more than it saves
 * (2^26 Zipf(1.4) keys over 2^24 406 and 417). */
template <bool kPacked>
struct CountWarp;

template <>
struct CountWarp<false> {
    uint32_t seen = 0, hits = 0, off = 0, quiet = 0;
    bool on = true;

    __device__ __forceinline__ bool cache() const { return on; }
    __device__ __forceinline__ bool sampling() const { return seen < kCountSample; }
    /* 32 more keys of the sample, `more` of them hits */
    __device__ __forceinline__ void sampled(uint32_t more)
    {
        seen += 32;
        hits += more;
        if (seen >= kCountSample && hits * kCountMinHits < seen) {
            on = false;
            off = kCountAgain / 32;
        }
    }
    __device__ __forceinline__ void left_out()
    {
        if (--off == 0) {
            on = true;
            seen = kCountSample - kCountResample;
            hits = 0;
        }
    }
    __device__ __forceinline__ bool look_for_equal() const { return quiet < 4 || (quiet & 7) == 0; }
    __device__ __forceinline__ void equal(bool found) { quiet = found ? 1 : quiet + 1; }
};

template <>
struct CountWarp<true> {
    /* bits 0 to 3 seen / 32, 4 to 13 hits, 14 to 21 off, 22 on quiet (4 to 15,
     * going back to 8) */
    uint32_t bits = 0;

    __device__ __forceinline__ bool cache() const { return (bits >> 14 & 0xffu) == 0; }
    __device__ __forceinline__ bool sampling() const { return (bits & 0xfu) < kCountSample / 32; }
    __device__ __forceinline__ void sampled(uint32_t more)
    {
        bits += 1u + (more << 4);
        if (!sampling() && (bits >> 4 & 0x3ffu) * kCountMinHits < kCountSample)
            bits = (bits & ~0x3fffffu) | (kCountSample - kCountResample) / 32 |
                   (kCountAgain / 32) << 14;
    }
    __device__ __forceinline__ void left_out() { bits -= 1u << 14; }
    __device__ __forceinline__ bool look_for_equal() const
    {
        return bits >> 22 < 4 || bits >> 22 == 8;
    }
    __device__ __forceinline__ void equal(bool found)
    {
        if (found) bits &= 0x3fffffu;
        bits += bits >> 22 == 15 ? uint32_t(-7) << 22 : 1u << 22;
    }
};

struct CountArgs {
    TableView t;
    const void *keys;
    uint64_t n;
    uint64_t max_windows;
    uint32_t cache_bits; /* entries: 2^cache_bits */
};

/* entries of the largest cache: 128 KiB of u32 keys, 96 KiB of u64 keys, each
 * with a 32-bit count */
template <class K>
constexpr uint32_t count_cache_max_bits()
{
    return sizeof(K) == 4 ? 14 : 13;
}

template <class K>
constexpr uint32_t count_smem_bytes(uint32_t cache_bits)
{
    return (uint32_t(sizeof(K)) + 4u) * ((1u << cache_bits) + uint32_t(kCountWarps * kCountQueue));
}

/* the four keys of a cache set, as they are now */
template <class K>
__device__ __forceinline__ void load_set(const K *p, K (&e)[4])
{
    const uint32_t at = uint32_t(__cvta_generic_to_shared(p));
    if constexpr (sizeof(K) == 4) {
        asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3]) : "r"(at) : "memory");
    } else {
        asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                     : "=l"(e[0]), "=l"(e[1]) : "r"(at) : "memory");
        asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                     : "=l"(e[2]), "=l"(e[3]) : "r"(at + 16u) : "memory");
    }
}

template <class L, int W>
__global__ void __launch_bounds__(kCountThreads, 1) count_insert_kernel(const CountArgs a)
{
    using K = typename L::key_t;
    using V = typename L::val_t;
    using CW = typename std::conditional<sizeof(K) == 8, unsigned long long, unsigned int>::type;
    constexpr int SB = L::kSlotBytes;
    constexpr int WB = W * SB;
    static_assert(WB <= 128, "window of one lane");
    extern __shared__ uint4 s_mem[];
    const uint32_t entries = 1u << a.cache_bits;
    K *const s_key = reinterpret_cast<K *>(s_mem);
    K *const s_qkey = s_key + entries;
    uint32_t *const s_cnt = reinterpret_cast<uint32_t *>(s_qkey + kCountWarps * kCountQueue);
    uint32_t *const s_qcnt = s_cnt + entries;

    const TableView &t = a.t;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const K empty = K(t.empty_key), tomb = K(t.tombstone_key);
    unsigned char *const slots = reinterpret_cast<unsigned char *>(t.slots);
    K *const qkey = s_qkey + wib * kCountQueue;
    uint32_t *const qcnt = s_qcnt + wib * kCountQueue;
    int queued = 0;

    for (uint32_t c = threadIdx.x; c < entries; c += kCountThreads) {
        s_key[c] = empty;
        s_cnt[c] = 0;
    }
    __syncthreads();

    uint32_t join = 0;
    int live_delta = 0;

    /* queues the lanes' keys (those with `in`), each with count c */
    auto enqueue = [&](bool in, K key, uint32_t c) {
        const unsigned m = __ballot_sync(kFull, in);
        if (in) {
            const int p = queued + __popc(m & lanemask_lt);
            qkey[p] = key;
            qcnt[p] = c;
        }
        queued += __popc(m);
        __syncwarp();
    };

    /* probes the table for all keys that fetch() queues; fetch returns false
     * once it has none */
    auto probe = [&](auto fetch) {
        bool has = false, more = true;
        K key = empty;
        uint32_t c = 0;
        uint64_t bucket = 0, step = 0, wins = 0;
        int claim = -1; /* the slot of the window to be claimed, -1: read the window */
        V expect = 0;   /* the payload it is expected to hold */
        /* an add whose result has not been looked at */
        V *add_to = nullptr;
        V add_old = 0;
        uint32_t add_c = 0;
        for (;;) {
            while (more && queued < 32) more = fetch();
            const unsigned need = __ballot_sync(kFull, !has);
            const int idle = __popc(need);
            const int take = idle < queued ? idle : queued;
            if (take == 0 && need == kFull) break;
            const int r = __popc(need & lanemask_lt);
            if (!has && r < take) {
                key = qkey[queued - 1 - r];
                c = qcnt[queued - 1 - r];
                has = true;
                claim = -1;
                wins = 0;
                step = 0;
                bucket = probe_begin<K>(t, key);
                if (c > 1) join |= kStDuplicateKey;
            }
            queued -= take;
            __syncwarp();

            unsigned char *const window = slots + bucket * uint64_t(WB);
            uint32_t w[WB / 4];
            K old = empty;
            V old_payload = 0;
            if (has) {
                if (claim >= 0)
                    old = cas_slot<L>(window + claim * SB, empty, expect, key, V(c), &old_payload);
                else
                    load_window<WB>(window, w);
            }
            if (add_to) {
                if (V(add_old + V(add_c)) < add_old) {
                    join |= kStIndexOverflow;
                    atomic_exch_any(add_to, V(t.max_count));
                }
                add_to = nullptr;
            }
            if (!has) continue;
            int hit = -1;
            bool advance = false;
            if (claim >= 0) {
                if (old == empty && old_payload == expect) {
                    fp_store(t, bucket * W + uint64_t(claim), fingerprint(key));
                    ++live_delta;
                    has = false;
                } else if (old == key) {
                    hit = claim;
                } else if (old == empty) {
                    expect = old_payload; /* free slot, stale payload: again */
                } else {
                    claim = -1; /* taken by another key: read the window again */
                }
            } else {
                uint32_t h = 0, f = 0;
#pragma unroll
                for (int s = 0; s < W; ++s) {
                    const K sk = window_key<L>(w, s);
                    h |= uint32_t(sk == key) << s;
                    f |= uint32_t(sk == empty) << s;
                }
                if (h) {
                    hit = __ffs(h) - 1;
                } else if (f) {
                    claim = __ffs(f) - 1;
                    expect = window_val_at<L, W>(w, claim);
                } else {
                    advance = true;
                }
            }
            if (hit >= 0) {
                join |= kStDuplicateKey;
                add_to = slot_value_ptr<L>(window + hit * SB);
                add_c = c;
                add_old = atomic_add_any(add_to, V(c));
                has = false;
            }
            if (advance) {
                if (++wins >= a.max_windows) {
                    join |= kStProbingLengthExceeded;
                    has = false;
                } else {
                    if (wins == 1) step = probe_step<K>(t, key);
                    bucket = probe_next(t, bucket, step);
                }
            }
        }
        if (add_to && V(add_old + V(add_c)) < add_old) {
            join |= kStIndexOverflow;
            atomic_exch_any(add_to, V(t.max_count));
        }
    };

    /* ---- the input, through the cache ---- */
    {
        const uint64_t warp = uint64_t(blockIdx.x) * kCountWarps + wib;
        const uint64_t nwarps = uint64_t(gridDim.x) * kCountWarps;
        uint64_t per = (a.n + nwarps - 1) / nwarps;
        per = (per + 31) & ~uint64_t(31);
        const uint64_t wb = warp * per < a.n ? warp * per : a.n;
        const uint64_t m = wb + per < a.n ? per : a.n - wb;
        const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;
        uint64_t at = 0;
        K pfA = uint64_t(lane) < m ? ld_stream(keys + lane) : empty;
        K pfB = 32 + uint64_t(lane) < m ? ld_stream(keys + 32 + lane) : empty;
        CountWarp<sizeof(K) == 8> mem;
        probe([&]() {
            if (at >= m) return false;
            const K key = pfA;
            bool in = at + uint64_t(lane) < m;
            pfA = pfB;
            const uint64_t nx = at + 64 + uint64_t(lane);
            if (nx < m) pfB = ld_stream(keys + nx);
            at += 32;
            if (in && (key == empty || key == tomb)) {
                join |= kStInvalidKey;
                in = false;
            }
            if (mem.cache()) {
                bool known = false;
                if (in) {
                    const uint32_t set =
                        (sizeof(K) == 4
                             ? (uint32_t(key) * 0x9E3779B1u) >> (34 - a.cache_bits)
                             : uint32_t((uint64_t(key) * 0x9E3779B97F4A7C15ull) >>
                                        (66 - a.cache_bits))) * 4;
                    K e[4];
                    load_set(s_key + set, e);
                    /* entries of a set are taken in order and never given
                     * up, so equal keys meet on one entry */
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        if (!in) break;
                        K cur = e[p];
                        if (cur == empty) {
                            cur = K(atomicCAS(reinterpret_cast<CW *>(s_key + set + p), CW(empty),
                                              CW(key)));
                            if (cur == empty) cur = key;
                            else known = cur == key;
                        } else {
                            known = cur == key;
                        }
                        if (cur == key) {
                            atomicAdd(s_cnt + set + p, 1u);
                            in = false;
                        }
                    }
                    if (known) join |= kStDuplicateKey;
                }
                if (mem.sampling()) mem.sampled(uint32_t(__popc(__ballot_sync(kFull, known))));
            } else {
                mem.left_out();
            }
            /* equal keys among those left for the table */
            uint32_t c = 1;
            bool equal = false;
            if (mem.look_for_equal()) {
                const unsigned peers = __match_any_sync(kFull, in ? key : empty) &
                                       __ballot_sync(kFull, in);
                const bool merged = in && (peers & lanemask_lt);
                equal = __any_sync(kFull, merged);
                c = uint32_t(__popc(peers));
                in &= !merged;
            }
            mem.equal(equal);
            enqueue(in, key, c);
            return at < m;
        });
    }
    __syncthreads();
    /* ---- the cached keys ---- */
    {
        uint32_t at = uint32_t(wib) * 32u;
        probe([&]() {
            if (at >= entries) return false;
            const uint32_t e = at + uint32_t(lane);
            const K key = s_key[e];
            enqueue(key != empty, key, s_cnt[e]);
            at += uint32_t(kCountThreads);
            return at < entries;
        });
    }
    const uint32_t wjoin = __reduce_or_sync(kFull, join);
    const int wlive = int(__reduce_add_sync(kFull, unsigned(live_delta)));
    if (lane == 0) {
        join_status(t.status, wjoin);
        live_add(t, wlive);
    }
}

} // namespace b200
} // namespace warpcore

#endif /* WC_COUNT_CUH */
