/*
 * wc_multi.cuh -- lookups of the tables that hold several values per key
 * (multi-value, multi-bucket, bucket-list): the bulk num_values and the
 * bulk retrieve (multi_value_hash_table.cuh:371-520,
 * multi_bucket_hash_table.cuh:574-680, bucket_list_hash_table.cuh:337-466).
 * What differs between the tables, how a key's values are found and read,
 * comes from a Walk (MvWalk, MbWalk, BlWalk).
 *
 * The reference counts the values of every key, scans the counts into
 * offsets and walks every key again to copy its values.  Here two kernels
 * do it:
 *   multi_find_kernel counts.  A block takes a tile of keys, walks them and
 *     scans the counts in the block: every key gets its end offset within
 *     its tile, every tile its sum.  The block that finishes last turns the
 *     tiles' sums into the tiles' offsets.
 *   multi_values_kernel adds each tile's offset to its keys' offsets, walks
 *     the keys that have values, up to the window where the last of them is,
 *     and copies the values as it meets them.
 * No block waits for another: one walk may be as long as the whole table
 * (an absent key in a full one), and a slow tile then delays only the call.
 *
 * Both are bound by the latency of the walks' dependent reads.  A walk ends
 * at the first window with a free slot: at load 0.8 its mean is 2 to 3
 * windows and the longest of 32 is 8 to 9, so a warp that keeps one key per
 * lane until all are done leaves two lanes of three waiting.  Here each
 * lane issues one memory operation per step (a window, a bucket, a handle,
 * a list bucket) and a lane whose key is done draws the next key of the
 * block's tile.
 *
 * Shared memory is kept small on purpose: reads in flight need L1 space.
 * A form that noted the windows with values in shared memory while
 * counting, and copied from the notes without a second walk, needed 37 KiB
 * per block and ran slower the more blocks were resident (multi-value,
 * 2^23 lookups, half present with 4 values each: 736 / 859 / 1366 us with
 * 4 / 5 / 6 blocks per SM).
 */
#ifndef WC_MULTI_CUH
#define WC_MULTI_CUH

#include "wc_lane_kernels.cuh"
#include <warpcore/detail/mb_ops.cuh>

namespace warpcore {
namespace b200 {

/* resident 256-thread blocks per SM these kernels are built for */
#ifndef WC_MULTI_INSERT_BLOCKS
#define WC_MULTI_INSERT_BLOCKS 4
#endif
/* (count: u64 keys spill up to 120 bytes with 6 and are no slower for it: 2^22
 * lookups of multi-value u64 pairs 487 / 487 / 504 us with 6 / 5 / 4, multi-bucket
 * at CG 4 319 / 335 / 358, bucket list 293 / 294 / 309) */
#ifndef WC_MULTI_COUNT_BLOCKS
#define WC_MULTI_COUNT_BLOCKS 6
#endif
#ifndef WC_MULTI_VALUES_BLOCKS
#define WC_MULTI_VALUES_BLOCKS 5
#endif

/* what the bulk calls of all these tables pass */
struct MultiArgs {
    const void *keys;
    const void *values;             /* insert */
    void *values_out;               /* retrieve */
    unsigned long long *begin_out;  /* retrieve: offsets; NULL where begin_out
                                       would be end_out - 1 (begin_first) */
    unsigned long long *end_out;
    unsigned long long *begin_first;
    unsigned long long *counts_out; /* num_values: per key, or NULL */
    unsigned long long *look;       /* scratch words, see kLook* */
    void *status_out;
    uint64_t n;
    uint64_t max_windows;
    uint32_t tile;                  /* keys per tile */
    uint32_t bool_mask;
    int handler;
};

/* keys per tile: four per thread, so that a lane draws a few times before
 * the tile's last walks leave lanes idle */
constexpr int kMultiTile = 1024;
/* keys per tile of multi_find_kernel, whose last walks leave lanes idle at a
 * barrier (a quarter of its stalls at 1024 keys).  2048 where keys take 4
 * bytes and windows, of a width known here, at most 64; with more, the shared
 * memory of six blocks leaves L1 too small for the windows in flight (1024 /
 * 2048: u32 pairs 380 / 357 us, multi-bucket of u32 keys 586 / 550, u64 pairs
 * 280 / 436).  A run-time width (window_bytes 0) may be up to 128 bytes of
 * 4-byte keys: retrieves of multi-bucket tables at CG 4 / 16 / 32 259 / 283 / 370
 * us with 1024, 261 / 291 / 384 with 2048, of bucket lists 298 / 295 / 393 and
 * 306 / 305 / 407. */
constexpr int multi_find_tile(int key_bytes, int window_bytes)
{
    return key_bytes == 4 && window_bytes > 0 && window_bytes <= 64 ? 2 * kMultiTile : kMultiTile;
}
constexpr int kMultiThreads = 256;

/* scratch words: the next tile, the blocks that are done, the sum of all
 * counts, then (retrieve) one word per tile: its sum, later its offset.  The
 * first kLookTiles are zeroed before a call. */
constexpr int kLookTicket = 0, kLookDone = 1, kLookTotal = 2, kLookTiles = 4;

__device__ __forceinline__ void multi_write_status(const MultiArgs &a, uint64_t i, uint32_t st)
{
    if (!a.status_out) return;
    if (a.handler == kHandlerStatus)
        reinterpret_cast<uint32_t *>(a.status_out)[i] = st;
    else if (a.handler == kHandlerBoolean)
        reinterpret_cast<unsigned char *>(a.status_out)[i] =
            (unsigned char)((st & a.bool_mask) != 0);
}

/* exclusive scan over the block of one value per thread; returns the total */
__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long v,
                                                                   unsigned long long &excl)
{
    __shared__ unsigned long long warp_sums[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned long long w = lane < int(blockDim.x >> 5) ? warp_sums[lane] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, w, o);
            if (lane >= o) w += y;
        }
        warp_sums[lane] = w; /* inclusive over warps */
    }
    __syncthreads();
    const unsigned long long warp_base = wid ? warp_sums[wid - 1] : 0ull;
    excl = warp_base + x - v;
    const unsigned long long total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return total;
}

/* By the block that is done last: the tiles' sums to their offsets, in
 * place, and the sum of all.  The sums were written by other blocks of this
 * launch, each followed by a fence and the block's count in kLookDone. */
__device__ __forceinline__ void scan_tile_sums(unsigned long long *look, uint64_t ntiles)
{
    constexpr int kPer = 4;
    unsigned long long *const words = look + kLookTiles;
    unsigned long long before = 0;
    for (uint64_t at = 0; at < ntiles; at += uint64_t(blockDim.x) * kPer) {
        const uint64_t i0 = at + uint64_t(threadIdx.x) * kPer;
        unsigned long long c[kPer], sum = 0, excl = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            c[j] = i0 + j < ntiles ? __ldcg(words + i0 + j) : 0ull;
            sum += c[j];
        }
        const unsigned long long total = block_exclusive_scan(sum, excl);
        excl += before;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (i0 + j < ntiles) words[i0 + j] = excl;
            excl += c[j];
        }
        before += total;
    }
    if (threadIdx.x == 0) look[kLookTotal] = before;
}

/* A window of W keys read by one lane, loaded first and looked at later, so
 * that lanes doing other operations in the same step have theirs in flight
 * beside it.  A window of a known width comes in 32-byte loads, with one
 * compare per slot; the masks are built only where there is a match.  Other
 * widths are looked at as they are read. */
template <class K, int kW>
struct KeyWindow {
    static constexpr int WB = kW * int(sizeof(K));
    static constexpr bool kWords = kW > 0 && WB <= 128;
    using L = typename std::conditional<sizeof(K) == 4, LayoutSet32, LayoutSet64>::type;
    uint32_t w[kWords ? WB / 4 : 1];
    uint32_t hits, empties;

    __device__ __forceinline__ void load(const K *kw, uint32_t W, K key, K empty)
    {
        if constexpr (kWords) load_window<WB>(reinterpret_cast<const unsigned char *>(kw), w);
        else mb_window<K, kW>(kw, W, key, empty, hits, empties);
    }
    /* the slots that hold k */
    __device__ __forceinline__ uint32_t slots_of(K k, uint32_t seen) const
    {
        if constexpr (kWords) {
            uint32_t m = 0;
            if (has(k, seen)) {
#pragma unroll
                for (int i = 0; i < kW; ++i) m |= uint32_t(K(window_key<L>(w, i)) == k) << i;
            }
            return m;
        } else {
            return seen;
        }
    }
    __device__ __forceinline__ bool has(K k, uint32_t seen) const
    {
        if constexpr (kWords) {
            bool any = false;
#pragma unroll
            for (int i = 0; i < kW; ++i) any |= K(window_key<L>(w, i)) == k;
            return any;
        } else {
            return seen != 0;
        }
    }
    __device__ __forceinline__ uint32_t key_slots(K key) const { return slots_of(key, hits); }
    __device__ __forceinline__ uint32_t free_slots(K empty) const
    {
        return slots_of(empty, empties);
    }
    __device__ __forceinline__ bool any_free(K empty) const { return has(empty, empties); }
};

/* A lane's next key: the lanes of a warp without a key take the next ones
 * of the block's tile, `m` in all, in order.  `left` (uniform) turns false
 * with the last of them.  Returns whether this lane got key number `at`. */
__device__ __forceinline__ bool draw_key(bool has, int m, int *drawn, bool &left, int &at)
{
    const unsigned need = __ballot_sync(kFull, !has);
    if (!need || !left) return false;
    const int lane = threadIdx.x & 31;
    int from = 0;
    if (lane == 0) from = atomicAdd(drawn, __popc(need));
    from = __shfl_sync(kFull, from, 0);
    left = from + __popc(need) < m;
    if (has) return false;
    at = from + __popc(need & ((1u << lane) - 1u));
    return at < m;
}

/* num_values (kOffsets false): per-key counts, written as the walks end, and
 * their sum; the first half of retrieve (kOffsets): end offsets within the
 * tiles, the tiles' offsets and the sum.  (With a scan of every tile for the
 * sum alone, num_values of 4 M u32 keys in a multi-bucket table took 107 us, in
 * a bucket list 104; 94 and 93 without.) */
template <class Walk, bool kOffsets>
__global__ void __launch_bounds__(kMultiThreads, WC_MULTI_COUNT_BLOCKS)
    multi_find_kernel(const typename Walk::Args a)
{
    using K = typename Walk::key_t;
    constexpr int kTile = Walk::kFindTile;
    __shared__ K s_key[kTile];
    /* counts, then end offsets in the tile */
    __shared__ unsigned long long s_end[kOffsets ? kTile : 1];
    __shared__ int s_drawn;
    __shared__ uint64_t s_tile;

    const int lane = threadIdx.x & 31;
    const uint64_t ntiles = (a.n + a.tile - 1) / a.tile;
    const K *const keys = reinterpret_cast<const K *>(a.keys);
    const K empty = K(Walk::view(a).empty_key), tomb = K(Walk::view(a).tombstone_key);
    uint32_t join = 0;
    unsigned long long all = 0; /* num_values: this lane's counts */
    auto counted = [&](uint64_t base, int at, uint64_t num) {
        if constexpr (kOffsets) {
            s_end[at] = num;
        } else {
            all += num;
            if (a.counts_out) a.counts_out[base + uint64_t(at)] = num;
        }
    };

    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = atomicAdd(a.look + kLookTicket, 1ull);
            s_drawn = 0;
        }
        __syncthreads();
        const uint64_t tile = s_tile;
        if (tile >= ntiles) break;
        const uint64_t base = tile * a.tile;
        const int m = int(a.n - base < a.tile ? a.n - base : a.tile);
        for (int i = threadIdx.x; i < m; i += kMultiThreads) s_key[i] = ld_stream(keys + base + i);
        __syncthreads();

        /* ---- walk the keys ---- */
        {
            bool has = false, left = true;
            int at = 0;
            K key = 0;
            typename Walk::State s;
            for (;;) {
                if (draw_key(has, m, &s_drawn, left, at)) {
                    key = s_key[at];
                    if (key == empty || key == tomb) {
                        counted(base, at, 0);
                        join |= kStInvalidKey;
                        multi_write_status(a, base + uint64_t(at), kStInvalidKey);
                    } else {
                        has = true;
                        Walk::start(a, key, s);
                    }
                }
                if (!left && !__any_sync(kFull, has)) break;
                uint32_t st = kStNone;
                if (has && Walk::count_step(a, key, s, st)) {
                    counted(base, at, s.num);
                    join |= st;
                    multi_write_status(a, base + uint64_t(at), st);
                    has = false;
                }
            }
        }
        __syncthreads();

        if constexpr (kOffsets) {
            constexpr int kPer = kTile / kMultiThreads;
            unsigned long long c[kPer], sum = 0, excl = 0;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int i = int(threadIdx.x) * kPer + j;
                c[j] = i < m ? s_end[i] : 0ull;
                sum += c[j];
            }
            const unsigned long long total = block_exclusive_scan(sum, excl);
            if (threadIdx.x == 0) {
                a.look[kLookTiles + tile] = total;
                __threadfence();
            }
            unsigned long long run = excl;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                run += c[j];
                const int i = int(threadIdx.x) * kPer + j;
                if (i < m) s_end[i] = run;
            }
            __syncthreads();
            for (int i = threadIdx.x; i < m; i += kMultiThreads)
                a.end_out[base + uint64_t(i)] = s_end[i];
        }
        __syncthreads(); /* the shared rows are rewritten by the next tile */
    }
    const uint32_t wj = __reduce_or_sync(kFull, join);
    if (lane == 0) join_status(Walk::view(a).status, wj);
    if constexpr (kOffsets) {
        if (threadIdx.x == 0) {
            const bool last = atomicAdd(a.look + kLookDone, 1ull) + 1 == gridDim.x;
            __threadfence();
            s_drawn = int(last);
        }
        __syncthreads();
        if (s_drawn) scan_tile_sums(a.look, ntiles);
    } else {
        all = warp_sum_u64(all);
        if (lane == 0 && all) atomicAdd(a.look + kLookTotal, all);
    }
}

/* the second half of retrieve, with the tiles of the first: the keys'
 * offsets, and every key's values, inside its own segment [begin, end) only.
 * A tile is taken kMultiTile keys at a time; those without values are dropped
 * first. */
template <class Walk>
__global__ void __launch_bounds__(kMultiThreads, WC_MULTI_VALUES_BLOCKS)
    multi_values_kernel(const typename Walk::Args a)
{
    using K = typename Walk::key_t;
    using V = typename Walk::val_t;
    __shared__ K s_key[kMultiTile];
    __shared__ unsigned long long s_begin[kMultiTile], s_room[kMultiTile];
    __shared__ int s_drawn, s_found;

    const int lane = threadIdx.x & 31;
    const K *const keys = reinterpret_cast<const K *>(a.keys);
    if (a.begin_first && blockIdx.x == 0 && threadIdx.x == 0) *a.begin_first = 0;
    const uint64_t ntiles = (a.n + a.tile - 1) / a.tile;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t tile_base = tile * a.tile;
        const int tile_m = int(a.n - tile_base < a.tile ? a.n - tile_base : a.tile);
        const unsigned long long before = a.look[kLookTiles + tile];
        unsigned long long part_begin = 0; /* of the part, within the tile */
        for (int part = 0; part < tile_m; part += kMultiTile) {
            const uint64_t base = tile_base + uint64_t(part);
            const int m = tile_m - part < kMultiTile ? tile_m - part : kMultiTile;
            if (threadIdx.x == 0) {
                s_drawn = 0;
                s_found = 0;
            }
            /* ends within the tile; the loads of all rows before any store */
            constexpr int kPer = kMultiTile / kMultiThreads;
            unsigned long long begin[kPer], end[kPer];
            const unsigned long long part_end = a.end_out[base + uint64_t(m - 1)];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int i = int(threadIdx.x) + j * kMultiThreads;
                end[j] = i < m ? a.end_out[base + uint64_t(i)] : 0ull;
                begin[j] = i > 0 && i < m ? a.end_out[base + uint64_t(i) - 1] : part_begin;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int i = int(threadIdx.x) + j * kMultiThreads;
                const unsigned long long room = i < m ? end[j] - begin[j] : 0ull;
                if (i < m) {
                    a.end_out[base + uint64_t(i)] = before + end[j];
                    if (a.begin_out) a.begin_out[base + uint64_t(i)] = before + begin[j];
                }
                const unsigned found = __ballot_sync(kFull, room != 0);
                int p = 0;
                if (lane == 0 && found) p = atomicAdd(&s_found, __popc(found));
                p = __shfl_sync(kFull, p, 0) + __popc(found & ((1u << lane) - 1u));
                if (room) {
                    s_key[p] = ld_stream(keys + base + uint64_t(i));
                    s_begin[p] = before + begin[j];
                    s_room[p] = room;
                }
            }
            part_begin = part_end;
            __syncthreads();
            const int n = s_found;
            bool has = false, left = n > 0;
            int at = 0;
            K key = 0;
            V *out = nullptr;
            uint64_t room = 0;
            typename Walk::State s;
            while (left || __any_sync(kFull, has)) {
                if (draw_key(has, n, &s_drawn, left, at)) {
                    key = s_key[at];
                    out = reinterpret_cast<V *>(a.values_out) + s_begin[at];
                    room = s_room[at];
                    has = true;
                    Walk::start(a, key, s);
                }
                if (has && Walk::value_step(a, key, s, out, room)) has = false;
            }
            __syncthreads(); /* the shared rows are rewritten by the next part */
        }
    }
}

/* Bulk insert.  Each warp owns a contiguous range of the input and reads
 * it one 32-key buffer ahead; each lane holds one (key, value) and issues
 * one memory operation per step (Walk::issue: a window read or a claim's
 * compare-and-swap), all lanes' operations being in flight together before
 * any is looked at (Walk::look).  A lane whose pair is done takes the next
 * one, so no lane waits for the longest walk of its warp.  Measured on the
 * multi-value table (u32 pairs, 2^24 into 168 MB, four values per key): 981
 * us with one pair per lane until the warp was done, 679 now.  Used where a
 * step has two kinds: with the four or five kinds of a multi-bucket or
 * bucket-list insert, a warp runs most kinds in every step, so those tables
 * have kernels of their own. */
template <class Walk>
__global__ void __launch_bounds__(256, Walk::kInsertBlocks)
    multi_insert_kernel(const typename Walk::Args a)
{
    using K = typename Walk::key_t;
    using V = typename Walk::val_t;
    const int lane = threadIdx.x & 31;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    const uint32_t m = uint32_t(wb + per < a.n ? per : a.n - wb); /* pairs of this warp */

    const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;
    const V *const vals = reinterpret_cast<const V *>(a.values) + wb;
    uint32_t pf_base = 0, cursor = 0;
    K pfA = K(0), pfB = K(0);
    V pvA = V(0), pvB = V(0);
    if (uint32_t(lane) < m) {
        pfA = ld_stream(keys + lane);
        pvA = ld_stream(vals + lane);
    }
    if (32 + uint32_t(lane) < m) {
        pfB = ld_stream(keys + 32 + lane);
        pvB = ld_stream(vals + 32 + lane);
    }

    bool has = false;
    uint32_t at = 0;
    K key = K(0);
    V val = V(0);
    typename Walk::InsertState s;
    uint32_t join = 0;
    typename Walk::Counts counts = {};
    for (;;) {
        /* ---- lanes without a pair take the next ones, in input order ---- */
        const unsigned need = __ballot_sync(kFull, !has);
        const uint32_t idle = uint32_t(__popc(need)), avail = m - cursor;
        const uint32_t take = idle < avail ? idle : avail;
        if (take == 0 && need == kFull) break;
        if (take) {
            const uint32_t r = uint32_t(__popc(need & lanemask_lt));
            const uint32_t off = cursor - pf_base + r; /* < 64 for lanes that take one */
            const K ka = shfl_any(pfA, int(off & 31)), kb = shfl_any(pfB, int(off & 31));
            const V va = shfl_any(pvA, int(off & 31)), vb = shfl_any(pvB, int(off & 31));
            if (!has && r < take) {
                key = off < 32 ? ka : kb;
                val = off < 32 ? va : vb;
                at = cursor + r;
                const uint32_t st = Walk::insert_start(a, key, val, s);
                has = st == kStNone;
                if (!has) {
                    join |= st;
                    multi_write_status(a, wb + at, st);
                }
            }
            cursor += take;
            if (cursor - pf_base >= 32) {
                pf_base += 32;
                pfA = pfB;
                pvA = pvB;
                const uint32_t nx = pf_base + 32 + uint32_t(lane);
                if (nx < m) {
                    pfB = ld_stream(keys + nx);
                    pvB = ld_stream(vals + nx);
                }
            }
        }

        typename Walk::InsertIo io;
        if (has) Walk::issue(a, key, val, s, io);
        uint32_t st = kStNone;
        if (has && Walk::look(a, key, val, s, io, st, join, counts)) {
            multi_write_status(a, wb + at, st);
            has = false;
        }
    }
    const uint32_t wj = __reduce_or_sync(kFull, join);
    if (lane == 0) join_status(Walk::view(a).status, wj);
    Walk::add_counts(a, counts);
}

/* dry run of retrieve: every key's status is dry_run */
template <int kUnused = 0>
__global__ void __launch_bounds__(256) multi_dry_status_kernel(void *status_out, uint64_t n,
                                                               int handler, uint32_t bool_mask)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (handler == kHandlerStatus)
            reinterpret_cast<uint32_t *>(status_out)[i] = kStDryRun;
        else if (handler == kHandlerBoolean)
            reinterpret_cast<unsigned char *>(status_out)[i] =
                (unsigned char)((kStDryRun & bool_mask) != 0);
    }
}

} // namespace b200
} // namespace warpcore

#endif /* WC_MULTI_CUH */
