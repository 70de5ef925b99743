/*
 * wc_lane_kernels.cuh -- whole-window probing with one key per lane.
 *
 * Same bucket sequence, claim order (lowest free slot of a window first),
 * statuses and results as table_op_kernel (wc_kernels.cuh); the difference
 * is who reads a window.  table_op_kernel lets TPK lanes read one window
 * together and returns match / free masks to the owner lane with ballots:
 * for u64 pairs at CG 8 (TPK 8) a warp then spends about 35 instructions
 * per key on rounds of ballots and shuffles, and at 50 % issue-active the
 * insert is bound by instruction issue, not by memory.  Here every lane
 * reads its own key's window with 32-byte vector loads (sm_100; four for a
 * 128-byte window), tests the window's slots in registers and issues its
 * own compare-and-swap: no ballots, no shuffles, no shared memory.
 *
 * Each lane issues one memory operation per wave, a window read or a
 * claim's compare-and-swap, so a warp keeps 32 of them in flight.  A window
 * is looked at with one compare and at most two selects per slot, in four
 * chains for lookups, and places in the warp's range are 32 bits wide; with
 * masks of all slots and 64-bit places, u32 pairs took 137 / 144 us (insert
 * of 4 M / lookup of 8 M, load 0.76) against 131 / 121 now, a u32 set 213
 * against 187 (lookup of 16 M), mixed 4- and 8-byte pairs 66 against 68.  Keys are
 * refilled in input order from a double-buffered prefetch of the warp's
 * contiguous key range, as in table_op_kernel.  Equal keys need no merging
 * for their slots: every claim goes to the lowest free slot of the
 * window its lane read, so two claims of one key meet on one slot, and the
 * compare-and-swap that loses sees the key.  A claim that loses its slot to
 * another key reads the window again.
 *
 * Insert, retrieve and erase; counting inserts without statuses have a kernel
 * of this form with a count cache (wc_count.cuh), the others table_op_kernel.
 */
#ifndef WC_LANE_KERNELS_CUH
#define WC_LANE_KERNELS_CUH

#include "wc_kernels.cuh"

namespace warpcore {
namespace b200 {

/* resident 256-thread blocks per SM the lane kernels are built for: 4 for
 * u32 pairs with windows of at most 64 bytes (64 registers, no spills; the
 * u32/u32 insert of 2^20 keys into 2 097 496 slots ran 21.2-21.4 against
 * 20.2 G keys/s with 3, the retrieve unchanged, and 5 spilled and lost),
 * 3 elsewhere, where 4 spills */
template <class L, int W>
constexpr int lane_min_blocks()
{
    return (L::kSlotBytes == 8 && L::kHasValue && W * L::kSlotBytes <= 64) ? 4 : 3;
}

/* a bucket's window of WB bytes, read by one lane from L2 (.cg: a claim by
 * another lane is seen): 32-byte vector loads for windows of 32 bytes or
 * more, else one load of the window */
template <int WB>
__device__ __forceinline__ void load_window(const unsigned char *p, uint32_t (&w)[WB / 4])
{
    if constexpr (WB >= 32) {
#pragma unroll
        for (int c = 0; c < WB / 32; ++c) {
            asm volatile("ld.global.cg.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(w[8 * c + 0]), "=r"(w[8 * c + 1]), "=r"(w[8 * c + 2]),
                           "=r"(w[8 * c + 3]), "=r"(w[8 * c + 4]), "=r"(w[8 * c + 5]),
                           "=r"(w[8 * c + 6]), "=r"(w[8 * c + 7])
                         : "l"(p + 32 * c));
        }
    } else if constexpr (WB == 16) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(p));
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (WB == 8) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2 *>(p));
        w[0] = v.x; w[1] = v.y;
    } else {
        w[0] = __ldcg(reinterpret_cast<const unsigned int *>(p));
    }
}

/* key / payload of slot s of a window held as 32-bit words */
template <class L>
__device__ __forceinline__ typename L::key_t window_key(const uint32_t *w, int s)
{
    using K = typename L::key_t;
    constexpr int SB = L::kSlotBytes;
    if constexpr (SB == 16) {
        if constexpr (sizeof(K) == 8) return uint64_t(w[4 * s]) | (uint64_t(w[4 * s + 1]) << 32);
        else return w[4 * s];
    } else if constexpr (SB == 8 && L::kHasValue) {
        return w[2 * s];
    } else if constexpr (SB == 8) {
        return uint64_t(w[2 * s]) | (uint64_t(w[2 * s + 1]) << 32);
    } else {
        return w[s];
    }
}

template <class L>
__device__ __forceinline__ typename L::val_t window_val(const uint32_t *w, int s)
{
    using V = typename L::val_t;
    constexpr int SB = L::kSlotBytes;
    if constexpr (SB == 16) {
        if constexpr (sizeof(V) == 8) return uint64_t(w[4 * s + 2]) | (uint64_t(w[4 * s + 3]) << 32);
        else return w[4 * s + 2];
    } else if constexpr (SB == 8 && L::kHasValue) {
        return w[2 * s + 1];
    } else {
        return 0;
    }
}

/* payload of slot `target` (a run-time index): selected by an unrolled
 * loop, so that the window stays in registers */
template <class L, int W>
__device__ __forceinline__ typename L::val_t window_val_at(const uint32_t *w, int target)
{
    typename L::val_t v = 0;
#pragma unroll
    for (int s = 0; s < W; ++s)
        if (s == target) v = window_val<L>(w, s);
    return v;
}

/* Streams of repeated keys.  A lane reads a window of 128 bytes in four
 * requests, a group of lanes in one, and where many warps read and write one
 * hot window the requests queue at its place in L2 (about 20 ns each).  So an
 * insert with such windows looks for repeated keys among the first kSkewKeys
 * keys of the block's warps (a table of recent keys in shared memory); from
 * kSkewMin of them on, a warp gives the rest of its range to group_range.
 * Distinct keys never get there.  Equal keys among a warp's first kSkewKeys
 * are merged, with the value of the last, as group_range does: a call of at
 * most 32 keys stores each key's last value.  1.9 M inserts into 40 MB of u64
 * pairs, lanes only / groups only / this: distinct keys 91 / 123 / 95 us,
 * Zipf(0.8) 1 688 / 1 098 / 1 227, Zipf(1.1) 5 165 / 3 540 / 3 320, one key
 * 4 870 / 2 760 / 2 970; u64 set at CG 16: 76 / 133 / 79, 126 / 104 / 115, 179 / 97 /
 * 110, 154 / 55 / 55.  (Looking at 64 keys: Zipf(1.1) 3 815, distinct 98.) */
constexpr uint32_t kSkewKeys = 32;
constexpr uint32_t kSkewMin = 3;
constexpr int kSkewSeenBits = 9, kSkewSeen = 1 << kSkewSeenBits;
template <int WB, int OP>
constexpr bool lane_looks_for_skew()
{
    return OP == kOpInsert && WB > 64;
}

template <class L, int W, int OP>
__global__ void __launch_bounds__(256, lane_min_blocks<L, W>()) lane_op_kernel(const TableOpArgs a)
{
    using K = typename L::key_t;
    using V = typename L::val_t;
    constexpr int SB = L::kSlotBytes;
    constexpr int WB = W * SB;
    static_assert(WB <= 128 && WB >= 4, "window of one lane");
    static_assert(OP == kOpInsert || OP == kOpRetrieve || OP == kOpErase, "operation");
    constexpr bool kValueIn = OP == kOpInsert && L::kHasValue;
    constexpr bool kSkew = lane_looks_for_skew<WB, OP>();
    __shared__ K s_seen[kSkew ? kSkewSeen : 1];
    __shared__ uint32_t s_twice;
    __shared__ uint64_t sh_bucket[kSkew ? 8 : 1][32];
    __shared__ K sh_key[kSkew ? 8 : 1][32];
    __shared__ uint32_t sh_off[kSkew ? 8 : 1][32];

    const TableView &t = a.t;
    const int lane = threadIdx.x & 31;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;

    /* this warp's contiguous range of keys */
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    uint32_t m = uint32_t(wb + per < a.n ? per : a.n - wb);
    const uint32_t m_all = m;

    const K empty = K(t.empty_key);
    const K tomb = K(t.tombstone_key);
    unsigned char *const slots = reinterpret_cast<unsigned char *>(t.slots);
    const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;
    const V *const vals_in = reinterpret_cast<const V *>(a.values) + (kValueIn ? wb : 0);

    if constexpr (kSkew) {
        for (int i = threadIdx.x; i < kSkewSeen; i += blockDim.x) s_seen[i] = empty;
        if (threadIdx.x == 0) s_twice = 0;
        __syncthreads();
    }

    uint32_t pf_base = 0, cursor = 0;
    K pfA = uint32_t(lane) < m ? ld_stream(keys + lane) : empty;
    K pfB = 32 + uint32_t(lane) < m ? ld_stream(keys + 32 + lane) : empty;
    V pvA = 0, pvB = 0;
    if constexpr (kValueIn) {
        if (uint32_t(lane) < m) pvA = ld_stream(vals_in + lane);
        if (32 + uint32_t(lane) < m) pvB = ld_stream(vals_in + 32 + lane);
    }

    /* the key this lane owns: waiting for its window (claim < 0) or for the
     * compare-and-swap on slot `claim` of it, expected to hold the empty key
     * with payload claim_expect */
    bool has = false;
    int claim = -1;
    V claim_expect = 0;
    uint32_t at = 0; /* the key's place in the warp's range */
    uint64_t bucket = 0, step = 0, wins = 0;
    K key = empty;
    V val = 0;
    uint32_t join = 0;
    int live_delta = 0;

    /* a key is done: its flag (sets) and its status */
    auto finish = [&](uint32_t st, bool flag) {
        if constexpr (OP == kOpRetrieve) {
            if (a.is_set && st == kStNone)
                reinterpret_cast<unsigned char *>(a.out)[wb + at] = (unsigned char)flag;
        }
        if (a.status_out) {
            if (a.handler == kHandlerStatus)
                st_stream(reinterpret_cast<uint32_t *>(a.status_out) + wb + at, st);
            else if (a.handler == kHandlerBoolean)
                reinterpret_cast<unsigned char *>(a.status_out)[wb + at] =
                    (unsigned char)((st & a.bool_mask) != 0);
        }
        has = false;
    };

    for (;;) {
        /* ---- refill lanes whose key is done, in input order ---- */
        const unsigned need = __ballot_sync(kFull, !has);
        const uint32_t idle = uint32_t(__popc(need)), avail = m - cursor;
        const uint32_t take = idle < avail ? idle : avail;
        if (take == 0 && need == kFull) break;
        if (take) {
            const uint32_t r = uint32_t(__popc(need & lanemask_lt));
            const uint32_t off = cursor - pf_base + r; /* < 64 for refilling lanes */
            bool fresh = false;
            const K ka = shfl_any(pfA, int(off & 31u));
            const K kb = shfl_any(pfB, int(off & 31u));
            V va = 0, vb = 0;
            if constexpr (kValueIn) {
                va = shfl_any(pvA, int(off & 31u));
                vb = shfl_any(pvB, int(off & 31u));
            }
            if (!has && r < take) {
                key = off < 32 ? ka : kb;
                if constexpr (kValueIn) val = off < 32 ? va : vb;
                at = cursor + r;
                has = true;
                claim = -1;
                wins = 0;
                step = 0;
                fresh = key != empty && key != tomb;
                if (!fresh) {
                    join |= kStInvalidKey;
                    finish(kStInvalidKey, false);
                }
            }
            if constexpr (kSkew) {
                if (cursor < kSkewKeys) {
                    const unsigned peers = merge_equal_keys<K, V, kValueIn>(fresh, key, empty, val);
                    bool twice = false;
                    if (fresh) {
                        volatile K *const seen =
                            s_seen + (uint64_t(key) * 0x9E3779B97F4A7C15ull >> (64 - kSkewSeenBits));
                        twice = *seen == key || (peers & lanemask_lt);
                        *seen = key;
                        if (peers & lanemask_lt) {
                            join |= kStDuplicateKey;
                            finish(kStDuplicateKey, false);
                            fresh = false;
                        }
                    }
                    const unsigned tw = __ballot_sync(kFull, twice);
                    if (lane == 0 && tw) atomicAdd(&s_twice, uint32_t(__popc(tw)));
                }
            }
            if (fresh) bucket = probe_begin<K>(t, key);
            cursor += take;
            if (cursor - pf_base >= 32) {
                pf_base += 32;
                pfA = pfB;
                pvA = pvB;
                const uint32_t nx = pf_base + 32 + uint32_t(lane);
                if (nx < m) {
                    pfB = ld_stream(keys + nx);
                    if constexpr (kValueIn) pvB = ld_stream(vals_in + nx);
                }
                if constexpr (kSkew) {
                    if (cursor >= kSkewKeys &&
                        *reinterpret_cast<volatile uint32_t *>(&s_twice) >= kSkewMin)
                        m = cursor; /* the rest goes through group_range */
                }
            }
        }

        /* ---- one memory operation per lane with a key: its window, or its
         * claim; all lanes' operations are in flight together ---- */
        unsigned char *const bptr = slots + bucket * uint64_t(WB);
        uint32_t w[WB / 4];
        K cas_old = empty;
        V cas_old_payload = 0;
        if (has) {
            if constexpr (OP == kOpInsert) {
                if (claim >= 0)
                    cas_old = cas_slot<L>(bptr + claim * SB, empty, claim_expect, key, val,
                                          &cas_old_payload);
                else
                    load_window<WB>(bptr, w);
            } else {
                load_window<WB>(bptr, w);
            }
        }
        if (!has) continue;

        if constexpr (OP == kOpInsert) {
            if (claim >= 0) {
                if (cas_old == empty && cas_old_payload == claim_expect) {
                    fp_store(t, bucket * W + uint64_t(claim), fingerprint(key));
                    ++live_delta;
                    finish(kStNone, false);
                } else if (cas_old == key) {
                    join |= kStDuplicateKey;
                    store_value<L>(bptr + claim * SB, val);
                    finish(kStDuplicateKey, false);
                } else if (cas_old == empty) {
                    claim_expect = cas_old_payload; /* free slot, stale payload: again */
                } else {
                    claim = -1; /* taken by another key: read the window again */
                }
                continue;
            }
        }

        /* the slot that holds the key, a free slot: one compare and one or
         * two selects per slot, no masks */
        bool hit = false, any_free = false;
        if constexpr (OP == kOpRetrieve) {
            /* four chains of compares side by side */
            bool h[4] = {false, false, false, false}, f[4] = {false, false, false, false};
            V x[4] = {0, 0, 0, 0};
#pragma unroll
            for (int s = 0; s < W; ++s) {
                const K sk = window_key<L>(w, s);
                f[s & 3] |= sk == empty;
                h[s & 3] |= sk == key;
                if constexpr (L::kHasValue) x[s & 3] = sk == key ? window_val<L>(w, s) : x[s & 3];
            }
            hit = h[0] | h[1] | h[2] | h[3];
            any_free = f[0] | f[1] | f[2] | f[3];
            V v = x[0] | x[1] | x[2] | x[3]; /* a key has one slot */
            if (hit || any_free) {
                if constexpr (L::kHasValue) {
                    if (hit && !a.is_set) {
                        if (uint64_t(v) > t.max_count) v = V(t.max_count);
                        st_stream(reinterpret_cast<V *>(a.out) + wb + at, v);
                    }
                }
                const uint32_t st = hit || a.is_set ? kStNone : kStKeyNotFound;
                join |= st;
                finish(st, hit);
                continue;
            }
        } else {
            int hs = 0;
#pragma unroll
            for (int s = W - 1; s >= 0; --s) {
                const K sk = window_key<L>(w, s);
                if (sk == key) {
                    hit = true;
                    hs = s;
                }
                if constexpr (OP == kOpInsert) {
                    if (sk == empty) { /* the lowest free slot is left over */
                        any_free = true;
                        claim = s;
                        claim_expect = window_val<L>(w, s);
                    }
                } else {
                    any_free |= sk == empty;
                }
            }
            if (hit) {
                unsigned char *const sp = bptr + hs * SB;
                if constexpr (OP == kOpInsert) {
                    join |= kStDuplicateKey;
                    store_value<L>(sp, val);
                    finish(kStDuplicateKey, false);
                } else {
                    if (erase_slot<L>(sp, key, tomb)) {
                        fp_store(t, bucket * W + uint64_t(hs), kFpTomb);
                        --live_delta;
                    }
                    finish(kStNone, false);
                }
                continue;
            }
        }
        if (any_free) {
            if constexpr (OP == kOpErase) finish(a.is_set ? kStNone : kStKeyNotFound, false);
            continue; /* insert: the claim follows in the next wave */
        }
        if (++wins >= a.max_windows) {
            if constexpr (OP == kOpErase) {
                finish(a.is_set ? kStNone : kStProbingLengthExceeded, false);
            } else {
                join |= kStProbingLengthExceeded;
                finish(kStProbingLengthExceeded, false);
            }
        } else {
            if (wins == 1) step = probe_step<K>(t, key);
            bucket = probe_next(t, bucket, step);
        }
    }
    if constexpr (kSkew) {
        if (m < m_all) {
            const int wib = threadIdx.x >> 5;
            group_range<L, W, OP>(a, wb + m, wb + m_all, sh_bucket[wib], sh_key[wib], sh_off[wib],
                                  static_cast<K *>(nullptr), static_cast<V *>(nullptr), false, join,
                                  live_delta);
        }
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

#endif /* WC_LANE_KERNELS_CUH */
