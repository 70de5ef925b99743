/*
 * wc_fp_kernels.cuh -- fingerprint-first bulk kernels for tables that keep
 * one fingerprint byte per slot (b200_core.cuh, "fingerprints").
 *
 * The bucket sequence, the slot order of claims and every per-key status
 * are those of table_op_kernel (wc_kernels.cuh); only what is read per
 * bucket differs.  table_op_kernel reads each bucket's whole window of
 * slots (128 B for u64 pairs at CG 8).  This kernel reads the bucket's
 * cg_size fingerprint bytes and then only the slots whose fingerprint
 * equals the key's:
 *   - a miss at load 0.9 costs ~2.9 fingerprint words instead of ~2.9
 *     windows, and the fingerprint array (1 byte per slot, 1/16 of a u64
 *     pair table) mostly stays in L2;
 *   - a hit costs the fingerprint words plus one slot, read with an
 *     evict-first hint so that slot lines do not push fingerprints out
 *     (retrieve), or from L2 without an L1 copy (inserts: a claim's
 *     compare-and-swap lands in L2, and an equal key's lane must see it;
 *     erase: its compare-and-swap on the slot follows, with the words read
 *     as the expected value).
 *
 * Inserts run fp_insert_kernel, retrieve and erase fp_find_kernel, counting
 * inserts fp_count_kernel (or count_insert_kernel, wc_count.cuh).
 *
 * Each lane owns one key and issues one memory operation per wave: a
 * fingerprint load, a candidate slot load, or a compare-and-swap claim.
 * The 32 lanes' operations are independent, so a warp keeps 32 requests in
 * flight.  Keys are refilled in input order from a double-buffered
 * prefetch; inserts merge equal keys of a refill.
 */
#ifndef WC_FP_KERNELS_CUH
#define WC_FP_KERNELS_CUH

#include "wc_kernels.cuh"

namespace warpcore {
namespace b200 {

/* resident 256-thread blocks per SM the fingerprint kernels are compiled
 * for: inserts (which hold a key, a value and a claim in flight) and the
 * read-only retrieve / erase, which gain from more warps in flight */
#ifndef WC_FP_MIN_BLOCKS
#define WC_FP_MIN_BLOCKS 4
#endif
#ifndef WC_FP_MIN_BLOCKS_READ
#define WC_FP_MIN_BLOCKS_READ 6
#endif

/* L2 eviction priorities: fingerprint lines are loaded and stored with
 * evict_last and slot lines read by retrieve with evict_first (ld.cs),
 * so that the
 * random slot traffic of a table larger than L2 evicts slot lines before
 * fingerprint lines (a fingerprint byte written into an evicted sector
 * costs a DRAM read to merge). */

__device__ __forceinline__ uint64_t l2_policy_evict_last()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ uint32_t ld_hint_u32(const void *p, uint64_t pol)
{
    uint32_t v;
    asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint2 ld_hint_v2(const void *p, uint64_t pol)
{
    uint2 v;
    asm volatile("ld.global.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
                 : "=r"(v.x), "=r"(v.y) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint4 ld_hint_v4(const void *p, uint64_t pol)
{
    uint4 v;
    asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t ld_hint_u16(const void *p, uint64_t pol)
{
    uint16_t v;
    asm volatile("ld.global.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t ld_hint_u8(const void *p, uint64_t pol)
{
    uint16_t v;
    asm volatile("ld.global.L2::cache_hint.u8 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ void st_hint_u8(void *p, uint32_t v, uint64_t pol)
{
    asm volatile("st.global.L2::cache_hint.u8 [%0], %1, %2;" ::"l"(p), "h"(uint16_t(v)), "l"(pol)
                 : "memory");
}

/* 4 bytes of 0x00 / 0xff (a __vcmpeq4 result) to 4 bits, byte k -> bit k:
 * the multiplier moves bit 7 + 8k to bit 28 + k with no two terms meeting */
__device__ __forceinline__ uint32_t pack_bytes4(uint32_t v)
{
    return ((v & 0x80808080u) * 0x00204081u) >> 28;
}

/* load the W fingerprint bytes of a bucket; bit s of `match` / `empty`
 * says whether slot s holds fingerprint fp / is empty */
template <int W>
__device__ __forceinline__ void fp_masks(const unsigned char *p, uint32_t fp, uint32_t &match,
                                         uint32_t &empty, uint64_t pol)
{
    const uint32_t pat = fp * 0x01010101u;
    if constexpr (W >= 4) {
        constexpr int NW = W / 4;
        uint32_t w[NW];
        if constexpr (W == 4) {
            w[0] = ld_hint_u32(p, pol);
        } else if constexpr (W == 8) {
            const uint2 v = ld_hint_v2(p, pol);
            w[0] = v.x;
            w[1] = v.y;
        } else {
#pragma unroll
            for (int h = 0; h < W / 16; ++h) {
                const uint4 v = ld_hint_v4(p + 16 * h, pol);
                w[4 * h + 0] = v.x;
                w[4 * h + 1] = v.y;
                w[4 * h + 2] = v.z;
                w[4 * h + 3] = v.w;
            }
        }
        match = 0;
        empty = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            match |= pack_bytes4(__vcmpeq4(w[k], pat)) << (4 * k);
            empty |= pack_bytes4(__vcmpeq4(w[k], 0u)) << (4 * k);
        }
    } else {
        const uint32_t x = W == 2 ? ld_hint_u16(p, pol) : ld_hint_u8(p, pol);
        constexpr uint32_t lim = (1u << W) - 1u; /* the zero bytes above W are not slots */
        match = pack_bytes4(__vcmpeq4(x, pat)) & lim;
        empty = pack_bytes4(__vcmpeq4(x, 0u)) & lim;
    }
}

/* one slot, read once: evict-first, so that the fingerprints stay in L2 */
template <class L>
__device__ __forceinline__ LaneWords load_slot_once(const unsigned char *sp)
{
    LaneWords r{{0u, 0u, 0u, 0u}};
    if constexpr (L::kSlotBytes == 16) {
        const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(sp));
        r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w;
    } else if constexpr (L::kSlotBytes == 8) {
        const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(sp));
        r.w[0] = v.x; r.w[1] = v.y;
    } else {
        r.w[0] = __ldcs(reinterpret_cast<const unsigned int *>(sp));
    }
    return r;
}

/* Counting insert.  The steps of a wave (fingerprints, slot, claim) run one
 * after the other; duplicates in one refill are merged with __match_any_sync,
 * and without per-key statuses keys go through the per-block count cache, both
 * as in table_op_kernel. */
template <class L, int W>
__global__ void __launch_bounds__(256, WC_FP_MIN_BLOCKS) fp_count_kernel(const TableOpArgs a)
{
    using K = typename L::key_t;
    using V = typename L::val_t;
    constexpr int SB = L::kSlotBytes;
    enum : int { kPhaseFps = 0, kPhaseCheck = 1, kPhaseClaim = 2, kPhasePreload = 3 };
    const bool preload = (a.flags & kFlagPreloadClaim) != 0;
    const uint64_t pol_keep = l2_policy_evict_last(); /* fingerprint lines */

    const TableView &t = a.t;
    const int lane = threadIdx.x & 31;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;

    /* this warp's contiguous range of keys */
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    const uint64_t we = wb + per < a.n ? wb + per : a.n;

    const K empty = K(t.empty_key);
    const K tomb = K(t.tombstone_key);
    unsigned char *const slots = reinterpret_cast<unsigned char *>(t.slots);
    const K *const keys = reinterpret_cast<const K *>(a.keys);

    uint64_t pf_base = wb;
    K pfA = (wb + lane < we) ? ld_stream(keys + wb + lane) : empty;
    K pfB = (wb + 32 + lane < we) ? ld_stream(keys + wb + 32 + lane) : empty;
    uint64_t cursor = wb;

    bool has = false, pending = false;
    int phase = kPhaseFps;
    uint32_t cand = 0, emp = 0, fp = 0;
    V claim_expect = 0;
    uint64_t i = 0, bucket = 0, step = 0, wins = 0;
    K key = empty;
    uint32_t st = kStNone, join = 0, cnt_add = 1;
    int live_delta = 0; /* claims minus erases of this lane */

    constexpr int kCache = 1 << count_cache_bits<L>();
    __shared__ K sc_key[kCache];
    __shared__ V sc_cnt[kCache];
    const bool use_cache = a.handler == kHandlerNothing;
    if (use_cache) {
        for (int c = threadIdx.x; c < kCache; c += blockDim.x) {
            sc_key[c] = empty;
            sc_cnt[c] = 0;
        }
        __syncthreads();
    }

    for (;;) {
        /* ---- refill lanes whose key is done, in input order ---- */
        const unsigned need = __ballot_sync(kFull, !has);
        const uint64_t avail = we - cursor;
        const int take = int(uint64_t(__popc(need)) < avail ? uint64_t(__popc(need)) : avail);
        if (take == 0 && need == kFull) break;
        const int r = __popc(need & lanemask_lt);
        const bool refill = !has && r < take;
        const int off = int(cursor - pf_base) + r;
        const K ka = shfl_any(pfA, off & 31);
        const K kb = shfl_any(pfB, off & 31);
        if (refill) {
            key = off < 32 ? ka : kb;
            i = cursor + r;
            has = true;
            pending = true;
            st = kStNone;
            cnt_add = 1;
            wins = 0;
            step = 0;
            phase = kPhaseFps;
            cand = 0;
            emp = 0;
            claim_expect = 0;
            if (key == empty || key == tomb) {
                st = kStInvalidKey;
                join |= kStInvalidKey;
                pending = false;
            }
        }
        cursor += uint64_t(take);
        if (cursor - pf_base >= 32) {
            pf_base += 32;
            pfA = pfB;
            const uint64_t nx = pf_base + 32 + lane;
            pfB = nx < we ? ld_stream(keys + nx) : empty;
        }

        {
            const bool fresh = refill && pending;
            const unsigned fmask = __ballot_sync(kFull, fresh);
            const unsigned peers = __match_any_sync(kFull, fresh ? key : empty) & fmask;
            if (fresh) {
                const int leader = __ffs(peers) - 1;
                cnt_add = __popc(peers);
                if (lane != leader) {
                    st = kStDuplicateKey;
                    join |= kStDuplicateKey;
                    pending = false;
                }
            }
        }
        if (use_cache && refill && pending) {
            using CW = typename std::conditional<sizeof(K) == 8, unsigned long long,
                                                 unsigned int>::type;
            const uint32_t h = uint32_t((uint64_t(key) * 0x9E3779B97F4A7C15ull) >> (64 - count_cache_bits<L>()));
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int c = int((h + p) & (kCache - 1));
                K cur = *reinterpret_cast<volatile K *>(&sc_key[c]);
                bool first = false;
                if (cur == empty) {
                    cur = K(atomicCAS(reinterpret_cast<CW *>(&sc_key[c]), CW(empty), CW(key)));
                    first = cur == empty;
                    if (first) cur = key;
                }
                if (cur == key) {
                    atomic_add_any(&sc_cnt[c], V(cnt_add));
                    if (!first) join |= kStDuplicateKey;
                    st = kStNone;
                    pending = false;
                    break;
                }
            }
        }
        if (refill && pending) {
            bucket = probe_begin<K>(t, key);
            fp = fingerprint(key);
        }

        /* ---- one memory operation per pending lane ---- */
        if (pending) {
            const uint64_t base_slot = bucket * uint64_t(W);
            bool advance = false;
            if (phase == kPhaseFps) {
                uint32_t m = 0, e = 0;
                fp_masks<W>(t.fps + base_slot, fp, m, e, pol_keep);
                cand = m;
                emp = e;
            } else if (phase == kPhaseCheck) {
                const int s = __ffs(cand) - 1;
                unsigned char *const sp = slots + (base_slot + uint64_t(s)) * SB;
                /* read where the claims' atomics land (L2): an L1 copy may
                 * predate the claim of an equal key by another lane, which
                 * would then be inserted twice */
                const LaneWords sw = load_lane<SB>(sp);
                const K sk = slot_key<L>(sw, 0);
                if (sk == key) {
                    st = kStDuplicateKey;
                    join |= kStDuplicateKey;
                    count_add<L>(sp, cnt_add, t.max_count, st, join);
                    pending = false;
                } else {
                    /* a set fingerprint over a key that reads empty is
                     * left to the compare-and-swap, which sees the key */
                    if (sk == empty) emp |= 1u << s;
                    cand &= cand - 1u;
                }
            } else if (phase == kPhasePreload) {
                /* bring the claim's slot line into L2 with a plain load; a
                 * slot that is no longer empty is skipped (its key is
                 * another one: equal keys show up as fingerprint matches,
                 * or as the CAS's old key) */
                {
                    int s = __ffs(emp) - 1;
                    const LaneWords sw = load_lane<SB>(slots + (base_slot + uint64_t(s)) * SB);
                    const K sk = slot_key<L>(sw, 0);
                    if (sk == key) {
                        st = kStDuplicateKey;
                        join |= kStDuplicateKey;
                        unsigned char *const sp = slots + (base_slot + uint64_t(s)) * SB;
                        count_add<L>(sp, cnt_add, t.max_count, st, join);
                        pending = false;
                    } else if (sk != empty) {
                        emp &= emp - 1u;
                        if (!emp) advance = true;
                    } else {
                        phase = kPhaseClaim;
                        claim_expect = slot_val<L>(sw, 0);
                    }
                }
            } else {
                {
                    const int s = __ffs(emp) - 1;
                    unsigned char *const sp = slots + (base_slot + uint64_t(s)) * SB;
                    const V payload = V(cnt_add);
                    V old_payload = 0;
                    /* (atom.cas takes no L2 cache hint) */
                    const K old = cas_slot<L>(sp, empty, claim_expect, key, payload, &old_payload);
                    if (old == empty && old_payload == claim_expect) {
                        st_hint_u8(t.fps + base_slot + uint64_t(s), fp, pol_keep);
                        ++live_delta;
                        st = kStNone;
                        pending = false;
                    } else if (old == key) {
                        st = kStDuplicateKey;
                        join |= kStDuplicateKey;
                        count_add<L>(sp, cnt_add, t.max_count, st, join);
                        pending = false;
                    } else if (old == empty) {
                        claim_expect = old_payload; /* free slot, stale payload: again */
                    } else {
                        emp &= emp - 1u;
                        if (!emp) advance = true;
                        else if (preload) phase = kPhasePreload;
                    }
                }
            }

            /* a bucket with no candidate left decides: absent if it had a
             * free slot (claim it for inserts), else the next bucket */
            if (pending && phase != kPhaseClaim && phase != kPhasePreload && !advance) {
                if (cand) {
                    phase = kPhaseCheck;
                } else if (emp) {
                    phase = preload ? kPhasePreload : kPhaseClaim;
                    claim_expect = 0;
                } else {
                    advance = true;
                }
            }
            if (pending && advance) {
                phase = kPhaseFps;
                cand = 0;
                emp = 0;
                claim_expect = 0;
                if (++wins >= a.max_windows) {
                    pending = false;
                    st = kStProbingLengthExceeded;
                    join |= kStProbingLengthExceeded;
                } else {
                    if (wins == 1) step = probe_step<K>(t, key);
                    bucket = probe_next(t, bucket, step);
                }
            }
        }

        /* ---- keys that finished this wave write their results ---- */
        if (has && !pending) {
            if (a.status_out) {
                if (a.handler == kHandlerStatus)
                    st_stream(reinterpret_cast<uint32_t *>(a.status_out) + i, st);
                else if (a.handler == kHandlerBoolean)
                    reinterpret_cast<unsigned char *>(a.status_out)[i] =
                        (unsigned char)((st & a.bool_mask) != 0);
            }
            has = false;
        }
    }
    if (use_cache) {
        __syncthreads();
        for (int c = threadIdx.x; c < kCache; c += blockDim.x) {
            const K ck = sc_key[c];
            if (ck != empty)
                count_one<L, W>(t, ck, uint32_t(sc_cnt[c]), a.max_windows, join, live_delta);
        }
    }
    const uint32_t wjoin = __reduce_or_sync(kFull, join);
    const int wlive = int(__reduce_add_sync(kFull, unsigned(live_delta)));
    if (lane == 0) {
        join_status(t.status, wjoin);
        live_add(t, wlive);
    }
}

/* The W fingerprint bytes of a bucket as 32-bit words */
template <int W>
struct FpWords {
    static constexpr int NW = W >= 4 ? W / 4 : 1;
    uint32_t w[NW];

    __device__ __forceinline__ void load(const unsigned char *p, uint64_t pol)
    {
        if constexpr (W == 1) {
            w[0] = ld_hint_u8(p, pol);
        } else if constexpr (W == 2) {
            w[0] = ld_hint_u16(p, pol);
        } else if constexpr (W == 4) {
            w[0] = ld_hint_u32(p, pol);
        } else if constexpr (W == 8) {
            const uint2 v = ld_hint_v2(p, pol);
            w[0] = v.x;
            w[1] = v.y;
        } else {
#pragma unroll
            for (int h = 0; h < W / 16; ++h) {
                const uint4 v = ld_hint_v4(p + 16 * h, pol);
                w[4 * h + 0] = v.x;
                w[4 * h + 1] = v.y;
                w[4 * h + 2] = v.z;
                w[4 * h + 3] = v.w;
            }
        }
    }
    /* the top bit of each byte of x that is zero; a byte of 1 above a zero
     * byte may be marked too (the borrow), so "any" is exact and a marked
     * byte is a candidate */
    static __device__ __forceinline__ uint32_t zero_bytes(uint32_t x)
    {
        constexpr uint32_t kBytes = W >= 4 ? 0x80808080u : W == 2 ? 0x8080u : 0x80u;
        return (x - 0x01010101u) & ~x & kBytes;
    }
    __device__ __forceinline__ bool any_empty() const
    {
        uint32_t m = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) m |= zero_bytes(w[k]);
        return m != 0;
    }
    /* candidates for the pattern of four equal bytes: bit 8 b + k stands for
     * byte b of word k (slot_of) */
    __device__ __forceinline__ uint32_t candidates(uint32_t pat) const
    {
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) c |= (zero_bytes(w[k] ^ pat) >> 7) << k;
        return c;
    }
    static __device__ __forceinline__ int slot_of(int bit) { return (bit >> 3) + 4 * (bit & 7); }
    /* the empty slots, bit s for slot s (a tombstone above an empty slot may
     * be marked too: its claim fails) */
    __device__ __forceinline__ uint32_t empty_slots() const
    {
        uint32_t e = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) e |= pack_bytes4(zero_bytes(w[k])) << (4 * k);
        return e;
    }
};

/* Retrieve and erase on tables with fingerprints.  What a kernel in the form of
 * fp_count_kernel was bound by here is instruction issue (28 warp instructions per query, 77 %
 * issue-active): a wave ran the fingerprint and the slot step one after the
 * other, each waiting for its own load, built masks byte by byte and carried
 * 64-bit places.  Here the lanes' fingerprint and slot loads are in flight
 * together before any is looked at, a zero-byte test finds the empty and
 * the matching fingerprints of a word (a match is checked against the slot
 * anyway), and places in the warp's range are 32 bits wide.  Against it, u64 set of
 * 134 MB at load 0.9: 15 M lookups 584 -> 483 us, 3.75 M erases 171 -> 158; u64
 * pairs of 2.4 GB, 2^27 lookups 5.54 -> 5.34 ms (25.1 G/s; plain 8-byte reads
 * at random measured 38 there, and a hit needs two); u32 pairs of 269 MB 30 M
 * 991 -> 863 us; u32 set at CG 32 50 M 1611 -> 1126. */
template <class L, int W, int OP>
__global__ void __launch_bounds__(256, WC_FP_MIN_BLOCKS_READ) fp_find_kernel(const TableOpArgs a)
{
    using K = typename L::key_t;
    using V = typename L::val_t;
    static_assert(OP == kOpRetrieve || OP == kOpErase, "operation");
    constexpr int SB = L::kSlotBytes;
    const uint64_t pol_keep = l2_policy_evict_last(); /* fingerprint lines */

    const TableView &t = a.t;
    const int lane = threadIdx.x & 31;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;

    /* this warp's contiguous range of keys */
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    const uint32_t m = uint32_t(wb + per < a.n ? per : a.n - wb);
    const K empty = K(t.empty_key);
    const K tomb = K(t.tombstone_key);
    unsigned char *const slots = reinterpret_cast<unsigned char *>(t.slots);
    const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;

    uint32_t pf_base = 0, cursor = 0;
    K pfA = uint32_t(lane) < m ? ld_stream(keys + lane) : empty;
    K pfB = 32 + uint32_t(lane) < m ? ld_stream(keys + 32 + lane) : empty;

    /* the key this lane owns; cand: slots of its bucket still to be read (0:
     * the bucket's fingerprints are due), any_empty: the bucket has a free one */
    bool has = false, any_empty = false;
    uint32_t cand = 0, at = 0;
    uint64_t bucket = 0, step = 0, wins = 0;
    K key = empty;
    uint32_t join = 0;
    int live_delta = 0;

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
            const K ka = shfl_any(pfA, int(off & 31u));
            const K kb = shfl_any(pfB, int(off & 31u));
            if (!has && r < take) {
                key = off < 32 ? ka : kb;
                at = cursor + r;
                has = true;
                cand = 0;
                wins = 0;
                step = 0;
                if (key == empty || key == tomb) {
                    join |= kStInvalidKey;
                    finish(kStInvalidKey, false);
                } else {
                    bucket = probe_begin<K>(t, key);
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

        /* ---- one load per lane with a key: the bucket's fingerprints or a
         * candidate's slot ---- */
        const uint64_t base_slot = bucket * uint64_t(W);
        FpWords<W> f;
        LaneWords sw;
        unsigned char *const sp =
            slots + (base_slot + uint64_t(FpWords<W>::slot_of(__ffs(cand) - 1))) * SB;
        if (has) {
            if (cand == 0) f.load(t.fps + base_slot, pol_keep);
            /* (erase reads from L2, where its compare-and-swap follows) */
            else if constexpr (OP == kOpRetrieve) sw = load_slot_once<L>(sp);
            else sw = load_lane<SB>(sp);
        }
        if (!has) continue;

        if (cand == 0) {
            cand = f.candidates(fingerprint(key) * 0x01010101u);
            any_empty = f.any_empty();
            if (cand) continue; /* the slot follows in the next wave */
        } else {
            if (slot_key<L>(sw, 0) == key) {
                if constexpr (OP == kOpRetrieve) {
                    if constexpr (L::kHasValue) {
                        if (!a.is_set) {
                            V v = slot_val<L>(sw, 0);
                            if (uint64_t(v) > t.max_count) v = V(t.max_count);
                            st_stream(reinterpret_cast<V *>(a.out) + wb + at, v);
                        }
                    }
                } else if (erase_slot_seen<L>(sp, key, tomb, sw)) {
                    fp_store(t, base_slot + uint64_t(FpWords<W>::slot_of(__ffs(cand) - 1)), kFpTomb);
                    --live_delta;
                }
                finish(kStNone, true);
                continue;
            }
            cand &= cand - 1u;
            if (cand) continue;
        }
        /* no candidate left: absent if the bucket has a free slot */
        if (any_empty) {
            const uint32_t st = a.is_set ? kStNone : kStKeyNotFound;
            if constexpr (OP == kOpRetrieve) join |= st;
            finish(st, false);
        } else if (++wins >= a.max_windows) {
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
    const uint32_t wjoin = __reduce_or_sync(kFull, join);
    const int wlive = int(__reduce_add_sync(kFull, unsigned(live_delta)));
    if (lane == 0) {
        join_status(t.status, wjoin);
        live_add(t, wlive);
    }
}

/* Insert on tables with fingerprints, in the form of fp_find_kernel: the
 * lanes' fingerprint loads, slot reads and claims are in flight together.
 * Claims take the lowest slot with an empty fingerprint first, as in
 * fp_count_kernel.  Against a kernel in the form of that one, which ran the
 * three steps one after the other: u64 set of 134 MB at load 0.9, 15 M keys
 * 727 -> 597 us; u64 pairs of 161 MB, 9 M 491 -> 444; u32 pairs of 269 MB, 30 M
 * 1612 -> 1423; 65 536 updates of 575 MB of u64 pairs 41 -> 33.
 *
 * Equal keys that meet in one refill are merged, with the value of the last:
 * a call of at most 32 keys stores each key's last value, and a frequent key
 * sends one claim or store per refill instead of up to 32 that queue at one
 * address.  A warp that found no equal keys in kMergeQuiet refills in a row
 * looks through one refill of eight, so distinct keys pay little: 4 M
 * keys, without / with merging, u64 set 176 / 184 us, u32 pairs 224 / 225, u64
 * pairs 215 / 201; one key 4 M times 2 645 / 117, 2 617 / 565, 4 110 / 566;
 * Zipf(1.4) 780 / 216, 3 346 / 2 146, 3 528 / 2 095.
 *
 * In tables with values the merged lanes wait for the lane that has their key
 * (kHold), unless they are most of a refill.  Their places would be filled
 * with one or two keys at a time, and a frequent key that comes in more
 * and smaller refills reads and writes its slot's line more often: 4 M
 * Zipf(1.1) updates of u64 pairs 10.2 ms without waiting, 6.8 with it (and
 * without merging); keys in runs of 16 125 us with waiting always, 87 so.
 * Sets, which write nothing for a key that is there, gain nothing by it.
 *
 * kPreload: a claim's slot is loaded before its compare-and-swap. */
constexpr uint32_t kMergeQuiet = 4;

/* one more block than the other kernels where 48 registers do: 4 M u32 pairs
 * 238 -> 225 us, u64 set 204 -> 184 */
template <class L>
constexpr int fp_insert_min_blocks()
{
    return L::kSlotBytes <= 8 ? WC_FP_MIN_BLOCKS + 1 : WC_FP_MIN_BLOCKS;
}

template <class L, int W, bool kPreload>
__global__ void __launch_bounds__(256, fp_insert_min_blocks<L>()) fp_insert_kernel(const TableOpArgs a)
{
    using K = typename L::key_t;
    using V = typename L::val_t;
    constexpr int SB = L::kSlotBytes;
    constexpr bool kValueIn = L::kHasValue;
    constexpr bool kHold = kValueIn;
    const uint64_t pol_keep = l2_policy_evict_last(); /* fingerprint lines */

    const TableView &t = a.t;
    const int lane = threadIdx.x & 31;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;

    /* this warp's contiguous range of keys */
    uint64_t per = (a.n + nwarps - 1) / nwarps;
    per = (per + 31) & ~uint64_t(31);
    const uint64_t wb = warp * per < a.n ? warp * per : a.n;
    const uint32_t m = uint32_t(wb + per < a.n ? per : a.n - wb);
    const K empty = K(t.empty_key);
    const K tomb = K(t.tombstone_key);
    unsigned char *const slots = reinterpret_cast<unsigned char *>(t.slots);
    const K *const keys = reinterpret_cast<const K *>(a.keys) + wb;
    const V *const vals_in = reinterpret_cast<const V *>(a.values) + (kValueIn ? wb : 0);

    uint32_t pf_base = 0, cursor = 0;
    K pfA = uint32_t(lane) < m ? ld_stream(keys + lane) : empty;
    K pfB = 32 + uint32_t(lane) < m ? ld_stream(keys + 32 + lane) : empty;
    V pvA = 0, pvB = 0;
    if constexpr (kValueIn) {
        if (uint32_t(lane) < m) pvA = ld_stream(vals_in + lane);
        if (32 + uint32_t(lane) < m) pvB = ld_stream(vals_in + 32 + lane);
    }

    /* the key this lane owns: with cand its candidates are to be read, else
     * with `free` the lowest slot of it is to be claimed, else the bucket's
     * fingerprints are due */
    bool has = false;
    bool peeked = false; /* the claim's slot has been read (kPreload) */
    uint32_t cand = 0, free = 0, at = 0;
    uint32_t quiet = 0; /* refills since the last one with equal keys */
    /* waits: lane `first` inserts this lane's key too; held: some lane waits */
    bool waits = false, held = false;
    int first = 0;
    uint64_t bucket = 0, step = 0, wins = 0;
    K key = empty;
    V val = 0, expect = 0;
    uint32_t join = 0;
    int live_delta = 0;

    auto finish = [&](uint32_t st) {
        join |= st;
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
        /* ---- lanes whose key another lane inserts wait for it ---- */
        if (kHold && held) {
            const unsigned done = __ballot_sync(kFull, !has);
            if (waits && ((done >> first) & 1u)) has = waits = false;
            held = __any_sync(kFull, waits);
        }
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
                cand = 0;
                free = 0;
                peeked = false;
                wins = 0;
                step = 0;
                fresh = key != empty && key != tomb;
                if (!fresh) finish(kStInvalidKey);
            }
            bool merged = false;
            if (quiet < kMergeQuiet || (quiet & 7u) == 0) {
                const unsigned peers = merge_equal_keys<K, V, kValueIn>(fresh, key, empty, val);
                merged = fresh && (peers & lanemask_lt);
                const uint32_t gone = uint32_t(__popc(__ballot_sync(kFull, merged)));
                if (gone) quiet = 0;
                if constexpr (kHold) {
                    if (merged && gone * 4 <= take * 3) {
                        waits = true;
                        first = __ffs(peers) - 1;
                    }
                    held |= gone != 0;
                }
            }
            ++quiet;
            if (merged) finish(kStDuplicateKey);
            else if (fresh) bucket = probe_begin<K>(t, key);
            if constexpr (kHold) has |= waits;
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
            }
        }

        /* ---- one memory operation per lane with a key ---- */
        const uint64_t base_slot = bucket * uint64_t(W);
        FpWords<W> f;
        LaneWords sw;
        K old = empty;
        V old_payload = 0;
        const uint64_t s = cand ? base_slot + uint64_t(FpWords<W>::slot_of(__ffs(cand) - 1))
                                : base_slot + uint64_t(free ? __ffs(free) - 1 : 0);
        unsigned char *const sp = slots + s * SB;
        const bool checking = cand != 0, claiming = !checking && free != 0;
        const bool peeking = kPreload && claiming && !peeked;
        if (has && !waits) {
            /* slots are read where the claims' atomics land (L2): an L1 copy
             * may predate the claim of an equal key by another lane */
            if (checking || peeking) sw = load_lane<SB>(sp);
            else if (claiming) old = cas_slot<L>(sp, empty, expect, key, val, &old_payload);
            else f.load(t.fps + base_slot, pol_keep);
        }
        if (!has || waits) continue;

        bool advance = false;
        if (checking) {
            if (slot_key<L>(sw, 0) == key) {
                store_value<L>(sp, val);
                finish(kStDuplicateKey);
                continue;
            }
            /* a fingerprint seen before the key it was written after: the
             * slot's claim decides */
            if (slot_key<L>(sw, 0) == empty)
                free |= 1u << FpWords<W>::slot_of(__ffs(cand) - 1);
            cand &= cand - 1u;
            advance = cand == 0 && free == 0;
        } else if (claiming) {
            if (peeking) {
                old = slot_key<L>(sw, 0);
                old_payload = slot_val<L>(sw, 0);
                peeked = old == empty;
            } else if (old == empty && old_payload == expect) {
                st_hint_u8(t.fps + s, fingerprint(key), pol_keep);
                ++live_delta;
                finish(kStNone);
                continue;
            }
            if (old == key) {
                store_value<L>(sp, val);
                finish(kStDuplicateKey);
            } else if (old == empty) {
                expect = old_payload; /* free slot, its payload known now */
            } else {
                free &= free - 1u;
                expect = 0;
                peeked = false;
                advance = free == 0;
            }
        } else {
            cand = f.candidates(fingerprint(key) * 0x01010101u);
            free = f.any_empty() ? f.empty_slots() : 0u;
            expect = 0;
            advance = cand == 0 && free == 0;
        }
        if (advance) {
            if (++wins >= a.max_windows) {
                finish(kStProbingLengthExceeded);
            } else {
                if (wins == 1) step = probe_step<K>(t, key);
                bucket = probe_next(t, bucket, step);
            }
        }
    }
    const uint32_t wjoin = __reduce_or_sync(kFull, join);
    const int wlive = int(__reduce_add_sync(kFull, unsigned(live_delta)));
    if (lane == 0) {
        join_status(t.status, wjoin);
        live_add(t, wlive);
    }
}

/* Recompute every fingerprint from the slot array in one streaming pass.
 * Lane l of a warp reads 16-byte vector v + l (coalesced) and writes the
 * fingerprints of its 1, 2 or 4 slots as one store, so a warp writes 32,
 * 64 or 128 consecutive bytes; four vectors per thread are in flight.  A
 * large insert runs the whole-window kernel without fingerprint writes and
 * then this pass: streaming the slot array costs less than one random byte
 * write per key once a batch covers more than about 1/8 of a table larger
 * than L2.
 *
 * A slot read as empty leaves its fingerprint alone: an insert on another
 * stream may claim it and store its fingerprint between the read and the
 * write here, and a cleared fingerprint would hide its key for good.  (A
 * fingerprint never has to be cleared, since no slot becomes empty again.)
 * The stores of mixed vectors byte by byte cost under 1 % of an insert: 2^27
 * u64 pairs 8.76 -> 8.79 ms, 135 M u32 pairs 8.37 -> 8.40, 180 M keys into a
 * u32 set 9.42 -> 9.47. */
template <class L>
__device__ __forceinline__ uint32_t fp_of_slot_key(typename L::key_t k, typename L::key_t e,
                                                   typename L::key_t tb)
{
    return k == e ? kFpEmpty : (k == tb ? kFpTomb : fingerprint(k));
}

template <class L>
__global__ void __launch_bounds__(256) fp_rebuild_kernel(const void *slots, uint64_t capacity,
                                                         uint64_t empty, uint64_t tomb,
                                                         unsigned char *fps)
{
    using K = typename L::key_t;
    constexpr int SB = L::kSlotBytes;
    constexpr int SPV = 16 / SB; /* slots per 16-byte vector: 1, 2 or 4 */
    constexpr int kUnroll = 4;
    const K e = K(empty), tb = K(tomb);
    const uint4 *const vec = reinterpret_cast<const uint4 *>(slots);
    const uint64_t nvec = capacity / SPV;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t v0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v0 < nvec;
         v0 += stride * kUnroll) {
        uint4 x[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint64_t v = v0 + uint64_t(u) * stride;
            x[u] = v < nvec ? __ldcs(vec + v) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint64_t v = v0 + uint64_t(u) * stride;
            if (v >= nvec) break;
            const LaneWords lw{{x[u].x, x[u].y, x[u].z, x[u].w}};
            uint32_t f = 0;
#pragma unroll
            for (int s = 0; s < SPV; ++s) f |= fp_of_slot_key<L>(slot_key<L>(lw, s), e, tb) << (8 * s);
            bool all = true;
#pragma unroll
            for (int s = 0; s < SPV; ++s) all &= (f >> (8 * s) & 0xffu) != kFpEmpty;
            if (all) {
                if constexpr (SPV == 1) fps[v] = (unsigned char)f;
                else if constexpr (SPV == 2) reinterpret_cast<unsigned short *>(fps)[v] = (unsigned short)f;
                else reinterpret_cast<uint32_t *>(fps)[v] = f;
            } else if constexpr (SPV > 1) {
#pragma unroll
                for (int s = 0; s < SPV; ++s)
                    if (f >> (8 * s) & 0xffu) fps[v * SPV + s] = (unsigned char)(f >> (8 * s));
            }
        }
    }
    /* ragged tail: capacity need not be a multiple of SPV */
    if (blockIdx.x == 0 && threadIdx.x < capacity % SPV) {
        const uint64_t si = nvec * SPV + threadIdx.x;
        const K k = *reinterpret_cast<const K *>(reinterpret_cast<const unsigned char *>(slots) + si * SB);
        if (k != e) fps[si] = (unsigned char)fp_of_slot_key<L>(k, e, tb);
    }
}

} // namespace b200
} // namespace warpcore

#endif /* WC_FP_KERNELS_CUH */
