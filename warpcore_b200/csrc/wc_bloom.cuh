/*
 * wc_bloom.cuh -- pattern-blocked Bloom filter kernels
 * (the reference's BloomFilter::insert / retrieve, bloom_filter.cuh:168-237,
 * launched by kernels::bloom_filter::insert / retrieve, gpu_engine.cuh:130-171).
 *
 * A block is cg_size consecutive slots (words).  The bit pattern of a key is
 * the reference's: block = h(key+seed) % num_blocks, bit i (i < k) =
 * h(key+seed+i) % block_bits, owned by word bit / slot_bits of the block, and
 * the word index wraps modulo num_slots for a ragged last block.  A warp takes
 * 32 keys; lane l owns key l.  A block is read by TPK lanes with 16-byte
 * vector loads (one request per block) for all 32 keys before any is tested.
 * Insert ORs only the words that miss bits (one atomicOr per such word, as
 * the reference) or the whole mask in one bulk reduction (BulkOr), query
 * tests the whole block and writes one byte per key.
 */
#ifndef WC_BLOOM_CUH
#define WC_BLOOM_CUH

#include "wc_lane_kernels.cuh"

#include <cstring>

namespace warpcore {
namespace b200 {

struct BloomArgs {
    void *words;
    const void *keys;
    unsigned char *flags_out;
    uint64_t n;
    uint64_t num_slots;
    uint64_t num_blocks;
    uint64_t magic_blocks; /* barrett_magic(num_blocks) */
    uint64_t k;
    uint64_t seed;
    uint32_t hasher;
    /* a shard holds the blocks [block_base, block_base + local_blocks) of a
     * filter of num_blocks blocks (a whole filter: 0 and num_blocks); its
     * words start at block_base, and a key whose block it does not hold is
     * skipped (insert) or reported absent (query) */
    uint64_t block_base;
    uint64_t local_blocks;
    /* this launch serves only the keys whose local block lies in
     * [region_lo, region_hi) (bloom_lane_kernel; see region passes below);
     * region_lo == 0 also answers the keys of other shards */
    uint64_t region_lo;
    uint64_t region_hi;
};

template <class S>
__device__ __forceinline__ S lane_word(const LaneWords &lw, int s)
{
    if constexpr (sizeof(S) == 4) return lw.w[s];
    else return uint64_t(lw.w[2 * s]) | (uint64_t(lw.w[2 * s + 1]) << 32);
}

template <class T>
__device__ __forceinline__ T atomic_or_any(T *p, T v)
{
    if constexpr (sizeof(T) == 8)
        return T(atomicOr(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v));
    else
        return T(atomicOr(reinterpret_cast<unsigned int *>(p), (unsigned int)v));
}

/* bit masks of the CG words of key's block, computed once by the lane that
 * owns the key */
template <class K, class S, int CG>
__device__ __forceinline__ void block_masks(K key, K seed, uint32_t hasher, uint64_t k, S (&m)[CG])
{
    constexpr uint64_t kSlotBits = sizeof(S) * 8;
    constexpr uint64_t kBlockBits = kSlotBits * CG;
#pragma unroll
    for (int w = 0; w < CG; ++w) m[w] = 0;
    /* the hasher decided once for the k hashes, with MurmurHash (the
     * default) inlined: 27.9 against 27.2 G queries/s on the 2^32-bit
     * filter */
    if (hasher == kHashMurmur) {
        for (uint64_t j = 0; j < k; ++j) {
            const uint64_t h = hash_key<K>(kHashMurmur, K(key + seed + K(j))) & (kBlockBits - 1);
            const int word = int(h / kSlotBits);
            const S bit = S(1) << (h % kSlotBits);
#pragma unroll
            for (int w = 0; w < CG; ++w)
                if (word == w) m[w] |= bit;
        }
        return;
    }
    for (uint64_t j = 0; j < k; ++j) {
        const uint64_t h = hash_key<K>(hasher, K(key + seed + K(j))) & (kBlockBits - 1);
        const int word = int(h / kSlotBits);
        const S bit = S(1) << (h % kSlotBits);
#pragma unroll
        for (int w = 0; w < CG; ++w)
            if (word == w) m[w] |= bit;
    }
}

/* ORs a key's whole block mask into the filter as one bulk reduction from
 * this thread's row in shared memory (cp.reduce.async.bulk), for blocks of
 * 16 to 128 bytes.  Inserts are bound by their ORs at L2: one per word that
 * misses bits, 4.3 per key with 8 bits in 64 bytes, after a read of the
 * block to find those words.  A bulk reduction needs no read (see LookFirst)
 * and is one request per key.  2^28 keys into the 2^32-bit filter of 64-byte blocks:
 * 13.17 -> 12.12 ms; 6 M keys into a 16 MiB filter of 32-byte blocks, which
 * stays in L2: 191 -> 174 us.  Sending a quarter or half of the warps'
 * masks this way and the others as word ORs measured 15.2 / 13.9 ms and
 * 168 / 172 us, so the two do not add up: L2 is what both wait for. */
template <class S, int CG>
struct BulkOr {
    static constexpr int BB = CG * int(sizeof(S));
    static constexpr bool kUsed = BB >= 16;
    /* a row is followed by 16 bytes where that spreads the rows of eight
     * lanes' 16-byte stores over all banks */
    static constexpr int kRow = BB > 16 ? BB + 16 : 16;

    /* the mask into this thread's row, once the row's last reduction has
     * been read */
    static __device__ __forceinline__ void put(unsigned char *row, const S (&m)[CG])
    {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        constexpr int WPV = 16 / int(sizeof(S));
#pragma unroll
        for (int v = 0; v < BB / 16; ++v) {
            uint4 q;
            memcpy(&q, &m[v * WPV], 16);
            *reinterpret_cast<uint4 *>(row + 16 * v) = q;
        }
    }
    /* whether the block misses bits of the row's mask.  (The mask is read
     * back, so that it and the block are never both in registers.) */
    static __device__ __forceinline__ bool misses(const S *block, const unsigned char *row)
    {
        uint32_t w[BB / 4], miss = 0;
        load_window<BB>(reinterpret_cast<const unsigned char *>(block), w);
#pragma unroll
        for (int v = 0; v < BB / 16; ++v) {
            uint32_t q[4];
            asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3])
                         : "r"(uint32_t(__cvta_generic_to_shared(row)) + 16u * v) : "memory");
#pragma unroll
            for (int i = 0; i < 4; ++i) miss |= q[i] & ~w[4 * v + i];
        }
        return miss != 0;
    }
    static __device__ __forceinline__ void send(S *block, unsigned char *row)
    {
        const uint32_t sa = uint32_t(__cvta_generic_to_shared(row));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.or.b64 [%0], [%1], %2;"
                     :: "l"(block), "r"(sa), "r"(BB) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    static __device__ __forceinline__ void finish()
    {
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
};

/* a whole block into registers, by 32-byte loads where it has them: a load of
 * 32 lanes at random addresses costs one pass per lane whatever its width */
template <class S, int CG>
__device__ __forceinline__ void load_block(const S *p, S (&w)[CG])
{
    constexpr int BB = CG * int(sizeof(S));
    uint32_t x[BB / 4];
    load_window<BB>(reinterpret_cast<const unsigned char *>(p), x);
#pragma unroll
    for (int i = 0; i < CG; ++i) {
        if constexpr (sizeof(S) == 4) w[i] = S(x[i]);
        else w[i] = S(uint64_t(x[2 * i]) | (uint64_t(x[2 * i + 1]) << 32));
    }
}

/* Whether every one of the key's k bits is set in the block w, each bit
 * tested in the 32-bit word it falls in (the query needs no masks).  The
 * block's words stand in this thread's column of shared memory, `col`, one
 * of 256 columns, so that a word is picked by its address and no two lanes
 * meet on a bank.  With the block in registers and each word picked by a
 * tree of selects, queries were bound by instruction issue: 2^28 queries of
 * the 2^32-bit filter of 64-byte blocks, k 8, 6.55 -> 5.52 ms (48.7 G/s; plain
 * 64-byte reads at random measured 57), 12 M of a 16 MiB filter of 32-byte
 * blocks, k 6, 129 -> 111 us.  (Those 6.55 ms were 7.40 with 16-byte loads of
 * the blocks.) */
template <class K, class S, int CG>
__device__ __forceinline__ bool block_has_all(K key, K seed, uint32_t hasher, uint64_t k,
                                              const S (&w)[CG], uint32_t *col)
{
    constexpr uint32_t kBlockBits = uint32_t(sizeof(S)) * 8 * CG;
#pragma unroll
    for (int i = 0; i < CG; ++i) {
        if constexpr (sizeof(S) == 4) {
            col[i * 256] = uint32_t(w[i]);
        } else {
            col[2 * i * 256] = uint32_t(w[i]);
            col[(2 * i + 1) * 256] = uint32_t(uint64_t(w[i]) >> 32);
        }
    }
    uint32_t ok = 1;
    const uint32_t n = uint32_t(k);
    if (hasher == kHashMurmur) {
        for (uint32_t j = 0; j < n; ++j) {
            const uint32_t h = uint32_t(hash_key<K>(kHashMurmur, K(key + seed + K(j)))) &
                               (kBlockBits - 1);
            ok &= col[(h >> 5) * 256] >> (h & 31u);
        }
        return ok & 1u;
    }
    for (uint32_t j = 0; j < n; ++j) {
        const uint32_t h = uint32_t(hash_key<K>(hasher, K(key + seed + K(j)))) & (kBlockBits - 1);
        ok &= col[(h >> 5) * 256] >> (h & 31u);
    }
    return ok & 1u;
}

/* When a warp's inserts read a block before its bulk OR, so that a key whose
 * bits are all set sends nothing.  ORs of one block queue at its place in
 * L2, about 1 ns each, so a stream of repeated keys needs the read; for
 * distinct keys it is a second access for nothing.  A warp looks at its first
 * kSample keys, goes on looking while at least one of kFew looked at was there,
 * and else looks again after kSkip rounds.  2^32-bit filter of 64-byte
 * blocks, never / always / this: 2^28 distinct keys 12.13 / 12.82 / 12.31 ms,
 * inserted again 12.13 / 9.31 / 9.88, 2^27 Zipf(0.8) keys 10.0 / 5.3 / 5.4,
 * Zipf(1.1) 32.2 / 5.0 / 5.1, 2^24 times one key 17.2 / 0.53 / 0.48; 6 M keys into a
 * 16 MiB filter of 32-byte blocks: 171 / 197 / 177 us, 169 / 116 / 116, 171 / 155 /
 * 151, 478 / 186 / 145, 3 077 / 271 / 150.  The share is taken over several rounds:
 * a region holds some 16 keys of a tile, and with "two present in the last
 * round" Zipf(1.1) took 14.6 ms. */
struct LookFirst {
    static constexpr uint32_t kSample = 64, kFew = 32, kSkip = 15;
    uint32_t keys = 0, there = 0, skip = 0;

    __device__ __forceinline__ bool now() const { return skip == 0; }
    /* keys of a round that was looked at: which lanes had one, and had one
     * that was there */
    __device__ __forceinline__ void looked(bool in, bool present)
    {
        keys += uint32_t(__popc(__ballot_sync(kFull, in)));
        there += uint32_t(__popc(__ballot_sync(kFull, present)));
    }
    /* ends a round */
    __device__ __forceinline__ void next()
    {
        if (skip) {
            --skip;
            return;
        }
        if (keys >= kSample && there * kFew < keys) skip = kSkip;
        if (keys >= 4 * kSample) {
            keys /= 2;
            there /= 2;
        }
    }
};

constexpr uint64_t kNoBlock = ~0ull;

/* ORs a key into the block that starts at word `first` (kNoBlock: no key);
 * whether its bits were all there (bulk ORs with `read`: the block is read
 * first) */
template <class K, class S, int CG, bool kBulk>
__device__ __forceinline__ bool bloom_or(const BloomArgs &a, K key, uint64_t first,
                                         unsigned char *row, bool read)
{
    S *const words = reinterpret_cast<S *>(a.words);
    const bool whole = first != kNoBlock && first + CG <= a.num_slots;
    bool there = false;
    if (first != kNoBlock) {
        S w[CG];
        if constexpr (!kBulk) {
            if (whole) {
                load_block<S, CG>(words + first, w);
            } else {
                /* ragged last block: words wrap to the front */
#pragma unroll
                for (int s = 0; s < CG; ++s) w[s] = __ldcg(words + (first + s) % a.num_slots);
            }
        }
        S m[CG];
        block_masks<K, S, CG>(key, K(a.seed), a.hasher, a.k, m);
        if (kBulk && whole) {
            if constexpr (kBulk) {
                using Bulk = BulkOr<S, CG>;
                Bulk::put(row, m);
                there = read && !Bulk::misses(words + first, row);
                if (!there) Bulk::send(words + first, row);
            }
        } else {
#pragma unroll
            for (int s = 0; s < CG; ++s) {
                if (kBulk ? m[s] != 0 : (w[s] & m[s]) != m[s]) {
                    uint64_t wi = first + uint64_t(s);
                    if (wi >= a.num_slots) wi -= a.num_slots;
                    atomic_or_any(words + wi, m[s]);
                }
            }
        }
    }
    return there;
}

template <class K, class S, int CG, bool INSERT>
__global__ void __launch_bounds__(256) bloom_kernel(const BloomArgs a)
{
    constexpr int SB = sizeof(S);
    constexpr int BB = CG * SB;                 /* block bytes */
    constexpr int LB = BB < 16 ? BB : 16;       /* bytes per lane */
    constexpr int TPK = BB / LB;                /* lanes per block */
    constexpr int SPL = LB / SB;                /* words per lane */
    constexpr int G = 32 / TPK;
    constexpr uint64_t kSlotBits = SB * 8;
    constexpr uint64_t kBlockBits = kSlotBits * CG;
    constexpr uint32_t kGroupMask = TPK == 32 ? kFull : ((1u << TPK) - 1u);
    /* small blocks: the owner computes the masks once and the group lanes
     * receive their words by shuffles; large blocks: every group lane derives
     * the masks of its own words */
    constexpr bool kOwnerMasks = CG * SB <= 64;

    const int lane = threadIdx.x & 31;
    const int g = lane / TPK;
    const int q = lane % TPK;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    S *const words = reinterpret_cast<S *>(a.words);
    const K *const keys = reinterpret_cast<const K *>(a.keys);
    const K seed = K(a.seed);

    for (uint64_t base = warp * 32; base < a.n; base += nwarps * 32) {
        const uint64_t i = base + lane;
        const bool active = i < a.n;
        const K key = active ? ld_stream(keys + i) : K(0);
        const uint64_t blk = fast_mod(hash_key<K>(a.hasher, K(key + seed)), a.num_blocks, a.magic_blocks);
        S own_mask[kOwnerMasks ? CG : 1];
        if constexpr (kOwnerMasks) block_masks<K, S, CG>(key, seed, a.hasher, a.k, own_mask);

        LaneWords win[TPK];
#pragma unroll
        for (int r = 0; r < TPK; ++r) {
            const int o = r * G + g; /* owner lane of this round's block */
            const uint64_t b = shfl_any(blk, o);
            const uint64_t w0 = b * CG + uint64_t(q) * SPL;
            win[r] = LaneWords{{0u, 0u, 0u, 0u}};
            if ((base + o) < a.n) {
                if (b * CG + CG <= a.num_slots) {
                    win[r] = load_lane<LB>(words + w0);
                } else {
                    /* ragged last block: words wrap to the front */
#pragma unroll
                    for (int s = 0; s < SPL; ++s) {
                        const S v = __ldcg(reinterpret_cast<const S *>(words) + (w0 + s) % a.num_slots);
                        if constexpr (SB == 4) win[r].w[s] = uint32_t(v);
                        else { win[r].w[2 * s] = uint32_t(v); win[r].w[2 * s + 1] = uint32_t(uint64_t(v) >> 32); }
                    }
                }
            }
        }

        bool my_flag = false;
#pragma unroll
        for (int r = 0; r < TPK; ++r) {
            const int o = r * G + g;
            const bool own_ok = (base + o) < a.n;
            const uint64_t b = shfl_any(blk, o);
            S mask[SPL];
            if constexpr (kOwnerMasks) {
#pragma unroll
                for (int w = 0; w < CG; ++w) {
                    const S m = shfl_any(own_mask[w], o);
                    if (w / SPL == q) mask[w % SPL] = m;
                }
            } else {
                const K kr = shfl_any(key, o);
#pragma unroll
                for (int s = 0; s < SPL; ++s) mask[s] = 0;
                for (uint64_t j = 0; j < a.k; ++j) {
                    const uint64_t h = hash_key<K>(a.hasher, K(kr + seed + K(j))) & (kBlockBits - 1);
                    const int word = int(h / kSlotBits);
                    if (word / SPL == q) {
#pragma unroll
                        for (int s = 0; s < SPL; ++s)
                            if (word % SPL == s) mask[s] |= S(1) << (h % kSlotBits);
                    }
                }
            }
            bool ok = true;
#pragma unroll
            for (int s = 0; s < SPL; ++s) {
                const S w = lane_word<S>(win[r], s);
                const bool missing = (w & mask[s]) != mask[s];
                ok &= !missing;
                if (INSERT && own_ok && missing) {
                    uint64_t wi = b * CG + uint64_t(q) * SPL + s;
                    if (wi >= a.num_slots) wi -= a.num_slots; /* ragged last block */
                    atomic_or_any(words + wi, mask[s]);
                }
            }
            if constexpr (!INSERT) {
                const unsigned bad = __ballot_sync(kFull, !ok);
                /* lane r*G + gg owns the block read by group gg this round */
                if (lane / G == r) {
                    const int gg = lane - r * G;
                    my_flag = ((bad >> (gg * TPK)) & kGroupMask) == 0;
                }
            }
        }
        if constexpr (!INSERT) {
            if (active) a.flags_out[i] = (unsigned char)my_flag;
        }
    }
}

/* One key per lane, for blocks of at most 128 bytes: the lane computes its
 * key's masks, reads its own block with 32-byte vector loads and tests it.
 * An insert of blocks of 16 bytes or more ORs the whole mask (BulkOr) and
 * reads the block only where keys repeat (LookFirst); of smaller ones it ORs
 * only the words that miss bits.  Against the
 * cooperative kernel above it spends no shuffles on block indices and masks.
 * It serves the keys whose block lies in [region_lo, region_hi) (one pass:
 * the whole filter).
 *
 * Two keys per lane at a time pay for inserts of up to 32 bytes, which wait
 * for their keys (6 M into a 16 MiB filter of 32-byte blocks 174 -> 165 us);
 * for queries, bound by instruction issue, more than one costs registers
 * (12 M: 129 / 135 / 134 us with one / two / four). */
template <class S, int CG, bool INSERT>
constexpr int bloom_keys_per_lane()
{
    return INSERT && BulkOr<S, CG>::kUsed && CG * int(sizeof(S)) <= 32 ? 2 : 1;
}

/* resident blocks: inserts of blocks of up to 32 bytes keep the six they have
 * at 40 registers (43 without the bound: 182 us, 176 with it) */
template <class S, int CG, bool INSERT>
constexpr int bloom_lane_min_blocks()
{
    return INSERT && CG * sizeof(S) <= 32 ? 6 : 1;
}

template <class K, class S, int CG, bool INSERT>
__global__ void __launch_bounds__(256, bloom_lane_min_blocks<S, CG, INSERT>())
    bloom_lane_kernel(const BloomArgs a)
{
    constexpr int U = bloom_keys_per_lane<S, CG, INSERT>();
    static_assert(CG * sizeof(S) <= 128, "block of one lane");
    using Bulk = BulkOr<S, CG>;
    constexpr bool kBulk = INSERT && Bulk::kUsed;

    S *const words = reinterpret_cast<S *>(a.words);
    const K *const keys = reinterpret_cast<const K *>(a.keys);
    const K seed = K(a.seed);
    __shared__ alignas(16) unsigned char s_rows[kBulk ? 256 * Bulk::kRow : 16];
    __shared__ uint32_t s_words[INSERT ? 1 : CG * sizeof(S) / 4 * 256];
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    LookFirst look;
    /* (whole warps stay in the loop where look has its ballots) */
    const uint64_t end = kBulk ? a.n + (threadIdx.x & 31) : a.n;
    for (uint64_t i0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i0 < end;
         i0 += stride * U) {
        K key[U];
        uint64_t w0[U]; /* first word of the key's block, kNoBlock: not served */
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + uint64_t(u) * stride;
            key[u] = i < a.n ? ld_stream(keys + i) : K(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + uint64_t(u) * stride;
            const uint64_t blk = mod_hash<K>(hash_key<K>(a.hasher, K(key[u] + seed)),
                                             a.num_blocks, a.magic_blocks) - a.block_base;
            w0[u] = i < a.n && blk < a.local_blocks && blk >= a.region_lo && blk < a.region_hi
                        ? blk * CG : kNoBlock;
            if constexpr (!INSERT) {
                if (i < a.n && blk >= a.local_blocks && a.region_lo == 0) a.flags_out[i] = 0;
            }
        }
        if constexpr (INSERT) {
            const bool read = look.now();
            bool there[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                there[u] = bloom_or<K, S, CG, kBulk>(
                    a, key[u], w0[u], s_rows + (kBulk ? threadIdx.x * Bulk::kRow : 0), read);
            if constexpr (kBulk) {
                if (read) {
#pragma unroll
                    for (int u = 0; u < U; ++u) look.looked(w0[u] != kNoBlock, there[u]);
                }
                look.next();
            }
        } else {
            S w[U][CG];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (w0[u] == kNoBlock) continue;
                if (w0[u] + CG <= a.num_slots) {
                    load_block<S, CG>(words + w0[u], w[u]);
                } else {
                    /* ragged last block: words wrap to the front */
#pragma unroll
                    for (int s = 0; s < CG; ++s)
                        w[u][s] = __ldcg(words + (w0[u] + s) % a.num_slots);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (w0[u] != kNoBlock)
                    a.flags_out[i0 + uint64_t(u) * stride] =
                        (unsigned char)block_has_all<K, S, CG>(key[u], seed, a.hasher, a.k, w[u],
                                                               s_words + threadIdx.x);
        }
    }
    if constexpr (kBulk) Bulk::finish();
}

/* Region passes, for blocks of at most 128 bytes.  On B200, random reads
 * slow down sharply once the array they hit outgrows the GPU's
 * address-translation reach: 64-byte reads at random measured 64 G/s over
 * 256 MiB but 13.5 G/s over 512 MiB and 9.5 G/s over 4 GiB.  A filter
 * larger than one region is therefore processed in passes, one launch per
 * region of its blocks; each pass streams all keys and serves those whose
 * block lies in its region, so that its random reads (and an insert's
 * atomics) stay inside the region.
 *
 * A pass must keep many block reads in flight although only a fraction of
 * the keys it streams belongs to its region.  So a warp takes a tile of
 * region_kpl x 32 keys (region_kpl coalesced loads per lane in flight),
 * computes their blocks, and compacts the keys of its region into a list
 * in shared memory (ballot + prefix count, input order kept).  The lanes
 * then take the list densely, one entry per lane at a time, and write flags /
 * OR words as the one-key-per-lane kernel does.  One entry per lane with four resident
 * blocks per SM (64-byte blocks; two for 128-byte blocks, whose words take
 * twice the registers) keeps more warps issuing than four entries per lane
 * with two blocks: on the 2^32-bit filter of 64-byte blocks, 2^28 keys,
 * 20.3 / 27.2 G keys/s (insert / query) against 16.9 / 21.3; two entries
 * with three blocks 19.7 / 25.5 (masks in registers then; with the query's
 * columns in shared memory 5.52 ms, with three or five blocks 6.22 / 7.44).
 * Each key is served by exactly one
 * pass; a query's flag is written there (a key of another shard's block
 * gets 0 in the first pass). */
/* keys per lane per warp tile (the rows of 128-byte blocks leave shared
 * memory for half as many) */
constexpr int region_kpl(int block_bytes) { return block_bytes <= 64 ? 8 : 4; }
constexpr int kRegionWarps = 8; /* 256 threads */

template <class K, class S, int CG, bool INSERT>
__global__ void __launch_bounds__(256, CG * sizeof(S) <= 64 ? 4 : 2) bloom_region_kernel(const BloomArgs a)
{
    constexpr int SB = sizeof(S);
    constexpr int BB = CG * SB;
    constexpr int kRegionKpl = region_kpl(BB);
    constexpr int WT = 32 * kRegionKpl; /* keys per warp tile */
    static_assert(BB <= 128, "block of one lane");
    static_assert(WT <= 256, "tile offsets are one byte");

    __shared__ K s_key[kRegionWarps][WT];
    __shared__ uint32_t s_rel[kRegionWarps][WT];       /* block - region_lo */
    __shared__ unsigned char s_off[kRegionWarps][WT];  /* position in the tile */
    using Bulk = BulkOr<S, CG>;
    constexpr bool kBulk = INSERT && Bulk::kUsed && BB <= 64; /* 48 KiB in all */
    __shared__ alignas(16) unsigned char s_rows[kBulk ? 256 * Bulk::kRow : 16];
    __shared__ uint32_t s_words[INSERT ? 1 : BB / 4 * 256];

    S *const words = reinterpret_cast<S *>(a.words);
    const K *const keys = reinterpret_cast<const K *>(a.keys);
    const K seed = K(a.seed);
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const unsigned lanemask_lt = (1u << lane) - 1u;
    const uint64_t gwarp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;

    LookFirst look;
    for (uint64_t base = gwarp * WT; base < a.n; base += nwarps * WT) {
        K kk[kRegionKpl];
#pragma unroll
        for (int j = 0; j < kRegionKpl; ++j) {
            const uint64_t i = base + uint64_t(j) * 32 + lane;
            kk[j] = i < a.n ? ld_stream(keys + i) : K(0);
        }
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < kRegionKpl; ++j) {
            const uint64_t i = base + uint64_t(j) * 32 + lane;
            const uint64_t blk =
                mod_hash<K>(hash_key<K>(a.hasher, K(kk[j] + seed)), a.num_blocks, a.magic_blocks) -
                a.block_base;
            if constexpr (!INSERT) {
                if (i < a.n && a.region_lo == 0 && blk >= a.local_blocks) a.flags_out[i] = 0;
            }
            const bool in = i < a.n && blk < a.local_blocks && blk >= a.region_lo &&
                            blk < a.region_hi;
            const unsigned m = __ballot_sync(kFull, in);
            if (in) {
                const int pos = cnt + __popc(m & lanemask_lt);
                s_key[wib][pos] = kk[j];
                s_rel[wib][pos] = uint32_t(blk - a.region_lo);
                s_off[wib][pos] = (unsigned char)(j * 32 + lane);
            }
            cnt += __popc(m);
        }
        __syncwarp();
        for (int e0 = 0; e0 < cnt; e0 += 32) {
            const int e = e0 + lane;
            const K key = e < cnt ? s_key[wib][e] : K(0);
            const uint64_t w0 = e < cnt ? (a.region_lo + s_rel[wib][e]) * CG : kNoBlock;
            if constexpr (INSERT) {
                const bool read = look.now();
                const bool there = bloom_or<K, S, CG, kBulk>(
                    a, key, w0, s_rows + (kBulk ? threadIdx.x * Bulk::kRow : 0), read);
                if constexpr (kBulk) {
                    if (read) look.looked(w0 != kNoBlock, there);
                    look.next();
                }
            } else if (e < cnt) {
                S w[CG];
                if (w0 + CG <= a.num_slots) {
                    load_block<S, CG>(words + w0, w);
                } else {
#pragma unroll
                    for (int s = 0; s < CG; ++s) w[s] = __ldcg(words + (w0 + s) % a.num_slots);
                }
                a.flags_out[base + s_off[wib][e]] =
                    (unsigned char)block_has_all<K, S, CG>(key, seed, a.hasher, a.k, w,
                                                           s_words + threadIdx.x);
            }
        }
        __syncwarp();
    }
    if constexpr (kBulk) Bulk::finish();
}

} // namespace b200
} // namespace warpcore

#endif /* WC_BLOOM_CUH */
