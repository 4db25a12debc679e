// The lattice on compact keys: the main path of every operation.
//
// Every coordinate of a vertex key of remainder r is (d+1)*q_i + r with an integer quotient
// q_i (canonical[r][j] = r for j <= d-r, else r-(d+1), src/Permutohedral.h:247-254), so a key
// is r and d quotients.  A compact key packs them, each quotient biased by half its field's
// range, into 64 bits for d <= 7 (fields of 16 bits up to d = 3, then 15, 12, 10 and 8) or
// 128 bits for d >= 8 (14 bits at d = 8, 9 up to d = 12, 7 above).  Against keys of d int16
// lanes (16 to 48 bytes a slot):
//  * a sector of 32 bytes, one 256-bit load, holds four (two) slots.  The table probes by
//    sector: at the default load a lookup reads 1.02 (1.09) sectors and the longest of a
//    warp's 32 lookups 1.4 (2.3), where slot-by-slot probing took 1.3 and 4.7 dependent reads;
//  * a slot fills with one 64-bit (128-bit) compare-and-swap, so inserts of d >= 8 need no
//    pending state, fences or second read;
//  * the steps to the next remainder and to a neighbour are an add of one field, the hash
//    a few 32-bit multiplies.
// Quotients reach about 0.8 of a position in sigmas, so the fields hold images 2500 sigmas wide
// and more at d <= 5 and d = 8, 640 at d = 6, 155 at d = 7, 315 at d = 9 to 12 and 75 from d = 13
// on: 1080p does not fit d = 7 at sigma 8, nor d = 10 at sigma 4.  Images whose pixel coordinates
// leave that range start on the int16-lane keys; a point whose keys do not fit sets kStatusWide
// in the splat, before anything is written, and the host runs the lattice again on them.  A
// slice at other positions asks for no rerun: a position out of the fields' range takes the
// int16 arithmetic on its own (slice_far_point).
#pragma once

#include <type_traits>

#include "lattice_kernels.cuh"

namespace pgpu {

template <int D>
struct CompactKey {
    static constexpr bool kOneWord = D <= 7;          // 64 bits, else 128
    using T = typename std::conditional<kOneWord, uint64_t, uint4>::type;
    static constexpr int kBucket = kOneWord ? 4 : 2;  // slots of a 32-byte sector
    static constexpr int kRemBits = D + 1 <= 2 ? 1 : D + 1 <= 4 ? 2 : 3;   // of 64-bit keys
    static constexpr int kPerWord = (D + 3) / 4;      // 128-bit keys: fields per 32-bit word
    static constexpr int kFieldBits = kOneWord ? ((63 - kRemBits) / D < 16 ? (63 - kRemBits) / D : 16)
                                      : kPerWord == 2 ? 14 : kPerWord == 3 ? 9 : 7;
    // Largest quotient of a greedy point.  The walk back onto the hyperplane moves it by one, a
    // remainder's step lowers it by one and a neighbour lies one further either way, and all of
    // these have to stay inside the field: a carry would make another vertex's key of it.
    // And coordinates stay clear of the int16 range's ends, where the reference's short keys wrap.
    static constexpr int kMaxField = (1 << (kFieldBits - 1)) - 3;
    static constexpr int kMaxAbs = 32767 / (D + 1) - 2;
    static constexpr int kMaxQ = kMaxAbs < kMaxField ? kMaxAbs : kMaxField;
    static_assert(kMaxQ + 3 <= (1 << (kFieldBits - 1)) && kMaxQ + 2 < (1 << (kFieldBits - 1)),
                  "the neighbours of a point's vertices fit the fields");
    __host__ __device__ static constexpr int word(int i) { return kOneWord ? 0 : i / kPerWord; }
    __host__ __device__ static constexpr int shift(int i) {
        return kOneWord ? kRemBits + i * kFieldBits : (i % kPerWord) * kFieldBits;
    }
    // one of every field: all quotients a step up
    __host__ __device__ static constexpr uint64_t ones64() {
        uint64_t b = 0;
        for (int i = 0; i < D; ++i) b += 1ull << shift(i);
        return b;
    }
    __host__ __device__ static constexpr uint32_t ones32(int w) {
        uint32_t b = 0;
        for (int i = 0; i < D; ++i)
            if (word(i) == w) b += 1u << shift(i);
        return b;
    }
};

// 1 << s, 0 from s = 32 up
__device__ __forceinline__ uint32_t bit32(uint32_t s) {
    uint32_t r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(s));
    return r;
}

__device__ __forceinline__ bool ck_equal(uint64_t a, uint64_t b) { return a == b; }
__device__ __forceinline__ bool ck_equal(const uint4& a, const uint4& b) { return words_equal(a, b); }
// an empty slot is all ones.  No 32-bit word of a 128-bit key is all ones, so a word that is
// marks an empty slot, or a read that raced with its one-time fill (the compare-and-swap decides).
__device__ __forceinline__ bool ck_empty(uint64_t a) { return (int32_t)(a >> 32) < 0; }   // keys use 63 bits
__device__ __forceinline__ bool ck_empty(const uint4& a) { return maybe_empty(a); }
__device__ __forceinline__ uint64_t ck_swap(uint64_t* p, uint64_t k) {
    return atomicCAS(reinterpret_cast<unsigned long long*>(p), ~0ull, k);
}
__device__ __forceinline__ uint4 ck_swap(uint4* p, const uint4& k) {
    return atomicCAS(p, make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu), k);
}

// key of remainder 0 from the greedy point's quotients
template <int D>
__device__ __forceinline__ typename CompactKey<D>::T ck_first(const int (&q)[D + 1]) {
    using K = CompactKey<D>;
    if constexpr (K::kOneWord) {
        uint64_t k = K::ones64() << (K::kFieldBits - 1);
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const int s = K::shift(i);
            if (s < 31) k += (uint64_t)((int64_t)q[i] * (int64_t)(1 << s));
            else k += (uint64_t)((uint32_t)q[i] << (s - 32)) << 32;
        }
        return k;
    } else {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = K::ones32(j) << (K::kFieldBits - 1);
#pragma unroll
        for (int i = 0; i < D; ++i) w[K::word(i)] += (uint32_t)q[i] << K::shift(i);
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The code of coordinate i that a thread's scratch column holds by rank: the bit position of
// its field (64-bit keys; 64: the implied coordinate), or word * 32 + bit (128-bit keys;
// 128: implied).
template <int D>
__device__ __forceinline__ constexpr uint32_t ck_code(int i) {
    using K = CompactKey<D>;
    return i == D ? (K::kOneWord ? 64u : 128u) : (uint32_t)(K::word(i) * 32 + K::shift(i));
}

// Key of remainder r+1 from that of r: r grows by one, the quotient of the coordinate ranked
// d-r (code) drops by one.
template <int D>
__device__ __forceinline__ void ck_step(uint64_t& k, uint32_t code, int) {
    k += 1ull - (((uint64_t)bit32(code - 32u) << 32) | bit32(code));
}
template <int D>
__device__ __forceinline__ void ck_step(uint4& k, uint32_t code, int r) {
    const uint32_t bit = 1u << (code & 31u), w = code >> 5;
    k.x -= w == 0 ? bit : 0u;
    k.y -= w == 1 ? bit : 0u;
    k.z -= w == 2 ? bit : 0u;
    k.w -= w == 3 ? bit : 0u;
    // the remainder: four bits on top of word 3, the fifth on top of word 2
    k.w += 1u << 28;
    if (D >= 16 && r + 1 == 16) k.z += 1u << 28;
}

// 32-bit hash, its high bits used: a linear mix of the words, folded
__device__ __forceinline__ uint32_t ck_fold(uint32_t h) { return (h ^ (h >> 15)) * 0x2C1B3C6Du; }
__device__ __forceinline__ uint32_t ck_mix(uint64_t k) {
    return (uint32_t)k * 0x9E3779B1u + (uint32_t)(k >> 32) * 0x85EBCA77u;
}
__device__ __forceinline__ uint32_t ck_mix(const uint4& k) {
    return k.x * 0x9E3779B1u + k.y * 0x85EBCA77u + k.z * 0xC2B2AE3Du + k.w * 0x27D4EB2Fu;
}

// the key's remainder
template <int D>
__device__ __forceinline__ int ck_remainder(uint64_t k) {
    return (int)((uint32_t)k & ((1u << CompactKey<D>::kRemBits) - 1u));
}
template <int D>
__device__ __forceinline__ int ck_remainder(const uint4& k) {
    return (int)((k.w >> 28) + ((k.z >> 28) << 4));
}

// Neighbours (src/Permutohedral.h:446-451) one step up (+1) or down (-1) along axis j: every
// coordinate moves by one, the remainder with it, except coordinate j, which moves by -d, that is
// one and a quotient back.  ck_shift_all: all coordinates moved; ck_axis: quotient j put back
// (j == d, the implied coordinate: nothing).
template <int D>
__device__ __forceinline__ uint64_t ck_shift_all(uint64_t k, int sign) {
    const int r = ck_remainder<D>(k);
    if (sign > 0) return r < D ? k + 1ull : k - (uint64_t)D + CompactKey<D>::ones64();
    return r > 0 ? k - 1ull : k + (uint64_t)D - CompactKey<D>::ones64();
}
template <int D>
__device__ __forceinline__ uint4 ck_shift_all(uint4 k, int sign) {
    using K = CompactKey<D>;
    const int r = ck_remainder<D>(k);
    const int to = sign > 0 ? (r < D ? r + 1 : 0) : (r > 0 ? r - 1 : D);
    k.w = (k.w & 0x0FFFFFFFu) | ((uint32_t)to << 28);
    if (D >= 16) k.z = (k.z & 0x0FFFFFFFu) | ((uint32_t)(to >> 4) << 28);
    if (sign > 0 ? r == D : r == 0) {
        const uint32_t s = sign > 0 ? 1u : ~0u;   // all quotients a step up (down)
        k.x += s * K::ones32(0);
        k.y += s * K::ones32(1);
        k.z += s * K::ones32(2);
        k.w += s * K::ones32(3);
    }
    return k;
}
template <int D>
__device__ __forceinline__ uint64_t ck_axis(uint64_t k, int j, int sign) {
    if (j == D) return k;
    const uint64_t one = 1ull << CompactKey<D>::shift(j);
    return sign > 0 ? k - one : k + one;
}
template <int D>
__device__ __forceinline__ uint4 ck_axis(uint4 k, int j, int sign) {
    if (j == D) return k;
    const uint32_t one = sign > 0 ? 0u - (1u << CompactKey<D>::shift(j)) : 1u << CompactKey<D>::shift(j);
    const int w = CompactKey<D>::word(j);
    if (w == 0) k.x += one;
    else if (w == 1) k.y += one;
    else if (w == 2) k.z += one;
    else k.w += one;
    return k;
}

// the int16-lane key of a compact key (parity dumps)
template <int D>
__device__ __forceinline__ void ck_widen(const typename CompactKey<D>::T& k, Key<key_words(D)>& out) {
    using K = CompactKey<D>;
    const int r = ck_remainder<D>(k);
    int kc[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        uint32_t f;
        if constexpr (K::kOneWord) f = (uint32_t)(k >> K::shift(i));
        else f = word_u32(k, K::word(i)) >> K::shift(i);
        const int q = (int)(f & ((1u << K::kFieldBits) - 1u)) - (1 << (K::kFieldBits - 1));
        kc[i] = q * (D + 1) + r;
    }
    pack_key<D>(kc, out);
}

// ---------------------------------------------------------------------------------
// hash table: one sector (kBucket slots) per probe, sectors probed linearly; slots fill in
// order within a sector and are never emptied
// ---------------------------------------------------------------------------------
// a sector, read past L1 (other SMs fill slots meanwhile)
__device__ __forceinline__ void load_sector(const uint64_t* p, uint64_t (&k)[4]) {
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(k[0]), "=l"(k[1]), "=l"(k[2]), "=l"(k[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ uint4 pair_u4(uint64_t a, uint64_t b) {
    return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ void load_sector(const uint4* p, uint4 (&k)[2]) {
    uint64_t w[4];
    load_sector(reinterpret_cast<const uint64_t*>(p), w);
    k[0] = pair_u4(w[0], w[1]);
    k[1] = pair_u4(w[2], w[3]);
}
// a sector of a table that no thread modifies any more
__device__ __forceinline__ void read_sector(const uint64_t* p, uint64_t (&k)[4]) {
    asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
        : "=l"(k[0]), "=l"(k[1]), "=l"(k[2]), "=l"(k[3]) : "l"(p));
}
__device__ __forceinline__ void read_sector(const uint4* p, uint4 (&k)[2]) {
    uint64_t w[4];
    read_sector(reinterpret_cast<const uint64_t*>(p), w);
    k[0] = pair_u4(w[0], w[1]);
    k[1] = pair_u4(w[2], w[3]);
}

constexpr unsigned kStatusFailed = kStatusProbeLimit | kStatusSpinLimit | kStatusKeyRange | kStatusWide;

// Find-or-insert, from sector b whose slots the caller has loaded into k: the slot, or -1
// (status bit set).  *created is set when this call filled the slot.
template <int D>
__device__ __forceinline__ int ck_insert(typename CompactKey<D>::T* tab, uint32_t sectors,
                                         const typename CompactKey<D>::T& key, uint32_t b,
                                         typename CompactKey<D>::T (&k)[CompactKey<D>::kBucket], unsigned* status,
                                         bool* created) {
    constexpr int B = CompactKey<D>::kBucket;
#pragma unroll 1
    for (uint32_t probe = 0;; ++probe) {
        int hit = -1, free = B;
#pragma unroll
        for (int s = B - 1; s >= 0; --s) {
            hit = ck_equal(k[s], key) ? s : hit;
            free = ck_empty(k[s]) ? s : free;
        }
        if (hit >= 0) return (int)(b * B + hit);
        // the first empty slot, and those behind it if others fill it meanwhile
#pragma unroll 1
        for (; free < B; ++free) {
            const auto old = ck_swap(tab + (size_t)b * B + free, key);
            if (ck_equal(old, key)) return (int)(b * B + free);
            if (ck_empty(old)) {
                *created = true;
                return (int)(b * B + free);
            }
        }
        // A probe this long means a table (nearly) full; once the lattice has overflowed,
        // give up early, so a table sized too small fails fast and is rerun.
        if (probe + 1 == kMaxProbe / B) break;
        if ((probe & 63u) == 63u && (__ldcg(status) & kStatusProbeLimit)) return -1;
        b = b + 1 == sectors ? 0u : b + 1;
        load_sector(tab + (size_t)b * B, k);
    }
    atomicOr(status, kStatusProbeLimit);
    return -1;
}

// slot of a key in a finished table, from sector b already read into k; -1 if absent
template <int D>
__device__ __forceinline__ int ck_find(const typename CompactKey<D>::T* tab, uint32_t sectors,
                                       const typename CompactKey<D>::T& key, uint32_t b,
                                       typename CompactKey<D>::T (&k)[CompactKey<D>::kBucket]) {
    constexpr int B = CompactKey<D>::kBucket;
#pragma unroll 1
    for (int probe = 0; probe < kMaxProbe / B; ++probe) {
        int hit = -1;
        bool end = false;
#pragma unroll
        for (int s = 0; s < B; ++s) {
            hit = ck_equal(k[s], key) ? s : hit;
            end = end || ck_empty(k[s]);
        }
        if (hit >= 0) return (int)(b * B + hit);
        if (end) return -1;
        b = b + 1 == sectors ? 0u : b + 1;
        read_sector(tab + (size_t)b * B, k);
    }
    return -1;
}

// a slot's tag: odd, from hash bits that the home sector does not use
__device__ __forceinline__ uint8_t ck_tag(uint32_t mix) { return (uint8_t)(ck_fold(mix) | 1u); }

// Of eight slots' tags (slot 0's the low byte), those from slot `first` on that may be `tag`, up to
// the first empty slot: the top bit of each one's byte, counted from slot `first`.  Every tag that
// matches is among them (a byte next above one may be too, the key decides); slots behind the
// eight never are.  *end: one of them is empty.
__host__ __device__ __forceinline__ uint64_t tag_matches(uint64_t word, uint32_t first, uint8_t tag, bool* end) {
    constexpr uint64_t kOnes = 0x0101010101010101ull, kTops = 0x8080808080808080ull;
    const uint32_t sh = first * 8u;
    // behind the word's end, bytes that are not empty
    const uint64_t x = sh ? (word >> sh) | (0x0202020202020202ull << (64u - sh)) : word;
    const uint64_t empty = (x - kOnes) & ~x & kTops;   // lowest set: the first zero byte
    const uint64_t y = x ^ (tag * kOnes);
    uint64_t match = (y - kOnes) & ~y & kTops & (~0ull >> sh);
    if (empty) match &= (empty & (0 - empty)) - 1;
    *end = empty != 0;
    return match;
}

// the slot of a 128-bit key by the slots' tags, from slot s (a sector's first) on; word: the
// eight tags that hold s's.  -1 if absent.  Slots of a sector fill in order, so tags behind the
// first empty one are not the key's.  (As many slots as ck_insert tries: kMaxProbe, from s on,
// lie in one word more than kMaxProbe / 8 where s is not a word's first.)
__device__ __forceinline__ int ck_find_tagged(const uint4* tab, const uint64_t* tags, uint32_t cap, const uint4& key,
                                              uint32_t s, uint64_t word) {
    const uint8_t tag = ck_tag(ck_mix(key));
#pragma unroll 1
    for (int probe = 0; probe <= kMaxProbe / 8; ++probe) {
        bool end;
        uint64_t match = tag_matches(word, s & 7u, tag, &end);
        for (; match; match &= match - 1) {
            const uint32_t at = s + ((uint32_t)(__ffsll((long long)match) - 1) >> 3);
            if (words_equal(__ldg(tab + at), key)) return (int)at;
        }
        if (end) return -1;
        s = (s | 7u) + 1u;
        if (s >= cap) s = 0;
        word = __ldg(tags + (s >> 3));
    }
    return -1;
}

// ---------------------------------------------------------------------------------
// simplex
// ---------------------------------------------------------------------------------
// The simplex of one point (the arithmetic of compute_simplex, bit for bit): quotients of the
// greedy point in q, and in the thread's scratch column, by rank, the coordinate's delta and
// code.  False, with nothing to use, when a quotient is out of range or not a number.
// scr: d+1 entries, `stride` apart.
template <int D>
__device__ __forceinline__ bool compact_simplex(const float (&p)[D], const LatticeConsts& lc, int (&q)[D + 1],
                                                uint2* scr, int stride) {
    using K = CompactKey<D>;
    float e[D + 1];
    elevate<D>(p, lc, e);
    const float scale = lc.inv_d1;
    constexpr float dp1 = (float)(D + 1);
    float g[D + 1], diff[D + 1];
    int sum = 0;
    bool fits = true;
#pragma unroll
    for (int i = 0; i <= D; ++i) {
        const float fl = floorf(__fmul_rn(e[i], scale));
        const float down = __fmul_rn(fl, dp1);
        const float up = __fadd_rn(down, dp1);
        const bool pick_up = __fsub_rn(up, e[i]) < __fsub_rn(e[i], down);
        g[i] = pick_up ? up : down;
        fits = fits && fabsf(g[i]) <= (float)K::kMaxQ * dp1;
        q[i] = __float2int_rz(fl) + (pick_up ? 1 : 0);
        sum += q[i];
        diff[i] = __fsub_rn(e[i], g[i]);
    }
    // ranks (of equal differences, the later coordinate ranks higher): up to d = 7 as 4-bit
    // fields of one register
    uint32_t ranks = 0;
    int rank[D + 1];
    if constexpr (D <= 7) {
#pragma unroll
        for (int i = 1; i <= D; ++i) ranks += (uint32_t)i << (4 * i);
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = i + 1; j <= D; ++j)
                if (diff[i] < diff[j]) ranks += (1u << (4 * i)) - (1u << (4 * j));
    } else {
#pragma unroll
        for (int i = 0; i <= D; ++i) rank[i] = i;
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = i + 1; j <= D; ++j)
                if (diff[i] < diff[j]) rank[i] += 1, rank[j] -= 1;
    }
    // back onto the hyperplane (src/Permutohedral.h:326-348): ranks move by sum, and those
    // that leave 0..d (on sum's side) wrap around, their coordinate d+1 the other way
    const int turn = sum > 0 ? D + 1 : -(D + 1), step = sum > 0 ? 1 : -1;
    const float fturn = (float)turn;
#pragma unroll
    for (int i = 0; i <= D; ++i) {
        int t = (D <= 7 ? (int)((ranks >> (4 * (D <= 7 ? i : 0))) & 15u) : rank[i]) + sum;
        float gi = g[i];
        if ((unsigned)t > (unsigned)D) t -= turn, q[i] -= step, gi = __fsub_rn(gi, fturn);
        const float delta = __fmul_rn(__fsub_rn(e[i], gi), scale);
        scr[min((unsigned)t, (unsigned)D) * stride] = make_uint2(__float_as_uint(delta), ck_code<D>(i));
    }
    return fits;
}

// weight of remainder r from the deltas by rank: b[0] = delta(rank d) + (1 - delta(rank 0)),
// b[r] = delta(rank d-r) - delta(rank d+1-r) (compute_simplex)
template <int D>
__device__ __forceinline__ float compact_weight(const uint2* scr, int stride, int r) {
    if (r == 0)
        return __fadd_rn(__uint_as_float(scr[D * stride].x), __fadd_rn(1.0f, -__uint_as_float(scr[0].x)));
    return __fsub_rn(__uint_as_float(scr[(D - r) * stride].x), __uint_as_float(scr[(D + 1 - r) * stride].x));
}

// ---------------------------------------------------------------------------------
// splat
// ---------------------------------------------------------------------------------
struct CompactSplatArgs {
    const Segment* segs;
    int nseg;
    uint32_t n_total;      // points of the batch
    LatticeConsts lc;
    void* keys;            // the shared hash-slot array, all ones
    void* rows;            // accumulator rows (FP32, zeroed): by slot, or by vertex (number_rows)
    uint32_t* ft;          // first-touch entry per slot, all ones (parity dumps); null: not tracked
    uint32_t* rec_slot;    // optional [r][n_total] row of every (point, remainder)
    void* rec;             // optional replay record (store_record)
    unsigned* seg_status;  // one status word per segment
    uint32_t blocks;       // direct splat blocks of the batch
    uint32_t tile_blocks;  // tile splat blocks of the batch
    int tile_px;           // pixels per lane of the tile splat
    const Segment* host_segs;   // host copies, nseg <= kParamSegs: pass them as parameters; or null
    // The vertices, numbered in the order the splat creates them (null with ft, whose vertices
    // are numbered afterwards, by first touch): the creator writes a vertex's key and slot,
    // marks its lower neighbours absent (nbr_init), and leaves the number at the slot.
    uint32_t* vcount;      // vertices so far
    uint32_t* seg_counts;  // per segment (batches of several)
    void* vkey;
    uint32_t* vtx2slot;
    uint32_t* slot2vtx;    // number_rows: all ones before
    int* nbr_init;         // as CompactNbrArgs::nbr
    uint32_t nbr_stride;
    uint8_t* tags;         // optional tag per slot (CompactNbrArgs), zeros before
    // rows by vertex: the splat looks up each vertex's number (waiting, where another
    // warp created it a moment ago) and adds to rows[number]; otherwise to rows[slot]
    int number_rows;
};

template <int D>
__device__ __forceinline__ void publish_vertex(const CompactSplatArgs& a, uint32_t slot, uint32_t v,
                                               const typename CompactKey<D>::T& key) {
    reinterpret_cast<typename CompactKey<D>::T*>(a.vkey)[v] = key;
    a.vtx2slot[v] = slot;
    if (a.nbr_init)
        for (int j = 0; j <= D; ++j) a.nbr_init[(size_t)(2 * j + 1) * a.nbr_stride + v] = -1;
    if (D > 7 && a.tags) a.tags[slot] = ck_tag(ck_mix(key));
    // rows were zeroed before the launch and a reader of the number uses nothing else the
    // creator wrote, so no fence orders these stores
    __stcg(a.slot2vtx + slot, v);
}

// The number of the vertex in slot s, created by another warp: wait (bounded) until its
// creator has published it, which takes the creator's inserts and one atomic
// (microseconds); 0xFFFFFFFF with the spin-limit status bit if it is not published within
// kAwaitSpin polls, or at once when another wait of the lattice has given up already
constexpr int kAwaitSpin = 1 << 14;
__device__ __forceinline__ uint32_t await_vertex(const uint32_t* slot2vtx, uint32_t s, unsigned* status) {
    for (int spin = 0; spin < kAwaitSpin; ++spin) {
        const uint32_t v = __ldcg(slot2vtx + s);
        if (v != 0xFFFFFFFFu) return v;
        if ((spin & 63) == 63 && (__ldcg(status) & kStatusSpinLimit)) return 0xFFFFFFFFu;
        __nanosleep(64);
    }
    atomicOr(status, kStatusSpinLimit);
    return 0xFFFFFFFFu;
}

// inclusive sum over the warp's lanes
__device__ __forceinline__ uint32_t warp_sum_to(uint32_t n, unsigned lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, n, o);
        if (lane >= (unsigned)o) n += u;
    }
    return n;
}

// first number of n new vertices of a segment
__device__ __forceinline__ uint32_t reserve_numbers(const CompactSplatArgs& a, int kseg, uint32_t n) {
    if (n == 0) return 0;
    if (a.nseg > 1) atomicAdd(a.seg_counts + kseg, n);
    return atomicAdd(a.vcount, n);
}

// ---------------------------------------------------------------------------------
// tile splat: one block per 2D tile of kTileThreads * NP pixels of one frame (d <= 7)
// ---------------------------------------------------------------------------------
// Neighbouring pixels land on the same lattice vertices (on the 4K d=5 bilateral the 384
// (point, remainder) entries of 8x8 pixels touch about 78 distinct vertices), while the
// direct splat pays a probe of the global table, a trip to L2 or DRAM, per entry.  Here each
// warp takes 32 or 64 pixels of the block's tile, one or two per lane: it finds each
// vertex's entries in shared memory (phases A and B), inserts each distinct vertex into the
// global table once (phase C), and then every lane adds its rows to the global rows with
// fire-and-forget vector reductions and writes its replay records (phase D).  A vertex's
// first touch is the smallest entry that reached it, so the global minimum over warps is the
// reference's first insertion; the vertex set, keys and records equal the direct splat's,
// only the order of the FP32 additions differs.
//
// The warps of a block do not wait for one another after the start (but with
// number_rows, for the vertices' numbers): the latency of one warp's probes hides behind
// other warps' arithmetic.  The block's vertices are numbered by its last warp, with one
// atomic: every vertex number of a batch comes from one counter, which takes about
// 0.6 G atomics/s, and with an atomic per warp the 4K frame's splat took 0.74 ms at 64
// pixels per warp and 0.96 ms at 32, whatever the occupancy.
//
// Finding equal keys takes no atomics: every entry stores its key in its own place and its
// number in a claim table at its key's hash, whichever comes last; then it
// reads the claim back and compares the claimant's key with its own.  Entries of one key
// share a claim, so either all of them find the same claimant, which stands for the
// vertex, or, where another key's entry came last, none; those (3 % of a 4K frame's
// entries) each stand for their vertex themselves and find the same slot in the global table.
// (A compare-and-swap table starts empty in every tile, so nearly every probe met contended
// swaps: 12 shared-memory wavefronts per swap, 0.37 of the splat's 0.75 ms per 4K frame.)
constexpr int kTileThreads = 128;
constexpr int kTileWarps = kTileThreads / 32;
// Pixels per lane.  More pixels share more vertices (NP = 2: 8x8 pixels per warp, 78 vertices for
// 64 pixels of a 4K frame; NP = 1: 8x4, 55 for 32), a small image needs the warps (tile_px_for).
// Four pixels (16x8 per warp, 113 vertices for 128) leave too few warps: 0.66 ms per 4K frame
// against 0.56.
// claim table entries per warp, log2: they later list a warp's vertices and its new ones
__host__ __device__ constexpr int tile_claim_bits(int np) { return np == 1 ? 9 : 10; }
__host__ __device__ constexpr int tile_min_blocks(int d, int np) { return np == 1 ? (d <= 5 ? 12 : 8) : d <= 5 ? 8 : 6; }

// Dynamic shared memory of a tile splat block; per warp: 8 bytes per entry, for the simplex
// scratch, then the key, then (where the entry stands for a vertex) the vertex's row, and
// the claims, which later list the vertices.  (The rows are not summed in shared memory:
// float atomics there are compare-and-swap loops, and a variant that summed each tile's rows
// before one global reduction per vertex took 2.1 ms per 4K frame against 0.73 ms.)
__host__ __device__ constexpr size_t tile_warp_bytes(int d, int np) {
    return (size_t)(d + 1) * np * 32 * 8 + ((size_t)2 << tile_claim_bits(np));
}
__host__ __device__ constexpr size_t tile_smem_bytes(int d, int np) { return tile_warp_bytes(d, np) * kTileWarps; }

// first number of a block's new vertices, of which its warps have s_new
__device__ __forceinline__ uint32_t number_block(const CompactSplatArgs& a, int kseg, const uint32_t* s_new) {
    uint32_t n = 0;
#pragma unroll
    for (int w = 0; w < kTileWarps; ++w) n += s_new[w];
    return reserve_numbers(a, kseg, n);
}

// publish a warp's new vertices, numbered from `at` in list order
template <int D>
__device__ __forceinline__ void publish_list(const CompactSplatArgs& a, const uint16_t* list, const uint32_t* val,
                                             uint32_t count, uint32_t at, unsigned lane) {
#pragma unroll 1
    for (uint32_t j = lane; j < count; j += 32) {
        const uint32_t slot = val[2 * list[j]];
        publish_vertex<D>(a, slot, at + j, __ldcg(reinterpret_cast<const unsigned long long*>(a.keys) + slot));
    }
}

// claim of a key
template <int NP>
__device__ __forceinline__ uint32_t tile_claim(uint64_t k) { return ck_mix(k) >> (32 - tile_claim_bits(NP)); }

// Position and values of pixel (x, y, f).  The usual layouts are read without asking per
// channel: as many guide channels as positions but x and y (1, or 2 where the guide is the
// image), or but x, y and t (3, 4); 0, any other, is read by load_point_xyt.
template <int D, int VDP>
__device__ __forceinline__ int point_layout(const PointSource& s) {
    const int coords = s.coord_mask == 3 ? 2 : s.coord_mask == 7 ? 3 : 0;
    if (coords == 0 || D <= coords || s.pos_channels != D - coords || !s.homogeneous) return 0;
    const bool both = s.pos_is_val && s.val_channels == s.pos_channels && s.pos_channels < VDP;
    if (!both && s.val_channels >= VDP) return 0;
    return 2 * (coords - 2) + (both ? 2 : 1);
}
template <int D, int VDP, int COORDS, bool BOTH>
__device__ __forceinline__ void load_image_point(const PointSource& s, uint32_t x, uint32_t y, uint32_t f,
                                                 float (&p)[D], float (&v)[VDP]) {
    constexpr int NC = D > COORDS ? D - COORDS : 1;
    const float* at = s.pos.base + ((long long)f * s.pos.tstride + (long long)y * s.pos.ystride + x);
    float ch[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k, at += s.pos.cstride) ch[k] = __ldg(at);
#pragma unroll
    for (int k = 0; k < NC; ++k) p[k] = __fmul_rn(ch[k], s.pos_scale[k]);
    if constexpr (D > COORDS) {
        p[NC] = __fmul_rn((float)x, s.coord_scale[0]);
        p[NC + 1] = __fmul_rn((float)y, s.coord_scale[1]);
        if constexpr (COORDS == 3) p[NC + 2] = __fmul_rn((float)f, s.coord_scale[2]);
    }
    if constexpr (BOTH) {
#pragma unroll
        for (int k = 0; k < VDP; ++k) v[k] = k < NC ? ch[k < NC ? k : 0] : k == NC ? 1.0f : 0.0f;
    } else {
        const float* in = s.val.base + ((long long)f * s.val.tstride + (long long)y * s.val.ystride + x);
#pragma unroll
        for (int k = 0; k < VDP; ++k, in += s.val.cstride)
            v[k] = k < s.val_channels ? __ldg(in) : k == s.val_channels ? 1.0f : 0.0f;
    }
}

// Phases A and B of a warp's pixels (positions pp; valid: in the image, cleared where the keys
// are out of range, and kStatusWide set unless status is null): their weights, the list (in s_claim, after use) and number of their
// vertices, each the entry that stands for it, and loc2, each entry's vertex (two entries to a
// register).  The entry of remainder r of pixel k of a lane is e = b*32 + lane, b = k*(D+1) + r.
template <int D, int NP>
__device__ __forceinline__ uint32_t tile_vertices(const float (&pp)[NP][D], const LatticeConsts& lc,
                                                  unsigned* status, uint64_t* s_key, uint16_t* s_claim,
                                                  unsigned lane, bool (&valid)[NP], float (&bary)[NP][D + 1],
                                                  uint32_t (&loc2)[NP * (D + 1) / 2 + 1]) {
    // Phase A: simplices, keys and claims
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        if (!valid[k]) continue;
        uint2* scr = reinterpret_cast<uint2*>(s_key + k * (D + 1) * 32 + lane);
        int q[D + 1];
        if (!compact_simplex<D>(pp[k], lc, q, scr, 32)) {
            if (status) atomicOr(status, kStatusWide);
            valid[k] = false;
            continue;
        }
        float srt[D + 1];
        uint32_t code[D + 1];
#pragma unroll
        for (int i = 0; i <= D; ++i) {
            const uint2 e = scr[i * 32];
            srt[i] = __uint_as_float(e.x);
            code[i] = e.y;
        }
        bary[k][0] = __fadd_rn(srt[D], __fadd_rn(1.0f, -srt[0]));   // compact_weight
#pragma unroll
        for (int i = 1; i <= D; ++i) bary[k][i] = __fsub_rn(srt[D - i], srt[D + 1 - i]);
        uint64_t key = ck_first<D>(q);
#pragma unroll
        for (int r = 0; r <= D; ++r) {
            if (r > 0) ck_step<D>(key, code[D - (r - 1)], r - 1);
            const uint32_t e = (uint32_t)(k * (D + 1) + r) * 32 + lane;
            s_key[e] = key;
            s_claim[tile_claim<NP>(key)] = (uint16_t)e;
        }
    }
    __syncwarp();

    // Phase B: the entry that stands for each entry's vertex
    uint32_t stands = 0;   // bit b: entry b stands for its vertex
#pragma unroll
    for (int k = 0; k < NP; ++k)
#pragma unroll
        for (int r = 0; r <= D; ++r) {
            const int b = k * (D + 1) + r;
            const uint32_t e = (uint32_t)b * 32 + lane;
            uint32_t c = 0;
            if (valid[k]) {
                const uint64_t key = s_key[e];
                c = s_claim[tile_claim<NP>(key)];
                if (s_key[c] != key) c = e;   // the claim went to another key
                if (c == e) stands |= 1u << b;
            }
            if (b & 1) loc2[b >> 1] |= c << 16;
            else loc2[b >> 1] = c;
        }
    __syncwarp();
    const uint32_t n = (uint32_t)__popc(stands), end = warp_sum_to(n, lane);
    uint32_t at = end - n;
    for (uint32_t m = stands; m; m &= m - 1) s_claim[at++] = (uint16_t)((uint32_t)(__ffs(m) - 1) * 32 + lane);
    __syncwarp();
    return __shfl_sync(0xFFFFFFFFu, end, 31);
}
__device__ __forceinline__ uint32_t tile_loc(const uint32_t* loc2, int b) {
    return (b & 1) ? loc2[b >> 1] >> 16 : loc2[b >> 1] & 0xFFFFu;
}

template <int D, int VDP, int NP, bool PARAM>
__global__ void __launch_bounds__(kTileThreads, tile_min_blocks(D, NP))
compact_tile_kernel(CompactSplatArgs a, const __grid_constant__ SegSource<PARAM> ps) {
    using K = CompactKey<D>;
    static_assert(K::kOneWord, "the tile splat keeps 64-bit keys in shared memory");
    constexpr unsigned kAll = 0xFFFFFFFFu;
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t* s_key = reinterpret_cast<uint64_t*>(tile_smem + warp * tile_warp_bytes(D, NP));
    uint16_t* s_claim = reinterpret_cast<uint16_t*>(s_key + NP * (D + 1) * 32);
    uint16_t* s_list = s_claim;                           // the vertices of the warp's pixels, after the claims,
    uint16_t* s_made = s_claim + NP * (D + 1) * 32;       // and those that this warp created
    uint32_t* s_row = reinterpret_cast<uint32_t*>(s_key);   // a vertex's row, after its key: s_row[2*e]
    __shared__ Segment s_sg[1];
    __shared__ uint32_t s_new[kTileWarps];   // vertices each warp created
    __shared__ uint32_t s_done, s_first;
    if (threadIdx.x == 0) s_done = 0;
    int kseg;
    if constexpr (PARAM) {
        kseg = 0;
#pragma unroll
        for (int k = 1; k < kParamSegs; ++k) kseg += k < a.nseg && ps.seg[k].tile_base <= blockIdx.x ? 1 : 0;
        __syncthreads();
    } else {
        kseg = segment_by<&Segment::tile_base>(a.segs, a.nseg, blockIdx.x);
        load_segment(a.segs + kseg, s_sg[0]);   // ends with a barrier
    }
    const Segment& sg = segment_ref<PARAM>(ps, kseg, s_sg[0]);

    unsigned* status = a.seg_status + kseg;
    uint64_t* tab = reinterpret_cast<uint64_t*>(a.keys) + sg.slot_base;
    const uint32_t sectors = sg.cap / K::kBucket;
    uint32_t bt, tx;
    const uint32_t f = div_magic(blockIdx.x - sg.tile_base, sg.tiles_x * sg.tiles_y, sg.tile_fm, &bt);
    const uint32_t ty = div_magic(bt, sg.tiles_x, sg.tile_xm, &tx);
    const uint32_t wsh = sg.warp_shift, wrow = sg.tile_shift - wsh;   // log2 of the warp's width, of warps per row
    const uint32_t x0 = (tx << sg.tile_shift) + ((warp & ((1u << wrow) - 1u)) << wsh);
    const uint32_t y0 = ty * sg.tile_h + (warp >> wrow) * ((uint32_t)(32 * NP) >> wsh);
    const uint32_t W = (uint32_t)sg.src.width, H = (uint32_t)sg.src.height;

    float v[NP][VDP], bary[NP][D + 1];
    uint32_t gi[NP], count, loc2[NP * (D + 1) / 2 + 1];
    bool valid[NP];   // in the image, its keys in range
    {
        const int layout = point_layout<D, VDP>(sg.src);
        float pp[NP][D];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const uint32_t p = lane * NP + k;   // a lane's pixels are neighbours
            const uint32_t px = x0 + (p & ((1u << wsh) - 1u)), py = y0 + (p >> wsh);
            valid[k] = px < W && py < H;
            gi[k] = sg.point_base + (f * H + py) * W + px;
            if (valid[k]) {
                if (layout == 2) load_image_point<D, VDP, 2, true>(sg.src, px, py, f, pp[k], v[k]);
                else if (layout == 1) load_image_point<D, VDP, 2, false>(sg.src, px, py, f, pp[k], v[k]);
                else if (layout == 4) load_image_point<D, VDP, 3, true>(sg.src, px, py, f, pp[k], v[k]);
                else if (layout == 3) load_image_point<D, VDP, 3, false>(sg.src, px, py, f, pp[k], v[k]);
                else load_point_xyt<D, VDP>(sg.src, px, py, f, pp[k], v[k]);
            }
        }
        count = tile_vertices<D, NP>(pp, a.lc, status, s_key, s_claim, lane, valid, bary, loc2);
    }

    // Phase C: each vertex into the global table; its batch slot replaces its key.  (One that
    // cannot be placed fails the lattice, which is rerun: any row will do.)
    uint32_t made = 0;
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < count; j0 += 32) {
        bool created = false;
        uint32_t l = 0;
        if (j0 + lane < count) {
            l = s_list[j0 + lane];
            const uint64_t key = s_key[l];
            const uint32_t b = __umulhi(ck_fold(ck_mix(key)), sectors);
            uint64_t in[K::kBucket];
            load_sector(tab + (size_t)b * K::kBucket, in);
            const int s = ck_insert<D>(tab, sectors, key, b, in, status, &created);
            s_row[2 * l] = sg.slot_base + (uint32_t)max(s, 0);
        }
        const unsigned m = __ballot_sync(kAll, created);
        if (created) s_made[made + __popc(m & ((1u << lane) - 1u))] = (uint16_t)l;
        made += __popc(m);
    }
    // the last of the block's warps to come here numbers the vertices of all (with number_rows,
    // every warp its own); the counter's answer is on its way during phase D (and the
    // fences come before phase D's reductions and stores, for which they would wait)
    bool last = false;
    uint32_t at = 0;
    if (a.vcount) {
        if (lane == 0) s_new[warp] = made;
        __syncwarp();
        if (a.number_rows) {
            // number the block's vertices and publish them, then learn the numbers of
            // vertices other blocks created; a block's own are published by then, so no
            // wait can close a cycle
            __syncthreads();
            if (threadIdx.x == 0) s_first = number_block(a, kseg, s_new);
            __syncthreads();
            at = s_first;
            for (unsigned w = 0; w < warp; ++w) at += s_new[w];
            publish_list<D>(a, s_made, s_row, made, at, lane);
            __syncwarp();
#pragma unroll 1
            for (uint32_t j = lane; j < count; j += 32) {
                const uint32_t l = s_list[j], v = await_vertex(a.slot2vtx, s_row[2 * l], status);
                s_row[2 * l] = v != 0xFFFFFFFFu ? v : 0u;
            }
        } else {
            uint32_t done = 0;
            if (lane == 0) {
                __threadfence_block();
                done = atomicAdd(&s_done, 1u);
            }
            last = __shfl_sync(kAll, done, 0) == kTileWarps - 1;
            if (last) {
                __threadfence_block();
                if (lane == 0) at = number_block(a, kseg, s_new);
            }
        }
    }
    __syncwarp();

    // Phase D: every lane's rows into its vertices' rows, and the replay record.  A lane's
    // pixels often share a vertex (the same remainder of both): one reduction for them.
    float* acc = reinterpret_cast<float*>(a.rows);
    uint32_t rows[NP][D + 1];
#pragma unroll
    for (int r = 0; r <= D; ++r) {
        float c[NP][VDP];
        bool sends[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            rows[k][r] = s_row[2 * tile_loc(loc2, k * (D + 1) + r)];
            sends[k] = valid[k];
#pragma unroll
            for (int i = 0; i < VDP; ++i) c[k][i] = __fmul_rn(bary[k][r], v[k][i]);
#pragma unroll
            for (int j = 0; j < k; ++j) {
                const bool join = sends[k] && sends[j] && rows[j][r] == rows[k][r];
#pragma unroll
                for (int i = 0; i < VDP; ++i)
                    if (join) c[j][i] = __fadd_rn(c[j][i], c[k][i]);
                sends[k] = sends[k] && !join;
            }
        }
#pragma unroll
        for (int k = 0; k < NP; ++k)
            if (sends[k]) atomic_add_row<VDP>(acc + (size_t)rows[k][r] * VDP, c[k]);
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        if (!valid[k]) continue;
        if (a.ft) {
#pragma unroll
            for (int r = 0; r <= D; ++r) atomicMin(a.ft + rows[k][r], gi[k] * (uint32_t)(D + 1) + (uint32_t)r);
        }
        if (a.rec_slot) {
#pragma unroll
            for (int r = 0; r <= D; ++r) a.rec_slot[(size_t)r * a.n_total + gi[k]] = rows[k][r];
        }
        if (a.rec) store_record<D>(a.rec, a.n_total, gi[k], rows[k], bary[k]);
    }
    if (!last) return;
    at = __shfl_sync(kAll, at, 0);
#pragma unroll 1
    for (int w = 0; w < kTileWarps; ++w) {
        const uint64_t* w_key = reinterpret_cast<const uint64_t*>(tile_smem + w * tile_warp_bytes(D, NP));
        publish_list<D>(a, reinterpret_cast<const uint16_t*>(w_key + NP * (D + 1) * 32) + NP * (D + 1) * 32,
                        reinterpret_cast<const uint32_t*>(w_key), s_new[w], at, lane);
        at += s_new[w];
    }
}

// ---------------------------------------------------------------------------------
// direct splat: one thread per point, every entry into the global table.  For lattices
// whose points share few vertices (a learned density above the tile splat's limit) and for
// d >= 8.  The probes of kAhead remainders are in flight together.
// ---------------------------------------------------------------------------------
constexpr int kDirectThreads = 128;
// (d=16, 2M points: two probes in flight and 6 blocks per SM 4.30 ms, four and 4 blocks 4.48)
constexpr int kDirectMinBlocks = 6;
template <int D>
__host__ __device__ constexpr int direct_ahead() { return D <= 7 ? (D + 1 < 4 ? D + 1 : 4) : 2; }
__host__ __device__ constexpr size_t direct_smem_bytes(int d) { return (size_t)(d + 1) * kDirectThreads * 12; }

template <int D, int VDP>
__global__ void __launch_bounds__(kDirectThreads, kDirectMinBlocks) compact_direct_kernel(CompactSplatArgs a) {
    using K = CompactKey<D>;
    using T = typename K::T;
    constexpr int AH = direct_ahead<D>();
    extern __shared__ __align__(16) unsigned char direct_smem[];
    uint2* scr = reinterpret_cast<uint2*>(direct_smem) + threadIdx.x;          // the simplex by rank
    uint32_t* s_row = reinterpret_cast<uint32_t*>(reinterpret_cast<uint2*>(direct_smem) + (D + 1) * kDirectThreads) +
                      threadIdx.x;                                              // slot of each remainder
    __shared__ Segment sg;
    const int kseg = segment_by<&Segment::splat_base>(a.segs, a.nseg, blockIdx.x);
    load_segment(a.segs + kseg, sg);
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x - sg.splat_base) * (uint32_t)kDirectThreads + threadIdx.x;
    unsigned* status = a.seg_status + kseg;
    T* tab = reinterpret_cast<T*>(a.keys) + sg.slot_base;
    const uint32_t sectors = sg.cap / K::kBucket;
    const uint32_t gi = sg.point_base + i;
    bool valid = i < sg.n;
    float v[VDP];
    T first;
    uint32_t mine = 0;   // bit r: this lane created the vertex of remainder r
    if (valid) {
        float p[D];
        load_point<D, VDP>(sg.src, i, p, v);
        int q[D + 1];
        valid = compact_simplex<D>(p, a.lc, q, scr, kDirectThreads);
        if (!valid) atomicOr(status, kStatusWide);
        first = ck_first<D>(q);
    }
    if (valid) {
        T key = first;
#pragma unroll 1
        for (int r0 = 0; r0 <= D; r0 += AH) {
            T kk[AH], in[AH][K::kBucket];
            uint32_t b[AH];
#pragma unroll
            for (int j = 0; j < AH; ++j) {
                const int r = r0 + j;
                if (r > D) break;
                if (r > 0) ck_step<D>(key, scr[(D - (r - 1)) * kDirectThreads].y, r - 1);
                kk[j] = key;
                b[j] = __umulhi(ck_fold(ck_mix(key)), sectors);
                load_sector(tab + (size_t)b[j] * K::kBucket, in[j]);
            }
#pragma unroll
            for (int j = 0; j < AH; ++j) {
                const int r = r0 + j;
                if (r > D) break;
                bool created = false;
                const int s = ck_insert<D>(tab, sectors, kk[j], b[j], in[j], status, &created);
                uint32_t row = 0xFFFFFFFFu;
                if (s >= 0) {
                    row = sg.slot_base + (uint32_t)s;
                    if (a.ft) atomicMin(a.ft + row, gi * (uint32_t)(D + 1) + (uint32_t)r);
                    if (created) mine |= 1u << r;
                    const float w = compact_weight<D>(scr, kDirectThreads, r);
                    float c[VDP];
#pragma unroll
                    for (int k = 0; k < VDP; ++k) c[k] = __fmul_rn(w, v[k]);
                    atomic_add_row<VDP>(reinterpret_cast<float*>(a.rows) + (size_t)row * VDP, c);
                }
                s_row[r * kDirectThreads] = row;
                if (a.rec_slot) a.rec_slot[(size_t)r * a.n_total + gi] = row;
            }
        }
        if (a.rec) {
            uint4* pairs = reinterpret_cast<uint4*>(a.rec);
#pragma unroll 1
            for (int j = 0; j < (D + 1) / 2; ++j)
                pairs[(size_t)j * a.n_total + gi] =
                    make_uint4(s_row[2 * j * kDirectThreads], __float_as_uint(compact_weight<D>(scr, kDirectThreads, 2 * j)),
                               s_row[(2 * j + 1) * kDirectThreads],
                               __float_as_uint(compact_weight<D>(scr, kDirectThreads, 2 * j + 1)));
            if (D % 2 == 0)
                reinterpret_cast<uint2*>(pairs + (size_t)(D / 2) * a.n_total)[gi] =
                    make_uint2(s_row[D * kDirectThreads], __float_as_uint(compact_weight<D>(scr, kDirectThreads, D)));
        }
    }
    if (a.vcount) {
        // numbered remainder by remainder, so that a warp's stores to vertex order are runs
        const uint32_t end = warp_sum_to((uint32_t)__popc(mine), lane);
        uint32_t at = 0;
        if (lane == 31) at = reserve_numbers(a, kseg, end);
        at = __shfl_sync(0xFFFFFFFFu, at, 31);
        T key = first;
#pragma unroll 1
        for (int r = 0; r <= D; ++r) {
            const bool made = (mine >> r) & 1u;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, made);
            if (valid && r > 0) ck_step<D>(key, scr[(D - (r - 1)) * kDirectThreads].y, r - 1);
            if (made) publish_vertex<D>(a, s_row[r * kDirectThreads], at + __popc(m & ((1u << lane) - 1u)), key);
            at += __popc(m);
        }
    }
}

// ---------------------------------------------------------------------------------
// vertices in the reference's order (parity dumps): every occupied slot's index is the rank of
// its first touch among all first touches (the bitmap's prefix popcount)
// ---------------------------------------------------------------------------------
struct CompactRankArgs {
    const void* keys;
    uint32_t cap;
    const uint32_t* ft;
    const uint32_t* bitmap;
    const uint32_t* offs;
    void* vkey;
    uint32_t* vtx2slot;
    uint32_t* slot2vtx;
    int* nbr_init;
    uint32_t nbr_stride;
    uint8_t* tags;
    uint4* wide0;          // the int16-lane keys in vertex order: word 0 ...
    uint4* widen;          // ... and later words, (KW-1) x wide_stride
    uint32_t wide_stride;
};
template <int D>
__global__ void compact_rank_kernel(CompactRankArgs a) {
    using T = typename CompactKey<D>::T;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < a.cap; s += gridDim.x * blockDim.x) {
        const uint32_t f = a.ft[s];
        if (f == 0xFFFFFFFFu) continue;
        const uint32_t w = f >> 5;
        const uint32_t v = a.offs[w] + __popc(a.bitmap[w] & ((1u << (f & 31u)) - 1u));
        const T key = reinterpret_cast<const T*>(a.keys)[s];
        reinterpret_cast<T*>(a.vkey)[v] = key;
        a.vtx2slot[v] = s;
        a.slot2vtx[s] = v;
        if (a.nbr_init)
            for (int j = 0; j <= D; ++j) a.nbr_init[(size_t)(2 * j + 1) * a.nbr_stride + v] = -1;
        if (a.tags) a.tags[s] = ck_tag(ck_mix(key));
        Key<key_words(D)> k;
        ck_widen<D>(key, k);
        a.wide0[v] = k.w[0];
#pragma unroll
        for (int i = 1; i < key_words(D); ++i) a.widen[(size_t)(i - 1) * a.wide_stride + v] = k.w[i];
    }
}

// ---------------------------------------------------------------------------------
// neighbours, and the rows into vertex order
// ---------------------------------------------------------------------------------
enum RowGather { kRowsInPlace = 0, kRowsCopy, kRowsHalf, kRowsBf16, kRowsNormalise };

struct CompactNbrArgs {
    const void* keys;
    int nseg;
    const uint32_t* seg_slot_base;   // nseg + 1 slot boundaries
    const unsigned* seg_status;
    const void* vkey;
    const uint32_t* vtx2slot;
    const uint32_t* slot2vtx;
    const uint32_t* nverts;
    int* nbr;              // neighbours of axis j: up (n1) at 2j*stride, down (n2) at (2j+1)*stride
    uint32_t stride;
    // one lookup per axis: vertex v finds u = n1(v) and, as n2(u) = v, writes v as u's lower
    // neighbour; every lower neighbour is -1 beforehand
    int half;
    // One byte per slot, 0 where empty, else from the key's hash (d >= 8): most neighbours of
    // those lattices are absent and their keys lie all over a table larger than L2, while
    // the tags stay in L2 and tell all but 1 in 100 of the absent ones.
    const uint8_t* tags;
    // the splat's rows (slot space, FP32) copied into vertex order: as they are, rounded to
    // 16 bits, or (homogeneous rows) normalised by their weight, (m_0.., w); kRowsInPlace
    // with rows_in set: normalised in place (rows by vertex)
    int gather;
    const float* rows_in;
    void* rows_out;
    int vdp, wc;
};

template <int VDP>
__device__ __forceinline__ void gather_row(const CompactNbrArgs& a, uint32_t slot, uint32_t v) {
    float r[VDP];
    const uint32_t from = a.gather == kRowsInPlace ? v : slot;
    load_row<VDP, float, float>(a.rows_in, (int)from, r);
    if (a.gather == kRowsNormalise || a.gather == kRowsInPlace) {   // m = sum / w, 0 where w is 0
        float w = r[0];
#pragma unroll
        for (int k = 0; k < VDP; ++k) if (k == a.wc) w = r[k];
#pragma unroll
        for (int k = 0; k < VDP; ++k) r[k] = k == a.wc ? w : (k < a.wc && w != 0.0f) ? r[k] / w : 0.0f;
    }
    if (a.gather == kRowsHalf) store_row<VDP, __half, float>(reinterpret_cast<__half*>(a.rows_out), v, r);
    else if (a.gather == kRowsBf16) store_row<VDP, __nv_bfloat16, float>(reinterpret_cast<__nv_bfloat16*>(a.rows_out), v, r);
    else store_row<VDP, float, float>(reinterpret_cast<float*>(a.rows_out), v, r);
}

// Axes whose probes are in flight together, and blocks per SM: 64-bit keys, two axes and 6 blocks
// (4K d=5: 0.123 ms; six axes and 3 blocks 0.146); 128-bit keys with tags, six and 4 (2M
// points at d=16: 6.9 ms; four axes 7.2).
__host__ __device__ constexpr int nbr_ahead(int d) { return d <= 7 ? 2 : 6; }
__host__ __device__ constexpr int nbr_min_blocks(int d) { return d <= 7 ? 6 : 4; }
template <int D>
__global__ void __launch_bounds__(256, nbr_min_blocks(D)) compact_neighbours_kernel(CompactNbrArgs a) {
    using K = CompactKey<D>;
    using T = typename K::T;
    constexpr int AH = nbr_ahead(D);
    const uint32_t m = *a.nverts;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x) {
        const T key = reinterpret_cast<const T*>(a.vkey)[v];
        const uint32_t slot = __ldg(a.vtx2slot + v);
        // neighbours are looked up in the vertex's own lattice only
        const int kseg = a.nseg > 1 ? segment_of_slot(a.seg_slot_base, a.nseg, slot) : 0;
        // a lattice whose splat failed is rerun by the host: its full table would make every
        // lookup of an absent key probe to the limit, so skip it
        if (__ldcg(a.seg_status + kseg) & kStatusFailed) {
            // (its vertices still take part in the blur: none may be left a stale neighbour)
            for (int j = 0; j < 2 * (D + 1); ++j)
                if (!a.half || j % 2 == 0) a.nbr[(size_t)j * a.stride + v] = -1;
            continue;
        }
        if (a.rows_in) {
            if (a.vdp == 2) gather_row<2>(a, slot, v);
            else if (a.vdp == 4) gather_row<4>(a, slot, v);
            else gather_row<8>(a, slot, v);
        }
        const uint32_t base = __ldg(a.seg_slot_base + kseg);
        const uint32_t sectors = (__ldg(a.seg_slot_base + kseg + 1) - base) / K::kBucket;
        const T* tab = reinterpret_cast<const T*>(a.keys) + base;
        const uint64_t* tags = reinterpret_cast<const uint64_t*>(a.tags + (K::kOneWord ? 0 : base));
#pragma unroll 1
        for (int sign = 1; sign >= (a.half ? 1 : -1); sign -= 2) {
            const T all = ck_shift_all<D>(key, sign);
#pragma unroll
            for (int j0 = 0; j0 <= D; j0 += AH) {
                T in[AH][K::kBucket];
                uint64_t word[AH];
                uint32_t b[AH];
#pragma unroll
                for (int j = 0; j < AH; ++j) {
                    if (j0 + j > D) break;
                    const T k = ck_axis<D>(all, j0 + j, sign);
                    b[j] = __umulhi(ck_fold(ck_mix(k)), sectors);
                    if constexpr (K::kOneWord) read_sector(tab + (size_t)b[j] * K::kBucket, in[j]);
                    else word[j] = __ldg(tags + (b[j] * K::kBucket >> 3));
                }
#pragma unroll
                for (int j = 0; j < AH; ++j) {
                    if (j0 + j > D) break;
                    const T k = ck_axis<D>(all, j0 + j, sign);
                    int s;
                    if constexpr (K::kOneWord) s = ck_find<D>(tab, sectors, k, b[j], in[j]);
                    else s = ck_find_tagged(tab, tags, sectors * K::kBucket, k, b[j] * K::kBucket, word[j]);
                    const int u = s >= 0 ? (int)__ldg(a.slot2vtx + base + s) : -1;
                    int* nbr = a.nbr + (size_t)(2 * (j0 + j)) * a.stride;
                    nbr[(sign > 0 ? 0 : (size_t)a.stride) + v] = u;
                    if (a.half && u >= 0) nbr[(size_t)a.stride + u] = (int)v;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------
// re-elevation slice (src/Permutohedral.h:405-407): the lattice at other positions than the
// splat's; a vertex the splat never created contributes zero.  FP32 rows in slot space.
// ---------------------------------------------------------------------------------
struct CompactSliceArgs {
    const Segment* segs;    // the slice positions, with the splat's slot ranges
    int nseg;
    LatticeConsts lc;
    const void* keys;
    const float* rows;
    int vd;
    unsigned* seg_status;
    uint32_t blocks;
};

template <int VDP>
__device__ __forceinline__ void write_slice(const OutView& ov, int vd, uint32_t x, uint32_t y, uint32_t f,
                                            const float (&acc)[VDP]) {
    float* o = ov.base + (long long)f * ov.tstride + (long long)y * ov.ystride + x;
    float wsum = acc[0];
#pragma unroll
    for (int j = 0; j < VDP; ++j) if (j == vd - 1) wsum = acc[j];
#pragma unroll
    for (int k = 0; k < VDP; ++k)
        if (k < ov.channels) o[(long long)k * ov.cstride] = ov.normalize ? acc[k] / wsum : acc[k];
}

// A vertex's key from its int16 coordinates; false where they are no compact key
template <int D>
__device__ __forceinline__ bool ck_from_coords(const int (&k)[D], typename CompactKey<D>::T& key) {
    using K = CompactKey<D>;
    constexpr int kHalf = 1 << (K::kFieldBits - 1);
    const int r = ((k[0] % (D + 1)) + D + 1) % (D + 1);
    int q[D + 1];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        q[i] = (k[i] - r) / (D + 1);
        ok = ok && q[i] * (D + 1) + r == k[i] && q[i] >= -kHalf && q[i] < kHalf;
    }
    key = ck_first<D>(q);
    if constexpr (K::kOneWord) {
        key += (uint64_t)r;
    } else {
        key.w += (uint32_t)(r & 15) << 28;
        if (D >= 16) key.z += (uint32_t)(r >> 4) << 28;
    }
    return ok;
}

// The slice of a position whose greedy point does not fit a compact key: the reference's int16
// simplex (compute_simplex; a position beyond int16 sets kStatusKeyRange, which fails the
// call), and each vertex on its own.  All vertices of the splat are compact keys, so one that
// is none was never created and contributes zero.  (Deciding this here, and not by a rerun of
// the lattice, matters beyond time: other blocks have written by now, and the output may be
// one of the inputs.)  Rare, so kept out of the callers' registers.
template <int D, int VDP>
__device__ __noinline__ void slice_far_point(const CompactSliceArgs& a, const Segment& sg, uint32_t x, uint32_t y,
                                             uint32_t f, unsigned* status, float (&acc)[VDP]) {
    using K = CompactKey<D>;
    using T = typename K::T;
    constexpr int B = K::kBucket;
    float p[D];
    load_position_xyt<D>(sg.src, x, y, f, p);
    float delta[D + 1];
    unsigned char coord[D + 1];
    Simplex<D> sx;
    compute_simplex<D>(p, a.lc, sx, status, SimplexScratch{delta, coord, 1, 1});
    const T* tab = reinterpret_cast<const T*>(a.keys) + sg.slot_base;
    const uint32_t sectors = sg.cap / B;
#pragma unroll
    for (int k = 0; k < VDP; ++k) acc[k] = 0.0f;
#pragma unroll 1
    for (int r = 0; r <= D; ++r) {
        int kc[D];
        vertex_coords<D>(sx, r, kc);
        T key;
        if (!ck_from_coords<D>(kc, key)) continue;
        const uint32_t b = __umulhi(ck_fold(ck_mix(key)), sectors);
        T in[B];
        read_sector(tab + (size_t)b * B, in);
        const int s = ck_find<D>(tab, sectors, key, b, in);
        if (s < 0) continue;
        float row[VDP];
        load_row<VDP, float, float>(a.rows + (size_t)sg.slot_base * VDP, s, row);
#pragma unroll
        for (int k = 0; k < VDP; ++k) acc[k] = acc_add(acc[k], sx.bary[r] * row[k]);
    }
}

// d <= 7: as the tile splat, a warp finds the vertices of 64 pixels first and looks each up once
constexpr int kTileSlicePx = 2;
template <int D, int VDP>
__global__ void __launch_bounds__(kTileThreads, tile_min_blocks(D, 2)) compact_tile_slice_kernel(
    const __grid_constant__ CompactSliceArgs a) {
    using K = CompactKey<D>;
    constexpr int NP = kTileSlicePx;
    static_assert(kTileThreads * NP == kSliceThreads, "a slice block's pixels");
    extern __shared__ __align__(16) unsigned char slice_smem[];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t* s_key = reinterpret_cast<uint64_t*>(slice_smem + warp * tile_warp_bytes(D, NP));
    uint16_t* s_list = reinterpret_cast<uint16_t*>(s_key + NP * (D + 1) * 32);
    int* s_row = reinterpret_cast<int*>(s_key);
    __shared__ Segment sg;
    const int kseg = segment_of_block(a.segs, a.nseg, blockIdx.x);
    load_segment(a.segs + kseg, sg);
    uint32_t bt, tx;
    const uint32_t fr = div_magic(blockIdx.x - sg.block_base, sg.stiles_x * sg.stiles_y, sg.stile_fm, &bt);
    const uint32_t ty = div_magic(bt, sg.stiles_x, sg.stile_xm, &tx);
    const uint32_t wsh = sg.slice_th == 1 ? 6u : min(3u, sg.slice_shift);   // 64 pixels: 8x8, or a run
    const uint32_t wrow = sg.slice_shift - wsh;
    const uint32_t x0 = (tx << sg.slice_shift) + ((warp & ((1u << wrow) - 1u)) << wsh);
    const uint32_t y0 = ty * sg.slice_th + (warp >> wrow) * ((uint32_t)(32 * NP) >> wsh);
    unsigned* status = a.seg_status + kseg;
    float bary[NP][D + 1];
    uint32_t count, loc2[NP * (D + 1) / 2 + 1];
    bool valid[NP];
    {
        float pp[NP][D];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const uint32_t p = lane * NP + k;
            const uint32_t px = x0 + (p & ((1u << wsh) - 1u)), py = y0 + (p >> wsh);
            valid[k] = px < (uint32_t)sg.src.width && py < (uint32_t)sg.src.height;
            if (valid[k]) load_position_xyt<D>(sg.src, px, py, fr, pp[k]);
        }
        count = tile_vertices<D, NP>(pp, a.lc, nullptr, s_key, s_list, lane, valid, bary, loc2);
    }
    // a lattice whose splat failed is rerun by the host; its output may be its input, so
    // write nothing (the warp decides as one: its lanes look up each other's vertices)
    if (__any_sync(0xFFFFFFFFu, (__ldcg(status) & kStatusFailed) != 0)) return;
    const uint64_t* tab = reinterpret_cast<const uint64_t*>(a.keys) + sg.slot_base;
    const uint32_t sectors = sg.cap / K::kBucket;
#pragma unroll 1
    for (uint32_t j = lane; j < count; j += 32) {
        const uint32_t l = s_list[j];
        const uint64_t key = s_key[l];
        const uint32_t b = __umulhi(ck_fold(ck_mix(key)), sectors);
        uint64_t in[K::kBucket];
        read_sector(tab + (size_t)b * K::kBucket, in);
        s_row[2 * l] = ck_find<D>(tab, sectors, key, b, in);
    }
    __syncwarp();
    const float* rows = a.rows + (size_t)sg.slot_base * VDP;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const uint32_t p = lane * NP + k;
        const uint32_t px = x0 + (p & ((1u << wsh) - 1u)), py = y0 + (p >> wsh);
        float acc[VDP];
        if (!valid[k]) {
            if (px >= (uint32_t)sg.src.width || py >= (uint32_t)sg.src.height) continue;
            slice_far_point<D, VDP>(a, sg, px, py, fr, status, acc);
            write_slice<VDP>(sg.out, a.vd, px, py, fr, acc);
            continue;
        }
#pragma unroll
        for (int i = 0; i < VDP; ++i) acc[i] = 0.0f;
#pragma unroll
        for (int r = 0; r <= D; ++r) {
            const int s = s_row[2 * tile_loc(loc2, k * (D + 1) + r)];
            float row[VDP];
            load_row<VDP, float, float>(rows, s, row);   // zeros where absent
            if (s < 0) continue;
#pragma unroll
            for (int i = 0; i < VDP; ++i) acc[i] = acc_add(acc[i], bary[k][r] * row[i]);
        }
        write_slice<VDP>(sg.out, a.vd, px, py, fr, acc);
    }
}

template <int D, int VDP>
__global__ void __launch_bounds__(kSliceThreads) compact_slice_kernel(const __grid_constant__ CompactSliceArgs a) {
    using K = CompactKey<D>;
    using T = typename K::T;
    constexpr int AH = direct_ahead<D>();
    extern __shared__ __align__(16) unsigned char slice_smem[];
    uint2* scr = reinterpret_cast<uint2*>(slice_smem) + threadIdx.x;
    __shared__ Segment sg;
    const int kseg = segment_of_block(a.segs, a.nseg, blockIdx.x);
    load_segment(a.segs + kseg, sg);
    uint32_t bt, tx;
    const uint32_t fr = div_magic(blockIdx.x - sg.block_base, sg.stiles_x * sg.stiles_y, sg.stile_fm, &bt);
    const uint32_t ty = div_magic(bt, sg.stiles_x, sg.stile_xm, &tx);
    const uint32_t px = (tx << sg.slice_shift) + (threadIdx.x & (sg.slice_tw - 1));
    const uint32_t py = ty * sg.slice_th + (threadIdx.x >> sg.slice_shift);
    if (px >= (uint32_t)sg.src.width || py >= (uint32_t)sg.src.height) return;
    unsigned* status = a.seg_status + kseg;
    // a lattice whose splat failed is rerun by the host; its output may be its input, so
    // write nothing
    if (__ldcg(status) & kStatusFailed) return;
    float p[D];
    load_position_xyt<D>(sg.src, px, py, fr, p);
    int q[D + 1];
    float acc[VDP];
    if (!compact_simplex<D>(p, a.lc, q, scr, kSliceThreads)) {
        slice_far_point<D, VDP>(a, sg, px, py, fr, status, acc);
        write_slice<VDP>(sg.out, a.vd, px, py, fr, acc);
        return;
    }
    const T* tab = reinterpret_cast<const T*>(a.keys) + sg.slot_base;
    const float* rows = a.rows + (size_t)sg.slot_base * VDP;
    const uint32_t sectors = sg.cap / K::kBucket;
    T key = ck_first<D>(q);
#pragma unroll
    for (int k = 0; k < VDP; ++k) acc[k] = 0.0f;
#pragma unroll 1
    for (int r0 = 0; r0 <= D; r0 += AH) {
        T kk[AH], in[AH][K::kBucket];
        uint32_t b[AH];
#pragma unroll
        for (int j = 0; j < AH; ++j) {
            const int r = r0 + j;
            if (r > D) break;
            if (r > 0) ck_step<D>(key, scr[(D - (r - 1)) * kSliceThreads].y, r - 1);
            kk[j] = key;
            b[j] = __umulhi(ck_fold(ck_mix(key)), sectors);
            read_sector(tab + (size_t)b[j] * K::kBucket, in[j]);
        }
        int s[AH];
        float row[AH][VDP];
#pragma unroll
        for (int j = 0; j < AH; ++j) {
            if (r0 + j > D) break;
            s[j] = ck_find<D>(tab, sectors, kk[j], b[j], in[j]);
            load_row<VDP, float, float>(rows, s[j], row[j]);   // zeros where absent
        }
#pragma unroll
        for (int j = 0; j < AH; ++j) {
            const int r = r0 + j;
            if (r > D) break;
            if (s[j] < 0) continue;
            const float w = compact_weight<D>(scr, kSliceThreads, r);
#pragma unroll
            for (int k = 0; k < VDP; ++k) acc[k] = acc_add(acc[k], w * row[j][k]);
        }
    }
    write_slice<VDP>(sg.out, a.vd, px, py, fr, acc);
}

}  // namespace pgpu
