// mtt_device.cuh — device primitives shared by the sm_100a kernels.
//
// Hand evaluation reproduces the reference scoring function fast_7card_score
// (src/tools/mtt_ev_dumper.cu:53-83; copies at honest_multistreet_solver.cu:24-54
// and preflop_grid_generator.cu:47-77) bit for bit, including its
// non-standard parts: no kickers for quads/trips/pairs, a full house takes
// the second trips before the best pair, and high-card hands compare by the
// whole 7-rank mask.  Instead of the reference's per-thread count arrays and
// rank loops it keeps four rank bit-planes (rank seen >=1, >=2, >=3, 4 times),
// a byte of card count per suit and a 13-bit rank mask per suit, so every case
// is a handful of bit operations and at most four __clz with no local memory.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mtt {

struct Planes {
    uint32_t one, two, three, four;
    uint32_t cnt;            // byte s: cards of suit s
    uint32_t sm01, sm23;     // 16-bit halves: rank masks of suits 0, 1 and 2, 3
};

__host__ __device__ __forceinline__ void planes_clear(Planes& p) {
    p.one = p.two = p.three = p.four = 0u;
    p.cnt = p.sm01 = p.sm23 = 0u;
}

__host__ __device__ __forceinline__ void planes_add(Planes& p, int card) {
    const uint32_t b = 1u << (card >> 2);
    p.four |= p.three & b;
    p.three |= p.two & b;
    p.two |= p.one & b;
    p.one |= b;
    p.cnt += 1u << ((card & 3) * 8);
    const uint32_t h = b << ((card & 1) * 16);
    if (card & 2) p.sm23 |= h; else p.sm01 |= h;
}

// Highest set bit: its index (hi_bit: of a non-empty mask; hi_or: -1 for an
// empty one) and the bit itself (0 for an empty mask).
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ int hi_bit(uint32_t m) { return 31 - __clz(m); }
__device__ __forceinline__ int hi_or(uint32_t m) { return 31 - __clz(m); }
__device__ __forceinline__ uint32_t top_bit(uint32_t m) { return __funnelshift_rc(0x80000000u, 0u, __clz(m)); }
__device__ __forceinline__ int bit_count(uint32_t m) { return __popc(m); }
#else
inline int hi_bit(uint32_t m) { return 31 - __builtin_clz(m); }
inline int hi_or(uint32_t m) { return m ? hi_bit(m) : -1; }
inline uint32_t top_bit(uint32_t m) { return m ? 1u << hi_bit(m) : 0u; }
inline int bit_count(uint32_t m) { return __builtin_popcount(m); }
#endif

// Highest card of a 5-rank run in m, 3 for the wheel A-2-3-4-5, else -1
// (f_str, mtt_ev_dumper.cu:57-61).
__host__ __device__ __forceinline__ int straight_high(uint32_t m) {
    const uint32_t two = m & (m >> 1), s = two & (two >> 2) & (m >> 4);
    const int low = (m & 0x100Fu) == 0x100Fu ? 3 : -1;
    return s ? hi_or(s) + 4 : low;
}

// Mask of the suit holding >= 5 cards (at most one can with 7 cards), else 0.
__host__ __device__ __forceinline__ uint32_t flush_mask(const Planes& p) {
    const uint32_t f = (p.cnt + 0x7B7B7B7Bu) & 0x80808080u;   // a byte of 5 or more
    if (!f) return 0u;
    const uint32_t half = f & 0x80800000u ? p.sm23 : p.sm01;
    return (f & 0x80008000u ? half >> 16 : half) & 0x1FFFu;
}

// Score of a flush's rank mask, which holds fewer than five ranks where cards
// of the hand repeat: those add their ranks one by one.  (One test ahead costs
// 30 million hands nothing; one in every step made them 1% slower.)
__host__ __device__ __forceinline__ uint32_t score_flush(uint32_t fm) {
    const int sf = straight_high(fm);
    if (sf >= 0) return (8u << 24) | (uint32_t)sf;
    uint32_t m = fm, score = 5u << 24;
    if (bit_count(fm) < 5) {
        for (int shift = 16; m; shift -= 4) {
            const int r = hi_bit(m);
            score |= (uint32_t)r << shift;
            m ^= 1u << r;
        }
        return score;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int r = hi_bit(m);
        score |= (uint32_t)r << (4 * (4 - k));
        m ^= 1u << r;
    }
    return score;
}

// What the scores without a flush are made of: the highest quads or else
// trips, `rest` the other trips and the pairs (with two trips among 7 cards
// there is no pair, so its highest is the second trips before the best pair),
// `rest2` the pairs below that, and the straight.  Indices are -1 for none.
struct Groups {
    uint32_t sets, rest, rest2;
    int hs, hr, hr2, st;
    bool quads;
};
__host__ __device__ __forceinline__ Groups rank_groups(uint32_t one, uint32_t two, uint32_t three, uint32_t four) {
    Groups g;
    g.quads = four != 0u;
    const uint32_t trips = three & ~four;
    g.sets = four ? four : trips;
    g.hs = hi_or(g.sets);
    g.rest = (two & ~three) | (trips & ~top_bit(g.sets));
    g.hr = hi_or(g.rest);
    g.rest2 = g.rest & ~top_bit(g.rest);
    g.hr2 = hi_or(g.rest2);
    g.st = straight_high(one);
    return g;
}

// Exact reference score (uint32) of 7 cards without a flush.  Every category
// is formed and the highest that holds selected: a warp's lanes hold different
// ones (30 million hands took 230 us either way; the flop dump's keys 3.35 ms
// branching, 3.08 ms selected).
__host__ __device__ __forceinline__ uint32_t score_ranks(uint32_t one, uint32_t two, uint32_t three, uint32_t four) {
    const Groups g = rank_groups(one, two, three, four);
    const uint32_t hs = (uint32_t)g.hs, hr = (uint32_t)g.hr;
    uint32_t s = one;
    s = g.rest ? (1u << 24) | (hr << 12) : s;
    s = g.rest2 ? (2u << 24) | (hr << 8) | ((uint32_t)g.hr2 << 4) : s;
    s = g.sets ? (3u << 24) | (hs << 8) : s;
    s = g.st >= 0 ? (4u << 24) | (uint32_t)g.st : s;
    s = g.sets && g.rest ? (6u << 24) | (hs << 4) | hr : s;
    return g.quads ? (7u << 24) | (hs << 4) : s;
}

// Exact reference score (uint32) of the 7 cards in p.
__host__ __device__ __forceinline__ uint32_t score_planes(const Planes& p) {
    const uint32_t fm = flush_mask(p);
    return fm ? score_flush(fm) : score_ranks(p.one, p.two, p.three, p.four);
}

// Monotone 16-bit key of the same score: key(a) < key(b) <=> score(a) <
// score(b) and equal keys <=> equal scores.  Each category's payload is
// re-based into one contiguous range (high card and flush use their 13-bit
// rank masks, which order like the reference's nibble lists); 16,973 keys
// in all, never 0 and never 0xFFFF, which the scans use as sentinels.
constexpr uint32_t KEY_PAIR = 8192, KEY_TWO_PAIR = 8208, KEY_TRIPS = 8464,
                   KEY_STRAIGHT = 8480, KEY_FLUSH = 8496, KEY_FULL = 16688,
                   KEY_QUADS = 16944, KEY_SFLUSH = 16960;

__host__ __device__ __forceinline__ uint32_t key_planes(const Planes& p) {
    const uint32_t fm = flush_mask(p);
    if (fm) {
        const int sf = straight_high(fm);
        if (sf >= 0) return KEY_SFLUSH + (uint32_t)sf;
        uint32_t m = fm;
        while (bit_count(m) > 5) m &= m - 1u;   // drop the lowest ranks
        return KEY_FLUSH + m;
    }
    const Groups g = rank_groups(p.one, p.two, p.three, p.four);
    const uint32_t hs = (uint32_t)g.hs, hr = (uint32_t)g.hr;
    uint32_t k = p.one;
    k = g.rest ? KEY_PAIR + hr : k;
    k = g.rest2 ? KEY_TWO_PAIR + ((hr << 4) | (uint32_t)g.hr2) : k;
    k = g.sets ? KEY_TRIPS + hs : k;
    k = g.st >= 0 ? KEY_STRAIGHT + (uint32_t)g.st : k;
    k = g.sets && g.rest ? KEY_FULL + ((hs << 4) | hr) : k;
    return g.quads ? KEY_QUADS + hs : k;
}

// Exact reference score of 7 cards: the suits are only counted, and the rank
// mask of a flush, one hand in 33, is gathered when there is one. The
// enumeration of all 133,784,560 hands runs at 100 G hands/s with it, 93 G with
// a rank mask kept for each suit, 86 G with the packed masks of planes_add.
template <typename Card>
__host__ __device__ __forceinline__ uint32_t score7(const Card* c) {
    uint32_t one = 0u, two = 0u, three = 0u, four = 0u, cnt = 0u;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        const uint32_t b = 1u << (c[i] >> 2);
        four |= three & b; three |= two & b; two |= one & b; one |= b;
        cnt += 1u << ((c[i] & 3) * 8);
    }
    const uint32_t f = (cnt + 0x7B7B7B7Bu) & 0x80808080u;
    if (!f) return score_ranks(one, two, three, four);
    const int suit = f & 0xFFFFu ? (f & 0xFFu ? 0 : 1) : (f & 0xFFFFFFu ? 2 : 3);
    uint32_t fm = 0u;
#pragma unroll
    for (int i = 0; i < 7; ++i) fm |= (c[i] & 3) == suit ? 1u << (c[i] >> 2) : 0u;
    return score_flush(fm);
}

// combo id (0..1325) <-> cards, lexicographic over c1 < c2.
__host__ __device__ __forceinline__ int combo_id(int c1, int c2) {
    // pairs before (c1, c1+1): sum_{k<c1} (51-k) = c1*51 - c1*(c1-1)/2
    return c1 * 51 - (c1 * (c1 - 1)) / 2 + (c2 - c1 - 1);
}

}  // namespace mtt
