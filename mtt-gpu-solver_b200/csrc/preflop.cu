// preflop.cu — the preflop anchor chain (src/preflop/preflop_grid_generator.cu):
// the 169 x 169 all-in equity matrix, class-reduced flop equity matrices of
// a flop subset, and DCFR over the closed BTN-vs-BB preflop tree whose flop
// play is co-solved over those matrices.
//
// Two modes.  MTT_PF_REFERENCE reproduces the reference bit for bit where
// its arithmetic is integer (win/tie counts) or order-fixed float (the
// equities and their class averages): the all-in matrix's board samples are
// drawn with replacement from the reference's LCG and its class_to_cards
// mapping (:79-92) is used as written; the flop matrices cover only the
// first 1,176 combos in lexicographic order (:476-491), count a tie as a
// quarter win (wins += 2, ties += 1, total += 2 per runout, :169-171), and
// entries the reference never writes (hero combos touching the flop) are 0.
// MTT_PF_CORRECT draws boards without replacement from a valid card pair per
// class, uses every combo that avoids the flop and counts a tie as half.
//
// Flop matrices: per flop, every combo's 16-bit score key for every
// (turn, river) pair of the 49-card deck is evaluated once into a
// pair-major table, and each hero's list of runouts (the reference's
// subsample: turn index r1 = 0, 2, .. and river r2 = r1+1, r1+4, .. into the
// hero's 47-card deck) into (pair, key) words.  A CTA then holds 64 villains'
// part of the table in shared memory and its warps walk the heroes' lists,
// two villains per 32-bit word and lane.  The combo matrix is reduced to
// classes in the reference's summation order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "mtt_bulk.cuh"
#include "mtt_common.h"
#include "mtt_device.cuh"
#include "mtt_pairs.cuh"

namespace mtt {
namespace pf {

constexpr int NC = 169, PAD = 192, ALIVE = 1176, NPAIR = 1176;   // NPAIR = C(49, 2) turn-river pairs
constexpr int LD_REF = 1216, LD_OK = 1344;   // row length of the combo matrices (reference: 1,216)
constexpr int SAMPLES = 3000;

// class_to_cards of the reference (:79-92), boundary behaviour included: the
// last class of each rank group maps into the next group (A2s becomes two
// copies of the king of clubs).  For classes 90 and 168 the reference's loop
// only ends in signed overflow (undefined); those take their own cards.
__host__ __device__ inline void class_cards_ref(int cls, int& h1, int& h2) {
    if (cls < 13) { const int r = 12 - cls; h1 = r * 4; h2 = r * 4 + 1; return; }
    int base = cls < 91 ? 13 : 91, r1 = 12;
    while (r1 > 0 && base + (r1 - 1) <= cls) base += r1--;
    if (r1 == 0) { h1 = 4; h2 = cls < 91 ? 0 : 1; return; }
    const int r2 = r1 - 1 - (cls - base);
    h1 = r1 * 4;
    h2 = r2 * 4 + (cls < 91 ? 0 : 1);
}

// A valid pair of cards of class cls: pairs c/d, suited c/c, offsuit c/d.
__host__ __device__ inline void class_cards_ok(int cls, int& h1, int& h2) {
    if (cls < 13) { const int r = 12 - cls; h1 = r * 4; h2 = r * 4 + 1; return; }
    const bool suited = cls < 91;
    int k = cls - (suited ? 13 : 91), hi = 12;
    while (k >= hi) { k -= hi; --hi; }
    const int lo = hi - 1 - k;
    h1 = hi * 4;
    h2 = lo * 4 + (suited ? 0 : 1);
}

// First combo of class cls (fixed suit order) that avoids the cards in dead.
__host__ __device__ inline void class_cards_avoid(int cls, uint64_t dead, int& c1, int& c2) {
    int hi, lo;
    bool pair = cls < 13, suited = false;
    if (pair) { hi = lo = 12 - cls; }
    else {
        suited = cls < 91;
        int k = cls - (suited ? 13 : 91);
        hi = 12;
        while (k >= hi) { k -= hi; --hi; }
        lo = hi - 1 - k;
    }
    for (int s1 = 0; s1 < 4; ++s1)
        for (int s2 = 0; s2 < 4; ++s2) {
            if (pair ? s2 <= s1 : (suited ? s2 != s1 : s2 == s1)) continue;
            const int a = hi * 4 + s1, b = lo * 4 + s2;
            if (((dead >> a) & 1ull) || ((dead >> b) & 1ull)) continue;
            c1 = a; c2 = b;
            return;
        }
    c1 = hi * 4; c2 = lo * 4 + 1;   // not reached: two dead cards leave a combo of every class
}

// combo -> class (host set-up, :475-483).
__host__ __device__ constexpr int combo_class(int c1, int c2) {
    const int r1 = c1 / 4, s1 = c1 % 4, r2 = c2 / 4, s2 = c2 % 4;
    const int hi = r1 > r2 ? r1 : r2, lo = r1 < r2 ? r1 : r2;
    if (r1 == r2) return 12 - hi;
    int base = s1 == s2 ? 13 : 91;
    for (int r = 12; r > hi; --r) base += r;
    return base + (hi - 1 - lo);
}

// Rank and suit counts of cards that may repeat: rank counts are exact (a
// rank seen 5+ times is neither quads, trips nor a pair, as with the
// reference's rc[r] == 4 / 3 / 2 tests) and a suit flushes on its card count
// (sc[s] >= 5) with the ranks it holds (sm[s]), as the reference does.
struct DupCards {
    uint32_t one = 0, two = 0, three = 0, four = 0, five = 0;
    uint32_t cnt = 0;          // byte s: cards of suit s
    uint32_t sm01 = 0, sm23 = 0;   // 16-bit halves: ranks held of suits 0, 1 and 2, 3
    __device__ __forceinline__ void add(int card) {
        const uint32_t b = 1u << (card >> 2);
        five |= four & b; four |= three & b; three |= two & b; two |= one & b; one |= b;
        cnt += 1u << ((card & 3) * 8);
        const uint32_t h = b << ((card & 1) * 16);
        if (card & 2) sm23 |= h; else sm01 |= h;
    }
};

__device__ __forceinline__ uint32_t score_dup(const DupCards& d) {
    const uint32_t fl = (d.cnt + 0x7B7B7B7Bu) & 0x80808080u;   // a byte of 5 or more
    if (fl) {
        const int s = (31 - __clz(fl & (0u - fl))) >> 3;       // 7 cards: at most one suit
        const uint32_t ranks = ((s & 2 ? d.sm23 : d.sm01) >> ((s & 1) * 16)) & 0x1FFFu;
        const int sf = straight_high(ranks);
        if (sf >= 0) return (8u << 24) | (uint32_t)sf;
        uint32_t m = ranks, score = 5u << 24;
        for (int p = 0; p < 5 && m; ++p) {
            const int r = hi_bit(m);
            score |= (uint32_t)r << (4 * (4 - p));
            m ^= 1u << r;
        }
        return score;
    }
    const uint32_t quads = d.four & ~d.five, trips = d.three & ~d.four, pairs = d.two & ~d.three;
    if (quads) return (7u << 24) | ((uint32_t)hi_bit(quads) << 4);
    const int t1 = trips ? hi_bit(trips) : -1;
    const uint32_t trips2 = trips & ~(t1 >= 0 ? (1u << t1) : 0u);
    const int t2 = trips2 ? hi_bit(trips2) : -1;
    const int p1 = pairs ? hi_bit(pairs) : -1;
    const uint32_t pairs2 = pairs & ~(p1 >= 0 ? (1u << p1) : 0u);
    const int p2 = pairs2 ? hi_bit(pairs2) : -1;
    if (t1 >= 0 && (t2 >= 0 || p1 >= 0)) return (6u << 24) | ((uint32_t)t1 << 4) | (uint32_t)(t2 >= 0 ? t2 : p1);
    const int st = straight_high(d.one);
    if (st >= 0) return (4u << 24) | (uint32_t)st;
    if (t1 >= 0) return (3u << 24) | ((uint32_t)t1 << 8);
    if (p1 >= 0 && p2 >= 0) return (2u << 24) | ((uint32_t)p1 << 8) | ((uint32_t)p2 << 4);
    if (p1 >= 0) return (1u << 24) | ((uint32_t)p1 << 12);
    return d.one;
}

// The all-in sampler (kernel_gen_preflop_matrix, :95-127).  28,561 class
// pairs are 6 warps an SM, so one thread per pair left the chip waiting on
// dependent steps (9.3 ms, 3.1 us a sample; 1.8 ms now).  In the reference's mode boards
// are drawn with replacement, samples depend only on the generator, and
// AI_SPLIT threads of a pair take a share each, their generators started by
// the LCG's n-step map; counts add up exactly.  Without replacement the deck's
// order carries over from sample to sample, so there one thread keeps a pair,
// its deck in shared memory (AI_DECK words apart by thread: no bank
// conflicts).  Divisions by the deck size are multiplications by its
// reciprocal, exact for 16-bit dividends.
constexpr int AI_SPLIT = 8, AI_THREADS = 128, AI_SHARE = SAMPLES / AI_SPLIT;
static_assert(AI_SHARE * AI_SPLIT == SAMPLES && AI_THREADS % AI_SPLIT == 0, "equal shares");

template <int MODE>
__global__ void __launch_bounds__(AI_THREADS) k_pf_allin(float* __restrict__ out, int* __restrict__ wins_out,
                                                         int* __restrict__ ties_out) {
    constexpr bool REF = MODE == MTT_PF_REFERENCE;
    constexpr int SPLIT = REF ? AI_SPLIT : 1;
    __shared__ uint32_t deck[REF ? 1 : 52][AI_THREADS];
    const int tid = threadIdx.x;
    const int i = (blockIdx.x * AI_THREADS + tid) / SPLIT, part = tid % SPLIT;
    if (i >= NC * NC) return;                 // a pair's threads leave together
    const int hc = i / NC, vc = i % NC;
    if (hc == vc) {
        if (part == 0) {
            out[i] = 0.5f;
            if (wins_out) { wins_out[i] = 0; ties_out[i] = 0; }
        }
        return;
    }
    int h1, h2, v1, v2;
    if (REF) {
        class_cards_ref(hc, h1, h2);
        class_cards_ref(vc, v1, v2);
        if (h1 == v1 || h1 == v2 || h2 == v1 || h2 == v2) {   // the reference's suit switch (:104-107)
            if (h1 == v1 || h2 == v1) v1 = (v1 / 4) * 4 + 2;
            if (h1 == v2 || h2 == v2) v2 = (v2 / 4) * 4 + 3;
        }
    } else {
        class_cards_ok(hc, h1, h2);
        class_cards_avoid(vc, (1ull << h1) | (1ull << h2), v1, v2);
    }
    const uint64_t dead = (1ull << h1) | (1ull << h2) | (1ull << v1) | (1ull << v2);
    const int dsz = 52 - __popcll(dead);
    int gone[4];                              // dead cards ascending, 52 past the last
    {
        uint64_t m = dead;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            gone[k] = m ? __ffsll((long long)m) - 1 : 52;
            m &= m - 1ull;
        }
    }
    if (!REF)
        for (int c = 0, n = 0; c < 52; ++c) if (!((dead >> c) & 1ull)) deck[n++][tid] = (uint32_t)c;
    uint32_t recip[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) recip[k] = 0xFFFFFFFFu / (uint32_t)(dsz - k) + 1u;
    uint32_t rng = (uint32_t)(hc * 169 + vc) * 2654435761u + 0x9E3779B9u;
    if (REF) {                                // 5 * AI_SHARE * part steps ahead: x -> A x + C, squared bit by bit
        uint32_t A = 1664525u, C = 1013904223u;
        for (uint32_t n = 5u * AI_SHARE * (uint32_t)part; n; n >>= 1) {
            if (n & 1u) rng = rng * A + C;
            C = C * (A + 1u);
            A = A * A;
        }
    }
    DupCards hero, vill;
    hero.add(h1); hero.add(h2);
    vill.add(v1); vill.add(v2);
    int wins = 0, ties = 0;
    for (int s = 0; s < SAMPLES / SPLIT; ++s) {
        DupCards a = hero, b = vill;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            rng = rng * 1664525u + 1013904223u;
            const uint32_t x = rng >> 16;
            const int pick = k + (int)(x - __umulhi(x, recip[k]) * (uint32_t)(dsz - k));
            int card;
            if (REF) {                        // the pick-th live card: step over each dead card below it
                card = pick;
#pragma unroll
                for (int q = 0; q < 4; ++q) card += card >= gone[q];
            } else {                          // without replacement: partial Fisher-Yates
                card = (int)deck[pick][tid];
                deck[pick][tid] = deck[k][tid];
                deck[k][tid] = (uint32_t)card;
            }
            a.add(card);
            b.add(card);
        }
        const uint32_t sh = score_dup(a), sv = score_dup(b);
        wins += sh > sv;
        ties += sh == sv;
    }
    if (SPLIT > 1) {
        const unsigned mask = ((1u << SPLIT) - 1u) << ((tid & 31) / SPLIT * SPLIT);
#pragma unroll
        for (int o = SPLIT / 2; o > 0; o >>= 1) {
            wins += __shfl_down_sync(mask, wins, o, SPLIT);
            ties += __shfl_down_sync(mask, ties, o, SPLIT);
        }
        if (part) return;
    }
    out[i] = ((float)wins + 0.5f * (float)ties) / (float)SAMPLES;
    if (wins_out) { wins_out[i] = wins; ties_out[i] = ties; }
}

// Key table of one flop: KT[pair][combo] = hero half (mtt_pairs.cuh) of combo
// with the flop and the (turn, river) pair (dead where cards collide).
__global__ void __launch_bounds__(256) k_pf_keys(const uint8_t* __restrict__ flops, const uint16_t* __restrict__ cc,
                                                 int ncombo, int ld, uint16_t* __restrict__ KT) {
    const int f = blockIdx.y;
    const int p = blockIdx.x;            // pair index over the 49-card deck
    const uint8_t f0 = flops[3 * f], f1 = flops[3 * f + 1], f2 = flops[3 * f + 2];
    const uint64_t fm = (1ull << f0) | (1ull << f1) | (1ull << f2);
    // unrank p -> (a < b) over the 49-card deck
    int a = 0, k = p, row = 48;
    while (k >= row) { k -= row; ++a; --row; }
    const int b = a + 1 + k;
    int n = 0, ta = -1, tb = -1;
    for (int c = 0; c < 52; ++c) {
        if ((fm >> c) & 1ull) continue;
        if (n == a) ta = c;
        if (n == b) tb = c;
        ++n;
    }
    uint16_t* out = KT + ((size_t)f * NPAIR + p) * ld;
    for (int j = threadIdx.x; j < ld; j += blockDim.x) {
        uint16_t key = (uint16_t)KEY_H_DEAD;
        if (j < ncombo) {
            const int c1 = cc[2 * j], c2 = cc[2 * j + 1];
            const uint64_t m = (1ull << c1) | (1ull << c2);
            if (!(m & fm) && c1 != ta && c1 != tb && c2 != ta && c2 != tb) {
                Planes pl; planes_clear(pl);
                planes_add(pl, f0); planes_add(pl, f1); planes_add(pl, f2);
                planes_add(pl, c1); planes_add(pl, c2); planes_add(pl, ta); planes_add(pl, tb);
                key = (uint16_t)(key_planes(pl) + 1u);
            }
        }
        out[j] = key;
    }
}

// Runout k of a 47-card deck in the reference's order: r1 = 0, 2, .., r2 =
// r1 + 1, r1 + 4, ..; 192 of them.
constexpr int RUNS = 192;

// Position in a 49-card deck of card r of the 47-card deck that lacks
// positions a < b.
__device__ __forceinline__ int deck_pos(int r, int a, int b) {
    r += r >= a;
    return r + (r >= b);
}
__device__ __forceinline__ int flop_deck_pos(uint64_t fm, int card) {
    return card - __popcll(fm & ((1ull << card) - 1ull));
}

// Hero lists: HL[f][h][k] = pair index << 16 | hero half of combo h on its
// runout k.  Not written for combos that touch the flop.
__global__ void __launch_bounds__(RUNS) k_pf_runs(const uint8_t* __restrict__ flops, const uint16_t* __restrict__ cc,
                                                  int ncombo, int ld, const uint16_t* __restrict__ KT,
                                                  uint32_t* __restrict__ HL) {
    const int f = blockIdx.y, h = blockIdx.x, k = threadIdx.x;
    const uint64_t fm = (1ull << flops[3 * f]) | (1ull << flops[3 * f + 1]) | (1ull << flops[3 * f + 2]);
    const int c1 = cc[2 * h], c2 = cc[2 * h + 1];
    if (((fm >> c1) | (fm >> c2)) & 1ull) return;
    int r1 = 0, left = k;
    for (;;) {                                 // runouts with this r1: r2 = r1 + 1, r1 + 4, .. < 47
        const int n = (47 - r1 - 1 + 2) / 3;
        if (left < n) break;
        left -= n;
        r1 += 2;
    }
    const int r2 = r1 + 1 + 3 * left;
    const int a = flop_deck_pos(fm, c1), b = flop_deck_pos(fm, c2);
    const int x = deck_pos(r1, a, b), y = deck_pos(r2, a, b);
    const int p = x * 48 - (x * (x - 1)) / 2 + (y - x - 1);
    HL[((size_t)f * ncombo + h) * RUNS + k] = ((uint32_t)p << 16) | KT[((size_t)f * NPAIR + p) * ld + h];
}

// kernel_gen_100_flop_matrices (:130-183): E[f][h][j] = (wins + ties / 2) /
// total of hero h against villain j with the mode's tie weight.  One CTA
// holds EQ_VILL villains' keys of all 1,176 pairs in shared memory (150 KB, a
// word per two villains, 32 words a row: conflict-free) and its warps take
// heroes in turn; a hero's list is staged per warp as (row offset, doubled
// hero half) and read two runouts a 16-byte broadcast.  Per runout and 64
// pairs: one broadcast half, one row load, one packed clamp, its win bits and
// their adds.  Usable runouts are counted by inclusion and exclusion from the
// villain's positions in the hero's deck, not in the loop.  The kernel
// before read the table from L2 one 16-bit key at a time and wrote the matrix
// with a stride of a row: 29.9 ms for 100 flops, 3.5 ms now.
constexpr int EQ_VILL = 64, EQ_WARPS = 32, EQ_THREADS = 32 * EQ_WARPS;
constexpr int EQ_TABLE = NPAIR * EQ_VILL / 2;                       // words
constexpr int EQ_SMEM = 4 * EQ_TABLE + 8 * RUNS * EQ_WARPS;         // 199,680 B

__global__ void __launch_bounds__(EQ_THREADS, 1) k_pf_flop_eq(const uint8_t* __restrict__ flops,
                                                           const uint16_t* __restrict__ cc, int ncombo, int ld, int mode,
                                                           const uint16_t* __restrict__ KT,
                                                           const uint32_t* __restrict__ HL, float* __restrict__ E) {
    extern __shared__ __align__(16) uint32_t eq_smem[];
    __shared__ uint64_t adj[47];               // bit y of adj[x]: 47-card deck positions x and y are a runout
    const int f = blockIdx.y, j0 = blockIdx.x * EQ_VILL;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 47) {
        uint64_t m = 0;
        for (int y = 0; y < 47; ++y) {
            const int lo = min(tid, y), hi = max(tid, y);
            if (lo != hi && !(lo & 1) && (hi - lo - 1) % 3 == 0) m |= 1ull << y;
        }
        adj[tid] = m;
    }
    // ld is a multiple of EQ_VILL: every tile's words exist (dead past ncombo)
    const uint32_t* KTf = reinterpret_cast<const uint32_t*>(KT + (size_t)f * NPAIR * ld + j0);
    for (int e = tid; e < EQ_TABLE; e += EQ_THREADS)
        eq_smem[e] = villain_word(KTf[(size_t)(e >> 5) * (ld >> 1) + (e & 31)]);
    __syncthreads();
    uint2* list = reinterpret_cast<uint2*>(eq_smem + EQ_TABLE) + warp * RUNS;
    const char* table = reinterpret_cast<const char*>(eq_smem + lane);
    const uint64_t fm = (1ull << flops[3 * f]) | (1ull << flops[3 * f + 1]) | (1ull << flops[3 * f + 2]);
    const int j = j0 + 2 * lane;               // this lane's villains: j and j + 1
    int pos[2][2];                             // their positions in the flop's deck
    uint64_t vm[2];
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const int jj = min(j + v, ncombo - 1);
        const int c1 = cc[2 * jj], c2 = cc[2 * jj + 1];
        vm[v] = (1ull << c1) | (1ull << c2);
        pos[v][0] = flop_deck_pos(fm, c1);
        pos[v][1] = flop_deck_pos(fm, c2);
    }
    float* Ef = E + (size_t)f * ld * ld;
    for (int h = warp; h < ncombo; h += EQ_WARPS) {
        const int hc1 = cc[2 * h], hc2 = cc[2 * h + 1];
        const uint64_t hm = (1ull << hc1) | (1ull << hc2);
        float2 eq = make_float2(0.0f, 0.0f);   // heroes on the flop: the reference never writes these; here 0
        if (!(hm & fm)) {
            const uint32_t* src = HL + ((size_t)f * ncombo + h) * RUNS;
            __syncwarp();
#pragma unroll
            for (int k = lane; k < RUNS; k += 32) {
                const uint32_t w = src[k];
                list[k] = make_uint2((w >> 16) * (4u * 32u), (w & 0xFFFFu) * 0x00010001u);
            }
            __syncwarp();
            uint32_t sc = 0u, w2 = 0u;         // halves: 2 wins + ties; 2 wins (at most 2 * 192)
#pragma unroll 8
            for (int k = 0; k < RUNS; k += 2) {
                const uint4 l = *reinterpret_cast<const uint4*>(list + k);
                const uint32_t t0 = pair_2w_t(l.y, *reinterpret_cast<const uint32_t*>(table + l.x));
                const uint32_t t1 = pair_2w_t(l.w, *reinterpret_cast<const uint32_t*>(table + l.z));
                sc += t0 + t1;
                w2 += (t0 & 0x00020002u) + (t1 & 0x00020002u);
            }
            const int a = flop_deck_pos(fm, hc1), b = flop_deck_pos(fm, hc2);
            float r[2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                r[v] = 0.0f;
                if ((vm[v] & hm) || (vm[v] & fm) || j + v >= ncombo) continue;
                const int x = pos[v][0] - (pos[v][0] > a) - (pos[v][0] > b);
                const int y = pos[v][1] - (pos[v][1] > a) - (pos[v][1] > b);
                const int n = RUNS - __popcll(adj[x]) - __popcll(adj[y]) + (int)((adj[x] >> y) & 1ull);
                const int wins = (int)(v ? w2 >> 16 : w2 & 0xFFFFu);
                const int t = (int)(v ? sc >> 16 : sc & 0xFFFFu) - wins;
                const int ties = mode == MTT_PF_REFERENCE ? t : 2 * t;
                r[v] = n > 0 ? ((float)wins + 0.5f * (float)ties) / (float)(2 * n) : 0.0f;
            }
            eq = make_float2(r[0], r[1]);
        }
        *reinterpret_cast<float2*>(Ef + (size_t)h * ld + j) = eq;
    }
}

// kernel_reduce_combo_to_class_matrices (:189-223): out[f][v][h].
__global__ void k_pf_reduce(const float* __restrict__ E, int ld, const int* __restrict__ lists,
                            const int* __restrict__ counts, float* __restrict__ out) {
    const int f = blockIdx.y, hcl = blockIdx.x, vcl = threadIdx.x;
    if (hcl >= NC || vcl >= NC) return;
    const float* Ef = E + (size_t)f * ld * ld;
    float sum = 0.0f;
    int valid = 0;
    for (int i = 0; i < counts[hcl]; ++i) {
        const int ch = lists[hcl * 12 + i];
        for (int j = 0; j < counts[vcl]; ++j) {
            const float eq = Ef[(size_t)ch * ld + lists[vcl * 12 + j]];
            if (eq > 0.0f) { sum = __fadd_rn(sum, eq); valid++; }
        }
    }
    out[((size_t)f * NC + vcl) * NC + hcl] = valid > 0 ? __fdiv_rn(sum, (float)valid) : 0.5f;
}

// Combos of the matrix (reference: the first 1,176 in lexicographic order;
// correct: all 1,326, those touching a flop are zeroed per flop by the kernels)
// and up to CLS_CAP combos per class.  Part of the module: copied in by each
// call, a captured call's replay read the copy's source when it was gone.
constexpr int CLS_CAP = 12;              // the largest class (offsuit) has 12 combos
struct Lists {
    uint16_t cc[2 * 1326];               // 2 per combo
    int lists[NC * CLS_CAP], counts[NC];
    int ncombo;
};
constexpr Lists make_lists(int limit) {
    Lists L{};
    for (int c1 = 0; c1 < 52; ++c1)
        for (int c2 = c1 + 1; c2 < 52; ++c2) {
            if (L.ncombo >= limit) continue;
            const int cls = combo_class(c1, c2);
            L.cc[2 * L.ncombo] = (uint16_t)c1;
            L.cc[2 * L.ncombo + 1] = (uint16_t)c2;
            if (L.counts[cls] < CLS_CAP) L.lists[cls * CLS_CAP + L.counts[cls]++] = L.ncombo;
            ++L.ncombo;
        }
    return L;
}
__device__ const Lists g_lists_ref = make_lists(ALIVE), g_lists_ok = make_lists(1326);

}  // namespace pf
}  // namespace mtt

using namespace mtt;
using namespace mtt::pf;

extern "C" int mtt_pf_allin_matrix(int32_t mode, float* d_out, int32_t* d_wins, int32_t* d_ties, void* stream) {
    if (!d_out || (mode != MTT_PF_REFERENCE && mode != MTT_PF_CORRECT) || (!d_wins != !d_ties)) return MTT_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    if (mode == MTT_PF_REFERENCE)
        k_pf_allin<MTT_PF_REFERENCE><<<ceil_div(NC * NC * AI_SPLIT, AI_THREADS), AI_THREADS, 0, st>>>(d_out, d_wins, d_ties);
    else
        k_pf_allin<MTT_PF_CORRECT><<<ceil_div(NC * NC, AI_THREADS), AI_THREADS, 0, st>>>(d_out, d_wins, d_ties);
    MTT_CHECK_LAUNCH();
    return MTT_OK;
}

extern "C" int mtt_pf_flop_class_matrices(int32_t mode, const uint8_t* d_flops, int32_t n, float* d_out, void* stream) {
    if (!d_flops || !d_out || n < 0 || (mode != MTT_PF_REFERENCE && mode != MTT_PF_CORRECT)) return MTT_ERR_INVALID;
    if (n == 0) return MTT_OK;
    cudaStream_t st = as_stream(stream);
    const bool ref = mode == MTT_PF_REFERENCE;
    const int ncombo = ref ? ALIVE : 1326, ld = ref ? LD_REF : LD_OK;
    void* sym = nullptr;
    MTT_TRY_CUDA(ref ? cudaGetSymbolAddress(&sym, g_lists_ref) : cudaGetSymbolAddress(&sym, g_lists_ok));
    const Lists* L = static_cast<const Lists*>(sym);     // on the device
    // flops per pass: one CTA of k_pf_flop_eq per (villain tile, flop) and SM, as
    // many flops as fit three waves and the scratch that is kept between calls
    // (23 of the reference's 19 tiles, 223 MB), and fewer where the device has
    // not that much left
    const int tiles = ceil_div(ncombo, EQ_VILL);
    int dev = 0, sms = 0;
    MTT_TRY_CUDA(cudaGetDevice(&dev));
    MTT_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MTT_TRY_CUDA(cudaFuncSetAttribute(k_pf_flop_eq, cudaFuncAttributeMaxDynamicSharedMemorySize, EQ_SMEM));
    const size_t keys = (size_t)NPAIR * ld, runs = (size_t)ncombo * RUNS, eqs = (size_t)ld * ld;
    const int fit = (int)(SCRATCH_KEEP / (sizeof(uint16_t) * keys + sizeof(uint32_t) * runs + sizeof(float) * eqs));
    int chunk = std::max(1, std::min({n, 3 * sms / tiles, fit}));
    uint16_t* d_KT = nullptr;
    uint32_t* d_HL = nullptr;
    float* d_E = nullptr;
    auto drop = [st](auto*& p) {
        if (p) cudaFreeAsync(p, st);
        p = nullptr;
    };
    int s = MTT_OK;
    while (!s) {
        s = scratch_alloc(&d_KT, chunk * keys, st);
        if (!s) s = scratch_alloc(&d_HL, chunk * runs, st);
        if (!s) s = scratch_alloc(&d_E, chunk * eqs, st);
        if (s != MTT_ERR_NOMEM || chunk == 1) break;
        cudaGetLastError();                    // the refusal is dealt with here
        drop(d_KT); drop(d_HL); drop(d_E);
        chunk = (chunk + 1) / 2;
        s = MTT_OK;
    }
    for (int f0 = 0; f0 < n && !s; f0 += chunk) {
        const int nf = std::min(chunk, n - f0);
        const uint8_t* fl = d_flops + 3 * (size_t)f0;
        k_pf_keys<<<dim3(NPAIR, nf), 256, 0, st>>>(fl, L->cc, ncombo, ld, d_KT);
        k_pf_runs<<<dim3(ncombo, nf), RUNS, 0, st>>>(fl, L->cc, ncombo, ld, d_KT, d_HL);
        k_pf_flop_eq<<<dim3(tiles, nf), EQ_THREADS, EQ_SMEM, st>>>(fl, L->cc, ncombo, ld, mode, d_KT, d_HL, d_E);
        k_pf_reduce<<<dim3(NC, nf), PAD, 0, st>>>(d_E, ld, L->lists, L->counts, d_out + (size_t)f0 * NC * NC);
        s = cuda_status(cudaGetLastError());
    }
    drop(d_KT); drop(d_HL); drop(d_E);
    return s;
}

extern "C" int mtt_pf_combo_class(int32_t c1, int32_t c2) {
    if (c1 < 0 || c2 <= c1 || c2 > 51) return -1;
    return combo_class(c1, c2);
}

// ============================================================ preflop DCFR
namespace mtt {
namespace pf {

// Closed preflop tree state; blocks of [A][PAD] floats in node order BTN root
// (3), BB vs min-raise (3), BTN vs 3-bet jam (2), BB vs open jam (2).
__host__ __device__ constexpr int node_off(int k) { return k == 0 ? 0 : k == 1 ? 3 * PAD : k == 2 ? 6 * PAD : 8 * PAD; }
__host__ __device__ constexpr int node_actions(int k) { return k < 2 ? 3 : 2; }
constexpr int STATE = 10 * PAD;

struct PfDev {
    const float* fw;        // flop weights [nf]
    const float* mats;      // class matrices [nf][MAT] (v-major, rows of 169)
    const float* jam;       // all-in equity by step CTA: [tile][2][o][32 classes], as [o][cls] and transposed
    float *R, *G, *S;       // regrets, current strategy, strategy sums [STATE]
    float* Gn;              // the next strategy: every CTA of a step reads all classes of G
    float *root, *evb, *evbb;
    float *nb, *nbb;        // net flop EVs [nf][PAD]
    int nf;
    float stack, bf, dead;
};

constexpr int MAT = (NC * NC + 3) / 4 * 4;           // a class matrix padded to 16 bytes
constexpr int STEP_CLS = 32, STEP_WARPS = 7, STEP_THREADS = STEP_CLS * STEP_WARPS;
constexpr int STEP_TILES = (NC + STEP_CLS - 1) / STEP_CLS, STEP_JAM = 2 * NC * STEP_CLS;

// Copies of the matrices in the layouts that the iterations stage 16 bytes at
// a time: class matrices with padded stride, the all-in matrix in step tiles.
__global__ void __launch_bounds__(256) k_pf_layout(const float* __restrict__ mats, const float* __restrict__ allin, int nf,
                                                   float* __restrict__ om, float* __restrict__ oj) {
    const size_t total = (size_t)nf * MAT, stride = (size_t)gridDim.x * blockDim.x;
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i = i0; i < total; i += stride) {
        const int e = (int)(i % MAT);
        om[i] = e < NC * NC ? mats[i / MAT * (NC * NC) + e] : 0.0f;
    }
    for (size_t i = i0; i < (size_t)STEP_TILES * STEP_JAM; i += stride) {
        const int e = (int)(i % STEP_JAM), o = e / STEP_CLS % NC;
        const int col = min((int)(i / STEP_JAM) * STEP_CLS + e % STEP_CLS, NC - 1);
        oj[i] = e < NC * STEP_CLS ? allin[o * NC + col] : allin[col * NC + o];
    }
}

__global__ void k_pf_init(PfDev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < STATE) {
        d.R[i] = 0.0f;
        d.S[i] = 0.0f;
        d.G[i] = d.Gn[i] = i < 6 * PAD ? 1.0f / 3.0f : 0.5f;
    }
    if (i < PAD) {
        d.root[i] = i < NC ? (i < 13 ? 6.0f : i < 91 ? 4.0f : 12.0f) / 1326.0f : 0.0f;
        d.evb[i] = 0.0f;
        d.evbb[i] = 0.0f;
    }
}

// One DCFR iteration is two launches, chained by programmatic dependent
// launch: the reference's float sums run in a fixed order, so what can be
// spread is the independent sums, and what bounds each launch is one chain of
// 169 adds.  k_pf_cosolve: CTA per flop, thread per class and player;
// k_pf_step: warp per sum over 32 classes.  Both stage the matrices they read,
// which no iteration writes, in shared memory before they wait for the
// launch ahead, so those loads run under its tail: an iteration over 100 flops
// takes 11.5 us (most of it the two launches' hand-over), against 29 us with
// the loads left in the chains.  The five launches before (thread per flop
// over one class's strided column, all classes' sums in one CTA) took 80 us.

// Asynchronous copy of 4 bytes to shared memory; copies_done waits for this
// thread's copies, of 16 bytes too (a barrier must follow).
__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Net flop EVs of the reached classes (kernel_update_dynamic_reaches,
// :412-421, and the per-flop part of kernel_cosolve_100_board_matrices,
// :228-285).
constexpr int COSOLVE_SMEM = 4 * MAT;
__global__ void __launch_bounds__(2 * PAD) k_pf_cosolve(PfDev d) {
    extern __shared__ __align__(16) float eqm[];   // the flop's matrix: 169 is odd, so rows and columns are conflict-free
    __shared__ float rb[2][PAD];              // reach: BB's classes, BTN's classes
    __shared__ float rsum[2];
    const int f = blockIdx.x, tid = threadIdx.x;
    const int side = tid / PAD, cls = tid % PAD;   // side 0: BTN's EV, 1: BB's
    for (int i = tid; i < MAT / 4; i += 2 * PAD) copy_async16(eqm + 4 * i, d.mats + (size_t)f * MAT + 4 * i);
    grid_dep_wait();
    grid_dep_trigger();
    if (cls < NC)                             // side 0 sums over BB's reach, side 1 over BTN's
        rb[side][cls] = __fmul_rn(d.root[cls], d.G[node_off(1 - side) + PAD + cls]);
    copies_done();
    __syncthreads();
    float e = 0.0f;
    if (cls < NC) {
        const float* eq = eqm + (side ? cls * NC : cls);
        const float* r = rb[side];
        if (side) {
#pragma unroll 13
            for (int o = 0; o < NC; ++o) e = __fadd_rn(e, __fmul_rn(r[o], __fsub_rn(1.0f, eq[o])));
        } else {
#pragma unroll 13
            for (int o = 0; o < NC; ++o) e = __fadd_rn(e, __fmul_rn(r[o], eq[o * NC]));
        }
    } else if (cls == PAD - 1) {              // an idle thread of each side adds the reach up
        float sum = 0.0f;
#pragma unroll 13
        for (int o = 0; o < NC; ++o) sum = __fadd_rn(sum, rb[side][o]);
        rsum[side] = sum;
    }
    __syncthreads();
    if (cls >= NC) return;
    const float pot_flop = __fadd_rn(d.dead, 3.1f);
    if (rsum[side] > 1e-7f) e = __fdiv_rn(e, rsum[side]);
    const float sh = __fmul_rn(__fmul_rn(e, side ? 0.94f : 1.06f), pot_flop);
    (side ? d.nbb : d.nb)[(size_t)f * PAD + cls] =
        sh >= 2.1f ? __fsub_rn(sh, 2.1f) : -__fmul_rn(__fsub_rn(2.1f, sh), d.bf);
}

// The weighted flop average (:270-285), the action values of the four nodes
// (kernel_build_closed_preflop_cfvs, :290-385) and their regret and strategy
// update (kernel_dcfr_step, :387-410) for 32 classes per CTA.  The masses
// behind the action values are the same for every class: one warp forms the
// nine of them, a lane each.  Four warps form one equity sum each over their
// 32 classes and two the flop averages; then warp k updates node k.
constexpr int STEP_FLOPS = 128;           // flops staged at a time
constexpr int STEP_SMEM = 4 * (STEP_JAM + STEP_FLOPS * (2 * STEP_CLS + 1));
enum { M_M3, M_BF3, M_BC3, M_MJ, M_CJ, M_FM, M_CM, M_JM, M_FJ, N_MASS };   // mass order; the first of each equity sum's too
__global__ void __launch_bounds__(STEP_THREADS) k_pf_step(PfDev d, float wp, float ws) {
    extern __shared__ __align__(16) float step_smem[];
    __shared__ __align__(16) float G[STATE];                 // filled 16 bytes at a time
    __shared__ __align__(16) float root[PAD];
    __shared__ float reach[N_MASS][PAD];                     // summands of the masses
    __shared__ float mass[N_MASS];
    __shared__ float sums[6][STEP_CLS];                      // equity sums of warps 0..3, flop sums of warps 4, 5
    __shared__ float wsum;                                   // flop weights
    float* const Ac = step_smem;                             // all-in equity [o][cls] of this CTA's classes
    float* const Ar = Ac + NC * STEP_CLS;                    // [o][cls] of the transpose
    float* const nbs = Ar + NC * STEP_CLS;                   // net flop EVs [player][flop][cls]
    float* const fws = nbs + STEP_FLOPS * 2 * STEP_CLS;      // flop weights
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cls = blockIdx.x * STEP_CLS + lane;
    const int col = min(cls, NC - 1);
    for (int i = tid; i < STEP_JAM / 4; i += STEP_THREADS)
        copy_async16(step_smem + 4 * i, d.jam + (size_t)blockIdx.x * STEP_JAM + 4 * i);
    auto stage_flops = [&](int f0) {                         // flops [f0, f0 + STEP_FLOPS)
        const int n = min(STEP_FLOPS, d.nf - f0);
        for (int k = warp; k < n; k += STEP_WARPS) {
            copy4(nbs + k * STEP_CLS + lane, d.nb + (size_t)(f0 + k) * PAD + col);
            copy4(nbs + (STEP_FLOPS + k) * STEP_CLS + lane, d.nbb + (size_t)(f0 + k) * PAD + col);
        }
        for (int k = tid; k < n; k += STEP_THREADS) copy4(fws + k, d.fw + f0 + k);
    };
    grid_dep_wait();
    grid_dep_trigger();
    for (int i = tid; i < STATE / 4; i += STEP_THREADS) copy_async16(G + 4 * i, d.G + 4 * i);
    for (int i = tid; i < PAD / 4; i += STEP_THREADS) copy_async16(root + 4 * i, d.root + 4 * i);
    stage_flops(0);
    float Rc[3] = {0.0f, 0.0f, 0.0f}, Sc[3] = {0.0f, 0.0f, 0.0f};   // the updated node's rows of this class
    if (warp < 4 && cls < NC)
        for (int a = 0; a < node_actions(warp); ++a) {
            Rc[a] = d.R[node_off(warp) + a * PAD + cls];
            Sc[a] = d.S[node_off(warp) + a * PAD + cls];
        }
    copies_done();
    __syncthreads();
    const float *sbr = G + node_off(0), *sbd = G + node_off(1), *s3b = G + node_off(2), *sbj = G + node_off(3);
    for (int o = tid; o < NC; o += STEP_THREADS) {
        const float r = root[o], ro = __fmul_rn(r, sbr[PAD + o]);
        reach[M_M3][o] = __fmul_rn(r, sbd[2 * PAD + o]);
        reach[M_BF3][o] = __fmul_rn(ro, s3b[o]);
        reach[M_BC3][o] = __fmul_rn(ro, s3b[PAD + o]);
        reach[M_MJ][o] = __fmul_rn(r, sbr[2 * PAD + o]);
        reach[M_CJ][o] = __fmul_rn(r, sbj[PAD + o]);
        reach[M_FM][o] = __fmul_rn(r, sbd[o]);
        reach[M_CM][o] = __fmul_rn(r, sbd[PAD + o]);
        reach[M_JM][o] = reach[M_M3][o];
        reach[M_FJ][o] = __fmul_rn(r, sbj[o]);
    }
    __syncthreads();
    // equity sums: warp 0 BTN vs 3-bet jam (eqc), 1 BB's jam over the min-raise (eqj), 2 BB vs open jam (eqo),
    // 3 BTN's open jam (eo)
    if (warp < 4) {
        const float* r = reach[warp == 0 ? M_M3 : warp == 1 ? M_BC3 : warp == 2 ? M_MJ : M_CJ];
        float y = 0.0f;
        if (warp == 0 || warp == 3) {
            const float* A = Ar + lane;
#pragma unroll 13
            for (int o = 0; o < NC; ++o) y = __fadd_rn(y, __fmul_rn(r[o], A[o * STEP_CLS]));
        } else {
            const float* A = Ac + lane;
#pragma unroll 13
            for (int o = 0; o < NC; ++o) y = __fadd_rn(y, __fmul_rn(r[o], __fsub_rn(1.0f, A[o * STEP_CLS])));
        }
        sums[warp][lane] = y;
    } else if (warp == 6 && lane < N_MASS) {
        float x = 0.0f;
#pragma unroll 13
        for (int o = 0; o < NC; ++o) x = __fadd_rn(x, reach[lane][o]);
        mass[lane] = x;
    }
    float tw = 0.0f, fe = 0.0f;
    for (int f0 = 0; f0 < d.nf; f0 += STEP_FLOPS) {          // flop sums, in flop order: BTN (4) and BB (5)
        if (f0) {                                            // further flops of a large subset
            __syncthreads();
            stage_flops(f0);
            copies_done();
            __syncthreads();
        }
        if (warp != 4 && warp != 5) continue;
        const float* n = nbs + (warp == 4 ? 0 : STEP_FLOPS * STEP_CLS) + lane;
        const int nf = min(STEP_FLOPS, d.nf - f0);
#pragma unroll 4
        for (int f = 0; f < nf; ++f) {
            const float w = fws[f];
            tw = __fadd_rn(tw, w);
            fe = __fadd_rn(fe, __fmul_rn(w, n[f * STEP_CLS]));
        }
    }
    if (warp == 4 || warp == 5) {
        sums[warp][lane] = fe;
        if (warp == 4 && lane == 0) wsum = tw;
    }
    __syncthreads();
    if (warp >= 4 || cls >= NC) return;
    const float stack = d.stack, bf = d.bf, dead = d.dead;
    const float jam_pot = __fadd_rn(__fmul_rn(2.0f, stack), dead);
    const float jam_net = __fsub_rn(jam_pot, stack);
    // eq * (jam_pot - stack) - (1 - eq) * bf * stack, evaluated left to right
    auto jam_value = [&](float eq) {
        return __fsub_rn(__fmul_rn(eq, jam_net), __fmul_rn(__fmul_rn(__fsub_rn(1.0f, eq), bf), stack));
    };
    auto share = [&](int k, int m) {   // equity sum k over its mass
        return mass[m] > 1e-7f ? __fdiv_rn(sums[k][lane], mass[m]) : sums[k][lane];
    };
    // the flop EV of player k, kept from before when no flop has weight
    auto flop_ev = [&](int k, float* ev) {
        const float v = wsum > 0.0f ? __fdiv_rn(sums[4 + k][lane], wsum) : ev[cls];
        if (wsum > 0.0f) ev[cls] = v;
        return v;
    };
    float C[3];
    if (warp == 0) {            // BTN root
        const float c30 = __fmul_rn(-2.1f, bf), c31 = jam_value(share(0, M_M3));
        const float v3 = __fadd_rn(__fmul_rn(s3b[cls], c30), __fmul_rn(s3b[PAD + cls], c31));
        const float tb = __fadd_rn(__fadd_rn(__fadd_rn(mass[M_FM], mass[M_CM]), mass[M_JM]), 1e-9f);
        const float toj = __fadd_rn(__fadd_rn(mass[M_FJ], mass[M_CJ]), 1e-9f);
        const float evj = jam_value(share(3, M_CJ));
        C[0] = 0.0f;
        C[1] = __fdiv_rn(__fadd_rn(__fadd_rn(__fmul_rn(mass[M_FM], dead), __fmul_rn(mass[M_CM], flop_ev(0, d.evb))),
                                   __fmul_rn(mass[M_JM], v3)), tb);
        C[2] = __fdiv_rn(__fadd_rn(__fmul_rn(mass[M_FJ], dead), __fmul_rn(mass[M_CJ], evj)), toj);
    } else if (warp == 1) {     // BB vs min-raise
        const float tot3 = __fadd_rn(__fadd_rn(mass[M_BF3], mass[M_BC3]), 1e-9f);
        const float evsh = jam_value(share(1, M_BC3));
        C[0] = __fmul_rn(-1.0f, bf);
        C[1] = flop_ev(1, d.evbb);
        C[2] = __fdiv_rn(__fadd_rn(__fmul_rn(mass[M_BF3], __fadd_rn(dead, 2.1f)), __fmul_rn(mass[M_BC3], evsh)), tot3);
    } else if (warp == 2) {     // BTN vs 3-bet jam
        C[0] = __fmul_rn(-2.1f, bf);
        C[1] = jam_value(share(0, M_M3));
        C[2] = 0.0f;
    } else {                    // BB vs open jam
        C[0] = __fmul_rn(-1.0f, bf);
        C[1] = jam_value(share(2, M_MJ));
        C[2] = 0.0f;
    }
    const int A = node_actions(warp), off = node_off(warp);
    const float* g = G + off;
    float v = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) if (a < A) v = __fadd_rn(v, __fmul_rn(g[a * PAD + cls], C[a]));
    float pos = 0.0f, nxt[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (a >= A) continue;
        const int i = off + a * PAD + cls;
        const float nr = __fmul_rn(wp, fmaxf(0.0f, __fadd_rn(Rc[a], __fsub_rn(C[a], v))));
        d.R[i] = nr;
        pos = __fadd_rn(pos, nr);
        nxt[a] = nr;
        d.S[i] = __fadd_rn(Sc[a], __fmul_rn(__fmul_rn(ws, root[cls]), g[a * PAD + cls]));
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (a < A) d.Gn[off + a * PAD + cls] = pos > 1e-7f ? __fdiv_rn(nxt[a], pos) : __fdiv_rn(1.0f, (float)A);
}

}  // namespace pf
}  // namespace mtt

extern "C" int mtt_pf_dcfr(const float* d_flop_weights, const float* d_class_mats, int32_t n_flops,
                           const float* d_allin, const mtt_pf_params* p, float* d_sums, float* d_sigma, void* stream) {
    if (!d_flop_weights || !d_class_mats || n_flops < 1 || !d_allin || !p || p->iters < 0 || !d_sums)
        return MTT_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    float* buf = nullptr;
    const size_t nf = (size_t)n_flops;
    MTT_TRY_CUDA(cudaFuncSetAttribute(k_pf_cosolve, cudaFuncAttributeMaxDynamicSharedMemorySize, COSOLVE_SMEM));
    MTT_TRY_CUDA(cudaFuncSetAttribute(k_pf_step, cudaFuncAttributeMaxDynamicSharedMemorySize, STEP_SMEM));
    MTT_TRY(scratch_alloc(&buf, 4 * (size_t)STATE + 3 * (size_t)PAD + 2 * nf * PAD + nf * MAT + (size_t)STEP_TILES * STEP_JAM,
                          st));
    PfDev d{};
    d.fw = d_flop_weights;
    d.R = buf; d.G = d.R + STATE; d.Gn = d.G + STATE; d.S = d.Gn + STATE;
    d.root = d.S + STATE; d.evb = d.root + PAD; d.evbb = d.evb + PAD;
    d.nb = d.evbb + PAD; d.nbb = d.nb + nf * PAD;
    float* const om = d.nbb + nf * PAD;       // every part before it is a multiple of 64 floats
    float* const oj = om + nf * MAT;
    d.mats = om; d.jam = oj;
    d.nf = n_flops; d.stack = p->stack_bb; d.bf = p->bubble; d.dead = p->dead_pot;
    k_pf_init<<<ceil_div(STATE, 256), 256, 0, st>>>(d);
    k_pf_layout<<<592, 256, 0, st>>>(d_class_mats, d_allin, n_flops, om, oj);
    int s = cuda_status(cudaGetLastError());
    for (int t = 1; t <= p->iters && !s; ++t) {
        const float tf = (float)t;   // host powf, as the reference's loop (:589-591)
        const float wp = powf(tf, 1.5f) / (powf(tf, 1.5f) + 1.0f), ws = tf * tf;
        s = cuda_status(launch_pdl(k_pf_cosolve, (unsigned)n_flops, 2 * PAD, COSOLVE_SMEM, st, t > 1, d));
        if (!s) s = cuda_status(launch_pdl(k_pf_step, (unsigned)STEP_TILES, STEP_THREADS, STEP_SMEM, st, true, d, wp, ws));
        std::swap(d.G, d.Gn);
    }
    if (!s) s = cuda_status(cudaMemcpyAsync(d_sums, d.S, sizeof(float) * STATE, cudaMemcpyDeviceToDevice, st));
    if (!s && d_sigma) s = cuda_status(cudaMemcpyAsync(d_sigma, d.G, sizeof(float) * STATE, cudaMemcpyDeviceToDevice, st));
    cudaFreeAsync(buf, st);
    // the call returns with its results in place (a caller on another stream
    // reads them, and frees its inputs, at once), unless it is only recorded
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!s && p->iters > 0) s = cuda_status(cudaStreamIsCapturing(st, &cap));
    if (!s && p->iters > 0 && cap == cudaStreamCaptureStatusNone) s = cuda_status(cudaStreamSynchronize(st));
    return s;
}

extern "C" int mtt_pf_read_subset(const char* path, uint8_t* h_flops, float* h_weights, int32_t capacity, int32_t* n) {
    if (!n) return MTT_ERR_INVALID;
    const char* tries[2] = {path ? path : "data/mtt_subset.bin", path ? nullptr : "mtt_subset.bin"};
    FILE* fp = nullptr;
    for (const char* t : tries)
        if (t && (fp = fopen(t, "rb"))) break;
    if (!fp) return MTT_ERR_IO;
    uint32_t count = 0;
    int s = fread(&count, 4, 1, fp) == 1 ? MTT_OK : MTT_ERR_IO;
    if (!s && count > 100000u) s = MTT_ERR_IO;
    if (!s) *n = (int32_t)count;
    for (uint32_t i = 0; i < count && !s && h_flops; ++i) {
        uint8_t rec[8];
        if (fread(rec, 1, 8, fp) != 8) { s = MTT_ERR_IO; break; }
        if ((int32_t)i >= capacity) { s = MTT_ERR_INVALID; break; }
        h_flops[3 * i] = rec[0]; h_flops[3 * i + 1] = rec[1]; h_flops[3 * i + 2] = rec[2];
        if (rec[0] > 51 || rec[1] > 51 || rec[2] > 51) { s = MTT_ERR_IO; break; }
        if (h_weights) std::memcpy(&h_weights[i], rec + 4, 4);
    }
    fclose(fp);
    return s;
}
