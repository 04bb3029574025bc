// eval.cu — hand evaluation, board showdown counts and the flop-EV dumper chain.
//
//  * mtt_eval7: 7 bytes per hand in, uint32 reference score out.  Four hands
//    (seven words) a thread; the few flushes are scored in a second pass.
//  * mtt_eval7_enumerate: all C(52,7) hands, category histogram + checksum.
//  * mtt_board_showdown_counts: exact win/tie/loss counts per (hero,
//    villain) pair over every completion of a 3/4/5-card board
//    (kernel_gen_49_turn_matrices, honest_multistreet_solver.cu:56-86, as
//    integer counts).  Each (completion, hand) is evaluated ONCE into a
//    16-bit key; pairs are then counted two completions per 32-bit word with
//    one packed add-and-clamp per count on shared-memory tiles.
//  * mtt_flop_ev / mtt_ev_dump: the reference dumper (mtt_ev_dumper.cu:85-168)
//    with the same subsampled runouts, villain stride, ½ tie weight, FMA
//    accumulation order and host aggregation, reproduced bit-exactly.
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "mtt_common.h"
#include "mtt_device.cuh"
#include "mtt_pairs.cuh"

namespace mtt {

// ============================================================ mtt_eval7
constexpr int EV_THREADS = 256;
constexpr long long EV_QUAD_MIN = 4096;      // below this, a thread per hand: the shorter chain wins (1.9 us)

// Four hands a thread, read as seven aligned words.  Bound by the integer pipe
// (ALU 91% busy, 162 issue slots a hand): the suits are only counted (a byte each, in one word), so a
// hand costs its rank planes, the count and the scores without a flush; one
// hand in 33 holds a flush, and those are read again and scored after all
// four, when most warps have one pass of them left instead of up to four.
// 30,000,001 hands took 275 us with every suit's mask kept, tested by four
// popcounts, and staged by bulk copies whose error word the call then read
// back; 217 us now, and the call no longer waits.
template <bool VEC>
__global__ void __launch_bounds__(EV_THREADS)
k_eval7_quad(const uint8_t* __restrict__ cards, uint32_t* __restrict__ out, long long n) {
    const long long q = (long long)blockIdx.x * EV_THREADS + threadIdx.x, h0 = 4 * q;
    if (h0 >= n) return;
    if (h0 + 4 > n) {                              // the last hands, fewer than four
        for (long long h = h0; h < n; ++h) out[h] = score7(cards + 7 * h);
        return;
    }
    const uint32_t* w = reinterpret_cast<const uint32_t*>(cards) + 7 * q;
    uint32_t word[7], suit[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        word[k] = __ldg(w + k);
        suit[k] = (word[k] & 0x03030303u) << 3;    // 8 x suit in every byte
    }
    uint32_t s[4], flush = 0u;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        uint32_t one = 0u, two = 0u, three = 0u, four = 0u, cnt = 0u;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int byte = 7 * h + k, sh = 8 * (byte & 3);
            // shifts by the low five bits: the rank (bit 6 of a card is 0), and 8 x suit
            const uint32_t b = __funnelshift_l(0u, 1u, word[byte >> 2] >> (sh + 2));
            four |= three & b; three |= two & b; two |= one & b; one |= b;
            cnt += __funnelshift_l(0u, 1u, suit[byte >> 2] >> sh);
        }
        flush |= ((cnt + 0x7B7B7B7Bu) & 0x80808080u ? 1u : 0u) << h;
        s[h] = score_ranks(one, two, three, four);
    }
    while (flush) {
        const int h = __ffs((int)flush) - 1;
        flush &= flush - 1u;
        const uint32_t v = score7(cards + 7 * (h0 + h));
#pragma unroll
        for (int k = 0; k < 4; ++k) if (k == h) s[k] = v;
    }
    if (VEC) {
        *reinterpret_cast<uint4*>(out + h0) = make_uint4(s[0], s[1], s[2], s[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) out[h0 + k] = s[k];
    }
}

__global__ void k_eval7_plain(const uint8_t* __restrict__ cards, uint32_t* __restrict__ out,
                              long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = score7(cards + 7 * i);
}

static int sm_count(int* out) {
    int dev = 0;
    MTT_TRY_CUDA(cudaGetDevice(&dev));
    MTT_TRY_CUDA(cudaDeviceGetAttribute(out, cudaDevAttrMultiProcessorCount, dev));
    return MTT_OK;
}

// ============================================================ enumeration
constexpr int ENUM_CHUNK = 64;
constexpr long long N_HANDS7 = 133784560LL;

__device__ __forceinline__ unsigned long long binom_dev(int n, int k) {
    if (k < 0 || n < k) return 0ull;
    unsigned long long b = 1ull;
    for (int i = 0; i < k; ++i) b = b * (unsigned long long)(n - i) / (unsigned long long)(i + 1);
    return b;
}

// colex unranking: idx -> c0 < c1 < ... < c6
__device__ __forceinline__ void unrank7(unsigned long long idx, int c[7]) {
    int top = 52;
    for (int i = 7; i >= 1; --i) {
        int cc = top - 1;
        unsigned long long b = binom_dev(cc, i);
        while (b > idx) { b = b * (unsigned long long)(cc - i) / (unsigned long long)cc; --cc; }
        c[i - 1] = cc;
        idx -= b;
        top = cc;
    }
}

__global__ void __launch_bounds__(256)
k_enumerate7(unsigned long long* __restrict__ hist, unsigned long long* __restrict__ checksum,
             uint32_t* __restrict__ key_table, int* __restrict__ err) {
    __shared__ unsigned long long s_hist[9];
    if (threadIdx.x < 9) s_hist[threadIdx.x] = 0ull;
    __syncthreads();
    const long long n_chunks = (N_HANDS7 + ENUM_CHUNK - 1) / ENUM_CHUNK;
    unsigned int cnt[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) cnt[k] = 0u;
    unsigned long long cs = 0ull;
    for (long long ch = (long long)blockIdx.x * blockDim.x + threadIdx.x; ch < n_chunks;
         ch += (long long)gridDim.x * blockDim.x) {
        unsigned long long idx = (unsigned long long)ch * ENUM_CHUNK;
        int c[7];
        unrank7(idx, c);
        int c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3], c4 = c[4], c5 = c[5], c6 = c[6];
        const unsigned long long end = min((unsigned long long)N_HANDS7, idx + ENUM_CHUNK);
        for (; idx < end; ++idx) {
            const int hand[7] = {c0, c1, c2, c3, c4, c5, c6};
            const uint32_t s = score7(hand);
            const uint32_t cat = s >> 24;
#pragma unroll
            for (int k = 0; k < 9; ++k) cnt[k] += (cat == (uint32_t)k) ? 1u : 0u;
            cs += (unsigned long long)s * (idx + 1ull);
            if (key_table) {
                Planes p; planes_clear(p);
#pragma unroll
                for (int k = 0; k < 7; ++k) planes_add(p, hand[k]);
                const uint32_t key = key_planes(p);
                if (key_table[key] != s) {
                    const uint32_t old = atomicCAS(&key_table[key], 0xFFFFFFFFu, s);
                    if (old != 0xFFFFFFFFu && old != s) atomicOr(err, 2);
                }
            }
            // colex successor
            if (c0 + 1 < c1) { ++c0; }
            else if (c1 + 1 < c2) { ++c1; c0 = 0; }
            else if (c2 + 1 < c3) { ++c2; c0 = 0; c1 = 1; }
            else if (c3 + 1 < c4) { ++c3; c0 = 0; c1 = 1; c2 = 2; }
            else if (c4 + 1 < c5) { ++c4; c0 = 0; c1 = 1; c2 = 2; c3 = 3; }
            else if (c5 + 1 < c6) { ++c5; c0 = 0; c1 = 1; c2 = 2; c3 = 3; c4 = 4; }
            else { ++c6; c0 = 0; c1 = 1; c2 = 2; c3 = 3; c4 = 4; c5 = 5; }
        }
    }
    // warp reduce then shared then global
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        unsigned int v = cnt[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_hist[k], (unsigned long long)v);
    }
    for (int o = 16; o > 0; o >>= 1) cs += __shfl_down_sync(0xFFFFFFFFu, cs, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(checksum, cs);
    __syncthreads();
    if (threadIdx.x < 9 && s_hist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], s_hist[threadIdx.x]);
}

// ============================================================ board counts
// keys[w][h] packs the hero halves of completions 2w (low) and 2w+1 (high)
// for hand h.
__device__ __forceinline__ void pair_unrank(int k, int n, int& a, int& b) {
    // lexicographic (a<b) over n items
    a = 0;
    int row = n - 1;
    while (k >= row) { k -= row; ++a; --row; }
    b = a + 1 + k;
}

__global__ void k_completion_keys(const uint8_t* __restrict__ board, int nboard,
                                  const uint8_t* __restrict__ hands, int H, int Hp, int ncomp,
                                  uint32_t* __restrict__ keys) {
    __shared__ uint8_t rest[52];
    __shared__ int nrest;
    if (threadIdx.x == 0) {
        uint64_t bm = 0;
        for (int k = 0; k < nboard; ++k) bm |= 1ull << board[k];
        int n = 0;
        for (int c = 0; c < 52; ++c) if (!((bm >> c) & 1ull)) rest[n++] = (uint8_t)c;
        nrest = n;
    }
    __syncthreads();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    const int w = blockIdx.y;
    if (h >= Hp) return;
    uint32_t word = KEY_H_DEAD | (KEY_H_DEAD << 16);
    if (h < H) {
        const int hc1 = hands[2 * h], hc2 = hands[2 * h + 1];
        uint64_t bm = 0;
        for (int k = 0; k < nboard; ++k) bm |= 1ull << board[k];
        const uint64_t hm = (1ull << hc1) | (1ull << hc2);
        if (!(hm & bm) && hc1 != hc2) {
            Planes base; planes_clear(base);
            for (int k = 0; k < nboard; ++k) planes_add(base, board[k]);
            planes_add(base, hc1); planes_add(base, hc2);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int k = 2 * w + half;
                if (k >= ncomp) continue;
                Planes p = base;
                uint64_t cm = 0;
                if (nboard == 4) {
                    const int c = rest[k];
                    cm = 1ull << c;
                    planes_add(p, c);
                } else if (nboard == 3) {
                    int a, b;
                    pair_unrank(k, nrest, a, b);
                    cm = (1ull << rest[a]) | (1ull << rest[b]);
                    planes_add(p, rest[a]); planes_add(p, rest[b]);
                }
                if (cm & hm) continue;
                word ^= (KEY_H_DEAD ^ (key_planes(p) + 1u)) << (16 * half);
            }
        }
    }
    keys[(size_t)w * Hp + h] = word;
}

constexpr int BC_TILE = 64, BC_WCHUNK = 32;

// Bound by the packed clamps (4 instructions a word of two completions) and,
// for few completions, by the three H x H outputs.  Accumulator halves hold at
// most 2 * 588 (flop boards: 1,176 completions), so plain 32-bit adds do not
// carry across.
__global__ void __launch_bounds__(256)
k_board_counts(const uint32_t* __restrict__ keys, int ncw, int H, int Hp,
               const uint8_t* __restrict__ hands, const uint8_t* __restrict__ board, int nboard,
               int n_const, int32_t* __restrict__ W, int32_t* __restrict__ T, int32_t* __restrict__ L, uint32_t one) {
    __shared__ alignas(16) uint32_t hk[BC_WCHUNK][BC_TILE];
    __shared__ alignas(16) uint32_t vk[BC_WCHUNK][BC_TILE];
    const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
    const int i0 = blockIdx.x * BC_TILE, j0 = blockIdx.y * BC_TILE;
    uint32_t wc[4][4], sc[4][4];   // 2 wins; 2 wins + ties
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) { wc[a][b] = 0u; sc[a][b] = 0u; }
    for (int w0 = 0; w0 < ncw; w0 += BC_WCHUNK) {
        const int nw = min(BC_WCHUNK, ncw - w0);
        for (int e = tid; e < nw * BC_TILE; e += 256) {
            const int w = e / BC_TILE, x = e % BC_TILE;   // Hp is a multiple of the tile
            hk[w][x] = keys[(size_t)(w0 + w) * Hp + i0 + x];
            vk[w][x] = villain_word(keys[(size_t)(w0 + w) * Hp + j0 + x]);
        }
        __syncthreads();
#pragma unroll 4
        for (int w = 0; w < nw; ++w) {
            const uint4 h4 = *reinterpret_cast<const uint4*>(&hk[w][tj * 4]);
            const uint4 v4 = *reinterpret_cast<const uint4*>(&vk[w][ti * 4]);
            const uint32_t hv[4] = {h4.x, h4.y, h4.z, h4.w};
            const uint32_t vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t t = pair_2w_t(hv[a], vv[b]);
                    sc[a][b] = add_on_fma(sc[a][b], t, one);
                    wc[a][b] = add_on_fma(wc[a][b], t & 0x00020002u, one);
                }
        }
        __syncthreads();
    }
    // a thread's villains are 4 consecutive columns, so with H a multiple of 4
    // each output row part is one 16-byte store
    uint64_t bm = 0;
    for (int k = 0; k < nboard; ++k) bm |= 1ull << board[k];
    const int j0t = j0 + ti * 4;
    uint64_t mj[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int j = min(j0t + b, H - 1);
        mj[b] = (1ull << hands[2 * j]) | (1ull << hands[2 * j + 1]);
    }
    const bool vec = (H & 3) == 0 && j0t + 3 < H &&
                     ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(T) | reinterpret_cast<uintptr_t>(L)) & 15u) == 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int i = i0 + tj * 4 + a;
        if (i >= H) continue;
        const uint64_t mi = (1ull << hands[2 * i]) | (1ull << hands[2 * i + 1]);
        int32_t wv[4], tv[4], lv[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const bool ok = !(mi & mj[b]) && !(mi & bm) && !(mj[b] & bm);
            wv[b] = ok ? (int32_t)((wc[a][b] & 0xFFFFu) + (wc[a][b] >> 16)) / 2 : 0;
            tv[b] = ok ? (int32_t)((sc[a][b] & 0xFFFFu) + (sc[a][b] >> 16)) - 2 * wv[b] : 0;
            lv[b] = ok ? n_const - wv[b] - tv[b] : 0;
        }
        const size_t o = (size_t)i * H + j0t;
        if (vec) {
            *reinterpret_cast<int4*>(W + o) = make_int4(wv[0], wv[1], wv[2], wv[3]);
            *reinterpret_cast<int4*>(T + o) = make_int4(tv[0], tv[1], tv[2], tv[3]);
            *reinterpret_cast<int4*>(L + o) = make_int4(lv[0], lv[1], lv[2], lv[3]);
        } else {
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (j0t + b < H) { W[o + b] = wv[b]; T[o + b] = tv[b]; L[o + b] = lv[b]; }
        }
    }
}

// ============================================================ flop EV chain
// Runout subsample of the reference loop (mtt_ev_dumper.cu:98-103): turn
// index r1 = 0,2,..,46 into the 49-card deck, river index r2 = r1+1, r1+4,
// .. < 47.  192 (r1, r2) pairs, packed two per key word.
constexpr int FE_RUNOUTS = 192, FE_WORDS = 96, FE_ALIVE = 1176, FE_VILL = 294;
struct Runouts { uint8_t r1[FE_RUNOUTS], r2[FE_RUNOUTS]; };
constexpr Runouts make_runouts() {
    Runouts t{};
    int k = 0;
    for (int r1 = 0; r1 < 47; r1 += 2)
        for (int r2 = r1 + 1; r2 < 47; r2 += 3) { t.r1[k] = (uint8_t)r1; t.r2[k] = (uint8_t)r2; ++k; }
    return t;
}
// Part of the module: copied in by each call, a captured call's replay read the
// copy's source when it was gone, and indexed the deck with what was there.
__constant__ Runouts c_runouts = make_runouts();

__device__ __forceinline__ void flop_deck(const uint8_t* f, uint8_t* deck) {
    const uint64_t fm = (1ull << f[0]) | (1ull << f[1]) | (1ull << f[2]);
    int n = 0;
    for (int c = 0; c < 52; ++c) if (!((fm >> c) & 1ull)) deck[n++] = (uint8_t)c;
}

// keys[f][w][i] (hand-minor): hero halves of runouts 2w and 2w + 1 for hand i
__global__ void __launch_bounds__(128)
k_flop_keys(const uint8_t* __restrict__ flops, uint32_t* __restrict__ keys) {
    __shared__ uint8_t deck[52];
    const int f = blockIdx.y;
    const uint8_t* fl = flops + 3 * f;
    if (threadIdx.x == 0) flop_deck(fl, deck);
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= FE_ALIVE) return;
    int a, b;
    pair_unrank(i, 49, a, b);
    const int hc1 = deck[a], hc2 = deck[b];
    Planes base; planes_clear(base);
    planes_add(base, fl[0]); planes_add(base, fl[1]); planes_add(base, fl[2]);
    planes_add(base, hc1); planes_add(base, hc2);
    uint32_t* kout = keys + (size_t)f * FE_WORDS * FE_ALIVE + i;
    for (int w = 0; w < FE_WORDS; ++w) {
        uint32_t word = KEY_H_DEAD | (KEY_H_DEAD << 16);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = 2 * w + half;
            const int t = deck[c_runouts.r1[k]], r = deck[c_runouts.r2[k]];
            if (t == hc1 || t == hc2 || r == hc1 || r == hc2) continue;
            Planes p = base;
            planes_add(p, t); planes_add(p, r);
            word ^= (KEY_H_DEAD ^ (key_planes(p) + 1u)) << (16 * half);
        }
        kout[(size_t)w * FE_ALIVE] = word;
    }
}

// eqT[f][m][i]: equity of hero i vs villain j = 4m over the usable runouts
// ((2W+T)/(2N) as in mtt_ev_dumper.cu:105-110), -1 when the pair is skipped.
// The numerator is the sum of one packed clamp per word; N is counted from the
// hands' deck positions by inclusion and exclusion over the runout pairs (192
// less the runouts that hold a card of either hand), so the loop spends
// nothing on it.  Bound by the clamps: all 1,755 flops took 48.8 ms with
// half-word compares and a popcount of usable runouts per pair, 8.1 ms now.
constexpr int FE_TH = 64, FE_TV = 64, FE_WCH = 32;
__global__ void __launch_bounds__(256)
k_flop_pair_eq(const uint32_t* __restrict__ keys, float* __restrict__ eqT, uint32_t one) {
    __shared__ alignas(16) uint32_t hk[FE_WCH][FE_TH];
    __shared__ alignas(16) uint32_t vk[FE_WCH][FE_TV];
    __shared__ uint64_t adj[49];             // bit y of adj[x]: deck positions x and y are a runout
    __shared__ uint8_t pos[2][FE_TH][2];     // deck positions of the tile's heroes and villains
    __shared__ uint8_t usable[2][FE_TH];     // runouts that avoid each hand's two cards
    const int f = blockIdx.z;
    const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
    const int i0 = blockIdx.x * FE_TH, m0 = blockIdx.y * FE_TV;
    if (tid < 49) {
        uint64_t m = 0;
        for (int y = 0; y < 49; ++y) {
            const int lo = min(tid, y), hi = max(tid, y);
            if (lo != hi && !(lo & 1) && hi < 47 && (hi - lo - 1) % 3 == 0) m |= 1ull << y;
        }
        adj[tid] = m;
    }
    __syncthreads();
    if (tid < 2 * FE_TH) {
        const int side = tid / FE_TH, x = tid % FE_TH;
        const int hand = side ? min(4 * (m0 + x), FE_ALIVE - 1) : min(i0 + x, FE_ALIVE - 1);
        int a, b;
        pair_unrank(hand, 49, a, b);
        pos[side][x][0] = (uint8_t)a;
        pos[side][x][1] = (uint8_t)b;
        usable[side][x] = (uint8_t)(FE_RUNOUTS - __popcll(adj[a]) - __popcll(adj[b]) + (int)((adj[a] >> b) & 1ull));
    }
    const uint32_t* kf = keys + (size_t)f * FE_WORDS * FE_ALIVE;
    uint32_t sc[4][4];   // 2 wins + ties of each half, at most 2 * 96
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) sc[a][b] = 0u;
    for (int w0 = 0; w0 < FE_WORDS; w0 += FE_WCH) {
        for (int e = tid; e < FE_WCH * FE_TH; e += 256) {
            const int w = e / FE_TH, x = e % FE_TH;
            const int i = min(i0 + x, FE_ALIVE - 1), m = min(m0 + x, FE_VILL - 1);
            hk[w][x] = kf[(size_t)(w0 + w) * FE_ALIVE + i];
            vk[w][x] = villain_word(kf[(size_t)(w0 + w) * FE_ALIVE + 4 * m]);
        }
        __syncthreads();
#pragma unroll 4
        for (int w = 0; w < FE_WCH; w += 2) {   // two words a step: their adds fuse into one
            const uint4 h4 = *reinterpret_cast<const uint4*>(&hk[w][ti * 4]);
            const uint4 v4 = *reinterpret_cast<const uint4*>(&vk[w][tj * 4]);
            const uint4 g4 = *reinterpret_cast<const uint4*>(&hk[w + 1][ti * 4]);
            const uint4 u4 = *reinterpret_cast<const uint4*>(&vk[w + 1][tj * 4]);
            const uint32_t hv[4] = {h4.x, h4.y, h4.z, h4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
            const uint32_t gv[4] = {g4.x, g4.y, g4.z, g4.w}, uv[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    sc[a][b] = add_on_fma(sc[a][b], pair_2w_t(hv[a], vv[b]), one);
                    sc[a][b] = add_on_fma(sc[a][b], pair_2w_t(gv[a], uv[b]), one);
                }
        }
        __syncthreads();
    }
    const int i = i0 + ti * 4;   // FE_ALIVE is a multiple of 4
    if (i >= FE_ALIVE) return;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int m = m0 + tj * 4 + b;
        if (m >= FE_VILL) continue;
        const int x = pos[1][tj * 4 + b][0], y = pos[1][tj * 4 + b][1];
        float eq[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int c = pos[0][ti * 4 + a][0], d = pos[0][ti * 4 + a][1];
            eq[a] = -1.0f;
            if (c != x && c != y && d != x && d != y) {
                const uint64_t ac = adj[c], ad = adj[d];
                const int shared = (int)((ac >> x) & 1ull) + (int)((ac >> y) & 1ull) + (int)((ad >> x) & 1ull) +
                                   (int)((ad >> y) & 1ull);
                const int n = (int)usable[0][ti * 4 + a] + (int)usable[1][tj * 4 + b] - FE_RUNOUTS + shared;
                if (n > 0) {
                    const int num = (int)((sc[a][b] & 0xFFFFu) + (sc[a][b] >> 16));
                    eq[a] = __fdiv_rn((float)num, (float)(2 * n));
                }
            }
        }
        *reinterpret_cast<float4*>(eqT + ((size_t)f * FE_VILL + m) * FE_ALIVE + i) = make_float4(eq[0], eq[1], eq[2], eq[3]);
    }
}

// Per hero, villains in increasing order, the reference's contracted FMAs.
__global__ void k_flop_accumulate(const float* __restrict__ eqT, const float* __restrict__ reach0,
                                  const float* __restrict__ reach1, int nflops,
                                  float* __restrict__ ev0, float* __restrict__ ev1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= FE_ALIVE || f >= nflops) return;
    const float uni = __fdiv_rn(1.0f, 1176.0f);
    const float* e = eqT + (size_t)f * FE_VILL * FE_ALIVE + i;
    float t0 = 0.0f, t1 = 0.0f;
    constexpr int U = 14;                          // equities in flight: 2.28 ms of loads one by one, 0.88 ms so
    static_assert(FE_VILL % U == 0, "whole steps");
    for (int m0 = 0; m0 < FE_VILL; m0 += U) {
        float q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = e[(size_t)(m0 + u) * FE_ALIVE];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int m = m0 + u;
            const float eq = q[u];
            if (eq < 0.0f) continue;
            const float r1 = reach1 ? reach1[4 * m] : uni;
            const float r0 = reach0 ? reach0[4 * m] : uni;
            t0 = __fmaf_rn(r1, __fmaf_rn(eq, 2.0f, -1.0f), t0);
            t1 = __fmaf_rn(r0, __fmaf_rn(__fsub_rn(1.0f, eq), 2.0f, -1.0f), t1);
        }
    }
    ev0[(size_t)f * FE_ALIVE + i] = t0;
    ev1[(size_t)f * FE_ALIVE + i] = t1;
}

// dump[f][scen][player][class]: the host loop of mtt_ev_dumper.cu:160-168,
// one thread per output, its class's combos in increasing combo order.
__global__ void k_dump_aggregate(const uint8_t* __restrict__ flops, const float* __restrict__ ev0,
                                 const float* __restrict__ ev1, int nflops, float* __restrict__ out) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nflops * 4 * 2 * 169) return;
    const int cls = idx % 169, pl = (idx / 169) % 2, scen = (idx / 338) % 4, f = idx / 1352;
    const uint8_t* fl = flops + 3 * f;
    const uint64_t fm = (1ull << fl[0]) | (1ull << fl[1]) | (1ull << fl[2]);
    // class -> ranks (mtt_ev_dumper.cu:26-32 inverted)
    int hi, lo, kind;   // kind 0 pair, 1 suited, 2 offsuit
    if (cls < 13) { hi = lo = 12 - cls; kind = 0; }
    else {
        kind = cls < 91 ? 1 : 2;
        int off = cls - (kind == 1 ? 13 : 91);
        hi = 12;
        while (off >= hi) { off -= hi; --hi; }
        lo = hi - 1 - off;
    }
    const float* ev = (pl == 0 ? ev0 : ev1) + (size_t)f * FE_ALIVE;
    const float mult = __fadd_rn(1.0f, __fmul_rn(0.1f, (float)scen));
    float acc = 0.0f;
    for (int s1 = 0; s1 < 4; ++s1) {
        for (int s2 = 0; s2 < 4; ++s2) {
            int c1, c2;
            if (kind == 0) { if (s2 <= s1) continue; c1 = 4 * lo + s1; c2 = 4 * hi + s2; }
            else if (kind == 1) { if (s2 != s1) continue; c1 = 4 * lo + s1; c2 = 4 * hi + s2; }
            else { if (s2 == s1) continue; c1 = 4 * lo + s1; c2 = 4 * hi + s2; }
            if (((fm >> c1) & 1ull) || ((fm >> c2) & 1ull)) continue;
            // alive index = lexicographic pair index over the 49-card deck
            const int a = c1 - __popcll(fm & ((1ull << c1) - 1ull));
            const int b = c2 - __popcll(fm & ((1ull << c2) - 1ull));
            const int i = a * 49 - (a * (a + 1)) / 2 + (b - a - 1);
            acc = __fadd_rn(acc, __fmul_rn(ev[i], mult));
        }
    }
    out[idx] = acc;
}

constexpr int FE_BATCH = 64;    // flops per scratch batch: keys and equities (117 MB) stay in the 126 MB L2

static int flop_ev_batched(const uint8_t* d_flops, int nflops, const float* d_reach0,
                           const float* d_reach1, float* d_ev0, float* d_ev1, cudaStream_t st) {
    const int nb = nflops < FE_BATCH ? nflops : FE_BATCH;
    uint32_t* keys = nullptr;
    float* eqT = nullptr;
    MTT_TRY(scratch_alloc(reinterpret_cast<void**>(&keys), (size_t)nb * FE_WORDS * FE_ALIVE * 4, st));
    int s = scratch_alloc(reinterpret_cast<void**>(&eqT), (size_t)nb * FE_VILL * FE_ALIVE * 4, st);
    for (int f0 = 0; s == MTT_OK && f0 < nflops; f0 += nb) {
        const int n = (nflops - f0) < nb ? (nflops - f0) : nb;
        const uint8_t* fl = d_flops + 3 * (size_t)f0;
        k_flop_keys<<<dim3(ceil_div(FE_ALIVE, 128), n), 128, 0, st>>>(fl, keys);
        k_flop_pair_eq<<<dim3(ceil_div(FE_ALIVE, FE_TH), ceil_div(FE_VILL, FE_TV), n), 256, 0, st>>>(
            keys, eqT, 1u);
        k_flop_accumulate<<<dim3(ceil_div(FE_ALIVE, 128), n), 128, 0, st>>>(
            eqT, d_reach0, d_reach1, n, d_ev0 + (size_t)f0 * FE_ALIVE, d_ev1 + (size_t)f0 * FE_ALIVE);
        s = cuda_status(cudaGetLastError());
    }
    if (eqT) cudaFreeAsync(eqT, st);
    cudaFreeAsync(keys, st);
    return s;
}

}  // namespace mtt

using namespace mtt;

extern "C" int mtt_eval7(const uint8_t* d_cards7, uint32_t* d_out, int64_t n, void* stream) {
    if (n < 0 || (n > 0 && (!d_cards7 || !d_out))) return MTT_ERR_INVALID;
    if (n == 0) return MTT_OK;
    cudaStream_t st = as_stream(stream);
    if (n >= EV_QUAD_MIN && (reinterpret_cast<uintptr_t>(d_cards7) & 3u) == 0u) {
        const unsigned grid = (unsigned)ceil_div_ll(n, 4 * EV_THREADS);
        if ((reinterpret_cast<uintptr_t>(d_out) & 15u) == 0u) k_eval7_quad<true><<<grid, EV_THREADS, 0, st>>>(d_cards7, d_out, n);
        else k_eval7_quad<false><<<grid, EV_THREADS, 0, st>>>(d_cards7, d_out, n);
    } else {
        // few hands: spread over the SMs; many at an odd address: 3,000,000 take
        // 26.8 us in blocks of 256, 28.8 in blocks of 64
        const int block = n < EV_QUAD_MIN ? 64 : EV_THREADS;
        k_eval7_plain<<<(unsigned)ceil_div_ll(n, block), block, 0, st>>>(d_cards7, d_out, n);
    }
    MTT_CHECK_LAUNCH();
    return MTT_OK;
}

extern "C" int mtt_eval7_enumerate(uint64_t* d_hist9, uint64_t* d_checksum, uint32_t* d_key_table,
                                   int32_t* d_err, void* stream) {
    if (!d_hist9 || !d_checksum || !d_err) return MTT_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    int sms = 0;
    MTT_TRY(sm_count(&sms));
    MTT_TRY_CUDA(cudaMemsetAsync(d_hist9, 0, 9 * sizeof(uint64_t), st));
    MTT_TRY_CUDA(cudaMemsetAsync(d_checksum, 0, sizeof(uint64_t), st));
    MTT_TRY_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int32_t), st));
    if (d_key_table) MTT_TRY_CUDA(cudaMemsetAsync(d_key_table, 0xFF, 65536 * sizeof(uint32_t), st));
    k_enumerate7<<<sms * 8, 256, 0, st>>>(reinterpret_cast<unsigned long long*>(d_hist9),
                                          reinterpret_cast<unsigned long long*>(d_checksum), d_key_table,
                                          reinterpret_cast<int*>(d_err));
    MTT_CHECK_LAUNCH();
    return MTT_OK;
}

extern "C" int mtt_board_showdown_counts(const uint8_t* d_board, int32_t nboard, const uint8_t* d_hands,
                                         int32_t H, int32_t* d_w, int32_t* d_t, int32_t* d_l,
                                         void* stream) {
    if (nboard < 3 || nboard > 5 || H < 0 || H > 1326) return MTT_ERR_INVALID;
    if (H == 0) return MTT_OK;
    if (!d_board || !d_hands || !d_w || !d_t || !d_l) return MTT_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    const int nrest = 52 - nboard;
    const int ncomp = nboard == 5 ? 1 : nboard == 4 ? nrest : nrest * (nrest - 1) / 2;
    const int ncw = (ncomp + 1) / 2;
    const int Hp = (H + 63) / 64 * 64;
    // compatible pairs see every completion that avoids their 4 cards
    const int free_cards = nrest - 4;
    const int n_const = nboard == 5 ? 1 : nboard == 4 ? free_cards : free_cards * (free_cards - 1) / 2;
    uint32_t* keys = nullptr;
    MTT_TRY(scratch_alloc(reinterpret_cast<void**>(&keys), (size_t)ncw * Hp * sizeof(uint32_t), st));
    k_completion_keys<<<dim3(Hp / 64, ncw), 64, 0, st>>>(d_board, nboard, d_hands, H, Hp, ncomp, keys);
    int s = cuda_status(cudaGetLastError());
    if (s == MTT_OK) {
        k_board_counts<<<dim3(Hp / BC_TILE, Hp / BC_TILE), 256, 0, st>>>(keys, ncw, H, Hp, d_hands, d_board,
                                                                        nboard, n_const, d_w, d_t, d_l, 1u);
        s = cuda_status(cudaGetLastError());
    }
    cudaFreeAsync(keys, st);
    return s;
}

// ------------------------------------------------ counts without allocation
// Key scratch of mtt_board_showdown_counts_noalloc: one per device, in the
// module's static device memory, so a call needs no allocator.  1 MiB.
static __device__ __align__(256) uint32_t g_counts_scratch[MTT_COUNTS_NOALLOC_MAX_WORDS];

namespace mtt {
constexpr int kMaxDevices = 64;
static std::mutex g_counts_scratch_mu;
static uint32_t* g_counts_scratch_ptr[kMaxDevices] = {};
static unsigned long long g_counts_scratch_ctx[kMaxDevices] = {};

// Address of this device's scratch in the current context.  It is looked up
// with the device current on the first call in each context (the first call
// on the device, and again after a cudaDeviceReset replaced its context).
static int counts_scratch(uint32_t** out) {
    int dev = 0;
    MTT_TRY_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return MTT_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_counts_scratch_mu);
    const unsigned long long ctx = current_context_id();
    if (!g_counts_scratch_ptr[dev] || ctx == 0 || ctx != g_counts_scratch_ctx[dev]) {
        void* p = nullptr;
        MTT_TRY_CUDA(cudaGetSymbolAddress(&p, g_counts_scratch));   // makes the device's context current
        g_counts_scratch_ptr[dev] = static_cast<uint32_t*>(p);
        g_counts_scratch_ctx[dev] = current_context_id();
    }
    *out = g_counts_scratch_ptr[dev];
    return MTT_OK;
}
}  // namespace mtt

extern "C" int mtt_board_showdown_counts_noalloc(const uint8_t* d_board, int32_t nboard, const uint8_t* d_hands,
                                                 int32_t H, int32_t* d_w, int32_t* d_t, int32_t* d_l,
                                                 void* stream) {
    if (nboard < 3 || nboard > 5 || H < 0 || H > 1326) return MTT_ERR_INVALID;
    if (H == 0) return MTT_OK;
    if (!d_board || !d_hands || !d_w || !d_t || !d_l) return MTT_ERR_INVALID;
    const int nrest = 52 - nboard;
    const int ncomp = nboard == 5 ? 1 : nboard == 4 ? nrest : nrest * (nrest - 1) / 2;
    const int ncw = (ncomp + 1) / 2;
    const int Hp = (H + 63) / 64 * 64;
    if ((long long)ncw * Hp > MTT_COUNTS_NOALLOC_MAX_WORDS) return MTT_ERR_UNSUPPORTED;
    const int free_cards = nrest - 4;
    const int n_const = nboard == 5 ? 1 : nboard == 4 ? free_cards : free_cards * (free_cards - 1) / 2;
    uint32_t* keys = nullptr;
    MTT_TRY(counts_scratch(&keys));
    cudaStream_t st = as_stream(stream);
    // Nothing in the scratch has to start at zero: k_completion_keys writes
    // all ncw * Hp words before k_board_counts reads any of them.
    k_completion_keys<<<dim3(Hp / 64, ncw), 64, 0, st>>>(d_board, nboard, d_hands, H, Hp, ncomp, keys);
    MTT_TRY_CUDA(cudaGetLastError());
    k_board_counts<<<dim3(Hp / BC_TILE, Hp / BC_TILE), 256, 0, st>>>(keys, ncw, H, Hp, d_hands, d_board, nboard,
                                                                    n_const, d_w, d_t, d_l, 1u);
    MTT_TRY_CUDA(cudaGetLastError());
    return MTT_OK;
}

extern "C" int mtt_canonical_flops(uint8_t* h_out, int32_t capacity, int32_t* n_out) {
    if (!n_out) return MTT_ERR_INVALID;
    // mtt_ev_dumper.cu:34-51: trips, paired, then unpaired families, orbit weights 4/12/24
    std::vector<uint8_t> v;
    v.reserve(1755 * 4);
    auto mc = [](int r, int s) { return (uint8_t)(r * 4 + s); };
    auto push = [&](uint8_t a, uint8_t b, uint8_t c, uint8_t w) { v.push_back(a); v.push_back(b); v.push_back(c); v.push_back(w); };
    for (int r = 12; r >= 0; --r) push(mc(r, 0), mc(r, 1), mc(r, 2), 4);
    for (int rp = 12; rp >= 0; --rp)
        for (int rk = 12; rk >= 0; --rk) {
            if (rp == rk) continue;
            push(mc(rp, 0), mc(rp, 1), mc(rk, 0), 12);
            push(mc(rp, 0), mc(rp, 1), mc(rk, 2), 12);
        }
    for (int r1 = 12; r1 >= 2; --r1)
        for (int r2 = r1 - 1; r2 >= 1; --r2)
            for (int r3 = r2 - 1; r3 >= 0; --r3) {
                push(mc(r1, 0), mc(r2, 0), mc(r3, 0), 4);
                push(mc(r1, 0), mc(r2, 0), mc(r3, 1), 12);
                push(mc(r1, 0), mc(r2, 1), mc(r3, 0), 12);
                push(mc(r1, 1), mc(r2, 0), mc(r3, 0), 12);
                push(mc(r1, 0), mc(r2, 1), mc(r3, 2), 24);
            }
    *n_out = (int32_t)(v.size() / 4);
    if (h_out) {
        if (capacity < *n_out) return MTT_ERR_INVALID;
        std::memcpy(h_out, v.data(), v.size());
    }
    return MTT_OK;
}

extern "C" int mtt_flop_ev(const uint8_t* d_flops, int32_t nflops, const float* d_reach0,
                           const float* d_reach1, float* d_ev0, float* d_ev1, void* stream) {
    if (nflops < 0) return MTT_ERR_INVALID;
    if (nflops == 0) return MTT_OK;
    if (!d_flops || !d_ev0 || !d_ev1) return MTT_ERR_INVALID;
    return flop_ev_batched(d_flops, nflops, d_reach0, d_reach1, d_ev0, d_ev1, as_stream(stream));
}

extern "C" int mtt_ev_dump(const uint8_t* d_flops, int32_t nflops, float* d_out, void* stream) {
    if (nflops < 0) return MTT_ERR_INVALID;
    if (nflops == 0) return MTT_OK;
    if (!d_flops || !d_out) return MTT_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    float *ev0 = nullptr, *ev1 = nullptr;
    MTT_TRY(scratch_alloc(reinterpret_cast<void**>(&ev0), (size_t)nflops * FE_ALIVE * 4, st));
    int s = scratch_alloc(reinterpret_cast<void**>(&ev1), (size_t)nflops * FE_ALIVE * 4, st);
    if (s == MTT_OK) s = flop_ev_batched(d_flops, nflops, nullptr, nullptr, ev0, ev1, st);
    if (s == MTT_OK) {
        const int total = nflops * 1352;
        k_dump_aggregate<<<ceil_div(total, 256), 256, 0, st>>>(d_flops, ev0, ev1, nflops, d_out);
        s = cuda_status(cudaGetLastError());
    }
    if (ev1) cudaFreeAsync(ev1, st);
    cudaFreeAsync(ev0, st);
    return s;
}
