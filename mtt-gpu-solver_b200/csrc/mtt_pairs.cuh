// mtt_pairs.cuh — packed comparisons of 16-bit score keys (key_planes).
//
// Packed comparisons.  A hero word holds key + 1 of two completions as signed
// halves, a villain word -key, so their half-wise sum is key_h - key_v + 1 and
// one saturating __viaddmin_s16x2_relu gives, per half,
//   clamp(sum, 0, 2) = 2 for a win, 1 for a tie, 0 for a loss,
// which sums to 2W + T; its bit 1 sums to 2W.
// A completion that uses one of the hand's cards (or padding) is KEY_H_DEAD in
// a hero word and KEY_V_DEAD in a villain word.  Keys are 1..16,972, so a sum
// with one dead side is below 0 and one with both (-17,001) does not wrap:
// dead completions count 0.  Two packed compares and their mask, before, were
// about 30 instructions a word (no half-word compare instruction exists); the
// clamp is one, which is what makes the pair counts cheap.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "mtt_device.cuh"

namespace mtt {

constexpr uint32_t KEY_H_DEAD = 0xFFFFu;            // -1
constexpr uint32_t KEY_V_DEAD = 0x10000u - 17000u;  // -17,000
static_assert(KEY_SFLUSH + 12 + 1 < 17000, "a live key never reaches a dead villain's offset");

__device__ __forceinline__ uint32_t villain_half(uint32_t h) {
    return h == KEY_H_DEAD ? KEY_V_DEAD : ((1u - h) & 0xFFFFu);
}
__device__ __forceinline__ uint32_t villain_word(uint32_t hero) {
    return villain_half(hero & 0xFFFFu) | (villain_half(hero >> 16) << 16);
}
__device__ __forceinline__ uint32_t pair_2w_t(uint32_t hero, uint32_t villain) {
    return __viaddmin_s16x2_relu(hero, villain, 0x00020002u);
}

// sum + t with the addition as a multiply-add, which leaves the integer pipe
// to the clamps (`one` must be 1 and unknown to the compiler).  All 1,755
// flops' equities: 8.7 ms with plain adds, 8.1 ms; the counts of a turn board
// 13.8 -> 12.3 us; the preflop flop equities, with more other integer work a
// word, 3.5 -> 3.7 ms, and keep plain adds.  What is left is 4.4 cycles a
// clamp and scheduler.
__device__ __forceinline__ uint32_t add_on_fma(uint32_t sum, uint32_t t, uint32_t one) {
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(t), "r"(one), "r"(sum));
    return r;
}

}  // namespace mtt
