// e13_visit.cuh -- one visit of a Turing machine to a 32-cell tape word: the
// remembered form (memo entries) and the loop that makes one.  Used where a
// warp runs one machine a word at a time: long machines of the search
// (e13_macro.cuh) and the hash-free checkers (e13_walk.cuh).
//
// memo entry (uint4): x content on entry; z content on exit; w bits 0..11
// steps (0: single-step this visit), 12..17 the key (state, side entered from:
// 16 = right, 32 = valid), 18..23 the key for the word entered next, 24..29 the
// lowest bit reached + 1, 30..31 the next word minus this one (signed); y the
// table cells read (bit per cell), where they are asked for.  Keys are kept
// shifted to bits 12..17 (Key), so that one entry is checked and applied in
// few instructions: a visit is bound by their number.
//
// The routines are inlined where they are used: the table and the memory of
// visits are then known to be in shared memory (through pointers handed to a
// function every access would be a generic one).
#pragma once
#include <stdint.h>

namespace e13dev {

constexpr unsigned kAll = 0xFFFFFFFFu;
constexpr int kMemoMaxSteps = 2048;  // longest remembered visit

// A key: state and side, in place for a memo entry's w.
constexpr unsigned kKeyMask = 0x3F000u, kKeyRight = 16u << 12;
__device__ __forceinline__ unsigned make_key(int st, bool right) {
  return ((unsigned)st | 32u | (right ? 16u : 0u)) << 12;
}
__device__ __forceinline__ int key_state(unsigned key) { return (int)((key >> 12) & 15u); }
__device__ __forceinline__ int key_bit(unsigned key) { return (key & kKeyRight) ? 31 : 0; }  // the bit entered at
__device__ __forceinline__ int key_dir(unsigned key) { return (key & kKeyRight) ? -1 : 1; }

// The first of the two slots a visit may be in: the last one used comes first,
// the other second.  (With one slot each, two visits of a machine's sweep
// often shared it and each evicted the other 2000 times.)  BITS: the memory
// has 2^BITS entries.
template <int BITS>
__device__ __forceinline__ unsigned memo_slot(unsigned c, unsigned key) {
  return ((c * 0x9E3779B1u + key * 0x85EBCA6Bu) >> (33 - BITS)) << 1;
}
__device__ __forceinline__ bool memo_match(const uint4 &e, unsigned c, unsigned key) {
  return e.x == c && ((e.w ^ key) & kKeyMask) == 0u;
}
__device__ __forceinline__ unsigned memo_steps(const uint4 &e) { return e.w & 0xFFFu; }
__device__ __forceinline__ unsigned memo_next(const uint4 &e) { return (e.w >> 6) & kKeyMask; }
__device__ __forceinline__ int memo_move(const uint4 &e) { return (int)e.w >> 30; }
__device__ __forceinline__ int memo_lowest(const uint4 &e) { return (int)((e.w >> 24) & 63u) - 1; }

// act words: bit 0 flip, bits 3..6 next state, bit 7 not a plain move, bits
// 24..31 the head's move (64 for anything but a plain move: leaves the word)
constexpr unsigned kActSpecial = 0x80u;
__device__ __forceinline__ unsigned act_word(unsigned code, unsigned sym) {
  if (code & 0xC0u) return 0x40000000u | kActSpecial;
  return ((code ^ sym) & 1u) | ((code << 1) & 0x78u) | ((code & 2u) ? 0x01000000u : 0xFF000000u);
}

// Runs the machine inside one word of content c until it leaves it: the entry
// to remember.
template <bool READS, bool LOWEST>
__device__ __forceinline__ uint4 macro_visit(const uint2 *act, unsigned c, unsigned key) {
  unsigned w = c, reads = 0, x = 0, sw = 0;
  int st = key_state(key), q = key_bit(key), n = 0, low = q, sq = -1, ss = 0;
  for (int next = 64; next <= kMemoMaxSteps; next += 64) {
    do {
      const uint2 a = act[st];
      const unsigned sym = (w >> q) & 1u;
      x = sym ? a.y : a.x;
      if (READS) reads |= 1u << (2 * st + (int)sym);
      w ^= (x & 1u) << q;
      q += (int)x >> 24;
      if (LOWEST) low = min(low, q);
      st = (int)((x >> 3) & 15u);
      ++n;
    } while ((unsigned)q <= 31u && n < next);
    // every 64 steps: left, or (most loops have few steps) in a loop?
    if ((unsigned)q > 31u || (w == sw && q == sq && st == ss)) break;
    if ((n & (n - 1)) == 0) {
      sw = w;
      sq = q;
      ss = st;
    }
  }
  if ((unsigned)q <= 31u || (x & kActSpecial)) return make_uint4(c, 0u, c, key);
  return make_uint4(c, reads, w, (unsigned)n | key | (make_key(st, q < 0) << 6) | ((unsigned)(low + 1) << 24) |
                                     (q < 0 ? 0xC0000000u : 0x40000000u));
}

// The entry of a visit that is not first in its slots: remembered or made, and
// put first.  By the whole warp; first: what slot[0] holds.
template <bool READS, bool LOWEST>
__device__ __forceinline__ uint4 memo_fetch(uint4 *slot, const uint4 &first, const uint2 *act, unsigned c, unsigned key,
                                            int lane) {
  uint4 v = slot[1];
  if (!memo_match(v, c, key)) v = macro_visit<READS, LOWEST>(act, c, key);
  __syncwarp();
  if (lane == 0) {
    slot[1] = first;
    slot[0] = v;
  }
  __syncwarp();
  return v;
}

// Runs a machine (state st, head on cell q of the 32-cell window w) for at
// most `left` steps, until it leaves the window or meets a cell that is no plain
// move (special; the head is then on it).  The steps taken, with the window,
// head (-1 or 32: left) and state after them.  loop: 0, or the length of a
// loop that the machine is in.  For machines that visits do not help: those
// that turn inside a word for long or back and forth over an edge.
struct Window {
  unsigned w;
  int q, st, steps, loop;
  bool special;
};

template <bool READS>
__device__ __forceinline__ void window_run(const uint2 *act, Window &V, int left, unsigned &reads) {
  unsigned w = V.w, sw = ~w;
  int q = V.q, st = V.st, n = 0, sq = -1, ss = 0, sn = 0;
  V.loop = 0;
  V.special = false;
  for (int next = min(64, left); n < left; next = min(n + 64, left)) {
    unsigned x = 0;
    int last = st;
    while ((unsigned)q <= 31u && n < next) {
      const uint2 a = act[st];
      const unsigned sym = (w >> q) & 1u;
      x = sym ? a.y : a.x;
      last = st;
      if (READS) reads |= 1u << (2 * st + (int)sym);
      w ^= (x & 1u) << q;
      q += (int)x >> 24;
      st = (int)((x >> 3) & 15u);
      ++n;
    }
    if (x & kActSpecial) {  // that step is not taken
      q -= 64;
      st = last;
      --n;
      V.special = true;
      break;
    }
    if ((unsigned)q > 31u) break;
    if (w == sw && q == sq && st == ss) {
      V.loop = n - sn;
      break;
    }
    if ((n & (n - 1)) == 0) {
      sw = w;
      sq = q;
      ss = st;
      sn = n;
    }
  }
  V.w = w;
  V.q = q;
  V.st = st;
  V.steps = n;
}

}  // namespace e13dev
