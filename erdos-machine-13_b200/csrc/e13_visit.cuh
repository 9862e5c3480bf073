// e13_visit.cuh -- one visit of a Turing machine to a 32-cell tape word: the
// remembered form (memo entries) and the loop that makes one.  Used where a
// warp runs one machine a word at a time: long machines of the search
// (e13_macro.cuh) and the hash-free checkers (e13_walk.cuh).
//
// memo entry (uint4): x content on entry; y bits 0..5 the key (state, side
// entered from: 16 = right, 32 = valid), bits 6..11 the same for the word
// entered next, 16..31 steps (0: single-step this visit); z content on exit;
// w what the user of the entry wants noted.
//
// macro_visit is bound by its chain (row load, symbol select, position: 70
// cycles a step); both cells of a state come in one load, the rest of a step
// overlaps with it.
#pragma once
#include <stdint.h>

namespace e13dev {

constexpr unsigned kAll = 0xFFFFFFFFu;
constexpr int kMemoBits = 9;
constexpr int kMemoSize = 1 << kMemoBits;
constexpr int kMemoMaxSteps = 2048;  // longest remembered visit

__device__ __forceinline__ unsigned memo_slot(unsigned c, unsigned sk) {
  return (c * 0x9E3779B1u + sk * 0x85EBCA6Bu) >> (32 - kMemoBits);
}

// act words: bit 0 flip, bits 3..6 next state, bit 7 not a plain move, bits
// 24..31 the head's move (64 for anything but a plain move: leaves the word)
constexpr unsigned kActSpecial = 0x80u;
__device__ __forceinline__ unsigned act_word(unsigned code, unsigned sym) {
  if (code & 0xC0u) return 0x40000000u | kActSpecial;
  return ((code ^ sym) & 1u) | ((code << 1) & 0x78u) | ((code & 2u) ? 0x01000000u : 0xFF000000u);
}

// Runs the machine inside one word of content c until it leaves it: the entry
// to remember.  sk: the key (state and side).  NOTE: what the entry's w holds.
enum { kNoteNothing = 0, kNoteReads = 1, kNoteLowest = 2 };
template <int NOTE>
static __device__ __noinline__ uint4 macro_visit(const uint2 *act, unsigned c, unsigned sk) {
  unsigned w = c, reads = 0, x = 0, sw = 0;
  int st = (int)(sk & 15u), q = (sk & 16u) ? 31 : 0, n = 0, low = q, sq = -1, ss = 0;
  for (int next = 64; next <= kMemoMaxSteps; next += 64) {
    do {
      const uint2 a = act[st];
      const unsigned sym = (w >> q) & 1u;
      x = sym ? a.y : a.x;
      if (NOTE == kNoteReads) reads |= 1u << (2 * st + (int)sym);
      w ^= (x & 1u) << q;
      q += (int)x >> 24;
      if (NOTE == kNoteLowest) low = min(low, q);
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
  if ((unsigned)q <= 31u || (x & kActSpecial)) return make_uint4(c, sk, c, 0u);
  return make_uint4(c, sk | ((unsigned)(st | 32 | (q < 0 ? 16 : 0)) << 6) | ((unsigned)n << 16), w,
                    NOTE == kNoteLowest ? (unsigned)low : reads);
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
static __device__ __noinline__ void window_run(const uint2 *act, Window &V, int left, unsigned &reads) {
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
