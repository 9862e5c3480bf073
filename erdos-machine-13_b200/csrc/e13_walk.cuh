// e13_walk.cuh -- the hash-free checkers' simulator: one warp runs one machine
// on a wide tape a word at a time until a stage start, a limit, a cell that is
// no plain move, or the edge of the allowed cells (src/recheck.c:61-92,
// src/deep.c:49-80, src/check.py:55-77).
//
// The tape's busy part, cells -4096 .. -4096 + 32 W - 1, is in shared memory,
// the rest (if any) in device memory.  Visits to a word of it are remembered
// (e13_visit.cuh) and applied whole; a visit that leaves its word alone and
// goes on into an equal word in the same state is a sweep, whose next 32 words
// the lanes look at together.  What is single-stepped instead: visits during
// which a stage start could fall (the ones outside the word must then number
// exactly the block's cells outside it), visits that the step limit would cut,
// words with a cell that is not allowed.
//
// Bound by the number of instructions of one chain, 200-250 cycles a visit; a
// survivor's 13 million steps to stage 12 are about 60,000 visits and sweeps.
// One B200, one lane per machine before, one warp now: recheck of 61 survivors
// to stage 12 357 -> 6.8 ms, check.py on 8 survivors 580 -> 4.1 ms.  Words in
// device memory have a path of their own, some 600 cycles a visit: a survivor
// that zigzags 16,000 cells beyond the window for 1.3e8 steps took 31 s with a
// lane, 13.9 with a warp that single-steps there, 1.7 with this path.  A machine
// whose configuration repeats (inside one word, or inside three words that it
// has not left since) turns until its limit: whole turns are left out.
#pragma once
#include "e13_visit.cuh"

namespace e13dev {

typedef long long wi64;

constexpr int kWalkLeft = 4096;                       // the window starts at cell -4096
constexpr int kWalkZero = kWalkLeft >> 5;             // its word of cell 0
constexpr unsigned kBlockBits = 0xC0000000u;          // cells -2, -1 in the word before it
// Visits remembered.  More of them cost nothing where every machine has an SM
// to itself, and fewer are made again: 512 -> 1024 took recheck of 61 survivors
// from 7.6 to 6.6 ms and check.py on 8 from 4.2 to 3.6; 2048 gave 6.5 and 3.6.
constexpr int kWalkMemoBits = 10;
constexpr int kWalkWatch = 512;                       // visits between looks for a repeated configuration,
constexpr int kWalkWatchFor = 64;                     // each of this many visits

// A warp's tape.
struct WalkTape {
  unsigned *win;  // W words in shared memory
  int W;
  unsigned *g;    // the other words: word w of the window's numbering at g[w + gshift]
  wi64 gshift;
  __device__ __forceinline__ unsigned ld(int w) const {
    return (unsigned)w < (unsigned)W ? win[w] : g[w + gshift];
  }
  __device__ __forceinline__ void st(int w, unsigned v) const {
    if ((unsigned)w < (unsigned)W) win[w] = v;
    else g[w + gshift] = v;
  }
};

// When a stage starts: the ones at cells >= -2 are the block -1 .. size - 2,
// and the state and head match (any: they need not).
struct WalkStop {
  int size, st, want1, want2;
  bool any;
};

struct Walker {
  int head, st, ones, minhead;
  wi64 left;  // steps until the limit
};

enum { kWalkStop = 0, kWalkLimit = 1, kWalkCell = 2, kWalkRange = 3 };

__device__ __forceinline__ int walk_word(int cell) { return (cell + kWalkLeft) >> 5; }

// The cells >= -2 of word b.
__device__ __forceinline__ unsigned walk_mask(int b) {
  return b >= kWalkZero ? 0xFFFFFFFFu : (b == kWalkZero - 1 ? kBlockBits : 0u);
}

// The cells of the block -1 .. size - 2 in word b.
__device__ __forceinline__ unsigned walk_block(int b, int size) {
  const int first = 32 * b - kWalkLeft;
  const int lo = max(-1 - first, 0), hi = min(size - 2 - first, 31);
  if (lo > 31 || hi < lo) return 0u;
  return (0xFFFFFFFFu >> (31 - hi)) & (0xFFFFFFFFu << lo);
}

// By the whole warp: is all of the block set?
__device__ __forceinline__ bool walk_block_set(const WalkTape &T, int size, int lane) {
  bool ok = true;
  const int last = walk_word(size - 2);
  for (int b = kWalkZero - 1 + lane; b <= last; b += 32) {
    const unsigned m = walk_block(b, size);
    if ((T.ld(b) & m) != m) ok = false;
  }
  return __all_sync(kAll, ok);
}

// Runs to the next event.  CRAFT: check.py's order of tests before a step
// (edge, limit, stage start) instead of recheck.c's and deep.c's (stage start,
// limit, edge).  The head may be at cells lo .. hi.  For kWalkCell, W.st and
// *sym say which cell.  memo must be empty or hold this table's visits.
template <bool CRAFT>
__device__ __forceinline__ int walk_run(const WalkTape &T, uint4 *memo, const uint2 *act, int lane, Walker &W,
                                     const WalkStop &S, int lo, int hi, int *sym_out) {
  int head = W.head, ones = W.ones, minhead = W.minhead;
  wi64 left = W.left;
  int b = walk_word(head);
  const int a_lo = (lo + kWalkLeft + 31) >> 5, a_hi = ((hi + 1 + kWalkLeft) >> 5) - 1;  // words of allowed cells
  const int b_lo = max(a_lo, 0), b_hi = min(a_hi, T.W - 1);                             // ... in the window
  const int w1 = walk_word(S.want1), w2 = walk_word(S.want2);
  const int t1 = __popc(walk_block(w1, S.size)), t2 = __popc(walk_block(w2, S.size));
  const int q0 = (head + kWalkLeft) & 31;
  bool inside = q0 != 0 && q0 != 31;  // the head is inside its word, not on an edge
  bool single = inside || S.any;
  unsigned key = make_key(W.st, q0 != 0);
  int count = kWalkWatch, watch = 0;
  int snap_b = 0;
  wi64 snap_left = 0;
  unsigned snap_key = 0, snap0 = 0, snap1 = 0, snap2 = 0;
  bool far = true;      // left the words snap_b - 1 .. snap_b + 1 since the snapshot
  for (;;) {
    if (!single) {
      unsigned c, n;
      uint4 *slot, e;
      bool ok, in_range, clear;
      bool rep;  // the visit left its word alone and goes on in the same way
      do {
        in_range = b >= b_lo && b <= b_hi;
        c = T.win[in_range ? b : 0];
        slot = memo + memo_slot<kWalkMemoBits>(c, key);
        e = *slot;
        __syncwarp();  // every lane has read the word (here: while the loads are under way)
        n = memo_steps(e);
        const unsigned mask = walk_mask(b);
        const int was = __popc(c & mask);
        clear = (b != w1 || ones - was != S.size - t1) && (b != w2 || ones - was != S.size - t2);
        ok = in_range && clear && memo_match(e, c, key) && n != 0 && (wi64)n <= left;
        if (ok) T.win[b] = e.z;  // every lane writes the same value
        const unsigned next = memo_next(e);
        ones = ok ? ones + __popc(e.z & mask) - was : ones;
        minhead = ok ? min(minhead, 32 * b - kWalkLeft + memo_lowest(e)) : minhead;
        left = ok ? left - (wi64)n : left;
        rep = ok && e.z == c && next == key;
        key = ok ? next : key;
        b = ok ? b + memo_move(e) : b;
      } while (ok && !rep && --count > 0);
      if (rep) {
        // a sweep: lane i looks at the i-th word ahead (a word that a stage may
        // start in is left to the loop above)
        --count;
        const int dir = key_dir(key);
        const int w = b + dir * lane;
        const bool same = w >= b_lo && w <= b_hi && w != w1 && w != w2 && T.win[w] == c;
        const unsigned m = __ballot_sync(kAll, !same);
        int run = m ? __ffs(m) - 1 : 32;
        if ((wi64)run * n > left) run = 0;
        left -= (wi64)run * n;
        b += dir * run;
        // each visit went down to its lowest bit (and one past the word when going left)
        if (run > 0) minhead = min(minhead, 32 * (dir < 0 ? b + 1 : b - run) - kWalkLeft + memo_lowest(e));
      } else if (!ok) {
        if (in_range && clear && !memo_match(e, c, key)) {
          single = memo_steps(memo_fetch<false, true>(slot, e, act, c, key, lane)) == 0;
        } else if (!in_range && b >= a_lo && b <= a_hi) {
          // a word in device memory: the same rules, one visit or sweep
          --count;
          c = T.ld(b);
          slot = memo + memo_slot<kWalkMemoBits>(c, key);
          e = *slot;
          if (!memo_match(e, c, key)) e = memo_fetch<false, true>(slot, e, act, c, key, lane);
          n = memo_steps(e);
          const unsigned mask = walk_mask(b);
          const int was = __popc(c & mask);
          single = n == 0 || (wi64)n > left || (b == w1 && ones - was == S.size - t1) ||
                   (b == w2 && ones - was == S.size - t2);
          if (!single) {
            const int dir = key_dir(key);
            int run = 1;
            if (e.z == c && memo_next(e) == key) {
              const int w = b + dir * lane;
              const bool same = w >= a_lo && w <= a_hi && (unsigned)w >= (unsigned)T.W &&
                                (w == b || (w != w1 && w != w2)) && T.ld(w) == c;
              const unsigned m = __ballot_sync(kAll, !same);
              run = m ? __ffs(m) - 1 : 32;
              if ((wi64)run * n > left) run = 1;
            } else {
              __syncwarp();
              T.st(b, e.z);
              ones += __popc(e.z & mask) - was;
            }
            left -= (wi64)run * n;
            minhead = min(minhead, 32 * (dir < 0 ? b - run + 1 : b) - kWalkLeft + memo_lowest(e));
            b += run > 1 ? dir * run : memo_move(e);
            key = memo_next(e);
          }
        } else {
          single = true;
        }
      }
      if (!single) {
        if ((unsigned)(b - snap_b + 1) > 2u) far = true;
        if (count <= 0) {
          if (watch == 0) {  // a snapshot, and a look after each of the next visits
            if (b > a_lo && b < a_hi) {
              snap_b = b;
              snap_key = key;
              snap_left = left;
              snap0 = T.ld(b - 1);
              snap1 = T.ld(b);
              snap2 = T.ld(b + 1);
              far = false;
            }
            watch = kWalkWatchFor;
          } else {
            if (!far && b == snap_b && key == snap_key && T.ld(b) == snap1 && T.ld(b - 1) == snap0 &&
                T.ld(b + 1) == snap2) {
              left %= snap_left - left;
              far = true;
            }
            --watch;
          }
          if (watch == 0) {
            far = true;
            count = kWalkWatch;
          } else {
            count = 1;
          }
        }
        continue;
      }
    }

    // single steps until the head is in another word
    far = true;
    int st = key_state(key);
    if (!inside) head = 32 * b - kWalkLeft + key_bit(key);
    if (head < lo || head > hi) {
      // beyond the allowed cells, and perhaps beyond the tape: its word is not
      // touched (check.py's allowed cells fill its tape exactly)
      int ev = kWalkRange;
      if (!CRAFT) {
        if (ones == S.size && (S.any || (st == S.st && (head == S.want1 || head == S.want2))) &&
            walk_block_set(T, S.size, lane))
          ev = kWalkStop;
        else if (left <= 0)
          ev = kWalkLimit;
      }
      __syncwarp();
      W.head = head;
      W.st = st;
      W.ones = ones;
      W.minhead = minhead;
      W.left = left;
      return ev;
    }
    unsigned word = T.ld(b);
    __syncwarp();  // every lane has read the word
    const int first = 32 * b - kWalkLeft;
    unsigned lw = 0;  // a configuration inside this word seen earlier
    int lat = -1, lk = 0, lnext = 64, ev = -1;
    wi64 lleft = 0;
    do {
      if (CRAFT) {
        if (head < lo || head > hi) {
          ev = kWalkRange;
          break;
        }
        if (left <= 0) {
          ev = kWalkLimit;
          break;
        }
      }
      if (ones == S.size && (S.any || (st == S.st && (head == S.want1 || head == S.want2)))) {
        T.st(b, word);
        if (walk_block_set(T, S.size, lane)) {
          ev = kWalkStop;
          break;
        }
      }
      if (!CRAFT) {
        if (left <= 0) {
          ev = kWalkLimit;
          break;
        }
        if (head < lo || head > hi) {
          ev = kWalkRange;
          break;
        }
      }
      const int q = head - first;
      const uint2 a = act[st];
      const unsigned sym = (word >> q) & 1u;
      const unsigned x = sym ? a.y : a.x;
      if (x & kActSpecial) {
        *sym_out = (int)sym;
        ev = kWalkCell;
        break;
      }
      if (x & 1u) {
        word ^= 1u << q;
        if (head >= -2) ones += sym ? -1 : 1;
      }
      head += (int)x >> 24;
      minhead = min(minhead, head);
      st = (int)((x >> 3) & 15u);
      --left;
      if (++lk >= lnext) {  // (the first steps are not looked at)
        const int at = (head << 4) | st;
        if (lat != -1 && at == lat && word == lw) {  // it loops inside this word
          left %= lleft - left;
          lat = -1;
        } else if (lk >= 2 * lnext || lat == -1) {
          lat = at;
          lw = word;
          lleft = left;
          lnext = lk;
        }
      }
    } while ((unsigned)(head - first) <= 31u);
    T.st(b, word);
    if (ev >= 0) {
      __syncwarp();
      W.head = head;
      W.st = st;
      W.ones = ones;
      W.minhead = minhead;
      W.left = left;
      return ev;
    }
    b = walk_word(head);
    key = make_key(st, head < first);
    inside = false;
    single = S.any;
  }
}

}  // namespace e13dev
