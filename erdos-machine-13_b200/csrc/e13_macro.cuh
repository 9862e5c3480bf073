// e13_macro.cuh -- long machines: one warp runs one machine a tape word at a
// time.
//
// A machine that lives for thousands of steps sweeps over tape it has written
// before, so the same things happen inside the same words again and again.
// What a machine does inside one 32-cell word depends only on its state, the
// side it enters from and the word's content, so the warp remembers the
// outcome of each such visit (new content, exit side and state, steps) in a
// small table in shared memory and applies it in one go the next
// time.  An entry is made when it is first needed by running the machine
// inside the word.  A visit that leaves the word as it was and goes on into an
// equal word in the same state is a sweep: the lanes look at the next words
// together and the whole run is one action.
//
// What bounds it: the latency of one chain of dependent instructions, not
// issue slots.  All 32 lanes run the same scalar code; what can wait is put
// off and done by the lanes together: each visit is noted in one lane, and
// every 32 visits the lanes test all of them against the stage hash at once.
//
// Every result equals single-stepping (src/e13search.c:134-177):
//  * a remembered visit is applied only if all its steps pass the deadline;
//  * words 0 and 42, which hold the window's ends, are single-stepped;
//  * the stage test compares a 64-bit hash before every step.  Inside word b
//    the hash can only take values hb ^ s with s in the span (over GF(2)) of
//    the keys of b's cells.  32 linear functionals per word vanish on that
//    span, so if any of them is 1 on hb ^ TGT[nt], no step of the visit can
//    match.  Visits are undone back to the first one that fails this, and that
//    one is single-stepped with the test;
//  * a machine whose whole configuration repeats (inside one word, or inside
//    three words that it has not left since) with no stage reached on the way
//    runs on to its deadline and dies there (src/e13search.c:161).
#pragma once
#include "e13_device.cuh"
#include "e13_visit.cuh"

namespace e13dev {

constexpr int kWindowSteps = 4096;   // bare runs: steps of one turn in the window
constexpr int kYieldEvery = 4;       // ... batches of visits between looks at what they yield
constexpr int kStepCycles = 80;      // ... cycles a step in the window
constexpr int kLoopTries = 8;        // recurrences of a batch's first visit looked at
constexpr int kSnapEvery = 32;       // single-stepped visits between configuration snapshots
constexpr int kLastWord = kTapeWords - 1;
constexpr int kSpans = 32;           // functionals per word

// What one warp needs in shared memory.
template <int BITS>
struct MacroMem {
  uint4 memo[1 << BITS];
  u32 tape[kTapeWords + 1];
  uint2 act[16];  // the table for macro_visit
  u32 rows[16];
  u32 pad[4];
};

__device__ __forceinline__ unsigned long long macro_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// By the whole warp: has the clock passed t_end (kNoEnd: there is none)?  Lanes
// read clocks of their own, which may differ, and all take the way that follows
// from the answer: it is lane 0's.
constexpr unsigned long long kNoEnd = ~0ull;
__device__ __forceinline__ bool macro_late(unsigned long long t_end) {
  return t_end != kNoEnd && __shfl_sync(kAll, macro_clock() > t_end ? 1 : 0, 0) != 0;
}

// After a change of M.rows: the expanded table, and an empty memory of visits.
template <int BITS>
__device__ __forceinline__ void macro_table(MacroMem<BITS> &M, int lane) {
  __syncwarp();
  reinterpret_cast<u32 *>(M.act)[lane] = act_word((M.rows[lane >> 1] >> ((lane & 1) << 4)) & 0xFFu, (u32)lane & 1u);
  for (int i = lane; i < 1 << BITS; i += 32) M.memo[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
}

__device__ __forceinline__ u32 span_bit(u64 v, u64 f) {
  const u64 x = v & f;
  return __popc((u32)x ^ (u32)(x >> 32)) & 1u;
}

// Runs a machine (L, hb, M.tape, M.rows; the same in every lane) to its next
// event: kEvDead, kEvSurv, kEvCell (cell, ecell) or kEvRun when the clock
// passes t_end (HASH only).  HASH: the filter, hb being the full 64-bit hash.
// Otherwise the bare table runs until L.t is past L.deadline (kEvDead), and
// kEvOff says that a step left the window (L.p is then outside it, that step
// not counted).  READS: reads collects the table cells read.
enum { kEvOff = 5 };

template <bool HASH, bool READS = false, int BITS>
__device__ __forceinline__ int macro_run(Lane &L, u64 &hb, MacroMem<BITS> &M, const KeyTabs &K, const u64 *span,
                                         int lane, u32 &reads, int &cell, u32 &ecell, unsigned long long t_end) {
  int p = L.p, b = L.p >> 5;
  int left = L.deadline + 1 - L.t;  // steps that still pass the deadline test
  u64 tgt = HASH ? s_tgt[L.nt] : 0ull;
  u32 key = make_key(L.st, (p & 31) != 0);
  bool single = (p & 31) != 0 && (p & 31) != 31;  // this visit step by step
  bool inside = single;                           // the head is inside the word (at p), not on its edge
  // visits not yet tested: lane j holds the j-th (its word, key, steps left
  // before it and the cells it changed)
  int noted = 0, v_b = 0, v_left = 0;
  u32 v_key = 0, v_d = 0;
  int snap_b = 0, snaps = 0;
  u32 snap_at = 0, snap0 = 0, snap1 = 0, snap2 = 0;  // words snap_b - 1 .. snap_b + 1
  bool far = true;                  // left those words, or reached a stage, since the snapshot
  // bare runs: batches until the next look at what visits yield, steps left and
  // clock at the last one, steps still to take in the window
  int visits_left = kYieldEvery, yield_left = left, window_left = 0;
  long long yield_clock = HASH ? 0 : clock64();
  for (;;) {
    if (!single) {
      // remembered visits, one after another.  Nothing in this loop branches
      // but its end: what the visit changes is selected by `ok`
      u32 c, n;
      uint4 *slot, e;
      bool ok, in_range;
      bool rep;  // the visit left its word alone and goes on in the same way
      do {
        c = M.tape[b];
        slot = M.memo + memo_slot<BITS>(c, key);
        e = *slot;
        __syncwarp();  // every lane has read the word (here: while the loads are under way)
        n = memo_steps(e);
        in_range = (unsigned)(b - 1) < (unsigned)(kLastWord - 1);
        ok = in_range && memo_match(e, c, key) && n - 1u < (u32)left;
        const bool mine = ok && lane == noted;
        v_b = mine ? b : v_b;
        v_key = mine ? key : v_key;
        v_left = mine ? left : v_left;
        v_d = mine ? c ^ e.z : v_d;
        if (READS && ok) reads |= e.y;
        if (ok) M.tape[b] = e.z;  // every lane writes the same value
        const u32 next = memo_next(e);
        left = ok ? left - (int)n : left;
        noted = ok ? noted + 1 : noted;
        rep = ok && e.z == c && next == key;
        key = ok ? next : key;
        b = ok ? b + memo_move(e) : b;
      } while (ok && !rep && noted < 32);
      if (rep) {
        if (noted < 32) {
          // a sweep: the i-th free lane looks at the i-th word ahead
          const int dir = key_dir(key), i = lane - noted;
          const int w = b + dir * i;
          const bool same = i >= 0 && (unsigned)(w - 1) < (unsigned)(kLastWord - 1) && M.tape[w] == c;
          const u32 m = __ballot_sync(kAll, !same) >> noted;
          int run = m ? __ffs(m) - 1 : 32 - noted;
          if (run * (int)n > left) run = 0;
          if (i >= 0 && i < run) {
            v_b = w;
            v_key = key;
            v_left = left - i * (int)n;
            v_d = 0;
          }
          noted += run;
          left -= run * (int)n;
          b += dir * run;
          if (noted < 32) continue;
        }
      } else if (!ok) {
        if (in_range && !memo_match(e, c, key)) {
          if (memo_steps(memo_fetch<READS, false>(slot, e, M.act, c, key, lane))) continue;
          single = true;
        } else {
          single = true;  // an end of the window, a visit to be single-stepped, or too few steps left
        }
      }
    }

    if (noted) {
      // test the visits noted
      __syncwarp();
      const bool mine = lane < noted;
      bool bad = false;
      u64 sum = 0;
      const u64 start = hb;
      if (HASH) {
        if (__any_sync(kAll, mine && v_d)) {  // (sweeps change nothing)
          u32 lo = 0, hi = 0;
          for (u32 d = mine ? v_d : 0u; d; d &= d - 1) {
            const int i = 32 * v_b + __ffs(d) - 1;
            lo ^= K.lo[i];
            hi ^= K.hi[i];
          }
          const u32 lo0 = lo, hi0 = hi;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {  // running hash changes
            const u32 a = __shfl_up_sync(kAll, lo, o), c = __shfl_up_sync(kAll, hi, o);
            if (lane >= o) {
              lo ^= a;
              hi ^= c;
            }
          }
          sum = ((u64)(hi ^ hi0) << 32) | (lo ^ lo0);  // before this lane's visit
          hb ^= ((u64)__shfl_sync(kAll, hi, 31) << 32) | __shfl_sync(kAll, lo, 31);
        }
        const u64 v = start ^ sum ^ tgt;
        bad = mine;
        for (int j = 0; j < kSpans && __any_sync(kAll, bad); j += 8) {
          u32 any = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) any |= span_bit(v, span[(j + k) * kTapeWords + v_b]);
          if (any) bad = false;
        }
      }
      u32 m = __ballot_sync(kAll, bad);
      if (m) {
        // back to the first visit that a stage start might fall into
        const int j = __ffs(m) - 1;
        if (mine && lane >= j && v_d) atomicXor(&M.tape[v_b], v_d);
        __syncwarp();
        b = __shfl_sync(kAll, v_b, j);
        key = __shfl_sync(kAll, v_key, j);
        left = __shfl_sync(kAll, v_left, j);
        hb = start ^ (((u64)__shfl_sync(kAll, (u32)(sum >> 32), j) << 32) | __shfl_sync(kAll, (u32)sum, j));
        single = true;
        noted = j;
      }
      // do the visits that stand contain a turn of a loop?  Visit j enters the
      // same word in the same way as visit 0, and between them only visit 0's
      // word and its neighbours were entered and ended as they were
      const int b0 = __shfl_sync(kAll, v_b, 0);
      const u32 key0 = __shfl_sync(kAll, v_key, 0);
      if (HASH && __any_sync(kAll, lane < noted && (unsigned)(v_b - snap_b + 1) > 2u)) far = true;
      m = __ballot_sync(kAll, lane > 0 && lane < noted && v_b == b0 && v_key == key0);
      for (int tries = 0; m && tries < kLoopTries; ++tries, m &= m - 1) {
        const int j = __ffs(m) - 1;
        const bool in = lane < j;
        if (__any_sync(kAll, in && (unsigned)(v_b - b0 + 1) > 2u)) break;
        const u32 x0 = __reduce_xor_sync(kAll, (in && v_b == b0 - 1) ? v_d : 0u);
        const u32 x1 = __reduce_xor_sync(kAll, (in && v_b == b0) ? v_d : 0u);
        const u32 x2 = __reduce_xor_sync(kAll, (in && v_b == b0 + 1) ? v_d : 0u);
        if ((x0 | x1 | x2) == 0u) {
          if (HASH) {
            L.t = L.deadline + 1;
            return kEvDead;
          }
          left %= __shfl_sync(kAll, v_left, 0) - __shfl_sync(kAll, v_left, j);
          break;
        }
      }
      if (!HASH && --visits_left <= 0) {
        // visits that cost more than the steps they take: over to the window
        const long long now = clock64();
        // (lane 0's clock decides, as in macro_late)
        if (__shfl_sync(kAll, now - yield_clock > (long long)kStepCycles * (yield_left - left) ? 1 : 0, 0)) {
          single = true;
          window_left = kWindowSteps;
        }
        yield_left = left;
        yield_clock = now;
        visits_left = kYieldEvery;
      }
      noted = 0;
      if (HASH && macro_late(t_end)) {
        L.p = b * 32 + key_bit(key);
        L.st = key_state(key);
        L.t = L.deadline + 1 - left;
        return kEvRun;
      }
    }
    if (!single) continue;

    int st = key_state(key);
    if (!inside) p = b * 32 + key_bit(key);
    if (!HASH && p >= 18 && p <= kTapeCells - 18) {
      // a bare run: 32 cells around the head, all inside the window the machine
      // may not leave, step by step
      const int b0 = (p - 16) >> 5, sh = (p - 16) & 31;
      const u32 w0 = M.tape[b0], w1 = M.tape[b0 + 1];
      Window V;
      V.w = __funnelshift_r(w0, w1, sh);
      V.q = 16;
      V.st = st;
      u32 r = 0;
      window_run<READS>(M.act, V, left < kWindowSteps ? left : kWindowSteps, r);
      if (READS) reads |= r;
      __syncwarp();
      M.tape[b0] = (w0 & ~(0xFFFFFFFFu << sh)) | (V.w << sh);
      if (sh) M.tape[b0 + 1] = (w1 & (0xFFFFFFFFu << sh)) | (V.w >> (32 - sh));
      __syncwarp();
      left -= V.steps;
      if (V.loop) left %= V.loop;
      p += V.q - 16;
      st = V.st;
      b = p >> 5;
      key = make_key(st, (p & 31) != 0);
      inside = (p & 31) != 0 && (p & 31) != 31;
      yield_left = left;
      yield_clock = clock64();
      visits_left = kYieldEvery;
      window_left -= V.steps;
      if (V.special || left <= 0) {
        L.p = p;
        L.st = st;
        L.t = L.deadline + 1 - left;
        __syncwarp();
        if (!V.special) return kEvDead;
        const u32 sym = (M.tape[b] >> (p & 31)) & 1u;
        cell = (st << 1) | (int)sym;
        ecell = (M.rows[st] >> (sym << 4)) & 0xFFu;
        return kEvCell;
      }
      // inside a word still, or not yet done: on with the window
      single = inside || window_left > 0;
      continue;
    }
    // single steps until the head is in another word (bare runs: in the first
    // and last word only)
    if (HASH) {
      // a loop that passes through here every turn: the same configuration
      // again, on words not left since the snapshot?
      if ((unsigned)(b - snap_b + 1) > 2u) far = true;
      const u32 at_here = ((u32)p << 4) | (u32)st;
      if (!far && at_here == snap_at && M.tape[b] == snap1 && M.tape[b - 1] == snap0 && M.tape[b + 1] == snap2) {
        left = 0;
        far = true;
      }
      if (--snaps < 0 && (unsigned)(b - 1) < (unsigned)(kLastWord - 1)) {
        snaps = kSnapEvery;
        snap_b = b;
        snap_at = at_here;
        snap0 = M.tape[b - 1];
        snap1 = M.tape[b];
        snap2 = M.tape[b + 1];
        far = false;
        if (macro_late(t_end)) {
          L.p = p;
          L.st = st;
          L.t = L.deadline + 1 - left;
          return kEvRun;
        }
      }
    }
    u32 word = M.tape[b];
    __syncwarp();  // every lane has read the word (and its neighbours, above) before one writes it
    u32 lw = 0;    // a configuration inside this word seen earlier
    int lat = -1, lleft = 0, lk = 0, lnext = 32, ev = -1;
    do {
      if (left <= 0) {
        ev = kEvDead;
        break;
      }
      const uint2 a = M.act[st];
      const u32 sym = (word >> (p & 31)) & 1u;
      const u32 x = sym ? a.y : a.x;
      if (x & kActSpecial) {
        cell = (st << 1) | (int)sym;
        ecell = (M.rows[st] >> (sym << 4)) & 0xFFu;
        ev = kEvCell;
        break;
      }
      if (READS) reads |= 1u << ((st << 1) | (int)sym);
      if (x & 1u) {
        word ^= 1u << (p & 31);
        if (HASH) hb ^= ((u64)K.hi[p] << 32) | K.lo[p];
      }
      const int np = p + ((int)x >> 24);
      if ((unsigned)(np - 1) >= (unsigned)(kTapeCells - 2)) {  // head <= -64 or >= 1299
        ev = kEvDead;
        if (!HASH) {
          p = np;
          ev = kEvOff;
        }
        break;
      }
      p = np;
      st = (int)((x >> 3) & 15u);
      --left;
      if (HASH && hb == tgt) {
        M.tape[b] = word;
        L.hb = (u32)hb;
        L.p = p;
        L.st = st;
        L.t = L.deadline + 1 - left;
        const int nt = L.nt;
        ev = stage_check(L, M.tape, K, 1);
        __syncwarp();  // every lane has read the tape
        if (ev) break;
        ev = -1;
        if (L.nt != nt) {
          left = L.deadline + 1 - L.t;
          tgt = s_tgt[L.nt];
          lat = -1;
          far = true;
        }
      }
      if (++lk >= lnext) {  // (the first 31 steps are not looked at)
        const int at = (p << 4) | st;
        if (at == lat && word == lw) {  // it loops inside this word
          if (HASH) {
            left = 0;
            ev = kEvDead;
            break;
          }
          left %= lleft - left;
          lat = -1;
        } else if (lk >= 2 * lnext || lat < 0) {
          lat = at;
          lw = word;
          lleft = left;
          lnext = lk;
        }
      }
    } while ((p >> 5) == b);
    M.tape[b] = word;
    if (ev >= 0) {
      L.p = p;
      L.st = st;
      L.t = L.deadline + 1 - left;
      __syncwarp();
      return ev;
    }
    b = p >> 5;
    key = make_key(st, (p & 31) != 0);
    single = inside = false;
  }
}

}  // namespace e13dev
