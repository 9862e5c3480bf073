// e13_scratch.h -- device working memory that a context keeps between calls.
//
// cudaMalloc and cudaFree of a call's buffers cost more than many calls' work
// (recheck of 61 survivors: 11 ms of kernels in calls of 15 to 900 ms; a serve
// session's second stack is 5 GB), so each buffer of each call has a slot in
// the context that grows on demand.  A slot above kScratchKeep, or a second
// stack of more than kAltKeepNodes, is given back when its call or session is
// over; all of them when the context goes, and when another call or buffer of
// the context runs out of memory.  One host thread per context, as for every
// call.
#pragma once
#include <stddef.h>

struct e13_ctx;

enum {
  kScratchCheckTapes, kScratchCheckIn, kScratchCheckOut,
  kScratchCraftTables, kScratchCraftWalks, kScratchCraftTapes, kScratchCraftRuns, kScratchCraftRunOuts, kScratchCraftCells,
  kScratchRawCodes, kScratchRawOut, kScratchRawWork, kScratchRawList,
  kScratchFullTabs, kScratchFullOut, kScratchFullList,
  kScratchEstRoot, kScratchEstOut, kScratchEstNext,
  kScratchSplitStack, kScratchSplitOut, kScratchSplitCtl, kScratchSplitJobs, kScratchSplitCounts, kScratchSplitSurv,
  kScratchSlots
};
constexpr size_t kScratchKeep = (size_t)1 << 30;
constexpr long long kAltKeepNodes = 16LL << 20;  // a session's default frontier

// The call a slot belongs to.
inline int e13_scratch_call(int slot) {
  const int first[] = {kScratchCheckTapes, kScratchCraftTables, kScratchRawCodes, kScratchFullTabs, kScratchEstRoot,
                       kScratchSplitStack};
  int k = 0;
  while (k + 1 < (int)(sizeof first / sizeof first[0]) && slot >= first[k + 1]) ++k;
  return k;
}

// A slot's buffer of at least `bytes` (contents undefined), or null.
extern "C" void *e13_ctx_scratch(e13_ctx *c, int slot, size_t bytes);
// At the end of a call: gives back the slots above kScratchKeep.
extern "C" void e13_ctx_scratch_done(e13_ctx *c);

// Ends a call however it is left.
struct ScratchCall {
  e13_ctx *c;
  explicit ScratchCall(e13_ctx *ctx) : c(ctx) {}
  ~ScratchCall() { e13_ctx_scratch_done(c); }
  ScratchCall(const ScratchCall &) = delete;
  ScratchCall &operator=(const ScratchCall &) = delete;
};

// Whether a file's copy of the filter tables is uploaded (0: e13_estimate.cu).
extern "C" bool *e13_ctx_filter_tables(e13_ctx *c, int which);
