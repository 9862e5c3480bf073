// e13_check.cu -- hash-free deep check of survivors on the device.
//
// Re-runs each machine from the blank tape to stage nmax and records, at every
// stage start, the exact set of ones left of cell -2 (the counter).  Stage
// starts are found without hashing, as src/recheck.c:61-92 does: state st0,
// head at head0 (abs) or head0 + 2^n - 2 (rel), and the ones at cells >= -2
// exactly the block -1 .. 2^n - 2.  Two variants:
//   E13_CHECK_RECHECK  recheck.c: limit t + 8*4^n + 1e5, tape +-4,000,000,
//                      stops at the first counter change (src/recheck.c:63-91)
//   E13_CHECK_DEEP     deep.c: limit t + 64*4^n + 1e5, tape -4096 .. 2^nmax+4096,
//                      off tape below -4094 or past 2^n + 2000 (src/deep.c:56-64)
//
// One machine per warp (e13_walk.cuh), one warp per CTA.  The tape is
// bit-packed; cells -4096 .. 2^nmax + 4096 (all of deep's tape, the busy part
// of recheck's) sit in shared memory, the rest of recheck's +-4M cells in HBM.
#include <cuda_runtime.h>

#include <mutex>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "e13.h"
#include "e13_scratch.h"
#include "e13_walk.cuh"

using namespace e13dev;

namespace {

typedef unsigned int u32;
typedef long long i64;

constexpr i64 kRecheckSide = 4000000;  // recheck's tape: cells -4e6 .. 4e6 (src/recheck.c:16-17)

struct CheckParams {
  int n, nmax, deep;
  int W;          // window words per lane: cells -4096 .. -4096 + 32W - 1
  i64 gwords;     // recheck: global tape words per machine (cells -4e6 .. 4e6)
  i64 gshift;     // global word index of window word 0
  u32 *gtapes;
  const e13_check_in *in;
  e13_check_out *out;
};

__device__ __forceinline__ int first_of_class(int n) { return n <= 2 ? 1 : (n <= 8 ? 3 : 9); }

// Shared memory of one machine: the remembered visits, the table, the window.
size_t check_smem(int W) { return (sizeof(uint4) << kWalkMemoBits) + sizeof(uint2) * 16 + sizeof(u32) * (size_t)W; }

// Words of the window for stage nmax: cells -4096 .. 2^nmax + 4096.
int window_words(int nmax) { return (int)((kWalkLeft + (1LL << nmax) + 4096 + 31) / 32 + 2); }

// Cell entry of a machine: bit 0 write, bit 1 right, bits 2..5 next, bit 7 not
// a move.
__device__ u32 check_code(const e13_check_in &in, int s, int a) {
  const int i = 2 * s + a;
  if (s >= in.nq || in.kind[i] != 0) return 0x80u;
  return (u32)(in.write[i] & 1) | (in.move[i] > 0 ? 2u : 0u) | ((u32)(in.next[i] & 15) << 2);
}

__global__ void __launch_bounds__(32) check_kernel(const CheckParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4 *memo = reinterpret_cast<uint4 *>(smem_raw);
  uint2 *act = reinterpret_cast<uint2 *>(memo + (1 << kWalkMemoBits));
  const int m = blockIdx.x, lane = threadIdx.x;
  WalkTape T;
  T.win = reinterpret_cast<u32 *>(act + 16);
  T.W = P.W;
  T.g = P.deep ? nullptr : P.gtapes + (i64)m * P.gwords;
  T.gshift = P.gshift;
  const e13_check_in &in = P.in[m];
  e13_check_out &o = P.out[m];
  for (int i = lane; i < (1 << kWalkMemoBits); i += 32) memo[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int w = lane; w < P.W; w += 32) T.win[w] = 0;
  reinterpret_cast<u32 *>(act)[lane] = act_word(check_code(in, lane >> 1, lane & 1), (u32)lane & 1u);
  __syncwarp();
  const bool deep = P.deep != 0;
  const i64 side = deep ? 0 : kRecheckSide;
  if (lane == 0) {
    o.status = E13_CHK_OK;
    o.fail_stage = 0;
    o.stages_done = 0;
    o.fail_t = 0;
    o.fail_head = 0;
  }
  Walker M{0, 0, 0, 0, 0};
  i64 t = 0;
  for (int n = 1; n <= P.nmax; ++n) {
    const int blk = 1 << n;
    const i64 limit = t + (deep ? 64LL : 8LL) * (1LL << (2 * n)) + 100000;
    const i64 at = in.rel ? in.head0 + blk - 2 : in.head0;
    // a head position that no allowed tape has stands for every one out of reach
    const int want = at > (1 << 29) || at < -(1 << 29) ? 1 << 29 : (int)at;
    const WalkStop S{blk, in.st0, want, want, false};
    M.left = limit - t;
    int sym = 0;
    const int ev = walk_run<false>(T, memo, act, lane, M, S, deep ? -4096 + 2 : (int)(-side + 3),
                                   deep ? blk + 2000 : (int)(side - 3), &sym);
    t = limit - M.left;
    if (ev != kWalkStop) {
      if (lane == 0) {
        int fail = ev == kWalkLimit ? E13_CHK_LIMIT : E13_CHK_OFFTAPE;
        if (ev == kWalkCell) {
          fail = in.kind[2 * M.st + sym] == 2 ? E13_CHK_FREE_READ : E13_CHK_HALT;
          o.free_state = M.st;
          o.free_sym = sym;
        }
        o.status = fail;
        o.fail_stage = n;
        o.fail_t = t;
        o.fail_head = M.head;
      }
      return;
    }
    // stage start n: record the counter (all ones at cells <= -3, from -3
    // down), a lane per word
    int cnt = 0, leftmost = 0;
    const int lowest = deep ? -4096 + 1 : M.minhead - 1;
    for (int top = kWalkZero - 1; top >= walk_word(lowest); top -= 32) {
      const int w = top - lane;
      u32 x = w >= walk_word(lowest) ? T.ld(w) : 0u;
      if (w == kWalkZero - 1) x &= ~kBlockBits;
      const int first = 32 * w - kWalkLeft;
      if (first < lowest) x &= 0xFFFFFFFFu << (lowest - first > 31 ? 31 : lowest - first);
      int before = __popc(x);
      const int own = before;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(kAll, before, d);
        if (lane >= d) before += v;
      }
      const int all = __shfl_sync(kAll, before, 31);
      int k = cnt + before - own;
      for (u32 y = x; y; ++k) {
        const int hb = 31 - __clz(y);
        y &= ~(1u << hb);
        if (k < E13_CHECK_MAX_ONES) o.ones_cells[n][k] = first + hb;
      }
      const u32 has = __ballot_sync(kAll, x != 0);
      if (has) {
        const int last = 31 - __clz(has);
        leftmost = __shfl_sync(kAll, x ? first + __ffs(x) - 1 : 0, last);
      }
      cnt += all;
    }
    __syncwarp();
    if (lane == 0) {
      o.stages_done = n;
      o.stage_t[n] = t;
      o.minhead[n] = M.minhead;
      o.nones[n] = cnt;
      o.leftmost[n] = leftmost;
    }
    if (!deep) {
      const int f = first_of_class(n);
      __syncwarp();
      if (n != f) {
        bool same = cnt == o.nones[f];
        const int k = min(cnt, E13_CHECK_MAX_ONES);
        for (int j = lane; j < k && same; j += 32) same = o.ones_cells[n][j] == o.ones_cells[f][j];
        if (!__all_sync(kAll, same)) return;  // recheck stops at the first counter change
      }
    }
  }
}

}  // namespace

struct e13_ctx;
extern "C" int e13_ctx_device(const e13_ctx *c);
extern "C" cudaStream_t e13_ctx_stream(const e13_ctx *c);

extern "C" int e13_check(e13_ctx *ctx, const e13_check_in *in, int n, int nmax, int mode, e13_check_out *out) {
  if (!ctx || (n > 0 && (!in || !out)) || n < 0 || nmax < 1 || nmax > E13_CHECK_MAX_NMAX ||
      (mode != E13_CHECK_RECHECK && mode != E13_CHECK_DEEP))
    return E13_ERR_ARG;
  if (n == 0) return E13_OK;
  if (cudaSetDevice(e13_ctx_device(ctx)) != cudaSuccess) return E13_ERR_CUDA;
  const bool deep = mode == E13_CHECK_DEEP;
  const int W = window_words(nmax);
  const size_t smem = check_smem(W);
  const i64 gwords = deep ? 0 : (2 * kRecheckSide + 1 + 31) / 32 + 2;
  const int chunk = deep ? n : (int)std::min<i64>(n, std::max<i64>(1, (4LL << 30) / (gwords * 4)));
  int rc = E13_OK;
  const cudaStream_t st = e13_ctx_stream(ctx);
  u32 *d_tapes = deep ? nullptr : (u32 *)e13_ctx_scratch(ctx, kScratchCheckTapes, (size_t)chunk * gwords * 4);
  e13_check_in *d_in = (e13_check_in *)e13_ctx_scratch(ctx, kScratchCheckIn, sizeof(e13_check_in) * (size_t)chunk);
  e13_check_out *d_out = (e13_check_out *)e13_ctx_scratch(ctx, kScratchCheckOut, sizeof(e13_check_out) * (size_t)chunk);
  if ((!deep && !d_tapes) || !d_in || !d_out) rc = E13_ERR_CUDA;
  if (!rc && cudaFuncSetAttribute(check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    rc = E13_ERR_CUDA;
  for (int b = 0; b < n && rc == E13_OK; b += chunk) {
    const int k = std::min(chunk, n - b);
    CheckParams P;
    P.n = k;
    P.nmax = nmax;
    P.deep = deep ? 1 : 0;
    P.W = W;
    P.gwords = gwords;
    P.gshift = (kRecheckSide - kWalkLeft) / 32;
    P.gtapes = d_tapes;
    P.in = d_in;
    P.out = d_out;
    if ((!deep && cudaMemsetAsync(d_tapes, 0, (size_t)k * gwords * 4, st) != cudaSuccess) ||
        cudaMemsetAsync(d_out, 0, sizeof(e13_check_out) * (size_t)k, st) != cudaSuccess ||
        cudaMemcpyAsync(d_in, in + b, sizeof(e13_check_in) * (size_t)k, cudaMemcpyHostToDevice, st) != cudaSuccess) {
      rc = E13_ERR_CUDA;
      break;
    }
    check_kernel<<<k, 32, smem, st>>>(P);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(out + b, d_out, sizeof(e13_check_out) * (size_t)k, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = E13_ERR_CUDA;
      break;
    }
  }
  e13_ctx_scratch_done(ctx);
  return rc;
}

// ------------------------------------------------------------------------
// The same check for callers that cannot allocate device memory.
//
// All device memory this entry point uses is fixed at load time: the tapes,
// inputs and outputs of up to E13_CHECK_NOALLOC_MAX machines sit in the
// file-scope arrays below (about 16 MB; every GPU that loads the library keeps
// them until the process exits).  Host code cannot use these names as device
// addresses, so the first call on each device looks the addresses up with
// cudaGetSymbolAddress while that device is current and keeps them.

namespace {

constexpr i64 kNoAllocWords = (2 * kRecheckSide + 1 + 31) / 32 + 2;  // one recheck tape (cells -4e6 .. 4e6)

static __device__ __align__(256) u32 g_noalloc_tapes[E13_CHECK_NOALLOC_MAX * kNoAllocWords];
static __device__ __align__(256) e13_check_in g_noalloc_in[E13_CHECK_NOALLOC_MAX];
static __device__ __align__(256) e13_check_out g_noalloc_out[E13_CHECK_NOALLOC_MAX];

constexpr int kNoAllocMaxDevices = 64;
// Per device, filled once under std::call_once: the arrays' device addresses
// and a non-blocking stream of this entry point's own, so a call waits for its
// own work only (not for other streams of the device, and not for a capture
// another thread holds on the legacy default stream).
struct NoAllocDevice {
  std::once_flag once;
  int rc;
  u32 *tapes;
  e13_check_in *in;
  e13_check_out *out;
  cudaStream_t stream;
};
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];

// With `device` current.
int noalloc_device(int device, NoAllocDevice **out) {
  if (device < 0 || device >= kNoAllocMaxDevices) return E13_ERR_ARG;
  NoAllocDevice &d = g_noalloc_dev[device];
  std::call_once(d.once, [&d]() {
    d.rc = E13_OK;
    if (cudaGetSymbolAddress((void **)&d.tapes, g_noalloc_tapes) != cudaSuccess ||
        cudaGetSymbolAddress((void **)&d.in, g_noalloc_in) != cudaSuccess ||
        cudaGetSymbolAddress((void **)&d.out, g_noalloc_out) != cudaSuccess ||
        cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking) != cudaSuccess)
      d.rc = E13_ERR_CUDA;
  });
  *out = &d;
  return d.rc;
}

}  // namespace

extern "C" int e13_check_noalloc(int device, const e13_check_in *in, int n, int nmax, int mode, e13_check_out *out) {
  if ((n > 0 && (!in || !out)) || n < 0 || nmax < 1 || nmax > E13_CHECK_MAX_NMAX ||
      (mode != E13_CHECK_RECHECK && mode != E13_CHECK_DEEP))
    return E13_ERR_ARG;
  if (n > E13_CHECK_NOALLOC_MAX) return E13_ERR_NOALLOC_SIZE;
  if (n == 0) return E13_OK;
  if (cudaSetDevice(device) != cudaSuccess) return E13_ERR_CUDA;
  NoAllocDevice *a = nullptr;
  int rc = noalloc_device(device, &a);
  if (rc) return rc;
  const cudaStream_t st = a->stream;
  const bool deep = mode == E13_CHECK_DEEP;
  const int W = window_words(nmax);
  const size_t smem = check_smem(W);
  if (cudaFuncSetAttribute(check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return E13_ERR_CUDA;
  // the arrays keep the previous call's contents: clear the tapes and outputs
  if ((!deep && cudaMemsetAsync(a->tapes, 0, sizeof(u32) * (size_t)n * kNoAllocWords, st) != cudaSuccess) ||
      cudaMemsetAsync(a->out, 0, sizeof(e13_check_out) * (size_t)n, st) != cudaSuccess ||
      cudaMemcpyAsync(a->in, in, sizeof(e13_check_in) * (size_t)n, cudaMemcpyHostToDevice, st) != cudaSuccess)
    return E13_ERR_CUDA;
  CheckParams P;
  P.n = n;
  P.nmax = nmax;
  P.deep = deep ? 1 : 0;
  P.W = W;
  P.gwords = deep ? 0 : kNoAllocWords;
  P.gshift = (kRecheckSide - kWalkLeft) / 32;
  P.gtapes = a->tapes;
  P.in = a->in;
  P.out = a->out;
  check_kernel<<<n, 32, smem, st>>>(P);
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(out, a->out, sizeof(e13_check_out) * (size_t)n, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return E13_ERR_CUDA;
  return E13_OK;
}
