// e13_raw.cu -- the raw-simulator throughput set: whole tables run from the
// blank tape with no filter, at most max_steps steps each, stopping when the
// head leaves the 1364-cell window (steps (3)-(7) of src/e13search.c:163-175
// with the stage test and the deadline removed).
//
// Most random tables halt or leave the window within 1,300 steps; one in nine
// of 13 states loops in place to the limit, and these took 99 % of the steps.
// raw_kernel runs one machine per lane in the search's lock-step form for at
// most kRawSteps steps and lists the machines that live longer; raw_long_kernel
// runs each of those in a warp of its own, a tape word at a time
// (e13_macro.cuh), which leaves out whole turns of a repeated configuration.  A
// million machines of at most 2^18 steps, one B200: 132 ms in one kernel, now
// 4.9 ms and 19 ms (a call that returns totals 25 ms, one that copies the rows
// 28-31); the second is the time of the few machines that neither loop nor
// sweep (a counter in one word), 80 cycles a step.
#include <cuda_runtime.h>
#include <stdint.h>

#include "e13.h"
#include "e13_device.cuh"
#include "e13_macro.cuh"
#include "e13_scratch.h"

using namespace e13dev;

namespace {

constexpr int kRawBlock = 768;
constexpr int kRawSteps = 1024;           // steps before a machine is listed
constexpr long long kRawIntMax = 1 << 30; // longer limits are run in raw_kernel alone (its step counts are 64-bit)
constexpr int kRawLongBlock = 256;
constexpr int kRawLongPerSm = 3;          // 68 KB of shared memory a block
// 24 warps an SM with 512 visits each: the listed machines are many and short
// lived, so warps count for more than visits (a million machines with their
// rows, three seeds: 28-31 ms; 12 warps with 1024 visits 29-30, 6 with 2048
// 36-37).
typedef MacroMem<9> RawMem;

// Steps beyond kRawSteps from which the listed machines are better off in
// raw_long_kernel, which starts each of them anew and runs 3,552 at a time, than
// in the lanes that they have.  With 13 states the two take the same time at
// 230 steps for 500 machines, 435 for 20,000, 1480 for 100,000, 2900 for
// 200,000, 5000 for a million, 7200 for 4 million and 8000 for 16 million (a
// million: limit 2000 6.5 ms in lanes, 9.6 listed; limit 12,000 15.2 and 11.5);
// with two states, where fewer machines live, at 165, 310, 650, 1180, 4000,
// 6800 and 8700.
long long raw_list_from(long long n, int nq) {
  const long long by_count = n / 75 < 2200 + n / 400 ? n / 75 : 2200 + n / 400;
  return (200 + (by_count < 7500 ? by_count : 7500)) * (16 + nq) / 29;
}

__device__ __forceinline__ u64 splitmix_at(u64 seed, u64 k) {
  // draw k (1-based) of splitmix64 started at `seed`
  u64 z = seed + k * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ u32 raw_row(const unsigned char *__restrict__ codes, u64 seed, long long m, int nq, int s) {
  if (s >= nq) return kEntHalt | (kEntHalt << 16);
  u32 c0, c1;
  if (codes) {
    c0 = codes[m * 2 * nq + 2 * s];
    c1 = codes[m * 2 * nq + 2 * s + 1];
  } else {
    c0 = (u32)(splitmix_at(seed, (u64)(m * 2 * nq + 2 * s + 1)) % (u64)(4 * nq));
    c1 = (u32)(splitmix_at(seed, (u64)(m * 2 * nq + 2 * s + 2)) % (u64)(4 * nq));
  }
  if (c0 >= (u32)(4 * nq)) c0 = kEntHalt;
  if (c1 >= (u32)(4 * nq)) c1 = kEntHalt;
  return cell_slot(2 * s, c0, true) | (cell_slot(2 * s + 1, c1, true) << 16);
}

__device__ __forceinline__ void raw_result(long long *out, long long m, long long t, int status, int p, int ones) {
  out[4 * m] = t;
  out[4 * m + 1] = status;
  out[4 * m + 2] = p - kLeft;
  out[4 * m + 3] = ones;
}

struct RawWork {
  unsigned long long total, next_machine;  // steps; machines taken
  unsigned long long listed, taken;        // machines listed, and taken by raw_long_kernel
};

// Each lane takes its next machine from a global counter as soon as its
// current one ends, so long runs do not hold up lanes with short ones; every
// iteration is one step (or one run skip inside a word) for every lane.
__global__ void __launch_bounds__(kRawBlock) raw_kernel(const unsigned char *__restrict__ codes, u64 seed, long long n,
                                                         int nq, long long max_steps, long long park_steps,
                                                         long long *__restrict__ out, RawWork *__restrict__ work,
                                                         int *__restrict__ list) {
  extern __shared__ __align__(16) u32 raw_smem[];
  u32 *tape = raw_smem;                       // kTapeWords x kRawBlock
  u32 *rows = tape + kTapeWords * kRawBlock;  // 16 x kRawBlock
  __shared__ unsigned long long s_total;
  if (threadIdx.x == 0) s_total = 0;
  __syncthreads();
  const int stride = kRawBlock;
  u32 *tcol = tape + threadIdx.x;
  u32 *rcol = rows + threadIdx.x;
  unsigned long long my_steps = 0;
  long long m = -1;  // current machine
  int p = 0, st = 0;
  long long t = 0;
  for (;;) {
    if (m < 0) {
      m = (long long)atomicAdd(&work->next_machine, 1ull);
      if (m < n) {
        for (int w = 0; w < kTapeWords; ++w) tcol[w * stride] = 0;
        for (int s = 0; s < 16; ++s) rcol[s * stride] = raw_row(codes, seed, m, nq, s);
        p = kLeft;
        st = 0;
        t = 0;
      }
    }
    if (!__any_sync(0xFFFFFFFFu, m < n)) break;
    int status = -1;  // -1 still running
    if (m < n) {
      if (t >= park_steps) {
        status = t >= max_steps ? 0 : 3;
      } else {
        const int widx = (p >> 5) * stride;
        const u32 word = tcol[widx];
        const u32 sym = (word >> (p & 31)) & 1u;
        const u32 e = (rcol[st * stride] >> (sym << 4)) & 0x1FFu;
        if (e & kEntSpecial) {
          status = 2;
        } else {
          // k = 1, or on a self-loop cell the rest of the run inside this word
          const bool right = (e & 2u) != 0;
          const int b = p & 31;
          const u32 x = word ^ (0u - sym);
          const u32 xr = right ? x : __brev(x);
          const int bb = right ? b : 31 - b;
          const u32 up = xr >> bb;
          long long k = up ? __ffs(up) - 1 : 32 - bb;
          const long long left_steps = park_steps - t;
          const int room = right ? (kTapeCells - 2) - p : p - 1;
          k = k < left_steps ? k : left_steps;
          k = k < room ? k : room;
          k = ((e & kEntSelf) && k > 1) ? k : 1;
          if ((e ^ sym) & 1u) tcol[widx] = word ^ (1u << b);
          const int np = p + (int)(right ? k : -k);
          if ((unsigned)(np - 1) >= (unsigned)(kTapeCells - 2)) {
            status = 1;  // left the window: this step is not counted, as in run()
            p = np;
          } else {
            p = np;
            st = (int)((e >> 2) & 15u);
            t += k;
          }
        }
      }
      if (status == 3) {
        list[atomicAdd(&work->listed, 1ull)] = (int)m;
        m = -1;
      } else if (status >= 0) {
        if (out) {
          int ones = 0;
          for (int w = 0; w < kTapeWords; ++w) ones += __popc(tcol[w * stride]);
          raw_result(out, m, t, status, p, ones);
        }
        my_steps += (unsigned long long)t;
        m = -1;
      }
    }
    __syncwarp();
  }
  for (int o = 16; o > 0; o >>= 1) my_steps += __shfl_down_sync(0xFFFFFFFFu, my_steps, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_total, my_steps);
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(&work->total, s_total);
}

__global__ void __launch_bounds__(kRawLongBlock) raw_long_kernel(const unsigned char *__restrict__ codes, u64 seed,
                                                                 int nq, int max_steps, long long *__restrict__ out,
                                                                 RawWork *__restrict__ work,
                                                                 const int *__restrict__ list) {
  extern __shared__ __align__(16) unsigned char raw_long_smem[];
  const int lane = threadIdx.x & 31;
  RawMem &M = reinterpret_cast<RawMem *>(raw_long_smem)[threadIdx.x >> 5];
  const unsigned long long n = work->listed;
  unsigned long long steps = 0;
  for (;;) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(&work->taken, 1ull);
    k = __shfl_sync(kAll, k, 0);
    if (k >= n) break;
    const long long m = list[k];
    if (lane < 16) M.rows[lane] = raw_row(codes, seed, m, nq, lane);
    for (int w = lane; w < kTapeWords; w += 32) M.tape[w] = 0;
    macro_table(M, lane);
    Lane L;
    L.p = kLeft;
    L.st = 0;
    L.t = 0;
    L.deadline = max_steps - 1;
    u64 hb = 0;
    u32 reads = 0, ecell = 0;
    int cell = 0;
    const int ev = macro_run<false>(L, hb, M, KeyTabs(), nullptr, lane, reads, cell, ecell, 0ull);
    int ones = __popc(M.tape[lane]) + (lane + 32 < kTapeWords ? __popc(M.tape[lane + 32]) : 0);
    ones = __reduce_add_sync(kAll, ones);
    if (lane == 0) {
      steps += (unsigned long long)L.t;
      if (out) raw_result(out, m, L.t, ev == kEvDead ? 0 : ev == kEvOff ? 1 : 2, L.p, ones);
    }
    __syncwarp();
  }
  if (lane == 0 && steps) atomicAdd(&work->total, steps);
}

}  // namespace

struct e13_ctx;
extern "C" int e13_ctx_device(const e13_ctx *c);
extern "C" void e13_ctx_note_run(e13_ctx *c, double ms, long long launches);
extern "C" cudaStream_t e13_ctx_stream(const e13_ctx *c);

extern "C" int e13_raw_run(e13_ctx *ctx, const uint8_t *codes, uint64_t seed, int64_t n, int nq, int64_t max_steps,
                           int64_t *out, uint64_t *total_steps) {
  if (!ctx || n < 0 || nq < 1 || nq > 16 || max_steps < 0) return E13_ERR_ARG;
  if (n == 0) return E13_OK;
  if (cudaSetDevice(e13_ctx_device(ctx)) != cudaSuccess) return E13_ERR_CUDA;
  cudaStream_t s = e13_ctx_stream(ctx);
  unsigned char *d_codes = nullptr;
  long long *d_out = nullptr;
  RawWork *d_work = nullptr;
  int *d_list = nullptr;
  // the macro simulator counts steps in 32 bits and lists machines by int;
  // without room for the list (4 bytes a machine) the first kernel runs them all
  bool park = max_steps > kRawSteps + raw_list_from(n, nq) && max_steps <= kRawIntMax && n <= 0x7FFFFFFFLL;
  int rc = E13_OK;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  if (codes) d_codes = (unsigned char *)e13_ctx_scratch(ctx, kScratchRawCodes, (size_t)n * 2 * nq);
  if (out) d_out = (long long *)e13_ctx_scratch(ctx, kScratchRawOut, sizeof(long long) * 4 * (size_t)n);
  d_work = (RawWork *)e13_ctx_scratch(ctx, kScratchRawWork, sizeof(RawWork));
  if (park) d_list = (int *)e13_ctx_scratch(ctx, kScratchRawList, sizeof(int) * (size_t)n);
  park = d_list != nullptr;
  if ((codes && !d_codes) || (out && !d_out) || !d_work) rc = E13_ERR_CUDA;
  if (!rc) {
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e13_ctx_device(ctx));
    const size_t smem = (size_t)(kTapeWords + 16) * kRawBlock * 4;
    cudaFuncSetAttribute(raw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaEventRecord(e0, s);
    if (codes) cudaMemcpyAsync(d_codes, codes, (size_t)n * 2 * nq, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(d_work, 0, sizeof(RawWork), s);
    const long long need = (n + kRawBlock - 1) / kRawBlock;
    const int grid = (int)(need < (long long)nsm ? need : (long long)nsm);  // 177 KB of shared memory per CTA: one per SM
    raw_kernel<<<grid, kRawBlock, smem, s>>>(d_codes, seed, n, nq, max_steps, park ? kRawSteps : max_steps, d_out, d_work,
                                             d_list);
    if (park) {
      const size_t lsmem = sizeof(RawMem) * (kRawLongBlock / 32);
      cudaFuncSetAttribute(raw_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lsmem);
      raw_long_kernel<<<nsm * kRawLongPerSm, kRawLongBlock, lsmem, s>>>(d_codes, seed, nq, (int)max_steps, d_out, d_work,
                                                                        d_list);
    }
    if (cudaGetLastError() != cudaSuccess) rc = E13_ERR_CUDA;
    unsigned long long tot = 0;
    if (!rc && out) cudaMemcpyAsync(out, d_out, sizeof(long long) * 4 * (size_t)n, cudaMemcpyDeviceToHost, s);
    if (!rc) cudaMemcpyAsync(&tot, &d_work->total, sizeof tot, cudaMemcpyDeviceToHost, s);
    cudaEventRecord(e1, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) rc = E13_ERR_CUDA;
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    e13_ctx_note_run(ctx, ms, park ? 2 : 1);
    if (total_steps) *total_steps = tot;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  e13_ctx_scratch_done(ctx);
  return rc;
}
