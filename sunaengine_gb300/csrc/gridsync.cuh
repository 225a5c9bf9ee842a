// What the 2D and 3D engines share around a substep's launch: the graph's refresh,
// the grid barrier of a cooperative launch and a CTA's prefix sum.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace sn {

// One captured substep. After a change the executable graph is updated where the
// topology allows it (a new scene size does), and made anew where it does not.
struct SubstepGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool valid = false;
  uint64_t launches = 0;  // of a substep
  ~SubstepGraph() { release(); }
  void release() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
    valid = false;
  }
  cudaError_t refresh(cudaGraph_t fresh, uint64_t substepLaunches) {
    if (exec) {
      cudaGraphExecUpdateResultInfo info;
      if (cudaGraphExecUpdate(exec, fresh, &info) != cudaSuccess) {
        cudaGetLastError();  // refused: not an error of the stream
        cudaGraphExecDestroy(exec);
        exec = nullptr;
      }
    }
    if (graph) cudaGraphDestroy(graph);
    graph = fresh;
    launches = substepLaunches;
    const cudaError_t e = exec ? cudaSuccess : cudaGraphInstantiate(&exec, graph, 0);
    valid = e == cudaSuccess;
    return e;
  }
};

constexpr int FU_T = 1024;  // threads of a fused substep's CTA, one CTA to an SM
constexpr uint32_t ERR_BARRIER = 8u;
constexpr long long BARRIER_WAIT_CYCLES = 1ll << 31;  // about a second
constexpr char BARRIER_TEXT[] = "a grid barrier timed out; results past it are not valid";

// The barrier of a cooperative launch: the arrivals' word (zero when the launch
// begins), where a wait that ran out is reported on the device and to the host
// (mapped memory), and how long a CTA waits.
struct GridBar {
  uint32_t *count, *err, *errHost;
  long long limit;
};

// Grid barrier of a cooperative launch: `target` counts the arrivals every CTA
// waits for (monotonic over the launch). A CTA that waits longer than the limit
// raises ERR_BARRIER; false sends the whole CTA out. Nobody passes a barrier that
// some CTA has not reached, so the others run out at the next one at the latest.
__device__ __forceinline__ bool grid_wait(const GridBar& bar, uint32_t& target) {
  __syncthreads();
  int bad = 0;
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar.count) : "memory");
    const long long t0 = clock64();
    for (;;) {
      uint32_t v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar.count) : "memory");
      if ((int32_t)(v - target) >= 0) break;
      if (clock64() - t0 > bar.limit) {
        atomicOr(bar.err, ERR_BARRIER);
        *(volatile uint32_t*)bar.errHost = ERR_BARRIER;
        bad = 1;
        break;
      }
    }
  }
  return __syncthreads_or(bad) == 0;
}

// Exclusive prefix of x[0, n) in place by the whole CTA, the total in x[n];
// returns the largest element (to every thread).
__device__ __forceinline__ uint32_t cta_scan(uint32_t* x, uint32_t n, uint32_t* ws) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t per = (n + FU_T - 1) / FU_T, lo = min(tid * per, n), hi = min(lo + per, n);
  uint32_t sum = 0, most = 0;
  for (uint32_t k = lo; k < hi; ++k) {
    sum += x[k];
    most = max(most, x[k]);
  }
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += v;
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 31) ws[warp] = inc;
  if (lane == 0) ws[32 + warp] = most;
  __syncthreads();
  uint32_t run = inc - sum;
  for (uint32_t w = 0; w < warp; ++w) run += ws[w];
  for (uint32_t k = lo; k < hi; ++k) {
    const uint32_t v = x[k];
    x[k] = run;
    run += v;
  }
  if (tid == FU_T - 1) x[n] = run;
  most = __reduce_max_sync(0xffffffffu, ws[32 + lane]);
  __syncthreads();
  return most;
}

// The places of a crowded cell's slots. tmp[lo, hi) holds the slots as they
// arrived; each becomes lo + the cell's lower slots, with RANKED set. Everywhere
// else a particle counts the lower slots of its cell by itself, which is
// quadratic in a cell that a wall or a hand has piled full; here the whole CTA
// sets one bit for each slot and counts bits below, `words` words of 32 slots, as
// many at a time as sh (shWords words) has room for. us a substep with one cell of
// p particles, counting / so: 2D, 40 k particles, p = 600 170 / 170, 1,100 181 / 171,
// 4,000 231 / 173, 36,000 813 / 213; 3D, 32 k, p = 600 89 / 66, 4,000 260 / 68, 30,000
// 1559 / 87 (there with the list's count cut short too). The line lies where they
// meet; the pass and its barrier cost about 3 us.
constexpr uint32_t RANKED = 0x80000000u;
constexpr uint32_t CELL_PILE = 512;
__device__ __forceinline__ void rank_pile(uint32_t* tmp, uint32_t lo, uint32_t hi, uint32_t words, uint32_t* sh,
                                          uint32_t shWords, uint32_t* ws) {
  const uint32_t tid = threadIdx.x, cap = (shWords - 1u) / 2u;
  uint32_t *bits = sh, *below = sh + cap, base = lo;
  for (uint32_t w0 = 0; w0 < words; w0 += cap) {
    const uint32_t n = min(cap, words - w0);
    for (uint32_t w = tid; w < n; w += FU_T) bits[w] = 0u;
    __syncthreads();
    for (uint32_t q = lo + tid; q < hi; q += FU_T) {
      const uint32_t s = tmp[q], w = (s >> 5) - w0;
      if (!(s & RANKED) && w < n) atomicOr(bits + w, 1u << (s & 31u));
    }
    __syncthreads();
    for (uint32_t w = tid; w < n; w += FU_T) below[w] = (uint32_t)__popc(bits[w]);
    __syncthreads();
    cta_scan(below, n, ws);
    for (uint32_t q = lo + tid; q < hi; q += FU_T) {
      const uint32_t s = tmp[q], w = (s >> 5) - w0;
      if (!(s & RANKED) && w < n)
        tmp[q] = RANKED | (base + below[w] + (uint32_t)__popc(bits[w] & ((1u << (s & 31u)) - 1u)));
    }
    base += below[n];
    __syncthreads();
  }
}
// f(t) for each thread t of the CTA whose `mine` is set, in turn and by the whole CTA.
template <class F>
__device__ __forceinline__ void each_pile(bool mine, uint32_t* mask, F f) {
  const uint32_t bal = __ballot_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31u) == 0u) mask[threadIdx.x >> 5] = bal;
  __syncthreads();
  for (uint32_t w = 0; w < FU_T / 32; ++w)
    for (uint32_t m = mask[w]; m; m &= m - 1u) f(w * 32u + (uint32_t)__ffs((int)m) - 1u);
  __syncthreads();
}

}  // namespace sn
