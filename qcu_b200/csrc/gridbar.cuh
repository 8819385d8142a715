// All-reduce, and with it a barrier, over the blocks of a cooperatively
// launched kernel.  Every block is resident, so every wait ends; the limit on
// the polls only bounds the damage of a logic error.
//
// A block stores its partial sums and counts itself in; one thread of each block
// watches the counter, and every block then sums all partials in block order.
// 2.1 us a reduction for 128 blocks (2 and 8 sums alike), against 3.3-4.0 us
// with a flag per block that one block collects and answers and 3.5-4.2 us when
// every block watches every other's; watching with acquiring loads, or two
// loads a turn, costs several us more.
// The counter goes on rising from launch to launch (modulo 2^32): nothing has
// to be reset, and launches of different sizes may follow one another.
//
// After a wait that gave up the counter says nothing any more, so `failed` stays
// set and every later launch on the state returns at once (grid_red_failed); the
// host looks at it with the next scalars it reads, ends the call with an error,
// and clears the state where a call begins (grid_red_reset).
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>

#include "reduce.cuh"

namespace qcu {

constexpr int GRID_RED_BLOCKS = 592;  // room for so many blocks (four an SM); a launch takes no more
constexpr int GRID_RED_VALUES = 8;    // sums of one reduction, at most
struct GridRed {
  unsigned count;  // arrivals
  unsigned base;   // arrivals of the launches before
  int failed;      // set when a wait gave up
  double part[2][GRID_RED_VALUES][GRID_RED_BLOCKS];
};
constexpr unsigned GRID_RED_POLLS = 1u << 21;  // a second or two

struct GridRedShared {
  double in[32][GRID_RED_VALUES];
  int ok;
};

// one thread of a block counts it in and waits until the counter has reached target
__device__ __forceinline__ int grid_arrive_wait(GridRed *g, unsigned target) {
  __threadfence();
  atomicAdd(&g->count, 1u);
  unsigned c, polls = 0;
  do {
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&g->count) : "memory");
    if (++polls >= GRID_RED_POLLS) {
      atomicExch(&g->failed, 1);
      return 0;
    }
  } while ((int)(c - target) < 0);
  __threadfence();
  return 1;
}

// whether a wait of an earlier launch on this state gave up: then the kernel
// returns before its first reduction (every thread of every block calls this)
__device__ __forceinline__ bool grid_red_failed(const GridRed *g) {
  return __syncthreads_or(*static_cast<const volatile int *>(&g->failed)) != 0;
}

// grid_allreduce without sums: a barrier (it takes an epoch like one)
__device__ __forceinline__ bool grid_barrier(GridRed *g, unsigned base, unsigned epoch, GridRedShared &sh) {
  __syncthreads();
  if (threadIdx.x == 0) sh.ok = grid_arrive_wait(g, base + epoch * gridDim.x);
  __syncthreads();
  return sh.ok != 0;
}

// The sums over the grid of v[0..N) of the threads of every `step`-th warp of
// each block (the others' are not looked at), into tot (shared memory, N
// values).  epoch: 1 for the kernel's first reduction, and so on; base: g->base
// as the kernel found it.  What any thread of any block wrote to global memory
// before the call can be read after it, with loads that go to L2 (__ldcg).
// False, in every thread of the block, when the wait gave up: the kernel returns.
template <int N>
__device__ __forceinline__ bool grid_allreduce(GridRed *g, unsigned base, unsigned epoch, double (&v)[N], int step,
                                               double *tot, GridRedShared &sh) {
  static_assert(N <= GRID_RED_VALUES, "");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (warp % step == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < N; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < N; k++) sh.in[warp][k] = v[k];
  }
  __syncthreads();
  if (warp == 0) {
    if (lane < N) {
      double q = 0.0;
      for (int w = 0; w < nw; w += step) q += sh.in[w][lane];
      __stcg(&g->part[epoch & 1][lane][blockIdx.x], q);
    }
    __syncwarp();
    if (lane == 0) sh.ok = grid_arrive_wait(g, base + epoch * gridDim.x);
  }
  __syncthreads();
  if (!sh.ok) return false;
  double q[N];  // value k by warp k % nw; a warp's loads and sums side by side
#pragma unroll
  for (int k = 0; k < N; k++) {
    q[k] = 0.0;
    if (k % nw == warp)
      for (int i = lane; i < gridDim.x; i += 32) q[k] += __ldcg(&g->part[epoch & 1][k][i]);
  }
#pragma unroll
  for (int k = 0; k < N; k++)
    if (k % nw == warp) {
      q[k] = warp_sum(q[k]);
      if (lane == 0) tot[k] = q[k];
    }
  __syncthreads();
  return true;
}

// by one thread of the grid, after its last reduction of the kernel
__device__ __forceinline__ void grid_red_end(GridRed *g, unsigned base, unsigned epochs) {
  g->base = base + epochs * gridDim.x;
}

// host: a state as before its first launch, in stream order
inline cudaError_t grid_red_reset(GridRed *g, cudaStream_t s) { return cudaMemsetAsync(g, 0, offsetof(GridRed, part), s); }
// QCU_BARRIER_GIVE_UP = `name` ("inner" or "coarse") leaves the state as a wait that
// gave up leaves it, before a launch: the host-side way the tests drive the error
inline cudaError_t grid_red_inject(GridRed *g, const char *name, cudaStream_t s) {
  const char *e = getenv("QCU_BARRIER_GIVE_UP");
  return e && strcmp(e, name) == 0 ? cudaMemsetAsync(&g->failed, 1, sizeof(int), s) : cudaSuccess;
}

}  // namespace qcu
