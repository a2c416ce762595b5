// Pieces of the kernels that run every sweep of an iterative grid solve in one cooperative launch (Jacobi
// relaxation, the pseudo-field): the grid barrier between sweeps and each thread's walk over its items.
#pragma once

#include "qmt_common.cuh"

namespace qmt {

__device__ __forceinline__ uint64_t barrier_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long ld_acquire_gpu(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

constexpr unsigned long long kGaveUp = 1ull << 63;   // a wait ran out somewhere

// Waits (one thread) until *p, without its top bit, reaches `target`.  Gives up after wait_ns, raising
// *flag and the top bit of *p, or when another thread has raised that bit; returns false then.
__device__ __forceinline__ bool wait_count(unsigned long long* p, unsigned long long target, int* flag, uint64_t wait_ns) {
  uint64_t t0 = 0;
  for (uint32_t i = 0;; ++i) {
    const unsigned long long v = ld_acquire_gpu(p);
    if (v & kGaveUp) return false;
    if (v >= target) return true;
    if (wait_ns < 100000ull || (i & 15u) == 15u) {
      const uint64_t now = barrier_timer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > wait_ns) {
        atomicExch(flag, 1);
        atomicOr(p, kGaveUp);
        return false;
      }
    }
  }
}

// Grid barrier for a cooperative launch (all CTAs co-resident) on one counter, cleared before the
// launch: each CTA adds its arrival (released after its writes, which the CTA barrier ordered before) and
// polls until the arrivals of this round are in; `round` counts the CTA's barriers.  One atomic on its
// way and one poll on its way back, against a read of the generation, an arrival with its result, the
// release of the generation and a read of the give-up flag before (Jacobi 64^3 3.6 -> 2.6 us per sweep).
// False on every CTA, at this barrier or the next, once a wait ran out.
__device__ __forceinline__ bool grid_barrier(unsigned long long* count, unsigned long long& round, int* flag,
                                             unsigned nblocks, uint64_t wait_ns) {
  __shared__ int ok_s;
  __syncthreads();
  ++round;
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
    ok_s = wait_count(count, round * nblocks, flag, wait_ns);
  }
  __syncthreads();
  return ok_s != 0;
}

__device__ __forceinline__ float4 ldcg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }

// A thread's work items in a sweep: the grid-stride sequence tid, tid + nthreads, ... over
// items of w x ny x nz, as grid coordinates of the first item and of the stride, advanced by
// additions with carries -- no division per item (the stride is below w * ny * nz, so each
// carry needs one subtraction).  Set up once per launch.
struct GridWalk {
  int x, y, z;      // first item
  int sx, sy, sz;   // the stride
};

__device__ __forceinline__ GridWalk grid_walk(int width, int height, uint32_t nthreads, uint32_t tid) {
  const uint32_t w = (uint32_t)width, ny = (uint32_t)height;
  const uint32_t r = tid / w, rs = nthreads / w;
  return GridWalk{(int)(tid - r * w), (int)(r % ny), (int)(r / ny), (int)(nthreads - rs * w), (int)(rs % ny),
                  (int)(rs / ny)};
}

__device__ __forceinline__ void grid_step(const GridWalk& k, int w, int ny, int& x, int& y, int& z) {
  x += k.sx;
  if (x >= w) {
    x -= w;
    ++y;
  }
  y += k.sy;
  if (y >= ny) {
    y -= ny;
    ++z;
  }
  z += k.sz;
}

}  // namespace qmt
