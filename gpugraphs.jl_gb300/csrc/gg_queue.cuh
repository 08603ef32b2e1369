// gg_queue.cuh -- queue appends of the searches, grid barrier of the persistent ones.
//
// A frontier queue has one length counter, and atomics on one address pass L2 one after
// another (about 0.5 ns each on GB300).  One atomic per warp instruction that appends
// anything therefore bounded whole levels: R-MAT scale 24 issues about a million of
// them in one bottom-up BFS level, a 128-graph shortest-path call 24 million.  A warp
// here stages its appends in its own slice of shared memory (the count is a register:
// no atomic at all) and takes queue space once per ~100 entries.  With the wider loads
// made in the same step a scale-24 BFS went from 3.00 to 0.66 ms, a scale-22 Int32
// shortest-path search from 2.86 to 2.27 ms.
#pragma once

#include <stdint.h>

namespace gg {

struct WarpQueue {
  static const int kCap = 128;  // entries staged per warp: 512 bytes, 32 KB on a full SM
  int32_t* buf;
  int32_t* q;
  unsigned long long* len;
  int n;

  __device__ __forceinline__ WarpQueue(int32_t* warp_buf, int32_t* queue, unsigned long long* length)
      : buf(warp_buf), q(queue), len(length), n(0) {}

  // appends v of the lanes with `want`; the whole warp calls
  __device__ __forceinline__ void push(bool want, int32_t v) {
    const unsigned b = __ballot_sync(0xffffffffu, want);
    if (!b) return;
    if (want) buf[n + __popc(b & ((1u << (threadIdx.x & 31)) - 1u))] = v;
    n += __popc(b);
    if (n > kCap - 32) flush();
  }

  // writes the staged entries out; every warp calls it once more before it ends
  __device__ __forceinline__ void flush() {
    if (n == 0) return;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(len, (unsigned long long)n);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int i = lane; i < n; i += 32) q[base + i] = buf[i];
    __syncwarp();
    n = 0;
  }
};

// adds every lane's v into *out with one atomic per warp (none when the sum is 0)
__device__ __forceinline__ void warp_add(unsigned long long v, unsigned long long* out) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

// Grid barrier, the part of thread 0 of every block (between two block barriers): the
// arrival counter bar[0] only grows and `target` is its value once every block arrived
// (blocks x barriers so far, compared modulo 2^32), so one arrival and the polls of one
// word are all the traffic.  The wait is bounded by `limit` polls; running out sets the
// error word bar[2], which the waiting blocks look at every 16 polls.
__device__ __forceinline__ bool coop_leader_sync(unsigned* bar, unsigned target,
                                                 unsigned long long limit) {
  __threadfence();
  atomicAdd(bar, 1u);
  unsigned long long polls = 0;
  for (;;) {
    unsigned a;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(bar) : "memory");
    if ((int)(a - target) >= 0) return true;
    if (++polls > limit) {
      atomicExch(bar + 2, 1u);
      return false;
    }
    if ((polls & 15) == 0 && *((volatile unsigned*)(bar + 2))) return false;
  }
}

}  // namespace gg
