// Grid-wide sums for kernels whose blocks are all resident (cooperative
// launches) and that need one or two sums per step of a device loop: the
// blocks exchange their partial sums as tagged 16-byte slots instead of
// passing a barrier and re-reading the partials.
//
// What bounds it: L2 round trips.  A counter barrier costs two dependent
// ones (1.25 us on 148 SMs) and the partials a third (2.1 us together); a
// slot {value, epoch} written and polled as one 16-byte access carries the
// value with its arrival (0.8 us up to 37 blocks).  With more blocks polling
// the same lines it gets slower (148 blocks: 3.1 us), so above kTagFlat
// blocks the sum goes in two levels: the blocks of a group poll one
// another's slots, then each block polls one block of every group.
#pragma once

#include "internal.cuh"

namespace b200la {

struct alignas(16) TagSlot {
  double v;
  unsigned long long tag;
};

constexpr int kTagFlat = 32;       // blocks that sum in one level
constexpr int kTagMaxBlocks = 512;  // 16 groups of up to 32 blocks
constexpr int kTagMaxVals = 2;
// polls before a wait gives up (a few seconds), as the grid barriers
constexpr int kTagSpin = 1 << 22;

// Device scratch of one solver: slots [2 levels][2 parities][kTagMaxVals][kTagMaxBlocks],
// zero at creation; `err` is set by a wait that ran out.
struct TagSync {
  TagSlot *slots;
  unsigned *err;
};
constexpr size_t kTagSlotBytes = sizeof(TagSlot) * 2 * 2 * kTagMaxVals * kTagMaxBlocks;

__device__ __forceinline__ void tag_store(TagSlot *p, double v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}

__device__ __forceinline__ unsigned long long tag_load(const TagSlot *p, double *v) {
  long long a;
  unsigned long long t;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(a), "=l"(t)
               : "l"(p)
               : "memory");
  *v = __longlong_as_double(a);
  return t;
}

// Warp 0 only: lane l < count polls slot[k * kTagMaxBlocks + index of lane l]
// until it carries `epoch`; v[k] becomes the sum over the lanes in a fixed
// order (all lanes).  False in every lane when a wait ran out.
template <int NV>
__device__ __forceinline__ bool tag_gather(const TagSlot *slot, int index, bool mine, unsigned long long epoch,
                                           unsigned *err, double (&v)[NV]) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  if (mine) {
    int spins = 0;
    for (;;) {
      double t[NV];
      bool all = true;
#pragma unroll
      for (int k = 0; k < NV; ++k) all &= tag_load(slot + k * kTagMaxBlocks + index, &t[k]) == epoch;
      if (all) {
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = t[k];
        break;
      }
      ++spins;
      if (spins > kTagSpin || ((spins & 255) == 0 && *(volatile unsigned *)err != 0u)) {
        atomicExch(err, 1u);
        ok = false;
        break;
      }
    }
  }
  ok = __all_sync(0xffffffffu, ok);
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
  return ok;
}

// Sums v[] over every thread of every block; the totals are returned in all
// threads, the same bits everywhere (fixed order).  `epoch` (> 0) grows by
// one per call in all blocks alike and never repeats over the life of the
// slots.  PUBLISH: global stores made before the call by any thread are
// visible after it to every thread (fences on both sides); without it the
// call orders only what depends on the summed values.
// A slot of epoch e is overwritten at e + 2 by a block that has completed
// e + 1, for which every block published e + 1, after it had read all its
// slots of e.  False in every thread of the block after a wait ran out.
template <int NV, bool PUBLISH>
__device__ __forceinline__ bool tag_sum(double (&v)[NV], const TagSync &ts, unsigned long long epoch) {
  __shared__ double red[NV][32];
  __shared__ double tot[NV];
  __shared__ int okf;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = warp_sum(v[k]);
    if (lane == 0) red[k][warp] = v[k];
  }
  __syncthreads();
  if (warp == 0) {
    const int B = (int)gridDim.x, b = (int)blockIdx.x;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = warp_sum(lane < nw ? red[k][lane] : 0.0);
    TagSlot *s1 = ts.slots + (epoch & 1) * (kTagMaxVals * kTagMaxBlocks);
    if (lane == 0) {
      if (PUBLISH) __threadfence();
#pragma unroll
      for (int k = 0; k < NV; ++k) tag_store(s1 + k * kTagMaxBlocks + b, v[k], epoch);
    }
    bool ok;
    if (B <= kTagFlat) {
      ok = tag_gather<NV>(s1, lane, lane < B, epoch, ts.err, v);
    } else {
      // groups of gs consecutive blocks, at most 32 groups
      int gs = 12;
      while (gs * 32 < B) ++gs;
      const int ng = (B + gs - 1) / gs, g = b / gs, r = b - g * gs;
      const int members = min(gs, B - g * gs);
      ok = tag_gather<NV>(s1, g * gs + lane, lane < members, epoch, ts.err, v);
      TagSlot *s2 = s1 + 2 * kTagMaxVals * kTagMaxBlocks;
      // what each lane's slot published goes on with this block's own slot:
      // every polling lane fences, then lane 0 stores after all of them
      if (PUBLISH) __threadfence();
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) tag_store(s2 + k * kTagMaxBlocks + b, v[k], epoch);
      }
      const int peer = lane * gs + min(r, B - lane * gs - 1);  // block r of group `lane`, or its last
      ok = tag_gather<NV>(s2, peer, ok && lane < ng, epoch, ts.err, v) && ok;
    }
    if (PUBLISH) __threadfence();
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) tot[k] = v[k];
      okf = ok ? 1 : 0;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = tot[k];
  const bool ok = okf != 0;
  // red/tot are rewritten by the next call only after its first barrier
  return ok;
}

}  // namespace b200la
