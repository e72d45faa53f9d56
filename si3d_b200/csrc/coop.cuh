// Helpers of the cooperative (grid-barrier) kernels: block sums in a fixed order, every-block
// reduction of block partials, and a counting grid barrier with a bounded wait.
//
// Every barrier wait is bounded: after kSpinLimit polls (or the barrier record's own limit) a block
// records SI3D_ETIMEOUT as the solve's ier, raises the barrier's abort flag and returns false; the
// other blocks see the flag at their next wait and return too, so a kernel built on it always ends.
#pragma once
#include "../../include/si3d_gpu.h"
#include "kernels.h"

namespace si3d {
namespace coop {

constexpr int QB = 256;                       // threads per block
constexpr long long kSpinLimit = 1LL << 23;   // polls (an L2 round trip each) before a wait gives up: > 2 s

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Block-wide sums of NV values at once (fixed order) over blocks of BS threads; the totals are
// returned in v[] in every thread.  sh holds (BS / 32) * NV + NV doubles.
template <int NV, int BS = QB>
__device__ __forceinline__ void bsum(double (&v)[NV], double* sh) {
  constexpr int NW = BS / 32;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  if (ln == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) sh[i * NW + w] = v[i];
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = 0;
#pragma unroll
    for (int q = 0; q < NW; ++q) t += sh[threadIdx.x * NW + q];
    sh[NW * NV + threadIdx.x] = t;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = sh[NW * NV + i];
  __syncthreads();
}

// Totals of NV partial arrays (n entries each, arrays `stride` apart), in every thread.
template <int NV, int BS = QB>
__device__ __forceinline__ void all_partials(const double* part, int n, int stride, double (&v)[NV], double* sh) {
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = 0;
  for (int j = threadIdx.x; j < n; j += BS) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += __ldcg(part + i * stride + j);
  }
  bsum<NV, BS>(v, sh);
}

// Per-block state of the grid barrier, in shared memory: the outcome of the last wait, the
// number of barriers this block has passed, and, read at the first barrier of the launch, the
// arrivals a barrier waits for and the poll limit.  Zero `epoch` (thread 0) before the first
// barrier.
struct BarSt {
  int ok;
  unsigned int epoch;
  unsigned int expect;
  long long limit;
};

__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Grid barrier on a monotonic arrival counter: barrier e (1, 2, ...) of the launch is passed once
// the counter reaches e * (nblocks + absent), nblocks being the blocks that share this barrier
// record (the whole grid, or one basin's share of an ensemble launch).  An arrival is one release-add (no round trip, no
// reset; the release orders the block's writes, which __syncthreads ordered before thread 0's
// arrival, ahead of it); the wait polls with acquire loads, which order the block's later reads
// after the other blocks' arrivals.  `absent` and `limit` (zero in every solve; a test sets them
// to make the wait run out) are read once, at the first barrier, so a barrier costs one release
// and the polls.  Bounded: returns false (in every thread of the block) once this block gave up
// or any block has.
__device__ __forceinline__ bool grid_barrier(GridBar* bar, PcgScal* sc, BarSt* st, unsigned int nblocks) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (st->epoch == 0) {
      st->expect = nblocks + __ldcg(&bar->absent);
      const unsigned long long lim = __ldcg(&bar->limit);
      st->limit = lim ? (long long)lim : kSpinLimit;
    }
    int ok = 1;
    const unsigned long long target = (unsigned long long)(++st->epoch) * st->expect;
    const long long limit = st->limit;
    red_release_add(&bar->count, 1ull);
    long long spins = 0;
    while (ld_acquire64(&bar->count) < target) {
      if (++spins > limit || ((spins & 15) == 0 && ld_acquire(&bar->abort) != 0u)) { ok = 0; break; }
    }
    if (!ok && atomicExch(&bar->abort, 1u) == 0u) {
      sc->ier = SI3D_ETIMEOUT;
      sc->done = 1;
      __threadfence();
    }
    st->ok = ok;
  }
  __syncthreads();
  return st->ok != 0;
}

__device__ __forceinline__ bool grid_barrier(GridBar* bar, PcgScal* sc, BarSt* st) {
  return grid_barrier(bar, sc, st, gridDim.x);
}

// ---------------------------------------------------------------- all-gather barrier
// A grid barrier that carries the block sums: every block stores its values, tagged with the
// barrier's number, into its own slots, and the first warps of every block poll all slots and add
// the values in an order that is the same in every block.  One L2 round trip for the store and
// one for the poll, where a counting barrier followed by a reduction of block partials takes an
// atomic, a poll and a dependent load.  What the polling costs depends on when it starts and what
// it reads: a poll that arrives before the other blocks' stores slows those stores down.  Measured
// with 148 blocks of 512 threads, the block's own sums included, in SM cycles: counting barrier
// 3690; all slots polled at once until the last has arrived 4780; the missing slots only, from 300
// cycles after the own store on, 16 bytes apart, 2300 (2060 with up to 64 blocks).
//
// A value travels as {low word, tag, high word, tag}: each 8-byte half carries its own tag, so a
// reader that sees both tags has both words whatever the width the hardware moves them in.  The
// slots are double-buffered by the barrier's parity: a block writes barrier e + 2's slot only after
// barrier e + 1, which every block reaches after it has read barrier e.  Tags count up from 1 in a
// launch and the slots are zeroed before it.  REL: the block's earlier global writes are visible
// to the other blocks after the barrier; without it only the values are exchanged.  With REL the
// arrival goes through the barrier record's counter (one release-add, acquire polls by one thread)
// and the values are read from the slots after it: releasing through the slots, with a fence before
// the store and after the poll, took 4400 to 6600 cycles with 148 blocks, the counter 2600.
constexpr int kSlotVals = 2;                     // values per slot and parity
constexpr int kPollDelay = 300;                  // cycles from the own store to the first poll

struct SlotBar {
  uint4* slots;              // [parity][value][block]
  GridBar* bar;
  int bid;                   // this block among the blocks that share the slots
  int nslots;                // blocks to wait for (plus the test hook's absent ones)
  int plane;                 // entries of one (parity, value) plane
  unsigned int epoch;        // exchanges passed (the same in every thread)
  unsigned int counted;      // those that went through the counter
  long long limit;
};

// uint4 entries that a barrier over nblocks blocks needs: the planes hold the blocks that the
// wait-limit test hook asks for beyond the grid (never written) as well.
__host__ __device__ constexpr int slot_plane(int nblocks) { return nblocks + 1024; }
__host__ __device__ constexpr size_t slot_count(int nblocks) { return 2 * kSlotVals * (size_t)slot_plane(nblocks); }

// `most`: the blocks the slots were laid out for.
__device__ __forceinline__ SlotBar slot_bar(GridBar* bar, uint4* slots, int bid, int nb, int most) {
  const unsigned long long lim = __ldcg(&bar->limit);
  return SlotBar{slots, bar, bid, nb + (int)__ldcg(&bar->absent), slot_plane(most), 0u, 0u,
                 lim ? (long long)lim : kSpinLimit};
}

__device__ __forceinline__ uint4 ld_slot(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_slot(uint4* p, double v, unsigned int tag) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(p), "r"(__double2loint(v)), "r"(tag),
               "r"(__double2hiint(v)) : "memory");
}

__device__ __forceinline__ void wait_cycles(int n) {
  const long long t0 = clock64();
  while (clock64() - t0 < n) {}
}

// One arrival on the counter and the wait for everyone's (thread 0): releases the block's writes, acquires
// the others'.
__device__ __forceinline__ int count_wait(const SlotBar& B) {
  const unsigned long long target = (unsigned long long)B.counted * (unsigned int)B.nslots;
  red_release_add(&B.bar->count, 1ull);
  long long spins = 0;
  while (ld_acquire64(&B.bar->count) < target)
    if (++spins > B.limit || ((spins & 15) == 0 && ld_acquire(&B.bar->abort) != 0u)) return 0;
  return 1;
}

// The outcome of a wait, in every thread; the first block to give up raises the abort flag.
__device__ __forceinline__ bool bar_ok(int failed, const SlotBar& B, PcgScal* sc) {
  if (!failed) return true;
  if (threadIdx.x == 0 && atomicExch(&B.bar->abort, 1u) == 0u) {
    sc->ier = SI3D_ETIMEOUT;
    sc->done = 1;
    __threadfence();
  }
  return false;
}

// Sums of v[] over all threads of all blocks, in every thread.  sh: 2 * kSlotVals * NT / 32 doubles,
// the totals behind the warps' sums for every NV (a slow thread may still read them while the next
// call stores its warps' sums).  Each polling warp takes 32 slots; `mid(first, count)` runs in the
// other warps (this thread being `first` of `count`) between the block's arrival and the end of the
// wait, and returns false to make the barrier fail.
// Bounded as grid_barrier: false once this block or any other gave up.
template <int NV, bool REL, int NT, typename Mid>
__device__ __forceinline__ bool gather_sum(double (&v)[NV], SlotBar& B, PcgScal* sc, double* sh, Mid&& mid) {
  constexpr int NW = NT / 32;
  static_assert(NV <= kSlotVals && NW <= 32 && NW >= 2, "slot layout");
  double* const tot = sh + kSlotVals * NW;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  if (ln == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) sh[i * NW + w] = v[i];
  }
  __syncthreads();
  ++B.epoch;
  if (REL) ++B.counted;
  const int pw = REL ? 1 : min(NW - 1, (B.nslots + 31) >> 5);   // polling warps
  int ok = 1;
  if (w < pw) {
    double a[NV];
    uint4* const mine = B.slots + (size_t)(B.epoch & 1) * kSlotVals * B.plane;
    if (w == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        a[i] = ln < NW ? sh[i * NW + ln] : 0.0;
        for (int o = 16; o > 0; o >>= 1) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
      }
      if (B.nslots > 1 && ln == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) st_slot(mine + i * B.plane + B.bid, a[i], B.epoch);
        if (REL) ok = count_wait(B);
      }
      if (REL) ok = __shfl_sync(0xffffffffu, ok, 0);
    } else {
      wait_cycles(kPollDelay);   // the first warp's reduction of the block's sums
    }
    if (B.nslots > 1) {
      if (!REL) wait_cycles(kPollDelay);
#pragma unroll
      for (int i = 0; i < NV; ++i) a[i] = 0.0;
      long long spins = 0;
      for (int s = w * 32 + ln; s < B.nslots && ok; s += 32 * pw) {
        uint4 e[NV];
        for (;;) {
          bool got = true;
#pragma unroll
          for (int i = 0; i < NV; ++i) e[i] = ld_slot(mine + i * B.plane + s);
#pragma unroll
          for (int i = 0; i < NV; ++i) got = got && e[i].y == B.epoch && e[i].w == B.epoch;
          if (got) break;
          if (++spins > B.limit || ((spins & 15) == 0 && ld_acquire(&B.bar->abort) != 0u)) { ok = 0; break; }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) a[i] += __hiloint2double((int)e[i].z, (int)e[i].x);
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < NV; ++i)
        for (int o = 16; o > 0; o >>= 1) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
    }
    if (ln == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) tot[i * NW + w] = a[i];
    }
  } else if (!mid((int)threadIdx.x - 32 * pw, NT - 32 * pw)) {
    ok = 0;
  }
  if (!bar_ok(__syncthreads_or(!ok), B, sc)) return false;
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = tot[i * NW];
  for (int q = 1; q < pw; ++q) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += tot[i * NW + q];
  }
  return true;
}

template <int NV, bool REL, int NT>
__device__ __forceinline__ bool gather_sum(double (&v)[NV], SlotBar& B, PcgScal* sc, double* sh) {
  return gather_sum<NV, REL, NT>(v, B, sc, sh, [](int, int) { return true; });
}

}  // namespace coop
}  // namespace si3d
