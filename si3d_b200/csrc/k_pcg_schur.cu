// The MIC-CG iteration of the zeta solve (stopping test 5) on the black unknowns alone.
//
// In red-black order A = [D, -C; -C^T, D_B] with D and D_B diagonal, and MIC(0)'s red pivots are D
// itself, so M - A is zero outside the black diagonal block.  It follows that (A z)_R = r_R whenever
// z = M^-1 r, hence q_R = A p's red part is c r0_R and r_R is rho r0_R throughout the iteration (r0
// the first residual, c and rho scalars), and with t = r_B + C^T D^-1 r_R (the residual of the
// Schur complement S = D_B - C^T D^-1 C) the black parts obey
//     z_B = P^-1 t,   p_B = z_B + beta p_B,   t -= alpha S p_B,   u_B += alpha p_B
// with P the black MIC pivots, and the scalars of the full iteration are
//     (r, z) = t . z_B + rho^2 gamma,         gamma = r0_R . D^-1 r0_R,
//     (p, q) = p_B . S p_B + c^2 gamma,       c = rho + beta c,   rho -= alpha c,
//     (r, r) = |t - rho g|^2 + rho^2 delta,   g = C^T D^-1 r0_R,  delta = r0_R . r0_R.
// These are the alpha, beta, stopping values and iterates of the two-colour loop
// (k_pcg_persistent.cu), node for node, in exact arithmetic; the red solution follows at the end
// from D u_R = b_R - rho r0_R + C u_B.  S couples a black node to the eight black nodes at distance
// two (nine coefficients a node, formed once per solve).
//
// What that buys: half the vectors, and two grid-wide exchanges an iteration instead of three, both
// all-gather barriers that carry the dot products (coop.cuh).  A block owns consecutive black nodes
// and keeps their coefficients, neighbour indices and vectors in shared memory for the whole solve.
// Three forms share the arithmetic (the values are the same, bit for bit):
//   window  p of the block's nodes and of the `reach` nodes before and after them is in shared
//           memory (reach: the largest index distance of two coupled nodes), so S p reads shared
//           memory only.  A block publishes z as tagged words that carry their own arrival, like
//           the barrier's slots; the neighbours form the halo's p = z + beta p themselves.  No
//           fence is needed in the iteration.
//   stream  for blocks whose window does not fit or whose halo is long: z and p go through L2, with fences
//           at the exchange that follows their writes.
//   cluster the window form for up to eight blocks: one thread-block cluster, whose blocks exchange
//           sums and z through each other's shared memory, behind the cluster's barrier; a block has
//           at most one node a thread, with its coefficients in registers.  3924 unknowns, four
//           blocks: 4.5 -> 2.8 us an iteration.
// Nodes beyond the shared-memory capacity keep their coefficients and vectors in global scratch.
// The solve is bound by the latency of the two exchanges (about 1.2 us each) and of the FP64 chains
// between them until a block holds about a thousand nodes.  Time of an iteration, two-colour loop ->
// this loop: 3924 unknowns 13.0 -> 2.8 us, 129155 (FP32 inner solves) 13.3 -> 6.2 us with the
// refinement around them, 350000 16.9 -> 5.9 us.
#include <algorithm>
#include <type_traits>

#include "../../include/si3d_gpu.h"
#include "common.cuh"
#include "coop.cuh"
#include "kernels.h"

namespace si3d {

namespace {

using namespace coop;

constexpr int SB = 512;    // threads per block (one block per SM), in every launch: a basin's sums depend on
                           // the number of its blocks alone
constexpr int RN = 3;      // nodes of a thread whose vectors are in registers (1536 of a block)
constexpr int kSmemMax = 225 * 1024;
constexpr int kClusterMax = 8;   // blocks of a cluster (the portable limit)

// Shared memory of a node: nine coefficients and eight neighbours (16-bit in the window form).  The
// vectors of a thread's first RN nodes are in its registers, those of later nodes in global memory.
template <typename T, bool WIN>
__host__ __device__ constexpr int node_bytes() {
  return 9 * (int)sizeof(T) + 8 * (int)(WIN ? sizeof(unsigned short) : sizeof(int));
}
// Bytes of the window of a block with `per` nodes (a zero entry for absent neighbours at its end,
// then the halo's z).
template <typename T>
__host__ __device__ constexpr long long window_bytes(int per, int reach) {
  return ((long long)per + 4LL * reach + 1 + 3) / 4 * 4 * (long long)sizeof(T);
}
// The window form runs when the window leaves room for at least a quarter of the block's nodes
// (a block of 512 threads then still reads most of a phase's data from shared memory), its
// entries fit 16-bit indices, and the halo is short: its words are polled one after the other by each
// thread, some 1.5 us an iteration for every thousand nodes of reach, where the stream form pays for its
// fences and for reading z and p of the eight neighbours through L2.  Basins that are long along the
// numbering's fast index have a long reach.  Window / stream, us an iteration in FP64 and FP32 (the
// latter with the refinement around it), by reach and nodes a block:
//   1000,  500: 4.5 / 5.3 and 7.0 / 7.4     2000,  500: 6.7 / 5.7 and 9.0 / 7.7     2000, 640: 8.0 / 9.7, 10.5 / 10.0
//   1500, 1440: 8.8 / 11.4, 11.2 / 12.5     2000, 3200: 19.9 / 22.7, 20.7 / 22.2
//   4000,  500: 8.9 / 5.6 and 11.0 / 7.8    4000, 1280: 12.4 / 11.6, 14.7 / 10.9    4000, 2570: 18.8 / 18.6, 19.7 / 18.0
//   8000,  770: - / 11.9 and 20.6 / 10.3
// One block alone has no halo.
template <typename T>
__host__ __device__ inline bool window_fits(int per, int nb, int reach) {
  const long long w = window_bytes<T>(per, reach);
  const bool near = nb == 1 || (reach <= 3000 && 4LL * reach <= 13LL * per);
  return near && per + 2LL * reach + 1 < 65536 && w + (long long)node_bytes<T, true>() * (per / 4) <= kSmemMax;
}

// z of one node as a tagged word: every 8-byte part carries the tag (coop.cuh's slots).
__device__ __forceinline__ void put_z(uint4* zt, int j, double z, unsigned int tag) { st_slot(zt + j, z, tag); }
__device__ __forceinline__ void put_z(uint4* zt, int j, float z, unsigned int tag) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(reinterpret_cast<uint2*>(zt) + j),
               "r"(__float_as_uint(z)), "r"(tag) : "memory");
}
__device__ __forceinline__ bool get_z(const uint4* zt, int j, double& z, unsigned int tag) {
  const uint4 v = ld_slot(zt + j);
  z = __hiloint2double((int)v.z, (int)v.x);
  return v.y == tag && v.w == tag;
}
__device__ __forceinline__ bool get_z(const uint4* zt, int j, float& z, unsigned int tag) {
  uint2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y)
               : "l"(reinterpret_cast<const uint2*>(zt) + j) : "memory");
  z = __uint_as_float(v.x);
  return v.y == tag;
}

// Sums of v[] over all threads of the cluster's nb <= kClusterMax blocks, in every thread, in the order of
// gather_sum (the same bits).  A block leaves its sums in its shared memory (tot: [2][kSlotVals], used in
// turn), and after the cluster's barrier every warp reads all blocks'.  (Every warp reading the sums of
// all warps of all blocks spares a reduction before the barrier, but reading other blocks' shared
// memory is what takes the time: 925 us instead of 818 for 294 iterations.)  `then` loads what else
// the barrier ordered.  The barrier also orders the shared and global memory of the blocks.  It needs no
// limit: the blocks of a cluster run together, and all of them take the same path through the loop.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned int in_block(const void* p, int block) {   // p's address in another block
  unsigned int a = (unsigned int)__cvta_generic_to_shared(p);
  asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(block));
  return a;
}
__device__ __forceinline__ void ld_block(const double* p, int block, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(in_block(p, block)) : "memory");
}
__device__ __forceinline__ void ld_block(const float* p, int block, float& v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(in_block(p, block)) : "memory");
}
template <int NV, typename Then>
__device__ __forceinline__ void cluster_sum(double (&v)[NV], int nb, int& turn, double* sh, double* tot, Then&& then) {
  constexpr int NW = SB / 32;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  }
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  if (ln == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) sh[i * NW + w] = v[i];
  }
  __syncthreads();
  double* const mine = tot + turn * kSlotVals;
  turn ^= 1;
  if (w == 0) {
    double a[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) a[i] = ln < NW ? sh[i * NW + ln] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < NV; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
    }
    if (ln == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) mine[i] = a[i];
    }
    __syncwarp();
  }
  cluster_barrier();
  const int b = ln & (kClusterMax - 1);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = 0.0;
    if (b < nb) ld_block(mine + i, b, v[i]);
  }
  then();
#pragma unroll
  for (int o = kClusterMax / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  }
}

// One system, solved by the nb blocks that share `bar` and P.slots, this one being block bid; CL: by the
// nb blocks of a cluster (window form, ONE), which exchange sums and z through each other's shared
// memory.  ONE: at most one node a thread, all of the block's in shared memory (window form); its
// coefficients are read from registers, which takes 630 instead of 1180 cycles for S p of 491 nodes
// (129,155 unknowns in FP32, 436 nodes a block: 2.81 -> 2.60 ms of solves a step).
template <typename T, bool WIN, bool ONE, bool CL = false>
__device__ __forceinline__ void schur_body(const PcgDevT<T>& P, GridBar* bar, int bid, int nb, int smem) {
  constexpr int RK = ONE ? 1 : RN;
  using Idx = typename std::conditional<WIN, unsigned short, int>::type;
  extern __shared__ double dyn[];
  __shared__ double sh[2 * kSlotVals * SB / 32];
  __shared__ double s_tot[2 * kSlotVals];
  const PcgColorT<T> &R = P.R, &B = P.B;
  PcgScal* SC = P.sc;
  if (SC->done != 0) return;
  const int nB = B.n, per = (nB + nb - 1) / nb, reach = P.reach;
  const int lo = min(bid * per, nB), n = min(per, nB - lo);
  const int wbytes = WIN ? (int)window_bytes<T>(per, reach) : 0;
  const int zbytes = CL ? per * (int)sizeof(T) : 0;
  const int cap = ((smem - wbytes - zbytes) / node_bytes<T, WIN>()) & ~1, nres = min(n, cap);
  // window entry of global node o: o - w0; entry wz is zero
  T* const s_w = reinterpret_cast<T*>(dyn);
  const int w0 = lo - reach, wz = per + 2 * reach;
  T* const s_h = s_w + wz + 1;   // z of the halo nodes
  T* const s_cf = reinterpret_cast<T*>(reinterpret_cast<char*>(dyn) + wbytes);   // [9][cap]
  Idx* const s_nb = reinterpret_cast<Idx*>(s_cf + 9 * cap);                      // [8][cap]
  T* const s_z = reinterpret_cast<T*>(s_nb + 8 * cap);                           // CL: [per]
  T rt[RK], ru[RK], rv[RK], rg[RK], rd[RK], rp[RK];   // t, u, S p, g, 1 / pivot, p
  const int i0 = threadIdx.x, it = i0 + RK * SB;      // first node, first node past the registers
  const int hl = min(reach, lo), hr = min(reach, nB - lo - n);                   // halo nodes before and after
  SlotBar bs{};
  if (!CL) bs = slot_bar(bar, P.slots, bid, nb, P.slot_blocks);
  int turn = 0;
  T* const z = B.z;
  unsigned int tag = 1;
  // z of the halo nodes into shared memory, by the warps that do not poll the barrier, while it waits
  auto fetch_halo = [&](int first, int count) -> bool {
    if (!WIN) return true;
    wait_cycles(kPollDelay);
    for (int h = first; h < hl + hr; h += count) {
      const int o = h < hl ? lo - hl + h : lo + n + (h - hl);
      T zo;
      long long spins = 0;
      while (!get_z(P.zt, o, zo, tag))
        if (++spins > bs.limit || ((spins & 15) == 0 && ld_acquire(&bar->abort) != 0u)) return false;
      s_h[h] = zo;
    }
    return true;
  };
  // The same from the blocks of the cluster, by the threads that will use it: a thread's first in a
  // register, so that only its use waits for the load.
  T zh = (T)0;
  const int ho = (int)threadIdx.x < hl ? lo - hl + (int)threadIdx.x : lo + n + ((int)threadIdx.x - hl), hb = ho / per;
  auto cluster_halo = [&]() {
    if ((int)threadIdx.x < hl + hr) ld_block(s_z + (ho - hb * per), hb, zh);
    for (int h = threadIdx.x + SB; h < hl + hr; h += SB) {
      const int o = h < hl ? lo - hl + h : lo + n + (h - hl), b = o / per;
      ld_block(s_z + (o - b * per), b, s_h[h]);
    }
  };
  auto nothing = [] {};
  // ---- the Schur complement's rows, g and t = r_B + g of this block's nodes
  double v2[2] = {0.0, 0.0}, w2[2] = {0.0, 0.0};
  auto row = [&](int i, T& rt_, T& ru_, T& rg_, T& rd_) {
    const int j = lo + i;
    const int4 q = B.nbr[j];
    const T aW = R.sx[q.x], aS = R.sy[q.y], aN = B.sy[j], aE = B.sx[j];
    constexpr bool F32 = std::is_same<T, float>::value;
    double dW, dS, dN, dE;   // 1 / diagonal of the red neighbours
    if constexpr (!F32) { dW = R.dinv[q.x]; dS = R.dinv[q.y]; dN = R.dinv[q.z]; dE = R.dinv[q.w]; }
    const int nR = R.n;
    const int4 none = make_int4(nB, nB, nB, nB);
    const int4 kW = q.x < nR ? R.nbr[q.x] : none, kS = q.y < nR ? R.nbr[q.y] : none;
    const int4 kN = q.z < nR ? R.nbr[q.z] : none, kE = q.w < nR ? R.nbr[q.w] : none;
    // A system in FP32 has all this formed in 64 bits from its couplings and rounded once: the differences
    // in cf[0] and g, in FP32, left an inner solution 0.7 to 1.4 times as far from the 64-bit one as A's own
    // FP32 rows do; this, 0.15 to 0.6 times.
    if constexpr (F32) {
      auto inv = [&](int k, const int4& e) { return 1.0 / (1.0 + R.sx[k] + B.sx[e.x] + R.sy[k] + B.sy[e.y]); };
      dW = inv(q.x, kW); dS = inv(q.y, kS); dN = inv(q.z, kN); dE = inv(q.w, kE);
    }
    // an absent red neighbour's coupling is zero: it drops out of every product
    const double gW = q.x < nR ? aW : 0.0, gS = q.y < nR ? aS : 0.0, gN = q.z < nR ? aN : 0.0, gE = q.w < nR ? aE : 0.0;
    const double hW = gW * dW, hS = gS * dS, hN = gN * dN, hE = gE * dE;
    const double diag = B.diag ? B.diag[j] : 1.0 + B.sx[j] + aW + B.sy[j] + aS;
    // couplings of red k to its own W, S, N, E: B.sx[k.W], B.sy[k.S], R.sy[k], R.sx[k]
    auto cN = [&](int k, const int4& e) -> double { return e.z < nB ? R.sy[k] : (T)0; };
    auto cE = [&](int k, const int4& e) -> double { return e.w < nB ? R.sx[k] : (T)0; };
    const int o[8] = {kW.x, min(kW.y, kS.x), kS.y, min(kS.w, kE.y), min(kW.z, kN.x), kN.z, min(kN.w, kE.z), kE.w};
    const double cf[9] = {diag - (((hW * gW + hS * gS) + hN * gN) + hE * gE),
                     -(hW * B.sx[kW.x]),
                     -(hW * B.sy[kW.y] + hS * B.sx[kS.x]),
                     -(hS * B.sy[kS.y]),
                     -(hS * cE(q.y, kS) + hE * B.sy[kE.y]),
                     -(hW * cN(q.x, kW) + hN * B.sx[kN.x]),
                     -(hN * cN(q.z, kN)),
                     -(hN * cE(q.z, kN) + hE * cN(q.w, kE)),
                     -(hE * cE(q.w, kE))};
    const T g = (T)(((hW * R.r[q.x] + hS * R.r[q.y]) + hN * R.r[q.z]) + hE * R.r[q.w]);
    const T rb = B.r[j], t = rb + g, d = B.dinv[j], zj = t * d;
    const bool res = i < nres;
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      if (res) s_cf[m * cap + i] = (T)cf[m];
      else P.cf[(size_t)m * nB + j] = (T)cf[m];
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int x = WIN ? (o[m] < nB ? o[m] - w0 : wz) : o[m];
      if (res) s_nb[m * cap + i] = (Idx)x;
      else P.nb8[(size_t)m * nB + j] = x;
    }
    rt_ = t; ru_ = B.u[j]; rg_ = g; rd_ = d;
    if (CL) s_z[i] = zj;
    else if (WIN) put_z(P.zt, j, zj, 1u);
    else z[j] = zj;
    v2[0] += (double)t * (double)zj;
    v2[1] += (double)rb * (double)rb;
  };
#pragma unroll
  for (int k = 0; k < RK; ++k) rt[k] = ru[k] = rv[k] = rg[k] = rd[k] = rp[k] = (T)0;
#pragma unroll 1
  for (int i = i0, k = 0; i < n; i += SB, ++k) {
    T t, u, g, d;
    row(i, t, u, g, d);
    if (k >= RK) {
      B.r[lo + i] = t;
      B.q[lo + i] = g;
    }
#pragma unroll
    for (int m = 0; m < RK; ++m)
      if (k == m) { rt[m] = t; ru[m] = u; rg[m] = g; rd[m] = d; }
  }
  if (WIN)
    for (int i = threadIdx.x; i <= wz; i += SB) s_w[i] = (T)0;
  for (int k = bid * SB + threadIdx.x; k < R.n; k += nb * SB) {
    const double r0 = (double)R.r[k];
    w2[0] += r0 * r0 * (double)R.dinv[k];
    w2[1] += r0 * r0;
  }
  if (CL) {
    cluster_sum<2>(w2, nb, turn, sh, s_tot, nothing);
    cluster_sum<2>(v2, nb, turn, sh, s_tot, cluster_halo);
  } else {
    if (!gather_sum<2, false, SB>(w2, bs, SC, sh)) return;
    // (with a fence in both forms: after it no tagged word of an earlier solve is left)
    if (!gather_sum<2, true, SB>(v2, bs, SC, sh)) return;
    if (WIN) {   // the first halo, now that no word of an earlier solve is left
      double none[1] = {0.0};
      if (!gather_sum<1, false, SB>(none, bs, SC, sh, fetch_halo)) return;
    }
  }
  // ONE: the thread's node's coefficients and neighbours in registers too
  T cfr[9];
  int nbr[8];
  if (ONE && i0 < n) {
#pragma unroll
    for (int m = 0; m < 9; ++m) cfr[m] = s_cf[m * cap + i0];
#pragma unroll
    for (int m = 0; m < 8; ++m) nbr[m] = s_nb[m * cap + i0];
  }
  const double gamma = w2[0], delta = w2[1];
  double alpha = SC->alpha, beta = SC->beta, rzdot = SC->rzdot, dkm1 = SC->dkm1, rho = 1.0, c = 0.0, rrt = 0.0;
  double rdk = 0.0;   // 1 / rzdot, formed while the next exchange is under way
  const double bnorm = SC->bnorm, stop = bnorm * SC->zeta, stop2 = stop * stop;
  int in = SC->in, ier = 0, par = 0;
  const int itmax = SC->itmax, hist_cap = SC->hist_cap;
  for (;;) {
    const double rzt = v2[0] + rho * rho * gamma;
    rrt = v2[1] + rho * rho * delta;
    dkm1 = rzdot;
    rzdot = rzt;
    if (!(rzt > 0.0)) { ier = -7; break; }
    if (rrt < stop2) break;   // test 5, |r| < |b| zeta, in squares
    if (!(in < itmax)) { ier = 1; break; }
    if (in != 0) beta = rzdot * rdk;
    rdk = 1.0 / rzdot;
    // ---- p = z + beta p (the neighbours' too, from their z and the old p) and S p
    const T bt = (T)beta;
    T* const po = par ? B.p2 : B.p;
    T* const pn = par ? B.p : B.p2;
    double pq[1] = {0.0};
    if (WIN) {
      for (int h = threadIdx.x; h < hl + hr; h += SB) {
        const int x = (h < hl ? lo - hl + h : lo + n + (h - hl)) - w0;
        s_w[x] = (CL && h < SB ? zh : s_h[h]) + bt * s_w[x];
      }
#pragma unroll
      for (int k = 0; k < RK; ++k) {
        rp[k] = rt[k] * rd[k] + bt * rp[k];
        if (i0 + k * SB < n) s_w[reach + i0 + k * SB] = rp[k];
      }
      for (int i = it; i < n; i += SB) s_w[reach + i] = B.r[lo + i] * B.dinv[lo + i] + bt * s_w[reach + i];
      __syncthreads();
    }
    // S p of node i, whose p is pi
    auto apply = [&](int i, T pi) -> T {
      const int j = lo + i;
      T cf[9];
      int o[8];
      if (ONE) {
#pragma unroll
        for (int m = 0; m < 9; ++m) cf[m] = cfr[m];
#pragma unroll
        for (int m = 0; m < 8; ++m) o[m] = nbr[m];
      } else if (i < nres) {
#pragma unroll
        for (int m = 0; m < 9; ++m) cf[m] = s_cf[m * cap + i];
#pragma unroll
        for (int m = 0; m < 8; ++m) o[m] = s_nb[m * cap + i];
      } else {
#pragma unroll
        for (int m = 0; m < 9; ++m) cf[m] = P.cf[(size_t)m * nB + j];
#pragma unroll
        for (int m = 0; m < 8; ++m) o[m] = P.nb8[(size_t)m * nB + j];
      }
      T p8[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) p8[m] = WIN ? s_w[o[m]] : z[o[m]] + bt * po[o[m]];
      const T ya = (cf[0] * pi + cf[1] * p8[0]) + cf[2] * p8[1];
      const T yb = (cf[3] * p8[2] + cf[4] * p8[3]) + cf[5] * p8[4];
      const T yc = (cf[6] * p8[5] + cf[7] * p8[6]) + cf[8] * p8[7];
      return (ya + yb) + yc;
    };
#pragma unroll
    for (int k = 0; k < RK; ++k) {
      const int i = i0 + k * SB;
      if (i < n) {
        if (!WIN) {
          rp[k] = rt[k] * rd[k] + bt * rp[k];
          pn[lo + i] = rp[k];
        }
        rv[k] = apply(i, rp[k]);
        pq[0] += (double)rp[k] * (double)rv[k];
      }
    }
    for (int i = it; i < n; i += SB) {
      const T pi = WIN ? s_w[reach + i] : z[lo + i] + bt * po[lo + i];
      if (!WIN) pn[lo + i] = pi;
      const T y = apply(i, pi);
      P.sv[lo + i] = y;
      pq[0] += (double)pi * (double)y;
    }
    if (CL) cluster_sum<1>(pq, nb, turn, sh, s_tot, nothing);
    else if (!gather_sum<1, false, SB>(pq, bs, SC, sh)) return;
    c = rho + beta * c;
    const double pap = pq[0] + c * c * gamma;
    alpha = rzdot / pap;
    if (!(pap > 0.0)) { ier = -6; break; }
    in += 1;
    par ^= 1;
    ++tag;
    rho -= alpha * c;
    // ---- u += alpha p, t -= alpha S p, z = P^-1 t
    const T al = (T)alpha, rh = (T)rho;
    v2[0] = v2[1] = 0.0;
    auto take = [&](int i, T t, T g, T d) {
      const T zj = t * d, rb = t - rh * g;
      if (CL) s_z[i] = zj;
      else if (WIN) put_z(P.zt, lo + i, zj, tag);
      else z[lo + i] = zj;
      v2[0] += (double)t * (double)zj;
      v2[1] += (double)rb * (double)rb;
    };
#pragma unroll
    for (int k = 0; k < RK; ++k) {
      rt[k] = rt[k] - al * rv[k];
      if (i0 + k * SB < n) take(i0 + k * SB, rt[k], rg[k], rd[k]);
      ru[k] = ru[k] + al * rp[k];
    }
    for (int i = it; i < n; i += SB) {
      const int j = lo + i;
      const T t = B.r[j] - al * P.sv[j];
      B.r[j] = t;
      B.u[j] = B.u[j] + al * (WIN ? s_w[reach + i] : pn[j]);
      take(i, t, B.q[j], B.dinv[j]);
    }
    if (CL) cluster_sum<2>(v2, nb, turn, sh, s_tot, cluster_halo);
    else if (!gather_sum<2, !WIN, SB>(v2, bs, SC, sh, fetch_halo)) return;
    // (here, far from the next exchange: the cluster's barrier waits for stores under way)
    if (bid == 0 && threadIdx.x == 0 && in <= hist_cap) { P.hist_alpha[in - 1] = alpha; P.hist_beta[in - 1] = beta; }
  }
  // ---- u of the black nodes, then of the red nodes: D u_R = b_R - rho r0_R + C u_B (b = r0 from u = 0)
#pragma unroll
  for (int k = 0; k < RK; ++k)
    if (i0 + k * SB < n) B.u[lo + i0 + k * SB] = ru[k];
  double done[1] = {0.0};
  if (CL) {
    __threadfence();
    cluster_barrier();   // (also: no block leaves while another may read its sums)
  } else if (!gather_sum<1, true, SB>(done, bs, SC, sh)) {
    return;
  }
  const T rh = (T)rho;
  for (int k = bid * SB + threadIdx.x; k < R.n; k += nb * SB) {
    const int4 q = R.nbr[k];
    const T r0 = R.r[k], b = R.rhs ? R.rhs[k] : r0;
    T y = b - rh * r0;
    y = y + B.sx[q.x] * B.u[q.x];
    y = y + B.sy[q.y] * B.u[q.y];
    y = y + R.sy[k] * B.u[q.z];
    y = y + R.sx[k] * B.u[q.w];
    R.u[k] = y * R.dinv[k];
  }
  if (bid == 0 && threadIdx.x == 0) {
    SC->alpha = alpha; SC->beta = beta; SC->rzdot = rzdot; SC->dkm1 = dkm1;
    SC->in = in; SC->stptst = sqrt(rrt) / bnorm;
    if (ier) SC->ier = ier;
    SC->done = 1;
  }
}

// The form depends on the nodes per block and the reach alone, so every block of a system takes the same.
template <typename T>
__device__ __forceinline__ void schur_any(const PcgDevT<T>& P, GridBar* bar, int bid, int nb, int smem) {
  const int per = (P.B.n + nb - 1) / nb;
  const long long all = window_bytes<T>(per, P.reach) + (long long)((per + 1) / 2 * 2) * node_bytes<T, true>();
  if (!window_fits<T>(per, nb, P.reach)) schur_body<T, false, false>(P, bar, bid, nb, smem);
  else if (per <= SB && all <= smem) schur_body<T, true, true>(P, bar, bid, nb, smem);
  else schur_body<T, true, false>(P, bar, bid, nb, smem);
}

template <typename T>
__global__ void __launch_bounds__(SB, 1) k_schur_loop(PcgDevT<T> P, GridBar* bar, int smem) {
  schur_any<T>(P, bar, blockIdx.x, gridDim.x, smem);
}

template <typename T>
__global__ void __launch_bounds__(SB, 1) k_schur_cluster(PcgDevT<T> P, int smem) {
  schur_body<T, true, true, true>(P, nullptr, blockIdx.x, gridDim.x, smem);
}

// The FP64 loops of an ensemble's basins in one cooperative launch: basin m's system is solved by
// blocks [first, first + nblk) of the grid with its own barrier record and slots, so each basin
// iterates to its own convergence and the launch ends when the last one has.
__global__ void __launch_bounds__(SB, 1) k_schur_loop_ens(const PcgEnsItem* __restrict__ items, int nitems, int smem) {
  __shared__ __align__(16) unsigned char s_buf[sizeof(PcgEnsItem)];
  __shared__ int s_m;
  PcgEnsItem& s_it = *reinterpret_cast<PcgEnsItem*>(s_buf);
  if (threadIdx.x == 0) {
    int m = -1;
    for (int i = 0; i < nitems && m < 0; ++i)
      if ((int)blockIdx.x >= items[i].first && (int)blockIdx.x < items[i].first + items[i].nblk) m = i;
    s_m = m;
    if (m >= 0) s_it = items[m];
  }
  __syncthreads();
  if (s_m < 0) return;
  schur_any<double>(s_it.P, s_it.bar, (int)blockIdx.x - s_it.first, s_it.nblk, smem);
}

int coop_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int nblocks, int smem, cudaStream_t st) {
  cfg = {};
  cfg.gridDim = dim3(nblocks);
  cfg.blockDim = dim3(SB);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return 0;
}

template <typename T>
int launch_schur(const PcgDevT<T>& P, GridBar* bar, int nblocks, cudaStream_t st, const GridBar* init) {
  const int per = (P.B.n + nblocks - 1) / nblocks;
  const int pe = (std::max(per, 2) + 1) / 2 * 2;
  const long long win = window_bytes<T>(per, P.reach) + (long long)pe * node_bytes<T, true>();
  // Up to eight blocks (4096 nodes) run as one cluster, when all of a block fits its shared memory; the
  // test hook of the barriers' limit keeps to the grid's barriers.  More blocks than the portable cluster
  // size have the grid's exchanges.
  if (nblocks > 1 && nblocks <= kClusterMax && per <= SB && !init && win + (long long)per * (int)sizeof(T) <= kSmemMax) {
    const int smem = (int)(win + (long long)per * (int)sizeof(T));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(SB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nblocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_schur_cluster<T>, P, smem) == cudaSuccess ? 0 : -1;
  }
  if (init) {
    if (cudaMemcpyAsync(bar, init, sizeof(GridBar), cudaMemcpyHostToDevice, st) != cudaSuccess) return -1;
  } else if (cudaMemsetAsync(bar, 0, sizeof(GridBar), st) != cudaSuccess) {
    return -1;
  }
  const size_t pitch = sizeof(uint4) * (size_t)slot_plane(P.slot_blocks);
  if (cudaMemset2DAsync(P.slots, pitch, 0, sizeof(uint4) * (size_t)nblocks, 2 * kSlotVals, st) != cudaSuccess) return -1;
  const int smem = (int)std::min<long long>(kSmemMax, window_fits<T>(per, nblocks, P.reach) ? win : (long long)pe * node_bytes<T, false>());
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  coop_config(cfg, attr, nblocks, smem, st);
  return cudaLaunchKernelEx(&cfg, k_schur_loop<T>, P, bar, smem) == cudaSuccess ? 0 : -1;
}

}  // namespace

int schur_init() {
  if (cudaFuncSetAttribute(k_schur_loop<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
      cudaFuncSetAttribute(k_schur_loop<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
      cudaFuncSetAttribute(k_schur_cluster<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
      cudaFuncSetAttribute(k_schur_cluster<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
      cudaFuncSetAttribute(k_schur_loop_ens, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess)
    return -1;
  return 0;
}

// One block per SM at most, and no block with fewer nodes than threads.
int schur_blocks(int device, int nB) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return std::max(1, std::min(sms, (nB + SB - 1) / SB));
}

size_t schur_slots(int nblocks) { return slot_count(nblocks); }

int schur_loop(const PcgDev& P, GridBar* bar, int nblocks, cudaStream_t st, const GridBar* init) {
  return launch_schur<double>(P, bar, nblocks, st, init);
}

int schur_loop_f(const PcgDevF& F, GridBar* bar, int nblocks, cudaStream_t st, const GridBar* init) {
  return launch_schur<float>(F, bar, nblocks, st, init);
}

int pcg_loop_ens_blocks(int device) {
  int sms = 0, occ = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_schur_loop_ens, SB, kSmemMax);
  return sms * std::max(occ, 0);
}

int pcg_loop_ens(const PcgEnsItem* items, int nitems, int nblocks, GridBar* bars, uint4* slots, size_t slot_bytes,
                 cudaStream_t st) {
  if (cudaMemsetAsync(bars, 0, sizeof(GridBar) * (size_t)nitems, st) != cudaSuccess) return -1;
  if (cudaMemsetAsync(slots, 0, slot_bytes, st) != cudaSuccess) return -1;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  coop_config(cfg, attr, nblocks, kSmemMax, st);
  return cudaLaunchKernelEx(&cfg, k_schur_loop_ens, items, nitems, kSmemMax) == cudaSuccess ? 0 : -1;
}

}  // namespace si3d
