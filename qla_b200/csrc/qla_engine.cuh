// qla_engine.cuh -- the site-loop engine behind every level-1 QLA operator.
//
// QLA's generated functions are loops `for(i<n)` over AoS site records
// (lib/perl/formatting.pl:90-127).  On B200 such a loop is HBM-bound, and
// AoS records of 24/48/72/96 B are awkward for per-thread coalescing.  The
// engine therefore moves whole tiles of T consecutive sites of every
// contiguous operand with 1-D bulk (TMA) copies into shared memory, in an
// S-stage mbarrier pipeline, computes one site per thread from shared memory,
// and writes the destination tile back with one bulk store.  Operands reached
// through a pointer array (`pX`, 8 B per site) or an int32 index stream
// (`xX`, 4 B per site) stream their pointer/index tile through the same
// pipeline and gather the records with per-thread read-only loads.
//
// A second, warp-cooperative kernel runs the gang-index `x` variants, whose
// every operand is scattered, and any call whose pointers are not 16-B
// aligned (bulk copies require 16-B alignment); a third runs one site per
// thread, for operators and calls that either of these would slow down.  The
// kernels share the per-site code, so their results are identical.
//
// An operator type OP provides:
//   using R;                               site real type (float/double)
//   NIN, N0, N1, N2                        number of inputs, complex numbers per input record
//   NOUT                                   complex numbers per destination record (0 = none)
//   NACC                                   number of double accumulators (0 = not a reduction)
//   apply(p, x0, x1, x2, y)                destination record y (pre-loaded when p.out_read)
//   accum(p, x0, x1, x2, acc)              reduction contribution of one site
#pragma once
#include "qla_core.cuh"

namespace qlab {

enum OpndMode : int { OM_NONE = 0, OM_CONTIG = 1, OM_PTR = 2, OM_IDX = 3 };

struct Opnd {
  const void* base;         // CONTIG / IDX: record array
  const void* const* ptrs;  // PTR: device array of record pointers (one per site)
  const int* idx;           // IDX: int32 record index per site
  int mode;
};

struct SiteParams {
  Opnd in[3];
  void* out;         // destination field (record array)
  int out_read;      // destination is also read (peq / meq)
  const int* gang;   // gang index (x variants): site k = gang[i]
  long long n;       // loop length
  int eqop, mu, sign, aux;
  double sval, sval_im;  // scalar argument passed by value (host scalar)
  const void* sptr;      // scalar argument left on the device (read by the kernel)
  // reductions
  DD* partials;
  unsigned* counter;
  void* result;      // device address receiving the reduced value(s)
  unsigned* err;     // device error word (QLA_DEVERR_* bits)
  // bulk-copy pipeline layout (host-computed)
  unsigned stage_bytes, tx_bytes;
  unsigned off_in[3], off_out_in;
  int stages;        // pipeline depth S (1..8)
  long long ntiles;  // number of full tiles of T sites
};

template <int N>
struct ArrN {
  static constexpr int value = N > 0 ? N : 1;
};

// ---------------------------------------------------------------------------
// per-site work shared by both kernels

template <class OP, int N>
__device__ __forceinline__ void fetch_gathered(Cx<typename OP::R> (&x)[ArrN<N>::value], const Opnd& o, long long k) {
  using R = typename OP::R;
  constexpr int RB = N * (int)sizeof(Cx<R>);
  const void* src;
  if (o.mode == OM_PTR)
    src = o.ptrs[k];
  else if (o.mode == OM_IDX)
    src = static_cast<const char*>(o.base) + (long long)o.idx[k] * RB;
  else
    src = static_cast<const char*>(o.base) + k * RB;
  if constexpr (OP::NIN > 1)
    load_rec_here<R, ArrN<N>::value>(x, src);
  else
    load_rec_global<R, ArrN<N>::value>(x, src);
}

// Direct path: all operands read straight from global memory for site k.
template <class OP>
__device__ __forceinline__ void site_direct(const SiteParams& p, long long k, double* acc) {
  using R = typename OP::R;
  Cx<R> x0[ArrN<OP::N0>::value], x1[ArrN<OP::N1>::value], x2[ArrN<OP::N2>::value];
  if constexpr (OP::NIN > 0) fetch_gathered<OP, OP::N0>(x0, p.in[0], k);
  if constexpr (OP::NIN > 1) fetch_gathered<OP, OP::N1>(x1, p.in[1], k);
  if constexpr (OP::NIN > 2) fetch_gathered<OP, OP::N2>(x2, p.in[2], k);
  if constexpr (OP::NOUT > 0) {
    constexpr int OB = OP::NOUT * (int)sizeof(Cx<R>);
    char* dst = static_cast<char*>(p.out) + k * OB;
    Cx<R> y[OP::NOUT];
    if (p.out_read) load_rec_rw<R, OP::NOUT>(y, dst);
    OP::apply(p, x0, x1, x2, y);
    store_rec<R, OP::NOUT>(dst, y);
  } else {
    OP::accum(p, x0, x1, x2, acc);
  }
}

// Staged path: contiguous operands come from the shared-memory tile `st`,
// pointer/index operands take their pointer/index from the tile and gather.
template <class OP, int N>
__device__ __forceinline__ void fetch_staged(Cx<typename OP::R> (&x)[ArrN<N>::value], const Opnd& o,
                                             const unsigned char* st, unsigned off, int t) {
  using R = typename OP::R;
  constexpr int RB = N * (int)sizeof(Cx<R>);
  if (o.mode == OM_CONTIG) {
    load_rec<R, ArrN<N>::value>(x, st + off + (unsigned)t * RB);
  } else if (o.mode == OM_PTR) {
    const void* src = reinterpret_cast<const void* const*>(st + off)[t];
    load_rec_global<R, ArrN<N>::value>(x, src);
  } else {
    const int j = reinterpret_cast<const int*>(st + off)[t];
    load_rec_global<R, ArrN<N>::value>(x, static_cast<const char*>(o.base) + (long long)j * RB);
  }
}

// Block-level reduction of NACC double-double accumulators into the
// per-block partial slots, then a last-block-done finish that writes the
// total to p.result.  The summation order depends only on the grid, so
// results are deterministic run to run on a given device.
template <class OP>
__device__ void reduce_finish(const SiteParams& p, DD (&acc)[ArrN<OP::NACC>::value]) {
  constexpr int NA = ArrN<OP::NACC>::value;
  __shared__ DD red[32][NA];
  __shared__ bool is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int a = 0; a < NA; a++) {
    for (int m = 16; m >= 1; m >>= 1) dd_merge(acc[a], dd_shfl_xor(acc[a], m));
    if (lane == 0) red[warp][a] = acc[a];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int a = 0; a < NA; a++) {
      DD s = red[0][a];
      for (int w = 1; w < nwarps; w++) dd_merge(s, red[w][a]);
      p.partials[(long long)blockIdx.x * NA + a] = s;
    }
    __threadfence();
    unsigned ticket = atomicAdd(p.counter, 1u);
    is_last = (ticket == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // last block: fold the partials in a fixed order
  DD s[NA];
  for (int a = 0; a < NA; a++) s[a] = DD{0.0, 0.0};
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
    for (int a = 0; a < NA; a++) {
      volatile DD* vp = reinterpret_cast<volatile DD*>(&p.partials[(long long)b * NA + a]);
      DD v;
      v.hi = vp->hi;
      v.lo = vp->lo;
      dd_merge(s[a], v);
    }
  for (int a = 0; a < NA; a++) {
    for (int m = 16; m >= 1; m >>= 1) dd_merge(s[a], dd_shfl_xor(s[a], m));
    if (lane == 0) red[warp][a] = s[a];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot[NA];
    for (int a = 0; a < NA; a++) {
      DD t = red[0][a];
      for (int w = 1; w < nwarps; w++) dd_merge(t, red[w][a]);
      tot[a] = __dadd_rn(t.hi, t.lo);
    }
    OP::finish(p, tot);
    *p.counter = 0u;  // ready for the next launch on this scratch
  }
}

template <class OP>
__device__ __forceinline__ void acc_fold(DD (&dacc)[ArrN<OP::NACC>::value], const double* acc) {
#pragma unroll
  for (int a = 0; a < ArrN<OP::NACC>::value; a++) dd_add(dacc[a], acc[a]);
}

// ---------------------------------------------------------------------------
// Kernel 1: bulk-copy (TMA) pipeline, persistent, warp-specialised.
//
// Block = NW consumer warps (one site per lane per tile, T = 32*NW sites per
// tile) + 1 producer warp.  Per stage s there is a `full` mbarrier (completed
// by the bulk-copy transaction bytes) and an `empty` mbarrier (one arrival
// per consumer warp once it has read the stage).  The producer lane waits on
// `empty`, re-arms `full` and issues the next tile's loads; consumer warps
// wait on `full`, compute, release the stage, and write their 32 results
// through a per-warp double-buffered shared-memory slice with their own bulk
// store.  No block-wide barrier sits in the tile loop, so every warp runs at
// its own pace and the next loads go out as soon as a stage is released.
//
// Dynamic shared memory: [full[S], empty[S], abort flag | S stages |
//                         NW x 2 destination slices of 32 records].
// Every wait is time-bounded; a failed wait raises the abort flag so that all
// other waits of the block give up at once, and loads still in flight are
// drained (bounded) before the block exits.
template <class OP>
__global__ void __launch_bounds__(288) site_tma_kernel(const SiteParams p) {
  using R = typename OP::R;
  constexpr int OB = OP::NOUT * (int)sizeof(Cx<R>);
  constexpr int NA = ArrN<OP::NACC>::value;
  extern __shared__ __align__(128) unsigned char smem[];
  overlap_begin();
  const int S = p.stages;
  const int NW = (blockDim.x >> 5) - 1;  // consumer warps
  const int T = NW * 32;                 // sites per tile
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + 8;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 8 * 16);
  unsigned char* stages = smem + 256;
  unsigned char* outbuf = stages + (size_t)S * p.stage_bytes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long my =
      ((long long)blockIdx.x < p.ntiles) ? (p.ntiles - 1 - (long long)blockIdx.x) / gridDim.x + 1 : 0;

  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], (unsigned)NW);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();

  DD dacc[NA];
#pragma unroll
  for (int a = 0; a < NA; a++) dacc[a] = DD{0.0, 0.0};
  bool alive = true;
  long long issued = 0;  // tiles whose loads the producer issued

  if (warp == NW) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      const uint64_t pol = policy_evict_first();
      constexpr int RB[3] = {OP::N0 * (int)sizeof(Cx<R>), OP::N1 * (int)sizeof(Cx<R>),
                             OP::N2 * (int)sizeof(Cx<R>)};
      long long k = 0;
      int s = 0;
      long long round = 0;  // k / S
      for (; k < my; k++) {
        // stage s was last filled in round-1; wait until its consumers released it
        if (round > 0 && !mbar_wait_bounded(&empty[s], (uint32_t)((round - 1) & 1), p.err, 2000000000ull,
                                            abort_flag)) {
          *abort_flag = 1;
          break;
        }
        const long long site0 = ((long long)blockIdx.x + k * gridDim.x) * T;
        unsigned char* st = stages + (size_t)s * p.stage_bytes;
        mbar_arrive_expect_tx(&full[s], p.tx_bytes);
#pragma unroll
        for (int j = 0; j < OP::NIN; j++) {
          const Opnd& o = p.in[j];
          if (o.mode == OM_CONTIG)
            bulk_g2s(st + p.off_in[j], static_cast<const char*>(o.base) + site0 * RB[j], (unsigned)T * RB[j],
                     &full[s], pol);
          else if (o.mode == OM_PTR)
            bulk_g2s(st + p.off_in[j], o.ptrs + site0, (unsigned)T * 8u, &full[s], pol);
          else
            bulk_g2s(st + p.off_in[j], o.idx + site0, (unsigned)T * 4u, &full[s], pol);
        }
        if constexpr (OP::NOUT > 0) {
          if (p.out_read)
            bulk_g2s(st + p.off_out_in, static_cast<const char*>(p.out) + site0 * OB, (unsigned)T * OB, &full[s],
                     pol);
        }
        if (++s == S) {
          s = 0;
          round++;
        }
      }
      issued = k;
    }
  } else {
    // ------------------------------------------------------------ consumers
    const uint64_t pol = policy_evict_first();
    unsigned char* myout = outbuf + (size_t)warp * 2 * 32 * OB;
    int s = 0;
    uint32_t par = 0;
    for (long long k = 0; k < my; k++) {
      if (!mbar_wait_bounded(&full[s], par, p.err, 2000000000ull, abort_flag)) {
        *abort_flag = 1;
        alive = false;
        break;
      }
      const unsigned char* st = stages + (size_t)s * p.stage_bytes;
      const int t = warp * 32 + lane;
      Cx<R> x0[ArrN<OP::N0>::value], x1[ArrN<OP::N1>::value], x2[ArrN<OP::N2>::value];
      Cx<R> y[ArrN<OP::NOUT>::value];
      if constexpr (OP::NIN > 0) fetch_staged<OP, OP::N0>(x0, p.in[0], st, p.off_in[0], t);
      if constexpr (OP::NIN > 1) fetch_staged<OP, OP::N1>(x1, p.in[1], st, p.off_in[1], t);
      if constexpr (OP::NIN > 2) fetch_staged<OP, OP::N2>(x2, p.in[2], st, p.off_in[2], t);
      if constexpr (OP::NOUT > 0) {
        if (p.out_read) load_rec<R, OP::NOUT>(y, st + p.off_out_in + (unsigned)t * OB);
      }
      if constexpr (OP::NOUT > 0) {
        OP::apply(p, x0, x1, x2, y);
        unsigned char* ob = myout + (size_t)(k & 1) * 32 * OB;
        if (lane == 0) bulk_wait_read<1>();  // slice (k&1) no longer read by this warp's store k-2
        __syncwarp();
        store_rec_smem<R, OP::NOUT>(ob + (unsigned)lane * OB, y);
        // every lane orders its reads of the stage and its writes of the
        // slice before the async proxy: the slice's bulk store below, and
        // the producer's next bulk copy into the stage released here
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&empty[s]);  // this warp is done with the stage
          const long long site0 = ((long long)blockIdx.x + k * gridDim.x) * T + warp * 32;
          bulk_s2g(static_cast<char*>(p.out) + site0 * OB, ob, 32u * OB, pol);
          bulk_commit();
        }
      } else {
        release_stage(&empty[s], lane);  // this warp is done with the stage
        double acc[NA];
        OP::accum(p, x0, x1, x2, acc);
        acc_fold<OP>(dacc, acc);
      }
      if (++s == S) {
        s = 0;
        par ^= 1u;
      }
    }
    if constexpr (OP::NOUT > 0) {
      if (lane == 0) bulk_wait_all<0>();
    }
    // partial last tile: plain loads by the consumers of the last block
    if (alive && blockIdx.x == gridDim.x - 1) {
      const long long k0 = p.ntiles * T + warp * 32 + lane;
      if (k0 < p.n) {
        double acc[NA];
        site_direct<OP>(p, k0, acc);
        if constexpr (OP::NACC > 0) acc_fold<OP>(dacc, acc);
      }
    }
  }
  __syncthreads();
  if (*abort_flag && warp == NW && lane == 0) {
    // a wait failed: before the block's shared memory is released, wait
    // (bounded) until every load still in flight has landed
    for (long long kk = (issued > S ? issued - S : 0); kk < issued; kk++)
      if (!mbar_wait_bounded(&full[kk % S], (uint32_t)((kk / S) & 1), p.err, 200000000ull, nullptr))
        raise_dev_error(p.err, QLA_DEVERR_BULK_TIMEOUT);
  }
  // every block takes part in the finish, even after a failed wait, so that
  // the ticket counter returns to zero (the error word marks the result invalid)
  if constexpr (OP::NACC > 0) reduce_finish<OP>(p, dacc);
}

// ---------------------------------------------------------------------------
// Kernel 2: warp-cooperative, for the gang-index variants (every operand
// scattered) and operands that a bulk copy cannot move (not 16-B aligned).
//
// A warp takes 32 sites at a time.  Its lanes copy the sites' records into
// the warp's shared-memory slice with cp.async, piece by piece: consecutive
// lanes take consecutive 16-B (or 8-B) pieces of one record, so one
// instruction touches 4 to 10 records' lines instead of 32 (a thread reading
// its own record makes every instruction touch 32 lines, and the L1 then
// spends a cycle on each: that bound the one-site-per-thread form).  Then
// each lane computes one site from shared memory, and results leave the same
// way.  The gang index and the operands' pointers or indices of the next 32
// sites are loaded while the records are in flight, which takes two of the
// three dependent latencies out of the loop.  Shared record slots hold an odd
// number of 16-B (8-B) units: conflict-free for one record per lane.
// Measured, QLA_F3_D_xpeq_spproj_pMa_times_pD on the even sites of
// 32^3 x 64: 142 us with one site per thread, 112 so (5.9-6.0 TB/s of
// DRAM traffic: alternate records share their 64-B granules).
template <int RB>
struct CoopSlot {  // shared bytes of one record slot
  static constexpr unsigned value = (RB % 16 == 0 && (RB / 16) % 2 == 0) ? RB + 16 : RB;
};
template <class OP>
struct CoopLayout {
  using R = typename OP::R;
  static constexpr int C = (int)sizeof(Cx<R>);
  static constexpr unsigned S0 = OP::NIN > 0 ? CoopSlot<OP::N0 * C>::value : 0,
                            S1 = OP::NIN > 1 ? CoopSlot<OP::N1 * C>::value : 0,
                            S2 = OP::NIN > 2 ? CoopSlot<OP::N2 * C>::value : 0,
                            SO = OP::NOUT > 0 ? CoopSlot<OP::NOUT * C>::value : 0;
  static constexpr unsigned o1 = 32 * S0, o2 = o1 + 32 * S1, oo = o2 + 32 * S2;
  static constexpr unsigned warp_bytes = oo + 32 * SO;  // each part is a multiple of 256 B
};

// address of operand o's record of site k
template <class OP, int N>
__device__ __forceinline__ const char* rec_addr(const Opnd& o, long long k) {
  constexpr int RB = N * (int)sizeof(Cx<typename OP::R>);
  if (o.mode == OM_PTR) return static_cast<const char*>(o.ptrs[k]);
  return static_cast<const char*>(o.base) + (o.mode == OM_IDX ? (long long)o.idx[k] : k) * RB;
}

// Walk over the pieces of 32 records (P pieces each), a piece per lane:
// f(record, piece, live).  Records of up to 16 pieces go 32 / P at a time, so
// that a lane keeps its piece number and its addresses advance by constants;
// longer records in one run.  Every lane makes every call, so f may shuffle.
// (The empty asm keeps the offsets from being held in registers across the
// site loop.)
template <int P, class F>
__device__ __forceinline__ void for_pieces(int lane, F&& f) {
  asm volatile("" : "+r"(lane));
  if constexpr (P <= 16) {
    constexpr int G = 32 / P, ITS = (32 + G - 1) / G;
    const int r0 = lane / P, pc = lane - r0 * P;
#pragma unroll
    for (int it = 0; it < ITS; it++) f(it * G + r0, pc, r0 < G);
  } else {
#pragma unroll 4
    for (int it = 0; it < P; it++) {
      const int q = it * 32 + lane;
      f(q / P, q % P, true);
    }
  }
}

// copies the records at `addr` (one per lane, the first nv lanes valid) into slots
template <int RB>
__device__ __forceinline__ void coop_fetch(unsigned char* slots, const char* addr, int nv, int lane) {
  constexpr unsigned SL = CoopSlot<RB>::value;
  const unsigned long long a = reinterpret_cast<unsigned long long>(addr);
  const bool wide = RB % 16 == 0 && __all_sync(0xffffffffu, lane >= nv || (a & 15u) == 0);
  if (wide) {
    for_pieces<(RB % 16 == 0 ? RB / 16 : 1)>(lane, [&](int r, int pc, bool live) {
      const char* src = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, a, r & 31)) + pc * 16;
      if (live && r < nv) cp_async_16(slots + r * SL + pc * 16, src);
    });
  } else {
    for_pieces<RB / 8>(lane, [&](int r, int pc, bool live) {
      const char* src = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, a, r & 31)) + pc * 8;
      if (live && r < nv) cp_async_8(slots + r * SL + pc * 8, src);
    });
  }
}

// writes the records in the slots to `addr` (one per lane)
template <int RB>
__device__ __forceinline__ void coop_store(const unsigned char* slots, char* addr, int nv, int lane) {
  constexpr unsigned SL = CoopSlot<RB>::value;
  const unsigned long long a = reinterpret_cast<unsigned long long>(addr);
  const bool wide = RB % 16 == 0 && __all_sync(0xffffffffu, lane >= nv || (a & 15u) == 0);
  if (wide) {
    for_pieces<(RB % 16 == 0 ? RB / 16 : 1)>(lane, [&](int r, int pc, bool live) {
      char* dst = reinterpret_cast<char*>(__shfl_sync(0xffffffffu, a, r & 31)) + pc * 16;
      if (live && r < nv) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(slots + r * SL + pc * 16);
    });
  } else {
    for_pieces<RB / 8>(lane, [&](int r, int pc, bool live) {
      char* dst = reinterpret_cast<char*>(__shfl_sync(0xffffffffu, a, r & 31)) + pc * 8;
      if (live && r < nv) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(slots + r * SL + pc * 8);
    });
  }
}

// Operators whose arithmetic outweighs their bytes (specialised beside them)
// run on this kernel too: every thread computes, and up to 255 registers each.
template <class OP>
struct ComputeBound {
  static constexpr bool value = false;
};
// Operators that run one site per thread on global memory (specialised beside
// them): `contiguous` for aligned arrays too, `scattered` for gang-index calls
// and operands off a 16-B boundary.
template <class OP>
struct SitePerThread {
  static constexpr bool contiguous = false, scattered = false;
};
// Operators with slots so large that only three or four warps fit on an SM, where
// they lose to one site per thread (specialised beside them).
template <class OP>
struct FewWarps {
  static constexpr bool value = false;
};
// Operators whose arithmetic hides behind the movement of their records even
// with half the usual warps (specialised beside them).
template <class OP>
struct StreamsRecords {
  static constexpr bool value = false;
};
// Blocks of 128 threads an SM must hold, by the 32-bit registers that one
// site's records fill: 5 (102 registers), 3 (168) or 1 (255).  (Left to itself
// the compiler spills the 8-colour matrix products: 211 us against 55.)
template <class OP>
constexpr int coop_min_blocks() {
  constexpr int live = (OP::N0 + OP::N1 + OP::N2 + OP::NOUT) * (int)sizeof(Cx<typename OP::R>) / 4;
  return ComputeBound<OP>::value || live > 160 ? 1 : live > 70 ? 3 : 5;
}

template <class OP>
__global__ void __launch_bounds__(128, coop_min_blocks<OP>()) site_coop_kernel(const SiteParams p) {
  using R = typename OP::R;
  using L = CoopLayout<OP>;
  constexpr int NA = ArrN<OP::NACC>::value, C = (int)sizeof(Cx<R>);
  extern __shared__ __align__(128) unsigned char smem[];
  overlap_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned char* sl = smem + (size_t)warp * L::warp_bytes;
  DD dacc[NA];
#pragma unroll
  for (int a = 0; a < NA; a++) dacc[a] = DD{0.0, 0.0};
  const long long step = (long long)gridDim.x * nw * 32;
  const char *a0 = nullptr, *a1 = nullptr, *a2 = nullptr;
  char* ao = nullptr;
  auto addresses = [&](long long i) {  // this lane's record addresses for loop position i
    if (i >= p.n) return;
    const long long k = p.gang ? (long long)p.gang[i] : i;
    if constexpr (OP::NIN > 0) a0 = rec_addr<OP, OP::N0>(p.in[0], k);
    if constexpr (OP::NIN > 1) a1 = rec_addr<OP, OP::N1>(p.in[1], k);
    if constexpr (OP::NIN > 2) a2 = rec_addr<OP, OP::N2>(p.in[2], k);
    if constexpr (OP::NOUT > 0) ao = static_cast<char*>(p.out) + k * (OP::NOUT * C);
  };
  long long i0 = ((long long)blockIdx.x * nw + warp) * 32;
  addresses(i0 + lane);
  for (; i0 < p.n; i0 += step) {
    const int nv = p.n - i0 < 32 ? (int)(p.n - i0) : 32;
    if constexpr (OP::NIN > 0) coop_fetch<OP::N0 * C>(sl, a0, nv, lane);
    if constexpr (OP::NIN > 1) coop_fetch<OP::N1 * C>(sl + L::o1, a1, nv, lane);
    if constexpr (OP::NIN > 2) coop_fetch<OP::N2 * C>(sl + L::o2, a2, nv, lane);
    char* dst = ao;
    if constexpr (OP::NOUT > 0) {
      if (p.out_read) coop_fetch<OP::NOUT * C>(sl + L::oo, ao, nv, lane);
    }
    addresses(i0 + step + lane);
    cp_async_wait_all();
    __syncwarp();
    if (lane < nv) {
      Cx<R> x0[ArrN<OP::N0>::value], x1[ArrN<OP::N1>::value], x2[ArrN<OP::N2>::value];
      if constexpr (OP::NIN > 0) load_rec<R, ArrN<OP::N0>::value>(x0, sl + lane * L::S0);
      if constexpr (OP::NIN > 1) load_rec<R, ArrN<OP::N1>::value>(x1, sl + L::o1 + lane * L::S1);
      if constexpr (OP::NIN > 2) load_rec<R, ArrN<OP::N2>::value>(x2, sl + L::o2 + lane * L::S2);
      if constexpr (OP::NOUT > 0) {
        Cx<R> y[OP::NOUT];
        if (p.out_read) {
          load_rec<R, OP::NOUT>(y, sl + L::oo + lane * L::SO);
        } else {  // (undefined, it would stay live around the loop)
#pragma unroll
          for (int e = 0; e < OP::NOUT; e++) y[e] = Cx<R>{R(0), R(0)};
        }
        OP::apply(p, x0, x1, x2, y);
        store_rec_smem<R, OP::NOUT>(sl + L::oo + lane * L::SO, y);
      } else {
        double acc[NA];
        OP::accum(p, x0, x1, x2, acc);
        acc_fold<OP>(dacc, acc);
      }
    }
    __syncwarp();  // results in the slots; every lane is done with the inputs
    if constexpr (OP::NOUT > 0) {
      coop_store<OP::NOUT * C>(sl + L::oo, dst, nv, lane);
      __syncwarp();  // the slots are free for the next 32 sites
    }
  }
  if constexpr (OP::NACC > 0) reduce_finish<OP>(p, dacc);
}

// Kernel 3: one site per thread, records read and written where they lie, up to
// 255 registers a thread.  For operators whose arithmetic on one site outweighs
// its bytes and needs more registers, or more local memory, than the warps that
// share shared-memory slots can have (SitePerThread), for scattered calls whose
// records are too short or too long for those slots (SiteLauncher), and for the
// allocation-free entry point's unaligned calls.  Operators of two inputs load with ld_here: into
// local arrays, plain loads of the second record wait for the first one's stores
// (QLA_DN_M_xeq_M_inverse_M, nc = 8, 23,438 sites: 159 us with __ldg, 237 plain).
template <class OP>
__global__ void __launch_bounds__(256) site_direct_kernel(const SiteParams p) {
  overlap_begin();
  constexpr int NA = ArrN<OP::NACC>::value;
  DD dacc[NA];
#pragma unroll
  for (int a = 0; a < NA; a++) dacc[a] = DD{0.0, 0.0};
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += stride) {
    const long long k = p.gang ? (long long)p.gang[i] : i;
    double acc[NA];
    site_direct<OP>(p, k, acc);
    if constexpr (OP::NACC > 0) acc_fold<OP>(dacc, acc);
  }
  if constexpr (OP::NACC > 0) reduce_finish<OP>(p, dacc);
}

}  // namespace qlab
